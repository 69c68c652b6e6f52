// Circulant convolutions of the voxel Lp / P Toeplitz blocks, family-combined.
//
// The operator's circulant blocks act between six lattice families: three face
// families of the P tensor (reference families 12, 34, 56) and three edge
// directions of the Lp tensor. Every P block (three diagonal, three cross blocks
// applied in both directions) is a Toeplitz operator between two face families, and
// all six share one circulant grid L_P, so the P part of an operator application is
//   for each face family g: X_g = FFT3(x_g)            (3 forward transforms)
//   for each frequency:     Y_f = sum_g S_fg X_g       (3x3 Hermitian spectral matrix)
//   for each face family f: y_f = IFFT3(Y_f)           (3 inverse transforms)
// instead of the reference's twelve transform pairs. The Lp blocks are diagonal in
// the edge direction and keep one forward/inverse pair each.
//
// Each 3-D transform runs as passes over one axis at a time on a per-family buffer
// T_f[z][y][kx] (kx fastest, Lx x Ly x nz_f), in place: x forward (gather of the family's
// compact vector through its lattice map), y forward, z (forward, spectral product, inverse),
// y inverse, x inverse (plain store into the compact output through the lattice map; each
// compact index belongs to exactly one family). Only the occupied lattice octant is
// transformed in each pass (pruning). Two sets of kernels (fftconv_impl.cuh):
//   pair     k_xpair, k_ypair, k_zpair / k_zpair_wide: the even and the odd frequencies as
//            transforms of half the length on the occupied entries, in registers (FP32 and
//            float-float, up to 512 points along x and y and 128 along z)
//   direct   k_xfwd, k_ypass, k_zconv3 / k_zconv1, k_xinv: the padded lines in radix groups
//            (fft_reg.cuh), the first and last ones straight from and to global memory, the
//            middle ones in shared-memory tiles with contiguous sequences (element (pos, seq)
//            at pos*rs + seq, bank-conflict free); FP64 and longer lines. The staged z passes
//            are the direct ones with bulk-copied tiles.
// Spectra carry the 1/(Lx*Ly*Lz) normalisation (Spectrum).
#include <mutex>
#include <set>
#include <utility>

#include <algorithm>

#include "ctx.hpp"
#include "fft_reg.cuh"

namespace peec {

int conv_all_f32(const Family*, int, const Spectrum*, const void* const*, const c64*, c64*,
                 c64*, int64_t, const void*, int, cudaStream_t, cudaEvent_t*, const ZTune*);
int conv_all_f64(const Family*, int, const Spectrum*, const void* const*, const c64*, c64*,
                 c64*, int64_t, const void*, int, cudaStream_t, cudaEvent_t*, const ZTune*);
int conv_all_ff(const Family*, int, const Spectrum*, const void* const*, const c64*, c64*,
                c64*, int64_t, const void*, int, cudaStream_t, cudaEvent_t*, const ZTune*);

// prec: PEEC_PREC_FP64 (0), PEEC_PREC_FP32 (1), PEEC_PREC_FF (2); tw[prec] the matching
// master twiddle table
int conv_all(const Family* F, int nfam, const Spectrum* spec, const void* const* ph,
             const c64* x, c64* LpI, c64* PQ, int64_t m, int prec, const void* const* tw,
             int twmax, cudaStream_t st, cudaEvent_t* ev, const ZTune* zt) {
  if (prec == 0) return conv_all_f64(F, nfam, spec, ph, x, LpI, PQ, m, tw[0], twmax, st, ev, zt);
  if (prec == 2) return conv_all_ff(F, nfam, spec, ph, x, LpI, PQ, m, tw[2], twmax, st, ev, zt);
  return conv_all_f32(F, nfam, spec, ph, x, LpI, PQ, m, tw[1], twmax, st, ev, zt);
}

// The staged FP32 z passes need whole 16-column tiles (Lx a multiple of 16, so every
// staged row is 128 bytes at a 128-byte offset), at least two radix groups along z, and
// tiles that fit three (faces) / one (edges) per shared-memory budget; the edge families
// must share one circulant grid to share a launch.
static bool staged_grid(const Family& f, int zmin) {
  return f.L[0] >= 16 && f.L[0] % 16 == 0 && f.L[2] >= zmin && f.L[2] <= 128 &&
         f.dims[2] >= 1 && f.dims[2] <= f.L[2];
}

bool zpass_yz_faces(const Family* F, int nfam) {
  if (nfam < 3) return false;
  for (int f = 0; f < 3; ++f)
    if (!F[f].active || !staged_grid(F[f], 16)) return false;
  return true;
}

bool zpass_yz_edges(const Family* F, int nfam) {
  const Family* f0 = nullptr;
  for (int f = 3; f < nfam; ++f) {
    if (!F[f].active) continue;
    if (!staged_grid(F[f], 32)) return false;
    if (!f0) f0 = &F[f];
    else if (F[f].L[0] != f0->L[0] || F[f].L[1] != f0->L[1] || F[f].L[2] != f0->L[2])
      return false;
  }
  return f0 != nullptr;
}

int line_launches(const Family* F, int nfam, int prec, int ax) {
  int n = 0;
  bool direct = false;
  for (int f = 0; f < nfam; ++f) {
    if (!F[f].active) continue;
    if (prec == 0 || !line_pair_ok(F[f], ax)) {
      direct = true;
      continue;
    }
    bool first = true;  // of the families that share a launch
    for (int g = 0; g < f; ++g) first = first && !(line_pair_ok(F[g], ax) && F[g].L[ax] == F[f].L[ax]);
    n += first ? 1 : 0;
  }
  return n + (direct ? 1 : 0);
}

int zedge_launches(const Family* F, int nfam, int prec, const ZTune& zt) {
  if (prec == 1 && zt.edge == 2 && zpass_yz_edges(F, nfam)) return 1;
  const bool pair = prec == 2 || (prec == 1 && zt.edge == 3);
  int n = 0;
  for (int f = 3; f < nfam; ++f) {
    if (!F[f].active) continue;
    bool first = true;  // of the families that share a pair launch
    for (int g = 3; g < f && pair && zpair_ok(F[f]); ++g)
      first = first && !(zpair_ok(F[g]) && F[g].L[2] == F[f].L[2]);
    n += first ? 1 : 0;
  }
  return n;
}

// --------------------------------------------------------------------------- spectra
// The spectrum of a generating row: along each axis the embedded kernel
// K(e) = row[|s e + o|] is even (s = 1, o = 0) or even about a half-sample shift
// (s = 2, o = +-1, c = -o), so its transform is exp(-i pi c f / L) times a real, even R(f)
// and the three axes are three real transforms of the row's own octant:
//   x: (uz, uy, t) -> (uz, uy, fx)   y: -> (uz, fy, fx)   z: -> (fy, fz, fx) = R,
// u the used entries of an axis (every one, or the odd ones of an interleaved axis) and
// f = 0 .. L/2. A complex FFT of length L transforms two lines at once, one as the real and
// one as the imaginary part: after the shift's phase they separate by themselves. An eighth
// of the lines of the embedded complex transform, half of them again by the pairing; all
// rows of a set share each pass's launch. FP64 pipe bound. Measured at 128x128x64 (nine
// spectra): 1.65 ms, against 13.3 ms as complex transforms of the embedded kernels; a retarded
// frequency at 48x48x24 (eighteen spectra) 0.40 against 3.2 ms.
// ------------------------------------------------------------------------------------

struct SpecAxis {
  int L, n, na, nb, s, o, c;
  int M, U;  // entries of the row along the axis, and those used
};

__device__ __forceinline__ int embed_index(int j, const SpecAxis& d) {
  // offset e of circulant slot j: e = j for j < na, e = j - L for j > L - nb
  int e;
  if (j < d.na) e = j;
  else if (j > d.L - d.nb) e = j - d.L;
  else return -1;
  int t = d.s * e + d.o;
  t = t < 0 ? -t : t;
  return t < d.M ? t : -1;
}

struct SpecRow {
  SpecAxis ax[3];
  const double* row;
  double *A, *B, *oct;  // after the x and the y pass; R
  double scale;
};
constexpr int kSpecRows = 9;
struct SpecSet {
  SpecRow r[kSpecRows];
  int cta0[kSpecRows + 1];  // first CTA of each row in this pass
  int n;
};

// One pass along axis AX: 2^LC pairs of lines per CTA, tile element (pos, pair) at
// buf[pos * (C + 1) + pair].
template <int AX, int LC>
__global__ void __launch_bounds__(256) k_spec_pass(SpecSet S, const c64* __restrict__ twm,
                                                   int twmax) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int C = 1 << LC, RS = C + 1;
  int ri = 0;
#pragma unroll
  for (int i = 1; i < kSpecRows; ++i)
    if (i < S.n && (int)blockIdx.x >= S.cta0[i]) ri = i;
  const SpecRow& R = S.r[ri];
  const SpecAxis& d = R.ax[AX];
  const int ox = R.ax[0].L / 2 + 1, oy = R.ax[1].L / 2 + 1, oz = R.ax[2].L / 2 + 1;
  const int Uy = R.ax[1].U, Uz = R.ax[2].U;
  const int64_t lines = AX == 0 ? (int64_t)Uz * Uy : (AX == 1 ? (int64_t)Uz * ox : (int64_t)oy * ox);
  const int64_t l0 = (int64_t)((int)blockIdx.x - S.cta0[ri]) * (2 * C);
  const int L = d.L, half = L / 2 + 1;
  c64* W = reinterpret_cast<c64*>(smem_raw);
  c64* buf = W + L;
  load_twiddles<double>(W, twm, twmax, L);
  auto in = [&](int64_t l, int t) -> double {  // entry t of line l
    if (l >= lines) return 0.0;
    if (AX == 0) {
      const int uz = (int)(l / Uy), uy = (int)(l % Uy);
      const int tz = R.ax[2].s == 2 ? 2 * uz + 1 : uz, ty = R.ax[1].s == 2 ? 2 * uy + 1 : uy;
      return R.row[((size_t)tz * R.ax[1].M + ty) * d.M + t];
    }
    const int u = d.s == 2 ? t >> 1 : t;
    if (AX == 1) return R.A[((l / ox) * Uy + u) * ox + l % ox];
    return R.B[(int64_t)u * oy * ox + l];
  };
  // the lanes run along the axis where that is contiguous, else along the lines
  for (int q = threadIdx.x; q < L << LC; q += blockDim.x) {
    const int j = AX == 0 ? q & (L - 1) : q >> LC, col = AX == 0 ? q >> d.n : q & (C - 1);
    const int t = embed_index(j, d);
    c64 v = mk<double>(0, 0);
    if (t >= 0) v = mk<double>(in(l0 + 2 * col, t), in(l0 + 2 * col + 1, t));
    buf[j * RS + col] = v;
  }
  __syncthreads();
  for (int s = 0; s < d.n;) {
    const int q = min(3, d.n - s);
    smem_group_q<double, false, LC>(buf, RS, q, d.n, s, W);
    s += q;
    __syncthreads();
  }
  for (int q = threadIdx.x; q < half << LC; q += blockDim.x) {
    const int f = AX == 0 ? q % half : q >> LC, col = AX == 0 ? q / half : q & (C - 1);
    c64 v = buf[(d.n ? brev(f & (L - 1), d.n) : 0) * RS + col];
    if (d.c) {
      double sn, cs;
      sincospi((double)d.c * f / L, &sn, &cs);
      v = mk<double>(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
    }
    if (AX == 2) v = cscale(v, R.scale);
    double* out = AX == 0 ? R.A : (AX == 1 ? R.B : R.oct);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t l = l0 + 2 * col + h;
      if (l >= lines) break;
      int64_t at;
      if (AX == 0) at = l * ox + f;
      else if (AX == 1) at = ((l / ox) * oy + f) * ox + l % ox;
      else at = ((l / ox) * oz + f) * ox + l % ox;
      out[at] = h ? v.y : v.x;
    }
  }
}

// octant R (FP64, (fy, fz, fx)) -> the y/z-folded form ((fy, fz, px), px every DIF x position)
// in FP64 and FP32
__global__ void k_spec_yzfold(const double* __restrict__ o64, double* y64, float* y32, int Lx,
                              int Ly, int Lz) {
  const int ox = Lx / 2 + 1, oy = Ly / 2 + 1, oz = Lz / 2 + 1;
  const int nx = ilog2(Lx);
  const size_t n = (size_t)Lx * oy * oz;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < n;
       o += (size_t)gridDim.x * blockDim.x) {
    const int px = (int)(o & (Lx - 1));
    const size_t rr = o >> nx;  // fy * oz + fz
    const int k = nx ? (int)(__brev((unsigned)px) >> (32 - nx)) : 0;
    const int fx = k <= Lx / 2 ? k : Lx - k;
    const double v = o64[rr * ox + fx];
    y64[o] = v;
    y32[o] = (float)v;
  }
}

// phase tables of the shifted axes: E[p] = exp(-i*pi*k/L) for the signed frequency k of
// DIF position p (k = brev(p) folded into (-L/2, L/2]), FP64 and its FP32 rounding
__global__ void k_phase_table(int L, c64* e64, c32* e32) {
  const int n = ilog2(L);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < L; p += gridDim.x * blockDim.x) {
    int k = brev(p, n);
    if (k > L / 2) k -= L;
    double sn, cs;
    sincospi(-(double)k / L, &sn, &cs);
    e64[p] = mk<double>(cs, sn);
    e32[p] = mk<float>((float)cs, (float)sn);
  }
}

int phase_tables(const int L[3], void* e64[3], void* e32[3], cudaStream_t st) {
  for (int a = 0; a < 3; ++a) {
    if (e64[a]) cudaFree(e64[a]);
    if (e32[a]) cudaFree(e32[a]);
    e64[a] = e32[a] = nullptr;
    PEEC_CUDA_TRY(dev_alloc(&e64[a], sizeof(c64) * L[a]));
    PEEC_CUDA_TRY(dev_alloc(&e32[a], sizeof(c32) * L[a]));
    k_phase_table<<<(L[a] + 255) / 256, 256, 0, st>>>(L[a], (c64*)e64[a], (c32*)e32[a]);
  }
  PEEC_CUDA_TRY(cudaGetLastError());
  return 0;
}

template <int AX, int LC>
static int spec_pass(SpecSet& S, int ctas, const c64* tw, int twmax, cudaStream_t st) {
  size_t sm = 0;
  for (int i = 0; i < S.n; ++i)
    sm = std::max(sm, sizeof(c64) * (size_t)S.r[i].ax[AX].L * ((1 << LC) + 2));
  if (sm > 48 * 1024) {
    // the device's limit, the same for every context (the attribute is the function's, and
    // contexts of other sizes may launch it from other threads)
    int dev = 0, lim = 0;
    PEEC_CUDA_TRY(cudaGetDevice(&dev));
    PEEC_CUDA_TRY(cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PEEC_CUDA_TRY(cudaFuncSetAttribute(k_spec_pass<AX, LC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  }
  k_spec_pass<AX, LC><<<ctas, 256, sm, st>>>(S, tw, twmax);
  return 0;
}

template <int AX>
static int spec_axis(SpecSet& S, const c64* tw, int twmax, cudaStream_t st) {
  int Lmax = 1;
  for (int i = 0; i < S.n; ++i) Lmax = std::max(Lmax, S.r[i].ax[AX].L);
  // pairs of lines per CTA: sixteen while the tile leaves room for two CTAs per SM
  int lc = 4;
  while (lc > 0 && sizeof(c64) * (size_t)Lmax * ((1 << lc) + 2) > 110 * 1024) lc -= 2;
  int ctas = 0;
  for (int i = 0; i < S.n; ++i) {
    const SpecRow& R = S.r[i];
    const int64_t ox = R.ax[0].L / 2 + 1, oy = R.ax[1].L / 2 + 1;
    const int64_t lines = AX == 0 ? (int64_t)R.ax[2].U * R.ax[1].U
                                  : (AX == 1 ? R.ax[2].U * ox : oy * ox);
    S.cta0[i] = ctas;
    ctas += (int)((lines + (2 << lc) - 1) / (2 << lc));
  }
  S.cta0[S.n] = ctas;
  if (lc == 4) return spec_pass<AX, 4>(S, ctas, tw, twmax, st);
  if (lc == 2) return spec_pass<AX, 2>(S, ctas, tw, twmax, st);
  return spec_pass<AX, 0>(S, ctas, tw, twmax, st);
}

int spectra_build(const SpecJob* jobs, int njobs, const void* tw64, int twmax, cudaMemPool_t pool, cudaStream_t st) {
  if (njobs <= 0) return 0;
  if (njobs > kSpecRows) return set_error("too many spectra"), PEEC_ERR_UNSUPPORTED_INTERNAL;
  SpecSet set{};
  set.n = njobs;
  size_t na = 0, nb = 0, no = 0;
  for (int i = 0; i < njobs; ++i) {
    const SpecJob& J = jobs[i];
    Spectrum& S = *J.S;
    SpecRow& R = set.r[i];
    for (int a = 0; a < 3; ++a) {
      // half-sample shift per axis: |2e + o| is even about e = -o/2 (the embedding window is
      // symmetric about the same point because na - nb = -o there)
      S.c[a] = (!J.symmetric && J.sdim[a] == 2) ? -J.odim[a] : 0;
      R.ax[a] = SpecAxis{S.L[a], ilog2(S.L[a]), J.na[a], J.nb[a], J.sdim[a], J.odim[a], S.c[a],
                         J.M[a], J.sdim[a] == 2 ? J.M[a] / 2 : J.M[a]};
    }
    const size_t ny = (size_t)S.L[0] * (S.L[1] / 2 + 1) * (S.L[2] / 2 + 1);
    if (!S.yz[0]) PEEC_CUDA_TRY(dev_alloc(&S.yz[0], ny * sizeof(double)));
    if (!S.yz[1]) PEEC_CUDA_TRY(dev_alloc(&S.yz[1], ny * sizeof(float)));
    R.row = J.row;
    R.scale = 1.0 / ((double)S.L[0] * S.L[1] * S.L[2]);
    na += (size_t)R.ax[2].U * R.ax[1].U * (S.L[0] / 2 + 1);
    nb += (size_t)R.ax[2].U * (S.L[1] / 2 + 1) * (S.L[0] / 2 + 1);
    no += (size_t)(S.L[0] / 2 + 1) * (S.L[1] / 2 + 1) * (S.L[2] / 2 + 1);
  }
  double* scr = nullptr;
  PEEC_CUDA_TRY(scratch_alloc((void**)&scr, (na + nb + no + 1) * sizeof(double), pool, st));
  size_t oa = 0, ob = na, oo = na + nb;
  for (int i = 0; i < njobs; ++i) {
    SpecRow& R = set.r[i];
    R.A = scr + oa;
    R.B = scr + ob;
    R.oct = scr + oo;
    oa += (size_t)R.ax[2].U * R.ax[1].U * (R.ax[0].L / 2 + 1);
    ob += (size_t)R.ax[2].U * (R.ax[1].L / 2 + 1) * (R.ax[0].L / 2 + 1);
    oo += (size_t)(R.ax[2].L / 2 + 1) * (R.ax[1].L / 2 + 1) * (R.ax[0].L / 2 + 1);
  }
  const c64* tw = reinterpret_cast<const c64*>(tw64);
  CTX_CHECK(spec_axis<0>(set, tw, twmax, st));
  CTX_CHECK(spec_axis<1>(set, tw, twmax, st));
  CTX_CHECK(spec_axis<2>(set, tw, twmax, st));
  for (int i = 0; i < njobs; ++i) {
    Spectrum& S = *jobs[i].S;
    const size_t ny = (size_t)S.L[0] * (S.L[1] / 2 + 1) * (S.L[2] / 2 + 1);
    k_spec_yzfold<<<(unsigned)std::min<size_t>((ny + 255) / 256, 152 * 16), 256, 0, st>>>(
        set.r[i].oct, (double*)S.yz[0], (float*)S.yz[1], S.L[0], S.L[1], S.L[2]);
  }
  PEEC_CUDA_TRY(cudaGetLastError());
  PEEC_CUDA_TRY(cudaFreeAsync(scr, st));
  return 0;
}

}  // namespace peec
