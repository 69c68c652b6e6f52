// Pass kernels and launch sequence of the circulant convolutions, templated on the
// arithmetic (float, double, float-float); each arithmetic is instantiated in its own
// translation unit (fftconv_f32.cu, fftconv_f64.cu, fftconv_ff.cu) so they compile in
// parallel. The pipeline itself is described in fftconv.cu.
#pragma once
#include <mutex>
#include <set>
#include <type_traits>
#include <utility>

#include "ctx.hpp"
#include "fft_reg.cuh"
#include "tma.cuh"

namespace peec {

constexpr int TPB = 256;
// z passes: 128 threads, so that with Lz = 128 every phase splits evenly (first and
// last groups 3 x 16 columns x 8 pencils, fused step 16 x 16) and four CTAs share an SM
constexpr int ZTPB = 128;

// Family buffers stream through each pass once: loads and stores carry the streaming
// (evict-first) cache hint, so the L2 keeps the spectra and twiddles the passes reuse.
template <typename R>
struct StreamVec;
template <>
struct StreamVec<float> {
  using T = float2;
};
template <>
struct StreamVec<double> {
  using T = double2;
};
template <>
struct StreamVec<ff> {
  using T = float4;
};
template <typename R>
__device__ __forceinline__ cx<R> ld_stream(const cx<R>* p) {
  using V = typename StreamVec<R>::T;
  const V v = __ldcs(reinterpret_cast<const V*>(p));
  return *reinterpret_cast<const cx<R>*>(&v);
}
template <typename R>
__device__ __forceinline__ void st_stream(cx<R>* p, const cx<R>& x) {
  using V = typename StreamVec<R>::T;
  __stcs(reinterpret_cast<V*>(p), *reinterpret_cast<const V*>(&x));
}

// --------------------------------------------------------------------------- x passes
// CTA: TY = 16 consecutive y rows of one z plane. Tile element (pos, yy) at
// buf[pos*(TY+1) + yy]; the first/last group threads run along x so map reads and
// output gathers are contiguous.

constexpr int LTY = 4;
constexpr int TY = 1 << LTY;
constexpr int XRS = TY + 1;

template <typename R, int Q>
__device__ __forceinline__ void xfwd_first(const c64* __restrict__ xin,
                                           const int32_t* __restrict__ map, cx<R>* buf,
                                           const AxPlan& p, int y0, int z, int nx, int ny,
                                           const cx<R>* W) {
  constexpr int N = 1 << Q;
  const int lh = p.n - Q;
  const int tasks = TY << lh;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int k = t & ((1 << lh) - 1);
    const int yy = t >> lh;
    const int y = y0 + yy;
    cx<R> v[N];
    const int32_t* mrow = map + ((size_t)z * ny + y) * nx;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const int x = k + (r << lh);
      v[r] = mk<R>(0, 0);
      if (y < ny && x < nx) {
        const int idx = mrow[x];
        if (idx >= 0) v[r] = ccast<R>(xin[idx]);
      }
    }
    dft_dif<R, Q>(v);
    if (p.ng > 1) group_twiddle<R, Q, false>(v, k, 0, W);
#pragma unroll
    for (int r = 0; r < N; ++r) buf[(k + (r << lh)) * XRS + yy] = v[r];
  }
}

template <typename R, int Q, bool INV>
__device__ __forceinline__ void x_last_inplace(cx<R>* buf, const AxPlan& p) {
  // the group at the end of the stage order (forward) / its mirror (inverse):
  // contiguous positions, no table twiddles
  constexpr int N = 1 << Q;
  const int tasks = TY << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int yy = t & (TY - 1);
    const int start = (t >> LTY) << Q;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[(start + r) * XRS + yy];
    if (!INV) dft_dif<R, Q>(v);
    else dft_dit<R, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) buf[(start + r) * XRS + yy] = v[r];
  }
}

// One launch runs a pass over every active family: the CTAs of family i are
// [cta0, cta0 + gx * gy) of the 1-D grid, laid out as that family's own gx x gy grid.
// Separate launches per family left each pass a train of partial waves (at 128x128x64 a
// family's x pass is under one wave of CTAs) with a ramp-up and tail each.
template <typename R>
struct FamPass {
  cx<R>* T;             // family buffer
  const int32_t* map;   // x passes: lattice map
  c64* io;              // x passes: compact input (forward) / output (inverse)
  AxPlan p;             // transform plan along the pass axis
  int L_other;          // x passes: Ly; y passes: Lx
  int a, b;             // x passes: lattice nx, ny; y passes: rows read, rows written
  int gx;               // CTAs along the family grid's first axis
  int cta0;             // first CTA of the family
};
constexpr int kMaxFam = 6;
template <typename R>
struct PassSet {
  int nf;
  FamPass<R> f[kMaxFam];
};

// this CTA's family, and its (x, y) block index in that family's grid
template <typename R>
__device__ __forceinline__ FamPass<R> pick_family(const PassSet<R>& s, int& bx, int& by) {
  const int b = blockIdx.x;
  FamPass<R> F = s.f[0];
#pragma unroll
  for (int i = 1; i < kMaxFam; ++i)
    if (i < s.nf && b >= s.f[i].cta0) F = s.f[i];
  const int lb = b - F.cta0;
  bx = lb % F.gx;
  by = lb / F.gx;
  return F;
}

template <typename R>
__global__ void __launch_bounds__(TPB) k_xfwd(PassSet<R> s, const cx<R>* __restrict__ twm,
                                              int twmax) {
  extern __shared__ unsigned char smem_raw[];
  int bx, by;
  const FamPass<R> F = pick_family(s, bx, by);
  const c64* __restrict__ xin = F.io;
  const int32_t* __restrict__ map = F.map;
  cx<R>* T = F.T;
  const AxPlan& p = F.p;
  const int Ly = F.L_other, nx = F.a, ny = F.b;
  const int Lx = 1 << p.n;
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* buf = W + Lx;
  const int y0 = bx * TY, z = by;
  load_twiddles<R>(W, twm, twmax, Lx);
  __syncthreads();
  qswitch<4>(p.q[0], [&](auto QC) {
    xfwd_first<R, decltype(QC)::value>(xin, map, buf, p, y0, z, nx, ny, W);
  });
  __syncthreads();
  if (p.ng > 1) {
    middle_groups<R, false, LTY>(buf, XRS, p, W);
    qswitch<4>(p.q[p.ng - 1],
               [&](auto QC) { x_last_inplace<R, decltype(QC)::value, false>(buf, p); });
    __syncthreads();
  }
  for (int q = threadIdx.x; q < TY << p.n; q += blockDim.x) {
    const int yy = q >> p.n, kx = q & (Lx - 1);
    const int y = y0 + yy;
    if (y < ny) st_stream(T + ((size_t)z * Ly + y) * Lx + kx, buf[kx * XRS + yy]);
  }
}

template <typename R, int Q>
__device__ __forceinline__ void xinv_last(const cx<R>* buf, c64* yout,
                                          const int32_t* __restrict__ map, const AxPlan& p,
                                          int y0, int z, int nx, int ny, const cx<R>* W) {
  constexpr int N = 1 << Q;
  const int lh = p.n - Q;
  const int tasks = TY << lh;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int k = t & ((1 << lh) - 1);
    const int yy = t >> lh;
    const int y = y0 + yy;
    if (y >= ny || k >= nx) continue;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[(k + (r << lh)) * XRS + yy];
    if (p.ng > 1) group_twiddle<R, Q, true>(v, k, 0, W);
    dft_dit<R, Q>(v);
    const int32_t* mrow = map + ((size_t)z * ny + y) * nx;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const int x = k + (r << lh);
      if (x < nx) {
        const int idx = mrow[x];
        if (idx >= 0) yout[idx] = mk<double>((double)v[r].x, (double)v[r].y);
      }
    }
  }
}

template <typename R>
__global__ void __launch_bounds__(TPB) k_xinv(PassSet<R> s, const cx<R>* __restrict__ twm,
                                              int twmax) {
  extern __shared__ unsigned char smem_raw[];
  int bx, by;
  const FamPass<R> F = pick_family(s, bx, by);
  const cx<R>* __restrict__ T = F.T;
  c64* yout = F.io;
  const int32_t* __restrict__ map = F.map;
  const AxPlan& p = F.p;
  const int Ly = F.L_other, nx = F.a, ny = F.b;
  const int Lx = 1 << p.n;
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* buf = W + Lx;
  const int y0 = bx * TY, z = by;
  load_twiddles<R>(W, twm, twmax, Lx);
  for (int q = threadIdx.x; q < TY << p.n; q += blockDim.x) {
    const int yy = q >> p.n, kx = q & (Lx - 1);
    const int y = y0 + yy;
    buf[kx * XRS + yy] = (y < ny) ? ld_stream(T + ((size_t)z * Ly + y) * Lx + kx) : mk<R>(0, 0);
  }
  __syncthreads();
  if (p.ng > 1) {
    qswitch<4>(p.q[p.ng - 1],
               [&](auto QC) { x_last_inplace<R, decltype(QC)::value, true>(buf, p); });
    __syncthreads();
    middle_groups<R, true, LTY>(buf, XRS, p, W);
  }
  qswitch<4>(p.q[0], [&](auto QC) {
    xinv_last<R, decltype(QC)::value>(buf, yout, map, p, y0, z, nx, ny, W);
  });
}

// --------------------------------------------------------------------------- column passes
// y and z passes work on columns of TX = 16 consecutive kx: element (pos, col) of the
// tile at buf[pos*TX + col]; global row pos of the column tile at g + pos*gstride.

constexpr int LTX = 4;
constexpr int TX = 1 << LTX;

// forward first group from global rows < n_in (zero beyond), into registers, then the
// tile (or, for a single-group plan, back to global in full)
template <typename R, int Q>
__device__ __forceinline__ void col_first_fwd(const cx<R>* g, size_t gstride, int ncols,
                                              int n_in, cx<R>* buf, const AxPlan& p,
                                              const cx<R>* W, cx<R>* gout) {
  constexpr int N = 1 << Q;
  const int lh = p.n - Q;
  const int tasks = TX << lh;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int k = t >> LTX;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const int row = k + (r << lh);
      v[r] = (col < ncols && row < n_in) ? ld_stream(g + row * gstride + col) : mk<R>(0, 0);
    }
    dft_dif<R, Q>(v);
    if (p.ng > 1) {
      group_twiddle<R, Q, false>(v, k, 0, W);
#pragma unroll
      for (int r = 0; r < N; ++r) buf[((k + (r << lh)) << LTX) + col] = v[r];
    } else if (col < ncols) {
#pragma unroll
      for (int r = 0; r < N; ++r) st_stream(gout + r * gstride + col, v[r]);
    }
  }
}

// forward last group: tile -> global, contiguous positions
template <typename R, int Q>
__device__ __forceinline__ void col_last_fwd(const cx<R>* buf, cx<R>* g, size_t gstride,
                                             int ncols, const AxPlan& p) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[((start + r) << LTX) + col];
    dft_dif<R, Q>(v);
    if (col < ncols) {
#pragma unroll
      for (int r = 0; r < N; ++r) st_stream(g + (start + r) * gstride + col, v[r]);
    }
  }
}

// inverse first group (mirror of the forward last group): global -> tile, or for a
// single-group plan global -> global rows < n_out
template <typename R, int Q>
__device__ __forceinline__ void col_first_inv(const cx<R>* g, size_t gstride, int ncols,
                                              int n_out, cx<R>* buf, const AxPlan& p,
                                              cx<R>* gout) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r)
      v[r] = col < ncols ? ld_stream(g + (start + r) * gstride + col) : mk<R>(0, 0);
    dft_dit<R, Q>(v);
    if (p.ng > 1) {
#pragma unroll
      for (int r = 0; r < N; ++r) buf[((start + r) << LTX) + col] = v[r];
    } else if (col < ncols) {
#pragma unroll
      for (int r = 0; r < N; ++r)
        if (start + r < n_out) st_stream(gout + (start + r) * gstride + col, v[r]);
    }
  }
}

// inverse last group (mirror of the forward first group): tile -> global rows < n_out
template <typename R, int Q>
__device__ __forceinline__ void col_last_inv(const cx<R>* buf, cx<R>* g, size_t gstride,
                                             int ncols, int n_out, const AxPlan& p,
                                             const cx<R>* W) {
  constexpr int N = 1 << Q;
  const int lh = p.n - Q;
  const int tasks = TX << lh;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int k = t >> LTX;
    if (k >= n_out) continue;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[((k + (r << lh)) << LTX) + col];
    group_twiddle<R, Q, true>(v, k, 0, W);
    dft_dit<R, Q>(v);
    if (col < ncols) {
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const int row = k + (r << lh);
        if (row < n_out) st_stream(g + row * gstride + col, v[r]);
      }
    }
  }
}

// register-group caps per kernel (see make_plan): x/y passes 16 points at both ends;
// z passes hold three families (P) or one (Lp) at the fused spectral step
template <typename R>
struct QCap {
  static constexpr bool wide = sizeof(R) == 8;  // double and float-float registers
  static constexpr int XY = 4;
  static constexpr int Z3 = wide ? 2 : 3;
  static constexpr int Z1 = wide ? 3 : 4;
};
// buffers and spectra: FP32 passes use the FP32 copies, FP64 and float-float the FP64 ones
template <typename R>
constexpr int slot_of() {
  return std::is_same<R, float>::value ? 1 : 0;
}

// --------------------------------------------------------------------------- y pass
// planes z < nz; rows y < n_in are read (zero padded to Ly), rows y < n_out written
template <typename R, bool INV>
__global__ void __launch_bounds__(TPB) k_ypass(PassSet<R> s, const cx<R>* __restrict__ twm,
                                               int twmax) {
  extern __shared__ unsigned char smem_raw[];
  int bx, by;
  const FamPass<R> F = pick_family(s, bx, by);
  cx<R>* T = F.T;
  const AxPlan& p = F.p;
  const int Lx = F.L_other, n_in = F.a, n_out = F.b;
  const int Ly = 1 << p.n;
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* buf = W + Ly;
  const int kx0 = bx * TX, z = by;
  const int ncols = min(TX, Lx - kx0);
  cx<R>* col = T + (size_t)z * Ly * Lx + kx0;
  load_twiddles<R>(W, twm, twmax, Ly);
  __syncthreads();
  if (!INV) {
    qswitch<QCap<R>::XY>(p.q[0], [&](auto QC) { col_first_fwd<R, decltype(QC)::value>(col, (size_t)Lx, ncols, n_in, buf, p, W, col); });
    if (p.ng > 1) {
      __syncthreads();
      middle_groups<R, false, LTX>(buf, TX, p, W);
      qswitch<QCap<R>::XY>(p.q[p.ng - 1], [&](auto QC) { col_last_fwd<R, decltype(QC)::value>(buf, col, (size_t)Lx, ncols, p); });
    }
  } else {
    qswitch<QCap<R>::XY>(p.q[p.ng - 1], [&](auto QC) { col_first_inv<R, decltype(QC)::value>(col, (size_t)Lx, ncols, n_out, buf, p, col); });
    if (p.ng > 1) {
      __syncthreads();
      middle_groups<R, true, LTX>(buf, TX, p, W);
      qswitch<QCap<R>::XY>(p.q[0], [&](auto QC) { col_last_inv<R, decltype(QC)::value>(buf, col, (size_t)Lx, ncols, n_out, p, W); });
    }
  }
}

// --------------------------------------------------------------------------- pair x and y passes
// Lines whose occupied entries fill at most half the circulant (n <= L/2 + 1, always so here), as
// two transforms of half the length H = L/2, the even and the odd frequencies:
//   X(2f) = FFT_H(x_j + x_{j+H}),   X(2f+1) = FFT_H((x_j - x_{j+H}) w^j),   w = exp(-2 pi i / L),
// only j + H = H ever occupied, and mirrored for the inverse. The padding is neither loaded nor
// transformed. A line's H points sit in the registers of G threads, V = H/G each: V-point
// transforms over the entries k + G r of thread k, twiddles, a transpose through shared memory,
// G-point transforms; a thread then holds G consecutive positions of the bit-reversed order. y:
// a CTA takes 128 / G consecutive columns, whose rows are contiguous across the lanes. x: a
// line's threads are neighbouring lanes (no CTA barrier after the twiddles are there), its G
// positions leave in 32-byte stores and the lattice map's and the vectors' entries come in lane
// order, all of a thread's loads in flight at once.
// What bounds them: FP32 the memory (about 1.3 times the family buffers' bytes in DRAM) and the
// gathers' latency, float-float the FP32 pipes. The direct kernels (k_xfwd and so on) ran 37M and
// 52M warp instructions in x and y at 128x128x64, on padding and through three transposes in
// shared memory with CTA barriers. Operator application at 128x128x64, x / y / inverse y / inverse
// x: FP32 70 / 78 / 70 / 87 -> 51 / 53 / 65 / 47 us, float-float 262 / 291 / 311 / 258 -> 209 / 263
// / 278 / 177 us; FP32 at 64x64x32 13.9 / 16.3 / 14.9 / 15.5 -> 8.3 / 6.8 / 7.5 / 8.9 us. FP64
// stays direct, like its z passes (its pipe is the bound in either form).
__device__ __forceinline__ int brevn(int v, int n) {
  return n ? (int)(__brev((unsigned)v) >> (32 - n)) : 0;
}

constexpr int XP_TPB = 128;
template <typename R>
struct LineFam {
  cx<R>* T;
  const int32_t* map;  // x: lattice map
  c64* io;             // x: compact vector
  int lx, ly;          // log2 of the circulant's x and y lengths
  int n;               // occupied entries of a line
  int ny;              // x: lines of a z plane
  int lines;           // x: ny nz; y: nz << lx
  int cta0;
};
template <typename R>
struct LineSet {
  LineFam<R> f[kMaxFam];
  int nf;
};

__device__ __forceinline__ c32 line_swap(const c32& v, int m) {
  return mk<float>(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
__device__ __forceinline__ cff line_swap(const cff& v, int m) {
  return mk<ff>(ff(__shfl_xor_sync(0xffffffffu, v.x.hi, m), __shfl_xor_sync(0xffffffffu, v.x.lo, m)),
                ff(__shfl_xor_sync(0xffffffffu, v.y.hi, m), __shfl_xor_sync(0xffffffffu, v.y.lo, m)));
}

template <typename R>
__device__ __forceinline__ cx<R> line_sel(bool t, cx<R> a, cx<R> b) {  // by value: no addresses
  return t ? a : b;
}

// G <= V: a thread takes V/G of the second transforms whole. G = 2 V: two neighbouring threads
// take one, as V points each (even and odd) and a last pair step in which they swap half.
template <typename R, int A, int B>
struct HalfLine {
  static constexpr int V = 1 << A, G = 1 << B, H = V * G, L = 2 * H;
  // lines of a CTA: x 128 threads; y at least 16 columns (128 bytes of FP32 rows)
  static constexpr int CX = XP_TPB / G, CY = CX < 16 ? 16 : CX;
  static constexpr bool SPLIT = G > V;
  static_assert(!SPLIT || G == 2 * V, "at most two threads a second transform");
  // x: exchange strides of a frequency group and of a line (bank-disjoint)
  static constexpr int SJ = SPLIT ? G + 2 : G + 1, LS = V * SJ + 8;
  static constexpr int RUN = B == 0 || SPLIT ? V : G, NRUN = V / RUN;
  static constexpr size_t smem(bool x) {
    return sizeof(cx<R>) * (L + (B == 0 ? 0 : x ? LS * CX : 2 * H * CY));
  }
  template <bool WARP>
  static __device__ __forceinline__ void sync() {
    if (WARP) __syncwarp();
    else __syncthreads();
  }
  // run q of thread k after a forward half (registers q RUN ..): position within the half
  static __device__ __forceinline__ int pos(int q, int k) {
    if (SPLIT) return brevn(k >> 1, A) * G + (k & 1) * V;
    return B > 0 ? brevn(k + G * q, A) * G : 0;
  }
  // entries k + G r -> positions in runs; the exchange cell of frequency group j, point t is
  // xc[j * sj + t * st], the neighbour k ^ 1 is lane ^ nb
  template <bool WARP>
  static __device__ __forceinline__ void fwd(cx<R>* d, const cx<R>* W, int k, cx<R>* xc, int sj,
                                             int st, int nb) {
    dft_dif<R, A>(d);
    if constexpr (B > 0) {
      if (WARP) __syncwarp();
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const int j = brevq(r, A);
        xc[j * sj + k * st] = j ? d[r] * W[2 * j * k] : d[r];
      }
      sync<WARP>();
      if constexpr (SPLIT) {
        const int j = k >> 1, t = k & 1;
#pragma unroll
        for (int i = 0; i < V; ++i) d[i] = xc[j * sj + (t + 2 * i) * st];
        dft_dif<R, A>(d);
#pragma unroll
        for (int i = 1; i < V; ++i) d[i] = d[i] * W[t * brevq(i, A) * (L / G)];
        cx<R> e[V];
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          const cx<R> o = line_swap(line_sel<R>(t, d[i], d[i + V / 2]), nb);
          const cx<R> a = line_sel<R>(t, o, d[i]), b = line_sel<R>(t, d[i + V / 2], o);
          e[2 * i] = a + b;
          e[2 * i + 1] = a - b;
        }
#pragma unroll
        for (int i = 0; i < V; ++i) d[i] = e[i];
      } else {
#pragma unroll
        for (int q = 0; q < V / G; ++q) {
#pragma unroll
          for (int t = 0; t < G; ++t) d[q * G + t] = xc[(k + G * q) * sj + t * st];
          dft_dif<R, B>(d + q * G);
        }
      }
    }
  }
  // the conjugate transpose
  template <bool WARP>
  static __device__ __forceinline__ void inv(cx<R>* d, const cx<R>* W, int k, cx<R>* xc, int sj,
                                             int st, int nb) {
    if constexpr (B > 0) {
      if (WARP) __syncwarp();
      if constexpr (SPLIT) {
        const int j = k >> 1, t = k & 1;
        cx<R> e[V];
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          const cx<R> a = d[2 * i] + d[2 * i + 1], b = d[2 * i] - d[2 * i + 1];
          const cx<R> o = line_swap(line_sel<R>(t, a, b), nb);
          e[i] = line_sel<R>(t, o, a);
          e[i + V / 2] = line_sel<R>(t, b, o);
        }
#pragma unroll
        for (int i = 0; i < V; ++i) d[i] = i ? cmulc(e[i], W[t * brevq(i, A) * (L / G)]) : e[i];
        dft_dit<R, A>(d);
#pragma unroll
        for (int i = 0; i < V; ++i)
          xc[j * sj + (t + 2 * i) * st] = cmulc(d[i], W[2 * j * (t + 2 * i)]);
      } else {
#pragma unroll
        for (int q = 0; q < V / G; ++q) {
          dft_dit<R, B>(d + q * G);
          const int j = k + G * q;
#pragma unroll
          for (int t = 0; t < G; ++t)
            xc[j * sj + t * st] = t ? cmulc(d[q * G + t], W[2 * j * t]) : d[q * G + t];
        }
      }
      sync<WARP>();
#pragma unroll
      for (int r = 0; r < V; ++r) d[r] = xc[brevq(r, A) * sj + k * st];
    }
    dft_dit<R, A>(d);
  }
};

// this CTA's family
template <typename R>
__device__ __forceinline__ const LineFam<R>& line_family(const LineSet<R>& S) {
  int f = 0;
#pragma unroll
  for (int i = 1; i < kMaxFam; ++i)
    if (i < S.nf && (int)blockIdx.x >= S.f[i].cta0) f = i;
  return S.f[f];
}

// N consecutive elements, 32 bytes at a time where they fill that
template <typename R, int N>
__device__ __forceinline__ void st_run(cx<R>* p, const cx<R>* d) {
  if constexpr (sizeof(R) == 4 && N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + i),
                   "f"(d[i].x), "f"(d[i].y), "f"(d[i + 1].x), "f"(d[i + 1].y), "f"(d[i + 2].x),
                   "f"(d[i + 2].y), "f"(d[i + 3].x), "f"(d[i + 3].y)
                   : "memory");
  } else if constexpr (std::is_same<R, ff>::value && N % 2 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 2)
      asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + i),
                   "f"(d[i].x.hi), "f"(d[i].x.lo), "f"(d[i].y.hi), "f"(d[i].y.lo),
                   "f"(d[i + 1].x.hi), "f"(d[i + 1].x.lo), "f"(d[i + 1].y.hi), "f"(d[i + 1].y.lo)
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) st_stream(p + i, d[i]);
  }
}
template <typename R, int N>
__device__ __forceinline__ void ld_run(const cx<R>* p, cx<R>* d) {
  if constexpr (sizeof(R) == 4 && N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      asm volatile("ld.global.cs.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=f"(d[i].x), "=f"(d[i].y), "=f"(d[i + 1].x), "=f"(d[i + 1].y),
                     "=f"(d[i + 2].x), "=f"(d[i + 2].y), "=f"(d[i + 3].x), "=f"(d[i + 3].y)
                   : "l"(p + i)
                   : "memory");
  } else if constexpr (std::is_same<R, ff>::value && N % 2 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 2)
      asm volatile("ld.global.cs.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=f"(d[i].x.hi), "=f"(d[i].x.lo), "=f"(d[i].y.hi), "=f"(d[i].y.lo),
                     "=f"(d[i + 1].x.hi), "=f"(d[i + 1].x.lo), "=f"(d[i + 1].y.hi),
                     "=f"(d[i + 1].y.lo)
                   : "l"(p + i)
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = ld_stream(p + i);
  }
}
__device__ __forceinline__ c32 line_in(const c64& v, float) { return ccast<float>(v); }
__device__ __forceinline__ cff line_in(const c64& v, ff) {
  return mk<ff>(ff_split(v.x), ff_split(v.y));
}
__device__ __forceinline__ c64 line_out(const c32& v) { return mk<double>((double)v.x, (double)v.y); }
__device__ __forceinline__ c64 line_out(const cff& v) {
  return mk<double>(ff_join(v.x), ff_join(v.y));
}

// half par of a forward line: the entries x (xh: entry H) combined and rotated
template <typename R, int V, int G>
__device__ __forceinline__ void line_half(const cx<R>* x, const cx<R>& xh, const cx<R>* W, int k,
                                          int par, cx<R>* d) {
#pragma unroll
  for (int r = 0; r < V; ++r) d[r] = x[r];
  d[0] = par ? x[0] - xh : x[0] + xh;
  if (par) {
#pragma unroll
    for (int r = 0; r < V; ++r) d[r] = d[r] * W[k + G * r];
  }
}

template <typename R, int A, int B, bool INV, int MINB>
__global__ void __launch_bounds__(HalfLine<R, A, B>::CY << B, MINB)
k_ypair(LineSet<R> S, const cx<R>* __restrict__ twm, int twmax) {
  using HL = HalfLine<R, A, B>;
  constexpr int V = HL::V, G = HL::G, H = HL::H, L = HL::L, C = HL::CY;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  const LineFam<R>& F = line_family(S);
  const int c = threadIdx.x % C, k = threadIdx.x / C;
  cx<R>* xc = W + L + c;
  for (int e = threadIdx.x; e < L; e += C * G) W[e] = twm[e * (twmax / L)];
  const int line = ((int)blockIdx.x - F.cta0) * C + c, lx = F.lx, n = F.n;
  const bool on = line < F.lines;
  const size_t rs = (size_t)1 << lx;
  cx<R>* T = F.T + (on ? (((size_t)(line >> lx) << (A + B + 1 + lx)) + (line & ((1 << lx) - 1))) : 0);
  cx<R> x[V], d[V], xh = mk<R>(0, 0);
  if (!INV) {
#pragma unroll
    for (int r = 0; r < V; ++r)
      x[r] = on && k + G * r < n ? ld_stream(T + (k + G * r) * rs) : mk<R>(0, 0);
    if (on && k == 0 && n > H) xh = ld_stream(T + H * rs);
  }
  // inverse, FP32: both halves' loads in flight before the first is worked on (x holds the even
  // half until its turn; 67 -> 65 us in y, 49 -> 47 in x at 128x128x64, 8.1 -> 7.5 in y at 64x64x32)
  constexpr bool AHEAD = INV && sizeof(R) == 4 && V <= 8;
  if (AHEAD) {
#pragma unroll
    for (int q = 0; q < HL::NRUN; ++q) {
#pragma unroll
      for (int t = 0; t < HL::RUN; ++t) {
        const cx<R>* p = T + (HL::pos(q, k) + t) * rs;
        d[q * HL::RUN + t] = on ? ld_stream(p + H * rs) : mk<R>(0, 0);
        x[q * HL::RUN + t] = on ? ld_stream(p) : mk<R>(0, 0);
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    // forward: even, odd; inverse: odd, even
    const int par = INV ? 1 - h : h;
    cx<R>* xb = xc + h * (H * C);
    if (!INV) {
      line_half<R, V, G>(x, xh, W, k, par, d);
      HL::template fwd<false>(d, W, k, xb, G * C, C, C & 31);
    }
#pragma unroll
    for (int q = 0; q < HL::NRUN; ++q) {
      constexpr int RUN = HL::RUN;
      cx<R>* p = T + (par * H + HL::pos(q, k)) * rs;
#pragma unroll
      for (int t = 0; t < RUN; ++t) {
        if (!INV) {
          if (on) st_stream(p + t * rs, d[q * RUN + t]);
        } else if (!AHEAD) {
          d[q * RUN + t] = on ? ld_stream(p + t * rs) : mk<R>(0, 0);
        }
      }
    }
    if (INV) {
      HL::template inv<false>(d, W, k, xb, G * C, C, C & 31);
      if (h == 0) {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const cx<R> o = cmulc(d[r], W[k + G * r]);
          if (AHEAD) d[r] = x[r];
          x[r] = o;
        }
      }
    }
  }
  if (INV && on) {
#pragma unroll
    for (int r = 0; r < V; ++r)
      if (k + G * r < n) st_stream(T + (k + G * r) * rs, d[r] + x[r]);
    if (k == 0 && n > H) st_stream(T + H * rs, d[0] - x[0]);
  }
}

template <typename R, int A, int B, bool INV, int MINB>
__global__ void __launch_bounds__(XP_TPB, MINB) k_xpair(LineSet<R> S, const cx<R>* __restrict__ twm,
                                                        int twmax) {
  using HL = HalfLine<R, A, B>;
  constexpr int V = HL::V, G = HL::G, H = HL::H, L = HL::L, C = HL::CX;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  const LineFam<R>& F = line_family(S);
  const int c = threadIdx.x / G, k = threadIdx.x % G;
  cx<R>* xc = W + L + c * HL::LS;
  for (int e = threadIdx.x; e < L; e += XP_TPB) W[e] = twm[e * (twmax / L)];
  const int line = ((int)blockIdx.x - F.cta0) * C + c, n = F.n;
  const bool on = line < F.lines;
  const int z = on ? line / F.ny : 0, y = on ? line - z * F.ny : 0;
  cx<R>* T = F.T + ((((size_t)z << F.ly) + y) << (A + B + 1));
  const int32_t* map = F.map + (size_t)(on ? line : 0) * n;
  int id[V], ih = -1;
#pragma unroll
  for (int r = 0; r < V; ++r) id[r] = on && k + G * r < n ? map[k + G * r] : -1;
  if (on && k == 0 && n > H) ih = map[H];
  cx<R> x[V], d[V], xh = mk<R>(0, 0);
  if (!INV) {
#pragma unroll
    for (int r = 0; r < V; ++r) x[r] = id[r] >= 0 ? line_in(F.io[id[r]], R()) : mk<R>(0, 0);
    if (ih >= 0) xh = line_in(F.io[ih], R());
  }
  constexpr bool AHEAD = INV && sizeof(R) == 4 && V <= 8;  // as in k_ypair
  if (AHEAD) {
#pragma unroll
    for (int q = 0; q < HL::NRUN; ++q) {
      const cx<R>* p = T + HL::pos(q, k);
      ld_run<R, HL::RUN>(p + H, d + q * HL::RUN);
      ld_run<R, HL::RUN>(p, x + q * HL::RUN);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int par = INV ? 1 - h : h;
    if (!INV) {
      line_half<R, V, G>(x, xh, W, k, par, d);
      HL::template fwd<true>(d, W, k, xc, HL::SJ, 1, 1);
    }
#pragma unroll
    for (int q = 0; q < HL::NRUN; ++q) {
      constexpr int RUN = HL::RUN;
      cx<R>* p = T + par * H + HL::pos(q, k);
      if (!INV) {
        if (on) st_run<R, RUN>(p, d + q * RUN);
      } else if (!AHEAD) {
        ld_run<R, RUN>(p, d + q * RUN);  // (a line past the last reads the first one's)
      }
    }
    if (INV) {
      HL::template inv<true>(d, W, k, xc, HL::SJ, 1, 1);
      if (h == 0) {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const cx<R> o = cmulc(d[r], W[k + G * r]);
          if (AHEAD) d[r] = x[r];
          x[r] = o;
        }
      }
    }
  }
  if (INV) {
#pragma unroll
    for (int r = 0; r < V; ++r)
      if (id[r] >= 0) F.io[id[r]] = line_out(d[r] + x[r]);
    if (ih >= 0) F.io[ih] = line_out(d[0] - x[0]);
  }
}

// --------------------------------------------------------------------------- z passes

// The six P spectra (blocks 00, 11, 22, 01, 02, 12) in the y/z-folded form (Spectrum::yz) and
// the face grid's phase tables E_a[p] = exp(-i*pi*k/L_a), k the signed frequency of position
// p. The cross blocks' half-sample shifts pair up: block fg carries E of family f's axis
// (y, x, z for f = 0, 1, 2) and conj(E) of family g's. FP32 passes read the FP32
// tables, FP64 and float-float passes the FP64 ones.
struct PSpec {
  const void* y[6];
  const void* ex;
  const void* ey;
  const void* ez;
};

// storage type of the spectra and phase tables a pass of arithmetic type R reads: the
// float-float passes split the FP64 ones on load
template <typename R>
struct SpecOf {
  using T = R;
};
template <>
struct SpecOf<ff> {
  using T = double;
};
template <typename R>
__device__ __forceinline__ R spec_re(const void* p, size_t i) {
  return R(reinterpret_cast<const typename SpecOf<R>::T*>(p)[i]);
}
template <typename R>
__device__ __forceinline__ cx<R> spec_cx(const void* p, size_t i) {
  const auto v = reinterpret_cast<const cx<typename SpecOf<R>::T>*>(p)[i];
  return mk<R>(R(v.x), R(v.y));
}

// folded frequency at DIF position p of a length-2^n axis
__device__ __forceinline__ int fold_pos(int p, int n) {
  const int k = brevn(p, n), L = 1 << n;
  return k <= (L >> 1) ? k : L - k;
}

// spectrum index of a tile's column col at z position pz in the y/z-folded tables
struct YzIdx {
  size_t rowbase;  // fold(ky) * (Lz/2 + 1) * Lx + kx0
  int Lx, nz;
  __device__ __forceinline__ size_t at(int col, int pz) const {
    return rowbase + (size_t)fold_pos(pz, nz) * Lx + col;
  }
};

__device__ __forceinline__ YzIdx make_yzidx(int Lx, int Ly, int Lz, int kx0, int ky) {
  YzIdx y;
  y.Lx = Lx;
  y.nz = ilog2(Lz);
  y.rowbase = (size_t)fold_pos(ky, ilog2(Ly)) * (Lz / 2 + 1) * Lx + kx0;
  return y;
}

// Y_f = sum_g S_fg X_g at the frequency of (column col, z position pz) of the CTA; ex the column's
// x phase, ey the CTA's y phase. FP64, bound by its pipe, rotates families 1 and 2 to family 0's
// phase and back (psi_1 = E_x conj(E_y), psi_2 = E_z conj(E_y)): there the operator's error, against
// a reference with 64-bit significands, is that of complex tables either way.
template <typename R>
__device__ __forceinline__ void pspec_apply(const PSpec& S, const YzIdx& Y, int col, int pz,
                                            const cx<R>& ex, const cx<R>& ey, cx<R>& a0,
                                            cx<R>& a1, cx<R>& a2) {
  const size_t i = Y.at(col, pz);
  const cx<R> ez = spec_cx<R>(S.ez, pz);
  R r[6];
#pragma unroll
  for (int b = 0; b < 6; ++b) r[b] = spec_re<R>(S.y[b], i);
  if constexpr (std::is_same<R, double>::value) {
    const cx<R> p1 = cmulc(ex, ey), p2 = cmulc(ez, ey);
    const cx<R> x0 = a0, x1 = cmulc(a1, p1), x2 = cmulc(a2, p2);
    a0 = cscale(x0, r[0]) + cscale(x1, r[3]) + cscale(x2, r[4]);
    a1 = (cscale(x0, r[3]) + cscale(x1, r[1]) + cscale(x2, r[5])) * p1;
    a2 = (cscale(x0, r[4]) + cscale(x1, r[5]) + cscale(x2, r[2])) * p2;
  } else {
    pspec_product<R>(r, cmulc(ey, ex), cmulc(ey, ez), cmulc(ex, ez), a0, a1, a2);
  }
}

// single-group z transform of all three face families in registers
template <typename R, int Q>
__device__ __forceinline__ void z3_single(cx<R>* T0, cx<R>* T1, cx<R>* T2, int nz0, int nz1,
                                          int nz2, size_t pl, int ncols, const PSpec& S,
                                          const YzIdx& O, int kx0, const cx<R>& ey) {
  constexpr int N = 1 << Q;
  for (int col = threadIdx.x; col < TX; col += blockDim.x) {
    if (col >= ncols) continue;
    const cx<R> ex = spec_cx<R>(S.ex, kx0 + col);
    cx<R> v[3][N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      v[0][r] = r < nz0 ? ld_stream(T0 + r * pl + col) : mk<R>(0, 0);
      v[1][r] = r < nz1 ? ld_stream(T1 + r * pl + col) : mk<R>(0, 0);
      v[2][r] = r < nz2 ? ld_stream(T2 + r * pl + col) : mk<R>(0, 0);
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) dft_dif<R, Q>(v[f]);
#pragma unroll
    for (int r = 0; r < N; ++r) pspec_apply<R>(S, O, col, r, ex, ey, v[0][r], v[1][r], v[2][r]);
#pragma unroll
    for (int f = 0; f < 3; ++f) dft_dit<R, Q>(v[f]);
#pragma unroll
    for (int r = 0; r < N; ++r) {
      if (r < nz0) st_stream(T0 + r * pl + col, v[0][r]);
      if (r < nz1) st_stream(T1 + r * pl + col, v[1][r]);
      if (r < nz2) st_stream(T2 + r * pl + col, v[2][r]);
    }
  }
}

// fused middle step: last forward group of the three families, spectral product,
// first inverse group, tile -> tile (the three tiles are consecutive: tile f at
// buf + f*tsz)
template <typename R, int Q>
__device__ __forceinline__ void z3_fused(cx<R>* buf, size_t tsz, const AxPlan& p, int ncols,
                                         const PSpec& S, const YzIdx& O, int kx0, const cx<R>& ey) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    cx<R> v[3][N];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
#pragma unroll
      for (int r = 0; r < N; ++r) v[f][r] = buf[f * tsz + ((start + r) << LTX) + col];
      dft_dif<R, Q>(v[f]);
    }
    if (col < ncols) {
      const cx<R> ex = spec_cx<R>(S.ex, kx0 + col);
#pragma unroll
      for (int r = 0; r < N; ++r)
        pspec_apply<R>(S, O, col, start + r, ex, ey, v[0][r], v[1][r], v[2][r]);
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      dft_dit<R, Q>(v[f]);
#pragma unroll
      for (int r = 0; r < N; ++r) buf[f * tsz + ((start + r) << LTX) + col] = v[f][r];
    }
  }
}

// group size QFIX when the kernel is specialised for it (plans of the common lengths),
// else the runtime value through qswitch
template <int QFIX, int CAP, typename F>
__device__ __forceinline__ void qpick(int q, F&& f) {
  if constexpr (QFIX > 0) f(qconst<QFIX>{});
  else qswitch<CAP>(q, f);
}

// Q0 / QL > 0: instantiation for plans whose first / last groups have those sizes (only
// that register code is compiled: smaller kernels, fewer registers); 0: any plan
template <typename R, int Q0 = 0, int QL = 0>
__global__ void __launch_bounds__(ZTPB, 4) k_zconv3(cx<R>* T0, cx<R>* T1, cx<R>* T2, int nz0, int nz1,
                                                int nz2, PSpec S, int Lx, int Ly, AxPlan p,
                                                const cx<R>* __restrict__ twm, int twmax) {
  extern __shared__ unsigned char smem_raw[];
  const int Lz = 1 << p.n;
  const size_t tsz = (size_t)Lz << LTX;
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* buf = W + Lz;  // three tiles, family f at buf + f*tsz
  const int kx0 = blockIdx.x * TX, ky = blockIdx.y;
  const int ncols = min(TX, Lx - kx0);
  const size_t pl = (size_t)Ly * Lx;
  const size_t off = (size_t)ky * Lx + kx0;
  T0 += off;
  T1 += off;
  T2 += off;
  const YzIdx O = make_yzidx(Lx, Ly, Lz, kx0, ky);
  const cx<R> ey = spec_cx<R>(S.ey, ky);
  load_twiddles<R>(W, twm, twmax, Lz);
  __syncthreads();
  if constexpr (Q0 == 0) {
    if (p.ng == 1) {
      qswitch<QCap<R>::Z3>(p.q[0], [&](auto QC) { z3_single<R, decltype(QC)::value>(T0, T1, T2, nz0, nz1, nz2, pl, ncols, S, O, kx0, ey); });
      return;
    }
  }
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_first_fwd<R, decltype(QC)::value>(T0, pl, ncols, nz0, buf, p, W, T0); });
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_first_fwd<R, decltype(QC)::value>(T1, pl, ncols, nz1, buf + tsz, p, W, T1); });
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_first_fwd<R, decltype(QC)::value>(T2, pl, ncols, nz2, buf + 2 * tsz, p, W, T2); });
  __syncthreads();
  {
    int s = p.q[0];
    for (int g = 1; g + 1 < p.ng; ++g) {
      smem_group_q<R, false, LTX>(buf, TX, p.q[g], p.n, s, W);
      smem_group_q<R, false, LTX>(buf + tsz, TX, p.q[g], p.n, s, W);
      smem_group_q<R, false, LTX>(buf + 2 * tsz, TX, p.q[g], p.n, s, W);
      s += p.q[g];
      __syncthreads();
    }
  }
  qpick<QL, QCap<R>::Z3>(p.q[p.ng - 1], [&](auto QC) { z3_fused<R, decltype(QC)::value>(buf, tsz, p, ncols, S, O, kx0, ey); });
  __syncthreads();
  {
    int s = p.n - p.q[p.ng - 1];
    for (int g = p.ng - 2; g >= 1; --g) {
      s -= p.q[g];
      smem_group_q<R, true, LTX>(buf, TX, p.q[g], p.n, s, W);
      smem_group_q<R, true, LTX>(buf + tsz, TX, p.q[g], p.n, s, W);
      smem_group_q<R, true, LTX>(buf + 2 * tsz, TX, p.q[g], p.n, s, W);
      __syncthreads();
    }
  }
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_last_inv<R, decltype(QC)::value>(buf, T0, pl, ncols, nz0, p, W); });
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_last_inv<R, decltype(QC)::value>(buf + tsz, T1, pl, ncols, nz1, p, W); });
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_last_inv<R, decltype(QC)::value>(buf + 2 * tsz, T2, pl, ncols, nz2, p, W); });
}

// one edge family with its real spectrum
template <typename R, int Q>
__device__ __forceinline__ void z1_single(cx<R>* Tg, int nz, size_t pl, int ncols,
                                          const void* __restrict__ s, const YzIdx& O) {
  constexpr int N = 1 << Q;
  for (int col = threadIdx.x; col < TX; col += blockDim.x) {
    if (col >= ncols) continue;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = r < nz ? ld_stream(Tg + r * pl + col) : mk<R>(0, 0);
    dft_dif<R, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r)
      v[r] = cscale(v[r], spec_re<R>(s, O.at(col, r)));
    dft_dit<R, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r)
      if (r < nz) st_stream(Tg + r * pl + col, v[r]);
  }
}

template <typename R, int Q>
__device__ __forceinline__ void z1_fused(cx<R>* buf, const AxPlan& p, int ncols,
                                         const void* __restrict__ s, const YzIdx& O) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    cx<R> v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[((start + r) << LTX) + col];
    dft_dif<R, Q>(v);
    if (col < ncols) {
#pragma unroll
      for (int r = 0; r < N; ++r)
        v[r] = cscale(v[r], spec_re<R>(s, O.at(col, start + r)));
    }
    dft_dit<R, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) buf[((start + r) << LTX) + col] = v[r];
  }
}

template <typename R, int Q0 = 0, int QL = 0>
__global__ void __launch_bounds__(ZTPB, 4) k_zconv1(cx<R>* T0, int nz0, const void* __restrict__ s00,
                                                int Lx, int Ly, AxPlan p,
                                                const cx<R>* __restrict__ twm, int twmax) {
  extern __shared__ unsigned char smem_raw[];
  const int Lz = 1 << p.n;
  cx<R>* W = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* buf = W + Lz;
  const int kx0 = blockIdx.x * TX, ky = blockIdx.y;
  const int ncols = min(TX, Lx - kx0);
  const size_t pl = (size_t)Ly * Lx;
  cx<R>* Tg = T0 + (size_t)ky * Lx + kx0;
  const YzIdx O = make_yzidx(Lx, Ly, Lz, kx0, ky);
  load_twiddles<R>(W, twm, twmax, Lz);
  __syncthreads();
  if constexpr (Q0 == 0) {
    if (p.ng == 1) {
      qswitch<QCap<R>::Z1>(p.q[0], [&](auto QC) { z1_single<R, decltype(QC)::value>(Tg, nz0, pl, ncols, s00, O); });
      return;
    }
  }
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_first_fwd<R, decltype(QC)::value>(Tg, pl, ncols, nz0, buf, p, W, Tg); });
  __syncthreads();
  middle_groups<R, false, LTX>(buf, TX, p, W);
  qpick<QL, QCap<R>::Z1>(p.q[p.ng - 1], [&](auto QC) { z1_fused<R, decltype(QC)::value>(buf, p, ncols, s00, O); });
  __syncthreads();
  middle_groups<R, true, LTX>(buf, TX, p, W);
  qpick<Q0, QCap<R>::XY>(p.q[0], [&](auto QC) { col_last_inv<R, decltype(QC)::value>(buf, Tg, pl, ncols, nz0, p, W); });
}

// --------------------------------------------------------------------------- staged z passes
// FP32 z passes over persistent CTAs that walk the tiles (one ky row, 16 kx columns) in a
// grid-stride loop. One warp stages the next tile's occupied z rows of every family into a
// shared-memory buffer with bulk asynchronous copies (cp.async.bulk, 128-byte rows,
// mbarrier completion) while the CTA computes the current tile, so HBM reads overlap the
// FFT arithmetic instead of stalling it. The first group reads the staged rows; the
// middle, fused and last groups are those of k_zconv3 / k_zconv1. Spectra come from the
// y/z-folded FP32 tables (Spectrum::yz[1]), which stay largely resident in L2.
// Bounded waits: a copy wait that runs out sets *err, waits once more (bounded) for the
// copies in flight and ends the CTA.

constexpr int ZWAIT_LIMIT = 1 << 20;

// forward first group from the staged rows (row < nz; zero beyond) into the tile
template <int Q>
__device__ __forceinline__ void stg_first_fwd(const c32* stg, int nz, c32* buf, const AxPlan& p,
                                              const c32* W) {
  constexpr int N = 1 << Q;
  const int lh = p.n - Q;
  const int tasks = TX << lh;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int k = t >> LTX;
    c32 v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const int row = k + (r << lh);
      v[r] = row < nz ? stg[(row << LTX) + col] : mk<float>(0, 0);
    }
    dft_dif<float, Q>(v);
    group_twiddle<float, Q, false>(v, k, 0, W);
#pragma unroll
    for (int r = 0; r < N; ++r) buf[((k + (r << lh)) << LTX) + col] = v[r];
  }
}

// fused middle step of the three face families with the y/z-folded spectra
template <int Q>
__device__ __forceinline__ void z3_fused_yz(c32* buf, size_t tsz, const AxPlan& p,
                                            const PSpec& S, const YzIdx& Y, int kx0,
                                            const c32& ey) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    c32 v[3][N];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
#pragma unroll
      for (int r = 0; r < N; ++r) v[f][r] = buf[f * tsz + ((start + r) << LTX) + col];
      dft_dif<float, Q>(v[f]);
    }
    const c32 ex = spec_cx<float>(S.ex, kx0 + col);
#pragma unroll
    for (int r = 0; r < N; ++r) pspec_apply<float>(S, Y, col, start + r, ex, ey, v[0][r], v[1][r], v[2][r]);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      dft_dit<float, Q>(v[f]);
#pragma unroll
      for (int r = 0; r < N; ++r) buf[f * tsz + ((start + r) << LTX) + col] = v[f][r];
    }
  }
}

// fused middle step of one edge family (real y/z-folded spectrum)
template <int Q>
__device__ __forceinline__ void z1_fused_yz(c32* buf, const AxPlan& p, const float* __restrict__ sy,
                                            const YzIdx& Y) {
  constexpr int N = 1 << Q;
  const int tasks = TX << (p.n - Q);
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int col = t & (TX - 1);
    const int start = (t >> LTX) << Q;
    c32 v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = buf[((start + r) << LTX) + col];
    dft_dif<float, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = cscale(v[r], __ldg(sy + Y.at(col, start + r)));
    dft_dit<float, Q>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) buf[((start + r) << LTX) + col] = v[r];
  }
}

// One family's pencil rows of a tile, for the staging warp.
struct StageSrc {
  const c32* T;  // family buffer at the tile's (ky, kx0)
  int nz;        // occupied z rows
};

// the staging warp (warp 0): arm the barrier with the tile's bytes, then one bulk copy
// per staged row, lanes striding over the rows
__device__ __forceinline__ void stage_tile(uint64_t* bar, c32* stg, int nzs, const StageSrc* src,
                                           int nfam, size_t pl) {
  const int lane = threadIdx.x & 31;
  uint32_t bytes = 0;
  for (int f = 0; f < nfam; ++f) bytes += (uint32_t)src[f].nz * (TX * sizeof(c32));
  if (lane == 0) mbar_arrive_expect_tx(bar, bytes);
  __syncwarp();
  for (int f = 0; f < nfam; ++f)
    for (int z = lane; z < src[f].nz; z += 32)
      bulk_g2s(stg + ((size_t)f * nzs + z) * TX, src[f].T + (size_t)z * pl, TX * sizeof(c32), bar);
}

// every thread waits for the staged tile; false (for all threads alike) if any wait ran
// into its limit, after the copies in flight were waited for once more
__device__ __forceinline__ bool stage_wait(uint64_t* bar, uint32_t parity, int* err) {
  const bool ok = mbar_wait_bounded(bar, parity, ZWAIT_LIMIT);
  if (__syncthreads_and(ok)) return true;
  if (threadIdx.x == 0) atomicExch(err, 1);
  mbar_wait_bounded(bar, parity, ZWAIT_LIMIT);
  return false;
}

template <int Q0, int QL>
__global__ void __launch_bounds__(ZTPB, 3) k_zconv3_staged(c32* T0, c32* T1, c32* T2, int nz0,
                                                           int nz1, int nz2, int nzs, PSpec S,
                                                           int Lx, int Ly, AxPlan p,
                                                           const c32* __restrict__ twm,
                                                           int twmax, int ntiles, int* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int Lz = 1 << p.n;
  const size_t tsz = (size_t)Lz << LTX;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
  c32* W = reinterpret_cast<c32*>(smem_raw + 128);
  c32* buf = W + Lz;             // three work tiles, family f at buf + f*tsz
  c32* stg = buf + 3 * tsz;      // staged rows, family f at stg + f*nzs*TX
  const int ntx = Lx >> LTX;
  const size_t pl = (size_t)Ly * Lx;
  c32* Tf[3] = {T0, T1, T2};
  const int nzf[3] = {nz0, nz1, nz2};
  auto sources = [&](int tile, StageSrc* src) {
    const size_t off = (size_t)(tile / ntx) * Lx + ((tile % ntx) << LTX);
    for (int f = 0; f < 3; ++f) src[f] = StageSrc{Tf[f] + off, nzf[f]};
  };
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  int tile = blockIdx.x;
  if (threadIdx.x < 32 && tile < ntiles) {
    StageSrc src[3];
    sources(tile, src);
    stage_tile(bar, stg, nzs, src, 3, pl);
  }
  load_twiddles<float>(W, twm, twmax, Lz);
  __syncthreads();
  uint32_t parity = 0;
  for (; tile < ntiles; tile += gridDim.x) {
    const int ky = tile / ntx, kx0 = (tile % ntx) << LTX;
    if (!stage_wait(bar, parity, err)) return;
    parity ^= 1u;
    qpick<Q0, QCap<float>::XY>(p.q[0], [&](auto QC) {
      stg_first_fwd<decltype(QC)::value>(stg, nz0, buf, p, W);
      stg_first_fwd<decltype(QC)::value>(stg + (size_t)nzs * TX, nz1, buf + tsz, p, W);
      stg_first_fwd<decltype(QC)::value>(stg + 2 * (size_t)nzs * TX, nz2, buf + 2 * tsz, p, W);
    });
    __syncthreads();
    // the stage is free: fetch the next tile while this one computes
    const int next = tile + gridDim.x;
    if (threadIdx.x < 32 && next < ntiles) {
      fence_proxy_async_smem();
      StageSrc src[3];
      sources(next, src);
      stage_tile(bar, stg, nzs, src, 3, pl);
    }
    {
      int s = p.q[0];
      for (int g = 1; g + 1 < p.ng; ++g) {
        smem_group_q<float, false, LTX>(buf, TX, p.q[g], p.n, s, W);
        smem_group_q<float, false, LTX>(buf + tsz, TX, p.q[g], p.n, s, W);
        smem_group_q<float, false, LTX>(buf + 2 * tsz, TX, p.q[g], p.n, s, W);
        s += p.q[g];
        __syncthreads();
      }
    }
    const YzIdx Y = make_yzidx(Lx, Ly, Lz, kx0, ky);
    const c32 ey = spec_cx<float>(S.ey, ky);
    qpick<QL, QCap<float>::Z3>(p.q[p.ng - 1], [&](auto QC) {
      z3_fused_yz<decltype(QC)::value>(buf, tsz, p, S, Y, kx0, ey);
    });
    __syncthreads();
    {
      int s = p.n - p.q[p.ng - 1];
      for (int g = p.ng - 2; g >= 1; --g) {
        s -= p.q[g];
        smem_group_q<float, true, LTX>(buf, TX, p.q[g], p.n, s, W);
        smem_group_q<float, true, LTX>(buf + tsz, TX, p.q[g], p.n, s, W);
        smem_group_q<float, true, LTX>(buf + 2 * tsz, TX, p.q[g], p.n, s, W);
        __syncthreads();
      }
    }
    const size_t off = (size_t)ky * Lx + kx0;
    qpick<Q0, QCap<float>::XY>(p.q[0], [&](auto QC) {
      col_last_inv<float, decltype(QC)::value>(buf, T0 + off, pl, TX, nz0, p, W);
      col_last_inv<float, decltype(QC)::value>(buf + tsz, T1 + off, pl, TX, nz1, p, W);
      col_last_inv<float, decltype(QC)::value>(buf + 2 * tsz, T2 + off, pl, TX, nz2, p, W);
    });
    __syncthreads();  // the work tiles are rewritten by the next tile's first group
  }
}

// the edge families' z passes in one launch; all share one circulant grid (Lx, Ly, Lz)
struct EdgeSet {
  c32* T[3];
  int nz[3];
  const float* sy[3];
  int nf;
};

template <int Q0, int QL>
__global__ void __launch_bounds__(ZTPB, 4) k_zedge_staged(EdgeSet E, int nzs, int Lx, int Ly,
                                                          AxPlan p, const c32* __restrict__ twm,
                                                          int twmax, int tiles_per_fam,
                                                          int* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int Lz = 1 << p.n;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
  c32* W = reinterpret_cast<c32*>(smem_raw + 128);
  c32* buf = W + Lz;
  c32* stg = buf + ((size_t)Lz << LTX);
  const int ntx = Lx >> LTX;
  const size_t pl = (size_t)Ly * Lx;
  const int ntiles = tiles_per_fam * E.nf;
  auto source = [&](int tile, StageSrc* src) {
    const int f = tile / tiles_per_fam, t = tile - f * tiles_per_fam;
    const size_t off = (size_t)(t / ntx) * Lx + ((t % ntx) << LTX);
    src[0] = StageSrc{E.T[f] + off, E.nz[f]};
  };
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  int tile = blockIdx.x;
  if (threadIdx.x < 32 && tile < ntiles) {
    StageSrc src[1];
    source(tile, src);
    stage_tile(bar, stg, nzs, src, 1, pl);
  }
  load_twiddles<float>(W, twm, twmax, Lz);
  __syncthreads();
  uint32_t parity = 0;
  for (; tile < ntiles; tile += gridDim.x) {
    const int f = tile / tiles_per_fam, t = tile - f * tiles_per_fam;
    const int ky = t / ntx, kx0 = (t % ntx) << LTX;
    const int nz = E.nz[f];
    if (!stage_wait(bar, parity, err)) return;
    parity ^= 1u;
    qpick<Q0, QCap<float>::XY>(p.q[0], [&](auto QC) {
      stg_first_fwd<decltype(QC)::value>(stg, nz, buf, p, W);
    });
    __syncthreads();
    const int next = tile + gridDim.x;
    if (threadIdx.x < 32 && next < ntiles) {
      fence_proxy_async_smem();
      StageSrc src[1];
      source(next, src);
      stage_tile(bar, stg, nzs, src, 1, pl);
    }
    middle_groups<float, false, LTX>(buf, TX, p, W);
    const YzIdx Y = make_yzidx(Lx, Ly, Lz, kx0, ky);
    qpick<QL, QCap<float>::Z1>(p.q[p.ng - 1], [&](auto QC) {
      z1_fused_yz<decltype(QC)::value>(buf, p, E.sy[f], Y);
    });
    __syncthreads();
    middle_groups<float, true, LTX>(buf, TX, p, W);
    const size_t off = (size_t)ky * Lx + kx0;
    qpick<Q0, QCap<float>::XY>(p.q[0], [&](auto QC) {
      col_last_inv<float, decltype(QC)::value>(buf, E.T[f] + off, pl, TX, nz, p, W);
    });
    __syncthreads();
  }
}

// --------------------------------------------------------------------------- pair z passes
// z pass of columns whose occupied rows fill at most half the circulant (nz <= Lz/2 + 1, always
// so here): the even and the odd frequencies are two transforms of half the length h = Lz/2,
//   X(2f)   = FFT_h(x_j + x_{j+h}),      X(2f+1) = FFT_h((x_j - x_{j+h}) w^j),
//   y_j     = E_j + conj(w)^j O_j,       y_{j+h} = E_j - conj(w)^j O_j,
// with only j + h = h ever occupied, so no padding zero is loaded, transformed or multiplied
// and each half's inverse gives just the rows kept. A column's h points sit in the registers of
// G threads, V each (h = V G; V-point transforms over the rows k + G r of thread k, twiddles, a
// transpose through shared memory, G-point transforms); the transform, the spectral product and
// the inverse of a half run between two barriers. The three face families share the threads.
// Spectra: the y/z-folded tables of the half's frequencies go to shared memory by asynchronous
// copies while the rows load and the forward transform runs; both kz and Lz - kz read them.
// The cross blocks' coefficients are formed from the phases of x, y and z (pspec_product).
// FP32 keeps the rows in registers for the second half; the wider types read them again and
// leave the odd half's rows in their place until the even half's are there.
// What bounds them: FP32 instruction issue and loads, float-float the FP32 pipes; the pruning
// halves the arithmetic of the padded transforms. z passes of an operator application at
// 128x128x64, faces + edges: FP32 267 us in the direct and staged forms, 176 here;
// float-float 2541 us direct, 1443 here. FP64 stays direct (see conv_all_t).
template <typename R>
struct ZPairJob {
  cx<R>* T[3];        // face families (edges: T[0] only)
  int nz[3];
  const void* S[6];   // the folded tables (edges: S[0] only)
  const void *ex, *ey, *ez;
  int lx, ly;         // log2 Lx, log2 Ly
  int cta0;
};
template <typename R, int NJ>
struct ZPairSet {
  ZPairJob<R> j[NJ];
  int n;
};

__device__ __forceinline__ void zp_cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void zp_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr int ZP_TPB = 128;
template <typename R, int A, int B, int NF>
struct ZPairShape {
  using ST = typename SpecOf<R>::T;
  static constexpr int V = 1 << A, G = 1 << B, H = V * G, L = 2 * H, C = ZP_TPB / G;
  static constexpr int NT = NF == 3 ? 6 : 1, NS = H / 2 + 1;
  static constexpr bool KEEP = sizeof(R) == 4;
  static constexpr size_t w = 0, ez = w + sizeof(cx<R>) * L,
                          xch = ez + (NF == 3 ? sizeof(cx<R>) * L : 0),
                          spec = xch + (B || !KEEP ? sizeof(cx<R>) * NF * H * C : 0),
                          bytes = spec + sizeof(ST) * NT * NS * C;
};

// one CTA's columns of a pair pass
template <typename R, int A, int B, int NF>
struct ZPairCta {
  using Sh = ZPairShape<R, A, B, NF>;
  using ST = typename Sh::ST;
  static constexpr int V = Sh::V, G = Sh::G, H = Sh::H, L = Sh::L, C = Sh::C, NT = Sh::NT,
                       NS = Sh::NS;
  struct Rows {  // a thread's rows k + G r of every family, and row H (thread k = 0)
    cx<R> d[NF][V];
  };
  const ZPairJob<R>* P;
  cx<R>*W, *Ez, *xch;
  ST* sp;
  int c, k, col0, px, py;
  bool on;
  size_t pl, at0;
  cx<R> ex, ey, q01, xh[NF];

  // the CTA's job and columns; shared memory, the twiddles and the first spectra on their way
  template <typename Set>
  __device__ __forceinline__ void setup(const Set& J, unsigned char* sm, const cx<R>* twm,
                                        int twmax) {
    W = reinterpret_cast<cx<R>*>(sm + Sh::w);
    Ez = reinterpret_cast<cx<R>*>(sm + Sh::ez);
    xch = reinterpret_cast<cx<R>*>(sm + Sh::xch);
    sp = reinterpret_cast<ST*>(sm + Sh::spec);
    int ji = 0;
    if (NF == 1) {
#pragma unroll
      for (int i = 1; i < 3; ++i)
        if (i < J.n && (int)blockIdx.x >= J.j[i].cta0) ji = i;
    }
    P = &J.j[ji];
    const int tid = threadIdx.x, lx = P->lx;
    c = tid % C;
    k = tid / C;
    col0 = ((int)blockIdx.x - P->cta0) * C;
    const int col = col0 + c;
    on = col < (1 << (lx + P->ly));
    px = col & ((1 << lx) - 1);
    py = on ? col >> lx : 0;
    pl = (size_t)1 << (lx + P->ly);
    at0 = ((size_t)py << lx) + px;
    stage(1);
    for (int e = tid; e < L; e += ZP_TPB) {
      W[e] = twm[e * (twmax / L)];
      if (NF == 3) Ez[e] = spec_cx<R>(P->ez, brevn(e, A + B + 1));
    }
    // the column's x and y phases
    ex = ey = q01 = mk<R>(1, 0);
    if (NF == 3 && on) {
      ex = spec_cx<R>(P->ex, px);
      ey = spec_cx<R>(P->ey, py);
      q01 = cmulc(ey, ex);
    }
  }

  // the half's spectra: odd (par 1) or even folded z frequencies of the CTA's columns
  __device__ __forceinline__ void stage(int par) const {
    const int cnt = par ? (H + 1) / 2 : NS, lx = P->lx;
    constexpr int E16 = 16 / sizeof(ST);
    if ((1 << lx) >= C) {
      constexpr int CH = C / E16;  // 16-byte pieces of a row of C columns
      const size_t base =
          (((size_t)fold_pos(col0 >> lx, P->ly) * (H + 1)) << lx) + (col0 & ((1 << lx) - 1));
      for (int e = threadIdx.x; e < NT * cnt * CH; e += ZP_TPB) {
        const int ch = e % CH, i = (e / CH) % cnt, t = e / (CH * cnt);
        zp_cp_async16(sp + ((size_t)t * NS + i) * C + ch * E16,
                      reinterpret_cast<const ST*>(P->S[t]) + base + ((size_t)(2 * i + par) << lx) +
                          ch * E16);
      }
    } else {
      for (int e = threadIdx.x; e < NT * cnt * C; e += ZP_TPB) {
        const int cc = e % C, i = (e / C) % cnt, t = e / (C * cnt);
        const int q = col0 + cc, y = min(q >> lx, (1 << P->ly) - 1);
        sp[((size_t)t * NS + i) * C + cc] = reinterpret_cast<const ST*>(
            P->S[t])[(((size_t)fold_pos(y, P->ly) * (H + 1) + 2 * i + par) << lx) +
                     (q & ((1 << lx) - 1))];
      }
    }
  }

  __device__ __forceinline__ void load(Rows& x) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const cx<R>* T = P->T[f] + at0;
      const int nz = P->nz[f];
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const int n = k + G * r;
        x.d[f][r] = on && n < nz ? ld_stream(T + n * pl) : mk<R>(0, 0);
      }
      xh[f] = on && k == 0 && nz > H ? ld_stream(T + H * pl) : mk<R>(0, 0);
    }
  }

  // one half: transform, spectral product, inverse of the rows in place
  __device__ __forceinline__ void half(Rows& x, int par) const {
#pragma unroll
    for (int f = 0; f < NF; ++f) dft_dif<R, A>(x.d[f]);
    if constexpr (B > 0) {
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const int j = brevq(r, A);
        const cx<R> w = W[2 * j * k];
#pragma unroll
        for (int f = 0; f < NF; ++f)
          xch[((size_t)f * H + j * G + k) * C + c] = j ? x.d[f][r] * w : x.d[f][r];
      }
    }
    zp_cp_wait();
    __syncthreads();
    if constexpr (B > 0) {
#pragma unroll
      for (int f = 0; f < NF; ++f) {
#pragma unroll
        for (int q = 0; q < V / G; ++q) {
#pragma unroll
          for (int t = 0; t < G; ++t)
            x.d[f][q * G + t] = xch[((size_t)f * H + (k + G * q) * G + t) * C + c];
          dft_dif<R, B>(x.d[f] + q * G);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      // frequency j + V m of the half: j the thread's, m the register's (B = 0: j = register)
      const int fr = B > 0 ? (k + G * (i / G)) + V * brevq(i % G, B) : brevq(i, A);
      const int kz = 2 * fr + par, fz = kz <= H ? kz : L - kz;
      const ST* s = sp + (size_t)(fz >> 1) * C + c;
      if constexpr (NF == 1) {
        x.d[0][i] = cscale(x.d[0][i], R(s[0]));
      } else {
        constexpr size_t TS = (size_t)NS * C;
        const cx<R> e = Ez[kz];
        R rr[6];
#pragma unroll
        for (int b = 0; b < 6; ++b) rr[b] = R(s[b * TS]);
        pspec_product<R>(rr, q01, cmulc(ey, e), cmulc(ex, e), x.d[0][i], x.d[1][i], x.d[2][i]);
      }
    }
    if constexpr (B > 0) {
      // back through the cells this thread read itself: no barrier before the writes
#pragma unroll
      for (int f = 0; f < NF; ++f) {
#pragma unroll
        for (int q = 0; q < V / G; ++q) dft_dit<R, B>(x.d[f] + q * G);
      }
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int j = k + G * (i / G), t = i % G;
        const cx<R> w = W[2 * j * t];
#pragma unroll
        for (int f = 0; f < NF; ++f)
          xch[((size_t)f * H + j * G + t) * C + c] = t ? cmulc(x.d[f][i], w) : x.d[f][i];
      }
    }
    __syncthreads();
    if (par) stage(0);
    if constexpr (B > 0) {
#pragma unroll
      for (int f = 0; f < NF; ++f) {
#pragma unroll
        for (int r = 0; r < V; ++r)
          x.d[f][r] = xch[((size_t)f * H + brevq(r, A) * G + k) * C + c];
      }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) dft_dit<R, A>(x.d[f]);
  }

  // rows of family f from its even half e and odd half o (rotated back)
  __device__ __forceinline__ void store(int f, int r, const cx<R>& e, const cx<R>& o) const {
    const int n = k + G * r;
    cx<R>* T = P->T[f] + at0;
    if (on && n < P->nz[f]) st_stream(T + n * pl, e + o);
    if (r == 0 && on && k == 0 && P->nz[f] > H) st_stream(T + H * pl, e - o);
  }
};

template <typename R, int A, int B, int NF, int MINB>
__global__ void __launch_bounds__(ZP_TPB, MINB) k_zpair(ZPairSet<R, NF == 3 ? 1 : 3> J,
                                                        const cx<R>* __restrict__ twm, int twmax) {
  using Cta = ZPairCta<R, A, B, NF>;
  using Sh = typename Cta::Sh;
  constexpr int V = Cta::V, G = Cta::G;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Cta t;
  t.setup(J, smem_raw, twm, twmax);
  // x: the rows, then the odd half's rows; d: the half at work. One copy of the half's code (a
  // loop of two), which stays in the instruction cache.
  typename Cta::Rows x, d;
  t.load(x);
  __syncthreads();  // twiddles and phases are in place
#pragma unroll
  for (int r = 0; r < V; ++r) {
    const cx<R> w = t.W[t.k + G * r];
#pragma unroll
    for (int f = 0; f < NF; ++f) d.d[f][r] = (r == 0 ? x.d[f][r] - t.xh[f] : x.d[f][r]) * w;
  }
#pragma unroll 1
  for (int par = 1;; par = 0) {
    t.half(d, par);
    if (par == 0) break;
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const cx<R> w = t.W[t.k + G * r];
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const cx<R> o = cmulc(d.d[f][r], w);
        d.d[f][r] = r == 0 ? x.d[f][r] + t.xh[f] : x.d[f][r];
        x.d[f][r] = o;
      }
    }
  }
#pragma unroll
  for (int f = 0; f < NF; ++f) {
#pragma unroll
    for (int r = 0; r < V; ++r) t.store(f, r, d.d[f][r], x.d[f][r]);
  }
}

// The pair pass of the wider types: one family's rows in registers at a time, the others in
// shared memory, so that the code of a transform is there once (float-float's two copies of
// three families each ran to some 30,000 instructions, bound by their fetch) and half the
// registers do. Stage 0 starts the odd half, stage 1 ends it and starts the even one, stage 2
// ends that; the odd half's rows wait in the place of the rows read.
template <typename R, int A, int B, int NF, int MINB>
__global__ void __launch_bounds__(ZP_TPB, MINB) k_zpair_wide(ZPairSet<R, NF == 3 ? 1 : 3> J,
                                                             const cx<R>* __restrict__ twm,
                                                             int twmax) {
  using Cta = ZPairCta<R, A, B, NF>;
  using Sh = typename Cta::Sh;
  constexpr int V = Cta::V, G = Cta::G, H = Cta::H, L = Cta::L, C = Cta::C, NS = Cta::NS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Cta t;
  t.setup(J, smem_raw, twm, twmax);
  const int c = t.c, k = t.k;
  __syncthreads();  // twiddles and phases are in place
#pragma unroll 1
  for (int stage = 0; stage < 3; ++stage) {
#pragma unroll 1
    for (int f = 0; f < NF; ++f) {
      cx<R>* T = t.P->T[f] + t.at0;
      const int nz = t.P->nz[f];
      cx<R>* xf = t.xch + (size_t)f * H * C + c;
      cx<R> d[V], x[V], xh = mk<R>(0, 0);
      if (stage < 2 && t.on && k == 0 && nz > H) xh = ld_stream(T + H * t.pl);
      if (stage > 0) {
#pragma unroll
        for (int r = 0; r < V; ++r) d[r] = xf[(brevq(r, A) * G + k) * C];
        dft_dit<R, A>(d);
      }
      // the rows as they were, or (stage 2) the odd half's
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const int n = k + G * r;
        x[r] = t.on && n < nz ? ld_stream(T + n * t.pl) : mk<R>(0, 0);
      }
      if (stage == 2) {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const int n = k + G * r;
          if (t.on && n < nz) st_stream(T + n * t.pl, d[r] + x[r]);
          if (r == 0 && t.on && k == 0 && nz > H) st_stream(T + H * t.pl, d[0] - x[0]);
        }
        continue;
      }
      if (stage == 1) {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const int n = k + G * r;
          const cx<R> o = cmulc(d[r], t.W[n]);
          if (t.on && n < nz) st_stream(T + n * t.pl, o);
        }
      }
      x[0] = stage == 0 ? x[0] - xh : x[0] + xh;
      if (stage == 0) {
#pragma unroll
        for (int r = 0; r < V; ++r) x[r] = x[r] * t.W[k + G * r];
      }
      dft_dif<R, A>(x);
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const int j = brevq(r, A);
        xf[(j * G + k) * C] = (B > 0 && j) ? x[r] * t.W[2 * j * k] : x[r];
      }
    }
    if (stage == 2) break;
    const int par = stage == 0 ? 1 : 0;
    zp_cp_wait();
    __syncthreads();
    // this thread's cells: the rows j = k + G q of the half, every family
    if constexpr (B > 0) {
#pragma unroll 1
      for (int f = 0; f < NF; ++f) {
        cx<R>* xf = t.xch + ((size_t)f * H + k * G) * C + c;
#pragma unroll
        for (int q = 0; q < V / G; ++q) {
          cx<R> d[G];
#pragma unroll
          for (int u = 0; u < G; ++u) d[u] = xf[(q * G * G + u) * C];
          dft_dif<R, B>(d);
#pragma unroll
          for (int u = 0; u < G; ++u) xf[(q * G * G + brevq(u, B)) * C] = d[u];
        }
      }
    }
#pragma unroll 1
    for (int i = 0; i < V; ++i) {
      // B > 0: frequency j + V m at the cell (j, m); B = 0: j at the cell (brev j)
      const int j = B > 0 ? k + G * (i / G) : i, m = B > 0 ? i % G : 0;
      const int fr = j + V * m, kz = 2 * fr + par, fz = kz <= H ? kz : L - kz;
      const typename Cta::ST* s = t.sp + (size_t)(fz >> 1) * C + c;
      cx<R>* x = t.xch + (size_t)(j * G + m) * C + c;
      if constexpr (NF == 1) {
        *x = cscale(*x, R(s[0]));
      } else {
        constexpr size_t TS = (size_t)NS * C, XS = (size_t)H * C;
        const cx<R> e = t.Ez[kz];
        R rr[6];
#pragma unroll
        for (int b = 0; b < 6; ++b) rr[b] = R(s[b * TS]);
        pspec_product<R>(rr, t.q01, cmulc(t.ey, e), cmulc(t.ex, e), x[0], x[XS], x[2 * XS]);
      }
    }
    if constexpr (B > 0) {
#pragma unroll 1
      for (int f = 0; f < NF; ++f) {
        cx<R>* xf = t.xch + ((size_t)f * H + k * G) * C + c;
#pragma unroll
        for (int q = 0; q < V / G; ++q) {
          cx<R> d[G];
#pragma unroll
          for (int u = 0; u < G; ++u) d[u] = xf[(q * G * G + brevq(u, B)) * C];
          dft_dit<R, B>(d);
#pragma unroll
          for (int u = 0; u < G; ++u)
            xf[(q * G * G + u) * C] = u ? cmulc(d[u], t.W[2 * (k + G * q) * u]) : d[u];
        }
      }
    }
    __syncthreads();
    if (par) t.stage(0);
  }
}

// --------------------------------------------------------------------------- host side

// Dynamic shared memory above 48 KB needs a per-kernel opt-in. It is set once per
// kernel instantiation to the device maximum (at context set-up, outside any launch
// sequence), so operator applications only launch kernels.
template <typename K>
static int smem_optin(K kernel, size_t bytes) {
  // kernels sharing a signature share K, so the record is keyed by address and device
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  if (bytes > 227 * 1024) {
    set_error("shared memory tile exceeds 227 KB: z extent too large for the z-pass tiles");
    return PEEC_ERR_UNSUPPORTED_INTERNAL;
  }
  int dev = 0;
  PEEC_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair((const void*)kernel, dev);
  if (!done.count(key)) {
    int maxsm = 0;
    PEEC_CUDA_TRY(cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PEEC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm));
    done.insert(key);
  }
  return 0;
}

// radix plans per pass: x/y passes take up to 16 points per register group at both
// ends; the z passes hold 3 families (P) at the fused step, so their last group is
// smaller (FP64 registers are twice as wide)
template <typename R>
struct Plans {
  static AxPlan xy(int n) { return make_plan(n, 4, 4, 4); }
  static AxPlan z3(int n) {
    return QCap<R>::wide ? make_plan(n, 2, 4, 2) : make_plan(n, 3, 4, 3);
  }
  // alt (FP32 only): the alternative edge plan the tuner may pick (first group 16 points)
  static AxPlan z1(int n, int alt = 0) {
    if (QCap<R>::wide) return make_plan(n, 3, 4, 3);
    return alt ? make_plan(n, 4, 4, 3) : make_plan(n, 4, 4, 4);
  }
};

template <typename R>
struct LinePass;

template <typename R>
struct Launch {
  static cx<R>* buf(const Family& f) { return reinterpret_cast<cx<R>*>(f.T[slot_of<R>()]); }
  // kind 0: forward x, 1: inverse x, 2: forward y, 3: inverse y; io[f]: the compact
  // vector of family f (x passes)
  static int pass(int kind, const Family* F, int nfam, c64* const* io, const cx<R>* tw,
                  int twmax, cudaStream_t st) {
    PassSet<R> s{};
    bool done[kMaxFam] = {};
    if constexpr (!std::is_same<R, double>::value)
      CTX_CHECK(LinePass<R>::run(kind, F, nfam, io, tw, twmax, st, done));
    int ctas = 0;
    size_t sm = 0;
    for (int f = 0; f < nfam; ++f) {
      if (!F[f].active || done[f]) continue;
      if (s.nf == kMaxFam) return set_error("too many families in one pass"), PEEC_ERR_UNSUPPORTED_INTERNAL;
      const Family& fam = F[f];
      FamPass<R>& d = s.f[s.nf++];
      d.T = buf(fam);
      d.map = fam.map;
      d.io = io ? io[f] : nullptr;
      d.cta0 = ctas;
      int gy = fam.dims[2];
      if (kind < 2) {
        const int Lx = fam.L[0];
        d.p = Plans<R>::xy(fam.logL[0]);
        d.L_other = fam.L[1];
        d.a = fam.dims[0];
        d.b = fam.dims[1];
        d.gx = (fam.dims[1] + TY - 1) / TY;
        sm = std::max(sm, sizeof(cx<R>) * (Lx + (size_t)Lx * XRS));
      } else {
        const int Ly = fam.L[1];
        d.p = Plans<R>::xy(fam.logL[1]);
        d.L_other = fam.L[0];
        d.a = kind == 3 ? Ly : fam.dims[1];
        d.b = kind == 3 ? fam.dims[1] : Ly;
        d.gx = (fam.L[0] + TX - 1) / TX;
        sm = std::max(sm, sizeof(cx<R>) * (Ly + ((size_t)Ly << LTX)));
      }
      ctas += d.gx * gy;
    }
    if (s.nf == 0) return 0;
    switch (kind) {
      case 0:
        CTX_CHECK(smem_optin(k_xfwd<R>, sm));
        k_xfwd<R><<<ctas, TPB, sm, st>>>(s, tw, twmax);
        break;
      case 1:
        CTX_CHECK(smem_optin(k_xinv<R>, sm));
        k_xinv<R><<<ctas, TPB, sm, st>>>(s, tw, twmax);
        break;
      case 2:
        CTX_CHECK(smem_optin(k_ypass<R, false>, sm));
        k_ypass<R, false><<<ctas, TPB, sm, st>>>(s, tw, twmax);
        break;
      default:
        CTX_CHECK(smem_optin(k_ypass<R, true>, sm));
        k_ypass<R, true><<<ctas, TPB, sm, st>>>(s, tw, twmax);
        break;
    }
    return 0;
  }
  static int zconv3(const Family* F, const PSpec& S, const cx<R>* tw, int twmax,
                    cudaStream_t st) {
    const int Lz = F[0].L[2];
    const size_t sm = sizeof(cx<R>) * (Lz + 3 * ((size_t)Lz << LTX));
    const AxPlan p = Plans<R>::z3(F[0].logL[2]);
    constexpr int QL = QCap<R>::Z3;
    const bool spec = p.ng >= 2 && p.q[0] == 4 && p.q[p.ng - 1] == QL;
    auto kern = spec ? k_zconv3<R, 4, QL> : k_zconv3<R, 0, 0>;
    CTX_CHECK(smem_optin(kern, sm));
    dim3 g((F[0].L[0] + TX - 1) / TX, F[0].L[1]);
    kern<<<g, ZTPB, sm, st>>>(buf(F[0]), buf(F[1]), buf(F[2]), F[0].dims[2], F[1].dims[2],
                              F[2].dims[2], S, F[0].L[0], F[0].L[1], p, tw, twmax);
    return 0;
  }
  static int zconv1(const Family& f, const void* s, const cx<R>* tw, int twmax, cudaStream_t st,
                    int alt = 0) {
    const int Lz = f.L[2];
    const size_t sm = sizeof(cx<R>) * (Lz + ((size_t)Lz << LTX));
    const AxPlan p = Plans<R>::z1(f.logL[2], alt);
    constexpr int QL = QCap<R>::Z1;
    const int q0 = p.q[0], ql = p.q[p.ng - 1];
    auto kern = (p.ng >= 2 && q0 == 4 && ql == QL) ? k_zconv1<R, 4, QL>
                : (p.ng >= 2 && q0 == 4 && ql == 3)  ? k_zconv1<R, 4, 3>
                : (p.ng >= 2 && q0 == 3 && ql == QL) ? k_zconv1<R, 3, QL>
                                                     : k_zconv1<R, 0, 0>;
    CTX_CHECK(smem_optin(kern, sm));
    dim3 g((f.L[0] + TX - 1) / TX, f.L[1]);
    kern<<<g, ZTPB, sm, st>>>(buf(f), f.dims[2], s, f.L[0], f.L[1], p, tw, twmax);
    return 0;
  }
};

// x and y passes as pairs: kinds as in Launch::pass; a launch per circulant length, done[f]:
// family f was taken (lengths 2 to 512)
template <typename R>
struct LinePass {
  template <int A, int B>
  static int launch(int kind, LineSet<R>& S, const cx<R>* tw, int twmax, cudaStream_t st) {
    using HL = HalfLine<R, A, B>;
    int ctas = 0;
    const int C = kind < 2 ? HL::CX : HL::CY;
    for (int i = 0; i < S.nf; ++i) {
      S.f[i].cta0 = ctas;
      ctas += (S.f[i].lines + C - 1) / C;
    }
    // registers: 80 or 128 (FP32), 128 or 168 (float-float)
    constexpr int MINX = sizeof(R) == 4 ? (HL::V == 16 ? 4 : 6) : (HL::V == 16 ? 3 : 4);
    constexpr int MINY = HL::CY > HL::CX ? (MINX / 2 > 0 ? MINX / 2 : 1) : MINX;
    void (*kern)(LineSet<R>, const cx<R>*, int) =
        kind == 0   ? k_xpair<R, A, B, false, MINX>
        : kind == 1 ? k_xpair<R, A, B, true, MINX>
        : kind == 2 ? k_ypair<R, A, B, false, MINY>
                    : k_ypair<R, A, B, true, MINY>;
    const size_t sm = HL::smem(kind < 2);
    CTX_CHECK(smem_optin(kern, sm));
    kern<<<ctas, C << B, sm, st>>>(S, tw, twmax);
    return 0;
  }
  static int run(int kind, const Family* F, int nfam, c64* const* io, const cx<R>* tw, int twmax,
                 cudaStream_t st, bool* done) {
    const int ax = kind < 2 ? 0 : 1;
    for (int f = 0; f < nfam; ++f) {
      if (done[f] || !line_pair_ok(F[f], ax)) continue;
      LineSet<R> S{};
      for (int g = f; g < nfam; ++g) {
        if (done[g] || !line_pair_ok(F[g], ax) || F[g].L[ax] != F[f].L[ax]) continue;
        LineFam<R>& d = S.f[S.nf++];
        d.T = Launch<R>::buf(F[g]);
        d.map = F[g].map;
        d.io = io ? io[g] : nullptr;
        d.lx = F[g].logL[0];
        d.ly = F[g].logL[1];
        d.n = F[g].dims[ax];
        d.ny = F[g].dims[1];
        d.lines = ax == 0 ? F[g].dims[1] * F[g].dims[2] : F[g].dims[2] << F[g].logL[0];
        done[g] = true;
      }
      // H = V G: four entries a thread up to H = 16, then eight, sixteen at H = 256
      switch (F[f].logL[ax] - 1) {
        case 0: CTX_CHECK((launch<0, 0>(kind, S, tw, twmax, st))); break;
        case 1: CTX_CHECK((launch<1, 0>(kind, S, tw, twmax, st))); break;
        case 2: CTX_CHECK((launch<2, 0>(kind, S, tw, twmax, st))); break;
        case 3: CTX_CHECK((launch<2, 1>(kind, S, tw, twmax, st))); break;
        case 4: CTX_CHECK((launch<2, 2>(kind, S, tw, twmax, st))); break;
        case 5: CTX_CHECK((launch<3, 2>(kind, S, tw, twmax, st))); break;
        case 6: CTX_CHECK((launch<3, 3>(kind, S, tw, twmax, st))); break;
        case 7:
          // FP32 forward y: sixteen entries a thread keep more rows in flight (52 against 60 us at
          // 128x128x64; inverse y 76 against 67, x 53 against 50)
          if (sizeof(R) == 4 && kind == 2) CTX_CHECK((launch<4, 3>(kind, S, tw, twmax, st)));
          else CTX_CHECK((launch<3, 4>(kind, S, tw, twmax, st)));
          break;
        default: CTX_CHECK((launch<4, 4>(kind, S, tw, twmax, st))); break;
      }
    }
    return 0;
  }
};

template <typename R>
struct ZPair {
  template <int A, int B, int NF>
  static int launch(ZPairSet<R, NF == 3 ? 1 : 3>& J, const cx<R>* tw, int twmax, cudaStream_t st) {
    using Sh = ZPairShape<R, A, B, NF>;
    int ctas = 0;
    for (int i = 0; i < J.n; ++i) {
      J.j[i].cta0 = ctas;
      ctas += (int)((((int64_t)1 << (J.j[i].lx + J.j[i].ly)) + Sh::C - 1) / Sh::C);
    }
    constexpr int MINB = sizeof(R) == 4 ? (NF == 3 ? 4 : 6) : 4;
    void (*kern)(ZPairSet<R, NF == 3 ? 1 : 3>, const cx<R>*, int);
    if constexpr (Sh::KEEP) kern = k_zpair<R, A, B, NF, MINB>;
    else kern = k_zpair_wide<R, A, B, NF, MINB>;
    CTX_CHECK(smem_optin(kern, Sh::bytes));
    kern<<<ctas, ZP_TPB, Sh::bytes, st>>>(J, tw, twmax);
    return 0;
  }
  // h = V G: up to eight points a thread, sixteen or more points over several threads
  template <int NF>
  static int by_length(int logh, ZPairSet<R, NF == 3 ? 1 : 3>& J, const cx<R>* tw, int twmax,
                       cudaStream_t st) {
    switch (logh) {
      case 0: return launch<0, 0, NF>(J, tw, twmax, st);
      case 1: return launch<1, 0, NF>(J, tw, twmax, st);
      case 2: return launch<2, 0, NF>(J, tw, twmax, st);
      case 3: return launch<2, 1, NF>(J, tw, twmax, st);
      case 4: return launch<2, 2, NF>(J, tw, twmax, st);
      case 5: return launch<3, 2, NF>(J, tw, twmax, st);
      default: return launch<3, 3, NF>(J, tw, twmax, st);
    }
  }
  static int faces(const Family* F, const PSpec& S, const cx<R>* tw, int twmax, cudaStream_t st) {
    ZPairSet<R, 1> J{};
    J.n = 1;
    ZPairJob<R>& j = J.j[0];
    for (int f = 0; f < 3; ++f) {
      j.T[f] = Launch<R>::buf(F[f]);
      j.nz[f] = F[f].dims[2];
    }
    for (int i = 0; i < 6; ++i) j.S[i] = S.y[i];
    j.ex = S.ex;
    j.ey = S.ey;
    j.ez = S.ez;
    j.lx = F[0].logL[0];
    j.ly = F[0].logL[1];
    return by_length<3>(F[0].logL[2] - 1, J, tw, twmax, st);
  }
  // the edge families, one launch per circulant length; done[f]: taken here
  static int edges(const Family* F, int nfam, const Spectrum* spec, const cx<R>* tw, int twmax,
                   cudaStream_t st, bool* done) {
    for (int f = 3; f < nfam; ++f) {
      if (done[f] || !zpair_ok(F[f])) continue;
      ZPairSet<R, 3> J{};
      for (int g = f; g < nfam; ++g) {
        if (done[g] || !zpair_ok(F[g]) || F[g].L[2] != F[f].L[2]) continue;
        ZPairJob<R>& j = J.j[J.n++];
        j.T[0] = Launch<R>::buf(F[g]);
        j.nz[0] = F[g].dims[2];
        j.S[0] = spec[3 + g].yz[slot_of<R>()];
        j.lx = F[g].logL[0];
        j.ly = F[g].logL[1];
        done[g] = true;
      }
      CTX_CHECK(by_length<1>(F[f].logL[2] - 1, J, tw, twmax, st));
    }
    return 0;
  }
};

template <typename R>
static PSpec pspec_of(const Spectrum* spec, const void* const* ph) {
  const int p = slot_of<R>();
  PSpec S{};
  for (int i = 0; i < 6; ++i) S.y[i] = spec[i].yz[p];
  S.ex = ph[3 * p];
  S.ey = ph[3 * p + 1];
  S.ez = ph[3 * p + 2];
  return S;
}

// The FP32 z-pass forms (ZTune): pairs (k_zpair), direct (k_zconv3 / k_zconv1), staged.
// Templates, so that only the float instantiation compiles their kernels.
template <int UNUSED = 0>
static int zface_f32(const Family* F, int nfam, const PSpec& S, const c32* tw, int twmax,
                     const ZTune& zt, cudaStream_t st) {
  int form = zt.face;
  if (form == 3 && zpair_ok(F[0])) return ZPair<float>::faces(F, S, tw, twmax, st);
  if (form != 2 || !zpass_yz_faces(F, nfam)) return Launch<float>::zconv3(F, S, tw, twmax, st);
  const int Lz = F[0].L[2], Lx = F[0].L[0], Ly = F[0].L[1];
  const AxPlan p = Plans<float>::z3(F[0].logL[2]);
  constexpr int QL = QCap<float>::Z3;
  const bool spec = p.q[0] == 4 && p.q[p.ng - 1] == QL;
  c32* T0 = Launch<float>::buf(F[0]);
  c32* T1 = Launch<float>::buf(F[1]);
  c32* T2 = Launch<float>::buf(F[2]);
  const int nzs = std::max(F[0].dims[2], std::max(F[1].dims[2], F[2].dims[2]));
  const size_t sm = 128 + sizeof(c32) * (Lz + 3 * ((size_t)Lz << LTX) + 3 * (size_t)nzs * TX);
  auto kern = spec ? k_zconv3_staged<4, QL> : k_zconv3_staged<0, 0>;
  CTX_CHECK(smem_optin(kern, sm));
  const int ntiles = (Lx >> LTX) * Ly;
  const int per_sm = std::max(1, std::min(3, (int)((227 * 1024) / (sm + 1024))));
  const int grid = std::min(ntiles, zt.nsm * per_sm);
  kern<<<grid, ZTPB, sm, st>>>(T0, T1, T2, F[0].dims[2], F[1].dims[2], F[2].dims[2], nzs, S,
                               Lx, Ly, p, tw, twmax, ntiles, zt.err);
  return 0;
}

template <int UNUSED = 0>
static int zedge_f32(const Family* F, int nfam, const Spectrum* spec, const c32* tw, int twmax,
                     const ZTune& zt, cudaStream_t st) {
  if (zt.edge != 2 || !zpass_yz_edges(F, nfam)) {
    bool done[kMaxFam] = {};
    if (zt.edge == 3) CTX_CHECK(ZPair<float>::edges(F, nfam, spec, tw, twmax, st, done));
    for (int f = 3; f < nfam; ++f)
      if (F[f].active && !done[f])
        CTX_CHECK(Launch<float>::zconv1(F[f], spec[3 + f].yz[1], tw, twmax, st, zt.edge_plan));
    return 0;
  }
  EdgeSet E{};
  const Family* f0 = nullptr;
  int nzs = 0;
  for (int f = 3; f < nfam; ++f) {
    if (!F[f].active) continue;
    if (!f0) f0 = &F[f];
    E.T[E.nf] = Launch<float>::buf(F[f]);
    E.nz[E.nf] = F[f].dims[2];
    E.sy[E.nf] = (const float*)spec[3 + f].yz[1];
    nzs = std::max(nzs, F[f].dims[2]);
    ++E.nf;
  }
  if (!f0) return 0;
  const int Lz = f0->L[2], Lx = f0->L[0], Ly = f0->L[1];
  const AxPlan p = Plans<float>::z1(f0->logL[2], zt.edge_plan);
  const size_t sm = 128 + sizeof(c32) * (Lz + ((size_t)Lz << LTX) + (size_t)nzs * TX);
  const int q0 = p.q[0], ql = p.q[p.ng - 1];
  auto kern = (q0 == 4 && ql == 3) ? k_zedge_staged<4, 3>
              : (q0 == 3 && ql == 4) ? k_zedge_staged<3, 4>
                                     : k_zedge_staged<0, 0>;
  CTX_CHECK(smem_optin(kern, sm));
  const int per_fam = (Lx >> LTX) * Ly;
  const int per_sm = std::max(1, std::min(4, (int)((227 * 1024) / (sm + 1024))));
  const int grid = std::min(per_fam * E.nf, zt.nsm * per_sm);
  kern<<<grid, ZTPB, sm, st>>>(E, nzs, Lx, Ly, p, tw, twmax, per_fam, zt.err);
  return 0;
}

// ev (nullable): 6 events bracketing the five pass classes
// ph: the face grid's phase tables (x, y, z), complex FP64, then complex FP32
// zt (nullable): the FP32 z-pass forms (form 0 when null)
template <typename R>
int conv_all_t(const Family* F, int nfam, const Spectrum* spec, const void* const* ph,
               const c64* x, c64* LpI, c64* PQ, int64_t m, const cx<R>* tw, int twmax,
               cudaStream_t st, cudaEvent_t* ev, const ZTune* zt) {
  using Lc = Launch<R>;
  const int p = slot_of<R>();
  if (nfam > kMaxFam) return set_error("too many families"), PEEC_ERR_UNSUPPORTED_INTERNAL;
  c64* in[kMaxFam];
  c64* out[kMaxFam];
  for (int f = 0; f < nfam; ++f) {
    in[f] = const_cast<c64*>(F[f].lp ? x : x + m);
    out[f] = F[f].lp ? LpI : PQ;
  }
  if (ev) cudaEventRecord(ev[0], st);
  CTX_CHECK(Lc::pass(0, F, nfam, in, tw, twmax, st));
  if (ev) cudaEventRecord(ev[1], st);
  CTX_CHECK(Lc::pass(2, F, nfam, nullptr, tw, twmax, st));
  if (ev) cudaEventRecord(ev[2], st);
  const PSpec S = pspec_of<R>(spec, ph);
  if constexpr (std::is_same<R, float>::value) {
    const ZTune z0{};
    const ZTune& z = zt ? *zt : z0;
    CTX_CHECK(zface_f32(F, nfam, S, tw, twmax, z, st));
    CTX_CHECK(zedge_f32(F, nfam, spec, tw, twmax, z, st));
  } else {
    // float-float takes the pair passes; FP64 is bound by its pipe and the two forms' counts
    // of operations are alike (128x128x64: 4.42 against 4.57 ms, 57x57x13: 0.25 against 0.22)
    bool done[kMaxFam] = {};
    bool pair = false;
    if constexpr (std::is_same<R, ff>::value) {
      pair = zpair_ok(F[0]);
      if (pair) CTX_CHECK(ZPair<R>::faces(F, S, tw, twmax, st));
      CTX_CHECK(ZPair<R>::edges(F, nfam, spec, tw, twmax, st, done));
    }
    if (!pair) CTX_CHECK(Lc::zconv3(F, S, tw, twmax, st));
    for (int f = 3; f < nfam; ++f)
      if (F[f].active && !done[f])
        CTX_CHECK(Lc::zconv1(F[f], spec[3 + f].yz[p], tw, twmax, st));
  }
  if (ev) cudaEventRecord(ev[3], st);
  CTX_CHECK(Lc::pass(3, F, nfam, nullptr, tw, twmax, st));
  if (ev) cudaEventRecord(ev[4], st);
  CTX_CHECK(Lc::pass(1, F, nfam, out, tw, twmax, st));
  if (ev) cudaEventRecord(ev[5], st);
  return 0;
}

}  // namespace peec
