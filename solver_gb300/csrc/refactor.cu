// Numeric refactorisation of SS = Yle + A' diag(1/DZ) A + jw Gamma diag(1/P) Gamma' on the
// device, per frequency, in the pattern and permutations of a host factorisation done
// once (the reference factorises with UMFPACK on the host at every frequency,
// FFT_solver_QS_S_type.jl:118-119). SS's structure does not depend on the frequency, so
// the fill of Pr SS Pc = L U in a fixed pivot order does not either; SS is close to
// diagonally dominant (off-diagonal row sums at most ~1.04 of the diagonal's magnitude
// on the benchmark grids), so keeping the first frequency's pivot order is stable. Every
// pivot is checked: zero or non-finite pivots set an error word the host reports.
//
//   assemble: every slot of L (off-diagonal), of the diagonal D and of U (off-diagonal)
//             is the sum of its SS contributions, in a fixed order per slot (edges'
//             +-1/DZ, surfaces' jw/P, Yle entries); slots of fill start at zero
//   rows:     up-looking, a group of lanes per permuted row, rows of one L level per launch
//             (a row depends on the rows of its L pattern, all of earlier levels):
//               for k in L(p,:) in increasing order: L(p,k) = w(k) / D(k);
//                 w(j) -= L(p,k) U(k,j) for j in U(k,:)   (targets precomputed)
//             then D(p) is final; U.dinv(p) = 1 / D(p), L's diagonal stays 1
#include "ctx.hpp"

namespace peec {

// contribution codes of asm_src: type in the top two bits, index below
constexpr int RF_TPB = 128;
constexpr int RF_WIDE = 152 * 32;  // rows of a level that get a warp each at most
constexpr uint32_t RF_EDGE_DIAG = 0u, RF_EDGE_OFF = 1u, RF_SURF = 2u, RF_YLE = 3u;

__global__ void k_rf_assemble(int64_t nslot, const int64_t* __restrict__ ptr,
                              const uint32_t* __restrict__ src, const c64* __restrict__ invZ,
                              const double* __restrict__ invP, const c64* __restrict__ yle,
                              double w, int64_t nL, int64_t n, c64* Lval, c64* D, c64* Uval) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < nslot;
       s += (int64_t)gridDim.x * blockDim.x) {
    c64 acc = mk<double>(0, 0);
    for (int64_t q = ptr[s]; q < ptr[s + 1]; ++q) {
      const uint32_t code = src[q];
      const uint32_t t = code >> 30, i = code & 0x3fffffffu;
      if (t == RF_EDGE_DIAG || t == RF_EDGE_OFF) {
        const c64 iz = invZ[i];
        acc = t == RF_EDGE_DIAG ? acc + iz : acc - iz;
      } else if (t == RF_SURF) {
        acc = acc + mk<double>(0.0, w * invP[i]);
      } else {
        acc = acc + yle[i];
      }
    }
    if (s < nL) Lval[s] = acc;
    else if (s < nL + n) D[s - nL] = acc;
    else Uval[s - nL - n] = acc;
  }
}

// x / d from r = 1 / d rounded to nearest: the quotient's estimate corrected by its remainder
// (Markstein, IBM J. Res. Dev. 34, 1990), three dependent operations where a division takes some
// ten; plain division where the reciprocal leaves the range the correction needs. 4e8 random
// quotients, significands of all ones and zeros among them, gave the division's bits.
__device__ __forceinline__ double rf_quot(double x, double d, double r) {
  const double q = x * r;
  const double y = fma(fma(-q, d, x), r, q);
  return r > 1e-250 && r < 1e250 ? y : x / d;
}

// upd_tgt codes: -1 the row's own diagonal; bit 30 set: U.val index (low 30 bits); else
// L.val index
//
// LN lanes a row: the L entries in order, each one's updates over the lanes (a row's slots are
// distinct, and each gets its updates in the order of the L entries, so the sums are those of
// one thread). The row is worked on in shared memory (SM; cap: its entries at most), and the next
// entry's pivot and first updates are on their way while one is applied: what is left of an
// entry's latency is a quotient, a complex product and a difference, some 0.3 us. One thread a row, in
// global memory, took 25 to 41 us a level (22 levels 0.93 ms at 128x128x64, 18 levels 0.46 ms at
// 48x48x24); they take 0.72 and 0.31 ms so.
template <int LN, bool SM>
__global__ void __launch_bounds__(RF_TPB) k_rf_rows(const int32_t* __restrict__ rows, int nrows,
                                                    SfTri L, SfTri U, c64* D,
                                                    const int32_t* __restrict__ upd_off,
                                                    const int32_t* __restrict__ upd_tgt, int cap,
                                                    int* err) {
  extern __shared__ __align__(16) unsigned char rf_smem[];
  const int g = threadIdx.x / LN, lane = threadIdx.x % LN;
  const int t = blockIdx.x * (RF_TPB / LN) + g;
  if (t >= nrows) return;  // whole groups
  const unsigned mask =
      LN == 32 ? 0xffffffffu : ((1u << (LN & 31)) - 1u) << ((threadIdx.x & 31) / LN * LN);
  const int p = rows[t];
  c64* Lval = const_cast<c64*>(L.val);
  c64* Uval = const_cast<c64*>(U.val);
  const int l0 = L.ptr[p], nl = L.ptr[p + 1] - l0, u0 = U.ptr[p], nu = U.ptr[p + 1] - u0;
  c64* w = reinterpret_cast<c64*>(rf_smem) + (size_t)g * cap;
  // the row's entry i: its L entries, the diagonal, its U entries
  auto at = [&](int i) -> c64* {
    if (SM) return w + i;
    return i < nl ? Lval + l0 + i : (i == nl ? D + p : Uval + u0 + (i - nl - 1));
  };
  if (SM) {
    for (int i = lane; i < nl; i += LN) w[i] = Lval[l0 + i];
    for (int i = lane; i < nu; i += LN) w[nl + 1 + i] = Uval[u0 + i];
    if (lane == 0) w[nl] = D[p];
  }
  __syncwarp(mask);
  // of an L entry: its pivot, its updates' range, this lane's first target and factor
  struct Step {
    c64 d, u;
    double den, r;  // |d|^2 and its reciprocal
    int e0, e1, uk, tg;
  };
  auto fetch = [&](int q) {
    Step s;
    const int k = L.col[l0 + q];
    s.e0 = upd_off[l0 + q];
    s.e1 = upd_off[l0 + q + 1];
    s.uk = U.ptr[k];
    s.d = D[k];
    s.den = s.d.x * s.d.x + s.d.y * s.d.y;
    s.r = 1.0 / s.den;
    s.tg = 0;
    s.u = mk<double>(0, 0);
    if (s.e0 + lane < s.e1) {
      s.tg = upd_tgt[s.e0 + lane];
      s.u = Uval[s.uk + lane];
    }
    return s;
  };
  auto slot = [&](int tg) {
    return tg < 0 ? nl : (tg & 0x40000000) ? nl + 1 + (tg & 0x3fffffff) - u0 : tg - l0;
  };
  if (nl > 0) {
    Step s = fetch(0);
    for (int q = 0; q < nl; ++q) {
      const Step c = s;
      if (q + 1 < nl) s = fetch(q + 1);
      const c64 z = *at(q);
      const c64 l = mk<double>(rf_quot(z.x * c.d.x + z.y * c.d.y, c.den, c.r),
                               rf_quot(z.y * c.d.x - z.x * c.d.y, c.den, c.r));
      if (c.e0 + lane < c.e1) {
        c64* x = at(slot(c.tg));
        *x = *x - l * c.u;
      }
      for (int e = c.e0 + lane + LN; e < c.e1; e += LN) {
        c64* x = at(slot(upd_tgt[e]));
        *x = *x - l * Uval[c.uk + (e - c.e0)];
      }
      __syncwarp(mask);
      if (lane == 0) *at(q) = l;
    }
    __syncwarp(mask);
  }
  if (SM) {
    for (int i = lane; i < nl; i += LN) Lval[l0 + i] = w[i];
    for (int i = lane; i < nu; i += LN) Uval[u0 + i] = w[nl + 1 + i];
  }
  if (lane == 0) {
    const c64 d = *at(nl);
    if (SM) D[p] = d;
    const double den = d.x * d.x + d.y * d.y;
    if (!(den > 0.0) || !isfinite(den)) atomicExch(err, 1);
    const_cast<c64*>(U.dinv)[p] = mk<double>(d.x / den, -d.y / den);
    const_cast<c64*>(L.dinv)[p] = mk<double>(1.0, 0.0);
  }
}

int refactor_launch(const RefactorPlan& R, const SfTri& L, const SfTri& U, c64* Lval, c64* Uval,
                    const c64* invZ, const double* invP, const c64* yle, double w, int* err,
                    cudaStream_t st) {
  const int64_t nslot = R.nL + R.n + R.nU;
  int64_t blocks = (nslot + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (blocks < 1) blocks = 1;
  k_rf_assemble<<<(unsigned)blocks, 256, 0, st>>>(nslot, R.asm_ptr, R.asm_src, invZ, invP, yle, w,
                                                  R.nL, R.n, Lval, R.D, Uval);
  int launches = 1;
  for (size_t l = 0; l + 1 < R.lvl_off.size(); ++l) {
    const int a = R.lvl_off[l], b = R.lvl_off[l + 1];
    if (b <= a) continue;
    // a level of few rows (the upper ones, with long rows) gives each a warp, the others eight
    // lanes; rows beyond 48 KB a CTA stay in global memory
    const int cap = R.lvl_cap[l], ln = b - a <= RF_WIDE ? 32 : 8, per = RF_TPB / ln;
    const size_t sm = sizeof(c64) * (size_t)cap * per;
    const bool in_sm = sm <= 48 * 1024;
    auto kern = ln == 32 ? (in_sm ? k_rf_rows<32, true> : k_rf_rows<32, false>)
                         : (in_sm ? k_rf_rows<8, true> : k_rf_rows<8, false>);
    kern<<<(b - a + per - 1) / per, RF_TPB, in_sm ? sm : 0, st>>>(R.rows + a, b - a, L, U, R.D,
                                                                  R.upd_off, R.upd_tgt, cap, err);
    ++launches;
  }
  PEEC_CUDA_TRY(cudaGetLastError());
  return launches;
}

// The per-frequency edge impedances DZ on the device (FFT_solver_QS_S_type.jl:105-114):
//   Z_self = sum over the four edge halves of 1/(1/R + jw Cd), R, or 1/(jw Cd) where only
//            one of them is present (compute_Z_self.jl:1-15);
//   Zs     = escal_R * Zs0 * sqrt(w / escal_freq) (real part);
//   on surface edges: Z_self keeps only its imaginary part where Zs > Re(Z_self), Zs is
//            dropped where Zs < Re(Z_self);
//   DZ     = Z_self + Zs + jw Lp_self.
// The arithmetic is that of the host state (frequency.FrequencyState): the same
// operations on doubles, one edge per thread.
__global__ void k_edge_dz(int64_t m, const double* __restrict__ R4, const double* __restrict__ Cd4,
                          const double* __restrict__ Lpd, const double* __restrict__ Zs0,
                          const uint8_t* __restrict__ surf, double escal_R, double sq, double w,
                          c64* DZ) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m;
       e += (int64_t)gridDim.x * blockDim.x) {
    double zr = 0.0, zi = 0.0;
    for (int a = 0; a < 4; ++a) {
      const double r = R4[4 * e + a], cd = Cd4[4 * e + a];
      if (r != 0.0 && cd != 0.0) {
        // 1 / (1/r + j w cd)
        const double p = 1.0 / r, q = w * cd;
        const double den = p * p + q * q;
        zr += p / den;
        zi += -q / den;
      } else if (r != 0.0) {
        zr += r;
      } else if (cd != 0.0) {
        // 1 / (j w cd) = -j / (w cd)
        zi += -1.0 / (w * cd);
      }
    }
    double zs = escal_R * (Zs0[e] * sq);
    if (surf[e]) {
      const double d = zs - zr;
      if (d > 0) zr = 0.0;
      else if (d < 0) zs = 0.0;
    }
    DZ[e] = mk<double>(zr + zs, zi + w * Lpd[e]);
  }
}

void launch_edge_dz(int64_t m, const double* R4, const double* Cd4, const double* Lpd,
                    const double* Zs0, const uint8_t* surf, double escal_R, double sq, double w,
                    c64* DZ, cudaStream_t st) {
  int64_t b = (m + 255) / 256;
  if (b > 152 * 8) b = 152 * 8;
  if (b < 1) b = 1;
  k_edge_dz<<<(unsigned)b, 256, 0, st>>>(m, R4, Cd4, Lpd, Zs0, surf, escal_R, sq, w, DZ);
}

}  // namespace peec
