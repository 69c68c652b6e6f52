// Vector kernels of the Householder GMRES (compact-WY form).
//
// The reflector basis U (N x kmax, column-major) is applied whole instead of the reference's
// one dot and axpy per reflector (gmres_custom.jl:112-127): z = U(:,0:k)^H v, a product with the
// triangular factor T, v -= U(:,0:k) c. Reductions have a fixed order: partials per CTA, then a
// fixed-order sum.
#include <mutex>

#include "ctx.hpp"
#include "peec_gb300.h"

namespace peec {

// Basis storage: complex double (the FP64 solves) or complex float-float (the inner
// solves of the mixed solve), and the arithmetic follows the storage. GB300 runs FP64 at
// about 1/60 of its FP32 rate, and these kernels do eight flops per basis element and
// column, so with FP64 arithmetic they are FP64-pipe bound at a fraction of HBM speed;
// float-float arithmetic (FP32 error-free transformations, ~2^-48) keeps the basis at
// FP64-like accuracy with the same 16 bytes per element and runs at HBM speed.
template <typename T>
struct BasisArith;
template <>
struct BasisArith<c64> {
  using A = double;
  using S = double;  // sums over the lanes
};
template <>
struct BasisArith<cff> {
  using A = ff;
  using S = ffsum;
};
template <typename A, typename T>
__device__ __forceinline__ cx<A> as(const T& v) {
  return mk<A>((A)v.x, (A)v.y);
}
__device__ __forceinline__ double as_double(double v) { return v; }
__device__ __forceinline__ double as_double(ff v) { return ff_join(v); }
template <>
__device__ __forceinline__ cff as<ff, c64>(const c64& v) {
  return mk<ff>(ff_split(v.x), ff_split(v.y));
}
template <>
__device__ __forceinline__ c64 as<double, cff>(const cff& v) {
  return mk<double>(ff_join(v.x), ff_join(v.y));
}

constexpr int KB = 8;        // columns per multi-dot tile
constexpr int RED_TPB = 256;
constexpr int MD_BLOCKS_MAX = 152 * 2;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// partial[c0+c][blk] (complex) = sum over the CTA's rows of conj(U[i,c0+c]) * v[i],
// c < NC: the tile's columns are a template parameter, so loads, products and the
// shuffle reductions are exactly the ones needed; each thread walks at least eight rows
template <int NC>
__global__ void __launch_bounds__(RED_TPB) k_multidot(const c64* __restrict__ U, size_t ldu,
                                                      const c64* __restrict__ v, size_t N,
                                                      int c0, c64* partial) {
  __shared__ double red[RED_TPB / 32][2 * NC];
  c0 += blockIdx.y * NC;
  const c64* __restrict__ Uc = U + (size_t)c0 * ldu;
  double ar[NC], ai[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) ar[c] = ai[c] = 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += stride) {
    c64 u[NC];
    const c64 x = v[i];
#pragma unroll
    for (int c = 0; c < NC; ++c) u[c] = Uc[(size_t)c * ldu + i];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      ar[c] = ar[c] + (u[c].x * x.x + u[c].y * x.y);
      ai[c] = ai[c] + (u[c].x * x.y - u[c].y * x.x);
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const double sr = warp_sum(ar[c]), si = warp_sum(ai[c]);
    if (lane == 0) {
      red[wid][2 * c] = sr;
      red[wid][2 * c + 1] = si;
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * NC) {
    double s = 0.0;
    for (int w = 0; w < RED_TPB / 32; ++w) s += red[w][threadIdx.x];
    const int c = threadIdx.x >> 1;
    double* p = reinterpret_cast<double*>(partial + (size_t)(c0 + c) * gridDim.x + blockIdx.x);
    p[threadIdx.x & 1] = s;
  }
}

// out[c] = sum_b partial[c][b]: one warp per column, lane-strided then a shuffle tree
// (fixed order for a fixed block count)
__global__ void k_reduce_cols(const c64* __restrict__ partial, int nblk, int k, c64* out) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= k) return;  // whole warps leave together
  double sr = 0.0, si = 0.0;
  for (int b = lane; b < nblk; b += 32) {
    const c64 p = partial[(size_t)c * nblk + b];
    sr += p.x;
    si += p.y;
  }
  sr = warp_sum(sr);
  si = warp_sum(si);
  if (lane == 0) out[c] = mk<double>(sr, si);
}

// partial sums of |v[i]|^2 for i >= i0
__global__ void __launch_bounds__(RED_TPB) k_norm2(const c64* __restrict__ v, size_t N, size_t i0,
                                                   double* part) {
  __shared__ double red[RED_TPB / 32];
  double acc = 0.0;
  for (size_t i = i0 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x) {
    const c64 x = v[i];
    acc += x.x * x.x + x.y * x.y;
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < RED_TPB / 32; ++w) s += red[w];
    part[blockIdx.x] = s;
  }
}

// out = sum part[0..nb)
__global__ void k_sum_parts(const double* __restrict__ part, int nb, double* out) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) acc += part[b];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double s = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    s = warp_sum(s);
    if (threadIdx.x == 0) *out = s;
  }
}

// new reflector column: u = (w with entries [0,j) zeroed, w[j] += add) * scale
template <typename UT>
__global__ void k_make_reflector(const c64* __restrict__ w, size_t N, int j, c64 add,
                                 double scale, UT* u) {
  using A = typename BasisArith<UT>::A;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x) {
    c64 x = (i < (size_t)j) ? mk<double>(0, 0) : w[i];
    if (i == (size_t)j) x = x + add;
    const c64 y = cscale(x, scale);
    u[i] = mk<A>((A)y.x, (A)y.y);
  }
}

// out = a - b
__global__ void k_sub(const c64* __restrict__ a, const c64* __restrict__ b, size_t N, c64* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = a[i] - b[i];
}

// out = x + y_pad - sum_c U[i,c] coef[c] where y_pad holds ny leading entries
template <typename UT>
__global__ void k_xupdate(const c64* __restrict__ x, const UT* __restrict__ U, size_t ldu,
                          const c64* __restrict__ coef, const c64* __restrict__ ypad, int k,
                          size_t N, c64* out) {
  using A = typename BasisArith<UT>::A;
  extern __shared__ unsigned char sx_raw[];
  c64* yp = reinterpret_cast<c64*>(sx_raw);                 // k entries
  cx<A>* sc2 = reinterpret_cast<cx<A>*>(sx_raw + sizeof(c64) * k);  // k entries
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    yp[c] = ypad[c];
    sc2[c] = as<A>(coef[c]);
  }
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x) {
    c64 v = x[i];
    if (i < (size_t)k) v = v + yp[i];
    cx<A> s = mk<A>(0, 0);
    for (int c0 = 0; c0 < k; c0 += 8) {
      cx<A> u[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (c0 + q < k) u[q] = as<A>(U[(size_t)(c0 + q) * ldu + i]);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (c0 + q < k) s = s + u[q] * sc2[c0 + q];
    }
    out[i] = v - as<double>(s);
  }
}

__global__ void k_add(const c64* __restrict__ a, const c64* __restrict__ b, size_t N, c64* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = a[i] + b[i];
}

// Small dense triangular products of the compact-WY representation (T upper
// triangular, column-major with leading dimension ld), one CTA.
// mode 0: out = T(0:k,0:k) * in;
// mode 2: T(0:k, k) = -2 T(0:k,0:k) * in, T(k,k) = 2 (append a reflector)
__global__ void k_tri(c64* T, int ld, int k, const c64* __restrict__ in, c64* out, int mode) {
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    c64 s = mk<double>(0, 0);
    for (int j = i; j < k; ++j) s = s + T[(size_t)j * ld + i] * in[j];
    if (mode == 2) out[i] = cscale(s, -2.0);
    else out[i] = s;
  }
  if (mode == 2 && threadIdx.x == 0) out[k] = mk<double>(2.0, 0.0);
}

__device__ __forceinline__ double cabs2(c64 z) { return z.x * z.x + z.y * z.y; }
__device__ __forceinline__ c64 csign(c64 d) {
  if (d.x == 0.0 && d.y == 0.0) return mk<double>(1.0, 0.0);
  const double a = hypot(d.x, d.y);
  return mk<double>(d.x / a, d.y / a);
}

// ------------------------------- Arnoldi iteration --------------------------------
//
// One iteration of the Householder GMRES (gmres_custom.jl:96-171) is three kernels around the
// operator application w = A v. With P1..Pk = I - U T U^H, k = j + 1:
//   k_gm_vec:  v = e_j - U c, c = T conj(Utop(j, :)) from the iteration before; 1/|v|;
//   k_gm_dot:  z = U^H w, then c = T^H z / |v|;
//   k_gm_orth: x = w / |v| - U c; the new reflector u = x with the rows below initer = j + 1
//              zeroed and sign(x(initer)) |tail| added at initer, written as column k of U;
//              t = U^H u and |tail|^2 of the rows; then the scalar step, T(:, k) and the next c.
// The reflector is kept unscaled and its scale goes into T: T(k, k) = 2 / |u|^2 (scaled rows
// would take a second pass over the column). Each kernel ends in its last CTA, so the small
// products over T need no launch of their own; every sum has a fixed order, whichever CTA comes
// last.
// What bounds them: float-float's FP32 pipes (72 instructions a complex product and sum) and
// the basis, read once for v, once for z and twice (then from L1 or L2) for x and t; below some
// 100k rows the latency of the last CTA. FP64 instructions hold their pipe 64 cycles, so
// conversions are integer code, lanes' sums are exchanged in halves (16 additions a warp for
// eight columns instead of 80; of a float-float basis in three FP32 parts, ffsum: in FP64 they
// cost 5.6 % of a mixed solve at 64x64x32, so 1.0 %), and small systems
// spread over CTAs of 32 or 128 rows whose warps share out the columns.
// An iteration outside the operator, mean of a solve: 155 -> 72 us at 64x64x32 (N = 87k), 315 ->
// 200 us at 128x128x64 (N = 750k); the FP64 solve of 20x20x4 (N = 528) 3.49 -> 2.63 ms.
constexpr int GM_TPB = 256, GM_ROWS = 1024, GM_FAN = 16, GM_MAXB = 152 * 2;
constexpr int GM_SCR = 1536;   // complex doubles of shared memory for the last CTA's sums
constexpr int GM_FOLD1 = 8192; // partial sums the last CTA adds up by itself

struct GmGrid {
  unsigned nb, rows;  // CTAs, rows of each
  unsigned vb, vrows; // the same for k_gm_vec, whose registers let four CTAs share an SM
  int wr;             // warps over the rows (8, 4 or 1), the others over the columns
  size_t sm;          // rows held in shared memory and the last CTA's sums
};
// Up to 152 CTAs of 32 rows, then up to 152 of 128, so that every SM has rows and the FP64
// pipes (complex double) or the latency of a column tile (float-float) are shared out; larger
// systems in 256 rows and, from 304 CTAs on, equal parts.
static GmGrid gm_grid(size_t N) {
  GmGrid g;
  if (N <= 152 * 32) {
    g.wr = 1;
    g.rows = 32;
  } else if (N <= 152 * 128) {
    g.wr = 4;
    g.rows = 128;
  } else {
    g.wr = 8;
    g.rows = (unsigned)std::max<size_t>(256, ((N + GM_MAXB - 1) / GM_MAXB + 31) / 32 * 32);
  }
  g.vrows = g.rows;
  if (g.wr == 8)
    g.vrows = (unsigned)std::max<size_t>(256, ((N + 2 * GM_MAXB - 1) / (2 * GM_MAXB) + 31) / 32 * 32);
  g.nb = (unsigned)std::max<size_t>((N + g.rows - 1) / g.rows, 1);
  g.vb = (unsigned)std::max<size_t>((N + g.vrows - 1) / g.vrows, 1);
  g.sm = sizeof(c64) * std::max<size_t>(std::min<size_t>(g.rows, GM_ROWS), GM_SCR);
  return g;
}
// partial sums: two per column of each CTA and of each group
size_t gm_part_doubles(size_t N, int k) {
  const GmGrid g = gm_grid(N);
  return std::max<size_t>(2 * (size_t)(k + 1) * (g.nb + (g.nb + GM_FAN - 1) / GM_FAN), g.vb);
}

__device__ __forceinline__ double shfl_xor(double v, int m) {
  return __shfl_xor_sync(0xffffffffu, v, m);
}

__device__ __forceinline__ ffsum shfl_xor(const ffsum& v, int m) {
  return ffsum{__shfl_xor_sync(0xffffffffu, v.hi, m), __shfl_xor_sync(0xffffffffu, v.lo, m),
               __shfl_xor_sync(0xffffffffu, v.c, m)};
}
// t ? a : b by value: a choice between array elements would put the array in memory
__device__ __forceinline__ double lane_pick(bool t, double a, double b) { return t ? a : b; }
__device__ __forceinline__ ffsum lane_pick(bool t, ffsum a, ffsum b) {
  return ffsum{t ? a.hi : b.hi, t ? a.lo : b.lo, t ? a.c : b.c};
}
__device__ __forceinline__ double lane_sum(double v) { return v; }
__device__ __forceinline__ ffsum lane_sum(ff v) { return ffsum_of(v); }
__device__ __forceinline__ double lane_double(double v) { return v; }
__device__ __forceinline__ double lane_double(const ffsum& v) { return ffsum_double(v); }

// counts the CTA in; true for every thread of the last one, which then sees the others' writes
__device__ __forceinline__ bool gm_last(unsigned* tick, unsigned cnt) {
  __shared__ unsigned last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(tick, 1u) + 1 == cnt;
    if (last) *tick = 0;
  }
  __syncthreads();
  const bool l = last;
  __syncthreads();
  if (l) __threadfence();
  return l;
}

// out[v * os] = sum of in[v * n + i], i < n, v < nv: eight neighbouring lanes a value
__device__ __forceinline__ void gm_sums(const double* in, int nv, int n, double* out, int os) {
  const int l = threadIdx.x & 7;
  for (int v0 = 0; v0 < nv; v0 += GM_TPB / 8) {
    const int v = v0 + (threadIdx.x >> 3);
    double s = 0;
    if (v < nv) {
#pragma unroll 4
      for (int i = l; i < n; i += 8) s += __ldcg(in + (size_t)v * n + i);
    }
    s += shfl_xor(s, 1);
    s += shfl_xor(s, 2);
    s += shfl_xor(s, 4);
    if (v < nv && l == 0) out[(size_t)v * os] = s;
  }
}

// Sums part[v * nb + b] over the CTAs b into out[v], v < nv: true in the CTA that did it, the
// last one; many sums go through groups of GM_FAN CTAs, which lie behind each other (grouped
// layout: part + v * cnt of group grp at nv * GM_FAN * grp).
__device__ __forceinline__ size_t gm_slot(int v, int nv, int nb) {
  if (nv * nb <= GM_FOLD1) return (size_t)v * nb + blockIdx.x;
  const int grp = blockIdx.x / GM_FAN, cnt = min(GM_FAN, nb - grp * GM_FAN);
  return (size_t)nv * GM_FAN * grp + (size_t)v * cnt + (blockIdx.x - grp * GM_FAN);
}
__device__ bool gm_fold(GmDev* gs, double* part, int nv, int nb, double* out) {
  if (nv * nb <= GM_FOLD1) {
    if (!gm_last(&gs->tick[31], nb)) return false;
    gm_sums(part, nv, nb, out, 1);
  } else {
    const int grp = blockIdx.x / GM_FAN, ng = (nb + GM_FAN - 1) / GM_FAN;
    const int cnt = min(GM_FAN, nb - grp * GM_FAN);
    if (!gm_last(&gs->tick[grp], cnt)) return false;
    double* gpart = part + (size_t)nv * nb;
    gm_sums(part + (size_t)nv * GM_FAN * grp, nv, cnt, gpart + grp, ng);
    if (!gm_last(&gs->tick[31], ng)) return false;
    gm_sums(gpart, nv, ng, out, 1);
  }
  __syncthreads();
  return true;
}

// sum of U[i, c] coef[c] over the column chunks of eight that start at c0, c0 + step, ... (a
// chunk's loads before its products)
template <typename UT, typename A>
__device__ __forceinline__ cx<A> gm_row(const UT* __restrict__ U, size_t N, size_t i,
                                        const cx<A>* coef, int k, int c0, int step) {
  cx<A> s = mk<A>(0, 0);
  for (; c0 < k; c0 += step) {
    cx<A> u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (c0 + q < k) u[q] = as<A>(U[(size_t)(c0 + q) * N + i]);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (c0 + q < k) cmac(s, u[q], coef[c0 + q]);
  }
  return s;
}

// fn(r, i, sum of U[i, c] coef[c]) for the rows i = r0 + r, r < nr, of the CTA. WR < 8: at most
// 32 WR rows, the column chunks over 8 / WR warps, whose sums meet in shared memory.
template <int WR, typename UT, typename A, typename F>
__device__ __forceinline__ void gm_rows(const UT* __restrict__ U, size_t N, size_t r0, int nr,
                                        const cx<A>* coef, int k, F fn) {
  constexpr int WC = 8 / WR, NR = 32 * WR;
  const int tid = threadIdx.x;
  if constexpr (WC == 1) {
    for (int r = tid; r < nr; r += GM_TPB)
      fn(r, r0 + r, gm_row<UT, A>(U, N, r0 + r, coef, k, 0, 8));
  } else {
    __shared__ cx<A> ps[WC - 1][NR];
    const int r = tid % NR, wc = tid / NR;
    cx<A> s = mk<A>(0, 0);
    if (r < nr) s = gm_row<UT, A>(U, N, r0 + r, coef, k, 8 * wc, 8 * WC);
    if (wc) ps[wc - 1][r] = s;
    __syncthreads();
    if (wc == 0 && r < nr) {
      for (int q = 0; q < WC - 1 && 8 * (q + 1) < k; ++q) s = s + ps[q][r];
      fn(r, r0 + r, s);
    }
  }
}

// part, values 2c and 2c + 1: (+)= sum over the rows held in sx of conj(U[r0 + r, c]) sx[r];
// column tiles of eight, tile t by the warps of column group t mod 8 / WR
template <int WR, typename UT, typename A>
__device__ void gm_dots(const UT* __restrict__ U, size_t N, size_t r0, int rows, const cx<A>* sx,
                        int k, double* part, int nv, int nb, bool first) {
  constexpr int WC = 8 / WR;
  __shared__ double red[2][WC][WR][2 * KB];
  const int tid = threadIdx.x, lane = tid & 31, wr = (tid >> 5) % WR, wc = (tid >> 5) / WR;
  int buf = 0;
#pragma unroll 1
  for (int t0 = 0; t0 < k; t0 += KB * WC, buf ^= 1) {
    const int c0 = t0 + KB * wc, nc = min(KB, k - c0);
    if (nc > 0) {
      const UT* __restrict__ Uc = U + (size_t)c0 * N + r0;
      cx<A> acc[KB];
#pragma unroll
      for (int c = 0; c < KB; ++c) acc[c] = mk<A>(0, 0);
      for (int r = wr * 32 + lane; r < rows; r += 32 * WR) {
        cx<A> u[KB];
#pragma unroll
        for (int c = 0; c < KB; ++c)
          if (c < nc) u[c] = as<A>(Uc[(size_t)c * N + r]);
        const cx<A> x = sx[r];
#pragma unroll
        for (int c = 0; c < KB; ++c)
          if (c < nc) cmac_conj(acc[c], u[c], x);
      }
      // lanes' sums, with the precision of FP64: halves change hands, so a lane ends with the sum
      // of one of the 16 values
      typename BasisArith<UT>::S d[2 * KB];
#pragma unroll
      for (int c = 0; c < KB; ++c) {
        d[2 * c] = lane_sum(acc[c].x);
        d[2 * c + 1] = lane_sum(acc[c].y);
      }
#pragma unroll
      for (int s = KB; s >= 1; s >>= 1) {
        const bool up = lane & (2 * s);
#pragma unroll
        for (int i = 0; i < s; ++i) {
          const auto o = shfl_xor(lane_pick(up, d[i], d[i + s]), 2 * s);
          d[i] = lane_pick(up, d[i + s], d[i]) + o;
        }
      }
      d[0] = d[0] + shfl_xor(d[0], 1);
      if (!(lane & 1)) red[buf][wc][wr][lane >> 1] = lane_double(d[0]);
    }
    __syncthreads();
    if (tid < WC * 2 * KB) {
      const int g = tid / (2 * KB), v = tid % (2 * KB), val = 2 * (t0 + KB * g) + v;
      if (val < 2 * k) {
        double s = red[buf][g][0][v];
#pragma unroll
        for (int w = 1; w < WR; ++w) s += red[buf][g][w][v];
        double* p = part + gm_slot(val, nv, nb);
        *p = first ? s : *p + s;
      }
    }
  }
}

// the CTA's sum of acc into value v of part
__device__ __forceinline__ void gm_cta_sum(double acc, double* part, int v, int nv, int nb) {
  __shared__ double red[GM_TPB / 32];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = red[0];
    for (int w = 1; w < GM_TPB / 32; ++w) s += red[w];
    part[gm_slot(v, nv, nb)] = s;
  }
}

template <int WR, typename UT>
__global__ void __launch_bounds__(GM_TPB, WR == 8 ? 4 : 2) k_gm_vec(const UT* __restrict__ U, size_t N,
                                                      unsigned rows, GmDev* gs, c64* v,
                                                      double* part, double* rnorm) {
  using A = typename BasisArith<UT>::A;
  extern __shared__ __align__(16) unsigned char gm_smem[];
  cx<A>* coef = reinterpret_cast<cx<A>*>(gm_smem);
  __shared__ double tot[1];
  const int j = gs->j, k = j + 1;
  if (j < 0 || k > gs->inner) return;
  for (int c = threadIdx.x; c < k; c += GM_TPB) coef[c] = as<A>(gs->cvec[c]);
  __syncthreads();
  const size_t row0 = (size_t)blockIdx.x * rows, row1 = min(N, row0 + rows);
  double acc = 0;
  gm_rows<WR, UT, A>(U, N, row0, (int)(row1 - row0), coef, k,
                     [&](int, size_t i, const cx<A>& sum) {
                       const c64 s = as<double>(sum);
                       c64 x = mk<double>(-s.x, -s.y);
                       if (i == (size_t)j) x.x += 1.0;
                       v[i] = x;
                       acc += x.x * x.x + x.y * x.y;
                     });
  gm_cta_sum(acc, part, 0, 1, gridDim.x);
  if (!gm_fold(gs, part, 1, gridDim.x, tot)) return;
  if (threadIdx.x == 0) *rnorm = 1.0 / sqrt(tot[0]);
}

// sink(i, sum over q = i .. k - 1 of T[q * ld + i] h(q)), i < k, by threads 64 to 255: 64 rows
// and three parts of the columns at a time (a warp's FP64 instruction takes its quarter of the
// SM for 64 cycles, so the sums of a row are spread)
template <typename H, typename S>
__device__ __forceinline__ void gm_tri(const c64* T, int ldT, int k, H h, S sink) {
  __shared__ c64 comb[2][64];
  const int part = (threadIdx.x >> 6) - 1, i64 = threadIdx.x & 63;
  for (int i0 = 0; i0 < k; i0 += 64) {
    const int i = i0 + i64;
    c64 s = mk<double>(0, 0);
    if (i < k) {
#pragma unroll 2
      for (int q = i + part; q < k; q += 3) s = s + T[(size_t)q * ldT + i] * h(q);
    }
    if (part) comb[part - 1][i64] = s;
    asm volatile("bar.sync 1, 192;" ::: "memory");
    if (!part && i < k) sink(i, s + comb[0][i64] + comb[1][i64]);
    asm volatile("bar.sync 1, 192;" ::: "memory");
  }
}

// z = U^H w and c = T^H z / |v|; CTA nb: the part of the next v's coefficients from the columns
// there so far, cpart = T conj(Utop(j + 1, :))
template <int WR, typename UT>
__global__ void __launch_bounds__(GM_TPB, 2) k_gm_dot(const UT* __restrict__ U, size_t N,
                                                      unsigned rows, const c64* __restrict__ w,
                                                      const c64* __restrict__ T, int ldT,
                                                      GmDev* gs, double* part,
                                                      const double* __restrict__ rnorm,
                                                      c64* coef) {
  using A = typename BasisArith<UT>::A;
  extern __shared__ __align__(16) unsigned char gm_smem[];
  const int j = gs->j, k = j + 1, tid = threadIdx.x;
  if (j < 0 || k > gs->inner) return;
  const int nb = gridDim.x - 1;
  if ((int)blockIdx.x == nb) {
    if (k >= gs->headlen || tid < 64) return;  // no such row: there is no next iteration
    const c64* h = gs->Utop + k;
    const int ld = gs->ld;
    c64* out = gs->cpart;
    gm_tri(T, ldT, k, [&](int q) { return cconj(h[(size_t)q * ld]); },
           [&](int i, c64 s) { out[i] = s; });
    return;
  }
  cx<A>* sx = reinterpret_cast<cx<A>*>(gm_smem);
  const size_t row0 = (size_t)blockIdx.x * rows, row1 = min(N, row0 + rows);
  for (size_t r0 = row0; r0 < row1; r0 += GM_ROWS) {
    const int nr = (int)min((size_t)GM_ROWS, row1 - r0);
    __syncthreads();
    for (int r = tid; r < nr; r += GM_TPB) sx[r] = as<A>(w[r0 + r]);
    __syncthreads();
    gm_dots<WR, UT, A>(U, N, r0, nr, sx, k, part, 2 * k, nb, r0 == row0);
  }
  __syncthreads();
  c64* z = k <= GM_SCR ? reinterpret_cast<c64*>(gm_smem) : gs->scr;
  if (!gm_fold(gs, part, 2 * k, nb, reinterpret_cast<double*>(z))) return;
  const double inv = *rnorm;
  // four threads a row, neighbouring lanes
  for (int i = tid >> 2; i < k; i += GM_TPB / 4) {
    c64 s = mk<double>(0, 0);
    for (int q = tid & 3; q <= i; q += 4) s = s + cconj(T[(size_t)i * ldT + q]) * z[q];
    const unsigned m = 0xfu << (tid & 28);
    s.x += __shfl_xor_sync(m, s.x, 1);
    s.y += __shfl_xor_sync(m, s.y, 1);
    s.x += __shfl_xor_sync(m, s.x, 2);
    s.y += __shfl_xor_sync(m, s.y, 2);
    if (!(tid & 3)) coef[i] = cscale(s, inv);
  }
}

// The rotations of the earlier columns applied to the new one, by one warp: lanes 0 and 1 run
// the chain cur <- Jc h(c + 1) - Js cur, one the real and one the imaginary part (two dependent
// FMAs a rotation); what is off the chain all lanes form before and after:
// Rc[c] = conj(Jc) cur_c + conj(Js) h(c + 1). h: the column's head; p, js, cu: k entries of
// scratch each. Returns cur (all lanes).
__device__ c64 gm_chain(const c64* h, const c64* J, int j, c64* p, c64* js, c64* cu, c64* Rc) {
  const int lane = threadIdx.x & 31;
  for (int c = lane; c < j; c += 32) {
    p[c] = J[2 * c] * h[c + 1];
    js[c] = J[2 * c + 1];
  }
  __syncwarp();
  double a = lane == 0 ? h[0].x : h[0].y;
  if (lane < 2 && j > 0) {
    double* cud = reinterpret_cast<double*>(cu);
    const double* pd = reinterpret_cast<const double*>(p);
    double pn = pd[lane];
    c64 sn = js[0];
    for (int c = 0; c < j; ++c) {
      const double pc = pn;
      const c64 sc = sn;
      if (c + 1 < j) {
        pn = pd[2 * c + 2 + lane];
        sn = js[c + 1];
      }
      cud[2 * c + lane] = a;
      const double o = __shfl_xor_sync(3u, a, 1);
      // Js cur = (x a - y b, x b + y a), a and b the real and imaginary parts
      a = fma(lane == 0 ? sc.y : -sc.y, o, fma(-sc.x, a, pc));
    }
  }
  __syncwarp();
  const c64 cur = mk<double>(__shfl_sync(0xffffffffu, a, 0), __shfl_sync(0xffffffffu, a, 1));
  for (int c = lane; c < j; c += 32) Rc[c] = cconj(J[2 * c]) * cu[c] + cconj(js[c]) * h[c + 1];
  return cur;
}

// |z|: the plain root where its square neither overflows nor loses digits
__device__ __forceinline__ double gm_abs(const c64& z) {
  const double q = cabs2(z);
  return q > 1e-280 && q < 1e280 ? sqrt(q) : hypot(z.x, z.y);
}

// The end of an iteration, in k_gm_orth's last CTA: sums[0 .. k) = U^H u over the rows beyond
// initer, sums[k].x = |x|^2 of the rows from initer on (gmres_custom.jl:129-171), in FP64:
//   * warp 1: the reflector's entry at initer, its scale, its leading rows in Utop;
//   * warp 0: the earlier Givens rotations applied to the new column, a new rotation that zeroes
//     its subdiagonal, the rotated right-hand side w, the column of R, and |w(initer + 1)|, the
//     residual estimate, into res[initer] and the state;
//   * the others: T(0:k, k) and the coefficients of the next v;
// and the WHILE node's condition: go on while the estimate is above tolb, the cycle has
// iterations left and the host asked for no early exit. Every path sets it, and the iteration
// count grows by one per call, so a loop ends after at most `inner` iterations.
template <typename UT>
__device__ void gm_step(GmDev& g, UT* U, size_t N, c64* T, int ldT, c64* sums, c64* scr,
                        cudaGraphConditionalHandle cond, int use_cond) {
  using A = typename BasisArith<UT>::A;
  const int tid = threadIdx.x, lane = tid & 31;
  const int j = g.j, initer = j + 1, k = j + 1, inner = g.inner, headlen = g.headlen, n = g.n;
  __shared__ c64 sh_a, sh_u;
  __shared__ double sh_tau;
  __shared__ int sh_refl;
  const c64 zero = mk<double>(0, 0);
  c64* Rc = g.R + (size_t)j * inner;
  c64 vj = zero;
  if (tid < 32) {
    vj = gm_chain(g.head, g.J, j, scr, scr + k, scr + 2 * k, Rc);
  } else if (tid == 32) {
    int refl = 0;
    c64 a = zero, u = zero;
    double tau = 0;
    if (initer != n) {
      const double alpha2 = sums[k].x, alpha = sqrt(alpha2);
      if (alpha != 0) {
        const c64 v1 = g.head[initer];
        const double q = cabs2(v1);
        a = q > 1e-280 && q < 1e280 ? cscale(v1, alpha * rsqrt(q)) : cscale(csign(v1), alpha);
        u = v1 + a;
        tau = 2.0 / (alpha2 - q + cabs2(u));
        refl = 1;
      }
      const cx<A> us = as<A>(u);
      U[(size_t)k * N + initer] = us;
      u = as<double>(us);  // as stored
    }
    sh_u = u;
    sh_a = a;
    sh_tau = tau;
    sh_refl = refl;
  }
  __syncthreads();
  const int refl = sh_refl;
  const c64 a = sh_a, ui = sh_u;
  if (tid < 32) {
    // the new column before the rotations: x's head, -a at initer, zero below
    const int nv = min(inner + 1, headlen);
    c64 vj1 = refl ? mk<double>(-a.x, -a.y) : (initer < nv ? g.head[initer] : zero);
    c64 w1 = g.wv[j + 1];
    if (initer != n) {
      const double rho = sqrt(cabs2(vj) + cabs2(vj1));
      // the four quotients by four lanes
      const double q = (lane == 0 ? vj.x : lane == 1 ? vj.y : lane == 2 ? vj1.x : vj1.y) / rho;
      const c64 Jc = mk<double>(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
      const c64 Js = mk<double>(__shfl_sync(0xffffffffu, q, 2), __shfl_sync(0xffffffffu, q, 3));
      const c64 wj = g.wv[j];
      __syncwarp();
      const c64 t = Js * wj;
      w1 = mk<double>(-t.x, -t.y);
      if (lane == 0) {
        g.J[2 * j] = Jc;
        g.J[2 * j + 1] = Js;
        g.wv[j + 1] = w1;
        g.wv[j] = cconj(Jc) * wj;
      }
      vj = mk<double>(rho, 0.0);
      vj1 = zero;
    }
    for (int i = j + 2 + lane; i < inner; i += 32) Rc[i] = refl || i >= nv ? zero : g.head[i];
    if (lane == 0) {
      Rc[j] = vj;
      if (j + 1 < inner) Rc[j + 1] = vj1;
      const double normr = gm_abs(w1);
      g.res[initer] = normr;
      g.normr = normr;
      g.j = initer;
      const bool go = normr > g.tolb && initer < inner && initer != n && !g.exit_now;
      if (use_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
    }
    return;
  }
  if (tid < 64) {
    c64* ucol = g.Utop + (size_t)initer * g.ld;
    for (int i = lane; i < headlen; i += 32)
      ucol[i] = !refl || i < initer ? zero : (i == initer ? ui : g.head[i]);
    return;
  }
  c64* cvec = g.cvec;
  const c64* cpart = g.cpart;
  if (!refl) {
    for (int i = tid - 64; i <= k; i += GM_TPB - 64) cvec[i] = i < k ? cpart[i] : zero;
    return;
  }
  // t: the row at initer joins; then T(0:k, k) = -tau T t
  const double tau = sh_tau;
  for (int c = tid - 64; c < k; c += GM_TPB - 64)
    sums[c] = sums[c] + cconj(as<double>(U[(size_t)c * N + initer])) * ui;
  asm volatile("bar.sync 1, 192;" ::: "memory");
  c64* Tk = T + (size_t)k * ldT;
  gm_tri(T, ldT, k, [&](int q) { return sums[q]; },
         [&](int i, c64 s) {
           s = cscale(s, -tau);
           Tk[i] = s;
           cvec[i] = cpart[i] + s * cconj(ui);
         });
  if (tid == 64) {
    Tk[k] = mk<double>(tau, 0.0);
    cvec[k] = cscale(cconj(ui), tau);
  }
}

template <int WR, typename UT>
__global__ void __launch_bounds__(GM_TPB, 2) k_gm_orth(UT* U, size_t N, unsigned rows,
                                                       const c64* __restrict__ w, c64* T, int ldT,
                                                       GmDev* gs, double* part,
                                                       const double* __restrict__ rnorm,
                                                       const c64* __restrict__ coef_g,
                                                       cudaGraphConditionalHandle cond,
                                                       int use_cond) {
  using A = typename BasisArith<UT>::A;
  extern __shared__ __align__(16) unsigned char gm_smem[];
  const int j = gs->j, k = j + 1, tid = threadIdx.x, nb = gridDim.x, nv = 2 * k + 2;
  if (j < 0 || k > gs->inner) {
    if (use_cond && tid == 0 && blockIdx.x == 0) cudaGraphSetConditional(cond, 0u);
    return;
  }
  cx<A>* sx = reinterpret_cast<cx<A>*>(gm_smem);
  cx<A>* coef = sx + min(rows, (unsigned)GM_ROWS);
  for (int c = tid; c < k; c += GM_TPB) coef[c] = as<A>(coef_g[c]);
  const double inv = *rnorm;
  const size_t head = gs->headlen, initer = (size_t)k;
  c64* headv = gs->head;
  UT* Uk = U + (size_t)k * N;
  const size_t row0 = (size_t)blockIdx.x * rows, row1 = min(N, row0 + rows);
  double acc = 0;
  for (size_t r0 = row0; r0 < row1; r0 += GM_ROWS) {
    const int nr = (int)min((size_t)GM_ROWS, row1 - r0);
    __syncthreads();
    gm_rows<WR, UT, A>(U, N, r0, nr, coef, k, [&](int r, size_t i, const cx<A>& s) {
      // one FP64 subtraction per part; the basis takes its rounding
      const c64 wi = w[i], sd = as<double>(s);
      const c64 xd = mk<double>(fma(wi.x, inv, -sd.x), fma(wi.y, inv, -sd.y));
      if (i < head) headv[i] = xd;
      if (i >= initer) acc += xd.x * xd.x + xd.y * xd.y;
      const cx<A> u = i > initer ? as<A>(xd) : mk<A>(0, 0);
      if (i != initer) Uk[i] = u;
      sx[r] = u;
    });
    __syncthreads();
    gm_dots<WR, UT, A>(U, N, r0, nr, sx, k, part, nv, nb, r0 == row0);
  }
  gm_cta_sum(acc, part, 2 * k, nv, nb);
  if (tid == 0) part[gm_slot(2 * k + 1, nv, nb)] = 0;
  // sums (k + 1), the chain's three arrays (k each)
  c64* scr = 4 * (k + 1) <= GM_SCR ? reinterpret_cast<c64*>(gm_smem) : gs->scr;
  if (!gm_fold(gs, part, nv, nb, reinterpret_cast<double*>(scr))) return;
  gm_step<UT>(*gs, U, N, T, ldT, scr, scr + k + 1, cond, use_cond);
}

__global__ void k_cast_down(const c64* __restrict__ a, size_t N, c32* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = ccast<float>(a[i]);
}

// ------------------------------- launchers ----------------------------------------

static inline unsigned g_stream(size_t n) {
  size_t g = (n + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  if (g < 1) g = 1;
  return (unsigned)g;
}

int red_blocks(size_t N) { return (int)g_stream(N); }

// multi-dot CTAs per column tile: at least 8 rows per thread, at most 2 CTAs per SM
static inline unsigned md_blocks(size_t N) {
  size_t g = (N + 8 * RED_TPB - 1) / (8 * RED_TPB);
  if (g > MD_BLOCKS_MAX) g = MD_BLOCKS_MAX;
  if (g < 1) g = 1;
  return (unsigned)g;
}

// returns the number of kernels launched
int launch_multidot(const c64* U, size_t ldu, const c64* v, size_t N, int k, c64* partial,
                    c64* out, cudaStream_t st) {
  if (k <= 0) return 0;
  const unsigned nb = md_blocks(N);
  const int full = k / KB, rem = k - full * KB;
  if (full) k_multidot<KB><<<dim3(nb, full), RED_TPB, 0, st>>>(U, ldu, v, N, 0, partial);
  const int c0 = full * KB;
  switch (rem) {
    case 1: k_multidot<1><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 2: k_multidot<2><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 3: k_multidot<3><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 4: k_multidot<4><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 5: k_multidot<5><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 6: k_multidot<6><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    case 7: k_multidot<7><<<nb, RED_TPB, 0, st>>>(U, ldu, v, N, c0, partial); break;
    default: break;
  }
  k_reduce_cols<<<(k + 7) / 8, 256, 0, st>>>(partial, nb, k, out);
  return (full ? 1 : 0) + (rem ? 1 : 0) + 1;
}

void launch_norm2(const c64* v, size_t N, size_t i0, double* part, double* out, cudaStream_t st) {
  const unsigned nb = g_stream(N);
  k_norm2<<<nb, RED_TPB, 0, st>>>(v, N, i0, part);
  k_sum_parts<<<1, 1024, 0, st>>>(part, nb, out);
}

void launch_make_reflector(const c64* w, size_t N, int j, c64 add, double scale, c64* u,
                           cudaStream_t st) {
  k_make_reflector<c64><<<g_stream(N), 256, 0, st>>>(w, N, j, add, scale, u);
}
void launch_make_reflector(const c64* w, size_t N, int j, c64 add, double scale, cff* u,
                           cudaStream_t st) {
  k_make_reflector<cff><<<g_stream(N), 256, 0, st>>>(w, N, j, add, scale, u);
}

void launch_sub(const c64* a, const c64* b, size_t N, c64* out, cudaStream_t st) {
  k_sub<<<g_stream(N), 256, 0, st>>>(a, b, N, out);
}

void launch_add(const c64* a, const c64* b, size_t N, c64* out, cudaStream_t st) {
  k_add<<<g_stream(N), 256, 0, st>>>(a, b, N, out);
}

// out += i * b (the imaginary-part convolutions of the Rcc operator joined to the real ones)
__global__ void k_add_i(const c64* __restrict__ b, size_t N, c64* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x) {
    const c64 u = out[i], v = b[i];
    out[i] = mk<double>(u.x - v.y, u.y + v.x);
  }
}

__global__ void k_set_scalar(double* p, double v) { *p = v; }

// *p = v in stream order (the value travels as a kernel argument, so no host buffer has to
// outlive the call)
void launch_set_scalar(double* p, double v, cudaStream_t st) { k_set_scalar<<<1, 1, 0, st>>>(p, v); }

void launch_add_i(const c64* b, size_t N, c64* out, cudaStream_t st) {
  k_add_i<<<g_stream(N), 256, 0, st>>>(b, N, out);
}

// flag |= 1 when a and b differ anywhere (bitwise on the doubles)
__global__ void k_differs(const c64* __restrict__ a, const c64* __restrict__ b, size_t N,
                          int* flag) {
  int d = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
       i += (size_t)gridDim.x * blockDim.x) {
    const c64 u = a[i], v = b[i];
    d |= (__double_as_longlong(u.x) != __double_as_longlong(v.x)) |
         (__double_as_longlong(u.y) != __double_as_longlong(v.y));
  }
  if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

void launch_differs(const c64* a, const c64* b, size_t N, int* flag, cudaStream_t st) {
  k_differs<<<g_stream(N), 256, 0, st>>>(a, b, N, flag);
}

void launch_tri(c64* T, int ld, int k, const c64* in, c64* out, int mode, cudaStream_t st) {
  k_tri<<<1, 256, 0, st>>>(T, ld, k, in, out, mode);
}

// The three kernels of an iteration (see k_gm_vec); gm_pre before and gm_post after w = A v
template <int WR, typename UT>
static int gm_launch(const GmBody& B, UT* U, const GmGrid& g, bool pre) {
  if (pre) {
    k_gm_vec<WR, UT><<<g.vb, GM_TPB, sizeof(c64) * (B.kmax + 1), B.st>>>(U, B.N, g.vrows, B.gs, B.v,
                                                                        B.part, B.scal);
    return 1;
  }
  // up to 24 KB of rows and sums and 32 KB of coefficients; the limit is one for all contexts
  // (the attribute is the function's, and contexts of other sizes launch it from other threads)
  const size_t sm2 = g.sm + sizeof(c64) * (B.kmax + 1);
  cudaFuncSetAttribute(k_gm_orth<WR, UT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  k_gm_dot<WR, UT><<<g.nb + 1, GM_TPB, g.sm, B.st>>>(U, B.N, g.rows, B.w, B.T, B.ldT, B.gs, B.part,
                                                     B.scal, B.coef);
  k_gm_orth<WR, UT><<<g.nb, GM_TPB, sm2, B.st>>>(U, B.N, g.rows, B.w, B.T, B.ldT, B.gs, B.part,
                                                 B.scal, B.coef, B.cond, B.use_cond);
  return 2;
}
template <typename UT>
static int gm_kernels(const GmBody& B, UT* U, bool pre) {
  const GmGrid g = gm_grid(B.N);
  if (g.wr == 1) return gm_launch<1>(B, U, g, pre);
  if (g.wr == 4) return gm_launch<4>(B, U, g, pre);
  return gm_launch<8>(B, U, g, pre);
}

int gm_pre(const GmBody& B) {
  return B.U32 ? gm_kernels(B, B.U32, true) : gm_kernels(B, B.U, true);
}
int gm_post(const GmBody& B) {
  return B.U32 ? gm_kernels(B, B.U32, false) : gm_kernels(B, B.U, false);
}

// the coefficients and the head in shared memory: 64 KB at the longest cycle (2,047 columns). The
// limit beyond 48 KB is one for all contexts, as in gm_launch.
template <typename UT>
static void xupdate(const c64* x, const UT* U, size_t ldu, const c64* coef, const c64* ypad, int k,
                    size_t N, c64* out, cudaStream_t st) {
  const size_t sm = (sizeof(c64) + sizeof(UT)) * (size_t)(k > 0 ? k : 1);
  if (sm > 48 * 1024)
    cudaFuncSetAttribute(k_xupdate<UT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  k_xupdate<UT><<<g_stream(N), 256, sm, st>>>(x, U, ldu, coef, ypad, k, N, out);
}
void launch_xupdate(const c64* x, const c64* U, size_t ldu, const c64* coef, const c64* ypad,
                    int k, size_t N, c64* out, cudaStream_t st) {
  xupdate(x, U, ldu, coef, ypad, k, N, out, st);
}
void launch_xupdate(const c64* x, const cff* U, size_t ldu, const c64* coef, const c64* ypad,
                    int k, size_t N, c64* out, cudaStream_t st) {
  xupdate(x, U, ldu, coef, ypad, k, N, out, st);
}

// ------------------------------------------------------------------------------------
// Allocation-free batched inner products (peec_multidot_noalloc)
//
// Some callers cannot call cudaMalloc at the point where they need these
// reductions: a host runtime whose device memory is entirely owned by its own
// pool allocator, or a latency-critical loop in which the implicit device
// synchronisation of cudaMalloc/cudaFree is not acceptable. For them the partial
// sums live in a fixed file-scope device array instead of caller- or
// context-owned scratch. It holds NOALLOC_BLOCKS x PEEC_NOALLOC_MAX_K complex
// doubles (1.25 MB) and stays resident on every GPU that loads this library until
// the process exits.
// ------------------------------------------------------------------------------------

constexpr int NOALLOC_BLOCKS = MD_BLOCKS_MAX;  // the multi-dot launcher's grid cap
static_assert(NOALLOC_BLOCKS >= MD_BLOCKS_MAX, "scratch smaller than the multi-dot grid");
static __device__ __align__(256) c64 g_noalloc_partials[(size_t)NOALLOC_BLOCKS * PEEC_NOALLOC_MAX_K];

// The array's device address belongs to the CUDA context that loaded this module. A
// cudaDeviceReset or a re-created primary context reloads the module and may move the
// array, so the looked-up address is cached per device together with the unique id of
// the context it was looked up in, and looked up again when the current context differs.
// The two driver calls are reached through the runtime, so the library needs no link
// against libcuda.
struct NoallocSlot {
  unsigned long long ctx_id = 0;
  void* addr = nullptr;
};
static std::mutex g_noalloc_mu;
static NoallocSlot g_noalloc_slot[256];
// held from launch to completion: calls on one device (any thread, any stream) take
// the shared array in turn
static std::mutex g_noalloc_run_mu[256];

typedef int (*drv_ctx_get_current_t)(void** ctx);
typedef int (*drv_ctx_get_id_t)(void* ctx, unsigned long long* id);
static std::once_flag g_drv_once;
static drv_ctx_get_current_t g_ctx_get_current = nullptr;
static drv_ctx_get_id_t g_ctx_get_id = nullptr;

static void resolve_driver_calls() {
  void* f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
          cudaSuccess && q == cudaDriverEntryPointSuccess)
    g_ctx_get_current = (drv_ctx_get_current_t)f;
  f = nullptr;
  if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) ==
          cudaSuccess && q == cudaDriverEntryPointSuccess)
    g_ctx_get_id = (drv_ctx_get_id_t)f;
  cudaGetLastError();
}

// the unique id of the calling thread's current context; 0 when it cannot be told
static unsigned long long current_context_id() {
  std::call_once(g_drv_once, resolve_driver_calls);
  if (!g_ctx_get_current || !g_ctx_get_id) return 0;
  void* c = nullptr;
  unsigned long long id = 0;
  if (g_ctx_get_current(&c) != 0 || !c) return 0;
  if (g_ctx_get_id(c, &id) != 0) return 0;
  return id;
}

}  // namespace peec

extern "C" int peec_multidot_noalloc(const void* U, int64_t ldu, const void* v, int64_t N, int k,
                                     void* out, void* stream) {
  using namespace peec;
  if (!U || !v || !out || N < 1 || ldu < N) {
    set_error("peec_multidot_noalloc: null pointer or N < 1 or ldu < N");
    return PEEC_ERR_BADARG;
  }
  if (k < 1 || k > PEEC_NOALLOC_MAX_K) {
    set_error("peec_multidot_noalloc: k = " + std::to_string(k) + " outside 1.." +
              std::to_string(PEEC_NOALLOC_MAX_K) + " (the fixed scratch holds " +
              std::to_string(PEEC_NOALLOC_MAX_K) + " columns)");
    return PEEC_ERR_BADARG;
  }
  int dev = 0;
  PEEC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) {
    set_error("peec_multidot_noalloc: device ordinal out of range");
    return PEEC_ERR_BADARG;
  }
  void* scratch = nullptr;
  {
    // set-up once per device and context, with that device current: the host-side
    // name of the array is not a device address, so ask the runtime for it. The first
    // lookup in a context loads this module there, which places the array.
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoallocSlot& slot = g_noalloc_slot[dev];
    unsigned long long id = current_context_id();
    if (!slot.addr || id == 0 || slot.ctx_id != id) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
      if (e != cudaSuccess) {
        cudaGetLastError();
        set_error(std::string("peec_multidot_noalloc: could not place the fixed scratch on "
                              "device ") + std::to_string(dev) + " (" + cudaGetErrorString(e) +
                  "); the first call on a device loads the library's device code there");
        return e == cudaErrorMemoryAllocation ? PEEC_ERR_OOM : PEEC_ERR_CUDA;
      }
      if (id == 0) id = current_context_id();  // the lookup made the primary context current
      slot.addr = p;
      slot.ctx_id = id;
    }
    scratch = slot.addr;
  }
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> run(g_noalloc_run_mu[dev]);
  // every partial[c][b] the reduction reads (c < k, b < grid) is written by this call's
  // multi-dot first, so the array needs no clearing between calls
  launch_multidot((const c64*)U, (size_t)ldu, (const c64*)v, (size_t)N, k, (c64*)scratch,
                  (c64*)out, st);
  PEEC_CUDA_TRY(cudaGetLastError());
  PEEC_CUDA_TRY(cudaStreamSynchronize(st));
  return PEEC_OK;
}
