// Block-sparse epilogue of the PEEC operator and its block preconditioner.
//
// After the convolutions have produced LpI = Lp*I (per edge) and PQ = P*Q (per
// surface), the operator rows of compute_Matrix_vector_fft.jl:29-77 are
//   Y1 = jw*LpI + DZ.*I + A*Phi,   Y2 = PQ - Gamma'*Phi,
//   Y3 = -A'*I + Yle*Phi + jw*Gamma*Q,
// and the preconditioner (precond_3_3_vector, :84-146) is applied with one sparse
// LU solve instead of three, using linearity of F\ :
//   M  = F \ (A'*invZ*Y1 - jw*Gamma*invP*Y2 + Y3)
//   y1 = invZ.*(Y1 - A*M),  y2 = invP.*(Y2 + Gamma'*M),  y3 = M.
// A has two entries per edge (-1 at n1, +1 at n2); Gamma one entry per surface.
// Node-side sums use host-built CSR lists (node -> edges, node -> surfaces).
#include <algorithm>
#include <mutex>

#include "ctx.hpp"

namespace peec {

// The operator rows of edges and surfaces that the preconditioner's node sums and the final
// rows need, in one launch. With g = jw*LpI + A*Phi the edge rows are Y1 = DZ.*I + g, so
// invZ.*Y1 = I + V1 with V1 = invZ.*g, and the node sums take A'*(invZ*Y1 - I) = A'*V1: the
// currents cancel before any rounding, and 1/DZ (formed once per frequency) replaces two
// divisions per edge. Surfaces: h = PQ - Phi, V2 = Q - invP.*h.
// Bound by the FP64 pipe (about ten instructions an edge, six a surface) and the gathers: 9.8 us
// at 128x128x64, 17.5 us as two kernels with the divisions.
__global__ void __launch_bounds__(256) k_branch_rows(
    const c64* __restrict__ Q, const c64* __restrict__ Phi, const c64* __restrict__ LpI,
    const c64* __restrict__ PQ, const c64* __restrict__ invZ, const int32_t* __restrict__ n1,
    const int32_t* __restrict__ n2, const int32_t* __restrict__ snode,
    const double* __restrict__ invP, const double* __restrict__ wp, int m, int ns, c64* V1,
    c64* V2, c64* G) {
  const double w = *wp;
  const int total = m + ns;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    if (i < m) {
      const c64 l = LpI[i], a = Phi[n2[i]] - Phi[n1[i]];
      const c64 g = mk<double>(fma(-w, l.y, a.x), fma(w, l.x, a.y));
      G[i] = g;
      V1[i] = g * invZ[i];
    } else {
      const int s = i - m;
      const c64 h = PQ[s] - Phi[snode[s]], q = Q[s];
      const double p = invP[s];
      G[i] = h;
      V2[s] = mk<double>(fma(-p, h.x, q.x), fma(-p, h.y, q.y));
    }
  }
}

// the node sums (NodeSums) as a vector, for solves that are not all in groups
__global__ void k_node_rows(NodeSums S, const int32_t* __restrict__ ne_ptr,
                            const int32_t* __restrict__ ne_idx, const int32_t* __restrict__ ns_ptr,
                            const int32_t* __restrict__ ns_idx, int n, c64* out) {
  const double w = *S.w;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    c64 t = mk<double>(0, 0), q = mk<double>(0, 0);
    for (int p = ne_ptr[v]; p < ne_ptr[v + 1]; ++p) {
      const int code = ne_idx[p];  // 2 * edge + (A = +1)
      const c64 x = S.V1[code >> 1];
      t = (code & 1) ? t + x : t - x;
    }
    for (int p = ns_ptr[v]; p < ns_ptr[v + 1]; ++p) q = q + S.V2[ns_idx[p]];
    // Yle*Phi by itself: a large admittance between two nodes at almost the same potential
    // cancels to a few digits, which a running sum would take from the other terms
    c64 yp = mk<double>(0, 0);
    for (int p = S.yle_ptr[v], e = S.yle_ptr[v + 1]; p < e; ++p)
      yp = yp + S.yle_val[p] * S.Phi[S.yle_col[p]];
    out[v] = mk<double>(fma(-w, q.y, t.x), fma(w, q.x, t.y)) + yp;
  }
}

// y1 = invZ.*(Y1 - A*M) = I + invZ.*(g - A*M), y2 = invP.*(h + Gamma'*M), y3 = M (skipped
// where M already is y's node block); G: g per edge, then h per surface. I and G null: zero.
__global__ void __launch_bounds__(256) k_final_rows(
    const c64* __restrict__ I, const c64* __restrict__ G, const c64* M,
    const c64* __restrict__ invZ, const int32_t* __restrict__ n1, const int32_t* __restrict__ n2,
    const int32_t* __restrict__ snode, const double* __restrict__ invP, int m, int ns, int n,
    c64* y) {
  const int total = M == y + m + ns ? m + ns : m + ns + n;
  const c64 zero = mk<double>(0, 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    if (i < m) {
      const c64 d = (G ? G[i] : zero) - (M[n2[i]] - M[n1[i]]), z = invZ[i];
      const c64 b = I ? I[i] : zero;
      y[i] = mk<double>(b.x + (d.x * z.x - d.y * z.y), b.y + (d.x * z.y + d.y * z.x));
    } else if (i < m + ns) {
      const int s = i - m;
      y[i] = cscale((G ? G[i] : zero) + M[snode[s]], invP[s]);
    } else {
      y[i] = M[i - m - ns];
    }
  }
}

// 1/DZ
__global__ void k_inv_dz(const c64* __restrict__ DZ, int64_t m, c64* invZ) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const c64 d = DZ[e];
    const double den = d.x * d.x + d.y * d.y;
    invZ[e] = mk<double>(d.x / den, -d.y / den);
  }
}

// U's rows times their inverse diagonals (SfTri::sval), one row per thread
__global__ void k_scale_u(const int32_t* __restrict__ ptr, const c64* __restrict__ val,
                          const c64* __restrict__ dinv, int64_t n, c64* sval) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const c64 d = dinv[r];
    for (int p = ptr[r], e = ptr[r + 1]; p < e; ++p) sval[p] = val[p] * d;
  }
}

// ---------------------------------------------------------------------------------------
// sparse LU solve x = Pc * (U \ (L \ (Pr * (Rs .* b)))), both triangles in one launch,
// synchronisation-free: every row carries a ready flag (the solve's epoch once its value
// is final); a warp claims 32 rows of one level at a time from a global counter, in
// level order (all L levels, then all U levels), waits until the rows it depends on are
// flagged, and publishes its results with release stores. A row only ever waits on rows
// claimed before it, by warps that are already running, so the solve always progresses;
// every wait is bounded nonetheless (after the limit the kernel records an error in
// ctl[2] and stops waiting, and all later waits return at once).
// ---------------------------------------------------------------------------------------

__global__ void k_perm_gather(const c64* __restrict__ b, const int32_t* __restrict__ perm,
                              const double* __restrict__ rs, int n, c64* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int j = perm[i];
    out[i] = rs ? cscale(b[j], rs[j]) : b[j];
  }
}

// L2-coherent loads and stores of values other SMs publish during the same launch
__device__ __forceinline__ c64 ld_cg(const c64* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return mk<double>(v.x, v.y);
}
__device__ __forceinline__ void st_cg(c64* p, c64 v) {
  __stcg(reinterpret_cast<double2*>(p), make_double2(v.x, v.y));
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ctl[0] epoch, ctl[1] row claim counter, ctl[2] error flag, ctl[3] unused
__global__ void k_sptrsv_begin(int* ctl) {
  ctl[0] += 1;
  ctl[1] = 0;
  ctl[3] = 0;
}

// One CTA per group (GrpPlan): components of the factors, several small ones packed
// together or one large one. The CTA first brings everything the group's solve reads into
// shared memory -- per row the right-hand side (the terms of its node's sum, one thread a
// term, or b gathered through Pr; scaled by Rs) and the inverse diagonal, per entry its value
// and positions -- by asynchronous copies, all in flight at once. Then the levels of L and of U by
// columns: once a level's values are final, every row with entries in that level's columns
// takes its update, x_i -= a_ij x_j, a barrier, the next level.
//
// What bounds it is the FP64 pipe's latency and issue: on GB300 a warp's FP64 instruction
// holds its sub-partition's pipe for 64 cycles whatever the number of its active lanes
// (19 cycles per instruction with all four sub-partitions busy). By rows, a level's chain is
// a row's whole sum: its products and a tree over the lanes that share it. By columns it is
// the entries in the one level before, mostly one: two instructions, as the real and the
// imaginary part of a product go to two lanes. A lane keeps its row through the level's
// passes (a row with k entries in the level's columns takes k), so that only levels need
// barriers. U's rows come divided by their diagonals (SfTri::sval), which leaves one product
// per row before the U levels; L's columns are divided by theirs while they are staged
// (skipped when L's diagonal is one). The next pass's entries are loaded before the barrier.
// Every row's updates come in a fixed order, so results do not depend on scheduling.
// Measured, one solve with its node sums on an idle GPU: 128x128x64 (183,490 rows, 60,943
// components, 29 levels of L and U in the deepest) 37.8 us; 96x96x48 copper (largest component
// 291 rows) 34.4 us; the 20x20x4 crossbar (one component, 100 levels) 30.0 us. By rows with a
// tree over each row's lanes: 44.4, 39.8 and 57.7 us, and the node sums 46.8, 20.2 and 6.8 us
// in a kernel of their own; one warp per group 72.5 (beside 72.1), 128.1 and 111.4 us.
__device__ __forceinline__ void grp_passes(c64* xs, const c64* ev, const int32_t* eij,
                                           const int32_t* rec, int nrec) {
  const int slot = threadIdx.x >> 1;
  const bool im = threadIdx.x & 1;
  constexpr int SLOTS = SF_GRP_TPB / 2;
  double* xd = reinterpret_cast<double*>(xs) + (im ? 1 : 0);
  auto cnt = [](int r) { return r < 0 ? ~r : r; };
  // an update a = a - c1 x.x + c2 x.y: its row's part, its column, and the coefficients
  // (re -= v.x x.x - v.y x.y, im -= v.y x.x + v.x x.y; the sign by its bit, as a negation
  // may cost an FP64 instruction)
  struct Upd {
    double* a;
    const double2* x;
    double c1, c2;
  };
  const int flip = im ? (int)0x80000000 : 0;
  auto fetch = [&](int e) {
    const int ij = eij[e];
    const c64 v = ev[e];
    return Upd{xd + 2 * (ij & 0xffff), reinterpret_cast<const double2*>(xs + (ij >> 16)),
               im ? v.y : v.x,
               __hiloint2double(__double2hiint(im ? v.x : v.y) ^ flip,
                                __double2loint(im ? v.x : v.y))};
  };
  int off = 0;
  int cur = nrec > 0 ? rec[0] : 0;
  int nxt = nrec > 1 ? rec[1] : 0;
  Upd u = {};
  if (slot < cnt(cur)) u = fetch(slot);
  for (int k = 0; k < nrec; ++k) {
    const int n = cnt(cur);
    const bool bar = cur < 0;
    const int nn = k + 2 < nrec ? rec[k + 2] : 0;
    Upd un = {};
    if (slot < n) {
      const double2 x = *u.x;
      const double a = *u.a;
      // the next pass's first entry, while this one's operands and products are under way
      if (slot < cnt(nxt)) un = fetch(off + n + slot);
      *u.a = fma(u.c2, x.y, fma(-u.c1, x.x, a));
      for (int t = slot + SLOTS; t < n; t += SLOTS) {
        const Upd v = fetch(off + t);
        const double2 y = *v.x;
        *v.a = fma(v.c2, y.y, fma(-v.c1, y.x, *v.a));
      }
    } else if (slot < cnt(nxt)) {
      un = fetch(off + n + slot);
    }
    off += n;
    cur = nxt;
    nxt = nn;
    u = un;
    if (bar) __syncthreads();
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <bool NODE>
__global__ void __launch_bounds__(SF_GRP_TPB) k_sptrsv_grp(GrpPlan P, int g0, int R, int E, int G,
                                                           const c64* __restrict__ Lval,
                                                           const c64* __restrict__ Uval,
                                                           const c64* __restrict__ Ldinv,
                                                           const c64* __restrict__ Udinv,
                                                           const c64* __restrict__ b, NodeSums S,
                                                           const double* __restrict__ rs,
                                                           c64* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char grp_sm[];
  const int tid = threadIdx.x;
  c64* xs = reinterpret_cast<c64*>(grp_sm);
  c64* du = xs + R;
  short4* gi = reinterpret_cast<short4*>(du + R);
  int2* yy = reinterpret_cast<int2*>(gi + R);
  c64* ev = reinterpret_cast<c64*>(yy + R);
  c64* gat = ev + E;
  int32_t* eij = reinterpret_cast<int32_t*>(gat + (NODE ? G : 0));
  int32_t* rec = eij + E;
  const GrpHead h = P.head[g0 + blockIdx.x];
  // indices into registers, then every value straight into shared memory, all in flight
  constexpr int B = 8;
  GrpRow row = {};
  if (tid < h.nr) row = P.rows[h.q0 + tid];
  const int nmax = NODE && h.nt > h.ne ? h.nt : h.ne;
  for (int t0 = tid; t0 < nmax; t0 += B * SF_GRP_TPB) {
    int gi[B], es[B], ej[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * SF_GRP_TPB;
      if (NODE && t < h.nt) gi[u] = P.gsrc[h.t0 + t];
      if (t < h.ne) {
        es[u] = P.esrc[h.e0 + t];
        ej[u] = P.eij[h.e0 + t];
      }
    }
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * SF_GRP_TPB;
      if (NODE && t < h.nt) cp_async16(gat + t, gi[u] >= 0 ? S.V1 + gi[u] : S.V2 + ~gi[u]);
      if (t < h.ne) {
        cp_async16(ev + t, es[u] >= 0 ? Lval + es[u] : Uval + ~es[u]);
        eij[t] = ej[u];
      }
    }
  }
  for (int t = tid; t < h.nrec; t += SF_GRP_TPB) rec[t] = P.rec[h.r0 + t];
  for (int q = tid; q < h.nr; q += SF_GRP_TPB) {
    const GrpRow pr = q == tid ? row : P.rows[h.q0 + q];
    cp_async16(du + q, Udinv + pr.r);
    if (!NODE) cp_async16(xs + q, b + pr.j);
    gi[q] = make_short4(pr.g0, pr.g1, pr.g2, pr.g3);
    yy[q] = make_int2(pr.y0, pr.y1);
  }
  const double w = NODE ? *S.w : 0.0;
  cp_async_wait_all();
  __syncthreads();
  if constexpr (NODE) {
    // two lanes a row: the parts of its node's sum, t + jw s
    const int part = tid & 1;
    const double ws = part ? w : -w;
    double* xd = reinterpret_cast<double*>(xs);
    const double* gt = reinterpret_cast<const double*>(gat) + part;
    const double* gs = reinterpret_cast<const double*>(gat) + 1 - part;
    for (int q = tid >> 1; q < h.nr; q += SF_GRP_TPB / 2) {
      const short4 g = gi[q];
      const int2 y = yy[q];
      double t = 0.0, s = 0.0;
      for (int p = g.x; p < g.y; ++p) t -= gt[2 * p];
      for (int p = g.y; p < g.z; ++p) t += gt[2 * p];
      for (int p = g.z; p < g.w; ++p) s += gs[2 * p];
      t = fma(ws, s, t);
      if (y.x < y.y) {  // Yle*Phi by itself, as in k_node_rows
        c64 yp = mk<double>(0, 0);
        for (int p = y.x; p < y.y; ++p) yp = yp + S.yle_val[p] * S.Phi[S.yle_col[p]];
        t += part ? yp.y : yp.x;
      }
      xd[2 * q + part] = rs ? t * rs[P.rows[h.q0 + q].j] : t;
    }
  } else if (rs) {
    for (int q = tid; q < h.nr; q += SF_GRP_TPB) xs[q] = cscale(xs[q], rs[P.rows[h.q0 + q].j]);
  }
  if (!P.unit_l) {  // L's columns over their diagonals; its rows take theirs with U's
    for (int e = tid; e < h.nl; e += SF_GRP_TPB)
      ev[e] = ev[e] * Ldinv[P.rows[h.q0 + (eij[e] >> 16)].r];
    for (int q = tid; q < h.nr; q += SF_GRP_TPB) du[q] = du[q] * Ldinv[P.rows[h.q0 + q].r];
  }
  __syncthreads();
  grp_passes(xs, ev, eij, rec, h.nrl);
  for (int q = tid; q < h.nr; q += SF_GRP_TPB) xs[q] = xs[q] * du[q];
  __syncthreads();
  grp_passes(xs, ev + h.nl, eij + h.nl, rec + h.nrl, h.nrec - h.nrl);
  for (int q = tid; q < h.nr; q += SF_GRP_TPB) out[q == tid ? row.o : P.rows[h.q0 + q].o] = xs[q];
}

__device__ __forceinline__ void sf_wait(const int* f, int epoch, int* err, int limit) {
  int it = 0;
  while (ld_acquire(f) != epoch) {
    ++it;
    if (it >= limit) {
      atomicExch(err, 1);
      return;
    }
    if ((it & 63) == 0) {
      if (*(volatile int*)err) return;
      __nanosleep(64);
    }
  }
}

constexpr int SF_CHUNK = 4;  // row entries whose column and value are held in registers

__global__ void __launch_bounds__(SF_TPB) k_sptrsv(const int32_t* __restrict__ ord, int nL,
                                                   int total, SfTri L, SfTri U,
                                                   const c64* __restrict__ b,
                                                   const int32_t* __restrict__ g_in,
                                                   const double* __restrict__ rs, c64* y,
                                                   c64* z, int* ctl, int limit) {
  const int lane = threadIdx.x & 31;
  const int epoch = ctl[0];
  int* err = ctl + 2;
  for (;;) {
    int base = 0;
    if (lane == 0) base = atomicAdd(ctl + 1, 32);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= total) break;
    const int r = ord[base + lane];
    if (r >= 0) {
      // L rows: y = L \ (Pr b); U rows: z = U \ y. Separate outputs: a U row may finish
      // while an L row that reads the same index is still pending.
      const bool up = base >= nL;
      const SfTri& T = up ? U : L;
      c64* out = up ? z : y;
      // everything that does not depend on other rows is loaded before the first wait
      const int p0 = T.ptr[r], p1 = T.ptr[r + 1];
      const c64 dr = T.dinv[r];
      c64 acc;
      if (!up) {
        const int j = g_in[r];
        acc = rs ? cscale(b[j], rs[j]) : b[j];
      }
      int cc[SF_CHUNK];
      c64 vv[SF_CHUNK];
#pragma unroll
      for (int q = 0; q < SF_CHUNK; ++q) {
        if (p0 + q < p1) {
          cc[q] = T.col[p0 + q];
          vv[q] = T.val[p0 + q];
        }
      }
      if (up) {
        sf_wait(L.flag + r, epoch, err, limit);
        acc = ld_cg(y + r);
      }
      for (int p = p0; p < p1; p += SF_CHUNK) {
        if (p > p0) {
#pragma unroll
          for (int q = 0; q < SF_CHUNK; ++q) {
            if (p + q < p1) {
              cc[q] = T.col[p + q];
              vv[q] = T.val[p + q];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < SF_CHUNK; ++q) {
          if (p + q < p1) {
            sf_wait(T.flag + cc[q], epoch, err, limit);
            acc = acc - vv[q] * ld_cg(out + cc[q]);
          }
        }
      }
      st_cg(out + r, acc * dr);
      st_release(T.flag + r, epoch);
    }
  }
}

static inline unsigned grid_for(long long n, int tpb = 256) {
  long long g = (n + tpb - 1) / tpb;
  if (g < 1) g = 1;
  if (g > 152 * 16) g = 152 * 16;
  return (unsigned)g;
}

void launch_branch_rows(const c64* Q, const c64* Phi, const c64* LpI, const c64* PQ,
                        const c64* invZ, const int32_t* n1, const int32_t* n2,
                        const int32_t* snode, const double* invP, const double* w, int m, int ns,
                        c64* V1, c64* V2, c64* G, cudaStream_t st) {
  if (m + ns > 0)
    k_branch_rows<<<grid_for((long long)m + ns), 256, 0, st>>>(Q, Phi, LpI, PQ, invZ, n1, n2, snode,
                                                              invP, w, m, ns, V1, V2, G);
}
void launch_node_rows(const NodeSums& S, const int32_t* ne_ptr, const int32_t* ne_idx,
                      const int32_t* ns_ptr, const int32_t* ns_idx, int n, c64* t,
                      cudaStream_t st) {
  k_node_rows<<<grid_for(n), 256, 0, st>>>(S, ne_ptr, ne_idx, ns_ptr, ns_idx, n, t);
}
void launch_final_rows(const c64* I, const c64* G, const c64* M, const c64* invZ,
                       const int32_t* n1, const int32_t* n2, const int32_t* snode,
                       const double* invP, int m, int ns, int n, c64* y, cudaStream_t st) {
  k_final_rows<<<grid_for((long long)m + ns + n), 256, 0, st>>>(I, G, M, invZ, n1, n2, snode,
                                                               invP, m, ns, n, y);
}
void launch_inv_dz(const c64* DZ, int64_t m, c64* invZ, cudaStream_t st) {
  if (m > 0) k_inv_dz<<<grid_for(m), 256, 0, st>>>(DZ, m, invZ);
}
void launch_scale_u(const int32_t* ptr, const c64* val, const c64* dinv, int64_t n, c64* sval,
                    cudaStream_t st) {
  k_scale_u<<<grid_for(n, 128), 128, 0, st>>>(ptr, val, dinv, n, sval);
}
void launch_perm_gather(const c64* b, const int32_t* perm, const double* rs, int n, c64* out,
                        cudaStream_t st) {
  k_perm_gather<<<grid_for(n), 256, 0, st>>>(b, perm, rs, n, out);
}
// Raises the shared memory the group kernel may be launched with on the current device
// to at least smem_bytes (the default limit is 48 KB per block). The limit belongs to the
// kernel, not to a context, so it only ever grows: contexts of other geometries on the
// same device keep what their plans need.
int sptrsv_grp_prepare(size_t smem_bytes) {
  static std::mutex mu;
  static size_t granted[256] = {};
  int dev = 0;
  PEEC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) return fail_cuda(cudaErrorInvalidDevice, "device", __FILE__, __LINE__);
  std::lock_guard<std::mutex> lock(mu);
  // set every time (a re-created context starts from the default again)
  const size_t v = std::max(smem_bytes, granted[dev]);
  PEEC_CUDA_TRY(cudaFuncSetAttribute(k_sptrsv_grp<false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v));
  PEEC_CUDA_TRY(cudaFuncSetAttribute(k_sptrsv_grp<true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v));
  granted[dev] = v;
  return 0;
}

// returns the number of kernels launched. S: the right-hand side is the node sums, formed by
// the groups themselves (only when every row is in a group, GrpPlan::direct); else b.
// One launch over all groups when the large ones fit the shared memory of a few resident
// CTAs; else the large groups go to st2 (forked from st with ev_fork, joined back with
// ev_join; under stream capture the fork and join become graph edges) so that they run
// beside the packed groups without widening these groups' shared memory.
int launch_sptrsv(const GrpPlan& P, cudaStream_t st2, cudaEvent_t ev_fork, cudaEvent_t ev_join,
                  const int32_t* ord, int nL, int total, const SfTri& L, const SfTri& U,
                  const c64* b, const NodeSums* S, const int32_t* g_in, const double* rs, c64* y,
                  c64* z, c64* x, int* ctl, cudaStream_t st) {
  int launches = 0;
  c64* out = P.direct ? x : z;
  auto groups = [&](int a, int e, int R, int E, int K, int G, cudaStream_t s) {
    if (e <= a) return;
    if (S)
      k_sptrsv_grp<true><<<e - a, SF_GRP_TPB, grp_smem(R, E, K, G), s>>>(
          P, a, R, E, G, L.val, U.sval, L.dinv, U.dinv, nullptr, *S, rs, out);
    else
      k_sptrsv_grp<false><<<e - a, SF_GRP_TPB, grp_smem(R, E, K, 0), s>>>(
          P, a, R, E, 0, L.val, U.sval, L.dinv, U.dinv, b, NodeSums(), rs, out);
    ++launches;
  };
  const int R = std::max(P.rb, P.rp), E = std::max(P.eb, P.ep), K = std::max(P.kb, P.kp),
            G = std::max(P.gb, P.gp);
  if (P.nbig == 0 || P.nbig == P.ngroups || grp_smem(R, E, K, S ? G : 0) <= SF_ONE_LAUNCH_SMEM) {
    groups(0, P.ngroups, R, E, K, G, st);
  } else {
    if (st2) {
      cudaEventRecord(ev_fork, st);
      cudaStreamWaitEvent(st2, ev_fork, 0);
    }
    groups(0, P.nbig, P.rb, P.eb, P.kb, P.gb, st2 ? st2 : st);
    if (st2) cudaEventRecord(ev_join, st2);
    groups(P.nbig, P.ngroups, P.rp, P.ep, P.kp, P.gp, st);
    if (st2) cudaStreamWaitEvent(st, ev_join, 0);
  }
  if (total <= 0) return launches;
  k_sptrsv_begin<<<1, 1, 0, st>>>(ctl);
  launches += 2;
  // at most two CTAs (eight warps) per SM: warps that wait on earlier rows take issue
  // slots from kernels of other streams, and more warps do not shorten the chain of
  // levels (the widest level at 128x128x64 is about 1,400 warp batches)
  const int warps = (total + 31) / 32;
  int blocks = (warps + SF_TPB / 32 - 1) / (SF_TPB / 32);
  if (blocks > 152 * 2) blocks = 152 * 2;
  if (blocks < 1) blocks = 1;
  k_sptrsv<<<blocks, SF_TPB, 0, st>>>(ord, nL, total, L, U, b, g_in, rs, y, z, ctl,
                                        1 << 20);
  return launches;
}

// The bounded-wait failure path of k_sptrsv on a two-row lower triangle whose second row
// depends on the first, with only the second row in the claim order: the first row's
// flag is never set, so the dependency wait runs into `limit` polls, records the error
// word and returns. Returns the error word (1 when the wait gave up).
int selftest_wait_limit(int limit, cudaStream_t st, int* err_out) {
  struct Host {
    int32_t ptr[3] = {0, 0, 1};
    int32_t col[1] = {0};
    c64 val[1];
    c64 dinv[2];
    int32_t ord[32];
    c64 b[2];
    int32_t g_in[2] = {0, 1};
    int ctl[4] = {0, 0, 0, 0};
    int flag[2] = {0, 0};
  } h;
  h.val[0] = mk<double>(0.5, 0);
  h.dinv[0] = h.dinv[1] = mk<double>(1, 0);
  h.b[0] = h.b[1] = mk<double>(1, 0);
  h.ord[0] = 1;
  for (int i = 1; i < 32; ++i) h.ord[i] = -1;
  Host* d = nullptr;
  c64* yz = nullptr;
  PEEC_CUDA_TRY(cudaMalloc(&d, sizeof(Host)));
  if (cudaMalloc(&yz, 4 * sizeof(c64)) != cudaSuccess) {
    cudaFree(d);
    return fail_cuda(cudaErrorMemoryAllocation, "selftest buffers", __FILE__, __LINE__);
  }
  cudaMemcpyAsync(d, &h, sizeof(Host), cudaMemcpyHostToDevice, st);
  SfTri L{d->ptr, d->col, d->val, d->dinv, d->flag};
  SfTri U = L;
  k_sptrsv_begin<<<1, 1, 0, st>>>(d->ctl);
  k_sptrsv<<<1, SF_TPB, 0, st>>>(d->ord, 32, 32, L, U, d->b, d->g_in, nullptr, yz, yz + 2, d->ctl,
                                  limit);
  int e = 0;
  cudaMemcpyAsync(&e, d->ctl + 2, sizeof(int), cudaMemcpyDeviceToHost, st);
  const cudaError_t rc = cudaStreamSynchronize(st);
  cudaFree(d);
  cudaFree(yz);
  if (rc != cudaSuccess) return fail_cuda(rc, "selftest_wait_limit", __FILE__, __LINE__);
  *err_out = e;
  return 0;
}

}  // namespace peec
