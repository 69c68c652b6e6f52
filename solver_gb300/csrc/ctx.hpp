// Internal declarations shared by the translation units of libpeec_gb300.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "common.cuh"

namespace peec {

int fail_cuda(cudaError_t e, const char* expr, const char* file, int line);
void set_error(const std::string& msg);

#define PEEC_ERR_UNSUPPORTED_INTERNAL (-6)

// one triangle of the synchronisation-free LU solve (CSR without the diagonal)
struct SfTri {
  const int32_t* ptr;
  const int32_t* col;
  const c64* val;
  const c64* dinv;
  int* flag;  // per row: the epoch of the solve that last finished the row
  const c64* sval = nullptr;  // U: each row's entries times the row's inverse diagonal
};
constexpr int SF_TPB = 128;

// The operands of the node sums t = sum_e A(e, node) V1[e] + jw sum_s V2[s] + (Yle Phi)[node]
// (sparse.cu, branch_rows), which the group solves form for their own rows
struct NodeSums {
  const c64 *V1 = nullptr, *V2 = nullptr, *Phi = nullptr;
  const int32_t *yle_ptr = nullptr, *yle_col = nullptr;  // (the groups know their rows of Yle)
  const c64* yle_val = nullptr;
  const double* w = nullptr;
};

// Groups of the LU solves (sparse.cu, k_sptrsv_grp). The rows of L and U fall into
// connected components (rows linked by a factor entry) that never depend on one another.
// Components of at most SF_PACK_COMP rows and SF_PACK_E / 2 entries are packed, in order of
// their depth, into groups of up to SF_PACK_R rows; larger ones (up to SF_COMP_MAX rows)
// form a group each. One CTA solves a group: it loads all of the group's rows, entries and
// right-hand sides into shared memory, then runs the group's L levels and U levels there.
constexpr int SF_COMP_MAX = 512;
constexpr int SF_PACK_COMP = 64;  // rows of a component that may be packed with others
constexpr int SF_PACK_R = 256;    // rows of a packed group
constexpr int SF_PACK_E = 1024;   // its entries (L and U off-diagonal)
constexpr int SF_GRP_TPB = 128;   // one warp per SM sub-partition, each with its FP64 pipe
struct alignas(16) GrpRow {
  int32_t r;           // factor row
  int32_t j;           // original row of its right-hand side (Pr)
  int32_t o;           // where its result goes: the original column (Pc), or r (GrpPlan::direct)
  int16_t g0, g1, g2, g3;  // node j's sum in the group's gather list: edges with A = -1
                           // [g0, g1), with A = +1 [g1, g2), surfaces [g2, g3)
  int32_t y0, y1;      // its row of Yle
  int32_t pad;
};
struct alignas(16) GrpHead {
  int32_t q0, nr;            // its rows
  int32_t r0, nrec, nrl;     // its update passes, the first nrl of them L's
  int32_t e0, ne, nl;        // its entries, the first nl of them L's
  int32_t t0, nt;            // its gather list
  int32_t pad0, pad1;
};
struct GrpPlan {
  const GrpHead* head = nullptr;  // per group
  const GrpRow* rows = nullptr;   // the groups' rows
  const int32_t* rec = nullptr;   // update passes of the L levels, then of the U levels: the
                                  // number of entries, < 0 (~number) when a barrier follows
                                  // (the level's last pass)
  const int32_t* esrc = nullptr;  // per entry, in pass order: its index in L's values, or
                                  // ~index in U's
  const int32_t* eij = nullptr;   // its row (low 16 bits) and column as positions in the group
  const int32_t* gsrc = nullptr;  // gather lists: edge, or ~surface
  int nbig = 0, ngroups = 0;      // groups [0, nbig) hold one large component each
  // the large groups' largest row, entry, pass and gather counts, and the packed groups'
  int rb = 0, eb = 0, kb = 0, gb = 0;
  int rp = 0, ep = 0, kp = 0, gp = 0;
  bool direct = false;            // results go through Pc already (no global-scheme rows)
  bool sums = false;              // the groups can form their nodes' sums
  bool unit_l = false;            // L's diagonal is one
};
constexpr size_t SF_ONE_LAUNCH_SMEM = 56 * 1024;  // four resident CTAs per SM
constexpr int SF_GATHER_MAX = 2048;  // a group's gather list, above which node sums run apart
// shared memory of a group of R rows, E entries, K passes and G gathered values: the vector,
// 1/U(i,i) and the node sums' ranges, the entries' values and positions, the passes, the node
// sums' terms
__host__ __device__ inline size_t grp_smem(int R, int E, int K, int G) {
  return (48 * (size_t)R + 20 * (size_t)E + 4 * (size_t)K + 16 * (size_t)G + 15) & ~(size_t)15;
}

// Device refactorisation of SS in a fixed pattern (refactor.cu): slots are the off-diagonal
// entries of L, then the diagonal of U (D), then the off-diagonal entries of U
struct RefactorPlan {
  int64_t n = 0, nL = 0, nU = 0;
  int64_t* asm_ptr = nullptr;    // per slot, its contributions in asm_src
  uint32_t* asm_src = nullptr;   // contribution codes (type << 30 | index)
  int32_t* rows = nullptr;       // rows grouped by L level
  std::vector<int> lvl_off;      // level offsets into rows (host)
  std::vector<int> lvl_cap;      // most entries (L, diagonal, U) of a level's rows (host)
  int32_t* upd_off = nullptr;    // per L entry (p, k): its targets in upd_tgt
  int32_t* upd_tgt = nullptr;    // per entry of U(k,:): its slot in row p
  c64* D = nullptr;              // diagonal of U
};
int refactor_launch(const RefactorPlan& R, const SfTri& L, const SfTri& U, c64* Lval, c64* Uval,
                    const c64* invZ, const double* invP, const c64* yle, double w, int* err,
                    cudaStream_t st);

// Device-resident state of one Householder GMRES cycle (the Arnoldi loop's scalar work
// runs in gm_step, krylov.cu). The host writes the header before a run of iterations
// and reads back the header, res and wv after it; Utop and R only when its convergence
// check needs them. All arrays live in one allocation after the header.
struct GmDev {
  int j;          // inner iterations done in this cycle (the next one's 0-based index)
  int inner;      // iterations per cycle
  int n;          // system size (the reference's initer != n tests)
  int headlen;    // min(N, inner + 1): rows of the reflectors kept in Utop
  int ld;         // inner + 1, leading dimension of Utop
  int exit_now;   // host: leave the loop after the next iteration
  unsigned tick[32];  // CTAs done of each group of a reduction, and groups done (zero between)
  double tolb;    // tol * |b|: the loop continues while |w(j+1)| > tolb
  double normr;   // |w(j+1)| after the last iteration
  double* res;    // [inner + 2] residual estimates, res[initer] = |w(initer)|
  c64* wv;        // [inner + 1] Givens-rotated right-hand side w
  c64* J;         // [2 * inner] Givens rotations (c, s) per column
  c64* Utop;      // [ld * ld] leading rows of the reflectors, column-major
  c64* R;         // [inner * inner] upper-triangular R, column-major, ld = inner
  c64* cvec;      // [ld] coefficients of the next iteration's v: T conj(Utop(j, :))
  c64* cpart;     // [ld] their part from the columns before the newest
  c64* head;      // [ld] leading rows of the orthogonalised vector
  c64* scr;       // [4 * ld + 4] scratch of the reductions' last CTAs
};

// Buffers of the device loop's Arnoldi body (krylov.cu): the basis is U (complex double)
// or U32 (complex float-float), whichever is set; T the compact-WY factor (ld ldT); v the
// iteration's vector (not normalised, *scal its inverse norm), w = A v; kmax the largest column
// count of the cycle (inner).
struct GmBody {
  c64* U = nullptr;
  cff* U32 = nullptr;
  size_t N = 0;
  c64* T = nullptr;
  int ldT = 0, kmax = 0;
  GmDev* gs = nullptr;
  c64 *v = nullptr, *w = nullptr, *coef = nullptr;
  double *part = nullptr, *scal = nullptr;  // partial sums: gm_part_doubles(N, kmax + 1)
  cudaGraphConditionalHandle cond = 0;
  int use_cond = 0;  // 1 inside the WHILE node's body graph, 0 for a single eager iteration
  cudaStream_t st = nullptr;
};
size_t gm_part_doubles(size_t N, int k);
int gm_pre(const GmBody& B);   // returns the kernels launched
int gm_post(const GmBody& B);

// cudaMalloc, and stream-ordered scratch from a context's pool (nullptr: the device's default
// pool, which gives its memory back at every synchronisation and maps it again at the next
// allocation). A refusal for lack of memory leaves nothing for later error checks to find.
cudaError_t dev_alloc(void** p, size_t bytes);
cudaError_t scratch_alloc(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t st);

#define CTX_CHECK(expr)      \
  do {                       \
    int _r = (expr);         \
    if (_r) return _r;       \
  } while (0)

// A lattice family: one face family of the P tensor (reference families 12, 34, 56)
// or one edge direction of the Lp tensor. Its lattice is both the input and the
// output lattice of its circulant blocks.
struct Family {
  bool active = false;
  bool lp = false;       // edge family (compact vector I, output LpI) vs face family (Q, PQ)
  int dims[3] = {0, 0, 0};  // lattice extents, x fastest
  int L[3] = {1, 1, 1}, logL[3] = {0, 0, 0};  // circulant grid
  int32_t* map = nullptr;   // lattice cell -> compact index or -1
  void* T[2] = {nullptr, nullptr};  // work buffer per precision: [z < dims[2]][y < Ly][kx < Lx]
};

// A block spectrum, scaled by 1/(Lx*Ly*Lz). Along each axis the kernel is even (c = 0) or even
// about a half-sample shift (c = +-1), so S(k) = R(|k_x|, |k_y|, |k_z|) *
// prod_a exp(-i*pi*c_a*k_a/L_a) with k_a in (-L_a/2, L_a/2] and R real. Kept y/z-folded: R at
// the folded y and z frequencies but at every x position, layout (fy, fz, px), px the DIF
// position, so that consecutive columns of a z pass read contiguous values;
// Lx(Ly/2+1)(Lz/2+1) values in FP64 (FP64 and float-float passes) and FP32 (FP32 passes), a
// quarter of the positions. Cross blocks take their phases from the phase tables.
struct Spectrum {
  int L[3] = {1, 1, 1};
  int c[3] = {0, 0, 0};
  void* yz[2] = {nullptr, nullptr};  // [0] fp64, [1] fp32
};

// Launchers (fftconv.cu). prec: 0 = fp64, 1 = fp32, 2 = float-float; tw[prec] the master
// twiddle table of that arithmetic. x (input) / LpI / PQ are complex double; families
// 0..2 are the face families, 3..5 the edge families; spectra 0..5 = P blocks
// (00, 11, 22, 01, 02, 12), 6..8 = Lp blocks of families 3..5.
// FP32 z-pass forms, chosen per grid by measurement (tune_zpass in ctx.cu). Face / edge
// form 0 (and 1, kept as a name): register-direct kernels; 2: staged kernels (persistent CTAs,
// bulk-copied tiles; the edge families in one launch); 3: pair kernels (half-length transforms
// of the even and odd frequencies). edge_plan: the edge families' z radix plan of forms 0 to 2
// (0: make_plan(n, 4, 4, 4), 1: make_plan(n, 4, 4, 3); 8 x 16 and 16 x 8 at Lz = 128).
struct ZTune {
  int* err = nullptr;  // error word set by a staged kernel whose copy wait ran into its limit
  int nsm = 0;         // SM count of the device
  int face = 0, edge = 0, edge_plan = 0;
};
// ev (nullable): 6 events around the five pass classes. ph: the face grid's phase tables,
// FP64 (x, y, z) then FP32 (x, y, z). zt (nullable: form 0): the FP32 z-pass choice.
int conv_all(const Family* F, int nfam, const Spectrum* spec, const void* const* ph,
             const c64* x, c64* LpI, c64* PQ, int64_t m, int prec, const void* const* tw,
             int twmax, cudaStream_t st, cudaEvent_t* ev, const ZTune* zt);
// one FP32 z pass alone, in the forms of zt (which 0: the face families, 1: the edge
// families), on the current family buffers; the tuner times it
int zpass_f32(const Family* F, int nfam, const Spectrum* spec, const void* const* ph,
              const void* tw, int twmax, const ZTune& zt, int which, cudaStream_t st);
// phase tables exp(-i*pi*k/L) per DIF position of the three face-grid axes, complex FP64
// (e64) and FP32 (e32)
int phase_tables(const int L[3], void* e64[3], void* e32[3], cudaStream_t st);
// whether the face / edge families' FP32 z passes can take forms 1 and 2 (whole 16-column
// tiles, enough z points; the edge families on one shared grid)
bool zpass_yz_faces(const Family* F, int nfam);
bool zpass_yz_edges(const Family* F, int nfam);
// lines along axis ax (x, y) the pair passes take: a circulant of 2 to 512 points
inline bool line_pair_ok(const Family& f, int ax) {
  return f.active && f.L[ax] >= 2 && f.L[ax] <= 512 && f.dims[ax] <= f.L[ax] / 2 + 1 &&
         ((int64_t)f.dims[2] << f.logL[0]) < ((int64_t)1 << 30) &&
         (int64_t)f.dims[1] * f.dims[2] < ((int64_t)1 << 30);
}
// launches of the x (ax 0) or y passes' one direction in a precision
int line_launches(const Family* F, int nfam, int prec, int ax);
// launches of the edge families' z passes in a precision (0 fp64, 1 fp32, 2 float-float)
int zedge_launches(const Family* F, int nfam, int prec, const ZTune& zt);
// z extents the pair passes take: a circulant of 2 to 128 points (half of it in registers)
inline bool zpair_ok(const Family& f) {
  return f.active && f.L[2] >= 2 && f.L[2] <= 128 && f.dims[2] <= f.L[2] / 2 + 1 &&
         (int64_t)f.L[0] * f.L[1] < ((int64_t)1 << 30);
}
// A spectrum to build from a generating row on the device: the row's extents, the output and
// input family extents, stride and offset per axis (K(e) = row[|sdim e + odim|])
struct SpecJob {
  Spectrum* S;
  const double* row;
  const int *M, *na, *nb, *sdim, *odim;
  int symmetric;
};
int spectra_build(const SpecJob* jobs, int njobs, const void* tw64, int twmax, cudaMemPool_t pool,
                  cudaStream_t st);

}  // namespace peec
