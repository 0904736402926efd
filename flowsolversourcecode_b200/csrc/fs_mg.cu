// fs_mg.cu -- element-agglomeration multigrid on the GPU.
//
// Hierarchy (host, once per context): AgglomorateLevelGeometricallyElement
// (AlgebraicMultiGrid/AgglomorateALevelGeometricallyElementBased.for:4-318)
// restated in C++ -- greedy seeds in cell order, immediate neighbours, then
// neighbours of neighbours, capped at 8/4/3/2 children by level, orphans
// joined with and then without the cap -- and the coarse connectivity in the
// reference's discovery order.  Coarsening stops as in Agglomorate
// (AgglomorateGrid.for:36-72).  The parent maps depend on connectivity only.
//
// Per solve: coarse matrices (AssembleElementBasedAgglomoratedLHS.for:45-150) in
// the reference's summation order (seed, then children, each with its slots),
// so they are bit-identical to the CPU restatement: entry by entry from static
// lists in the layout of the one-phase V-cycle (k_mg_coarse), by a per-parent
// gather in mesh order for 'amg' and the general V-cycle (k_mg_lhs).
//
// Cycles run inside ONE persistent cooperative kernel.  Levels with more than
// FS_MG_SMALL rows are processed by the whole grid (grid barriers between
// colours of the Gauss-Seidel sweeps); smaller levels by CTA 0 alone with
// block barriers, so the coarse tail of a cycle costs no grid barriers.  A
// phase of a latency-bound sweep costs about one dependent-load chain per row a
// thread handles, so CTA 0 wins below ~8 rows per thread (2048 rows).
//   k_mg_solve      : AlgebraicMultigrid (AlgebraicMultiGridMainRoutine.for:330-345)
//                     with V/F/W cycles (MultiGridCycle.for), smoothing sweeps
//                     that stop on sum|r| <= rrF*IResiduals (SolveEquationsWithMultiGrid.for),
//                     multicolour symmetric Gauss-Seidel in place of the
//                     sequential sweep, coarse corrections kept between cycles
//                     as the reference does.
//   k_amg_bicgstab  : FP64 BiCGSTAB right-preconditioned by one V-cycle with
//                     over-weighted coarse corrections -- no reference row;
//                     templated on the V-cycle precision (double, or float
//                     with FP32 copies of every level's matrix: iterative
//                     refinement) and its form: damped Jacobi in one phase per
//                     level and leg with a dense FP64 inverse of the coarsest
//                     level (MODE 1), the same with Gauss-Seidel smoothing on
//                     level 0 (MODE 2), and PCycle (MODE 0) for more than one
//                     sweep or no level small enough for the inverse.
#include "fs_internal.cuh"
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

namespace cg = cooperative_groups;

#define FS_MG_SMALL 2048
#define FS_MG_DIRECT 160   // largest coarsest level inverted densely (n^2 doubles in shared memory)
#define FS_MG_MAXLEV 16
#define FS_SUMK (FS_GUESS_MAX * (FS_GUESS_MAX + 1) / 2 + FS_GUESS_MAX + 1)   // sums of the guess fit
// preconditioner V-cycle: Jacobi weight and coarse-correction factor
// (over-correction compensates the energy of piecewise-constant prolongation)
#ifndef FS_MG_OMEGA
#define FS_MG_OMEGA 0.9
#endif
// CTAs per SM the preconditioned Krylov kernel is compiled for (register cap)
#ifndef FS_AMG_MINB
#define FS_AMG_MINB 1
#endif
#ifndef FS_MG_ALPHA
#define FS_MG_ALPHA 1.8
#endif
// level 0 (the fine matrix) may take its own weight and correction factor
#ifndef FS_MG_OMEGA0
#define FS_MG_OMEGA0 0.8
#endif
#ifndef FS_MG_ALPHA0
#define FS_MG_ALPHA0 FS_MG_ALPHA
#endif

template <class R>
struct LevelDev {
  int n, w, ncolors;
  const int32_t *ncf, *nbr, *color_ptr, *color_rows;
  const R *ac, *anb;
  R *b, *x, *r, *t;
  const int32_t *parent;        // this level -> next coarser (nullptr on the coarsest)
  const int32_t *rptr, *rlist;  // restriction into this level: finer rows per coarse row, ascending
};

// One level of the V-cycle (fs_amg_core.cuh).  Rows of levels >= 1 are numbered
// aggregate by aggregate, so the rows of coarse row P are [kp[P], kp[P+1]); row
// a of level 0 is cell cells[a].  Off-diagonals: levels >= 1 in slices of 32
// rows, slot j of row a at (a/32 * w + j) * 32 + a % 32 (unused slots: value 0
// and the row itself); level 0 slot j at j * n + a, columns in mesh order,
// unused slots -1.
template <class R>
struct VcLevel {
  int n, w;
  const int32_t *col, *cells;
  const R *val, *ac;
  const int32_t *kp;
  R *b, *x, *r;
};
template <class R>
struct VcDev {
  int lc;
  // set by each CTA of the kernel: lanes per row (log2), its aggregates and their rows
  int G[FS_MG_MAXLEV], p0[FS_MG_MAXLEV], p1[FS_MG_MAXLEV], e0[FS_MG_MAXLEV], e1[FS_MG_MAXLEV];
  VcLevel<R> L[FS_MG_MAXLEV];
  R *x1;                 // result of level 1
  const double *sinv;
  LevelDev<R> L0;        // level 0 in mesh order
  const int32_t *par0;   // level-1 row of each cell
  // Row patterns of level 0 (npat = 0: none): cell i's neighbour in slot u is
  // i + offs[8 pat[i] + u] (FS_PAT_NONE: unused slot); patL in level 0's layout
  int npat;
  const uint8_t *pat, *patL;
  const int32_t *offs;
};

template <class R>
struct AmgKArgs {
  int N, W;
  const int32_t *ncf, *cn;
  const double *ac, *anb, *bc;
  double *x, *r, *r0, *p, *v, *s, *t, *y, *z, *dphi;
  const LevelDev<R> *lev;   // with the one-phase V-cycle level 0 alone
  const VcDev<R> *vc;
  int lc, direct, pre, post, maxit;
  const double *sinv;
  double tol;
  double *part;
  int32_t *iters;
  double *diag;
  const double *xs[FS_GUESS_MAX];   // initial-guess basis: previous p' solutions, the network's guess
  int nx;             // vectors in xs (0: zero start)
  int32_t *fit;       // [0]: k_guess_fit found a guess (device)
  int32_t *nncnt;     // [fallbacks, uses] of the initial guess, or nullptr
  unsigned *gridbar;  // grid barrier counts: the solve's, then (FS_GRIDBAR_FIT) the guess fit's; zero at launch
  unsigned *teambar;  // team barrier words of PCycle (zeroed before the launch)
  int32_t *status;    // [0] set when a bounded wait gave up (grid or team barrier)
  int team_extra;     // fs_test_wait_timeout
  long spin_limit;    // polls of a grid barrier before it gives up
};

// sums of a level's matrix entries that make up the next level's: entry q from
// idx[ptr[q] .. ptr[q+1]), c >= 0 entry c of val, c < 0 row -1-c of ac
struct CoarseSums {
  int32_t *ptr = nullptr, *idx = nullptr;
};

struct fs_mg_dev {
  // hierarchy (host)
  int nlev = 0;
  int n[FS_MG_MAXLEV] = {}, w[FS_MG_MAXLEV] = {}, ncol[FS_MG_MAXLEV] = {};
  std::vector<int32_t> h_parent[FS_MG_MAXLEV];
  std::vector<int32_t> h_nnb[FS_MG_MAXLEV], h_nbr[FS_MG_MAXLEV], h_cptr[FS_MG_MAXLEV], h_clist[FS_MG_MAXLEV];
  int lc = 0;                           // coarsest level of the preconditioner
  bool direct = false;                  // lev[lc] inverted densely
  int per_sm = 0;                       // co-resident CTAs per SM of the multigrid kernels
  std::vector<void *> allocs;           // device memory of the parts built so far
  // Mesh order (mg_mesh_build, mg_mesh_vectors): connectivity, matrices and, per
  // precision, vectors and the FP32 matrices -- for 'amg', the general V-cycle and
  // fs_mg_coarse_matrix
  bool mesh_ready = false, mesh_vec[2] = {false, false};
  int32_t *nnb[FS_MG_MAXLEV] = {}, *nbr[FS_MG_MAXLEV] = {}, *parent[FS_MG_MAXLEV] = {};
  int32_t *cptr[FS_MG_MAXLEV] = {}, *clist[FS_MG_MAXLEV] = {}, *cmap[FS_MG_MAXLEV] = {};
  int32_t *rptr[FS_MG_MAXLEV] = {}, *rlist[FS_MG_MAXLEV] = {};
  int32_t *colors[FS_MG_MAXLEV] = {};   // rows by colour, then ncol+1 offsets
  double *ac[FS_MG_MAXLEV] = {}, *anb[FS_MG_MAXLEV] = {}, *b[FS_MG_MAXLEV] = {}, *x[FS_MG_MAXLEV] = {}, *r[FS_MG_MAXLEV] = {};
  double *t[FS_MG_MAXLEV] = {};
  float *acf[FS_MG_MAXLEV] = {}, *anbf[FS_MG_MAXLEV] = {}, *bf[FS_MG_MAXLEV] = {}, *xf[FS_MG_MAXLEV] = {}, *rf[FS_MG_MAXLEV] = {};
  float *tf[FS_MG_MAXLEV] = {};
  double *sinv = nullptr;
  LevelDev<double> *lev64 = nullptr;
  LevelDev<float> *lev32 = nullptr;
  double *red = nullptr;                // partial sums
  unsigned *gridbar = nullptr;
  // The one-phase V-cycle's layout (mg_vc_build): maps and index arrays, then
  // matrices and vectors per precision
  bool vc_map = false, vc_ready[2] = {false, false};
  int32_t *vcol[FS_MG_MAXLEV] = {}, *vkp[FS_MG_MAXLEV] = {}, *cells = nullptr, *par0 = nullptr;
  int vnpos[FS_MG_MAXLEV] = {};
  CoarseSums csum[FS_MG_MAXLEV], cdiag[FS_MG_MAXLEV];   // level l's entries and diagonals from level l-1
  // FP64 matrices (the source of the next level's in either precision; level 0's in the FP32 cycle: scratch), FP32 copies
  double *vval[FS_MG_MAXLEV] = {}, *vac[FS_MG_MAXLEV] = {}, *val0[2] = {}, *ac0[2] = {};
  float *vvalf[FS_MG_MAXLEV] = {}, *vacf[FS_MG_MAXLEV] = {}, *acm = nullptr, *anbm = nullptr;   // acm, anbm: level 0 in mesh order
  int npat = 0;                                      // row patterns of level 0
  uint8_t *pat = nullptr, *patL = nullptr;
  int32_t *offs = nullptr;
  unsigned *vbar[2] = {nullptr, nullptr};            // barrier counts, partial sums and coarsest inverse
  double *vpart[2] = {nullptr, nullptr}, *vinv[2] = {nullptr, nullptr};
  VcDev<double> *vc64 = nullptr;
  VcDev<float> *vc32 = nullptr;
  // preconditioner reuse (pc_refresh): the system, precision and layout (the
  // V-cycle's, else mesh order) the coarse levels and the dense inverse were
  // last built for, and the solves since
  int built_nf = 0, age = 0;
  bool built_f32 = false, built_vc = false;
  // the Krylov launch a deferred solve prepared (pc_defer): its arguments and
  // form (fs_pc_batch_form), for fs_pc_batch_launch
  AmgKArgs<double> pend64{};
  AmgKArgs<float> pend32{};
  int pend_form = -1;
};

namespace {

// ---------------------------------------------------------------- device helpers
__device__ __forceinline__ double wsum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// block sum broadcast to the whole block
__device__ double bsum(double v) {
  __shared__ double sh[33];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = wsum(v);
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    double r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.;
    r = wsum(r);
    if (lane == 0) sh[32] = r;
  }
  __syncthreads();
  double r = sh[32];
  __syncthreads();
  return r;
}


// V-cycle work split (PCycle): levels up to FS_PC_SMALL rows on CTA 0 alone,
// up to FS_PC_TEAM_MAX rows on a team of the first FS_PC_TEAM CTAs with a
// bounded barrier of its own, larger ones on every CTA
#ifndef FS_PC_TEAM
#define FS_PC_TEAM 32
#endif
#define FS_PC_SMALL 256
#ifndef FS_PC_TEAM_MAX
#define FS_PC_TEAM_MAX 4096   // levels up to this many rows run on the CTA team
#endif
// Polls of a barrier before it reports a timeout (0.7 s on B200).  Where one CTA
// or a team works through small levels while the others wait, the sweeps it
// makes are the user's to choose (mg_pre, mg_post): the grid barrier's limit
// grows by FS_PHASE_POLLS (0.2 ms) per phase of that work, each of which takes
// microseconds.
#define FS_PC_SPIN_LIMIT (1L << 20)
#define FS_PHASE_POLLS 256L
#define FS_VC_SLOTS 6          // slots of level 0 that the row patterns give; the others come from the index table
#define FS_VC_ROWS 2048        // residuals of a down leg that a CTA keeps in shared memory
// Level 0's neighbours as a pattern per row: on meshes numbered in rows and
// planes the offsets of a cell's neighbours take few combinations (27 on a
// box), and a byte per row replaces an index per slot -- 24 of 104 bytes of a
// row's product, and six registers of the loads kept a row ahead.  Used when
// every row has at most 8 slots and the mesh at most this many combinations
// (their table sits in shared memory, 32 bytes each); other meshes read the
// index table.  p' kernel, B200, table against patterns: 128^3 54.7 and 45.6 ms
// for 92 iterations, 295k cells 21.5 and 19.1 for 130, 857k cells FP32 23.4 and
// 21.1 for 98, 124k cells 13.8 and 12.9 for 124.
#define FS_PAT_MAX 64
#define FS_PAT_NONE ((int32_t)0x80000000)
#define FS_GRIDBAR_FIT 32     // word of the guess fit's barrier count (another cache line)
#define FS_GRIDBAR_WORDS 64

// the same Krylov/V-cycle code for one system on the whole grid (g1) and for
// groups of CTAs that each solve their own system (gb)
namespace g1 {
#define FS_GROUPS 0
#include "fs_amg_core.cuh"
#undef FS_GROUPS
}  // namespace g1
namespace gb {
#define FS_GROUPS 1
#include "fs_amg_core.cuh"
#undef FS_GROUPS
}  // namespace gb
using namespace g1;

template <class R>
__device__ __forceinline__ Scope scope_of(const LevelDev<R> &L) { Scope s; s.grid = L.n > FS_MG_SMALL; return s; }

__device__ __forceinline__ void scope_sync(Sync &S, const Scope &sc) {
  if (sc.grid) S.all(); else __syncthreads();
}

// sum over a level: grid-wide or CTA 0
__device__ double scope_sum(Sync &S, const Scope &sc, double v) {
  if (sc.grid) { double o, d; S.sum2(v, 0., o, d); return o; }
  return bsum(v);
}

// one symmetric multicolour Gauss-Seidel sweep (SORMultiGrid.for:20-66)
template <class R>
// `last`: colour of the previous pass over x; a pass repeating it (the
// backward pass's first colour, the next sweep's first) would rewrite the same
// values -- rows of one colour read only other colours -- and is skipped
__device__ void gs_sweep(Sync &S, const Scope &sc, const LevelDev<R> L, const R *b, R *x, int &last) {
  const int n = L.n;
  for (int pass = 0; pass < 2; pass++)
    for (int cc = 0; cc < L.ncolors; cc++) {
      int c = pass == 0 ? cc : L.ncolors - 1 - cc;
      if (c == last) continue;
      last = c;
      int r0 = L.color_ptr[c], r1 = L.color_ptr[c + 1];
      for (long q = r0 + sc.tid0(); q < r1; q += sc.nth()) {
        int i = L.color_rows[q];
        R l = ell_acc<8, true>(b[i], n, L.w, L.nbr, L.anb, i, [&](int k) { return x[k]; });
        x[i] = l / L.ac[i];
      }
      scope_sync(S, sc);
    }
}

// r = b - A x on a level; returns sum |r| (CalculateResidualsMG + CheckConvergenceMG)
template <class R>
__device__ double residual(Sync &S, const Scope &sc, const LevelDev<R> L, const R *b, const R *x, R *r) {
  const int n = L.n;
  double s = 0.;
  for (long i = sc.tid0(); i < n; i += sc.nth()) {
    R t = ell_acc<8, true>(b[i] - L.ac[i] * x[i], n, L.w, L.nbr, L.anb, i, [&](int k) { return x[k]; });
    r[i] = t;
    s += fabs((double)t);
  }
  return scope_sum(S, sc, s);
}

// SolveEquationMG: sweeps until sum|r| <= rrF*IRes or itmax (checked=true), or
// exactly itmax sweeps (checked=false)
template <class R>
__device__ void smooth(Sync &S, const Scope &sc, const LevelDev<R> &L, const R *b, R *x, R *r,
                       double rrf, double ires, int itmax, bool checked) {
  double fres = ires;
  int iter = 0, last = -1;
  while ((!checked || fres > rrf * ires) && iter < itmax) {
    gs_sweep(S, sc, L, b, x, last);
    if (checked) fres = residual(S, sc, L, b, x, r);
    iter++;
  }
}

// b_{l+1}[P] = sum of r_l over P's fine rows in ascending order (AssembleAgglomeratedRHS)
template <class R>
__device__ void restrict_rhs(const Scope &sc, const LevelDev<R> &Lc, const R *r_f) {
  for (long P = sc.tid0(); P < Lc.n; P += sc.nth()) {
    R s = 0.;
    for (int q = Lc.rptr[P]; q < Lc.rptr[P + 1]; q++) s = s + r_f[Lc.rlist[q]];
    Lc.b[P] = s;
  }
}

// x_l[i] += x_{l+1}[parent[i]] (CorrectFinerLevelSolution)
template <class R>
__device__ void prolong(const Scope &sc, const LevelDev<R> &Lf, R *x_f, const R *x_c) {
  for (long i = sc.tid0(); i < Lf.n; i += sc.nth()) x_f[i] = x_f[i] + x_c[Lf.parent[i]];
}

// a V/F/W cycle; level 0 uses (b0, x0, r0), coarser levels their own arrays.
// Every CTA walks the same sequence of operations; an operation on a small
// level is done by CTA 0 while the others skip to the next grid barrier.
template <class R>
struct Cycle {
  Sync &S;
  const LevelDev<R> *lev;
  int nlev;
  const R *b0; R *x0; R *r0;
  double rrf, ires;
  int pre, post;
  bool checked;
  bool last_grid;   // scope of the previous operation
  __device__ const R *B(int l) const { return l == 0 ? b0 : lev[l].b; }
  __device__ R *X(int l) const { return l == 0 ? x0 : lev[l].x; }
  __device__ R *Rr(int l) const { return l == 0 ? r0 : lev[l].r; }
  __device__ void enter(const Scope &sc) {
    // a grid barrier whenever the whole grid is involved on either side,
    // else a block barrier (CTA 0 works alone on small levels)
    if (sc.grid || last_grid) S.all(); else __syncthreads();
    last_grid = sc.grid;
  }
  __device__ void op_smooth(int l, int itmax) {
    Scope sc = scope_of(lev[l]);
    enter(sc);
    if (sc.active()) smooth(S, sc, lev[l], B(l), X(l), Rr(l), rrf, ires, itmax, checked);
  }
  __device__ void op_residual(int l) {
    Scope sc = scope_of(lev[l]);
    enter(sc);
    if (sc.active()) residual(S, sc, lev[l], B(l), X(l), Rr(l));
  }
  __device__ void op_restrict(int l) {   // Restrict(l): smooth, residual, coarse rhs
    op_smooth(l, pre);
    op_residual(l);
    Scope sc = scope_of(lev[l + 1]);
    Scope sf = scope_of(lev[l]);
    Scope su; su.grid = sc.grid || sf.grid;
    enter(su);
    if (su.active()) restrict_rhs(su, lev[l + 1], Rr(l));
  }
  __device__ void op_prolong(int lc) {   // Prolongate(lc): correct level lc-1, smooth it
    int l = lc - 1;
    Scope sf = scope_of(lev[l]);
    enter(sf);
    if (sf.active()) prolong(sf, lev[l], X(l), X(lc));
    op_smooth(l, post);
  }
  __device__ void run(int type) {
    int L = nlev - 1;
    for (int l = 0; l < L; l++) op_restrict(l);
    op_smooth(L, post);
    op_residual(L);
    if (type != 0) {
      for (int l1 = L - 1; l1 >= 1; l1--) {
        for (int l = L; l >= l1 + 1; l--) op_prolong(l);
        for (int l = l1; l < L; l++) op_restrict(l);
        op_smooth(L, post);
        op_residual(L);
      }
      if (type == 2)
        for (int l1 = 2; l1 <= L - 1; l1++) {
          for (int l = L; l >= l1 + 1; l--) op_prolong(l);
          for (int l = l1; l < L; l++) op_restrict(l);
          op_smooth(L, post);
          op_residual(L);
        }
    }
    for (int l = L; l >= 1; l--) op_prolong(l);
    Scope g; g.grid = true;
    enter(g);     // final barrier: level-0 x complete
  }
};

struct MgSolveArgs {
  const LevelDev<double> *lev;
  int nlev, type, pre, post, maxcycles;
  const double *b0; double *x0; double *r0;
  double rrf; const double *ires;
  double *part;
  int32_t *iters;
  unsigned *gridbar;
  int32_t *status;
  long spin_limit;
};

// AlgebraicMultigrid cycle loop (AlgebraicMultiGridMainRoutine.for:330-345)
__global__ void __launch_bounds__(FS_COOP_BLOCK) k_mg_solve(MgSolveArgs a) {
  Sync S(a.part, a.gridbar, a.status, 0, a.spin_limit);
  // dphiMG = 0 on every level
  for (int l = 0; l < a.nlev; l++) {
    Scope sc; sc.grid = true;
    double *x = l == 0 ? a.x0 : a.lev[l].x;
    for (long i = sc.tid0(); i < a.lev[l].n; i += sc.nth()) x[i] = 0.;
  }
  S.all();
  double ires = *a.ires, fres = ires;
  Cycle<double> C{S, a.lev, a.nlev, a.b0, a.x0, a.r0, a.rrf, ires, a.pre, a.post, true, true};
  int ncycle = 1;
  while (ncycle <= a.maxcycles && fres > a.rrf * ires) {
    C.last_grid = true;
    C.run(a.type);
    Scope g; g.grid = true;
    fres = residual(S, g, a.lev[0], a.b0, a.x0, a.r0);
    ncycle++;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.iters = ncycle - 1;
}

// the initial guess of k_amg_bicgstab on the whole cooperative grid
// (guess_fit_body in fs_amg_core.cuh)
template <class R, int NX>
__global__ void __launch_bounds__(FS_COOP_BLOCK, 1) k_guess_fit(AmgKArgs<R> a) {
  g1::guess_fit_body<R, NX>(a);
}

// right-preconditioned BiCGSTAB with the V-cycle on the whole cooperative grid
// (amg_bicgstab_body in fs_amg_core.cuh)
template <class R, int MODE>
__global__ void __launch_bounds__(FS_COOP_BLOCK, FS_AMG_MINB) k_amg_bicgstab(const __grid_constant__ AmgKArgs<R> a) {
  g1::amg_bicgstab_body<R, MODE>(a);
}

// the same solve for n systems at once (the p' solves of an ensemble, one
// cooperative launch): CTAs [start[q], start[q+1]) solve system q behind their
// own bounded barrier, so systems of uneven size share the GPU instead of each
// holding all of it in turn
template <class R, int MODE>
__global__ void __launch_bounds__(FS_COOP_BLOCK, FS_AMG_MINB)
    k_amg_bicgstab_batch(const AmgKArgs<R> *__restrict__ as, const int32_t *__restrict__ start, int n) {
  gb::GridState &G = gb::gstate();
  if (threadIdx.x == 0) {
    int q = 0;
    while (q + 1 < n && (int)blockIdx.x >= start[q + 1]) q++;
    G.q = q;
    G.cta = (int)blockIdx.x - start[q];
    G.ncta = start[q + 1] - start[q];
  }
  __syncthreads();
  gb::amg_bicgstab_body<R, MODE>(as[G.q]);
}

// the initial guesses of the batched solves, in the same CTA groups (a group
// whose system has no basis vectors does nothing)
template <class R, int NX>
__global__ void __launch_bounds__(FS_COOP_BLOCK, 1)
    k_guess_fit_batch(const AmgKArgs<R> *__restrict__ as, const int32_t *__restrict__ start, int n) {
  gb::GridState &G = gb::gstate();
  if (threadIdx.x == 0) {
    int q = 0;
    while (q + 1 < n && (int)blockIdx.x >= start[q + 1]) q++;
    G.q = q;
    G.cta = (int)blockIdx.x - start[q];
    G.ncta = start[q + 1] - start[q];
  }
  __syncthreads();
  const AmgKArgs<R> a = as[G.q];
  if (a.nx == NX) gb::guess_fit_body<R, NX>(a);   // groups of other basis sizes take another launch
}

// the fit kernels by basis size (1 .. FS_GUESS_MAX): each instance keeps its
// sums in registers
template <class R>
static const void *guess_fit_kernel(int nx) {
  switch (nx) {
    case 1: return (const void *)k_guess_fit<R, 1>;
    case 2: return (const void *)k_guess_fit<R, 2>;
    case 3: return (const void *)k_guess_fit<R, 3>;
    case 4: return (const void *)k_guess_fit<R, 4>;
    case 5: return (const void *)k_guess_fit<R, 5>;
    case 6: return (const void *)k_guess_fit<R, 6>;
    case 7: return (const void *)k_guess_fit<R, 7>;
    case 8: return (const void *)k_guess_fit<R, 8>;
  }
  return nullptr;
}
template <class R>
static const void *guess_fit_batch_kernel(int nx) {
  switch (nx) {
    case 1: return (const void *)k_guess_fit_batch<R, 1>;
    case 2: return (const void *)k_guess_fit_batch<R, 2>;
    case 3: return (const void *)k_guess_fit_batch<R, 3>;
    case 4: return (const void *)k_guess_fit_batch<R, 4>;
    case 5: return (const void *)k_guess_fit_batch<R, 5>;
    case 6: return (const void *)k_guess_fit_batch<R, 6>;
    case 7: return (const void *)k_guess_fit_batch<R, 7>;
    case 8: return (const void *)k_guess_fit_batch<R, 8>;
  }
  return nullptr;
}

// coarse matrix of level lc from level lc-1 (AssembleElementBasedAgglomoratedLHS.for:45-150)
// one thread per coarse row (AssembleElementBasedAgglomoratedLHS.for:45-150):
// the children in list order, each child's diagonal then its neighbour slots in
// slot order, so every coarse entry is summed in the reference's order.  The
// coarse row's off-diagonal sums live in shared memory (wc doubles per thread,
// column-major across the block).  WF > 0 bounds the fine width: a child's
// slots are then loaded all at once (independent loads in flight) before the
// additions, instead of one dependent load chain per slot.
template <int WF>
__global__ void k_mg_lhs(int nf, const int32_t *__restrict__ ncf_f, const double *__restrict__ ac_f,
                         const double *__restrict__ anb_f, int nc, int wc, const int32_t *__restrict__ cptr,
                         const int32_t *__restrict__ clist, const int32_t *__restrict__ cmap,
                         double *__restrict__ ac_c, double *__restrict__ anb_c,
                         float *__restrict__ acf_c, float *__restrict__ anbf_c) {
  extern __shared__ double sacc[];
  int P = blockIdx.x * blockDim.x + threadIdx.x;
  const int T = blockDim.x;
  double *acc_nb = sacc + threadIdx.x;
  for (int k = 0; k < wc; k++) acc_nb[(long)k * T] = 0.;
  if (P >= nc) return;
  double acc = 0.;
  const int q0 = cptr[P], q1 = cptr[P + 1];
  for (int q = q0; q < q1; q++) {
    const int c = clist[q];
    const double a0 = ac_f[c];
    const int nn = ncf_f[c];
    if (WF > 0) {
      int t[WF > 0 ? WF : 1];
      double a[WF > 0 ? WF : 1];
#pragma unroll
      for (int j = 0; j < WF; j++) {
        t[j] = -1; a[j] = 0.;
        if (j < nn) { t[j] = cmap[(long)j * nf + c]; a[j] = anb_f[(long)j * nf + c]; }
      }
      acc = acc + a0;
#pragma unroll
      for (int j = 0; j < WF; j++) {
        if (t[j] == -2) acc = acc + a[j];
        else if (t[j] >= 0) acc_nb[(long)t[j] * T] = acc_nb[(long)t[j] * T] + a[j];
      }
    } else {
      acc = acc + a0;
      for (int j = 0; j < nn; j++) {
        const int tj = cmap[(long)j * nf + c];
        const double aj = anb_f[(long)j * nf + c];
        if (tj == -2) acc = acc + aj;
        else if (tj >= 0) acc_nb[(long)tj * T] = acc_nb[(long)tj * T] + aj;
      }
    }
  }
  ac_c[P] = acc;
  for (int k = 0; k < wc; k++) anb_c[(long)k * nc + P] = acc_nb[(long)k * T];
  if (acf_c) {   // the FP32 copy of the coarse level, when the preconditioner is FP32
    acf_c[P] = (float)acc;
    for (int k = 0; k < wc; k++) anbf_c[(long)k * nc + P] = (float)acc_nb[(long)k * T];
  }
}

__global__ void k_to_f32(long n, const double *a, float *b) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

// Dense inverse of the coarsest level (one CTA of 16 warps, n <= 32 CT): in-place
// Gauss-Jordan without pivoting, one block barrier per pivot.  Warp y holds
// rows y + 16 a, lane x columns x + 32 b in registers; the pivot row and column
// of step k, and the pivot's reciprocal, are read from buffers (by the parity
// of k) that step k-1 filled.  The update is a multiplication and a subtraction
// per entry; the pivot row, column and reciprocal are handled outside it, by the
// warp or the lanes they belong to.  Bound by FP64 rate (64 a clock and SM: 0.4
// us a pivot at n = 157) and the chain barrier - reciprocal - barrier.  With the
// matrix in shared memory, or a select or branch per entry, a pivot took 4 us at
// n = 157 (0.64 ms in all); the set-up of the 64x64 cavity's p' solve went from
// 0.67 to 0.25 ms.  Every entry goes through the same operations as an in-place
// elimination.
// The agglomerated matrices are diagonally dominant.  A pure-Neumann level
// (every row sum ~0: the pressure correction with walls only) is singular with
// the constant null space; its last equation is replaced by x_{n-1} = 0 and the
// last column of the inverse is zeroed, so sinv*b solves the remaining
// equations -- the consistent systems the V-cycle restricts.  A zero pivot
// drops its unknown.
template <int CT>
__global__ void __launch_bounds__(512, 1) k_mg_dense_inverse(int n, int w, const int32_t *nbr, const double *ac,
                                                             const double *anb, bool sliced, double *sinv) {
  constexpr int RT = 2 * CT;
  extern __shared__ double A[];
  __shared__ double prow[2][32 * CT], pcol[2][32 * CT], pinv[2];
  __shared__ int singular;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
  for (int q = tid; q < n * n; q += nt) A[q] = 0.;
  if (tid == 0) singular = 1;
  __syncthreads();
  for (int i = tid; i < n; i += nt) {
    double d = ac[i], rs = d;
    A[(long)i * n + i] = d;
    for (int j = 0; j < w; j++) {
      const long q = sliced ? ((long)(i >> 5) * w + j) * 32 + (i & 31) : (long)j * n + i;
      const int k = nbr[q];
      if (k >= 0 && k != i) { double a = anb[q]; A[(long)i * n + k] += a; rs += a; }
    }
    if (fabs(rs) > 1e-9 * fabs(d)) singular = 0;
  }
  __syncthreads();
  const bool sing = singular != 0;
  if (sing)
    for (int j = tid; j < n; j += nt) A[(long)(n - 1) * n + j] = j == n - 1 ? 1. : 0.;
  __syncthreads();
  double v[RT][CT];
#pragma unroll
  for (int a = 0; a < RT; a++)
#pragma unroll
    for (int b = 0; b < CT; b++) {
      const int i = wid + 16 * a, j = lane + 32 * b;
      v[a][b] = i < n && j > 0 && j < n ? A[(long)i * n + j] : 0.;   // column 0 is published
    }
  for (int j = tid; j < 32 * CT; j += nt) {
    prow[0][j] = j < n ? A[j] : 0.;
    pcol[0][j] = j < n ? A[(long)j * n] : 0.;
  }
  if (tid == 0) pinv[0] = A[0] != 0. ? 1. / A[0] : 0.;
  __syncthreads();
  for (int k = 0; k < n; k++) {
    const int c = k & 1, d = c ^ 1, k1 = k + 1;
    const double p = pinv[c];
    double rk[CT];
#pragma unroll
    for (int b = 0; b < CT; b++) rk[b] = lane + 32 * b == k ? p : prow[c][lane + 32 * b] * p;
    // every entry v - c rk (column k holds 0 since it was published) ...
#pragma unroll
    for (int a = 0; a < RT; a++) {
      const double ci = pcol[c][wid + 16 * a];
#pragma unroll
      for (int b = 0; b < CT; b++) v[a][b] = v[a][b] - ci * rk[b];
    }
    // ... but row k, which becomes rk; then row and column k+1 for the next step.
    // (Bit tests, not a == k / 16: the compiler would index v with k / 16, in memory.)
    if (wid == (k & 15)) {
#pragma unroll
      for (int a = 0; a < RT; a++)
        if (1u << (k >> 4) & 1u << a)
#pragma unroll
          for (int b = 0; b < CT; b++) v[a][b] = rk[b];
    }
    if (wid == (k1 & 15)) {
#pragma unroll
      for (int a = 0; a < RT; a++)
        if (1u << (k1 >> 4) & 1u << a)
#pragma unroll
          for (int b = 0; b < CT; b++) prow[d][lane + 32 * b] = v[a][b];
      if (lane == (k1 & 31) && k1 < n) {   // its own store
        const double next = prow[d][k1];
        pinv[d] = next != 0. ? 1. / next : 0.;
      }
    }
    if (lane == (k1 & 31)) {
#pragma unroll
      for (int b = 0; b < CT; b++)
        if (1u << (k1 >> 5) & 1u << b)
#pragma unroll
          for (int a = 0; a < RT; a++) {
            pcol[d][wid + 16 * a] = v[a][b];
            v[a][b] = 0.;
          }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < RT; a++)
#pragma unroll
    for (int b = 0; b < CT; b++) {
      const int i = wid + 16 * a, j = lane + 32 * b;
      if (i < n && j < n) sinv[(long)i * n + j] = sing && j == n - 1 ? 0. : v[a][b];
    }
}

// level 0 into the V-cycle's layout (row a is cell cells[a]; FP64, and FP32 when
// that is the cycle's precision, then with an FP32 copy in mesh order too).
// Unused slots are copied as they are: no one reads them.
__global__ void k_mg_level0(int n, int w, const int32_t *__restrict__ cells, const double *__restrict__ ac,
                            const double *__restrict__ anb, double *__restrict__ acL, double *__restrict__ anbL,
                            float *__restrict__ acLf, float *__restrict__ anbLf, float *__restrict__ acf,
                            float *__restrict__ anbf) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  const long i = cells[a];
  const double d = ac[i];
  acL[a] = d;
  if (acf) { acLf[a] = (float)d; acf[a] = (float)ac[a]; }
  for (int j = 0; j < w; j++) {
    const double v = anb[(long)j * n + i];
    anbL[(long)j * n + a] = v;
    if (acf) { anbLf[(long)j * n + a] = (float)v; anbf[(long)j * n + a] = (float)anb[(long)j * n + a]; }
  }
}

// the next level's matrix (AssembleElementBasedAgglomoratedLHS.for:45-150) in
// the V-cycle's layout: a thread per entry, then per diagonal, sums its static
// list -- the children in list order, each child's diagonal then its slots --
// so every entry is summed in the reference's order.  The rows of an
// aggregate are consecutive in the layout, so neighbouring threads gather from
// neighbouring lines; a thread per coarse row over the mesh-ordered matrix
// (k_mg_lhs) reads a sector per value.
__global__ void k_mg_coarse(int npos, int n, const int32_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                            const int32_t *__restrict__ dptr, const int32_t *__restrict__ didx,
                            const double *__restrict__ acF, const double *__restrict__ anbF, double *__restrict__ acC,
                            double *__restrict__ anbC, float *__restrict__ acCf, float *__restrict__ anbCf) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  const bool diag = q >= npos;
  if (diag) q -= npos;
  if (diag && q >= n) return;
  const int32_t *pp = diag ? dptr : ptr, *ii = diag ? didx : idx;
  const int c1 = pp[q + 1];
  double t = 0.;
  for (int c = pp[q]; c < c1; c += 4) {
    int e[4];
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) e[u] = c + u < c1 ? ii[c + u] : 0;
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = c + u < c1 ? (e[u] >= 0 ? anbF[e[u]] : acF[-1 - e[u]]) : 0.;
#pragma unroll
    for (int u = 0; u < 4; u++) if (c + u < c1) t = t + v[u];
  }
  if (diag) {
    acC[q] = t;
    if (acCf) acCf[q] = (float)t;
  } else {
    anbC[q] = t;
    if (anbCf) anbCf[q] = (float)t;
  }
}

}  // namespace

// ================================================================ host: hierarchy
struct HostLevel {
  int n = 0, w = 0;
  std::vector<int32_t> nnb, nbr;   // nbr[j*n+i]
};

// AgglomorateLevelGeometricallyElement restated (see file header); fills the
// coarse level and the parent map / child lists of the fine one.
static void agglomerate(const HostLevel &f, int lc, HostLevel &c, std::vector<int32_t> &parent,
                        std::vector<int32_t> &cptr, std::vector<int32_t> &clist) {
  const int n = f.n;
  const int maxc = lc == 1 ? 8 : lc == 2 ? 4 : lc == 3 ? 3 : 2;
  parent.assign(n, -1);
  std::vector<int32_t> seed;
  std::vector<std::vector<int32_t>> ch;
  for (int s = 0; s < n; s++) {
    if (parent[s] != -1) continue;
    int ip = (int)seed.size();
    parent[s] = ip;
    std::vector<int32_t> list;
    int cnt = 0;
    for (int j = 0; j < f.nnb[s]; j++) {
      int q = f.nbr[(size_t)j * n + s];
      if (q >= 0 && parent[q] == -1) {
        if (cnt >= maxc) break;
        parent[q] = ip; list.push_back(q); cnt++;
      }
    }
    int cnt2 = cnt;
    if (cnt < maxc)
      for (int k = 0; k < cnt2; k++) {
        if (cnt >= maxc) break;
        int cc = list[k];
        for (int j = 0; j < f.nnb[cc]; j++) {
          if (cnt >= maxc) break;
          int q = f.nbr[(size_t)j * n + cc];
          if (q >= 0 && parent[q] == -1) { parent[q] = ip; list.push_back(q); cnt++; }
        }
      }
    if (cnt == 0) parent[s] = -1;
    else { seed.push_back(s); ch.push_back(list); }
  }
  for (int pass = 0; pass < 2; pass++)
    for (int o = 0; o < n; o++) {
      if (parent[o] == -1) {
        bool found = false;
        for (int j = 0; j < f.nnb[o]; j++) {
          int q = f.nbr[(size_t)j * n + o];
          if (q >= 0 && parent[q] != -1 && !found) {
            found = true;
            int P = parent[q];
            if (pass == 0 && (int)ch[P].size() >= maxc) continue;
            parent[o] = P; ch[P].push_back(o);
          }
        }
      }
      if (pass == 1 && parent[o] == -1) {
        parent[o] = (int)seed.size(); seed.push_back(o); ch.emplace_back();
      }
    }
  const int nc = (int)seed.size();
  std::vector<std::vector<int32_t>> cn(nc);
  for (int e = 0; e < n; e++)
    for (int j = 0; j < f.nnb[e]; j++) {
      int q = f.nbr[(size_t)j * n + e];
      if (q < 0 || parent[e] == parent[q]) continue;
      auto &v = cn[parent[e]];
      if (std::find(v.begin(), v.end(), parent[q]) == v.end()) v.push_back(parent[q]);
    }
  int wc = 1;
  for (auto &v : cn) wc = std::max(wc, (int)v.size());
  c.n = nc; c.w = wc;
  c.nnb.assign(nc, 0);
  c.nbr.assign((size_t)wc * nc, -1);
  for (int P = 0; P < nc; P++) {
    c.nnb[P] = (int)cn[P].size();
    for (int k = 0; k < c.nnb[P]; k++) c.nbr[(size_t)k * nc + P] = cn[P][k];
  }
  cptr.assign(nc + 1, 0);
  clist.clear();
  for (int P = 0; P < nc; P++) {
    cptr[P] = (int)clist.size();
    clist.push_back(seed[P]);
    clist.insert(clist.end(), ch[P].begin(), ch[P].end());
  }
  cptr[nc] = (int)clist.size();
}

static std::vector<int32_t> color_level(const HostLevel &L, int &ncol) {
  std::vector<int> col(L.n, -1);
  ncol = 0;
  for (int i = 0; i < L.n; i++) {
    uint64_t used = 0;
    for (int j = 0; j < L.nnb[i]; j++) {
      int k = L.nbr[(size_t)j * L.n + i];
      if (k >= 0 && col[k] >= 0 && col[k] < 64) used |= 1ull << col[k];
    }
    int c = 0;
    while (c < 63 && (used & (1ull << c))) c++;
    col[i] = c;
    ncol = std::max(ncol, c + 1);
  }
  std::vector<int32_t> ptr(ncol + 1, 0), rows(L.n);
  for (int i = 0; i < L.n; i++) ptr[col[i] + 1]++;
  for (int c = 0; c < ncol; c++) ptr[c + 1] += ptr[c];
  std::vector<int32_t> pos(ptr.begin(), ptr.end() - 1);
  for (int i = 0; i < L.n; i++) rows[pos[col[i]]++] = i;
  rows.insert(rows.end(), ptr.begin(), ptr.end());
  return rows;
}

template <class T>
static int mg_alloc(fs_ctx *ctx, T **d, size_t n) {
  FS_CK(fs_alloc(ctx, (void **)d, std::max<size_t>(n, 1) * sizeof(T)));
  ctx->mg->allocs.push_back(*d);
  return FS_OK;
}
template <class T>
static int upv(fs_ctx *ctx, T **d, const std::vector<T> &h) {
  int rc = mg_alloc(ctx, d, h.size());
  if (rc) return rc;
  if (!h.empty()) FS_CK(fs_upload(ctx, *d, h.data(), h.size() * sizeof(T)));
  return FS_OK;
}

// a part of the hierarchy: what a failed build holds is given back
template <class F>
static int mg_part(fs_ctx *ctx, F &&build) {
  std::vector<void *> &a = ctx->mg->allocs;
  const size_t before = a.size();
  const int rc = build();
  if (rc) {
    cudaStreamSynchronize(ctx->st);
    while (a.size() > before) { cudaFree(a.back()); a.pop_back(); }
  }
  return rc;
}

// the hierarchy and what follows from it on the host; device memory is
// allocated by the parts that a solver uses (mg_mesh_*, mg_vc_build)
int fs_mg_build(fs_ctx *ctx) {
  if (ctx->mg) return FS_OK;
  // cooperative grid: smallest co-resident count of the kernels
  int per = INT_MAX;
  const void *kernels[] = {(const void *)k_mg_solve, (const void *)k_amg_bicgstab<double, 0>,
                           (const void *)k_amg_bicgstab<float, 0>, (const void *)k_amg_bicgstab<double, 1>,
                           (const void *)k_amg_bicgstab<float, 1>, (const void *)k_amg_bicgstab<float, 2>};
  for (const void *k : kernels) {
    int a = 0;
    FS_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k, FS_COOP_BLOCK, 0));
    per = std::min(per, a);
  }
  if (per < 1) { ctx->err = "multigrid kernels do not fit on an SM"; return FS_E_CUDA; }
  // the dense inverse's attribute belongs to the function, shared by every
  // context of the process: set it for the largest coarsest level any may have
  const int sm = (int)(sizeof(double) * FS_MG_DIRECT * FS_MG_DIRECT);
  const void *ks[] = {(const void *)k_mg_dense_inverse<1>, (const void *)k_mg_dense_inverse<2>,
                      (const void *)k_mg_dense_inverse<3>, (const void *)k_mg_dense_inverse<4>,
                      (const void *)k_mg_dense_inverse<5>};
  for (const void *k : ks) FS_CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  fs_mg_dev *M = new fs_mg_dev();
  ctx->mg = M;
  M->per_sm = per;   // occupancy limit; the grid follows the launch shape at each solve
  HostLevel f;
  f.n = ctx->N; f.w = ctx->W; f.nnb = ctx->h_ncf; f.nbr = ctx->h_cn;
  int l = 0;
  const int maxlev = std::min(ctx->cfg.mg_max_levels, FS_MG_MAXLEV);
  for (;;) {
    M->n[l] = f.n; M->w[l] = f.w;
    HostLevel c;
    const bool more = l + 1 < maxlev && f.n > 2 * ctx->cfg.mg_min_parents;
    if (more) agglomerate(f, l + 1, c, M->h_parent[l], M->h_cptr[l + 1], M->h_clist[l + 1]);
    if (l > 0) { M->h_nnb[l] = std::move(f.nnb); M->h_nbr[l] = std::move(f.nbr); }
    if (!more) break;
    f = std::move(c);
    l++;
  }
  M->nlev = l + 1;
  // preconditioner: stop at the first level small enough for the dense inverse
  M->lc = M->nlev - 1;
  for (int q = 0; q < M->nlev; q++)
    if (q > 0 && M->n[q] <= FS_MG_DIRECT) { M->lc = q; break; }
  M->direct = M->lc > 0 && M->n[M->lc] <= FS_MG_DIRECT;
  return FS_OK;
}

// neighbour counts and lists of a level (host)
static const std::vector<int32_t> &mg_nnb(const fs_ctx *ctx, int l) { return l ? ctx->mg->h_nnb[l] : ctx->h_ncf; }
static const std::vector<int32_t> &mg_nbr(const fs_ctx *ctx, int l) { return l ? ctx->mg->h_nbr[l] : ctx->h_cn; }

static int mg_mesh_tables(fs_ctx *ctx) {
  fs_mg_dev *M = ctx->mg;
  int rc;
  M->ncol[0] = ctx->ncolors;
  M->colors[0] = ctx->color_rows;   // the same greedy colouring in cell order
  M->nnb[0] = ctx->ncf; M->nbr[0] = ctx->cn;
  M->ac[0] = ctx->ac; M->anb[0] = ctx->anb;
  for (int q = 0; q < M->nlev; q++) {
    const std::vector<int32_t> &nnb = mg_nnb(ctx, q), &nbr = mg_nbr(ctx, q);
    const size_t n = M->n[q], w = M->w[q];
    if (q > 0) {
      HostLevel h;
      h.n = M->n[q]; h.w = M->w[q]; h.nnb = nnb; h.nbr = nbr;
      if ((rc = upv(ctx, &M->colors[q], color_level(h, M->ncol[q])))) return rc;
      if ((rc = upv(ctx, &M->nnb[q], nnb)) || (rc = upv(ctx, &M->nbr[q], nbr))) return rc;
      if ((rc = mg_alloc(ctx, &M->ac[q], n)) || (rc = mg_alloc(ctx, &M->anb[q], n * w))) return rc;
      FS_CK(cudaMemsetAsync(M->anb[q], 0, sizeof(double) * n * w, ctx->st));
    }
    if (q + 1 == M->nlev) break;
    const std::vector<int32_t> &par = M->h_parent[q], &cnn = M->h_nnb[q + 1], &cnb = M->h_nbr[q + 1];
    const int nc = M->n[q + 1];
    if ((rc = upv(ctx, &M->parent[q], par))) return rc;
    // LHS lists and slot map (fine slot -> coarse slot / internal / none)
    if ((rc = upv(ctx, &M->cptr[q + 1], M->h_cptr[q + 1])) || (rc = upv(ctx, &M->clist[q + 1], M->h_clist[q + 1])))
      return rc;
    std::vector<int32_t> cmap(n * w, -1);
    for (size_t i = 0; i < n; i++) {
      const int P = par[i];
      for (int j = 0; j < nnb[i]; j++) {
        const int nb = nbr[j * n + i];
        if (nb < 0) continue;
        const int Q = par[nb];
        if (Q == P) { cmap[j * n + i] = -2; continue; }
        for (int k = 0; k < cnn[P]; k++)
          if (cnb[(size_t)k * nc + P] == Q) { cmap[j * n + i] = k; break; }
      }
    }
    if ((rc = upv(ctx, &M->cmap[q + 1], cmap))) return rc;
    // restriction lists: fine rows of each coarse row in ascending order
    std::vector<int32_t> rptr(nc + 1, 0), rlist(n);
    for (size_t i = 0; i < n; i++) rptr[par[i] + 1]++;
    for (int P = 0; P < nc; P++) rptr[P + 1] += rptr[P];
    std::vector<int32_t> pos(rptr.begin(), rptr.end() - 1);
    for (size_t i = 0; i < n; i++) rlist[pos[par[i]]++] = (int32_t)i;
    if ((rc = upv(ctx, &M->rptr[q + 1], rptr)) || (rc = upv(ctx, &M->rlist[q + 1], rlist))) return rc;
  }
  if (M->direct && (rc = mg_alloc(ctx, &M->sinv, (size_t)M->n[M->lc] * M->n[M->lc]))) return rc;
  if ((rc = mg_alloc(ctx, &M->red, (6 + FS_SUMK + 9) * (size_t)FS_RED_BLOCKS))) return rc;
  return mg_alloc(ctx, &M->gridbar, FS_GRIDBAR_WORDS);
}

static int mg_mesh_tables_once(fs_ctx *ctx) {
  if (ctx->mg->mesh_ready) return FS_OK;
  int rc = mg_part(ctx, [&] { return mg_mesh_tables(ctx); });
  if (rc) return rc;
  ctx->mg->mesh_ready = true;
  return FS_OK;
}

template <class R>
static int mg_mesh_vectors(fs_ctx *ctx) {
  constexpr bool f32 = sizeof(R) == sizeof(float);
  fs_mg_dev *M = ctx->mg;
  int rc;
  std::vector<LevelDev<R>> L(M->nlev);
  for (int q = 0; q < M->nlev; q++) {
    const size_t n = M->n[q];
    LevelDev<R> d{};
    if constexpr (f32) {
      if ((rc = mg_alloc(ctx, &M->acf[q], n)) || (rc = mg_alloc(ctx, &M->anbf[q], n * M->w[q])) ||
          (rc = mg_alloc(ctx, &M->bf[q], n)) || (rc = mg_alloc(ctx, &M->xf[q], n)) || (rc = mg_alloc(ctx, &M->rf[q], n)) ||
          (rc = mg_alloc(ctx, &M->tf[q], n)))
        return rc;
      d.ac = M->acf[q]; d.anb = M->anbf[q]; d.b = M->bf[q]; d.x = M->xf[q]; d.r = M->rf[q]; d.t = M->tf[q];
    } else {
      if ((rc = mg_alloc(ctx, &M->b[q], n)) || (rc = mg_alloc(ctx, &M->x[q], n)) || (rc = mg_alloc(ctx, &M->r[q], n)) ||
          (rc = mg_alloc(ctx, &M->t[q], n)))
        return rc;
      d.ac = M->ac[q]; d.anb = M->anb[q]; d.b = M->b[q]; d.x = M->x[q]; d.r = M->r[q]; d.t = M->t[q];
    }
    d.n = M->n[q]; d.w = M->w[q]; d.ncolors = M->ncol[q]; d.ncf = M->nnb[q]; d.nbr = M->nbr[q];
    d.color_rows = M->colors[q]; d.color_ptr = M->colors[q] + M->n[q];
    d.parent = q + 1 < M->nlev ? M->parent[q] : nullptr;
    d.rptr = M->rptr[q]; d.rlist = M->rlist[q];
    L[q] = d;
  }
  LevelDev<R> *dev = nullptr;
  if ((rc = upv(ctx, &dev, L))) return rc;
  if constexpr (f32) M->lev32 = dev; else M->lev64 = dev;
  return FS_OK;
}

// the mesh-ordered levels for cycles in R
template <class R>
static int mg_mesh_build(fs_ctx *ctx) {
  int rc = mg_mesh_tables_once(ctx);
  if (rc) return rc;
  bool &ready = ctx->mg->mesh_vec[sizeof(R) == sizeof(float)];
  if (ready) return FS_OK;
  if ((rc = mg_part(ctx, [&] { return mg_mesh_vectors<R>(ctx); }))) return rc;
  ready = true;
  return FS_OK;
}

int fs_mg_free(fs_ctx *ctx) {
  fs_mg_dev *M = ctx->mg;
  if (!M) return FS_OK;
  for (void *x : M->allocs) cudaFree(x);
  delete M;
  ctx->mg = nullptr;
  return FS_OK;
}

// coarse matrices of levels 1..last for the current fine system (every call:
// the fine matrix changes), FP32 copies of levels 0..last when asked
static int mg_coarse_matrices(fs_ctx *ctx, int last, bool f32) {
  fs_mg_dev *M = ctx->mg;
  for (int q = 1; q <= last; q++) {
    // block of T threads with T * w doubles of shared accumulators (<= 48 KB)
    int T = 128;
    while (T > 32 && (size_t)T * M->w[q] * sizeof(double) > 48 * 1024) T /= 2;
    const size_t sm = (size_t)T * M->w[q] * sizeof(double);
    if (sm > 48 * 1024) { ctx->err = "coarse level too wide for the coarse-matrix kernel"; return FS_E_UNSUPPORTED; }
    const int wf = M->w[q - 1];
#define FS_LHS_ARGS M->n[q - 1], M->nnb[q - 1], M->ac[q - 1], M->anb[q - 1], M->n[q], M->w[q], M->cptr[q], \
                    M->clist[q], M->cmap[q], M->ac[q], M->anb[q], f32 ? M->acf[q] : nullptr, f32 ? M->anbf[q] : nullptr
    if (wf <= 8) k_mg_lhs<8><<<fs_grid(M->n[q], T), T, sm, ctx->st>>>(FS_LHS_ARGS);
    else if (wf <= 32) k_mg_lhs<32><<<fs_grid(M->n[q], T), T, sm, ctx->st>>>(FS_LHS_ARGS);
    else k_mg_lhs<0><<<fs_grid(M->n[q], T), T, sm, ctx->st>>>(FS_LHS_ARGS);
#undef FS_LHS_ARGS
    FS_LAUNCH_CHECK();
  }
  if (f32)
    for (int q = 0; q <= 0; q++) {   // coarse levels got their FP32 copy from k_mg_lhs
      long n = M->n[q], nw = (long)M->w[q] * M->n[q];
      k_to_f32<<<fs_grid(n), FS_BLOCK, 0, ctx->st>>>(n, M->ac[q], M->acf[q]);
      FS_LAUNCH_CHECK();
      k_to_f32<<<fs_grid(nw), FS_BLOCK, 0, ctx->st>>>(nw, M->anb[q], M->anbf[q]);
      FS_LAUNCH_CHECK();
    }
  return FS_OK;
}

// the coarsest level's dense inverse (sliced: the V-cycle's layout, whose unused
// slots hold 0 and the row itself; else slot-major, unused slots -1)
static int dense_inverse(fs_ctx *ctx, int n, int w, const int32_t *nbr, const double *ac, const double *anb, bool sliced,
                         double *sinv) {
  const size_t sm = sizeof(double) * (size_t)n * n;
  const int ct = (n + 31) / 32;
#define FS_INV(CT) k_mg_dense_inverse<CT><<<1, 512, sm, ctx->st>>>(n, w, nbr, ac, anb, sliced, sinv)
  if (ct <= 1) FS_INV(1);
  else if (ct == 2) FS_INV(2);
  else if (ct == 3) FS_INV(3);
  else if (ct == 4) FS_INV(4);
  else FS_INV(5);
#undef FS_INV
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// position of slot j of row a in level l's layout
static size_t vc_pos(int l, int n, int w, int a, int j) {
  return l == 0 ? (size_t)j * n + a : ((size_t)(a / 32) * w + j) * 32 + a % 32;
}

// the V-cycle's number of every row of levels 0..lc: aggregate by aggregate, within
// an aggregate in ascending original order; the coarsest level keeps its numbering
static std::vector<std::vector<int32_t>> vc_numbers(const fs_mg_dev *M) {
  std::vector<std::vector<int32_t>> id(M->lc + 1);
  id[M->lc].resize(M->n[M->lc]);
  for (int i = 0; i < M->n[M->lc]; i++) id[M->lc][i] = i;
  for (int l = M->lc - 1; l >= 0; l--) {
    const std::vector<int32_t> &par = M->h_parent[l], &up = id[l + 1];
    std::vector<int32_t> at(M->n[l + 1] + 1, 0);
    for (int i = 0; i < M->n[l]; i++) at[up[par[i]] + 1]++;
    for (int P = 0; P < M->n[l + 1]; P++) at[P + 1] += at[P];
    id[l].resize(M->n[l]);
    for (int i = 0; i < M->n[l]; i++) id[l][i] = at[up[par[i]]]++;
  }
  return id;
}

// the entries of level l-1 that each entry and diagonal of level l sums, in the
// reference's order (children in list order, a child's diagonal, then its slots)
static int mg_vc_sums(fs_ctx *ctx, int l, const std::vector<int32_t> &idf, const std::vector<int32_t> &idc) {
  fs_mg_dev *M = ctx->mg;
  const int n = M->n[l - 1], w = M->w[l - 1], nc = M->n[l], wc = M->w[l];
  const std::vector<int32_t> &nnb = mg_nnb(ctx, l - 1), &nbr = mg_nbr(ctx, l - 1);
  const std::vector<int32_t> &par = M->h_parent[l - 1], &cnn = M->h_nnb[l], &cnb = M->h_nbr[l];
  const std::vector<int32_t> &cptr = M->h_cptr[l], &clist = M->h_clist[l];
  const size_t np = M->vnpos[l];
  std::vector<int32_t> ptr(np + 1, 0), dptr(nc + 1, 0), slot((size_t)n * w, -1);
  // pass 1: the coarse slot of every fine slot (-2 inside the aggregate), counts
  for (int P = 0; P < nc; P++) {
    const int p = idc[P];
    for (int q = cptr[P]; q < cptr[P + 1]; q++) {
      const int c = clist[q];
      dptr[p + 1]++;
      for (int j = 0; j < nnb[c]; j++) {
        const int k = nbr[(size_t)j * n + c];
        if (k < 0) continue;
        const int Q = par[k];
        if (Q == P) { slot[(size_t)j * n + c] = -2; dptr[p + 1]++; continue; }
        for (int m = 0; m < cnn[P]; m++)
          if (cnb[(size_t)m * nc + P] == Q) { slot[(size_t)j * n + c] = m; ptr[vc_pos(l, nc, wc, p, m) + 1]++; break; }
      }
    }
  }
  for (size_t q = 0; q < np; q++) ptr[q + 1] += ptr[q];
  for (int p = 0; p < nc; p++) dptr[p + 1] += dptr[p];
  std::vector<int32_t> idx(ptr[np]), didx(dptr[nc]), at(ptr.begin(), ptr.end() - 1), dat(dptr.begin(), dptr.end() - 1);
  for (int P = 0; P < nc; P++) {
    const int p = idc[P];
    for (int q = cptr[P]; q < cptr[P + 1]; q++) {
      const int c = clist[q], a = idf[c];
      didx[dat[p]++] = -1 - a;
      for (int j = 0; j < nnb[c]; j++) {
        const int t = slot[(size_t)j * n + c];
        const int32_t e = (int32_t)vc_pos(l - 1, n, w, a, j);
        if (t == -2) didx[dat[p]++] = e;
        else if (t >= 0) idx[at[vc_pos(l, nc, wc, p, t)]++] = e;
      }
    }
  }
  int rc;
  if ((rc = upv(ctx, &M->csum[l].ptr, ptr)) || (rc = upv(ctx, &M->csum[l].idx, idx)) ||
      (rc = upv(ctx, &M->cdiag[l].ptr, dptr)) || (rc = upv(ctx, &M->cdiag[l].idx, didx)))
    return rc;
  return FS_OK;
}

// the row patterns of level 0, when there are few enough
static int mg_vc_patterns(fs_ctx *ctx, const std::vector<int32_t> &id) {
  fs_mg_dev *M = ctx->mg;
  M->npat = 0;
  const int n = ctx->N, w = ctx->W;
  if (w > 8) return FS_OK;
  const std::vector<int32_t> &cn = ctx->h_cn;
  std::vector<int32_t> offs;
  std::vector<uint8_t> pat(n), patL(n);
  int last = 0, np = 0;
  for (int i = 0; i < n; i++) {
    int32_t o[8];
    for (int u = 0; u < 8; u++) {
      const int k = u < w ? cn[(size_t)u * n + i] : -1;
      o[u] = k >= 0 ? k - i : FS_PAT_NONE;
    }
    auto same = [&](int p) { return std::memcmp(o, offs.data() + (size_t)8 * p, sizeof(o)) == 0; };
    int p = last;
    if (np == 0 || !same(last))
      for (p = 0; p < np && !same(p); p++) {}
    if (p == np) {
      if (np == FS_PAT_MAX) return FS_OK;
      offs.insert(offs.end(), o, o + 8);
      np++;
    }
    pat[i] = (uint8_t)p;
    last = p;
  }
  for (int i = 0; i < n; i++) patL[id[i]] = pat[i];
  int rc;
  if ((rc = upv(ctx, &M->pat, pat)) || (rc = upv(ctx, &M->patL, patL)) || (rc = upv(ctx, &M->offs, offs))) return rc;
  M->npat = np;
  return FS_OK;
}

// ---------------------------------------------------------------- V-cycle layout
// Once per context: levels 1 .. lc-1 renumbered aggregate by aggregate (the
// coarsest keeps its numbering, so its dense inverse is used as it is; within
// an aggregate rows stay in ascending original order, which keeps every sum's
// order), their sliced layout, and for the
// precision asked for the arrays and the descriptor.

// first row of each of level l+1's aggregates among level l's rows
static std::vector<int32_t> vc_first(const fs_mg_dev *M, int l, const std::vector<std::vector<int32_t>> &ids) {
  std::vector<int32_t> kp(M->n[l + 1] + 1, 0);
  for (int i = 0; i < M->n[l]; i++) kp[ids[l + 1][M->h_parent[l][i]] + 1]++;
  for (int P = 0; P < M->n[l + 1]; P++) kp[P + 1] += kp[P];
  return kp;
}

// column indices of level l in the layout (unused slots: level 0 -1, else the row itself)
static std::vector<int32_t> vc_columns(const fs_ctx *ctx, int l, const std::vector<int32_t> &id) {
  const int n = ctx->mg->n[l], w = ctx->mg->w[l];
  const std::vector<int32_t> &nnb = mg_nnb(ctx, l), &nbr = mg_nbr(ctx, l);
  std::vector<int32_t> col(ctx->mg->vnpos[l]);
  if (l > 0)
    for (size_t q = 0; q < col.size(); q++) col[q] = std::min<int>((int)(q / (32 * (size_t)w) * 32 + q % 32), n - 1);
  for (int j = 0; j < w; j++)
    for (int i = 0; i < n; i++) {
      const int k = j < nnb[i] ? nbr[(size_t)j * n + i] : -1;
      if (l == 0) col[vc_pos(l, n, w, id[i], j)] = k;
      else if (k >= 0) col[vc_pos(l, n, w, id[i], j)] = id[k];
    }
  return col;
}

static int mg_vc_map(fs_ctx *ctx, const std::vector<std::vector<int32_t>> &ids) {
  fs_mg_dev *M = ctx->mg;
  const int n = M->n[0];
  int rc;
  for (int l = 0; l <= M->lc; l++)
    M->vnpos[l] = (int)((size_t)(l == 0 ? n : (M->n[l] + 31) / 32 * 32) * M->w[l]);
  std::vector<int32_t> p0(n), cells(n);
  for (int i = 0; i < n; i++) { p0[i] = ids[1][M->h_parent[0][i]]; cells[ids[0][i]] = i; }
  if ((rc = upv(ctx, &M->par0, p0)) || (rc = upv(ctx, &M->cells, cells)) ||
      (rc = upv(ctx, &M->vkp[0], vc_first(M, 0, ids))) || (rc = mg_vc_patterns(ctx, ids[0])))
    return rc;
  // level 0's columns: without patterns, or for the slots that they do not cover
  M->vcol[0] = nullptr;
  if ((M->npat == 0 || M->w[0] > FS_VC_SLOTS) && (rc = upv(ctx, &M->vcol[0], vc_columns(ctx, 0, ids[0])))) return rc;
  for (int l = 1; l <= M->lc; l++)
    if ((rc = mg_vc_sums(ctx, l, ids[l - 1], ids[l]))) return rc;
  return FS_OK;
}

// What the cycle touches of the levels >= 1 goes into one block, the coarsest
// level first, with the barrier count and the partial sums: the small levels
// share a few pages instead of one allocation (and page) per array.  Device
// memory with everything else of the hierarchy, 3.4 M cells: 189 bytes a cell in
// FP64 and 195 in FP32 (24 more where level 0 has no row patterns); the
// mesh-ordered levels of the general V-cycle take 140 and 168.
template <class R>
static int mg_vc_arrays(fs_ctx *ctx, const std::vector<std::vector<int32_t>> &ids) {
  constexpr bool f32 = sizeof(R) == sizeof(float);
  fs_mg_dev *M = ctx->mg;
  const int lc = M->lc;
  const size_t N = M->n[0], W = M->w[0];
  int rc;
  char *base = nullptr;
  size_t off = 0;
  auto take = [&](auto **d, size_t n) {
    *d = base ? reinterpret_cast<std::remove_reference_t<decltype(*d)>>(base + off) : nullptr;
    off += (std::max<size_t>(n, 1) * sizeof(**d) + 255) / 256 * 256;
  };
  VcDev<R> v{};
  R *val[FS_MG_MAXLEV] = {}, *ac[FS_MG_MAXLEV] = {};
  int32_t *kp[FS_MG_MAXLEV] = {}, *col[FS_MG_MAXLEV] = {};
  // Level 0: the matrix in the layout, x and r.  The FP32 cycle reads FP32 copies (in mesh
  // order too, for the up leg); the FP64 matrix in the layout is then only the source of
  // level 1's and sits in the gradient routine's scratch during the set-up.  Allocated ahead
  // of the block: where arrays come to lie moves the kernel by a percent or two, and the
  // other way round the p' solves of a 295k-cell run took 2.4 % longer (19.42 against 18.96
  // ms, FP64; other runs within 1 % either way).
  R *x0 = nullptr, *r0 = nullptr;
  if ((rc = mg_alloc(ctx, &x0, N)) || (rc = mg_alloc(ctx, &r0, N))) return rc;
  if constexpr (f32) {
    if ((rc = mg_alloc(ctx, &val[0], W * N)) || (rc = mg_alloc(ctx, &ac[0], N)) || (rc = mg_alloc(ctx, &M->anbm, W * N)) ||
        (rc = mg_alloc(ctx, &M->acm, N)))
      return rc;
  }
  if (f32 && W + 1 <= FS_GTMP_BLOCKS) { M->val0[f32] = ctx->gtmp; M->ac0[f32] = ctx->gtmp + W * N; }
  else if ((rc = mg_alloc(ctx, &M->val0[f32], W * N)) || (rc = mg_alloc(ctx, &M->ac0[f32], N))) return rc;
  for (int pass = 0; pass < 2; pass++) {
    if (pass == 1 && (rc = mg_alloc(ctx, &base, off))) return rc;
    off = 0;
    take(&M->vbar[f32], FS_GRIDBAR_WORDS);
    take(&M->vpart[f32], (9 + FS_SUMK) * (size_t)FS_RED_BLOCKS);
    take(&M->vinv[f32], (size_t)M->n[lc] * M->n[lc]);
    for (int l = lc; l >= 1; l--) {
      VcLevel<R> &d = v.L[l];
      take(&ac[l], M->n[l]);
      take(&d.b, M->n[l]);
      take(&d.x, M->n[l]);
      take(&d.r, M->n[l]);
      if (l < lc) take(&kp[l], M->n[l + 1] + 1);
      take(&col[l], M->vnpos[l]);
      take(&val[l], M->vnpos[l]);
    }
    take(&v.x1, M->n[1]);   // the result of level 1
  }
  for (int l = 1; l <= lc; l++) {
    if (l < lc) {
      const std::vector<int32_t> h = vc_first(M, l, ids);
      FS_CK(fs_upload(ctx, kp[l], h.data(), sizeof(int32_t) * h.size()));
    }
    const std::vector<int32_t> h = vc_columns(ctx, l, ids[l]);
    FS_CK(fs_upload(ctx, col[l], h.data(), sizeof(int32_t) * h.size()));
  }
  // FP64 matrices of the other levels, shared by both precisions
  double *fval[FS_MG_MAXLEV] = {}, *fac[FS_MG_MAXLEV] = {};
  for (int l = 1; l <= lc; l++) {
    if constexpr (!f32) { fval[l] = val[l]; fac[l] = ac[l]; }
    else if (M->vc_ready[0]) { fval[l] = M->vval[l]; fac[l] = M->vac[l]; }
    else if ((rc = mg_alloc(ctx, &fval[l], M->vnpos[l])) || (rc = mg_alloc(ctx, &fac[l], M->n[l]))) return rc;
  }
  if constexpr (!f32) { val[0] = M->val0[0]; ac[0] = M->ac0[0]; }
  kp[0] = M->vkp[0]; col[0] = M->vcol[0];
  v.lc = lc;
  for (int l = 0; l <= lc; l++) {
    VcLevel<R> &d = v.L[l];
    d.n = M->n[l]; d.w = M->w[l];
    d.col = col[l]; d.val = val[l]; d.ac = ac[l]; d.kp = kp[l];
  }
  v.L[0].cells = M->cells;
  v.L[0].r = r0;
  v.sinv = M->vinv[f32];
  LevelDev<R> &q = v.L0;
  q.n = M->n[0]; q.w = M->w[0]; q.ncolors = ctx->ncolors; q.ncf = ctx->ncf; q.nbr = ctx->cn;
  q.color_rows = ctx->color_rows; q.color_ptr = ctx->color_rows + N;
  if constexpr (f32) { q.ac = M->acm; q.anb = M->anbm; } else { q.ac = ctx->ac; q.anb = ctx->anb; }
  q.x = x0; q.r = r0;
  v.par0 = M->par0;
  v.npat = M->npat; v.pat = M->pat; v.patL = M->patL; v.offs = M->offs;
  VcDev<R> *dev = nullptr;
  if ((rc = mg_alloc(ctx, &dev, 1))) return rc;
  FS_CK(fs_upload(ctx, dev, &v, sizeof(v)));
  // nothing fails from here on: what both precisions use may change
  for (int l = 1; l <= lc; l++) { M->vkp[l] = kp[l]; M->vcol[l] = col[l]; M->vval[l] = fval[l]; M->vac[l] = fac[l]; }
  if constexpr (f32) {
    for (int l = 0; l <= lc; l++) { M->vvalf[l] = val[l]; M->vacf[l] = ac[l]; }
    M->vc32 = dev;
  } else M->vc64 = dev;
  M->vc_ready[f32] = true;
  return FS_OK;
}

static int mg_vc_build(fs_ctx *ctx, bool f32) {
  fs_mg_dev *M = ctx->mg;
  if (M->vc_ready[f32]) return FS_OK;
  const std::vector<std::vector<int32_t>> ids = vc_numbers(M);
  int rc;
  if (!M->vc_map) {
    if ((rc = mg_part(ctx, [&] { return mg_vc_map(ctx, ids); }))) return rc;
    M->vc_map = true;
  }
  return mg_part(ctx, [&] { return f32 ? mg_vc_arrays<float>(ctx, ids) : mg_vc_arrays<double>(ctx, ids); });
}

// the current matrices in the V-cycle's layout (level0: level 0 alone, the
// coarse levels being kept)
static int mg_vc_values(fs_ctx *ctx, bool f32, bool level0) {
  fs_mg_dev *M = ctx->mg;
  k_mg_level0<<<fs_grid(M->n[0]), FS_BLOCK, 0, ctx->st>>>(
      M->n[0], M->w[0], M->cells, ctx->ac, ctx->anb, M->ac0[f32], M->val0[f32], f32 ? M->vacf[0] : nullptr,
      f32 ? M->vvalf[0] : nullptr, f32 ? M->acm : nullptr, f32 ? M->anbm : nullptr);
  FS_LAUNCH_CHECK();
  for (int l = 1; l <= M->lc && !level0; l++) {
    k_mg_coarse<<<fs_grid((long)M->vnpos[l] + M->n[l]), FS_BLOCK, 0, ctx->st>>>(
        M->vnpos[l], M->n[l], M->csum[l].ptr, M->csum[l].idx, M->cdiag[l].ptr, M->cdiag[l].idx,
        l > 1 ? M->vac[l - 1] : M->ac0[f32], l > 1 ? M->vval[l - 1] : M->val0[f32], M->vac[l], M->vval[l], f32 ? M->vacf[l] : nullptr, f32 ? M->vvalf[l] : nullptr);
    FS_LAUNCH_CHECK();
  }
  return FS_OK;
}

// phases of one cycle of k_mg_solve (Cycle::run) if CTA 0 did all of it: the
// visits of a level times its colour passes, residuals, restriction and prolongation
static long mg_cycle_phases(const fs_mg_dev *M, int type, int pre, int post) {
  const int L = M->nlev - 1;
  long visits = 2L * L + 1;
  if (type != 0) for (int l = L - 1; l >= 1; l--) visits += 2L * (L - l) + 1;
  if (type == 2) for (int l = 2; l <= L - 1; l++) visits += 2L * (L - l) + 1;
  const long colours = *std::max_element(M->ncol, M->ncol + M->nlev);
  return visits * (std::max({pre, post, 1}) * (2 * colours + 1) + 3);
}

int fs_mg_solve(fs_ctx *ctx, int nf, double rrf, int solver) {
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  fs_mg_dev *M = ctx->mg;
  const bool gs = solver == FS_SOLVER_AMG32GS_BICGS;
  const bool f32 = solver == FS_SOLVER_AMG32_BICGS || gs;
  if (gs && !(M->direct && M->lc > 0)) {
    ctx->err = "the Gauss-Seidel V-cycle needs a coarsest level small enough for the dense inverse";
    return FS_E_UNSUPPORTED;
  }
  const int G = std::min(ctx->num_sms * fs_coop_per_sm(ctx, M->per_sm), FS_RED_BLOCKS);
  if (solver == FS_SOLVER_AMG) {
    if ((rc = mg_mesh_build<double>(ctx))) return rc;
    if ((rc = mg_coarse_matrices(ctx, M->nlev - 1, false))) return rc;
    M->built_nf = 0;
    MgSolveArgs a{};
    a.lev = M->lev64; a.nlev = M->nlev; a.type = ctx->cfg.mg_cycle; a.pre = ctx->cfg.mg_pre; a.post = ctx->cfg.mg_post;
    a.maxcycles = ctx->cfg.mg_max_cycles; a.b0 = ctx->bc; a.x0 = ctx->dphi; a.r0 = M->r[0];
    a.rrf = rrf; a.ires = ctx->resblk + RB_ABS + (nf - 1); a.part = M->red; a.iters = ctx->d_iters + (nf - 1);
    a.gridbar = M->gridbar; a.status = ctx->d_status;
    a.spin_limit = FS_PC_SPIN_LIMIT + FS_PHASE_POLLS * mg_cycle_phases(M, a.type, a.pre, a.post);
    FS_CK(cudaMemsetAsync(M->gridbar, 0, sizeof(unsigned) * FS_GRIDBAR_WORDS, ctx->st));
    void *args[] = {&a};
    if (!ctx->graph_mode) ctx->wait_open = true;
    FS_TIMING(FS_CK(cudaEventRecord(ctx->kev[nf - 1][0], ctx->st)));
    FS_CK(fs_coop_launch((const void *)k_mg_solve, G, fs_coop_block(ctx), args, ctx->st));
    FS_LAUNCH_CHECK();
    FS_TIMING(FS_CK(cudaEventRecord(ctx->kev[nf - 1][1], ctx->st)));
    return FS_OK;
  }
  // coarse levels and the dense coarsest inverse: rebuilt every pc_refresh solves
  // of the same system (1: every solve); in between the V-cycle keeps them and
  // only level 0 (the current system) is new -- a fixed preconditioner within
  // each solve, which still runs to its tolerance
  // the one-phase V-cycle needs one pre- and one post-sweep and a dense coarsest level
  const bool fused = std::max(1, ctx->cfg.mg_pre) == 1 && M->direct && M->lc > 0;
  const bool vc = gs || fused;
  if ((rc = vc ? mg_vc_build(ctx, f32) : f32 ? mg_mesh_build<float>(ctx) : mg_mesh_build<double>(ctx))) return rc;
  const int refresh = std::max(1, ctx->cfg.pc_refresh);
  const bool reuse = M->built_nf == nf && M->built_f32 == f32 && M->built_vc == vc && M->age + 1 < refresh;
  if (reuse) M->age++;
  else { M->built_nf = nf; M->built_f32 = f32; M->built_vc = vc; M->age = 0; }
  if (vc) {
    if ((rc = mg_vc_values(ctx, f32, reuse))) return rc;
  } else if (!reuse) {
    if ((rc = mg_coarse_matrices(ctx, M->lc, f32))) return rc;
  } else if (f32) {   // level 0 in FP32 from the current system
    const long n = M->n[0], nw = (long)M->w[0] * M->n[0];
    k_to_f32<<<fs_grid(n), FS_BLOCK, 0, ctx->st>>>(n, M->ac[0], M->acf[0]);
    FS_LAUNCH_CHECK();
    k_to_f32<<<fs_grid(nw), FS_BLOCK, 0, ctx->st>>>(nw, M->anb[0], M->anbf[0]);
    FS_LAUNCH_CHECK();
  }
  // team-barrier counters of the V-cycle start at zero for every launch
  FS_CK(cudaMemsetAsync(ctx->d_status + 4, 0, sizeof(int32_t) * 2, ctx->st));
  unsigned *gridbar = vc ? M->vbar[f32] : M->gridbar;
  FS_CK(cudaMemsetAsync(gridbar, 0, sizeof(unsigned) * FS_GRIDBAR_WORDS, ctx->st));
  if (M->direct && !reuse) {
    const int q = M->lc;
    if ((rc = vc ? dense_inverse(ctx, M->n[q], M->w[q], M->vcol[q], M->vac[q], M->vval[q], true, M->vinv[f32])
                 : dense_inverse(ctx, M->n[q], M->w[q], M->nbr[q], M->ac[q], M->anb[q], false, M->sinv)))
      return rc;
  }
  auto fill = [&](auto &a) {
    a.N = ctx->N; a.W = ctx->W; a.ncf = ctx->ncf; a.cn = ctx->cn; a.ac = ctx->ac; a.anb = ctx->anb; a.bc = ctx->bc;
    a.x = ctx->kx; a.r = ctx->kr; a.r0 = ctx->kr0; a.p = ctx->kp; a.v = ctx->kv; a.s = ctx->ks; a.t = ctx->kt;
    a.y = ctx->ky; a.z = ctx->kz; a.dphi = ctx->dphi;
    // one V-cycle per application: one pre- and one post-sweep (MultiGridpreSweep)
    a.lc = M->lc; a.direct = M->direct; a.sinv = M->sinv;
    a.pre = std::max(1, ctx->cfg.mg_pre); a.post = std::max(1, ctx->cfg.mg_pre);
    a.maxit = ctx->cfg.krylov_maxit; a.tol = ctx->cfg.krylov_tol; a.part = vc ? M->vpart[f32] : M->red;
    a.iters = ctx->d_iters + (nf - 1); a.diag = ctx->resblk + RB_DIAG;
    a.nx = 0;
    if (nf == FS_VAR_PC)
      for (int j = 0; j < ctx->pc_nguess && j < FS_GUESS_MAX; j++) a.xs[a.nx++] = ctx->pc_guess[j];
    a.fit = ctx->d_status + 6;
    a.nncnt = ctx->pc_nn ? fs_nn_counters(ctx) : nullptr;   // the network's guess is in the basis
    a.gridbar = gridbar;
    // PCycle's team and CTA 0 work on the coarse levels alone: their sweeps of two phases,
    // restrictions, prolongations and the coarsest level's 20 sweeps
    a.spin_limit = FS_PC_SPIN_LIMIT + (vc ? 0 : FS_PHASE_POLLS * ((2L * (a.pre + (long)a.post) + 4) * M->lc + 48));
    a.teambar = (unsigned *)(ctx->d_status + 4);
    a.status = ctx->d_status;
    a.team_extra = ctx->test_wait_extra >= 0 ? ctx->test_wait_extra : ctx->graph_mode ? -ctx->test_wait_extra : 0;
  };
  if (ctx->pc_defer && nf == FS_VAR_PC) {   // prepared here, launched with other contexts' by fs_pc_batch_launch
    int form = -1;
    if ((rc = fs_pc_batch_form(ctx, &form))) return rc;
    if (form < 0) { ctx->err = "this p' solver cannot join a batched launch"; return FS_E_UNSUPPORTED; }
    M->pend_form = form;   // the initial-guess fit runs in the batched launch too
    if (!f32) {
      M->pend64 = AmgKArgs<double>{};
      fill(M->pend64);
      M->pend64.lev = vc ? &M->vc64->L0 : M->lev64; M->pend64.vc = M->vc64;
    } else {
      M->pend32 = AmgKArgs<float>{};
      fill(M->pend32);
      M->pend32.lev = vc ? &M->vc32->L0 : M->lev32; M->pend32.vc = M->vc32;
    }
    return FS_OK;
  }
  if (!ctx->graph_mode) ctx->wait_open = true;   // graphs copy the status word themselves
  if (!f32) {
    AmgKArgs<double> a{};
    fill(a);
    a.lev = vc ? &M->vc64->L0 : M->lev64; a.vc = M->vc64;
    void *args[] = {&a};
    if (a.nx > 0) FS_CK(fs_coop_launch(guess_fit_kernel<double>(a.nx), G, fs_coop_block(ctx), args, ctx->st));
    FS_TIMING(FS_CK(cudaEventRecord(ctx->kev[nf - 1][0], ctx->st)));
    FS_CK(fs_coop_launch(fused ? (const void *)k_amg_bicgstab<double, 1> : (const void *)k_amg_bicgstab<double, 0>,
                         G, fs_coop_block(ctx), args, ctx->st));
  } else {
    AmgKArgs<float> a{};
    fill(a);
    a.lev = vc ? &M->vc32->L0 : M->lev32; a.vc = M->vc32;
    void *args[] = {&a};
    if (a.nx > 0) FS_CK(fs_coop_launch(guess_fit_kernel<float>(a.nx), G, fs_coop_block(ctx), args, ctx->st));
    FS_TIMING(FS_CK(cudaEventRecord(ctx->kev[nf - 1][0], ctx->st)));
    const void *k = gs ? (const void *)k_amg_bicgstab<float, 2>
                    : fused ? (const void *)k_amg_bicgstab<float, 1> : (const void *)k_amg_bicgstab<float, 0>;
    FS_CK(fs_coop_launch(k, G, fs_coop_block(ctx), args, ctx->st));
  }
  FS_LAUNCH_CHECK();
  FS_TIMING(FS_CK(cudaEventRecord(ctx->kev[nf - 1][1], ctx->st)));
  (void)rrf;
  return FS_OK;
}

extern "C" int fs_mg_levels(fs_ctx *ctx, int32_t *n_levels, int32_t *level_sizes, int max_levels) {
  if (!ctx) return FS_E_ARG;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  if (n_levels) *n_levels = ctx->mg->nlev;
  if (level_sizes)
    for (int q = 0; q < ctx->mg->nlev && q < max_levels; q++) level_sizes[q] = ctx->mg->n[q];
  return FS_OK;
}

extern "C" int fs_mg_parents(fs_ctx *ctx, int level, int32_t *parents, size_t n) {
  if (!ctx || !parents) return FS_E_ARG;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  if (level < 0 || level + 1 >= ctx->mg->nlev || n != ctx->mg->h_parent[level].size()) return FS_E_ARG;
  memcpy(parents, ctx->mg->h_parent[level].data(), sizeof(int32_t) * n);
  return FS_OK;
}

extern "C" int fs_mg_info(fs_ctx *ctx, int32_t *widths, int max_levels, int32_t *prec_coarsest, int32_t *direct) {
  if (!ctx) return FS_E_ARG;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  if (widths)
    for (int q = 0; q < ctx->mg->nlev && q < max_levels; q++) widths[q] = ctx->mg->w[q];
  if (prec_coarsest) *prec_coarsest = ctx->mg->lc;
  if (direct) *direct = ctx->mg->direct ? 1 : 0;
  return FS_OK;
}

extern "C" int fs_mg_coarse_matrix(fs_ctx *ctx, int level, double *ac, int32_t *n_nbr, int32_t *nbr, double *anb,
                                   size_t n, size_t w) {
  if (!ctx || !ac || !n_nbr || !nbr || !anb) return FS_E_ARG;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  fs_mg_dev *M = ctx->mg;
  if (level < 1 || level >= M->nlev || n != (size_t)M->n[level] || w != (size_t)M->w[level]) return FS_E_ARG;
  cudaSetDevice(ctx->dev);
  if ((rc = mg_mesh_tables_once(ctx)) || (rc = mg_coarse_matrices(ctx, level, false))) return rc;
  FS_CK(cudaMemcpyAsync(ac, M->ac[level], sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->st));
  FS_CK(cudaMemcpyAsync(anb, M->anb[level], sizeof(double) * n * w, cudaMemcpyDeviceToHost, ctx->st));
  FS_CK(cudaMemcpyAsync(n_nbr, M->nnb[level], sizeof(int32_t) * n, cudaMemcpyDeviceToHost, ctx->st));
  FS_CK(cudaMemcpyAsync(nbr, M->nbr[level], sizeof(int32_t) * n * w, cudaMemcpyDeviceToHost, ctx->st));
  FS_CK(cudaStreamSynchronize(ctx->st));
  return FS_OK;
}

// The same level as the one-phase V-cycle holds it, in the numbering and slots of
// fs_mg_coarse_matrix (0 in the slots past n_nbr; f32: the FP32 cycle's copy).
// For tests: the two are assembled by different kernels.
extern "C" int fs_mg_vcycle_matrix(fs_ctx *ctx, int level, int f32, double *ac, double *anb, size_t n, size_t w) {
  if (!ctx || !ac || !anb) return FS_E_ARG;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  fs_mg_dev *M = ctx->mg;
  if (!M->direct || level < 1 || level > M->lc || n != (size_t)M->n[level] || w != (size_t)M->w[level]) return FS_E_ARG;
  cudaSetDevice(ctx->dev);
  if ((rc = mg_vc_build(ctx, f32 != 0)) || (rc = mg_vc_values(ctx, f32 != 0, false))) return rc;
  M->built_nf = 0;   // the coarse levels are this system's now
  auto read = [&](auto *dac, auto *dval) -> int {
    std::vector<std::remove_pointer_t<decltype(dac)>> a(n), v(M->vnpos[level]);
    FS_CK(cudaMemcpyAsync(a.data(), dac, sizeof(a[0]) * a.size(), cudaMemcpyDeviceToHost, ctx->st));
    FS_CK(cudaMemcpyAsync(v.data(), dval, sizeof(v[0]) * v.size(), cudaMemcpyDeviceToHost, ctx->st));
    FS_CK(cudaStreamSynchronize(ctx->st));
    const std::vector<int32_t> id = vc_numbers(M)[level];
    for (size_t i = 0; i < n; i++) {
      ac[i] = a[id[i]];
      for (size_t j = 0; j < w; j++) anb[j * n + i] = v[vc_pos(level, (int)n, (int)w, id[i], (int)j)];
    }
    return FS_OK;
  };
  return f32 ? read(M->vacf[level], M->vvalf[level]) : read(M->vac[level], M->vval[level]);
}

// Test of the bounded device waits (no reference counterpart): with extra > 0
// the grid barriers of the AMG solves wait for more CTAs than take part (with
// extra < 0 those of solves inside a captured graph alone), so their polls run
// out; the solve then ends and the call that reads its results reports
// FS_E_TIMEOUT.
extern "C" int fs_test_wait_timeout(fs_ctx *ctx, int extra) {
  if (!ctx || extra < -64 || extra > 64) return FS_E_ARG;
  ctx->test_wait_extra = extra;
  return FS_OK;
}

extern "C" int fs_test_alloc_failure(fs_ctx *ctx, int nth) {
  if (!ctx || nth < 0) return FS_E_ARG;
  ctx->test_alloc_left = nth;
  return FS_OK;
}

// ------------------------------------------------------------ batched p' solves
// Several contexts' AMG-BiCGSTAB solves in one cooperative launch of
// k_amg_bicgstab_batch (no reference counterpart; the ensemble form).  Form:
// 0/1 FP64 V-cycle run()/fused, 2/3 FP32 run()/fused, 4 FP32 Gauss-Seidel; -1
// when the context's p' solver is not an AMG-BiCGSTAB one.
int fs_pc_batch_form(fs_ctx *ctx, int *form) {
  if (!ctx || !form) return FS_E_ARG;
  *form = -1;
  const int sv = ctx->cfg.solver_cont;
  if (sv != FS_SOLVER_AMG_BICGS && sv != FS_SOLVER_AMG32_BICGS && sv != FS_SOLVER_AMG32GS_BICGS) return FS_OK;
  int rc = fs_mg_build(ctx);
  if (rc) return rc;
  const fs_mg_dev *M = ctx->mg;
  const bool gs = sv == FS_SOLVER_AMG32GS_BICGS, f32 = sv != FS_SOLVER_AMG_BICGS;
  if (gs && !(M->direct && M->lc > 0)) return FS_OK;
  const bool fused = std::max(1, ctx->cfg.mg_pre) == 1 && M->direct && M->lc > 0;
  *form = !f32 ? (fused ? 1 : 0) : gs ? 4 : fused ? 3 : 2;
  return FS_OK;
}

struct fs_pc_batch {
  int n = 0, form = -1, ncta = 0;
  size_t argsz = 0;
  void *h_args = nullptr;       // pinned: the n argument blocks, copied to d_args by each launch
  void *d_args = nullptr;
  int32_t *d_start = nullptr;   // n + 1 CTA offsets
  unsigned *d_words = nullptr;  // per context FS_GRIDBAR_WORDS barrier counts, then 2 team words each (zero at each launch)
  std::vector<int32_t> start;
};

static const void *batch_kernel(int form) {
  switch (form) {
    case 0: return (const void *)k_amg_bicgstab_batch<double, 0>;
    case 1: return (const void *)k_amg_bicgstab_batch<double, 1>;
    case 2: return (const void *)k_amg_bicgstab_batch<float, 0>;
    case 3: return (const void *)k_amg_bicgstab_batch<float, 1>;
    case 4: return (const void *)k_amg_bicgstab_batch<float, 2>;
  }
  return nullptr;
}

void fs_pc_batch_free(fs_pc_batch *B) {
  if (!B) return;
  if (B->h_args) cudaFreeHost(B->h_args);
  if (B->d_args) cudaFree(B->d_args);
  if (B->d_start) cudaFree(B->d_start);
  if (B->d_words) cudaFree(B->d_words);
  delete B;
}

// CTAs of one co-resident launch (1024 threads each, one per SM) split among
// the n contexts in proportion to weight[q] (fs_cta_split)
int fs_pc_batch_create(fs_ctx **cs, int n, const double *weight, fs_pc_batch **out) {
  if (!cs || n < 1 || !weight || !out) return FS_E_ARG;
  *out = nullptr;
  fs_ctx *ctx = cs[0];
  int form = -1;
  for (int q = 0; q < n; q++) {
    int f = -1;
    int rc = fs_pc_batch_form(cs[q], &f);
    if (rc) { if (cs[q] != ctx) ctx->err = cs[q]->err; return rc; }
    if (f < 0 || (q > 0 && f != form)) { ctx->err = "contexts cannot share a batched p' launch"; return FS_E_UNSUPPORTED; }
    form = f;
  }
  int occ = 0;
  FS_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_kernel(form), FS_COOP_BLOCK, 0));
  const int cap = std::min(ctx->num_sms * std::max(occ, 0), FS_RED_BLOCKS);
  if (cap < n) { ctx->err = "more contexts than co-resident CTAs for a batched p' launch"; return FS_E_UNSUPPORTED; }
  const std::vector<int32_t> split = fs_cta_split(cap, weight, n);
  fs_pc_batch *B = new fs_pc_batch;
  B->n = n; B->form = form;
  B->argsz = form <= 1 ? sizeof(AmgKArgs<double>) : sizeof(AmgKArgs<float>);
  B->start = split;
  B->ncta = B->start[n];
  cudaError_t e;
  if ((e = cudaHostAlloc(&B->h_args, B->argsz * n, cudaHostAllocDefault)) != cudaSuccess ||
      (e = cudaMalloc(&B->d_args, B->argsz * n)) != cudaSuccess ||
      (e = cudaMalloc(&B->d_start, sizeof(int32_t) * (n + 1))) != cudaSuccess ||
      (e = cudaMalloc(&B->d_words, sizeof(unsigned) * (FS_GRIDBAR_WORDS + 2) * n)) != cudaSuccess ||
      (e = fs_upload(ctx, B->d_start, B->start.data(), sizeof(int32_t) * (n + 1))) != cudaSuccess) {
    ctx->err = std::string("batched p' set-up: ") + cudaGetErrorString(e);
    fs_pc_batch_free(B);
    return FS_E_CUDA;
  }
  *out = B;
  return FS_OK;
}

// launch the solves every context prepared with pc_defer (fs_mg_solve), on st;
// each context's status word records a barrier timeout as in its own launches
int fs_pc_batch_launch(fs_pc_batch *B, fs_ctx **cs, int n, cudaStream_t st) {
  if (!B || !cs || n != B->n) return FS_E_ARG;
  fs_ctx *ctx = cs[0];
  unsigned nx_mask = 0;
  for (int q = 0; q < n; q++) {
    fs_mg_dev *M = cs[q]->mg;
    if (!M || M->pend_form != B->form) { ctx->err = "batched p' launch: a context prepared no matching solve"; return FS_E_ARG; }
    char *dst = (char *)B->h_args + B->argsz * q;
    if (B->form <= 1) {
      AmgKArgs<double> a = M->pend64;
      a.gridbar = B->d_words + (size_t)FS_GRIDBAR_WORDS * q;
      a.teambar = B->d_words + (size_t)FS_GRIDBAR_WORDS * n + 2 * q;
      if (a.nx > 0 && a.nx <= FS_GUESS_MAX) nx_mask |= 1u << a.nx;
      memcpy(dst, &a, sizeof(a));
    } else {
      AmgKArgs<float> a = M->pend32;
      a.gridbar = B->d_words + (size_t)FS_GRIDBAR_WORDS * q;
      a.teambar = B->d_words + (size_t)FS_GRIDBAR_WORDS * n + 2 * q;
      if (a.nx > 0 && a.nx <= FS_GUESS_MAX) nx_mask |= 1u << a.nx;
      memcpy(dst, &a, sizeof(a));
    }
    M->pend_form = -1;
  }
  FS_CK(cudaMemcpyAsync(B->d_args, B->h_args, B->argsz * n, cudaMemcpyHostToDevice, st));
  void *args[] = {&B->d_args, &B->d_start, &B->n};
  // the initial guesses, same groups: one launch per basis size present (a
  // group sits out the launches of other sizes); the barrier words start from
  // zero for each launch
  for (int nx = 1; nx <= FS_GUESS_MAX; nx++) {
    if (!(nx_mask & (1u << nx))) continue;
    FS_CK(cudaMemsetAsync(B->d_words, 0, sizeof(unsigned) * (FS_GRIDBAR_WORDS + 2) * n, st));
    FS_CK(fs_coop_launch(B->form <= 1 ? guess_fit_batch_kernel<double>(nx) : guess_fit_batch_kernel<float>(nx),
                         B->ncta, FS_COOP_BLOCK, args, st));
    FS_LAUNCH_CHECK();
  }
  FS_CK(cudaMemsetAsync(B->d_words, 0, sizeof(unsigned) * (FS_GRIDBAR_WORDS + 2) * n, st));
  FS_CK(fs_coop_launch(batch_kernel(B->form), B->ncta, FS_COOP_BLOCK, args, st));
  FS_LAUNCH_CHECK();
  return FS_OK;
}
