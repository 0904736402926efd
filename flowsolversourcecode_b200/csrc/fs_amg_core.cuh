// Krylov solve with the V-cycle preconditioner and the grid reductions it
// uses.  Included twice by fs_mg.cu:
//   FS_GROUPS 0: the whole cooperative grid solves one system;
//   FS_GROUPS 1: the CTAs of one cooperative launch are split into groups, one
//     per system (the batched p' solve of an ensemble); CTA index and count are
//     relative to the group, held in shared memory.
// Either way the grid barrier is a bounded one in global memory among the CTAs
// of the system.
struct GridState {
  int cta, ncta, q;    // this CTA within its group, the group's CTAs, its system
  unsigned target;     // arrivals in all when the next barrier opens, less `arrivals`
  unsigned arrivals;   // arrivals per barrier
  unsigned *bar;       // arrival count, zero at launch, never reset
  long limit;          // polls of a barrier before it reports a timeout
  int32_t *status;     // [0] set when a barrier timed out
  double *part;        // partial sums
  int buf;             // buffer of the next sums
};
__device__ __forceinline__ GridState &gstate() {
  __shared__ GridState g;
  return g;
}
#if FS_GROUPS
__device__ __forceinline__ int cta_id() { return gstate().cta; }
__device__ __forceinline__ int cta_count() { return gstate().ncta; }
#else
__device__ __forceinline__ int cta_id() { return (int)blockIdx.x; }
__device__ __forceinline__ int cta_count() { return (int)gridDim.x; }
#endif
// before the first barrier, by every thread; `extra` arrivals never come (only
// to test the timeout)
__device__ __forceinline__ void grid_state_init(double *part, unsigned *bar, int32_t *status, int extra, long limit) {
  if (threadIdx.x == 0) {
    GridState &G = gstate();
    G.target = 0;
    G.arrivals = (unsigned)(cta_count() + extra);
    G.bar = bar;
    G.limit = limit;
    G.status = status;
    G.part = part;
    G.buf = 0;
  }
  __syncthreads();
}
// Barrier among the system's CTAs, all co-resident (cooperative launch): one
// release-add per CTA on a count that only grows, then acquire polls until it
// reaches the next multiple of the CTA count -- one round trip to the L2 for
// the arrival and one for the poll that sees the last one (1.2 us for 148 CTAs
// on B200, the empty barrier), no reset and no second word.  Polls are bounded;
// a timeout is recorded in the system's status word, and once that is set no
// barrier waits for long any more.
//
// Nothing that the solve needs later is left in registers across a barrier
// (arguments, descriptors and the iteration's scalars live in shared memory):
// the loops of every phase get the 64 registers that 1024 threads have.
__device__ __noinline__ void grid_barrier() {
  __syncthreads();
  if (threadIdx.x == 0) {
    GridState &G = gstate();
    const unsigned target = G.target + G.arrivals;
    unsigned *bar = G.bar;
    const long limit = G.limit;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    long spins = 0;
    unsigned seen;
    while (true) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if ((int)(seen - target) >= 0) break;
      if ((++spins & 63) == 0) {
        if (*(const volatile int32_t *)G.status != 0) break;
        if (spins > limit) { atomicExch(G.status, 1); break; }
      }
    }
    G.target = target;
  }
  __syncthreads();
}

// grid-deterministic sums of K <= 3 values (every CTA gets the same results):
// the warps' sums into shared memory, warp k adds them and writes the CTA's
// partial of value k; behind the barrier warp k adds the CTAs' partials, 32 at a
// time, and the sums of those.  Two block barriers beside the grid barrier's
// two; three buffers, so a CTA still reading one sum is not overwritten by the
// next.
struct Sum3 { double a, b, c; };
template <int K>
__device__ __forceinline__ Sum3 grid_sums(Sum3 in) {
  __shared__ double sh[3][33];
  GridState &S = gstate();
  const int G = cta_count(), lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double w0 = wsum(in.a), w1 = K > 1 ? wsum(in.b) : 0., w2 = K > 2 ? wsum(in.c) : 0.;
  if (lane == 0) {
    sh[0][wid] = w0;
    if (K > 1) sh[1][wid] = w1;
    if (K > 2) sh[2][wid] = w2;
  }
  __syncthreads();
  double *pb = S.part + (long)(3 * S.buf + wid) * G;
  if (wid < K) {
    const double v = wsum(lane < nw ? sh[wid][lane] : 0.);
    if (lane == 0) pb[cta_id()] = v;
  }
  grid_barrier();
  if (wid < K) {
    double r = 0.;
    for (int c0 = 0; c0 < nw && c0 * 32 < G; c0 += 5) {   // 148 CTAs: one round
      double v[5];
#pragma unroll
      for (int c = 0; c < 5; c++) {
        const int q = (c0 + c) * 32 + lane;
        v[c] = c0 + c < nw && q < G ? 0. + pb[q] : 0.;
        if (c0 + c < nw) for (int m = q + blockDim.x; m < G; m += blockDim.x) v[c] += pb[m];
      }
#pragma unroll
      for (int c = 0; c < 5; c++) {
        const double t = __shfl_sync(0xffffffffu, wsum(v[c]), 0);
        if (lane == c0 + c) r = t;
      }
    }
    r = wsum(r);
    if (lane == 0) sh[wid][32] = r;
  }
  if (threadIdx.x == 0) S.buf = (S.buf + 1) % 3;
  __syncthreads();
  return Sum3{sh[0][32], K > 1 ? sh[1][32] : 0., K > 2 ? sh[2][32] : 0.};
}

struct Sync {
  __device__ Sync(double *part, unsigned *bar, int32_t *status, int extra, long limit) {
    grid_state_init(part, bar, status, extra, limit);
  }
  __device__ __forceinline__ void gbar() { grid_barrier(); }
  __device__ __forceinline__ void all() { grid_barrier(); }
  __device__ __forceinline__ void sum2(double a0, double a1, double &o0, double &o1) {
    const Sum3 r = grid_sums<2>(Sum3{a0, a1, 0.});
    o0 = r.a; o1 = r.b;
  }
  // grid-deterministic sums of K <= FS_SUMK values, in the partial slots after
  // the three buffers of sums (every CTA gets the same results), with one
  // block barrier before and one after the grid barrier: warp sums into shared
  // memory, thread k adds the warps' and then the CTAs' partials of value k in
  // a fixed order
  template <int K>
  __device__ void sumKt(const double (&in)[K], double (&out)[K]) {
    __shared__ double sh[K][33];
    const int G = cta_count(), lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double *pk = gstate().part + 9L * G;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const double v = wsum(in[k]);
      if (lane == 0) sh[k][wid] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < K) {
      const int k = threadIdx.x;
      double t = 0.;
      for (int w = 0; w < nw; w++) t += sh[k][w];
      pk[(long)k * G + cta_id()] = t;
    }
    gbar();
    if ((int)threadIdx.x < K) {
      const int k = threadIdx.x;
      double t = 0.;
      for (int q = 0; q < G; q++) t += pk[(long)k * G + q];
      sh[k][32] = t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = sh[k][32];
  }
};

// which threads work on a level, and how they synchronise
// the first FS_PC_TEAM CTAs: mid-sized preconditioner levels (PCycle)
__device__ __forceinline__ int team_size() { return cta_count() < FS_PC_TEAM ? cta_count() : FS_PC_TEAM; }

struct Scope {
  bool grid = false;   // whole grid
  bool team = false;   // else the first team_size() CTAs; else CTA 0 only
  __device__ bool active() const { return grid || (team ? cta_id() < team_size() : cta_id() == 0); }
  __device__ long tid0() const {
    return (grid || team) ? (long)cta_id() * blockDim.x + threadIdx.x : (long)threadIdx.x;
  }
  __device__ long nth() const {
    return grid ? (long)cta_count() * blockDim.x : team ? (long)team_size() * blockDim.x : (long)blockDim.x;
  }
};

// One V-cycle with zero initial guesses as the preconditioner M^-1 of the Krylov
// solver.  Damped Jacobi (omega) on every level, so each sweep is one phase of
// independent rows; the first pre-sweep from zero is fused into the restriction
// that makes the level's rhs, and the coarsest level is solved by a dense FP64
// inverse (k_mg_dense_inverse).  The coarse correction is over-weighted,
// x += alpha*x_c[parent] with alpha > 1, which compensates the energy of
// piecewise-constant prolongation.  On levels with a thread per row the
// prolongation is a phase of its own before the first post-sweep; on levels
// with G lanes per row it is formed on the fly inside the sweep for the row and
// its neighbours.  A cycle over levels 0..lc costs 3*lc+2 barrier phases plus one
// per thread-per-row level.  Level-0 rhs and result are FP64 in either
// precision; up-leg results go to each level's r.
//
// Rows with fewer than two threads each are handled a thread per row, two rows
// per step (ell_acc2).  Coarse rows have 10-30 neighbours and coarse levels
// fewer rows than the grid has threads, so there a row is handled by G
// consecutive lanes (G = 2..8 from the threads per row) that split its
// neighbour loop and combine by shuffles.  Levels up to FS_PC_SMALL rows run on
// CTA 0 alone; levels up to FS_PC_TEAM_MAX rows on a team of the first
// FS_PC_TEAM CTAs with a bounded barrier of their own in global memory -- a
// barrier over all CTAs costs several microseconds, and those phases have too
// little work to use the whole grid anyway.

template <class R>
__device__ __forceinline__ Scope pc_scope(const LevelDev<R> &L) {
  Scope s;
  s.grid = L.n > FS_PC_TEAM_MAX;
  s.team = !s.grid && L.n > FS_PC_SMALL;
  return s;
}

template <int G, class T>
__device__ __forceinline__ T gsum(T v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// rows [0,n) by groups of G consecutive lanes; the trip count is uniform per
// warp, so every lane reaches the group shuffles (f must not return early)
template <int G, class F>
__device__ __forceinline__ void group_rows(const Scope &sc, int n, F &f) {
  constexpr int GPW = 32 / G;
  const long w0 = sc.tid0() >> 5, nw = sc.nth() >> 5;
  const int lane = threadIdx.x & 31, grp = lane / G, q = lane % G;
  for (long wb = w0 * GPW; wb < n; wb += nw * GPW) {
    long i = wb + grp;
    f(std::integral_constant<int, G>{}, i, i < n, q);
  }
}

// G from the threads per row (callers handle fewer than 2 threads per row)
template <class F>
__device__ __forceinline__ void level_rows(const Scope &sc, int n, int level, F &&f) {
  const long per = sc.nth() / (n > 0 ? n : 1);
  (void)level;
  if (per < 4) group_rows<2>(sc, n, f);
  else if (per < 8) group_rows<4>(sc, n, f);
  else group_rows<8>(sc, n, f);
}

template <class R>
struct PCycle {
  Sync &S;
  const LevelDev<R> *lev;
  int lc;              // coarsest level used by the preconditioner
  bool direct;         // coarsest by the dense inverse, else coarse_sweeps sweeps
  const double *sinv;  // lev[lc].n^2, row-major
  int pre, post, coarse_sweeps;
  R omega, alpha;        // Jacobi weight and coarse-correction factor on levels >= 1
  Scope last;            // scope of the previous phase
  R omega0, alpha0;      // the same on level 0
  unsigned *bar;         // team barrier: [0] arrivals, [1] generation (zero at launch)
  int32_t *status;       // [0] set when a team barrier timed out
  unsigned gen;          // generation this CTA waits to leave
  int extra;             // arrivals waited for beyond the team (0; >0 only to test the timeout)
  __device__ R om(int l) const { return l == 0 ? omega0 : omega; }
  __device__ R al(int l) const { return l == 0 ? alpha0 : alpha; }
  // barrier among the team CTAs: the arrival count in global memory, the last
  // arrival resets it and bumps the generation the others poll; polls are
  // bounded, and a timeout is recorded (later team barriers then stop
  // waiting).  The FP64 cycle calls it out of line (inlined at every phase it
  // doubled that kernel's register spills); the FP32 cycle, with fewer live
  // registers, runs faster with it inline.
  __device__ __noinline__ void team_sync_call() { team_sync_body(); }
  __device__ __forceinline__ void team_sync() {
    if (sizeof(R) == sizeof(double)) team_sync_call();
    else team_sync_body();
  }
  __device__ __forceinline__ void team_sync_body() {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned g = gen, T = (unsigned)(team_size() + extra);
      if (atomicAdd(&bar[0], 1u) == T - 1) {
        atomicExch(&bar[0], 0u);
        __threadfence();
        atomicAdd(&bar[1], 1u);
      } else {
        const volatile unsigned *vg = bar + 1;
        const volatile int32_t *vs = status;
        long spins = 0;
        while (*vg == g && *vs == 0) {
          if (++spins > FS_PC_SPIN_LIMIT) { atomicExch(status, 1); break; }
          __nanosleep(64);
        }
      }
      __threadfence();
    }
    gen++;
    __syncthreads();
  }
  // the barrier before a phase: grid-wide when the grid is involved on either
  // side, among the team when the team is, else within CTA 0
  __device__ void enter(const Scope &sc) {
    if (sc.grid || last.grid) S.all();
    else if (sc.team || last.team) { if (cta_id() < team_size()) team_sync(); }
    else __syncthreads();
    last = sc;
  }
  // r (into dst) = b - A x on level l; level 0 takes b from `in`
  __device__ void residual(int l, const double *__restrict__ in, const R *__restrict__ x, R *__restrict__ dst) {
    const LevelDev<R> L = lev[l];
    Scope sc = pc_scope(L);
    enter(sc);
    if (!sc.active()) return;
    if (l == 0 || sc.nth() < 2L * L.n) {   // a thread per row, two rows per step
      const long t0 = sc.tid0(), nt = sc.nth();
      for (long i = t0; i < L.n; i += 2 * nt) {
        const long i2 = i + nt;
        const bool h2 = i2 < L.n;
        R t1 = 0., t2 = 0.;
        ell_acc2<6, false>(t1, t2, L.n, L.w, L.nbr, L.anb, i, i2, h2, [&](int k) { return x[k]; });
        dst[i] = (l == 0 ? (R)in[i] : L.b[i]) - L.ac[i] * x[i] - t1;
        if (h2) dst[i2] = (l == 0 ? (R)in[i2] : L.b[i2]) - L.ac[i2] * x[i2] - t2;
      }
      return;
    }
    level_rows(sc, L.n, l, [&](auto g, long i, bool act, int q) {
      constexpr int G = decltype(g)::value;
      R t = 0.;
      if (act) t = ell_part<G, G == 1 ? 8 : 4>(L.n, L.w, L.nbr, L.anb, i, q, [&](int k) { return x[k]; });
      t = gsum<G>(t);
      if (act && q == 0) dst[i] = (l == 0 ? (R)in[i] : L.b[i]) - L.ac[i] * x[i] - t;
    });
  }
  // further Jacobi sweeps in place: residual into t, then the update
  __device__ void sweeps(int l, const double *in, R *x, int n) {
    const LevelDev<R> L = lev[l];
    Scope sc = pc_scope(L);
    for (int s = 0; s < n; s++) {
      residual(l, in, x, L.t);
      enter(sc);
      if (sc.active()) for (long i = sc.tid0(); i < L.n; i += sc.nth()) x[i] = x[i] + om(l) * L.t[i] / L.ac[i];
    }
  }
  // out = M^-1 in.  Callers have made `in` visible grid-wide.
  __device__ void run(const double *__restrict__ in, double *__restrict__ out) {
    Scope g; g.grid = true;
    {
      const LevelDev<R> L0 = lev[0];
      for (long i = g.tid0(); i < L0.n; i += g.nth()) L0.x[i] = omega0 * (R)in[i] / L0.ac[i];
    }
    last.grid = true;
    last.team = false;
    sweeps(0, in, lev[0].x, pre - 1);
    for (int l = 0; l < lc; l++) {
      const LevelDev<R> L = lev[l], C = lev[l + 1];
      residual(l, in, L.x, L.r);
      Scope scc = pc_scope(C);
      enter(scc);
      const bool first_sweep = l + 1 < lc || !direct;
      if (scc.active() && scc.nth() < 2L * C.n) {   // a thread per coarse row
        for (long P = scc.tid0(); P < C.n; P += scc.nth()) {
          R s = 0.;
          const int c0 = C.rptr[P], c1 = C.rptr[P + 1];
          for (int c = c0; c < c1; c++) s = s + L.r[C.rlist[c]];
          C.b[P] = s;
          if (first_sweep) C.x[P] = om(l + 1) * s / C.ac[P];
        }
      } else if (scc.active())
        level_rows(scc, C.n, l + 1, [&](auto gg, long P, bool act, int q) {
          constexpr int G = decltype(gg)::value;
          R s = 0.;
          if (act)
            for (int c = C.rptr[P] + q; c < C.rptr[P + 1]; c += G) s = s + L.r[C.rlist[c]];
          s = gsum<G>(s);
          if (act && q == 0) {
            C.b[P] = s;
            if (first_sweep) C.x[P] = om(l + 1) * s / C.ac[P];
          }
        });
      if (l + 1 < lc) sweeps(l + 1, in, C.x, pre - 1);
    }
    const LevelDev<R> Cc = lev[lc];
    if (direct) {
      Scope c0; c0.grid = false;
      enter(c0);
      if (cta_id() == 0) {
        const int n = Cc.n, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        for (int i = threadIdx.x >> 5; i < n; i += nw) {
          double t = 0.;
          for (int j = lane; j < n; j += 32) t += sinv[(long)i * n + j] * (double)Cc.b[j];
          t = wsum(t);
          if (lane == 0) Cc.r[i] = (R)t;
        }
      }
    } else {
      sweeps(lc, in, Cc.x, coarse_sweeps - 1);
      Scope sc = pc_scope(Cc);
      enter(sc);
      if (sc.active()) for (long i = sc.tid0(); i < Cc.n; i += sc.nth()) Cc.r[i] = Cc.x[i];
    }
    for (int l = lc - 1; l >= 0; l--) {
      const LevelDev<R> L = lev[l];
      const R *__restrict__ xc = lev[l + 1].r;
      Scope sl = pc_scope(L);
      const bool to_out = l == 0 && post == 1;
      enter(sl);
      if (sl.active() && (l == 0 || sl.nth() < 2L * L.n)) {
        // a thread per row: prolong in place (x += alpha x_c[parent], each row
        // its own), then the smoothing sweep gathers x directly -- two memory
        // latencies per slot round instead of three
        const long t0 = sl.tid0(), nt = sl.nth();
        for (long i = t0; i < L.n; i += nt) L.x[i] = L.x[i] + al(l) * xc[L.parent[i]];
        enter(sl);
        for (long i = t0; i < L.n; i += 2 * nt) {
          const long i2 = i + nt;
          const bool h2 = i2 < L.n;
          R t1 = 0., t2 = 0.;
          ell_acc2<6, false>(t1, t2, L.n, L.w, L.nbr, L.anb, i, i2, h2, [&](int k) { return L.x[k]; });
          R xi = L.x[i], bi = l == 0 ? (R)in[i] : L.b[i];
          R xn = xi + om(l) * (bi - L.ac[i] * xi - t1) / L.ac[i];
          if (to_out) out[i] = (double)xn; else L.r[i] = xn;
          if (h2) {
            R xj = L.x[i2], bj = l == 0 ? (R)in[i2] : L.b[i2];
            R xm = xj + om(l) * (bj - L.ac[i2] * xj - t2) / L.ac[i2];
            if (to_out) out[i2] = (double)xm; else L.r[i2] = xm;
          }
        }
      } else if (sl.active())
        level_rows(sl, L.n, l, [&](auto gg, long i, bool act, int q) {
          constexpr int G = decltype(gg)::value;
          R t = 0.;
          if (act)
            t = ell_part<G, G == 1 ? 8 : 4>(L.n, L.w, L.nbr, L.anb, i, q,
                                            [&](int k) { return L.x[k] + al(l) * xc[L.parent[k]]; });
          t = gsum<G>(t);
          if (act && q == 0) {
            R xi = L.x[i] + al(l) * xc[L.parent[i]];
            R bi = l == 0 ? (R)in[i] : L.b[i];
            R xn = xi + om(l) * (bi - L.ac[i] * xi - t) / L.ac[i];
            if (to_out) out[i] = (double)xn; else L.r[i] = xn;
          }
        });
      if (!to_out) sweeps(l, in, L.r, post - 1);
    }
    if (post > 1 || lc == 0) {   // a hierarchy of level 0 alone has no up leg that writes out
      enter(g);
      const LevelDev<R> L0 = lev[0];
      for (long i = g.tid0(); i < L0.n; i += g.nth()) out[i] = (double)L0.r[i];
    }
    enter(g);
  }

};

// ------------------------------------------------------------ V-cycle in one phase per level and leg
// One damped-Jacobi pre- and post-sweep per level and a dense coarsest solve,
// with the arithmetic and the order of every sum of PCycle::run():
//   down  the residual of each row of level l and its sum over the aggregates
//         in one phase: a CTA takes consecutive aggregates, whose rows are
//         consecutive too (levels >= 1 are renumbered aggregate by aggregate,
//         level 0 has a copy of the matrix in that order), so a block barrier
//         stands between the residuals and their sums instead of a grid barrier;
//   up    the post-sweep of a row, then its prolongation x += alpha x_row into
//         the consecutive rows of its aggregate on the finer level; level 0
//         forms x_0 + alpha x_1[parent] on the fly for a row and its neighbours.
// A level costs two grid barriers a cycle where separate residual,
// restriction, prolongation and sweep phases cost three to four, and the passes
// over the level that went with them.  What bounds a phase on a small level is
// the barrier (1.2 us) and its chain of dependent loads, on a large one DRAM.
// Separate phases (PCycle) take 1.65 times as long at 128^3 and 2.3 times at 124k
// cells (p' kernels, B200: 75.1 and 29.5 ms against 45.6 and 12.9, with level 0's
// neighbours from row patterns).  Tried and slower: a warp per chunk of aggregates with the
// residuals in its own shared array (a chain of six dependent loads per chunk:
// level 0 of 128^3 72 us against 63, level 1 54 against 19).
template <class R>
__device__ __forceinline__ VcDev<R> &vstate() {
  __shared__ VcDev<R> s;
  return s;
}
// the solve's arguments, for the phases
template <class R>
__device__ __forceinline__ AmgKArgs<R> &astate() {
  __shared__ AmgKArgs<R> s;
  return s;
}
template <class T>
__device__ __forceinline__ void copy_words(T &dst, const T &src) {
  for (int q = threadIdx.x; q < (int)(sizeof(T) / 4); q += blockDim.x) ((int32_t *)&dst)[q] = ((const int32_t *)&src)[q];
}

// Level 0's neighbour indices of a row, from the table (PAT false: slot u of row
// a at nbr[u n + a], loaded a row ahead) or from its pattern (a byte a row ahead,
// the offsets in shared memory)
__device__ __forceinline__ int32_t *pat_offs() {
  __shared__ __align__(16) int32_t s[FS_PAT_MAX * 8];
  return s;
}
template <bool PAT>
struct RowIdx;
template <>
struct RowIdx<false> {
  int k[6];
  __device__ __forceinline__ void load(const int32_t *__restrict__ nbr, const uint8_t *, int n, int w, long a, bool h) {
#pragma unroll
    for (int u = 0; u < 6; u++) k[u] = h && u < w ? __ldg(nbr + (long)u * n + a) : -1;
  }
  __device__ __forceinline__ void get(int (&o)[6], int, bool) const {
#pragma unroll
    for (int u = 0; u < 6; u++) o[u] = k[u];
  }
};
template <>
struct RowIdx<true> {
  int p;
  __device__ __forceinline__ void load(const int32_t *, const uint8_t *__restrict__ pat, int, int, long a, bool h) {
    p = h ? __ldg(pat + a) : 0;
  }
  __device__ __forceinline__ void get(int (&o)[6], int i, bool h) const {
    const int32_t *s = pat_offs() + 8 * p;
    const int4 q = *reinterpret_cast<const int4 *>(s);
    const int2 r = *reinterpret_cast<const int2 *>(s + 4);
    const int f[6] = {q.x, q.y, q.z, q.w, r.x, r.y};
#pragma unroll
    for (int u = 0; u < 6; u++) o[u] = h && f[u] != FS_PAT_NONE ? i + f[u] : -1;
  }
};

// log2 of the lanes per row of a level, from the threads that the cycle of PCycle gives it
// (pc_scope, level_rows): it fixes the order of a row's sum
__device__ __forceinline__ int vc_lanes(int n) {
  const long nth = (long)blockDim.x * (n > FS_PC_TEAM_MAX ? cta_count() : n > FS_PC_SMALL ? team_size() : 1);
  const long per = nth / (n > 0 ? n : 1);
  return per < 2 ? 0 : per < 4 ? 1 : per < 8 ? 2 : 3;
}

// lanes per row and this CTA's aggregates of every level: consecutive ones
// holding an equal share of the level's rows
template <class R>
__device__ __forceinline__ void vc_split() {
  VcDev<R> &V = vstate<R>();
  const int t = threadIdx.x;
  if (t <= V.lc) V.G[t] = vc_lanes(V.L[t].n);
  if (t < 2 * V.lc) {
    const int l = t >> 1, nc = V.L[l + 1].n;
    const long want = (long)V.L[l].n * (cta_id() + (t & 1)) / cta_count();
    int lo = 0, hi = nc;   // first aggregate whose rows start at or after `want`
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      if (V.L[l].kp[m] >= want) hi = m; else lo = m + 1;
    }
    if (t & 1) { V.p1[l] = lo; V.e1[l] = V.L[l].kp[lo]; }
    else { V.p0[l] = lo; V.e0[l] = V.L[l].kp[lo]; }
  }
}

// the grid's warps over the items of a phase
struct Warps {
  int w0, nw;
  // with items for every warp a CTA takes neighbouring ones; with fewer they
  // are spread over the CTAs
  __device__ Warps(int items) {
    const int wid = threadIdx.x >> 5, wpc = blockDim.x >> 5;
    nw = wpc * cta_count();
    w0 = items >= nw ? cta_id() * wpc + wid : wid * cta_count() + cta_id();
  }
};

// sum over the 2^g lanes of a row
template <class R>
__device__ __forceinline__ R lanes_sum(R v, int g) {
  for (int o = 1 << g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the down legs' residuals, one array for all of them
template <class R>
__device__ __forceinline__ R *vc_rows() {
  __shared__ R sh[FS_VC_ROWS];
  return sh;
}

// Sums of the residuals of the CTA's rows (rs, from row e0 of level l) over its
// aggregates: b of level l+1, and unless that is the coarsest its first sweep
// from zero x = omega b / ac.  2^gc lanes an aggregate; AggFirst: the thread's
// first aggregate, its rows and diagonal, loaded before the residuals were done.
template <class R>
struct AggFirst { int P, c0, c1; R d; };
template <class R>
__device__ __forceinline__ AggFirst<R> vc_agg(const VcDev<R> &V, int l, int gc, bool sweep, int P) {
  AggFirst<R> f{P, 0, 0, (R)1};
  if (P < V.p1[l]) {
    const int32_t *__restrict__ kp = V.L[l].kp;
    const int e0 = V.e0[l];
    f.c0 = __ldg(kp + P) - e0 + ((threadIdx.x & 31) & ((1 << gc) - 1));
    f.c1 = __ldg(kp + P + 1) - e0;
    if (sweep) f.d = __ldg(V.L[l + 1].ac + P);
  }
  return f;
}
template <class R>
__device__ __forceinline__ void vc_restrict(const VcDev<R> &V, int l, int gc, bool sweep, const R *rs, AggFirst<R> f) {
  const int lane = threadIdx.x & 31, P1 = V.p1[l], Gc = 1 << gc;
  while (f.P - (lane >> gc) < P1) {
    R s = (R)0;
    for (int c = f.c0; c < f.c1; c += 4 * Gc) {
      R v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = c + u * Gc < f.c1 ? rs[c + u * Gc] : (R)0;
#pragma unroll
      for (int u = 0; u < 4; u++) if (c + u * Gc < f.c1) s = s + v[u];
    }
    if (gc) s = lanes_sum(s, gc);
    if (f.P < P1 && (lane & (Gc - 1)) == 0) {
      V.L[l + 1].b[f.P] = s;
      if (sweep) V.L[l + 1].x[f.P] = (R)FS_MG_OMEGA * s / f.d;
    }
    f = vc_agg(V, l, gc, sweep, f.P + (int)(blockDim.x >> gc));
  }
}

// Down leg of level l >= 1.  A CTA takes the aggregates [p0, p1) and with them
// the consecutive rows [e0, e1): residuals first (2^g lanes a row), kept in
// shared memory or, when they do not fit, in the level's r, then behind a block
// barrier their sums.  Every phase ends with a grid barrier.  Lane counts are
// powers of two and kept as shifts, and a warp without rows goes straight to
// the barrier: on a small level the other warps' index arithmetic was most of
// the phase (32 warps a CTA share four issue slots).
template <class R>
__device__ __forceinline__ void vc_down(int l, int gc, bool sweep) {
  constexpr int U = 8;
  const VcDev<R> &V = vstate<R>();
  const VcLevel<R> &F = V.L[l];
  const int g = V.G[l], e0 = V.e0[l], e1 = V.e1[l], lane = threadIdx.x & 31;
  R *rs = e1 - e0 <= FS_VC_ROWS ? vc_rows<R>() : F.r + e0;
  int a0 = e0 + (int)((threadIdx.x & ~31u) >> g);   // the warp's first row
  const int P0 = V.p0[l] + (int)((threadIdx.x & ~31u) >> gc);
  const bool sums = P0 < V.p1[l];
  AggFirst<R> first{P0, 0, 0, (R)1};
  if (sums) first = vc_agg(V, l, gc, sweep, P0 + (lane >> gc));
  if (a0 < e1) {
    const int32_t *__restrict__ col = F.col;
    const R *__restrict__ val = F.val, *__restrict__ ac = F.ac;
    const R *x = F.x, *b = F.b;
    const int G = 1 << g, q = lane & (G - 1), w = F.w, rpp = (int)(blockDim.x >> g);
    for (; a0 < e1; a0 += rpp) {
      const int a = a0 + (lane >> g);
      const bool h = a < e1;
      const long p = ((long)(a >> 5) * w) * 32 + (a & 31);
      const R bi = h ? b[a] : (R)0, xi = h ? x[a] : (R)0, d = h ? __ldg(ac + a) : (R)0;
      R t = (R)0;
      for (int j0 = q; j0 < w; j0 += U * G) {
        int k[U];
        R c[U], y[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool in = h && j0 + u * G < w;
          k[u] = in ? __ldg(col + p + (long)(j0 + u * G) * 32) : -1;
          c[u] = in ? __ldg(val + p + (long)(j0 + u * G) * 32) : (R)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) y[u] = k[u] >= 0 ? x[k[u]] : (R)0;
#pragma unroll
        for (int u = 0; u < U; u++) t = t + c[u] * y[u];
      }
      if (g) t = lanes_sum(t, g);
      if (h && q == 0) rs[a - e0] = bi - d * xi - t;
    }
  }
  __syncthreads();
  if (sums) vc_restrict(V, l, gc, sweep, rs, first);
  grid_barrier();
}

// The same for level 0: b = in and x = x0 in mesh order, row a is cell cells[a],
// a thread per row.
template <class R, bool PAT>
__device__ __forceinline__ void vc_down_fine(int gc, const double *in, const R *x0) {
  constexpr int U = 6;
  const VcDev<R> &V = vstate<R>();
  R *sh = vc_rows<R>();
  const VcLevel<R> &F = V.L[0];
  const int e0 = V.e0[0], e1 = V.e1[0], n = F.n, w = F.w;
  const bool sweep = V.lc > 1;
  R *rs = e1 - e0 <= FS_VC_ROWS ? sh : F.r + e0;
  const int32_t *__restrict__ col = F.col, *__restrict__ cells = F.cells;
  const uint8_t *__restrict__ pat = V.patL;
  const R *__restrict__ val = F.val, *__restrict__ ac = F.ac;
  int a = e0 + (int)threadIdx.x, i = a < e1 ? __ldg(cells + a) : 0;
  RowIdx<PAT> ix;
  ix.load(col, pat, n, w, a, a < e1);
  const AggFirst<R> first = vc_agg(V, 0, gc, sweep, V.p0[0] + (int)(threadIdx.x >> gc));
  while (a < e1) {
    int k[U];
    R c[U], g[U];
    ix.get(k, i, true);
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = k[u] >= 0 ? __ldg(val + (long)u * n + a) : (R)0;
      g[u] = k[u] >= 0 ? x0[k[u]] : (R)0;
    }
    const R bi = (R)in[i], xi = x0[i], d = __ldg(ac + a);
    const int an = a + (int)blockDim.x;
    i = an < e1 ? __ldg(cells + an) : 0;
    ix.load(col, pat, n, w, an, an < e1);
    R t = (R)0;
#pragma unroll
    for (int u = 0; u < U; u++) t = t + c[u] * g[u];
    for (int j = U; j < w; j++) {
      const int kj = __ldg(col + (long)j * n + a);
      if (kj >= 0) t = t + __ldg(val + (long)j * n + a) * x0[kj];
    }
    rs[a - e0] = bi - d * xi - t;
    a = an;
  }
  __syncthreads();
  vc_restrict(V, 0, gc, sweep, rs, first);
  grid_barrier();
}

// post-sweep of level l's rows, then the prolongation into the finer level's x
// (level 1: the result goes to x1)
template <class R>
__device__ __forceinline__ void vc_up(int l) {
  constexpr int U = 8;
  const VcDev<R> &V = vstate<R>();
  const VcLevel<R> &L = V.L[l], &F = V.L[l - 1];
  const int g = V.G[l], n = L.n;
  const Warps w((n + (32 >> g) - 1) >> (5 - g));
  if (w.w0 << (5 - g) < n) {
    const int lane = threadIdx.x & 31, G = 1 << g, q = lane & (G - 1), wd = L.w;
    const int32_t *__restrict__ col = L.col, *__restrict__ kp = F.kp;
    const R *__restrict__ val = L.val, *__restrict__ ac = L.ac;
    const R *x = L.x, *b = L.b;
    R *xf = F.x, *x1 = V.x1;
    for (int s = w.w0; s << (5 - g) < n; s += w.nw) {
      const int i = (s << (5 - g)) + (lane >> g);
      const bool act = i < n;
      const long p = ((long)(i >> 5) * wd) * 32 + (i & 31);
      const R xi = act ? x[i] : (R)0, bi = act ? b[i] : (R)0, d = act ? __ldg(ac + i) : (R)1;
      int c = 0, c1 = 0;
      R f0 = (R)0, f1 = (R)0;
      if (l > 1 && act) {
        c = __ldg(kp + i) + q;
        c1 = __ldg(kp + i + 1);
        if (c < c1) f0 = xf[c];
        if (c + G < c1) f1 = xf[c + G];
      }
      R t = (R)0;
      for (int j0 = q; j0 < wd; j0 += U * G) {
        int k[U];
        R v[U], y[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool in = act && j0 + u * G < wd;
          k[u] = in ? __ldg(col + p + (long)(j0 + u * G) * 32) : -1;
          v[u] = in ? __ldg(val + p + (long)(j0 + u * G) * 32) : (R)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) y[u] = k[u] >= 0 ? x[k[u]] : (R)0;
#pragma unroll
        for (int u = 0; u < U; u++) t = t + v[u] * y[u];
      }
      if (g) t = lanes_sum(t, g);
      if (!act) continue;
      const R xn = xi + (R)FS_MG_OMEGA * (bi - d * xi - t) / d;
      if (l == 1) {
        if (q == 0) x1[i] = xn;
      } else {
        const R add = (R)FS_MG_ALPHA * xn;
        if (c < c1) xf[c] = f0 + add;
        if (c + G < c1) xf[c + G] = f1 + add;
        for (c += 2 * G; c < c1; c += G) xf[c] = xf[c] + add;
      }
    }
  }
  grid_barrier();
}

// the coarsest level by its dense inverse (a warp per row), prolonged into the
// next finer level, or left in x1 when that is level 0
template <class R>
__device__ __forceinline__ void vc_dense() {
  const VcDev<R> &V = vstate<R>();
  const VcLevel<R> &C = V.L[V.lc], &F = V.L[V.lc - 1];
  const double *__restrict__ sinv = V.sinv;
  const bool last = V.lc == 1;
  R *x1 = V.x1;
  const int lane = threadIdx.x & 31, n = C.n;
  const Warps w(n);
  const R *b = C.b;
  R *xf = F.x;
  for (int i = w.w0; i < n; i += w.nw) {
    double m[5], y[5];   // n <= FS_MG_DIRECT = 160
#pragma unroll
    for (int u = 0; u < 5; u++) {
      const int j = lane + 32 * u;
      m[u] = j < n ? __ldg(sinv + (long)i * n + j) : 0.;
      y[u] = j < n ? (double)b[j] : 0.;
    }
    double t = 0.;
#pragma unroll
    for (int u = 0; u < 5; u++) if (lane + 32 * u < n) t += m[u] * y[u];
    t = wsum(t);
    const R xn = (R)__shfl_sync(0xffffffffu, t, 0);
    if (last) {
      if (lane == 0) x1[i] = xn;
    } else {
      const R add = (R)FS_MG_ALPHA * xn;
      for (int c = __ldg(F.kp + i) + lane; c < __ldg(F.kp + i + 1); c += 32) xf[c] = xf[c] + add;
    }
  }
  grid_barrier();
}

// levels 1 and below: from b_1, x_1 to the corrected x_1 in V.x1.  GS: the
// restriction sums a coarse row's children in sequence.
template <class R, bool GS>
__device__ __forceinline__ void vcycle_coarse() {
  const VcDev<R> &V = vstate<R>();
  const int lc = V.lc;
  for (int l = 1; l < lc; l++) vc_down<R>(l, GS ? 0 : V.G[l + 1], l + 1 < lc);
  vc_dense<R>();
  for (int l = lc - 1; l >= 1; l--) vc_up<R>(l);
}

// level 0's post-sweep into out, with its correction formed on the fly
template <class R, bool PAT>
__device__ __forceinline__ void vc_up_fine(const double *in, double *out) {
  constexpr int U = 6;
  const VcDev<R> &V = vstate<R>();
  const LevelDev<R> &L = V.L0;
  const long nt = (long)cta_count() * blockDim.x;
  long i = (long)cta_id() * blockDim.x + threadIdx.x;
  const int n = L.n, w = L.w;
  const int32_t *__restrict__ nbr = L.nbr, *__restrict__ par = V.par0;
  const uint8_t *__restrict__ pat = V.pat;
  const R *__restrict__ anb = L.anb, *__restrict__ ac = L.ac;
  const R *x0 = L.x, *x1 = V.x1;
  const R al0 = (R)FS_MG_ALPHA0, om0 = (R)FS_MG_OMEGA0;
  RowIdx<PAT> ix;
  ix.load(nbr, pat, n, w, i, i < n);
  while (i < n) {
    R c[U], y[U], z[U];
    int k[U], q[U];
    ix.get(k, (int)i, true);
    const int qi = __ldg(par + i);
#pragma unroll
    for (int u = 0; u < U; u++) q[u] = k[u] >= 0 ? __ldg(par + k[u]) : 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = k[u] >= 0 ? __ldg(anb + (long)u * n + i) : (R)0;
      y[u] = k[u] >= 0 ? x0[k[u]] : (R)0;
    }
    const R aci = __ldg(ac + i), bi = (R)in[i], yi = x0[i], zi = x1[qi];
#pragma unroll
    for (int u = 0; u < U; u++) z[u] = k[u] >= 0 ? x1[q[u]] : (R)0;
    const long in1 = i + nt;
    ix.load(nbr, pat, n, w, in1, in1 < n);
    R t = (R)0;
#pragma unroll
    for (int u = 0; u < U; u++) t = t + c[u] * (y[u] + al0 * z[u]);
    for (int j = U; j < w; j++) {
      const int kj = __ldg(nbr + (long)j * n + i);
      if (kj >= 0) t = t + __ldg(anb + (long)j * n + i) * (x0[kj] + al0 * x1[__ldg(par + kj)]);
    }
    const R xi = yi + al0 * zi;
    out[i] = (double)(xi + om0 * (bi - aci * xi - t) / aci);
    i = in1;
  }
  grid_barrier();
}

// out = M^-1 in.  The caller has set x_0 = omega0 in / ac_0 and passed a grid
// barrier; ends with one.
template <class R>
__device__ __forceinline__ void vcycle(const double *in, double *out) {
  const VcDev<R> &V = vstate<R>();
  if (V.npat) vc_down_fine<R, true>(V.G[1], in, V.L0.x);
  else vc_down_fine<R, false>(V.G[1], in, V.L0.x);
  vcycle_coarse<R, false>();
  if (V.npat) vc_up_fine<R, true>(in, out);
  else vc_up_fine<R, false>(in, out);
}

// Level 0's rows of one colour (positions [q0, q1) of the colour lists) solved
// from their neighbours: (in - sum a x) / ac, the sum in slot order, two rows at
// a time.  xv(k): a neighbour's value; put(i, x): the row's.
template <class R, bool PAT, class XF, class PF>
__device__ __forceinline__ void gs_rows(const double *in, int q0, int q1, XF &&xv, PF &&put) {
  constexpr int U = 6;
  const VcDev<R> &V = vstate<R>();
  const LevelDev<R> &L = V.L0;
  const long nt = (long)cta_count() * blockDim.x;
  const int n = L.n, w = L.w;
  const int32_t *__restrict__ nbr = L.nbr, *__restrict__ list = L.color_rows;
  const uint8_t *__restrict__ pat = V.pat;
  const R *__restrict__ anb = L.anb, *__restrict__ ac = L.ac;
  for (long q = q0 + (long)cta_id() * blockDim.x + threadIdx.x; q < q1; q += 2 * nt) {
    const bool h = q + nt < q1;
    const int i = __ldg(list + q), j = h ? __ldg(list + q + nt) : i;
    RowIdx<PAT> ixi, ixj;
    ixi.load(nbr, pat, n, w, i, true);
    ixj.load(nbr, pat, n, w, j, h);
    int k[U], m[U];
    ixi.get(k, i, true);
    ixj.get(m, j, h);
    R a[U], b[U], x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      a[u] = k[u] >= 0 ? __ldg(anb + (long)u * n + i) : (R)0;
      b[u] = m[u] >= 0 ? __ldg(anb + (long)u * n + j) : (R)0;
      x[u] = k[u] >= 0 ? xv(k[u]) : (R)0;
      y[u] = m[u] >= 0 ? xv(m[u]) : (R)0;
    }
    const R bi = (R)in[i], bj = (R)in[j], di = __ldg(ac + i), dj = __ldg(ac + j);
    R t = (R)0, s = (R)0;
#pragma unroll
    for (int u = 0; u < U; u++) { t = t + a[u] * x[u]; s = s + b[u] * y[u]; }
    for (int v = U; v < w; v++) {
      const int ki = __ldg(nbr + (long)v * n + i), kj = h ? __ldg(nbr + (long)v * n + j) : -1;
      if (ki >= 0) t = t + __ldg(anb + (long)v * n + i) * xv(ki);
      if (kj >= 0) s = s + __ldg(anb + (long)v * n + j) * xv(kj);
    }
    put(i, (bi - t) / di);
    if (h) put(j, (bj - s) / dj);
  }
}

// The V-cycle with symmetric multicolour Gauss-Seidel smoothing on level 0 (a
// forward pass from zero before the restriction and, after the correction
// x += alpha x_1[parent], a backward pass, each colour a phase) and damped Jacobi
// on the others.  out = M^-1 in; callers have made `in` visible.
// The forward pass's first colour starts from zero, so its rows are in / ac and
// it shares a phase with clearing the others.  With two colours (hexahedral
// meshes) the correction is formed on the fly for the neighbours of the backward
// pass's first colour, whose own values it does not need, and the rows go to out
// as they are solved: five level-0 phases a cycle instead of eight
// (B200, 389k distorted cells, 90 iterations: 16.2 -> 14.8 ms).
template <class R, bool PAT>
__device__ __forceinline__ void vcycle_gs(const double *in, double *out) {
  const VcDev<R> &V = vstate<R>();
  const LevelDev<R> &L = V.L0;
  const long t0 = (long)cta_id() * blockDim.x + threadIdx.x, nt = (long)cta_count() * blockDim.x;
  R *x = L.x;
  const int32_t *cp = L.color_ptr;
  {
    const int c1 = cp[1];
    for (long q = t0; q < L.n; q += nt) {
      const int i = L.color_rows[q];
      x[i] = q < c1 ? (R)in[i] / L.ac[i] : (R)0.;
    }
  }
  grid_barrier();
  for (int c = 1; c < L.ncolors; c++) {
    gs_rows<R, PAT>(in, cp[c], cp[c + 1], [&](int k) { return x[k]; }, [&](int i, R v) { x[i] = v; });
    grid_barrier();
  }
  vc_down_fine<R, PAT>(0, in, x);
  vcycle_coarse<R, true>();
  const R al0 = (R)FS_MG_ALPHA0;
  const R *x1 = V.x1;
  const int32_t *__restrict__ par = V.par0;
  if (L.ncolors == 2) {
    gs_rows<R, PAT>(in, cp[1], cp[2], [&](int k) { return x[k] + al0 * x1[__ldg(par + k)]; },
                    [&](int i, R v) { x[i] = v; out[i] = (double)v; });
    grid_barrier();
    gs_rows<R, PAT>(in, 0, cp[1], [&](int k) { return x[k]; }, [&](int i, R v) { out[i] = (double)v; });
  } else {
    for (long i = t0; i < L.n; i += nt) x[i] = x[i] + al0 * x1[par[i]];
    for (int c = L.ncolors - 1; c >= 0; c--) {
      grid_barrier();
      gs_rows<R, PAT>(in, cp[c], cp[c + 1], [&](int k) { return x[k]; },
                      [&](int i, R v) { x[i] = v; out[i] = (double)v; });
    }
  }
  grid_barrier();
}

// apply the preconditioner: out (FP64) = M^-1 in (FP64), via the R-precision
// V-cycle.  MODE: 0 the V-cycle of PCycle::run(), 1 vcycle() (the caller has
// set x_0 = omega0 in / ac_0), 2 vcycle_gs()
template <class R, int MODE>
__device__ __forceinline__ void apply_prec(Sync &S, const double *in, double *out, unsigned &gen) {
  if (MODE == 1) vcycle<R>(in, out);
  else if (MODE == 2) {
    if (vstate<R>().npat) vcycle_gs<R, true>(in, out);
    else vcycle_gs<R, false>(in, out);
  }
  else {
    const AmgKArgs<R> &a = astate<R>();
    Scope all;
    all.grid = true;
    PCycle<R> C{S, a.lev, a.lc, a.direct != 0, a.sinv, a.pre, a.post, 20, (R)FS_MG_OMEGA, (R)FS_MG_ALPHA, all,
                (R)FS_MG_OMEGA0, (R)FS_MG_ALPHA0, a.teambar, a.status, gen, a.team_extra};
    C.run(in, out);
    gen = C.gen;
  }
}

// ------------------------------------------------------------ the passes of the Krylov iteration
// y = A x over the thread's rows in grid-stride order, with the products its
// sums need: (y.e, y.y, y.f) or (e.y) alone.  The next row's indices are loaded
// while a row gathers.  Every pass loads all it needs of a row before it
// stores, so the stores do not hold up the loads.
template <class R, int K, bool PAT>
__device__ __forceinline__ Sum3 krylov_ax_rows(const double *x, double *y, const double *e, const double *f) {
  constexpr int U = 6;
  const AmgKArgs<R> &A = astate<R>();
  const int n = A.N, w = A.W;
  const int32_t *__restrict__ nbr = A.cn;
  const double *__restrict__ anb = A.anb, *__restrict__ ac = A.ac;
  const long nt = (long)cta_count() * blockDim.x;
  long i = (long)cta_id() * blockDim.x + threadIdx.x;
  Sum3 s{0., 0., 0.};
  const uint8_t *__restrict__ pat = PAT ? vstate<R>().pat : nullptr;
  RowIdx<PAT> ix;
  ix.load(nbr, pat, n, w, i, i < n);
  while (i < n) {
    int k[U];
    double c[U], g[U];
    ix.get(k, (int)i, true);
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = k[u] >= 0 ? __ldg(anb + (long)u * n + i) : 0.;
      g[u] = k[u] >= 0 ? x[k[u]] : 0.;
    }
    const double aci = __ldg(ac + i), xi = x[i], ei = e[i], fi = K > 1 ? f[i] : 0.;
    const long in = i + nt;
    ix.load(nbr, pat, n, w, in, in < n);
    double t = aci * xi;
#pragma unroll
    for (int u = 0; u < U; u++) t = t + c[u] * g[u];
    for (int j = U; j < w; j++) {
      const int kj = __ldg(nbr + (long)j * n + i);
      if (kj >= 0) t = t + __ldg(anb + (long)j * n + i) * x[kj];
    }
    y[i] = t;
    s.a += t * ei;
    if (K > 1) { s.b += t * t; s.c += fi * t; }
    i = in;
  }
  return s;
}
template <class R, int MODE, int K>
__device__ __forceinline__ Sum3 krylov_ax(const double *x, double *y, const double *e, const double *f) {
  if (MODE != 0 && vstate<R>().npat) return krylov_ax_rows<R, K, true>(x, y, e, f);
  return krylov_ax_rows<R, K, false>(x, y, e, f);
}

// s = r - alpha v with |s|^2 and r0.s, and x_0 = omega0 s / ac_0 of the V-cycle
template <class R, int MODE>
__device__ __forceinline__ Sum3 krylov_s(double alpha) {
  const AmgKArgs<R> &A = astate<R>();
  const int n = A.N;
  const long nt = (long)cta_count() * blockDim.x;
  const double *r = A.r, *v = A.v, *r0 = A.r0;
  const R *__restrict__ ac0 = A.lev[0].ac;
  double *s = A.s;
  R *x0 = A.lev[0].x;
  const R om0 = (R)FS_MG_OMEGA0;
  Sum3 o{0., 0., 0.};
  for (long i = (long)cta_id() * blockDim.x + threadIdx.x; i < n; i += 2 * nt) {
    const long j = i + nt;
    const bool h = j < n;
    const double r1 = r[i], v1 = v[i], q1 = r0[i], r2 = h ? r[j] : 0., v2 = h ? v[j] : 0., q2 = h ? r0[j] : 0.;
    const R d1 = MODE == 1 ? __ldg(ac0 + i) : (R)1, d2 = MODE == 1 && h ? __ldg(ac0 + j) : (R)1;
    const double s1 = r1 - alpha * v1, s2 = r2 - alpha * v2;
    s[i] = s1;
    o.a += s1 * s1;
    o.b += q1 * s1;
    if (MODE == 1) x0[i] = om0 * (R)s1 / d1;
    if (h) {
      s[j] = s2;
      o.a += s2 * s2;
      o.b += q2 * s2;
      if (MODE == 1) x0[j] = om0 * (R)s2 / d2;
    }
  }
  return o;
}

// x += alpha y + omega z, r = s - omega t, and p = r + beta (p - omega v) of the
// next iteration with x_0 = omega0 p / ac_0
template <class R, int MODE>
__device__ __forceinline__ void krylov_xrp(double alpha, double omega, double beta) {
  const AmgKArgs<R> &A = astate<R>();
  const int n = A.N;
  const long nt = (long)cta_count() * blockDim.x;
  const double *y = A.y, *z = A.z, *s = A.s, *t = A.t, *v = A.v;
  double *x = A.x, *r = A.r, *p = A.p;
  const R *__restrict__ ac0 = A.lev[0].ac;
  R *x0 = A.lev[0].x;
  const R om0 = (R)FS_MG_OMEGA0;
  for (long i = (long)cta_id() * blockDim.x + threadIdx.x; i < n; i += 2 * nt) {
    const long j = i + nt;
    const bool h = j < n;
    double x1 = x[i], y1 = y[i], z1 = z[i], s1 = s[i], t1 = t[i], p1 = p[i], v1 = v[i];
    double x2 = 0., y2 = 0., z2 = 0., s2 = 0., t2 = 0., p2 = 0., v2 = 0.;
    if (h) { x2 = x[j]; y2 = y[j]; z2 = z[j]; s2 = s[j]; t2 = t[j]; p2 = p[j]; v2 = v[j]; }
    const R d1 = MODE == 1 ? __ldg(ac0 + i) : (R)1, d2 = MODE == 1 && h ? __ldg(ac0 + j) : (R)1;
    x[i] = x1 + alpha * y1 + omega * z1;
    const double r1 = s1 - omega * t1;
    r[i] = r1;
    const double n1 = r1 + beta * (p1 - omega * v1);
    p[i] = n1;
    if (MODE == 1) x0[i] = om0 * (R)n1 / d1;
    if (h) {
      x[j] = x2 + alpha * y2 + omega * z2;
      const double r2 = s2 - omega * t2;
      r[j] = r2;
      const double n2 = r2 + beta * (p2 - omega * v2);
      p[j] = n2;
      if (MODE == 1) x0[j] = om0 * (R)n2 / d2;
    }
  }
  grid_barrier();
}

// mean of the right-hand side of a pure-Neumann system (every row sums to
// zero), else 0; the same grid-deterministic sums in every kernel that calls it
template <class R>
__device__ double rhs_mean(Sync &S, const AmgKArgs<R> &a) {
  const int N = a.N;
  const long t0 = (long)cta_id() * blockDim.x + threadIdx.x, nt = (long)cta_count() * blockDim.x;
  double nonsing = 0., bsum = 0.;
  for (long i = t0; i < N; i += nt) {
    double rs = a.ac[i];
    for (int j = 0; j < a.W; j++)
      if (a.cn[(long)j * N + i] >= 0) rs += a.anb[(long)j * N + i];
    nonsing += fabs(rs) > 1e-9 * fabs(a.ac[i]) ? 1. : 0.;
    bsum += a.bc[i];
  }
  double n_nonsing, b_total;
  S.sum2(nonsing, bsum, n_nonsing, b_total);
  return n_nonsing == 0. ? b_total / N : 0.;
}

// The initial guess of k_amg_bicgstab, one cooperative launch before it: the
// combination x = sum_j c_j x_j of the basis vectors (previous p' solutions,
// the network's guess) that minimises |b - A x|, least squares over their
// span, so |b - A x| <= |b|.  The normal equations (Gram matrix of the A x_j)
// are solved by every CTA alike from grid-deterministic sums, by a Cholesky
// factorisation with a relative diagonal shift.  x goes to a.x and fit[0] = 1;
// a failed factorisation leaves fit[0] = 0 (the solve starts from zero).
template <class R, int NX>
__device__ __forceinline__ void guess_fit_body(const AmgKArgs<R> a) {
  constexpr int NG = NX * (NX + 1) / 2, K = NG + NX + 1;
  Sync S(a.part, a.gridbar + FS_GRIDBAR_FIT, a.status, a.team_extra, a.spin_limit);
  const double bmean = rhs_mean(S, a);
  double c[NX];
  bool fell_back;
  const int N = a.N, W = a.W;
  const long t0 = (long)cta_id() * blockDim.x + threadIdx.x, nt = (long)cta_count() * blockDim.x;
  const double *xs[NX];
#pragma unroll
  for (int j = 0; j < NX; j++) xs[j] = a.xs[j];
  // Gram matrix G_jk = (A x_j).(A x_k) (upper triangle), g_j = (A x_j).b, |b|^2;
  // each row of A is read once for all basis vectors, its slots in order
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; k++) acc[k] = 0.;
  for (long i = t0; i < N; i += nt) {
    double y[NX];
    const double aci = a.ac[i];
#pragma unroll
    for (int j = 0; j < NX; j++) { double t = 0.; t = t + aci * xs[j][i]; y[j] = t; }
    for (int w0 = 0; w0 < W; w0 += 4) {
      int kk[4];
      double av[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const bool in = w0 + u < W;
        kk[u] = in ? a.cn[(long)(w0 + u) * N + i] : -1;
        av[u] = in ? a.anb[(long)(w0 + u) * N + i] : 0.;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (kk[u] >= 0)
#pragma unroll
          for (int j = 0; j < NX; j++) y[j] = y[j] + av[u] * xs[j][kk[u]];
    }
    const double b1 = a.bc[i] - bmean;
    int q = 0;
#pragma unroll
    for (int j = 0; j < NX; j++)
#pragma unroll
      for (int k = j; k < NX; k++) acc[q++] += y[j] * y[k];
#pragma unroll
    for (int j = 0; j < NX; j++) acc[NG + j] += y[j] * b1;
    acc[NG + NX] += b1 * b1;
  }
  double tot[K];
  S.sumKt<K>(acc, tot);
  // Cholesky of G + 1e-12 max(diag) I, then the two triangular solves (row-major L)
  double L[NX][NX];
  double dmax = 0.;
  {
    int q = 0;
#pragma unroll
    for (int j = 0; j < NX; j++)
#pragma unroll
      for (int k = j; k < NX; k++) { L[k][j] = tot[q]; if (k == j) dmax = fmax(dmax, tot[q]); q++; }
  }
  bool ok = dmax > 0. && isfinite(dmax);
#pragma unroll
  for (int j = 0; j < NX; j++) {
    if (!ok) break;
    double d = L[j][j] + 1e-12 * dmax;
    for (int k = 0; k < j; k++) d -= L[j][k] * L[j][k];
    if (!(d > 1e-14 * dmax)) { ok = false; break; }
    d = sqrt(d);
    L[j][j] = d;
#pragma unroll
    for (int r = j + 1; r < NX; r++) {
      double v = L[r][j];
      for (int k = 0; k < j; k++) v -= L[r][k] * L[j][k];
      L[r][j] = v / d;
    }
  }
  if (ok) {
    double z[NX];
#pragma unroll
    for (int j = 0; j < NX; j++) {
      double v = tot[NG + j];
      for (int k = 0; k < j; k++) v -= L[j][k] * z[k];
      z[j] = v / L[j][j];
    }
#pragma unroll
    for (int j = NX - 1; j >= 0; j--) {
      double v = z[j];
      for (int k = j + 1; k < NX; k++) v -= L[k][j] * c[k];
      c[j] = v / L[j][j];
    }
#pragma unroll
    for (int j = 0; j < NX; j++) if (!isfinite(c[j])) ok = false;
  }
  if (!ok)
#pragma unroll
    for (int j = 0; j < NX; j++) c[j] = 0.;
  fell_back = !ok;
  for (long i = t0; i < N; i += nt) {
    double xi = 0.;
#pragma unroll
    for (int j = 0; j < NX; j++) xi += c[j] * xs[j][i];
    a.x[i] = xi;
  }
  if (cta_id() == 0 && threadIdx.x == 0) {
    a.fit[0] = fell_back ? 0 : 1;
    if (a.nncnt) { a.nncnt[1] += 1; if (fell_back) a.nncnt[0] += 1; }
  }
}


// right-preconditioned BiCGSTAB (van der Vorst 1992) with a multigrid V-cycle:
// MODE 0 PCycle::run(), 2 vcycle_gs() (multicolour Gauss-Seidel smoothing), 1
// vcycle() (one pre- and one post-sweep, dense coarsest level), whose first
// sweep from zero, x_0 = omega0 in / ac_0, rides on the loops that form p and s.
// Four grid synchronisations per iteration besides the V-cycles': the sums
// after v = A y and after s, the sums after t = A z, and the barrier after one
// pass that updates x and r and forms the next p.  That pass needs beta
// before |r|^2 and r0.r of the new r are summed; both come from the t-pass
// sums instead: r0.r_new = r0.s - omega r0.t, and |s - omega t|^2 = |s|^2 -
// omega t.s (omega = t.s / t.t), with |s|^2 summed fresh from s, so the
// estimate's rounding is relative to |s|^2 of this iteration.  Only an
// iteration whose estimate says it has converged (or the last one) sums |r|^2
// and r0.r of the stored r instead, so the exit is always decided on a
// residual summed from its vector, and a solve that has not really converged
// continues with p formed in a separate pass.
struct KrylovState {
  double alpha, omega, rho, rho_next, ss, r0s, resn, normb;
  int k;
  bool p_ready;
};
template <class R, int MODE>
__device__ __forceinline__ void amg_bicgstab_body(const AmgKArgs<R> &ap) {
  copy_words(astate<R>(), ap);
  if (MODE != 0) copy_words(vstate<R>(), *ap.vc);
  __syncthreads();
  if (MODE != 0) {
    vc_split<R>();
    for (int q = threadIdx.x; q < 8 * vstate<R>().npat; q += blockDim.x) pat_offs()[q] = vstate<R>().offs[q];
  }
  const AmgKArgs<R> &a = astate<R>();
  Sync S(a.part, a.gridbar, a.status, a.team_extra, a.spin_limit);
  unsigned gen = 0;   // team-barrier generation (the counters are zeroed before the launch)
  const int N = a.N;
  Scope g; g.grid = true;
  const long t0 = g.tid0(), nt = g.nth();
  R *__restrict__ x0v = a.lev[0].x;
  const R *__restrict__ ac0 = a.lev[0].ac;
  const R om0 = (R)FS_MG_OMEGA0;
  // start from the initial guess k_guess_fit left in x (the least-squares
  // combination of the basis vectors; fit[0] = 0 when it fell back), or from zero.
  // A pure-Neumann system (every row sums to zero: the closed-cavity p'
  // system) is singular.  Its right-hand side is taken with its mean removed,
  // the part a solution can match; otherwise, once the outer iterations have
  // converged the mean (rounding in the mass fluxes) is no longer small
  // against |b|, the tolerance cannot be met and the iterates drift.  The
  // constant null vector is left to the caller (pressure reference cell).
  const double bmean = rhs_mean(S, a);
  const bool has_x = a.nx > 0 && a.fit[0] != 0;
  double l0 = 0., l1 = 0.;
  for (long i = t0; i < N; i += nt) {
    const double b1 = a.bc[i] - bmean;
    double ri = b1;
    if (has_x) {
      double t = 0.;
      t = t + a.ac[i] * a.x[i];
      t = ell_acc<8, false>(t, a.N, a.W, a.cn, a.anb, i, [&](int k) { return a.x[k]; });
      ri = ri - t;
    } else {
      a.x[i] = 0.;
    }
    // the first p is r (beta's factors are 1 and p = v = 0 before it)
    a.r[i] = ri; a.r0[i] = ri; a.p[i] = ri; a.v[i] = 0.;
    if (MODE == 1) x0v[i] = om0 * (R)ri / ac0[i];
    l0 += ri * ri;
    l1 += b1 * b1;
  }
  double rr, bb;
  S.sum2(l0, l1, rr, bb);
  // rho = r0 . r of the iteration; rho_next that of the next one, summed from
  // the stored r when p still has to be formed (p_ready false).  Thread 0
  // writes, everyone reads behind a barrier.
  __shared__ KrylovState K;
  if (threadIdx.x == 0) {
    K.normb = sqrt(bb); K.resn = sqrt(rr); K.alpha = K.omega = 1.; K.rho = K.rho_next = rr; K.k = 0;
    // rr = 0 or not finite: the loop's breakdown test takes it
    K.p_ready = rr != 0. && isfinite(rr);
  }
  __syncthreads();
  while (K.k < a.maxit && K.resn > a.tol * K.normb && K.normb > 0.) {
    if (!K.p_ready) {
      const double rho1 = K.rho_next;
      // breakdown (r0 . r vanished: r at round-off): keep x.  Every CTA holds
      // the same sums, so every CTA takes the same branch.
      if (!(rho1 != 0.) || !isfinite(rho1)) {
        __syncthreads();
        if (threadIdx.x == 0) K.k++;
        break;
      }
      const double beta = (rho1 / K.rho) * (K.alpha / K.omega), omega = K.omega;
      for (long i = t0; i < N; i += nt) {
        const double pi = a.r[i] + beta * (a.p[i] - omega * a.v[i]);
        a.p[i] = pi;
        if (MODE == 1) a.lev[0].x[i] = om0 * (R)pi / a.lev[0].ac[i];
      }
      S.all();
      if (threadIdx.x == 0) K.rho = rho1;
    }
    __syncthreads();
    if (threadIdx.x == 0) { K.k++; K.p_ready = false; }
    apply_prec<R, MODE>(S, a.p, a.y, gen);                          // y = M^-1 p
    const double rv = grid_sums<1>(krylov_ax<R, MODE, 1>(a.y, a.v, a.r0, nullptr)).a;   // v = A y
    if (!(rv != 0.) || !isfinite(K.rho / rv)) break;
    {
      const double alpha = K.rho / rv;
      if (threadIdx.x == 0) K.alpha = alpha;
      const Sum3 sq = grid_sums<2>(krylov_s<R, MODE>(alpha));
      if (threadIdx.x == 0) { K.ss = sq.a; K.r0s = sq.b; }
      if (sqrt(sq.a) <= a.tol * K.normb) {
        for (long i = t0; i < N; i += nt) a.x[i] = a.x[i] + alpha * a.y[i];
        if (threadIdx.x == 0) K.resn = sqrt(sq.a);
        break;
      }
    }
    apply_prec<R, MODE>(S, a.s, a.z, gen);                          // z = M^-1 s
    const Sum3 tq = grid_sums<3>(krylov_ax<R, MODE, 3>(a.z, a.t, a.s, a.r0));   // t = A z
    const double ts = tq.a, tt = tq.b, alpha = K.alpha;
    if (!(tt > 0.) || !(ts != 0.) || !isfinite(ts / tt)) {
      // t = A z vanished or is orthogonal to s: take the half step and stop
      for (long i = t0; i < N; i += nt) a.x[i] = a.x[i] + alpha * a.y[i];
      if (threadIdx.x == 0) K.resn = sqrt(K.ss);
      break;
    }
    const double omega = ts / tt;
    const double rn_est = fmax(K.ss - omega * ts, 0.);
    const double rho_est = K.r0s - omega * tq.c;
    if (K.k < a.maxit && sqrt(rn_est) > a.tol * K.normb && rho_est != 0. && isfinite(rho_est)) {
      // x and r of this iteration and p of the next in one pass
      krylov_xrp<R, MODE>(alpha, omega, (rho_est / K.rho) * (alpha / omega));
      if (threadIdx.x == 0) { K.omega = omega; K.rho = rho_est; K.resn = sqrt(rn_est); K.p_ready = true; }
    } else {
      l0 = 0.; l1 = 0.;
      for (long i = t0; i < N; i += nt) {
        a.x[i] = a.x[i] + alpha * a.y[i] + omega * a.z[i];
        const double ri = a.s[i] - omega * a.t[i];
        a.r[i] = ri;
        l0 += ri * ri;
        l1 += a.r0[i] * ri;
      }
      double rn, r0r;
      S.sum2(l0, l1, rn, r0r);
      if (threadIdx.x == 0) { K.omega = omega; K.rho_next = r0r; K.resn = sqrt(rn); }
    }
    __syncthreads();
  }
  __syncthreads();
  S.all();
  for (long i = t0; i < N; i += nt) a.dphi[i] = a.x[i];
  if (cta_id() == 0 && threadIdx.x == 0) { *a.iters = K.k; a.diag[0] = K.resn; a.diag[1] = K.normb; }
}
