// The resident engine: one LP per thread-block cluster, on chip.
//
// A PDHG iteration of a small LP is bound by latency, not by bytes: the team
// engine (engine.cu) meets two L2 barriers per iteration, re-stages the tiles
// and gathers the other side's direction from L2, 12 to 20 us for an LP whose
// matrix would stream in 0.1 us.  Here an LP whose matrix and vectors fit the
// shared memory of a cluster of 1 to 16 SMs is stepped by that cluster alone:
//   * each CTA holds a contiguous share of the LP's row tiles and of its column
//     tiles (values, 16-bit indices, pointers, and the vectors of their rows)
//     and a whole copy of the two direction vectors dx and dy;
//   * a pass takes the products of the CTA's entries, one after another over
//     its threads, adds each row, and writes its part of the direction into
//     every CTA's copy (distributed shared memory);
//   * a cluster barrier (hardware) ends the pass;
//   * the line search's sums travel as tile partials in the same way; every
//     thread adds them and advances its own copy of the state (RunState), so no
//     pass of an iteration or line search touches global memory.
// The other modes (set-up, checks, restarts, final pass) run the generic tile
// code of engine_passes.cuh on the slot's arrays, the cluster's warps sharing
// the tiles, with the same barrier.  A run of iterations between two of them
// loads the resident data from the arena (9 us) and writes the vectors back.
//
// Measured on B200, alone, us per iteration with set-up and checks, team engine
// against this one: 3 x 5 (704 iterations) 11.2 / 4.4, 230 x 2,025 (448) 17.6 / 6.9,
// 347 x 2,776 (1,024) 16.7 / 6.6.  By clock stamps of an earlier build of the same
// loop an iteration of 230 x 2,025 on eight SMs takes 7,500 cycles: 1,200 products
// (bound by bank conflicts of the scattered 8-byte reads), 3,300 row sums and
// steps (a chain of dependent float64 adds and a division per row), 1,600
// barriers with the remote stores they wait for, 950 the line search's share; a
// generic step takes about 20 us, and a solve of 448 iterations has about 54 of
// them.  At 16 SMs the products shrink and nothing else does.
//
// Row sums, element-wise steps, tile partials and reduction trees are those of
// engine_passes.cuh, operand for operand, so every LP's bits are the same in
// either engine, whatever the cluster size.
#pragma once

#include "engine_passes.cuh"

namespace pdlp {

constexpr int kResWarps = 12;
constexpr int kResThreads = 32 * kResWarps;
constexpr int kResSmem = 227 * 1024;           // dynamic shared memory of a CTA
constexpr int kResMaxCluster = 16;

// The CTA's fixed area: the block flags, the LP's descriptor and state, and a
// copy of the scheduling fields per warp for the generic passes.
struct __align__(16) ResHeader {
  int flags[4];            // block_flags()
  int failed[2];           // rank 0's view of the launch's error word, by generic step
  int bad;                 // bounds-checked builds: a check of some CTA's resident data failed
  int pad;
  Inst inst;
  State st;
  TeamCopy team[kResWarps];
};

static_assert((sizeof(ResHeader) + 15) / 16 * 16 + kResWarps * sizeof(WarpSmem) <= kResSmem,
              "the generic passes' areas fit beside the header");

// Byte offsets of the resident data after the header.  They are the same in
// every CTA of the cluster (sized by the largest share), so that a local
// address maps to the same array in a peer.
struct ResLayout {
  int dx, dy, part, prod, rv, cv, rval, cval, rptr, cptr, rtile, ctile, ridx, cidx, bytes;
  int rrows, crows;        // capacity in rows of one row-side / column-side vector
};

// The largest share of one side over the CTAs of a cluster.
struct ResShare {
  int tiles, rows, nnz;
};

// What one cluster of a launch steps.
struct ResidentLP {
  int inst;
  int budget;              // steps it may run in this launch
  ResShare r, c;
};

__host__ __device__ inline int res_up16(int v) { return (v + 15) & ~15; }

__host__ __device__ inline ResLayout res_layout(int m, int n, int tiles, ResShare r, ResShare c,
                                                int word) {
  ResLayout l;
  int o = res_up16((int)sizeof(ResHeader));
  auto take = [&](long long bytes) {
    const int at = o;
    // far past any CTA's memory: too big, without overflowing
    o = bytes > (1 << 28) || o > (1 << 28) ? (1 << 29) : o + res_up16((int)bytes);
    return at;
  };
  l.rrows = r.rows;
  l.crows = c.rows;
  l.dx = take((long long)n * word);
  l.dy = take((long long)m * word);
  l.part = take(16LL * tiles);
  l.prod = take((long long)(r.nnz > c.nnz ? r.nnz : c.nnz) * word);
  l.rv = take(56LL * r.rows);
  l.cv = take(56LL * c.rows);
  l.rval = take((long long)r.nnz * word);
  l.cval = take((long long)c.nnz * word);
  l.rptr = take(4LL * (r.rows + 1));
  l.cptr = take(4LL * (c.rows + 1));
  l.rtile = take(8LL * r.tiles);
  l.ctile = take(8LL * c.tiles);
  l.ridx = take(2LL * r.nnz);
  l.cidx = take(2LL * c.nnz);
  l.bytes = o;
  return l;
}

// The tiles of CTA `rank` of `size`: an even split by count.
__host__ __device__ inline int res_first(int tiles, int rank, int size) {
  return (int)((long long)tiles * rank / size);
}

// ---- cluster primitives ------------------------------------------------------

__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}

__device__ __forceinline__ int cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return (int)r;
}

// Every thread of the cluster; orders their shared-memory writes, remote ones
// included, before the others' reads.
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same for global memory: the generic passes' stores and the bulk copies
// and L1 gathers of the pass that follows.
__device__ __forceinline__ void cluster_sync_global(int lane) {
  __threadfence();
  cluster_sync();
  __threadfence();
  if (lane == 0) fence_proxy_async_global();
}

// v into the same shared-memory word of every CTA of the cluster.
__device__ __forceinline__ void cluster_put(double* p, double v, int size) {
  const unsigned a = smem_addr(p);
  for (int r = 0; r < size; ++r) {
    unsigned ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
  }
}
__device__ __forceinline__ void cluster_put(float* p, float v, int size) {
  const unsigned a = smem_addr(p);
  for (int r = 0; r < size; ++r) {
    unsigned ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
  }
}

__device__ __forceinline__ void cluster_put(int* p, int v, int size) {
  const unsigned a = smem_addr(p);
  for (int r = 0; r < size; ++r) {
    unsigned ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
  }
}

__device__ __forceinline__ void mbar_inval(unsigned long long* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ double res_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float res_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double res_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float res_add(float a, float b) { return __fadd_rn(a, b); }

// ---- a pass ------------------------------------------------------------------

// The products of the CTA's entries, one after another over its threads:
// rounded, as gather_products leaves them.
template <typename T>
__device__ __forceinline__ void res_products(const T* __restrict__ val,
                                             const uint16_t* __restrict__ idx,
                                             const T* __restrict__ x, T* __restrict__ prod,
                                             int entries) {
  constexpr int kU = 4;
  int q = threadIdx.x;
  for (; q + (kU - 1) * kResThreads < entries; q += kU * kResThreads) {
    T v[kU], g[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      v[u] = val[q + u * kResThreads];
      g[u] = x[idx[q + u * kResThreads]];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) prod[q + u * kResThreads] = res_mul(v[u], g[u]);
  }
  for (; q < entries; q += kResThreads) prod[q] = res_mul(val[q], x[idx[q]]);
}

// One lane's part of a row: products q, q + L, ... below e, added in order
// (staged_row_sums' order).
template <typename T>
__device__ __forceinline__ T res_sum(const T* __restrict__ prod, int q, int e, int L) {
  T a = T(0);
  for (; q + 7 * L < e; q += 8 * L) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = prod[q + u * L];
#pragma unroll
    for (int u = 0; u < 8; ++u) a = res_add(a, v[u]);
  }
  if (q + 3 * L < e) {
    T v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = prod[q + u * L];
#pragma unroll
    for (int u = 0; u < 4; ++u) a = res_add(a, v[u]);
    q += 4 * L;
  }
  if (q + L < e) {
    const T v0 = prod[q], v1 = prod[q + L];
    a = res_add(res_add(a, v0), v1);
    q += 2 * L;
  }
  if (q < e) a = res_add(a, prod[q]);
  return a;
}

// ---- the sums of a line search ------------------------------------------------

// The instance's two sums from its tiles' partials, by every warp for itself,
// in warp_finish's order: groups of 64 tiles, then the groups.
__device__ __forceinline__ void res_total(const double* part, int tiles, double* s0, double* s1,
                                          int lane) {
  const int groups = (tiles + kGroupTiles - 1) / kGroupTiles;
  double t0 = 0.0, t1 = 0.0;                   // lane l: groups l, l + 32, ...
  for (int g = 0; g < groups; ++g) {
    double a = 0.0, b = 0.0;
    const int end = min(tiles, (g + 1) * kGroupTiles);
    for (int t = g * kGroupTiles + lane; t < end; t += 32) {
      a += part[2 * t];
      b += part[2 * t + 1];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a += __shfl_xor_sync(kFull, a, off);
      b += __shfl_xor_sync(kFull, b, off);
    }
    if (groups == 1) {
      t0 = a;
      t1 = b;
    } else if ((g & 31) == lane) {
      t0 += a;
      t1 += b;
    }
  }
  if (groups > 1) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      t0 += __shfl_xor_sync(kFull, t0, off);
      t1 += __shfl_xor_sync(kFull, t1, off);
    }
  }
  *s0 = t0;
  *s1 = t1;
}

// The fields of the State that iterations and line searches change, in every
// thread's registers; a run writes them back at its end.
struct RunState {
  double eta, omega, dxdx, sum_eta;
  long long k, attempts;
  int done, rejected;                // iterations and rejected trials of this run
  int kc, ks;                        // k modulo check_every, stepsize_every
  int rmode, cmode, cprimal, xcommit, ycommit, trials;
  int final_status;                  // a final pass was scheduled with this status, or -1
};

__device__ __forceinline__ RunState run_load(const State& s, const Inst& I) {
  RunState c;
  c.eta = s.eta;
  c.omega = s.omega;
  c.dxdx = s.dxdx;
  c.sum_eta = s.sum_eta;
  c.k = s.k;
  c.attempts = s.attempts;
  c.done = 0;
  c.rejected = 0;
  c.kc = (int)(s.k % I.check_every);
  c.ks = (int)(s.k % I.stepsize_every);
  c.rmode = s.rmode;
  c.cmode = s.cmode;
  c.cprimal = s.cprimal;
  c.xcommit = s.xcommit;
  c.ycommit = s.ycommit;
  c.trials = s.trials;
  c.final_status = -1;
  return c;
}

__device__ void run_store(const RunState& c, State* S) {
  S->eta = c.eta;
  S->dxdx = c.dxdx;
  S->sum_eta = c.sum_eta;
  S->k = c.k;
  S->epoch += c.done;
  S->iters_done += c.done;
  S->attempts = c.attempts;
  S->rejected += c.rejected;
  S->rmode = c.rmode;
  S->cmode = c.cmode;
  S->cprimal = c.cprimal;
  S->xcommit = c.xcommit;
  S->ycommit = c.ycommit;
  S->trials = c.trials;
  if (c.final_status >= 0) schedule_final(S, c.final_status, 0);
}

// plan_primal(k + 1)
__device__ __forceinline__ int run_plan(const RunState& c, const Inst& I) {
  const int kc = c.kc + 1 == I.check_every ? 0 : c.kc + 1;
  const int ks = c.ks + 1 == I.stepsize_every ? 0 : c.ks + 1;
  if (kc == 0 || c.k + 1 >= I.max_iter) return P_NONE;
  return ks == 0 ? P_TRIAL : P_NORMAL;
}

// r_finish of a trial.
__device__ __forceinline__ void run_trial(RunState& c, const Inst& I, double dyadx, double dydy) {
  c.attempts += 1;
  c.trials += 1;
  double eta_new;
  const bool accepted = step_test(c.eta, c.omega, c.dxdx, dyadx, dydy, c.attempts, &eta_new);
  c.eta = eta_new;
  c.ycommit = 0;
  if (accepted) {
    c.trials = 0;
    c.ycommit = 1;
    c.xcommit = 1;
    c.cprimal = run_plan(c, I);
    c.cmode = C_ITER;
  } else {
    c.rejected += 1;
    if (c.trials >= kMaxLineSearch) {
      c.cmode = C_NONE;
      c.rmode = R_FINAL;
      c.final_status = PDLP_STATUS_NUMERICAL;
    } else {
      c.cprimal = P_TRIAL;
      c.cmode = C_PRIMAL;
    }
  }
}

// c_finish of an iteration or a primal step.
__device__ __forceinline__ void run_advance(RunState& c, const Inst& I, double dxdx) {
  const int kind = c.cprimal;
  if (c.cmode == C_ITER) {
    c.xcommit = 0;
    c.sum_eta += c.eta;
    c.k += 1;
    c.done += 1;
    c.kc = c.kc + 1 == I.check_every ? 0 : c.kc + 1;
    c.ks = c.ks + 1 == I.stepsize_every ? 0 : c.ks + 1;
    if (kind == P_NONE) {
      if (c.kc == 0) {
        c.rmode = R_CHECK_A;
        c.cmode = C_CHECK_A;
      } else {
        c.cmode = C_NONE;
        c.rmode = R_FINAL;
        c.final_status = PDLP_STATUS_ITERATION_LIMIT;
      }
      return;
    }
  }
  if (kind == P_TRIAL) {
    c.dxdx = dxdx;
    c.rmode = R_TRIAL;
    c.cmode = C_NONE;
  } else {
    c.cprimal = run_plan(c, I);
    c.rmode = R_ITER;
    c.cmode = C_ITER;
  }
}

// Modes that run on chip.
__device__ __forceinline__ bool res_hot(int rmode, int cmode) {
  return rmode == R_ITER || rmode == R_TRIAL || (rmode == R_NONE && cmode == C_PRIMAL);
}

// ---- a run of iterations --------------------------------------------------------

// Row pointer i of a CTA's share (`rows` rows, cnt entries from entry base on).
// Bounds-checked builds test it as tile_ptrs_ok does and keep it in the share.
__device__ __forceinline__ int res_pointer(const EngineArgs& A, const int* ptr, int i, int rows,
                                           int base, int cnt, int where) {
  if (rows == 0) return 0;
  const int v = ld_ro(ptr + i) - base;
#ifdef PDLP_BOUNDS_CHECK
  const int next = i < rows ? ld_ro(ptr + i + 1) - base : cnt;
  if (v < 0 || v > next || next > cnt || (i == 0 && v != 0) || (i == rows && v != cnt)) {
    if (atomicCAS(&A.ctl->error, 0, PDLP_ERR_BOUNDS) == 0) A.ctl->error_where = where;
    block_fail();
    return min(max(v, 0), cnt);
  }
#endif
  return v;
}

// Index j of an entry, below len: index_ok's test before the index is narrowed;
// a bad one is kept out of the products.
__device__ __forceinline__ uint16_t res_index(const EngineArgs& A, int j, int len, int where) {
  return index_ok(A, j, len, where) ? (uint16_t)j : (uint16_t)0;
}

// Steps the LP from global memory's state until a mode that does not run on
// chip, or until `step` reaches the budget.  Returns the step count; the
// vectors and the state are back in global memory then.  (-1, with nothing
// stepped: bounds-checked builds, when a check of the loaded data failed.)
template <typename T>
__device__ __forceinline__ int res_run(const EngineArgs& A, const ResidentLP& lp, State* S, int rank,
                                       int size, int step) {
  const int budget = lp.budget;
  unsigned char* const smem = g_smem;      // the symbol itself: shared-memory addressing
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ResHeader& H = *reinterpret_cast<ResHeader*>(smem);
  const Inst& I = H.inst;
  const int nrt = I.rt_end - I.rt_begin, nct = I.ct_end - I.ct_begin;
  const ResLayout lay = res_layout(I.m, I.n, nrt + nct, lp.r, lp.c, (int)sizeof(T));
  T* const dx = reinterpret_cast<T*>(smem + lay.dx);
  T* const dy = reinterpret_cast<T*>(smem + lay.dy);
  double* const part = reinterpret_cast<double*>(smem + lay.part);
  T* const prod = reinterpret_cast<T*>(smem + lay.prod);
  double* const rv = reinterpret_cast<double*>(smem + lay.rv);   // ax y rl ru sum_y y_new adx
  double* const cv = reinterpret_cast<double*>(smem + lay.cv);   // aty x c lo hi sum_x x_new
  T* const rval = reinterpret_cast<T*>(smem + lay.rval);
  T* const cval = reinterpret_cast<T*>(smem + lay.cval);
  int* const rptr = reinterpret_cast<int*>(smem + lay.rptr);
  int* const cptr = reinterpret_cast<int*>(smem + lay.cptr);
  int2* const rtile = reinterpret_cast<int2*>(smem + lay.rtile);
  int2* const ctile = reinterpret_cast<int2*>(smem + lay.ctile);
  uint16_t* const ridx = reinterpret_cast<uint16_t*>(smem + lay.ridx);
  uint16_t* const cidx = reinterpret_cast<uint16_t*>(smem + lay.cidx);
  const int RR = lay.rrows, CR = lay.crows;

  // this CTA's share: tiles, rows and entries
  const int rt0 = res_first(nrt, rank, size), rt1 = res_first(nrt, rank + 1, size);
  const int ct0 = res_first(nct, rank, size), ct1 = res_first(nct, rank + 1, size);
  int rb = 0, rn = 0, rp0 = 0, rq = 0, cb = 0, cn = 0, cp0 = 0, cq = 0;
  if (rt1 > rt0) {
    const Tile &ta = A.rtiles[I.rt_begin + rt0], &tb = A.rtiles[I.rt_begin + rt1 - 1];
    rb = ta.begin;
    rn = tb.end - ta.begin;
    rp0 = ta.p0;
    rq = tb.p0 + tb.cnt - ta.p0;
  }
  if (ct1 > ct0) {
    const Tile &ta = A.ctiles[I.ct_begin + ct0], &tb = A.ctiles[I.ct_begin + ct1 - 1];
    cb = ta.begin;
    cn = tb.end - ta.begin;
    cp0 = ta.p0;
    cq = tb.p0 + tb.cnt - ta.p0;
  }
  {
    const int tid = threadIdx.x;
    const T* const gx = sizeof(T) == 4 ? reinterpret_cast<const T*>(I.rx32) : reinterpret_cast<const T*>(I.rx);
    const T* const gc = sizeof(T) == 4 ? reinterpret_cast<const T*>(I.cx32) : reinterpret_cast<const T*>(I.cx);
    const T* const gd = sizeof(T) == 4 ? reinterpret_cast<const T*>(I.dx32) : reinterpret_cast<const T*>(I.dx);
#pragma unroll 4
    for (int q = tid; q < rq; q += kResThreads) {
      rval[q] = __ldcg(gx + rp0 + q);
      ridx[q] = res_index(A, ld_ro(I.ri + rp0 + q), I.n, rb);
    }
#pragma unroll 4
    for (int q = tid; q < cq; q += kResThreads) {
      cval[q] = __ldcg(gc + cp0 + q);
      cidx[q] = res_index(A, ld_ro(I.ci + cp0 + q), I.m, cb);
    }
    for (int i = tid; i <= rn; i += kResThreads) rptr[i] = res_pointer(A, I.rp + rb, i, rn, rp0, rq, rb);
    for (int i = tid; i <= cn; i += kResThreads) cptr[i] = res_pointer(A, I.cp + cb, i, cn, cp0, cq, cb);
    for (int i = tid; i < rt1 - rt0; i += kResThreads) {
      const Tile& t = A.rtiles[I.rt_begin + rt0 + i];
      rtile[i] = make_int2(t.begin - rb, t.end - rb);
    }
    for (int i = tid; i < ct1 - ct0; i += kResThreads) {
      const Tile& t = A.ctiles[I.ct_begin + ct0 + i];
      ctile[i] = make_int2(t.begin - cb, t.end - cb);
    }
    for (int i = tid; i < rn; i += kResThreads) {
      rv[i] = ld_mut(I.ax + rb + i);
      rv[RR + i] = ld_mut(I.y + rb + i);
      rv[2 * RR + i] = ld_mut(I.rl + rb + i);
      rv[3 * RR + i] = ld_mut(I.ru + rb + i);
      rv[4 * RR + i] = ld_mut(I.sumy + rb + i);
      rv[5 * RR + i] = ld_mut(I.ynew + rb + i);
      rv[6 * RR + i] = ld_mut(I.adx + rb + i);
    }
    for (int i = tid; i < cn; i += kResThreads) {
      cv[i] = ld_mut(I.aty + cb + i);
      cv[CR + i] = ld_mut(I.x + cb + i);
      cv[2 * CR + i] = ld_mut(I.c + cb + i);
      cv[3 * CR + i] = ld_mut(I.lo + cb + i);
      cv[4 * CR + i] = ld_mut(I.hi + cb + i);
      cv[5 * CR + i] = ld_mut(I.sumx + cb + i);
      cv[6 * CR + i] = ld_mut(I.xnew + cb + i);
    }
    for (int i = tid; i < I.n; i += kResThreads) dx[i] = __ldcg(gd + i);
    const int* src = reinterpret_cast<const int*>(S);
    int* dst = reinterpret_cast<int*>(&H.st);
    for (int i = tid; i < (int)(sizeof(State) / sizeof(int)); i += kResThreads) dst[i] = ld_mut(src + i);
  }
  __syncthreads();
  RunState c = run_load(H.st, I);
  const int Lr = I.lanes_r, Lc = I.lanes_c;
  // thread `tid` adds rows tid / L, tid / L + threads / L, ..., L lanes each
  const int rgrp = threadIdx.x / Lr, rsub = threadIdx.x & (Lr - 1), rstep = kResThreads / Lr;
  const int cgrp = threadIdx.x / Lc, csub = threadIdx.x & (Lc - 1), cstep = kResThreads / Lc;
  double sigma = c.eta * c.omega, tau = c.eta / c.omega;
  cluster_sync();          // no peer writes into this CTA before it has loaded
#ifdef PDLP_BOUNDS_CHECK
  if (threadIdx.x == 0 && block_flags()[1]) cluster_put(&H.bad, 1, size);
  cluster_sync();
  if (H.bad) return -1;
#endif

  while (step < budget && res_hot(c.rmode, c.cmode)) {
    if (c.rmode != R_NONE) {
      const double eta = c.eta;
      const bool trial = c.rmode == R_TRIAL, commit = c.ycommit != 0;
      res_products<T>(rval, ridx, dx, prod, rq);
      __syncthreads();
      for (int r0 = 0; r0 < rn; r0 += rstep) {
        const int v = r0 + rgrp;
        const bool own = v < rn && rsub == 0;
        double ax = 0.0, y = 0.0, sumy = 0.0, rl = 0.0, ru = 0.0, yc = 0.0, adxc = 0.0;
        if (own) {
          ax = rv[v];
          y = rv[RR + v];
          rl = rv[2 * RR + v];
          ru = rv[3 * RR + v];
          sumy = rv[4 * RR + v];
          if (commit) {
            yc = rv[5 * RR + v];
            adxc = rv[6 * RR + v];
          }
        }
        T s = v < rn ? res_sum<T>(prod, rptr[v] + rsub, rptr[v + 1], Lr) : T(0);
        for (int off = Lr >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
        if (own) {
          const double a = (double)s;
          if (commit) {                     // pdlp.py:385-389
            const double yn = yc;
            y = yn;
            ax = ax + adxc;
            sumy = sumy + eta * yn;
            rv[RR + v] = y;
            rv[v] = ax;
            rv[4 * RR + v] = sumy;
          }
          if (!trial) {                     // backend.py:260-279
            const double axn = ax + a;
            rv[v] = axn;
            const double w = y + sigma * (axn + a);
            const double yn = prox(w, sigma, rl, ru);
            cluster_put(dy + rb + v, (T)(yn - y), size);
            rv[RR + v] = yn;
            rv[4 * RR + v] = sumy + eta * yn;
          } else {                          // pdlp.py:347-356
            rv[6 * RR + v] = a;
            const double axb = ax + 2.0 * a;
            const double w = y + sigma * axb;
            const double yn = prox(w, sigma, rl, ru);
            rv[5 * RR + v] = yn;
            cluster_put(dy + rb + v, (T)(yn - y), size);
          }
        }
      }
      if (trial) {
        // each tile's sums of dy adx and dy dy, in hot_rtile's lanes and order
        __syncthreads();
        for (int t = warp; t < rt1 - rt0; t += kResWarps) {
          const int2 tl = rtile[t];
          double acc[2] = {0.0, 0.0};
          for (int v = tl.x + lane; v < tl.y; v += 32) {
            const double d = rv[5 * RR + v] - rv[RR + v], a = rv[6 * RR + v];
            acc[0] += d * a;
            acc[1] += d * d;
          }
#pragma unroll
          for (int s = 0; s < 2; ++s) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc[s] += __shfl_xor_sync(kFull, acc[s], off);
          }
          if (lane < 2) cluster_put(part + 2 * (rt0 + t) + lane, lane ? acc[1] : acc[0], size);
          __syncwarp();
        }
      }
      cluster_sync();
      if (trial) {
        double s0, s1;
        res_total(part, nrt, &s0, &s1, lane);
        run_trial(c, I, s0, s1);
        sigma = c.eta * c.omega;
        tau = c.eta / c.omega;
      } else {
        c.ycommit = 0;
      }
    }
    if (c.cmode == C_ITER || c.cmode == C_PRIMAL) {
      const double eta = c.eta;
      const bool iter = c.cmode == C_ITER, xc = iter && c.xcommit != 0;
      const int kind = c.cprimal;
      if (iter) {
        res_products<T>(cval, cidx, dy, prod, cq);
        __syncthreads();
      }
      for (int r0 = 0; r0 < cn; r0 += cstep) {
        const int v = r0 + cgrp;
        const bool own = v < cn && csub == 0;
        double xv = 0.0, atyv = 0.0, cc = 0.0, lo = 0.0, hi = 0.0, sumx = 0.0;
        if (own) {
          xv = xc ? cv[6 * CR + v] : cv[CR + v];
          atyv = cv[v];
          cc = cv[2 * CR + v];
          lo = cv[3 * CR + v];
          hi = cv[4 * CR + v];
          if (iter) sumx = cv[5 * CR + v];
        }
        T s = T(0);
        if (iter) {
          if (v < cn) s = res_sum<T>(prod, cptr[v] + csub, cptr[v + 1], Lc);
          for (int off = Lc >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
        }
        if (own) {
          if (iter) {                       // backend.py:282-291
            atyv = atyv + (double)s;
            cv[v] = atyv;
            cv[5 * CR + v] = sumx + eta * xv;
          }
          if (kind == P_NONE) {
            if (xc) cv[CR + v] = xv;
          } else {                          // backend.py:204-215 / 241-255
            const double xn = clip(xv - tau * (cc + atyv), lo, hi);
            cluster_put(dx + cb + v, (T)(xn - xv), size);
            if (kind == P_TRIAL) {
              cv[6 * CR + v] = xn;
              if (xc) cv[CR + v] = xv;
            } else {
              cv[CR + v] = xn;
            }
          }
        }
      }
      if (kind == P_TRIAL) {
        // each tile's sum of dx dx, in hot_ctile's lanes and order
        __syncthreads();
        for (int t = warp; t < ct1 - ct0; t += kResWarps) {
          const int2 tl = ctile[t];
          double acc = 0.0;
          for (int v = tl.x + lane; v < tl.y; v += 32) {
            const double d = cv[6 * CR + v] - cv[CR + v];
            acc += d * d;
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(kFull, acc, off);
          if (lane == 0) cluster_put(part + 2 * (nrt + ct0 + t), acc, size);
          __syncwarp();
        }
      }
      cluster_sync();
      double s0 = 0.0, s1;
      if (kind == P_TRIAL) res_total(part + 2 * nrt, nct, &s0, &s1, lane);
      run_advance(c, I, s0);
    }
    ++step;
  }

  // back to global memory: the vectors this CTA owns, and the state (the same
  // in every CTA)
  __syncthreads();
  if (threadIdx.x == 0) run_store(c, &H.st);
  __syncthreads();
  {
    const int tid = threadIdx.x;
    T* const gd = sizeof(T) == 4 ? reinterpret_cast<T*>(I.dx32) : reinterpret_cast<T*>(I.dx);
    for (int i = tid; i < rn; i += kResThreads) {
      I.ax[rb + i] = rv[i];
      I.y[rb + i] = rv[RR + i];
      I.sumy[rb + i] = rv[4 * RR + i];
      I.ynew[rb + i] = rv[5 * RR + i];
      I.adx[rb + i] = rv[6 * RR + i];
    }
    for (int i = tid; i < cn; i += kResThreads) {
      I.aty[cb + i] = cv[i];
      I.x[cb + i] = cv[CR + i];
      I.sumx[cb + i] = cv[5 * CR + i];
      I.xnew[cb + i] = cv[6 * CR + i];
      gd[cb + i] = dx[cb + i];
    }
    if (rank == 0) {
      int* dst = reinterpret_cast<int*>(S);
      const int* src = reinterpret_cast<const int*>(&H.st);
      for (int i = tid; i < (int)(sizeof(State) / sizeof(int)); i += kResThreads) dst[i] = src[i];
    }
  }
  cluster_sync_global(lane);
  return step;
}

// ---- the kernel -----------------------------------------------------------------

// One cluster per LP of the launch (any number of them; clusters are
// independent and take SMs as they become free).  T: the precision of the
// iteration's products.  A kernel per precision and 12 warps of 168 registers,
// so that nothing spills: a spilled register is reloaded from L2, since every
// cluster barrier empties L1 (16 warps of 128 registers: an iteration of
// 230 x 2,025 took 13,500 cycles instead of 7,500; both precisions in one
// kernel, 36 bytes spilled: 35 LPs of up to 1,500 rows 70 ms instead of 50).
template <typename T>
__global__ void __launch_bounds__(kResThreads, 1) engine_resident(EngineArgs A,
                                                                  const ResidentLP* __restrict__ lps,
                                                                  int* __restrict__ steps_done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = cluster_rank(), size = cluster_size();
  const ResidentLP lp = lps[blockIdx.x / size];
  State* const S = A.st + lp.inst;
  ResHeader& H = *reinterpret_cast<ResHeader*>(g_smem);
  {
    const int* src = reinterpret_cast<const int*>(A.inst + lp.inst);
    int* dst = reinterpret_cast<int*>(&H.inst);
    for (int i = threadIdx.x; i < (int)(sizeof(Inst) / sizeof(int)); i += kResThreads) dst[i] = src[i];
    if (threadIdx.x == 0) H.failed[0] = H.failed[1] = H.bad = H.flags[1] = 0;
    __syncthreads();
  }
  const Inst& I = H.inst;
  // the generic passes' areas share the memory of the resident data
  WarpSmem& W = reinterpret_cast<WarpSmem*>(g_smem + res_up16((int)sizeof(ResHeader)))[warp];
  TeamCopy& C = H.team[warp];
  const int nw = size * kResWarps, gw = rank * kResWarps + warp;
  const int nrt = I.rt_end - I.rt_begin, nct = I.ct_end - I.ct_begin;
  const int r0 = I.rt_begin + res_first(nrt, gw, nw), r1 = I.rt_begin + res_first(nrt, gw + 1, nw);
  const int c0 = I.ct_begin + res_first(nct, gw, nw), c1 = I.ct_begin + res_first(nct, gw + 1, nw);
  int step = 0;
  int turn = 0;
  bool started = false;                // every CTA has met a barrier of this kernel
  while (step < lp.budget) {
    // A warp without tiles in a pass may still be reading the State while that
    // pass's finisher writes it.  It takes the same way through the barriers
    // all the same: before an A pass of this loop rmode alone decides, and no A
    // pass's finisher changes it (a line search runs in res_run); a step
    // without an A pass is a C_PRIMAL, in res_run, which copies the State
    // before a barrier; and the second load below decides no barrier.
    team_load(C, S, lane);
    if (C.rmode == R_NONE && C.cmode == C_NONE) break;           // the LP is done
    if (res_hot(C.rmode, C.cmode)) {
      __syncthreads();                                           // every warp has read C
      const int done = res_run<T>(A, lp, S, rank, size, step);
      if (done < 0) break;
      step = done;
      continue;
    }
    // one step of the generic passes
    // (the descriptor comes from the CTA's copy: W shares its memory with the
    // resident data)
    {
      const int* src = reinterpret_cast<const int*>(&H.inst);
      int* dst = reinterpret_cast<int*>(&W.inst);
      for (int i = lane; i < (int)(sizeof(Inst) / sizeof(int)); i += 32) dst[i] = src[i];
    }
    if (lane == 0) {
      W.inst_id = lp.inst;
      mbar_init(&W.bar[0]);
      mbar_init(&W.bar[1]);
      mbar_init_fence();
      fence_proxy_async();
    }
    __syncwarp();
    BulkPhase ph;
    if (C.rmode != R_NONE) {
      PassCache pc;
      pc.copy(lp.inst, C.rmode, 0, C.ycommit, C.eta, C.omega);
      for (int t = r0; t < r1; ++t) {
        const Tile cur = A.rtiles[t];
        ph.flush = t + 1 >= r1 || A.rtiles[t + 1].group != cur.group;
        process_rtile(A, cur, t, W, lane, pc, ph, &C);
      }
      cluster_sync_global(lane);
      started = true;
      team_load(C, S, lane);
    }
    if (C.cmode != C_NONE) {
      PassCache pc;
      pc.copy(lp.inst, C.cmode, C.cprimal, C.xcommit, C.eta, C.omega);
      for (int t = c0; t < c1; ++t) {
        const Tile cur = A.ctiles[t];
        ph.flush = t + 1 >= c1 || A.ctiles[t + 1].group != cur.group;
        process_ctile(A, cur, t, W, lane, pc, ph, &C, false);
      }
    }
    __syncwarp();
    if (lane == 0) {
      mbar_inval(&W.bar[0]);
      mbar_inval(&W.bar[1]);
    }
    // a bounded wait that gave up (in an earlier pass, here or elsewhere in the
    // launch): every CTA of the cluster leaves on rank 0's word, written once
    // every CTA is known to run
    if (rank == 0 && threadIdx.x == 0) {
      const int e = *(volatile int*)&A.ctl->error;
      if (started) cluster_put(&H.failed[turn], e, size);
    }
    cluster_sync_global(lane);
    started = true;
    ++step;
    // two words in turn: this one is next written after every thread has read it
    if (H.failed[turn] != 0) break;
    turn ^= 1;
  }
  if (rank == 0 && threadIdx.x == 0) steps_done[blockIdx.x / size] = step;
  cluster_sync();                // no CTA leaves while a peer may write into it
}

using ResidentKernel = void (*)(EngineArgs, const ResidentLP*, int*);

inline ResidentKernel resident_kernel(bool f32) {
  return f32 ? engine_resident<float> : engine_resident<double>;
}

}  // namespace pdlp
