// Batched node relaxation (BNR): K node LPs that share one scaled problem
// (matrix, costs and row bounds) and differ only in their column bounds,
// advanced together by a fixed number of PDHG iterations with a step size per
// node, then bounded from below by the safe dual bound of each node.  The
// algorithm is the reference's BNREngine.solve_batch (src/sovopt/mip/bnr.py:
// 176-301) with safe_dual_bound_batch (src/sovopt/mip/safebound.py:194-235).
//
// Layout: every per-node block is (rows, K) with the node index fastest, so a
// sparse product reads A once for all K nodes (A X with X (n, K)).  One
// iteration is three launches, each a programmatic dependent of the one before:
//   A^T dY and the primal step (+ sum dX dX)  ->  A dX and the dual step
//   (+ sums dY AdX, dY dY)  ->  per-node accept / step size,
// or, for wide batches, five, with the two products on their own.
// A taken trial is not stored but redone by the next step, which reads the
// same inputs anyway (see bnr_cols).
// The iterations of one call are captured once into a CUDA graph, keyed by
// (K, iterations, step exponents), and replayed.
//
// Products and sums keep the reference's operations in the same order
// (explicit round-to-nearest multiplies and adds: no fused multiply-add), so
// element-wise results equal the reference's CPU results.  The per-node sums
// are fixed-order trees, which differ from the reference's sequential sums
// only by rounding.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"

namespace pdlp {
namespace {

constexpr double kBnrInf = 1.0e30;               // core/tolerances.py:16
constexpr double kQuotientMax = 1.0715086071862673e301;   // 2^1000 (tolerances.py:23)
constexpr int kRowsPerBlock = 64;                // rows per block of the per-node sums

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
// numpy.minimum / numpy.maximum: a NaN operand gives NaN (fmin/fmax would drop it)
__device__ __forceinline__ double np_min(double a, double b) {
  return (isnan(a) || isnan(b)) ? a + b : fmin(a, b);
}
__device__ __forceinline__ double np_max(double a, double b) {
  return (isnan(a) || isnan(b)) ? a + b : fmax(a, b);
}
__device__ __forceinline__ double clipd(double v, double lo, double hi) {
  return np_min(np_max(v, lo), hi);     // numpy.clip: maximum, then minimum
}

// Y (rows, k) = A X with X (cols, k) node-fastest.  One thread per (row, V
// consecutive nodes): V = 2 when k is even (16-byte gathers and stores), else
// 1.  Each node's entries are added in storage order (the reference's CSR
// SpMM order).  The entries are taken two at a time, both gathers issued
// before the adds, with eight blocks resident per SM.  The products are bound
// by the latency of gathers that L2 serves; among one, two or four nodes per
// thread, two to eight entries per batch and one to eight blocks per SM, this
// form measured fastest on B200.
template <int V>
struct Lanes;
template <>
struct Lanes<1> {
  double v[1];
  __device__ static Lanes load(const double* p) { return Lanes{{*p}}; }
  __device__ void store(double* p) const { *p = v[0]; }
};
template <>
struct Lanes<2> {
  double v[2];
  __device__ static Lanes load(const double* p) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    return Lanes{{t.x, t.y}};
  }
  __device__ void store(double* p) const { *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]); }
};

template <int V>
__global__ void __launch_bounds__(256, 8) bnr_spmm(int rows, int k, const int64_t* __restrict__ rp,
                                                const int* __restrict__ ri,
                                                const double* __restrict__ rx,
                                                const double* X, double* Y) {
  constexpr int kBatch = 2;
  grid_dep_wait();
  const int groups = k / V;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)rows * groups) return;
  const long long r = g / groups;
  const int col = (int)(g - r * groups) * V;
  const double* Xc = X + col;
  long long p = __ldg(rp + r);
  const long long end = __ldg(rp + r + 1);
  double acc[V];
#pragma unroll
  for (int u = 0; u < V; ++u) acc[u] = 0.0;
  for (; p + kBatch <= end; p += kBatch) {
    double v[kBatch];
    Lanes<V> x[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      v[u] = __ldg(rx + p + u);
      x[u] = Lanes<V>::load(Xc + (long long)__ldg(ri + p + u) * k);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
#pragma unroll
      for (int e = 0; e < V; ++e) acc[e] = add(acc[e], mul(v[u], x[u].v[e]));
  }
  for (; p < end; ++p) {
    const double v = __ldg(rx + p);
    const Lanes<V> x = Lanes<V>::load(Xc + (long long)__ldg(ri + p) * k);
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = add(acc[e], mul(v, x.v[e]));
  }
  Lanes<V> out;
#pragma unroll
  for (int e = 0; e < V; ++e) out.v[e] = acc[e];
  out.store(Y + r * k + col);
}

// ---- one iteration: a product fused with the step that uses it -----------------
//
// A block takes 64 consecutive rows and a tile of at most 16 nodes: 2^txs
// threads along the nodes, V nodes each (two when K is even: 16-byte gathers
// and vectors), the others along the rows.  Before it waits for the launch
// before it (programmatic dependent launch) it stages the rows' pointers,
// indices and values, which no launch changes, in shared memory; then the
// gathers of the product and the vectors of the step are in flight together,
// and the product goes to memory only where a later step needs it.
//
// Small batches are bound by the chain of launches and round trips: five
// launches per iteration (primal, A dX, dual, A^T dY, accept) took 23 to 31 us
// whatever the size; three take 10 to 20.  Per 60 iterations, split against
// fused on B200: 2,000 x 3,000, 8 nodes 1.50 / 0.68 ms, 64 nodes 1.42 / 0.97;
// 20,000 x 30,000, 8 nodes 1.86 / 1.26, 16 nodes 1.91 / 1.67.  Wide batches are
// bound by the gathers, which L2 serves (245 MB per product at 128 nodes), and
// want the most warps, which the split kernels have: 128 nodes 8.14 / 8.4 ms at
// best.  See fused_shape for the line between them.
//
// The per-node sums over rows run in a fixed order: blocks of kRowsPerBlock
// rows; in a block, phase p (8 phases) adds rows r0 + p + 8 j for j ascending
// from 0.0; the phases are added in order; then bnr_accept adds the blocks.
// The rows' terms go through shared memory.  Output pair of row block b and
// node j at part[2 (j pstride + b)], pstride = mblocks + nblocks + 1, so one
// node's partials are contiguous for the warp that adds them: m-side blocks
// [0, mblocks), n-side blocks [mblocks, mblocks + nblocks).
constexpr int kStageCap = 1024;      // entries of a block's rows that are staged
constexpr int kBnrThreads = 256;
constexpr int kTileNodes = 16;       // nodes of a block's tile, at most

struct BnrStage {
  double term[2][kRowsPerBlock * kTileNodes];   // the sums' terms: [row * tile + node]
  int off[kRowsPerBlock + 1];        // from the block's first entry (nnz fits an int)
  double val[kStageCap];
  int idx[kStageCap];
};

template <int V>
struct BnrTile {
  int x, y, ty, tile, node, nr;      // thread's place, node tile width, first node, rows
  bool live;
};

template <int V>
__device__ __forceinline__ BnrTile<V> bnr_tile(int rows, int k, int txs) {
  BnrTile<V> t;
  t.x = threadIdx.x & ((1 << txs) - 1);
  t.y = threadIdx.x >> txs;
  t.ty = kBnrThreads >> txs;
  t.tile = V << txs;
  t.node = (blockIdx.y << txs) * V + t.x * V;
  t.nr = min(kRowsPerBlock, rows - (int)blockIdx.x * kRowsPerBlock);
  t.live = t.node < k;
  return t;
}

// Stages the block's rows.  Returns whether their entries fit (else they are
// read from memory) and sets *first to the block's first entry.
__device__ __forceinline__ bool bnr_stage(BnrStage& S, int r0, int nr, const int64_t* __restrict__ rp,
                                          const int* __restrict__ ri,
                                          const double* __restrict__ rx, int* first) {
  const int p0 = (int)__ldg(rp + r0);
  *first = p0;
  if ((int)threadIdx.x <= nr) S.off[threadIdx.x] = (int)__ldg(rp + r0 + threadIdx.x) - p0;
  __syncthreads();
  const int cnt = S.off[nr];
  if (cnt > kStageCap) return false;
  for (int q = threadIdx.x; q < cnt; q += kBnrThreads) {
    S.idx[q] = __ldg(ri + p0 + q);
    S.val[q] = __ldg(rx + p0 + q);
  }
  __syncthreads();
  return true;
}

// Row r of the block times the nodes' columns of X, the entries added in
// storage order, kB gathers in flight.
template <int V>
__device__ __forceinline__ Lanes<V> bnr_row(const BnrStage& S, bool staged, int r, int k,
                                            const int* __restrict__ ri,
                                            const double* __restrict__ rx,
                                            const double* Xc) {
  constexpr int kB = 4;
  Lanes<V> a;
#pragma unroll
  for (int e = 0; e < V; ++e) a.v[e] = 0.0;
  const int* const idx = staged ? S.idx : ri;
  const double* const val = staged ? S.val : rx;
  int q = S.off[r];
  const int end = S.off[r + 1];
  for (; q + kB <= end; q += kB) {
    Lanes<V> x[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) x[u] = Lanes<V>::load(Xc + (long long)idx[q + u] * k);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const double v = val[q + u];
#pragma unroll
      for (int e = 0; e < V; ++e) a.v[e] = add(a.v[e], mul(v, x[u].v[e]));
    }
  }
  if (q < end) {                      // the last 1 .. kB - 1 entries, in flight together
    Lanes<V> x[kB - 1];
#pragma unroll
    for (int u = 0; u < kB - 1; ++u)
      if (q + u < end) x[u] = Lanes<V>::load(Xc + (long long)idx[q + u] * k);
#pragma unroll
    for (int u = 0; u < kB - 1; ++u)
      if (q + u < end) {
        const double v = val[q + u];
#pragma unroll
        for (int e = 0; e < V; ++e) a.v[e] = add(a.v[e], mul(v, x[u].v[e]));
      }
  }
  return a;
}

// The block's sums per node from the rows' terms; NS sums.
template <int V, int NS>
__device__ __forceinline__ void bnr_sums(BnrStage& S, const BnrTile<V>& t, int k, int pstride,
                                         int part_block, double* part) {
  const int tile = t.tile;
  __syncthreads();                    // the rows' terms are in place
  for (int w = threadIdx.x; w < 8 * tile; w += kBnrThreads) {
    const int ph = w / tile, j = w - ph * tile;
    double a[NS] = {};
    for (int r = ph; r < t.nr; r += 8) {
#pragma unroll
      for (int c = 0; c < NS; ++c) a[c] = add(a[c], S.term[c][r * tile + j]);
    }
    // rows ph + 8 j are this thread's alone: its sum may replace the first
#pragma unroll
    for (int c = 0; c < NS; ++c) S.term[c][ph * tile + j] = a[c];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < tile; j += kBnrThreads) {
    const int node = (int)blockIdx.y * tile + j;
    if (node >= k) continue;
    double* out = part + ((long long)node * pstride + part_block) * 2;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      double a = 0.0;
      if (c < NS) {
        a = S.term[c][j];
        for (int y = 1; y < 8; ++y) a = add(a, S.term[c][y * tile + j]);
      }
      out[c] = a;
    }
  }
}

// A taken trial is not stored: the next step recomputes it.  pend[j] says
// that node j's last trial was taken, and eta_prev[j] is the step size that
// trial used.  The next primal and dual steps read X, AtY, Y and AX anyway;
// for a pending node they first redo the trial from them with the same
// operations, which gives the same bits, and store it as the current
// iterate together with the reference's other updates on acceptance,
// AtY += AtdY and AX += AdX (bnr.py:262-265).  Nothing is copied, and one
// buffer per iterate suffices.

// For a node with a taken trial, AtdY = A^T dY (of that trial) and the update;
// then Xn = clip(X - tau (c + AtY), L, U), dX = Xn - X (bnr.py:233-236), and the
// node's sum of dX dX over the block's columns.
template <int V>
__global__ void __launch_bounds__(kBnrThreads, 2) bnr_cols(
    int n, int k, int txs, int mblocks, int pstride, const int64_t* __restrict__ cp,
    const int* __restrict__ ci, const double* __restrict__ cx, const double* __restrict__ c,
    const double* eta, const double* eta_prev, const double* __restrict__ omega, const int* pend,
    double* X, double* AtY, const double* dY, const double* __restrict__ L,
    const double* __restrict__ U, double* dX, double* part) {
  __shared__ BnrStage S;
  const BnrTile<V> t = bnr_tile<V>(n, k, txs);
  const int r0 = blockIdx.x * kRowsPerBlock;
  grid_dep_release();
  int first;
  const bool staged = bnr_stage(S, r0, t.nr, cp, ci, cx, &first);
  grid_dep_wait();
  if (t.live) {
    double tau[V], tau_prev[V];
    bool taken[V], any = false;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const double om = omega[t.node + e];
      tau[e] = eta[t.node + e] / om;
      tau_prev[e] = eta_prev[t.node + e] / om;
      taken[e] = pend[t.node + e] != 0;
      any |= taken[e];
    }
    for (int r = t.y; r < t.nr; r += t.ty) {
      const long long g = (long long)(r0 + r) * k + t.node;
      const double cr = __ldg(c + r0 + r);
      const Lanes<V> lo = Lanes<V>::load(L + g), hi = Lanes<V>::load(U + g);
      Lanes<V> x = Lanes<V>::load(X + g), aty = Lanes<V>::load(AtY + g), d;
      if (any) {
        const Lanes<V> atdy = bnr_row<V>(S, staged, r, k, ci + first, cx + first, dY + t.node);
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (taken[e]) {
            x.v[e] = clipd(sub(x.v[e], mul(tau_prev[e], add(cr, aty.v[e]))), lo.v[e], hi.v[e]);
            aty.v[e] = add(aty.v[e], atdy.v[e]);
          }
        x.store(X + g);
        aty.store(AtY + g);
      }
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const double xn = clipd(sub(x.v[e], mul(tau[e], add(cr, aty.v[e]))), lo.v[e], hi.v[e]);
        d.v[e] = sub(xn, x.v[e]);
        S.term[0][r * t.tile + t.x * V + e] = mul(d.v[e], d.v[e]);
      }
      d.store(dX + g);
    }
  }
  bnr_sums<V, 1>(S, t, k, pstride, mblocks + blockIdx.x, part);
}

// The dual trial of a node with step sigma (bnr.py:238-242).
__device__ __forceinline__ double dual_trial(double y, double ax, double adx, double sigma,
                                             double lo, double hi) {
  const double w = add(y, mul(sigma, add(ax, mul(2.0, adx))));
  return sub(w, mul(sigma, clipd(w / sigma, lo, hi)));
}

// AdX = A dX; W = Y + sigma (AX + 2 AdX); Yn = W - sigma clip(W / sigma, rl, ru);
// dY = Yn - Y (bnr.py:238-242), and the node's sums of dY AdX and dY dY over
// the block's rows.  AdX_prev is the previous step's A dX, which the redone
// trial uses.
template <int V>
__global__ void __launch_bounds__(kBnrThreads, 2) bnr_rows(
    int m, int k, int txs, int pstride, const int64_t* __restrict__ rp, const int* __restrict__ ri,
    const double* __restrict__ rx, const double* __restrict__ rl, const double* __restrict__ ru,
    const double* eta, const double* eta_prev, const double* __restrict__ omega, const int* pend,
    double* Y, double* AX, const double* AdX_prev, const double* dX, double* AdX, double* dY,
    double* part) {
  __shared__ BnrStage S;
  const BnrTile<V> t = bnr_tile<V>(m, k, txs);
  const int r0 = blockIdx.x * kRowsPerBlock;
  grid_dep_release();
  int first;
  const bool staged = bnr_stage(S, r0, t.nr, rp, ri, rx, &first);
  grid_dep_wait();
  if (t.live) {
    double sigma[V], sigma_prev[V];
    bool taken[V], any = false;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const double om = omega[t.node + e];
      sigma[e] = eta[t.node + e] * om;
      sigma_prev[e] = eta_prev[t.node + e] * om;
      taken[e] = pend[t.node + e] != 0;
      any |= taken[e];
    }
    for (int r = t.y; r < t.nr; r += t.ty) {
      const long long g = (long long)(r0 + r) * k + t.node;
      const double lo = __ldg(rl + r0 + r), hi = __ldg(ru + r0 + r);
      Lanes<V> y = Lanes<V>::load(Y + g), ax = Lanes<V>::load(AX + g), d, prev;
      if (any) prev = Lanes<V>::load(AdX_prev + g);
      const Lanes<V> adx = bnr_row<V>(S, staged, r, k, ri + first, rx + first, dX + t.node);
      adx.store(AdX + g);
      if (any) {
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (taken[e]) {
            y.v[e] = dual_trial(y.v[e], ax.v[e], prev.v[e], sigma_prev[e], lo, hi);
            ax.v[e] = add(ax.v[e], prev.v[e]);
          }
        y.store(Y + g);
        ax.store(AX + g);
      }
#pragma unroll
      for (int e = 0; e < V; ++e) {
        d.v[e] = sub(dual_trial(y.v[e], ax.v[e], adx.v[e], sigma[e], lo, hi), y.v[e]);
        S.term[0][r * t.tile + t.x * V + e] = mul(d.v[e], adx.v[e]);
        S.term[1][r * t.tile + t.x * V + e] = mul(d.v[e], d.v[e]);
      }
      d.store(dY + g);
    }
  }
  bnr_sums<V, 2>(S, t, k, pstride, blockIdx.x, part);
}

// ---- the steps alone, for wide batches ------------------------------------------
//
// With many rows times nodes the products run faster as kernels of their own,
// one row and two nodes per thread (bnr_spmm): see fused_shape.  Block (32, 8)
// with threadIdx.x the node within a 32-node tile; same sums, same order.
__device__ __forceinline__ void bnr_block_sums(double s0, double s1, int k, int node,
                                               int pstride, int part_block,
                                               double* part) {
  __shared__ double sh[2][8][32];
  sh[0][threadIdx.y][threadIdx.x] = s0;
  sh[1][threadIdx.y][threadIdx.x] = s1;
  __syncthreads();
  if (threadIdx.y == 0 && node < k) {
    double a = sh[0][0][threadIdx.x], c2 = sh[1][0][threadIdx.x];
    for (int y = 1; y < 8; ++y) {
      a = add(a, sh[0][y][threadIdx.x]);
      c2 = add(c2, sh[1][y][threadIdx.x]);
    }
    double* out = part + ((long long)node * pstride + part_block) * 2;
    out[0] = a;
    out[1] = c2;
  }
}

// Xn = clip(X - tau (c + AtY), L, U), dX = Xn - X (bnr.py:233-236), and the
// node's sum of dX dX over the block's rows.
__global__ void __launch_bounds__(256) bnr_primal(int n, int k, int mblocks, int pstride,
                                                  const double* __restrict__ c,
                                                  const double* eta, const double* eta_prev,
                                                  const double* __restrict__ omega,
                                                  const int* pend, double* X, double* AtY,
                                                  const double* AtdY,
                                                  const double* __restrict__ L,
                                                  const double* __restrict__ U,
                                                  double* dX, double* part) {
  grid_dep_wait();
  const int node = blockIdx.y * 32 + threadIdx.x;
  double s = 0.0;
  if (node < k) {
    const double tau = eta[node] / omega[node];
    const bool taken = pend[node] != 0;
    const double tau_prev = eta_prev[node] / omega[node];
    const int r0 = blockIdx.x * kRowsPerBlock, r1 = min(n, r0 + kRowsPerBlock);
    for (int r = r0 + threadIdx.y; r < r1; r += 8) {
      const long long g = (long long)r * k + node;
      const double cr = __ldg(c + r), lo = L[g], hi = U[g];
      double x = X[g], aty = AtY[g];
      if (taken) {
        x = clipd(sub(x, mul(tau_prev, add(cr, aty))), lo, hi);
        aty = add(aty, AtdY[g]);
        X[g] = x;
        AtY[g] = aty;
      }
      const double xn = clipd(sub(x, mul(tau, add(cr, aty))), lo, hi);
      const double d = sub(xn, x);
      dX[g] = d;
      s = add(s, mul(d, d));
    }
  }
  bnr_block_sums(s, 0.0, k, node, pstride, mblocks + blockIdx.x, part);
}

// W = Y + sigma (AX + 2 AdX); Yn = W - sigma clip(W / sigma, rl, ru); dY = Yn - Y
// (bnr.py:238-242), and the node's sums of dY AdX and dY dY over the block's
// rows.  AdX_prev is the previous step's A dX, which the redone trial uses.
__global__ void __launch_bounds__(256) bnr_dual(int m, int k, int pstride,
                                                const double* __restrict__ rl,
                                                const double* __restrict__ ru,
                                                const double* eta, const double* eta_prev,
                                                const double* __restrict__ omega,
                                                const int* pend, double* Y, double* AX,
                                                const double* AdX_prev, const double* AdX,
                                                double* dY, double* part) {
  grid_dep_wait();
  const int node = blockIdx.y * 32 + threadIdx.x;
  double s0 = 0.0, s1 = 0.0;
  if (node < k) {
    const double sigma = eta[node] * omega[node];
    const bool taken = pend[node] != 0;
    const double sigma_prev = eta_prev[node] * omega[node];
    const int r0 = blockIdx.x * kRowsPerBlock, r1 = min(m, r0 + kRowsPerBlock);
    for (int r = r0 + threadIdx.y; r < r1; r += 8) {
      const long long g = (long long)r * k + node;
      const double lo = __ldg(rl + r), hi = __ldg(ru + r), adx = AdX[g];
      double y = Y[g], ax = AX[g];
      if (taken) {
        const double adx_prev = AdX_prev[g];
        y = dual_trial(y, ax, adx_prev, sigma_prev, lo, hi);
        ax = add(ax, adx_prev);
        Y[g] = y;
        AX[g] = ax;
      }
      const double d = sub(dual_trial(y, ax, adx, sigma, lo, hi), y);
      dY[g] = d;
      s0 = add(s0, mul(d, adx));
      s1 = add(s1, mul(d, d));
    }
  }
  bnr_block_sums(s0, s1, k, node, pstride, blockIdx.x, part);
}

// The sum over nb row blocks (from block b0) of slot c of a node's partials,
// by one warp: lane l adds blocks l, l + 32, ... in order from 0.0, then the
// 32 lane sums are added in lane order.  Every lane returns the total.
__device__ __forceinline__ double lanes_total(double s) {
  double a = __shfl_sync(0xffffffffu, s, 0);
  for (int l = 1; l < 32; ++l) a = add(a, __shfl_sync(0xffffffffu, s, l));
  return a;
}

__device__ __forceinline__ double warp_blocks_sum(const double* __restrict__ part, int pstride,
                                                  int node, int b0, int nb, int c, int lane) {
  const double* p = part + ((long long)node * pstride + b0) * 2 + c;
  double s = 0.0;
#pragma unroll 8
  for (int b = lane; b < nb; b += 32) s = add(s, p[2 * b]);
  return lanes_total(s);
}

// Per node (one warp each): the step-size test's sums over the row blocks,
// then the test and the next step size (bnr.py:244-270).  A taken trial sets
// accept[node] (the next step's pend); eta_prev keeps the step it used.  fac holds the iteration's (1 - t^-growth,
// 1 + t^-damp), computed on the host with the C library's pow, as the
// reference computes them.
__global__ void __launch_bounds__(128) bnr_accept(int k, int mblocks, int nblocks,
                                                  const double* part, double* eta,
                                                  double* eta_prev,
                                                  const double* __restrict__ omega, int* accept,
                                                  const double* __restrict__ fac) {
  const int lane = threadIdx.x & 31;
  const int node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  grid_dep_release();
  grid_dep_wait();
  if (node >= k) return;            // whole warps leave together
  const int pstride = mblocks + nblocks + 1;
  // the three sums, each in warp_blocks_sum's order, in one loop so that the
  // loads of both sides are in flight together; their lane totals interleaved
  // as three independent chains
  const double* base = part + (long long)node * pstride * 2;
  const double2* pm = reinterpret_cast<const double2*>(base);
  const double* pn = base + 2 * (long long)mblocks;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  const int nmax = max(mblocks, nblocks);
  constexpr int kU = 8;             // blocks per lane in flight, added in order
  for (int b0 = lane; b0 < nmax; b0 += 32 * kU) {
    double2 v[kU];
    double w[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int b = b0 + 32 * u;
      v[u] = b < mblocks ? pm[b] : make_double2(0.0, 0.0);
      w[u] = b < nblocks ? pn[2 * b] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int b = b0 + 32 * u;
      if (b < mblocks) {
        s0 = add(s0, v[u].x);
        s1 = add(s1, v[u].y);
      }
      if (b < nblocks) s2 = add(s2, w[u]);
    }
  }
  double dyadx = __shfl_sync(0xffffffffu, s0, 0), dydy = __shfl_sync(0xffffffffu, s1, 0),
         dxdx = __shfl_sync(0xffffffffu, s2, 0);
  for (int l = 1; l < 32; ++l) {
    dyadx = add(dyadx, __shfl_sync(0xffffffffu, s0, l));
    dydy = add(dydy, __shfl_sync(0xffffffffu, s1, l));
    dxdx = add(dxdx, __shfl_sync(0xffffffffu, s2, l));
  }
  if (lane != 0) return;
  const double om = omega[node];
  const double interaction = fabs(dyadx);
  const double movement = mul(0.5, add(mul(om, dxdx), dydy / om));
  const double floor_ = np_max(movement, 1.0) / kQuotientMax;
  const double limit = interaction > 0.0 ? movement / np_max(interaction, floor_) : INFINITY;
  const double e = eta[node];
  accept[node] = (e <= limit) || (movement == 0.0);
  eta_prev[node] = e;
  double en = np_min(mul(fac[0], limit), mul(fac[1], e));
  en = fmax(isfinite(en) ? en : 1.0, 1e-14);
  eta[node] = en;
}

// Each node's final iterates: for a node whose last trial was taken, that
// trial, redone as in bnr_primal / bnr_dual; otherwise X and Y as they are.
__global__ void bnr_resolve_x(long long total, int k, const int* __restrict__ pend,
                              const double* __restrict__ eta_prev,
                              const double* __restrict__ omega, const double* __restrict__ c,
                              const double* __restrict__ X, const double* __restrict__ AtY,
                              const double* __restrict__ L, const double* __restrict__ U,
                              double* __restrict__ out) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const int node = (int)(g % k);
  double x = X[g];
  if (pend[node]) {
    const double tau = eta_prev[node] / omega[node];
    x = clipd(sub(x, mul(tau, add(c[g / k], AtY[g]))), L[g], U[g]);
  }
  out[g] = x;
}

__global__ void bnr_resolve_y(long long total, int k, const int* __restrict__ pend,
                              const double* __restrict__ eta_prev,
                              const double* __restrict__ omega, const double* __restrict__ rl,
                              const double* __restrict__ ru, const double* __restrict__ Y,
                              const double* __restrict__ AX, const double* __restrict__ AdX,
                              double* __restrict__ out) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const int node = (int)(g % k);
  double y = Y[g];
  if (pend[node]) {
    const long long i = g / k;
    y = dual_trial(y, AX[g], AdX[g], eta_prev[node] * omega[node], rl[i], ru[i]);
  }
  out[g] = y;
}

// X = clip(X, L, U) (bnr.py:211)
__global__ void bnr_clip(long long total, double* __restrict__ X, const double* __restrict__ L,
                         const double* __restrict__ U) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < total) X[g] = clipd(X[g], L[g], U[g]);
}

// Safe dual bound terms (safebound.py:212-230), per-node partial sums and
// flags over blocks of rows: the m side from Y, the n side from d = c - A^T Y.
// The pair of (node, block), laid out as for the step sums, is (sum, flags):
// flag 1 = a vacuous term, flag 2 = an empty column box L > U + 1e-12
// (bnr.py:203).
__global__ void __launch_bounds__(256) bnr_bound_terms(
    int m, int n, int k, int mblocks, int pstride, const double* __restrict__ Y,
    const double* __restrict__ rl, const double* __restrict__ ru,
    const double* __restrict__ c, const double* __restrict__ aty,
    const double* __restrict__ L, const double* __restrict__ U, double* __restrict__ part) {
  __shared__ double sh[8][32];
  __shared__ int bad_sh[8][32];
  const bool mside = (int)blockIdx.x < mblocks;
  const int b = mside ? blockIdx.x : blockIdx.x - mblocks;
  const int rows = mside ? m : n;
  const int node = blockIdx.y * 32 + threadIdx.x;
  double s = 0.0;
  int bad = 0;
  if (node < k) {
    const int r0 = b * kRowsPerBlock, r1 = min(rows, r0 + kRowsPerBlock);
    for (int r = r0 + threadIdx.y; r < r1; r += 8) {
      const long long g = (long long)r * k + node;
      if (mside) {
        const double y = Y[g];
        const bool pos = y > 0.0;
        const bool rbad = (pos ? rl[r] <= -kBnrInf : ru[r] >= kBnrInf) && y != 0.0;
        const double pick = pos ? rl[r] : ru[r];
        s = add(s, rbad ? 0.0 : mul(y, pick));
        bad |= rbad;
      } else {
        const double d = sub(c[r], aty[g]);
        const bool pos = d > 0.0;
        const bool cbad = (pos ? L[g] <= -kBnrInf : U[g] >= kBnrInf) && d != 0.0;
        const double pick = pos ? L[g] : U[g];
        s = add(s, cbad ? 0.0 : mul(d, pick));
        bad |= cbad;
        if (L[g] > U[g] + 1e-12) bad |= 2;
      }
    }
  }
  sh[threadIdx.y][threadIdx.x] = s;
  bad_sh[threadIdx.y][threadIdx.x] = bad;
  __syncthreads();
  if (threadIdx.y == 0 && node < k) {
    double a = sh[0][threadIdx.x];
    int f = bad_sh[0][threadIdx.x];
    for (int yy = 1; yy < 8; ++yy) {
      a = add(a, sh[yy][threadIdx.x]);
      f |= bad_sh[yy][threadIdx.x];
    }
    double* out = part + ((long long)node * pstride + blockIdx.x) * 2;
    out[0] = a;
    out[1] = (double)f;
  }
}

// Per node: bound = (row sum + column sum + offset) / obj_scale, -inf when
// vacuous, +inf for an empty box; also the infeasible flag (bnr.py:203, 283-290).
__global__ void __launch_bounds__(128) bnr_bound_final(int k, int mblocks, int nblocks,
                                                       const double* __restrict__ part,
                                                       double obj_offset, double obj_scale,
                                                       double* __restrict__ bounds,
                                                       unsigned char* __restrict__ empty) {
  const int lane = threadIdx.x & 31;
  const int node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (node >= k) return;            // whole warps leave together
  const int pstride = mblocks + nblocks + 1;
  const double rs = warp_blocks_sum(part, pstride, node, 0, mblocks, 0, lane);
  const double cs = warp_blocks_sum(part, pstride, node, mblocks, nblocks, 0, lane);
  int flags = 0;
  for (int b = lane; b < mblocks + nblocks; b += 32)
    flags |= (int)part[((long long)node * pstride + b) * 2 + 1];
  flags = __reduce_or_sync(0xffffffffu, flags);
  if (lane != 0) return;
  const bool vac = flags & 1, emp = flags & 2;
  const double bound = vac ? -INFINITY : add(rs, cs);
  bounds[node] = emp ? INFINITY : (bound + obj_offset) / obj_scale;
  empty[node] = emp ? 1 : 0;
}

int blocks_for(long long total) { return (int)std::max(1LL, (total + 255) / 256); }

// Y (rows, k) = A X on stream s, two nodes per thread when k is even.
void launch_spmm(int rows, int k, const int64_t* rp, const int* ri, const double* rx,
                 const double* X, double* Y, cudaStream_t s) {
  if (k % 2 == 0)
    bnr_spmm<2><<<blocks_for((long long)rows * (k / 2)), 256, 0, s>>>(rows, k, rp, ri, rx, X, Y);
  else
    bnr_spmm<1><<<blocks_for((long long)rows * k), 256, 0, s>>>(rows, k, rp, ri, rx, X, Y);
}

}  // namespace
}  // namespace pdlp

using namespace pdlp;

struct pdlp_bnr {
  cudaStream_t stream = nullptr;
  int m = 0, n = 0;
  long long nnz = 0;
  double obj_scale = 1.0, obj_offset = 0.0;
  // shared problem (device)
  int64_t *rp = nullptr, *cp = nullptr;
  int *ri = nullptr, *ci = nullptr;
  double *rx = nullptr, *cx = nullptr, *c = nullptr, *rl = nullptr, *ru = nullptr;
  // per-node blocks, sized for cap nodes
  int cap = 0;
  // A dX in two buffers, alternating by iteration (a step redoes the
  // previous trial with the previous A dX)
  double *L = nullptr, *U = nullptr, *X = nullptr, *dX = nullptr, *AtY = nullptr,
         *AtdY = nullptr;
  double *Y = nullptr, *dY = nullptr, *AX = nullptr, *AdX0 = nullptr, *AdX1 = nullptr;
  double *eta = nullptr, *eta_prev = nullptr, *omega = nullptr, *part = nullptr,
         *bounds = nullptr;
  int* accept = nullptr;
  unsigned char* empty = nullptr;
  std::vector<double> h_eta, h_omega;   // persistent step sizes (bnr.py:168-171)
  // the captured iterations
  cudaStream_t cap_stream = nullptr;
  cudaGraphExec_t graph = nullptr;
  double* fac = nullptr;          // per iteration (1 - t^-growth, 1 + t^-damp)
  int g_k = -1, g_iters = -1;
  long long g_launches = 0;
  double g_growth = 0.0, g_damp = 0.0;
};

namespace {

void bnr_free_blocks(pdlp_bnr* b) {
  double** ds[] = {&b->L, &b->U, &b->X, &b->dX, &b->AtY, &b->AtdY, &b->Y, &b->dY, &b->AX,
                   &b->AdX0, &b->AdX1, &b->eta, &b->eta_prev, &b->omega, &b->part, &b->bounds};
  for (double** d : ds) { cudaFree(*d); *d = nullptr; }
  cudaFree(b->accept); b->accept = nullptr;
  cudaFree(b->empty); b->empty = nullptr;
  if (b->graph) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }
}

// Capacity for K nodes (the reference doubles its buffers: bnr.py:166-171).
int bnr_ensure(pdlp_bnr* b, int K) {
  if (K <= b->cap) return PDLP_OK;
  const int cap = std::max(K, b->cap * 2);
  PDLP_CUDA(cudaStreamSynchronize(b->stream));
  bnr_free_blocks(b);
  const size_t nk = (size_t)b->n * cap, mk = (size_t)b->m * cap;
  const int mblocks = (b->m + kRowsPerBlock - 1) / kRowsPerBlock;
  const int nblocks = (b->n + kRowsPerBlock - 1) / kRowsPerBlock;
  struct { double** p; size_t n; } want[] = {
      {&b->L, nk}, {&b->U, nk}, {&b->X, nk}, {&b->dX, nk}, {&b->AtY, nk}, {&b->AtdY, nk},
      {&b->Y, mk}, {&b->dY, mk}, {&b->AX, mk}, {&b->AdX0, mk}, {&b->AdX1, mk},
      {&b->eta, (size_t)cap}, {&b->eta_prev, (size_t)cap}, {&b->omega, (size_t)cap},
      {&b->part, (size_t)(mblocks + nblocks + 1) * cap * 2}, {&b->bounds, (size_t)cap}};
  for (auto& w : want) {
    const cudaError_t e = cudaMalloc(w.p, sizeof(double) * std::max<size_t>(w.n, 1));
    if (e != cudaSuccess) { bnr_free_blocks(b); b->cap = 0; return fail(PDLP_ERR_OOM, "bnr: cudaMalloc"); }
  }
  if (cudaMalloc(&b->accept, sizeof(int) * cap) != cudaSuccess ||
      cudaMalloc(&b->empty, (size_t)cap) != cudaSuccess) {
    bnr_free_blocks(b);
    b->cap = 0;
    return fail(PDLP_ERR_OOM, "bnr: cudaMalloc");
  }
  // growing restarts every node's step sizes at 1, as the reference's
  // buffer growth does (bnr.py:149-171); otherwise they persist across calls
  b->h_eta.assign(cap, 1.0);
  b->h_omega.assign(cap, 1.0);
  b->cap = cap;
  return PDLP_OK;
}

template <typename T>
int bnr_upload(T** dst, const T* src, size_t count, int memory, cudaStream_t st) {
  PDLP_CUDA(cudaMalloc(dst, sizeof(T) * std::max<size_t>(count, 1)));
  if (count == 0) return PDLP_OK;
  if (!src) return fail(PDLP_ERR_ARG, "bnr: a required array is NULL");
  PDLP_CUDA(cudaMemcpyAsync(*dst, src, sizeof(T) * count,
                            memory == PDLP_MEM_HOST ? cudaMemcpyHostToDevice
                                                    : cudaMemcpyDeviceToDevice, st));
  return PDLP_OK;
}

// The fused form for K nodes and `blocks` blocks of 64 rows (both sides), or 0
// for the split form.  Returns the node tiles and sets the threads along the
// nodes, 2^txs of V nodes each: four, or eight when four make more blocks than
// about three per SM.  Beyond five per SM, or with tiles of 32 nodes or more,
// the split form is as fast or faster (ms per 60 iterations, split against four
// / eight / sixteen threads: 2,000 x 3,000, 32 nodes 1.45 against 0.76 / 0.96 /
// 1.30, 128 nodes 1.49 against 1.51 / 1.33 / 1.47; 8,000 x 12,000, 32 nodes 1.58
// against 1.51 / 1.30 / 1.44, 64 nodes 1.84 against 2.60 / 1.97 / 1.85).
unsigned fused_shape(int blocks, int K, int V, int* txs) {
  constexpr long long kThreePerSM = 400, kFivePerSM = 800;
  auto tiles = [&](int x) { return ((long long)K + (V << x) - 1) / (V << x); };
  int x = 0;
  while (x < 2 && tiles(x) > 1) ++x;
  if (tiles(x) > 1 && blocks * tiles(x) > kThreePerSM) ++x;
  *txs = x;
  return blocks * tiles(x) <= kFivePerSM ? (unsigned)tiles(x) : 0u;
}

// The launches of `iters` iterations for K nodes, on stream s; returns how
// many kernels it launched.
long long bnr_enqueue_iterations(pdlp_bnr* b, int K, int iters, cudaStream_t s) {
  const int mblocks = (b->m + kRowsPerBlock - 1) / kRowsPerBlock;
  const int nblocks = (b->n + kRowsPerBlock - 1) / kRowsPerBlock;
  const int V = K % 2 == 0 ? 2 : 1;
  int txs = 0;
  const unsigned tiles = fused_shape(mblocks + nblocks, K, V, &txs);
  const bool fused = tiles > 0;
  const int pstride = mblocks + nblocks + 1;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  long long launches = 0;
  auto launch = [&](auto kernel, dim3 grid, dim3 block, auto... args) {
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cudaLaunchKernelEx(&cfg, kernel, args...);
    ++launches;
  };
  auto product = [&](int rows, const int64_t* rp, const int* ri, const double* rx,
                     const double* X, double* Y) {
    launch(V == 2 ? bnr_spmm<2> : bnr_spmm<1>, dim3((unsigned)blocks_for((long long)rows * (K / V))),
           dim3(256), rows, K, rp, ri, rx, X, Y);
  };
  for (int it = 0; it < iters; ++it) {
    double* adx = (it & 1) ? b->AdX1 : b->AdX0;              // this step's A dX
    const double* adx_prev = (it & 1) ? b->AdX0 : b->AdX1;   // the previous step's
    const double *c = b->c, *eta = b->eta, *eta_prev = b->eta_prev, *omega = b->omega;
    const int* pend = b->accept;
    // an empty side has no rows to step and no sums to write
    if (fused) {
      if (nblocks > 0)
        launch(V == 2 ? bnr_cols<2> : bnr_cols<1>, dim3((unsigned)nblocks, tiles), dim3(kBnrThreads),
               b->n, K, txs, mblocks, pstride, (const int64_t*)b->cp, (const int*)b->ci,
               (const double*)b->cx, c, eta, eta_prev, omega, pend, b->X, b->AtY,
               (const double*)b->dY, (const double*)b->L, (const double*)b->U, b->dX, b->part);
      if (mblocks > 0)
        launch(V == 2 ? bnr_rows<2> : bnr_rows<1>, dim3((unsigned)mblocks, tiles), dim3(kBnrThreads),
               b->m, K, txs, pstride, (const int64_t*)b->rp, (const int*)b->ri,
               (const double*)b->rx, (const double*)b->rl, (const double*)b->ru, eta, eta_prev,
               omega, pend, b->Y, b->AX, adx_prev, (const double*)b->dX, adx, b->dY, b->part);
    } else {
      const unsigned kt = (unsigned)((K + 31) / 32);
      if (nblocks > 0)
        launch(bnr_primal, dim3((unsigned)nblocks, kt), dim3(32, 8), b->n, K, mblocks, pstride,
               c, eta, eta_prev, omega, pend, b->X, b->AtY, (const double*)b->AtdY,
               (const double*)b->L, (const double*)b->U, b->dX, b->part);
      product(b->m, b->rp, b->ri, b->rx, b->dX, adx);
      if (mblocks > 0)
        launch(bnr_dual, dim3((unsigned)mblocks, kt), dim3(32, 8), b->m, K, pstride,
               (const double*)b->rl, (const double*)b->ru, eta, eta_prev, omega, pend, b->Y, b->AX,
               adx_prev, (const double*)adx, b->dY, b->part);
      if (it + 1 < iters) product(b->n, b->cp, b->ci, b->cx, b->dY, b->AtdY);
    }
    launch(bnr_accept, dim3((unsigned)((K + 3) / 4)), dim3(128), K, mblocks, nblocks,
           (const double*)b->part, b->eta, b->eta_prev, omega, b->accept,
           (const double*)(b->fac + 2 * it));
  }
  return launches;
}

}  // namespace

extern "C" {

int pdlp_bnr_create(const pdlp_problem_desc* P, double obj_scale, int32_t max_batch,
                    void* stream, pdlp_bnr** out) {
  if (!P || !out) return fail(PDLP_ERR_ARG, "NULL problem or output");
  *out = nullptr;
  if (P->m < 0 || P->n < 0 || P->nnz < 0) return fail(PDLP_ERR_ARG, "negative dimension");
  if (P->nnz > 0x7fffffffLL) return fail(PDLP_ERR_ARG, "nnz must fit in int32");
  if (P->memory != PDLP_MEM_HOST && P->memory != PDLP_MEM_DEVICE)
    return fail(PDLP_ERR_ARG, "memory must be PDLP_MEM_HOST or PDLP_MEM_DEVICE");
  if (!(obj_scale > 0.0) || !std::isfinite(obj_scale)) return fail(PDLP_ERR_ARG, "obj_scale must be positive");
  pdlp_bnr* b = new pdlp_bnr();
  b->stream = (cudaStream_t)stream;
  b->m = P->m; b->n = P->n; b->nnz = P->nnz;
  b->obj_scale = obj_scale;
  b->obj_offset = P->obj_offset;
  cudaStream_t st = b->stream;
  int rc = PDLP_OK;
  const int mem = P->memory;
  if ((rc = bnr_upload(&b->rp, P->rp, (size_t)P->m + 1, mem, st)) ||
      (rc = bnr_upload(&b->ri, P->ri, (size_t)P->nnz, mem, st)) ||
      (rc = bnr_upload(&b->rx, P->rx, (size_t)P->nnz, mem, st)) ||
      (rc = bnr_upload(&b->cp, P->cp, (size_t)P->n + 1, mem, st)) ||
      (rc = bnr_upload(&b->ci, P->ci, (size_t)P->nnz, mem, st)) ||
      (rc = bnr_upload(&b->cx, P->cx, (size_t)P->nnz, mem, st)) ||
      (rc = bnr_upload(&b->c, P->c, (size_t)P->n, mem, st)) ||
      (rc = bnr_upload(&b->rl, P->row_lb, (size_t)P->m, mem, st)) ||
      (rc = bnr_upload(&b->ru, P->row_ub, (size_t)P->m, mem, st)) ||
      (rc = bnr_ensure(b, std::max(1, (int)max_batch)))) {
    pdlp_bnr_destroy(b);
    return rc;
  }
  cudaError_t e = cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) { pdlp_bnr_destroy(b); return cuda_fail(e, "bnr create"); }
  *out = b;
  return PDLP_OK;
}

int pdlp_bnr_destroy(pdlp_bnr* b) {
  if (!b) return PDLP_OK;
  cudaStreamSynchronize(b->stream);
  bnr_free_blocks(b);
  void* arrays[] = {b->rp, b->ri, b->rx, b->cp, b->ci, b->cx, b->c, b->rl, b->ru};
  for (void* a : arrays) cudaFree(a);
  cudaFree(b->fac);
  if (b->cap_stream) cudaStreamDestroy(b->cap_stream);
  delete b;
  return PDLP_OK;
}

int pdlp_bnr_solve_batch(pdlp_bnr* b, int32_t K, const double* col_lb, const double* col_ub,
                         const double* warm_x, const double* warm_y, int32_t iters,
                         double step_growth, double step_damp, double* bounds, double* x,
                         double* y, uint8_t* infeasible, int32_t memory) {
  if (!b) return fail(PDLP_ERR_ARG, "NULL handle");
  if (K <= 0 || iters < 0) return fail(PDLP_ERR_ARG, "K must be positive and iters >= 0");
  if (!col_lb || !col_ub) return fail(PDLP_ERR_ARG, "col_lb / col_ub are NULL");
  if (memory != PDLP_MEM_HOST && memory != PDLP_MEM_DEVICE)
    return fail(PDLP_ERR_ARG, "memory must be PDLP_MEM_HOST or PDLP_MEM_DEVICE");
  if ((warm_x == nullptr) != (warm_y == nullptr)) return fail(PDLP_ERR_ARG, "warm_x and warm_y go together");
  int rc = bnr_ensure(b, K);
  if (rc) return rc;
  cudaStream_t st = b->stream;
  const cudaMemcpyKind in = memory == PDLP_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind outk = memory == PDLP_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  const size_t nk = (size_t)b->n * K, mk = (size_t)b->m * K;
  if (nk) {
    PDLP_CUDA(cudaMemcpyAsync(b->L, col_lb, sizeof(double) * nk, in, st));
    PDLP_CUDA(cudaMemcpyAsync(b->U, col_ub, sizeof(double) * nk, in, st));
  }
  if (warm_x) {
    if (nk) PDLP_CUDA(cudaMemcpyAsync(b->X, warm_x, sizeof(double) * nk, in, st));
    if (mk) PDLP_CUDA(cudaMemcpyAsync(b->Y, warm_y, sizeof(double) * mk, in, st));
  } else {
    if (nk) PDLP_CUDA(cudaMemsetAsync(b->X, 0, sizeof(double) * nk, st));
    if (mk) PDLP_CUDA(cudaMemsetAsync(b->Y, 0, sizeof(double) * mk, st));
  }
  // no trial pending at the start
  PDLP_CUDA(cudaMemsetAsync(b->accept, 0, sizeof(int) * K, st));
  PDLP_CUDA(cudaMemcpyAsync(b->eta, b->h_eta.data(), sizeof(double) * K, cudaMemcpyHostToDevice, st));
  PDLP_CUDA(cudaMemcpyAsync(b->omega, b->h_omega.data(), sizeof(double) * K, cudaMemcpyHostToDevice, st));
  PDLP_CUDA(cudaMemcpyAsync(b->eta_prev, b->h_eta.data(), sizeof(double) * K, cudaMemcpyHostToDevice, st));
  // X = clip(X, L, U); AX = A X; AtY = A^T Y
  bnr_clip<<<blocks_for((long long)nk), 256, 0, st>>>((long long)nk, b->X, b->L, b->U);
  launch_spmm(b->m, K, b->rp, b->ri, b->rx, b->X, b->AX, st);
  launch_spmm(b->n, K, b->cp, b->ci, b->cx, b->Y, b->AtY, st);
  count_launches(3);
  PDLP_CUDA(cudaGetLastError());
  // the iterations, from a graph captured once per (K, iters, exponents)
  if (iters > 0) {
    if (!b->graph || b->g_k != K || b->g_iters != iters || b->g_growth != step_growth ||
        b->g_damp != step_damp) {
      if (b->graph) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }
      // the step-size factors of iteration i use t = i + 2 (attempts + 1,
      // bnr.py:267), with the host's pow as in the reference
      std::vector<double> fac(2 * (size_t)iters);
      for (int it = 0; it < iters; ++it) {
        const double t = (double)(it + 2);
        fac[2 * it] = 1.0 - std::pow(t, -step_growth);
        fac[2 * it + 1] = 1.0 + std::pow(t, -step_damp);
      }
      PDLP_CUDA(cudaStreamSynchronize(st));
      cudaFree(b->fac);
      b->fac = nullptr;
      PDLP_CUDA(cudaMalloc(&b->fac, sizeof(double) * fac.size()));
      PDLP_CUDA(cudaMemcpy(b->fac, fac.data(), sizeof(double) * fac.size(), cudaMemcpyHostToDevice));
      PDLP_CUDA(cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeThreadLocal));
      b->g_launches = bnr_enqueue_iterations(b, K, iters, b->cap_stream);
      cudaGraph_t g = nullptr;
      const cudaError_t le = cudaGetLastError();
      const cudaError_t ce = cudaStreamEndCapture(b->cap_stream, &g);
      if (le != cudaSuccess) { if (g) cudaGraphDestroy(g); return cuda_fail(le, "bnr capture"); }
      if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
      const cudaError_t ie = cudaGraphInstantiate(&b->graph, g, 0);
      cudaGraphDestroy(g);
      if (ie != cudaSuccess) { b->graph = nullptr; return cuda_fail(ie, "cudaGraphInstantiate"); }
      b->g_k = K; b->g_iters = iters; b->g_growth = step_growth; b->g_damp = step_damp;
    }
    PDLP_CUDA(cudaGraphLaunch(b->graph, st));
    count_launches(b->g_launches);
  }
  // each node's final iterates, into dX (x) and dY (y); the last step's
  // A dX is in AdX[(iters - 1) % 2]
  bnr_resolve_x<<<blocks_for((long long)nk), 256, 0, st>>>(
      (long long)nk, K, b->accept, b->eta_prev, b->omega, b->c, b->X, b->AtY, b->L, b->U, b->dX);
  bnr_resolve_y<<<blocks_for((long long)mk), 256, 0, st>>>(
      (long long)mk, K, b->accept, b->eta_prev, b->omega, b->rl, b->ru, b->Y, b->AX,
      ((iters - 1) & 1) ? b->AdX1 : b->AdX0, b->dY);
  // the bound: A^T Y, its terms, then per node (safebound.py:194-235)
  const int mblocks = (b->m + kRowsPerBlock - 1) / kRowsPerBlock;
  const int nblocks = (b->n + kRowsPerBlock - 1) / kRowsPerBlock;
  launch_spmm(b->n, K, b->cp, b->ci, b->cx, b->dY, b->AtdY, st);
  bnr_bound_terms<<<dim3(std::max(1, mblocks + nblocks), (K + 31) / 32), dim3(32, 8), 0, st>>>(
      b->m, b->n, K, mblocks, mblocks + nblocks + 1, b->dY, b->rl, b->ru, b->c, b->AtdY, b->L,
      b->U, b->part);
  bnr_bound_final<<<(K + 3) / 4, 128, 0, st>>>(K, mblocks, nblocks, b->part, b->obj_offset,
                                               b->obj_scale, b->bounds, b->empty);
  count_launches(5);
  PDLP_CUDA(cudaGetLastError());
  // outputs; the step sizes stay with the engine for the next call
  if (bounds) PDLP_CUDA(cudaMemcpyAsync(bounds, b->bounds, sizeof(double) * K, outk, st));
  if (x && nk) PDLP_CUDA(cudaMemcpyAsync(x, b->dX, sizeof(double) * nk, outk, st));
  if (y && mk) PDLP_CUDA(cudaMemcpyAsync(y, b->dY, sizeof(double) * mk, outk, st));
  if (infeasible) PDLP_CUDA(cudaMemcpyAsync(infeasible, b->empty, (size_t)K, outk, st));
  PDLP_CUDA(cudaMemcpyAsync(b->h_eta.data(), b->eta, sizeof(double) * K, cudaMemcpyDeviceToHost, st));
  PDLP_CUDA(cudaStreamSynchronize(st));
  return PDLP_OK;
}

int pdlp_bnr_step_sizes(pdlp_bnr* b, int32_t K, double* eta, double* omega) {
  if (!b || K < 0) return fail(PDLP_ERR_ARG, "NULL handle or negative K");
  if (K > b->cap) return fail(PDLP_ERR_ARG, "K beyond the engine's capacity");
  for (int i = 0; i < K; ++i) {
    if (eta) eta[i] = b->h_eta[i];
    if (omega) omega[i] = b->h_omega[i];
  }
  return PDLP_OK;
}

}  // extern "C"
