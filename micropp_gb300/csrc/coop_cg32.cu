// coop_cg32.cu -- the mixed form's FP32 CG solves (1 or 6 right-hand sides, Jacobi or multigrid preconditioner),
// all iterations with their V-cycles in one cooperative launch.
//
// For batches that do not fill the GPU an iteration launched kernel by kernel is bound by latency: a V-cycle is
// about 12 launches, and a stencil kernel with one node per thread takes 15-50 us however small its grid, since a
// thread walks its 27 slots and 3 rows in turn on a few SMs.  Here a group of G blocks owns an instance and goes
// through the phases of its iterations with a barrier between them, and the rows of 32 nodes (a unit) are spread over
// 3 warps: one row of each node per warp with one right-hand side, two right-hand sides per warp with six.
//  - A unit's matrix values (243 rows of 128 bytes) go to shared memory by asynchronous copies, which need no
//    registers: about 190 KB per SM in flight.  A block whose units all fit keeps them for the whole solve (about
//    29,000 nodes on all SMs); a pass then waits for its vector entries only.
//  - The coarsest levels that fit in one block's shared memory (the tail) are its block's alone, from the
//    restriction to the interpolation: no barrier between their many short phases.
// Level-0 units are dealt to the blocks in runs, so that neighbouring units share vector rows in L1.  The level-0
// vectors of the 1-RHS solve are component-major here, as those of the 6-RHS solve (du32 and kinv32 alone stay
// node-interleaved): 32 nodes are one 128-byte access.
//
// A sum over an instance is formed over V parts, the blocks of a solve that has all SMs.  With fewer blocks (other handles
// are at work) a block has several parts and forms the sum of each as a block of its own would: the result does not depend
// on what else runs.  That is a kernel of its own (SHARED): in one body the solve with a part per block was 1.5-3% slower.
//
// Arithmetic: every FP32 sum -- the products of a row, a thread's part of a dot product, the 32 lanes of a warp --
// is formed as in the launched kernels (mixed_kernels.cu, mg_kernels.cu), in their order; the FP64 sums above a warp
// are not, which changes an FP32 scalar once in 1e8 or so.  The outputs of the two forms are the same but for that.
#include <cuda_runtime.h>

#include "coop.cuh"
#include "device.cuh"
#include "launch.h"

namespace mgb {
namespace {

// Warps of a block, a multiple of 6 (a warp's dot products are those of one right-hand side): 18 at 96 registers, for
// the vector entries that a thread has in flight.
constexpr int kWarps = 18, kThreads = 32 * kWarps;
constexpr int kSubs = 3, kGroups = kWarps / kSubs;  // warps per unit; units a block works on at a time
constexpr int kUnitFloats = kEllPerNode * 32;       // matrix values of a unit; each group of 3 warps holds one
constexpr int kHeldFloats = kGroups * kUnitFloats;
// Blocks per instance from which one of them keeps to the tail: below, a block more for the other levels is worth more.
constexpr int kTailBlocks = 8;

// Parts of the sums that a block sets down between two __syncthreads.
constexpr int kPass = 8;

// Batches solved by one cooperative launch: at most kCoopNodes nodes in all and kTailBlocks blocks for each instance,
// or with the V-cycle half as many blocks and kCoopNodesFew nodes.  One homogenization (stress and ctan, damage,
// multigrid), launched and here, ms: 60^3 x 1 20.3 and 14.5, x 4 47.3 and 44.5; 40^3 x 8 33.1 and 28.3, x 16 53.7 and
// 55.4; 30^3 x 32 46.9 and 49.2; 20^3 x 32 21.1 and 18.4, x 100 50.9 and 56.4; 10^3 x 32 9.7 and 5.9, x 200 25.2 and
// 26.6; Jacobi 20^3 x 32 24.2 and 25.2, 40^3 x 4 41.6 and 40.0.
//
// Handles homogenized together (launched, one launch with a share of the SMs, one launch with all of them; ms): multigrid,
// a point of 30^3 each, x 4 19.7, 11.6, 15.1, x 16 48.3, 33.6, 53.2; 40^3 x 16 82.3, 65.7, 82.7.  Jacobi 30^3 x 4 24.5,
// 18.6, 24.0, x 8 32.6, 31.8, 45.6, 40^3 x 3 36.4, 35.3, 38.1; above kCoopBeside nodes in all its solves are launched: 40^3 x
// 4 40.0, 45.1, 50.3, 30^3 x 16 54.8, 57.4, 87.2, 60^3 x 4 163, 200, 224 -- without the V-cycle's latencies the products
// bound an iteration, and those of six right-hand sides are slower here.
constexpr long long kCoopNodes = 950000, kCoopNodesFew = 300000, kCoopBeside = 250000;

// Nodes per warp of the launched kernels' dot products, in units of 32: blocks own whole multiples.
__host__ __device__ constexpr int own_units(int nr) { return nr == 1 ? 4 : 2; }

struct Grid {
  int nx, ny, nz, nxny, nn, np, units;
  int ix, iy, inner, iunits;  // interior nodes along x and y, interior nodes, units of 32 of them
};

struct Levels {
  Grid g[kMgMaxLevels];
  int n;     // levels of the V-cycle (1: Jacobi preconditioner)
  int tail;  // first level of the tail (n: none)
};

// A level of the tail in shared memory: the rows of its interior nodes, iterate and residual on all its nodes (zero on
// the boundary) and the right-hand side and inverse diagonal on the interior ones.
struct TailLevel {
  int A, x, t, b, k;  // offsets in the block's shared memory
  int si, sn;         // strides of a component on the interior nodes and on all nodes
};

__host__ __device__ inline int tail_floats(const Grid &g, int nr) {
  return g.inner * (kEllPerNode + 3 * nr + 3) + 2 * 3 * nr * g.nn;
}

// What the phases of a solve share, at the start of the block's shared memory.  The phases are functions of their own
// that read it: in one body their pointers and indices would take the registers of the products.
struct Ctx {
  Levels lv;
  MgInst mg;
  TailLevel tail[kMgMaxLevels];
  float *R, *Z, *P, *AP, *D, *T, *kinv;
  const float *ks, *vals;
  const double *b;
  double *red;
  unsigned int *ctr, polls;
  uint64_t policy;  // L2 eviction priority of the matrix values
  double min_err, rel_err;
  double tot[12], rz[6], pn0[6];
  float alpha[6], beta[6];
  int rdone[6], done, ok, bad;
  int held[kGroups];  // the unit (level << 24 | unit) whose values each group of 3 warps holds
  int me, workers;    // this block among those that work on the levels before the tail (me = -1: the tail's block)
  int u0, u1;         // its level-0 units, those of its parts v0 .. v1 - 1
  int V, v0, v1;
  int idle;           // parts without level-0 units: 1 where a solve with all SMs has a block for the tail
  int pairs;
  double warp[2][kPass][kWarps];
};
constexpr int kCtxBytes = (sizeof(Ctx) + 127) / 128 * 128;

extern __shared__ __align__(128) char g_smem[];
__device__ __forceinline__ Ctx &ctx() { return *reinterpret_cast<Ctx *>(g_smem); }
__device__ __forceinline__ float *held_values() { return reinterpret_cast<float *>(g_smem + kCtxBytes); }

__device__ __forceinline__ bool on_bnd(const Grid &g, int n) {
  const int i = n % g.nx, j = (n / g.nx) % g.ny, k = n / g.nxny;
  return i == 0 || j == 0 || k == 0 || i == g.nx - 1 || j == g.ny - 1 || k == g.nz - 1;
}

// The t-th interior node (t < g.inner) and its coordinates.
__device__ __forceinline__ int inner_node(const Grid &g, int t, int &i, int &j, int &k) {
  i = t % g.ix + 1;
  j = (t / g.ix) % g.iy + 1;
  k = t / (g.ix * g.iy) + 1;
  return k * g.nxny + j * g.nx + i;
}

// Lane 0: the sum over the warp, in warp_sum's order (reduce.cuh).
__device__ __forceinline__ float lane0_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Rows of a node that a warp forms: with one right-hand side row `sub`; with six the 3 rows of the right-hand sides
// 2 sub and 2 sub + 1.
template <int NR>
struct Share {
  static constexpr int kOut = NR == 1 ? 1 : 6;
  static __device__ __forceinline__ int comp(int sub, int o) { return NR == 1 ? sub : sub * 6 + o; }
};

// y = the warp's rows of A x at interior node n; products in the order of the slots, then the columns.  value(e): entry
// e = s * 9 + fi * 3 + fj of the node's rows.  x is component-major with component stride np; it was written by this
// kernel before a barrier and is read with ordinary loads.
template <int NR, class V>
__device__ __forceinline__ void row_products(int nx, int nxny, size_t np, V value, const float *x, int n, int sub,
                                             float (&y)[Share<NR>::kOut]) {
#pragma unroll
  for (int o = 0; o < Share<NR>::kOut; ++o) y[o] = 0.f;
  if constexpr (NR == 1) {
#pragma unroll 1
    for (int dz = 0; dz < 3; ++dz) {
      const float *xb = x + n + (dz - 1) * nxny - nx - 1;
      float K[27], xv[27];
#pragma unroll
      for (int q = 0; q < 27; ++q) xv[q] = xb[(size_t)(q % 3) * np + (q / 9) * nx + (q / 3) % 3];
#pragma unroll
      for (int q = 0; q < 27; ++q) K[q] = value((dz * 9 + q / 3) * 9 + sub * 3 + q % 3);
#pragma unroll
      for (int q = 0; q < 27; ++q) y[0] = fmaf(K[q], xv[q], y[0]);
    }
  } else {
    const float *xc = x + (size_t)(sub * 6) * np + n - 1;
#pragma unroll 1
    for (int dz = 0; dz < 3; ++dz) {
      const float *xb = xc + (dz - 1) * nxny - nx;
      float xv[3][2][3][3];
#pragma unroll
      for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int d = 0; d < 3; ++d) xv[dy][p][dx][d] = xb[(size_t)(p * 3 + d) * np + dy * nx + dx];
#pragma unroll
      for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
          for (int e = 0; e < 9; ++e) {
            const float K = value(((dz * 3 + dy) * 3 + dx) * 9 + e);
#pragma unroll
            for (int p = 0; p < 2; ++p) y[p * 3 + e / 3] = fmaf(K, xv[dy][p][dx][e % 3], y[p * 3 + e / 3]);
          }
    }
  }
}

// The matrix values of unit u to shared memory, by the 96 threads of a group of which this is the t-th; finished by the
// caller's cp_wait and barrier.  policy: the L2 eviction priority (see keep_fraction), 0 for the usual one.
__device__ __forceinline__ void copy_unit(float *dst, const float *vals, size_t np, int u, int t, uint64_t policy) {
  constexpr int kStep = 32 * kSubs / 8;  // rows per round of the group's threads, 8 of them to a row
  unsigned int d = (unsigned int)__cvta_generic_to_shared(dst + t * 4);
  const float *src = vals + (size_t)(t >> 3) * np + u * 32 + (t & 7) * 4;
  const size_t step = kStep * np;
  if (policy) {
    for (int row = t >> 3; row < kEllPerNode; row += kStep, d += kStep * 128, src += step)
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "l"(policy)
                   : "memory");
  } else {
    for (int row = t >> 3; row < kEllPerNode; row += kStep, d += kStep * 128, src += step)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  }
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float half_pow(int a) { return a == 0 ? 1.0f : 0.5f; }

// sum over the fine nodes around the coarse node at tc (2 x its coordinates on grid f): P^T t
__device__ __forceinline__ float restricted(const float *tc, const Grid &f) {
  float v[27], acc = 0.f;
#pragma unroll
  for (int q = 0; q < 27; ++q) v[q] = tc[(q / 9 - 1) * f.nxny + ((q / 3) % 3 - 1) * f.nx + q % 3 - 1];
#pragma unroll
  for (int q = 0; q < 27; ++q)
    acc = fmaf(half_pow(q % 3 - 1) * half_pow((q / 3) % 3 - 1) * half_pow(q / 9 - 1), v[q], acc);
  return acc;
}

// x + (P xc)(i, j, k): xc on the coarse grid gc.  All 8 loads go out together; a coordinate that is even has one
// parent, and the loads of the second are of the first again and unused.
__device__ __forceinline__ float interpolate(float x, const float *xc, const Grid &gc, int i, int j, int k) {
  const int oi = i & 1, oj = j & 1, ok = k & 1;
  const float w = (oi ? 0.5f : 1.f) * (oj ? 0.5f : 1.f) * (ok ? 0.5f : 1.f);
  const float *xq = xc + ((k >> 1) * gc.ny + (j >> 1)) * gc.nx + (i >> 1);
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = xq[(ok & (q >> 2)) * gc.nxny + (oj & (q >> 1)) * gc.nx + (oi & q)];
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if ((q & 1) <= oi && ((q >> 1) & 1) <= oj && (q >> 2) <= ok) x = fmaf(w, v[q], x);
  return x;
}

// The stencil phases.  in / out pick x, y or t of a coarse level (kSmooth).
enum Op {
  kResid,    // t = b - A x
  kSmooth,   // out = in + D^-1 (b - A in)
  kProduct,  // AP = A P, P itself on boundary nodes (level 0)
  kPost      // Z = t + D^-1 (R - A t) (level 0)
};

// One function for all of them, its products in a loop over the planes of the stencil, which keeps the solve's code
// small.
template <int NR>
__device__ __noinline__ void apply(int op, int l, int in_sel, int out_sel) {
  constexpr int kOut = Share<NR>::kOut;
  Ctx &c = ctx();
  if (c.me < 0) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, group = wid / kSubs, sub = wid - group * kSubs;
  const Grid &g = c.lv.g[l];
  const MgLevel &m = c.mg.lv[l];
  const size_t np = g.np;
  const float *A = l == 0 ? c.vals : m.vals;
  const float *x, *b = l == 0 ? c.R : m.b, *kd = l == 0 ? c.ks : m.kinv;
  float *out;
  if (op == kProduct) {
    x = c.P;
    out = c.AP;
  } else if (op == kPost) {
    x = c.T;
    out = c.Z;
  } else if (op == kResid) {
    x = l == 0 ? c.Z : m.x;
    out = m.t;
  } else {
    x = in_sel == 0 ? m.x : in_sel == 1 ? m.y : m.t;
    out = out_sel == 0 ? m.x : m.y;
  }
  const int first = l == 0 ? c.u0 : c.me, step = l == 0 ? 1 : c.workers, end = l == 0 ? c.u1 : g.units;
  int index = 0;  // of the level's first unit among the worker's units of all levels
  if (l > 0) {
    index = c.u1 - c.u0;
    for (int f = 1; f < l; ++f) index += (c.lv.g[f].units - c.me + c.workers - 1) / c.workers;
  }
  float *buf = held_values() + group * kUnitFloats;
  // the worker's units in turn over the groups of 3 warps, so that each keeps its own while there are no more
  int k = group - index % kGroups;
  if (k < 0) k += kGroups;
  for (; first + k * step < end; k += kGroups) {
    const int u = first + k * step, n = u * 32 + lane, want = l << 24 | u;
    if (c.held[group] != want) {
      asm volatile("bar.sync %0, 96;" ::"r"(group + 1) : "memory");
      copy_unit(buf, A, np, u, sub * 32 + lane, c.policy);
      if (sub == 0 && lane == 0) c.held[group] = want;
      cp_wait();
      asm volatile("bar.sync %0, 96;" ::"r"(group + 1) : "memory");
    }
    const bool live = n < g.nn, interior = live && !on_bnd(g, n);
    float y[kOut] = {};
    const float *v = buf + lane;
    if (interior) row_products<NR>(g.nx, g.nxny, np, [&](int e) { return v[e * 32]; }, x, n, sub, y);
    if (!live) continue;
    if (op == kProduct) {
#pragma unroll
      for (int q = 0; q < kOut; ++q) {
        const size_t o = (size_t)Share<NR>::comp(sub, q) * np + n;
        out[o] = interior ? y[q] : x[o];
      }
      continue;
    }
    float bv[kOut], kv[kOut], xv[kOut];
#pragma unroll
    for (int q = 0; q < kOut; ++q) {
      const int cc = Share<NR>::comp(sub, q);
      const size_t o = (size_t)cc * np + n;
      bv[q] = b[o];
      kv[q] = kd[(size_t)n * 3 + (NR == 1 ? cc : q % 3)];
      xv[q] = x[o];
    }
#pragma unroll
    for (int q = 0; q < kOut; ++q) {
      const float v = op == kResid ? bv[q] - y[q] : fmaf(kv[q], bv[q] - y[q], xv[q]);
      out[(size_t)Share<NR>::comp(sub, q) * np + n] = interior ? v : 0.f;
    }
  }
}

// b_{l+1} = P^T t_l, x_{l+1} = D^-1 b_{l+1} on the interior nodes of level l + 1 (the others stay zero)
template <int NR>
__device__ __noinline__ void restrict_down(int l) {
  constexpr int kComps = 3 * NR;
  Ctx &c = ctx();
  if (c.me < 0) return;
  const Grid &g = c.lv.g[l], &gc = c.lv.g[l + 1];
  const MgLevel &mc = c.mg.lv[l + 1];
  const float *tv = c.mg.lv[l].t;
  for (int it = threadIdx.x >> 5; c.me + (it / kComps) * c.workers < gc.iunits; it += kWarps) {
    const int t = (c.me + (it / kComps) * c.workers) * 32 + (threadIdx.x & 31), cc = it % kComps;
    if (t >= gc.inner) continue;
    int X, Y, W;
    const int n = inner_node(gc, t, X, Y, W);
    const float kv = mc.kinv[(size_t)n * 3 + cc % 3];
    const float acc = restricted(tv + (size_t)cc * g.np + ((2 * W) * g.ny + 2 * Y) * g.nx + 2 * X, g);
    mc.b[(size_t)cc * gc.np + n] = acc;
    mc.x[(size_t)cc * gc.np + n] = kv * acc;
  }
}

// t_l = x_l + P x_{l+1}
template <int NR>
__device__ __noinline__ void prolong_up(int l) {
  Ctx &c = ctx();
  if (c.me < 0) return;
  const Grid &g = c.lv.g[l], &gc = c.lv.g[l + 1];
  const float *xc = c.mg.lv[l + 1].x, *xl = l == 0 ? c.Z : c.mg.lv[l].x;
  float *tv = c.mg.lv[l].t;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (l == 0) {  // every node of the block's units, the 3 components of a right-hand side together
    for (int it = wid; it < (c.u1 - c.u0) * NR; it += kWarps) {
      const int n = (c.u0 + it / NR) * 32 + lane, c0 = it % NR * 3;
      if (n >= g.nn) continue;
      const int i = n % g.nx, j = (n / g.nx) % g.ny, k = n / g.nxny;
      const bool b = i == 0 || j == 0 || k == 0 || i == g.nx - 1 || j == g.ny - 1 || k == g.nz - 1;
      float v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        v[d] = b ? 0.f : interpolate(xl[(size_t)(c0 + d) * g.np + n], xc + (size_t)(c0 + d) * gc.np, gc, i, j, k);
#pragma unroll
      for (int d = 0; d < 3; ++d) tv[(size_t)(c0 + d) * g.np + n] = v[d];
    }
  } else {
    constexpr int kComps = 3 * NR;
    for (int it = wid; c.me + (it / kComps) * c.workers < g.iunits; it += kWarps) {
      const int t = (c.me + (it / kComps) * c.workers) * 32 + lane, cc = it % kComps;
      if (t >= g.inner) continue;
      int i, j, k;
      const int n = inner_node(g, t, i, j, k);
      const size_t q = (size_t)cc * g.np + n;
      tv[q] = interpolate(xl[q], xc + (size_t)cc * gc.np, gc, i, j, k);
    }
  }
}

// On a tail level: out = b - A in (the residual), or in + D^-1 (b - A in)
template <int NR>
__device__ __noinline__ void tail_apply(int l, int in, int out, bool smooth) {
  const Ctx &c = ctx();
  const Grid &g = c.lv.g[l];
  const TailLevel &q = c.tail[l];
  float *sm = held_values();
  const float *A = sm + q.A;
  const int inner = g.inner, nx = g.nx, nxny = g.nxny, si = q.si, sn = q.sn, qb = q.b, qk = q.k;
  for (int o = threadIdx.x; o < inner * kSubs; o += kThreads) {
    const int sub = o / inner, t = o - sub * inner;
    int i, j, k;
    const int n = inner_node(g, t, i, j, k);
    float y[Share<NR>::kOut];
    row_products<NR>(nx, nxny, sn, [&](int e) { return A[e * si + t]; }, sm + in, n, sub, y);
#pragma unroll
    for (int p = 0; p < Share<NR>::kOut; ++p) {
      const int cc = Share<NR>::comp(sub, p), e = cc * sn + n;
      const float r = sm[qb + cc * si + t] - y[p];
      sm[out + e] = smooth ? fmaf(sm[qk + (cc % 3) * si + t], r, sm[in + e]) : r;
    }
  }
  __syncthreads();
}

// The coarsest level's Jacobi sweeps x -> t -> x.  A thread keeps one row, with its 81 values, through all of them: a
// sweep then loads the vector entries only.
template <int NR>
__device__ __noinline__ void tail_sweeps() {
  const Ctx &c = ctx();
  const int l = c.lv.n - 1, pairs = c.pairs, inner = c.lv.g[l].inner;
  const TailLevel &q = c.tail[l];
  const int xs = q.x, ts = q.t;
  if (inner * 3 * NR > kThreads) {
    for (int p = 0; p < pairs; ++p) {
      tail_apply<NR>(l, xs, ts, true);
      tail_apply<NR>(l, ts, xs, true);
    }
    return;
  }
  float *sm = held_values();
  const int cc = threadIdx.x / inner, t = threadIdx.x - cc * inner, nx = c.lv.g[l].nx, nxny = c.lv.g[l].nxny, sn = q.sn;
  const bool live = cc < 3 * NR;
  int i, j, k;
  const int n = inner_node(c.lv.g[l], t, i, j, k), own = cc * sn + n, first = cc / 3 * 3 * sn + n - nxny - nx - 1;
  float K[81], b = 0.f, kd = 0.f, xo = 0.f;
  if (live) {
    const float *A = sm + q.A + cc % 3 * 3 * inner + t;
#pragma unroll
    for (int e = 0; e < 81; ++e) K[e] = A[(e / 3 * 9 + e % 3) * inner];
    b = sm[q.b + cc * inner + t];
    kd = sm[q.k + cc % 3 * inner + t];
    xo = sm[xs + own];
  }
  for (int p = 0; p < 2 * pairs; ++p) {
    if (live) {
      const float *x = sm + ((p & 1) ? ts : xs) + first;
      float y = 0.f;
#pragma unroll
      for (int zy = 0; zy < 9; ++zy) {
        const float *xz = x + (zy / 3) * nxny + (zy % 3) * nx;
#pragma unroll
        for (int e = 0; e < 9; ++e) y = fmaf(K[zy * 9 + e], xz[(e % 3) * sn + e / 3], y);
      }
      xo = fmaf(kd, b - y, xo);
      sm[((p & 1) ? xs : ts) + own] = xo;
    }
    __syncthreads();
  }
}

// b = P^T t of the finer level f (component stride `stride`), x = D^-1 b, on tail level l
template <int NR>
__device__ __noinline__ void tail_restrict(int l, const float *tf, size_t stride) {
  Ctx &c = ctx();
  const Grid &g = c.lv.g[l], &f = c.lv.g[l - 1];
  const TailLevel &q = c.tail[l];
  float *sm = held_values();
  for (int o = threadIdx.x; o < g.inner * 3 * NR; o += kThreads) {
    const int cc = o / g.inner, t = o - cc * g.inner;
    int X, Y, W;
    const int n = inner_node(g, t, X, Y, W);
    const float acc = restricted(tf + (size_t)cc * stride + ((2 * W) * f.ny + 2 * Y) * f.nx + 2 * X, f);
    sm[q.b + cc * q.si + t] = acc;
    sm[q.x + cc * q.sn + n] = sm[q.k + (cc % 3) * q.si + t] * acc;
  }
  __syncthreads();
}

// The tail's levels, from the residual t of the level above it to the iterate of its first level
template <int NR>
__device__ __noinline__ void tail_cycle() {
  Ctx &c = ctx();
  if (c.me >= 0) return;
  const int L = c.lv.n, top = c.lv.tail, tid = threadIdx.x;
  float *sm = held_values();
  tail_restrict<NR>(top, c.mg.lv[top - 1].t, c.lv.g[top - 1].np);
  for (int l = top; l + 1 < L; ++l) {
    tail_apply<NR>(l, c.tail[l].x, c.tail[l].t, false);
    tail_restrict<NR>(l + 1, sm + c.tail[l].t, c.tail[l].sn);
  }
  tail_sweeps<NR>();
  for (int l = L - 2; l >= top; --l) {
    const Grid &g = c.lv.g[l], &gc = c.lv.g[l + 1];
    const TailLevel &q = c.tail[l], &qc = c.tail[l + 1];
    for (int o = tid; o < g.inner * 3 * NR; o += kThreads) {
      const int cc = o / g.inner, t = o - cc * g.inner;
      int i, j, k;
      const int n = inner_node(g, t, i, j, k), e = cc * q.sn + n;
      sm[q.t + e] = interpolate(sm[q.x + e], sm + qc.x + cc * qc.sn, gc, i, j, k);
    }
    __syncthreads();
    tail_apply<NR>(l, q.t, q.x, true);
  }
  const Grid &g = c.lv.g[top];
  for (int o = tid; o < g.inner * 3 * NR; o += kThreads) {
    int i, j, k;
    const int cc = o / g.inner, n = inner_node(g, o - cc * g.inner, i, j, k);
    c.mg.lv[top].x[(size_t)cc * g.np + n] = sm[c.tail[top].x + cc * c.tail[top].sn + n];
  }
}

// The shared memory of the tail's block at the start of a solve.
template <int NR>
__device__ __noinline__ void fill_tail() {
  Ctx &c = ctx();
  const int tid = threadIdx.x;
  float *sm = held_values();
  if (c.me < 0) {
    if (tid == 0) {
      int p = 0;
      for (int l = c.lv.tail; l < c.lv.n; ++l) {
        const Grid &g = c.lv.g[l];
        TailLevel &q = c.tail[l];
        q.si = g.inner;
        q.sn = g.nn;
        q.A = p;
        q.x = q.A + q.si * kEllPerNode;
        q.t = q.x + 3 * NR * q.sn;
        q.b = q.t + 3 * NR * q.sn;
        q.k = q.b + 3 * NR * q.si;
        p = q.k + 3 * q.si;
      }
    }
    __syncthreads();
    for (int l = c.lv.tail; l < c.lv.n; ++l) {
      const Grid &g = c.lv.g[l];
      const TailLevel &q = c.tail[l];
      const MgLevel &m = c.mg.lv[l];
      for (int o = tid; o < g.inner * kEllPerNode; o += kThreads) {
        int i, j, k;
        const int e = o / g.inner, t = o - e * g.inner, n = inner_node(g, t, i, j, k);
        sm[q.A + e * q.si + t] = __ldg(m.vals + (size_t)e * g.np + n);
      }
      for (int o = tid; o < g.inner * 3; o += kThreads) {
        int i, j, k;
        const int d = o / g.inner, t = o - d * g.inner, n = inner_node(g, t, i, j, k);
        sm[q.k + d * q.si + t] = m.kinv[(size_t)n * 3 + d];
      }
      for (int o = tid; o < 2 * 3 * NR * q.sn; o += kThreads) sm[q.x + o] = 0.f;
    }
  }
  __syncthreads();
}

// First level-0 unit of part v (v = V: the end): runs of whole own_units.
template <int NR>
__device__ __forceinline__ int first_unit(const Ctx &c, int v) {
  const int runs = (c.lv.g[0].units + own_units(NR) - 1) / own_units(NR);
  if (v <= c.idle) return 0;
  return min(runs * (v - c.idle) / (c.V - c.idle) * own_units(NR), c.lv.g[0].units);
}

// Level-0 units u0 .. u1 - 1 of the block's part v
template <int NR, bool SHARED>
__device__ __forceinline__ int2 part_units(const Ctx &c, int v) {
  return SHARED ? make_int2(first_unit<NR>(c, v), first_unit<NR>(c, v + 1)) : make_int2(c.u0, c.u1);
}

// Warp `wid`'s share (lane 0) of x.y over the level-0 nodes of part v: `per` nodes per thread, as the launched kernel whose
// sum it is.
template <int NR, bool SHARED>
__device__ __noinline__ double dot0(const float *x, const float *y, int per, int v, int wid) {
  const Ctx &c = ctx();
  const int lane = threadIdx.x & 31, q = wid % NR, nn = c.lv.g[0].nn;
  const int2 u = part_units<NR, SHARED>(c, v);
  const size_t np = c.lv.g[0].np;
  double acc = 0.0;
  for (int w = wid / NR; w * per < u.y - u.x; w += kWarps / NR) {
    const int n = (u.x + w * per) * 32 + lane * per;
    float xv[4][3], yv[4][3], s = 0.f;
#pragma unroll
    for (int p = 0; p < 4; ++p)
      if (p < per && n + p < nn)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const size_t o = (size_t)(q * 3 + d) * np + n + p;
          xv[p][d] = x[o];
          yv[p][d] = y[o];
        }
#pragma unroll
    for (int p = 0; p < 4; ++p)
      if (p < per && n + p < nn)
#pragma unroll
        for (int d = 0; d < 3; ++d) s = fmaf(xv[p][d], yv[p][d], s);
    acc += (double)lane0_sum(s);
  }
  return acc;
}

// D += alpha P; R -= alpha AP; Z = D^-1 R (the V-cycle's start) or kinv R; for warp `wid` of part v, with its share of the
// stop test's norm and, with the Jacobi preconditioner, of r.z.  Rows are dealt to the parts and their warps as the
// launched updates deal them.
template <int NR, bool MG>
__device__ __noinline__ double2 update(int v, int wid) {
  const Ctx &c = ctx();
  const int lane = threadIdx.x & 31, nn = c.lv.g[0].nn;
  const size_t np = c.lv.g[0].np;
  float *R = c.R, *Z = c.Z, *D = c.D;
  const float *P = c.P, *AP = c.AP, *kinv = c.kinv, *ks = c.ks;
  double azz = 0.0, arz = 0.0;
  if (NR == 1) {
    const int nrow = nn * 3, ublocks = (nrow + 1023) / 1024, ustride = ublocks * 256;
    const float al = c.alpha[0];
    for (int w = wid * c.V + v; w < ublocks * 8; w += c.V * kWarps) {
      float zz = 0.f, rz = 0.f, pv[4], av[4], rv[4], dv[4], kv[4], sv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int row = w * 32 + lane + q * ustride, n = row / 3;
        if (row < nrow) {
          const size_t o = (size_t)(row - n * 3) * np + n;
          pv[q] = P[o]; av[q] = AP[o]; rv[q] = R[o]; dv[q] = D[row]; kv[q] = kinv[row];
          if (MG) sv[q] = ks[row];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int row = w * 32 + lane + q * ustride, n = row / 3;
        if (row < nrow) {
          const size_t o = (size_t)(row - n * 3) * np + n;
          D[row] = fmaf(al, pv[q], dv[q]);
          const float r = fmaf(-al, av[q], rv[q]), zj = kv[q] * r, z = MG ? sv[q] * r : zj;
          R[o] = r;
          Z[o] = z;
          zz = fmaf(zj, zj, zz);
          if (!MG) rz = fmaf(r, z, rz);
        }
      }
      azz += (double)lane0_sum(zz);
      if (!MG) arz += (double)lane0_sum(rz);
    }
  } else if (!c.rdone[wid % NR]) {
    const int q = wid % NR, wchunks = (nn + 1023) / 1024 * 8;
    const float al = c.alpha[q];
    for (int w = (wid / NR) * c.V + v; w < wchunks; w += c.V * (kWarps / NR)) {
      const int n0 = (w >> 3) * 1024 + (w & 7) * 32 + lane;
      float zz = 0.f, rz = 0.f;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float pv[4], av[4], rv[4], dv[4], kv[4], sv[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int n = n0 + p * 256;
          const size_t o = (size_t)(q * 3 + d) * np + n;
          if (n < nn) {
            pv[p] = P[o]; av[p] = AP[o]; rv[p] = R[o]; dv[p] = D[o]; kv[p] = kinv[(size_t)n * 3 + d];
            if (MG) sv[p] = ks[(size_t)n * 3 + d];
          }
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int n = n0 + p * 256;
          const size_t o = (size_t)(q * 3 + d) * np + n;
          if (n < nn) {
            D[o] = fmaf(al, pv[p], dv[p]);
            const float r = fmaf(-al, av[p], rv[p]), zj = kv[p] * r, z = MG ? sv[p] * r : zj;
            R[o] = r;
            Z[o] = z;
            zz = fmaf(zj, zj, zz);
            if (!MG) rz = fmaf(r, z, rz);
          }
        }
      }
      azz += (double)lane0_sum(zz);
      if (!MG) arz += (double)lane0_sum(rz);
    }
  }
  return make_double2(azz, arz);
}

// P = Z + beta P (start: P = Z) on the block's own nodes
template <int NR>
__device__ __noinline__ void direction(bool start) {
  const Ctx &c = ctx();
  const int len = (c.u1 - c.u0) * 8, total = len * 3 * NR;  // float4 per component and in all
  const size_t np4 = c.lv.g[0].np / 4;
  float4 *P4 = reinterpret_cast<float4 *>(c.P) + c.u0 * 8;
  const float4 *Z4 = reinterpret_cast<const float4 *>(c.Z) + c.u0 * 8;
  for (int it = threadIdx.x; it < total; it += 4 * kThreads) {
    float4 pv[4], zv[4];
    size_t o[4];
    float beta[4];
    bool live[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = it + q * kThreads, cc = e / len;
      live[q] = e < total && !c.rdone[cc / 3];
      if (!live[q]) continue;
      o[q] = cc * np4 + (e - cc * len);
      beta[q] = c.beta[cc / 3];
      zv[q] = Z4[o[q]];
      if (!start) pv[q] = P4[o[q]];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!live[q]) continue;
      const float4 z = zv[q], w = pv[q];
      P4[o[q]] = start ? z
                       : make_float4(fmaf(beta[q], w.x, z.x), fmaf(beta[q], w.y, z.y), fmaf(beta[q], w.z, z.z),
                                     fmaf(beta[q], w.w, z.w));
    }
  }
}

// Start of a 1-RHS solve: R = b, D = 0, the inverse diagonal, Z (P) and the share of warp `wid` of part v of ||kinv r||^2
// and r.z
template <bool MG, bool SHARED>
__device__ __noinline__ double2 setup1(int v, int wid) {
  const Ctx &c = ctx();
  const Grid &g = c.lv.g[0];
  const int2 units = part_units<1, SHARED>(c, v);
  const int lane = threadIdx.x & 31;
  const size_t np = g.np;
  double azz = 0.0, arz = 0.0;
  for (int u = units.x + wid; u < units.y; u += kWarps) {
    const int n = u * 32 + lane;
    float zz = 0.f, rz = 0.f;
    if (n < g.nn) {
      const bool b = on_bnd(g, n);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const size_t o = (size_t)d * np + n, row = (size_t)n * 3 + d;
        const float kd = b ? 1.0f : 1.0f / c.vals[(size_t)(13 * 9 + d * 4) * np + n];
        const float r = (float)c.b[row], zj = kd * r, z = MG ? c.ks[row] * r : zj;
        c.kinv[row] = kd;
        c.D[row] = 0.f;
        c.R[o] = r;
        c.Z[o] = z;
        if (!MG) c.P[o] = z;
        rz = fmaf(r, z, rz);
        zz = fmaf(zj, zj, zz);
      }
    }
    azz += (double)lane0_sum(zz);
    arz += (double)lane0_sum(rz);
  }
  return make_double2(azz, arz);
}

template <int NR, bool MG, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
    k_coop_cg32(Levels lv, const Inst *insts, const int *list, int G, int V, int idle, const double *rel_tols,
                double abs_tol, int max_its_arg, int pairs, float keep) {
  Ctx &c = ctx();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int a = blockIdx.x / G, rank = blockIdx.x - a * G;
  const bool tail = MG && lv.tail < lv.n;
  if (tid == 0) {
    // rank 0 keeps to the tail; the units of the other levels go to the workers, on level 0 by the parts of the sums
    c.lv = lv;
    c.V = V;
    c.idle = idle;
    c.pairs = pairs;
    uint64_t policy = 0;
    if (keep < 1.f)
      asm volatile("createpolicy.fractional.L2::evict_normal.L2::evict_first.b64 %0, %1;" : "=l"(policy) : "f"(keep));
    c.policy = policy;
    c.workers = tail ? G - 1 : G;
    c.me = tail ? rank - 1 : rank;
    const int first = tail ? 1 : 0;  // parts of rank 0 alone
    c.v0 = c.me < 0 ? 0 : first + (V - first) * c.me / c.workers;
    c.v1 = c.me < 0 ? 1 : first + (V - first) * (c.me + 1) / c.workers;
    c.u0 = first_unit<NR>(c, c.v0);
    c.u1 = first_unit<NR>(c, c.v1);
  }
  const Inst &I = insts[list[a]];
  Cg6State *c6s = I.cg6;
  if (NR == 6 && c6s->all_done) return;
  const int max_its = NR == 1 ? max_its_arg : c6s->max_its;
  __syncthreads();
  if (MG)
    for (int q = tid; q < (int)(sizeof(MgInst) / 4); q += kThreads)
      reinterpret_cast<int *>(&c.mg)[q] = reinterpret_cast<const int *>(I.mg)[q];
  if (NR == 6 && tid < 6) {
    c.rz[tid] = c6s->rz[tid];
    c.pn0[tid] = c6s->pnorm0[tid];
    c.rdone[tid] = c6s->done[tid];
  }
  if (tid < kGroups) c.held[tid] = -1;
  if (tid == 0) {
    c.R = NR == 1 ? I.r32 : I.R6;
    c.Z = NR == 1 ? I.z32 : I.Z6;
    c.P = NR == 1 ? I.p32 : I.P6;
    c.AP = NR == 1 ? I.Ap32 : I.AP6;
    c.D = NR == 1 ? I.du32 : I.D6;
    c.T = MG ? I.mg->lv[0].t : nullptr;
    c.kinv = I.kinv32;
    c.ks = MG ? I.mg->lv[0].kinv : I.kinv32;
    c.vals = I.vals32;
    c.b = I.b;
    c.red = I.red;
    c.ctr = I.ticket;
    c.polls = I.polls ? I.polls : kSpinLimit;
    c.min_err = NR == 1 ? abs_tol : c6s->min_err;
    c.rel_err = NR == 1 ? rel_tols[a] : c6s->rel_err;
    if (NR == 1) c.rdone[0] = 0;
    c.done = c.bad = 0;
  }
  __syncthreads();
  unsigned int target = 0;
  int its = 0, turn = 0;
  bool ok = true;
  auto barrier = [&]() {
    target += G;
    ok = group_barrier(c.ctr, target, &c.ok, c.polls);
    return ok;
  };
  // Sums over the instance of what share(v, w) returns in lane 0 for warp w of the block's part v (the values of warp w
  // belong to right-hand side w % NR): a barrier, after which c.tot[kind * NR + q] holds them.  Two buffers of partials in
  // turn: a block may write the next ones while another still reads these.
  auto reduce = [&](auto share, int kinds) {
    double *part = c.red + (size_t)turn * 2 * NR * V;
    turn ^= 1;
    // sum k of part p0 + i
    auto set_down = [&](int p0, int i, int k) {
      const int kind = k / NR, q = k - kind * NR;
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps / NR; ++w) v += c.warp[kind][i][w * NR + q];
      part[(size_t)k * V + p0 + i] = v;
    };
    auto keep_share = [&](double2 r, int i, int w) {
      if (lane == 0) {
        c.warp[0][i][w] = r.x;
        c.warp[1][i][w] = r.y;
      }
    };
    if constexpr (SHARED) {
      for (int p0 = c.v0; p0 < c.v1; p0 += kPass) {
        const int n = min(kPass, c.v1 - p0);
        // a part has fewer units than warps: the warps take turns at the first ones
        for (int i = 0, w = wid; i < n; ++i, w = w < kWarps - 6 ? w + 6 : w + 6 - kWarps) keep_share(share(p0 + i, w), i, w);
        __syncthreads();
        for (int e = tid; e < kinds * NR * n; e += kThreads) set_down(p0, e / (kinds * NR), e % (kinds * NR));
        if (p0 + kPass < c.v1) __syncthreads();
      }
    } else {
      keep_share(share(rank, wid), 0, wid);
      __syncthreads();
      if (tid < kinds * NR) set_down(rank, 0, tid);
    }
    if (!barrier()) return false;
    if (wid < kinds * NR) {
      double v = 0.0;
      for (int b = lane; b < V; b += 32) v += __ldcg(part + (size_t)wid * V + b);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) c.tot[wid] = v;
    }
    __syncthreads();
    return true;
  };
  // One V-cycle on R from the level-0 iterate Z = D^-1 R; Z becomes the preconditioned residual and c.tot the
  // products r.z.
  auto vcycle = [&]() {
    const int L = lv.n, dist = tail ? lv.tail : L;  // levels dealt to the workers
    for (int l = 0; l < dist && l + 1 < L; ++l) {
      apply<NR>(kResid, l, 0, 0);
      if (!barrier()) return false;
      if (l + 1 == dist) break;  // the tail's block restricts for itself
      restrict_down<NR>(l);
      if (!barrier()) return false;
    }
    if (tail) {
      tail_cycle<NR>();
      if (!barrier()) return false;
    } else {
      for (int p = 0; p < 2 * pairs; ++p) {  // the coarsest level's Jacobi sweeps x -> y -> x
        apply<NR>(kSmooth, L - 1, p & 1, ~p & 1);
        if (!barrier()) return false;
      }
    }
    for (int l = min(dist, L - 1) - 1; l >= 0; --l) {
      prolong_up<NR>(l);
      if (!barrier()) return false;
      if (l > 0) {
        apply<NR>(kSmooth, l, 2, 0);
        if (!barrier()) return false;
      }
    }
    apply<NR>(kPost, 0, 0, 0);
    __syncthreads();
    return reduce([&](int v, int w) { return make_double2(dot0<NR, SHARED>(c.R, c.Z, NR == 1 ? 1 : 2, v, w), 0.0); }, 1);
  };
  auto all_done = [&]() {
    __syncthreads();
    if (tid == 0) {
      int all = 1;
      for (int q = 0; q < NR; ++q) all &= c.rdone[q];
      c.done = all;
    }
    __syncthreads();
    return c.done != 0;
  };
  // Scalars after a V-cycle (start: the one before the first iteration); true when every right-hand side is done.
  auto vcycle_scalars = [&](bool start) {
    if (tid < NR && !c.rdone[tid]) {
      const double tot = c.tot[tid];
      if (!start) c.beta[tid] = (float)(tot / c.rz[tid]);
      c.rz[tid] = tot;
      if (!isfinite(tot)) {
        c.rdone[tid] = 1;
        if (NR == 1) c.bad = 1;
      }
    }
    return all_done();
  };
  bool run = true, maxed = false;
  double pnorm = 0.0;
  fill_tail<NR>();
  if (NR == 1) {
    run = reduce([&](int v, int w) { return setup1<MG, SHARED>(v, w); }, 2);
    if (run) {
      const double zz = c.tot[0], rz = c.tot[1], pn = sqrt(zz);
      pnorm = pn;
      const bool bad = !isfinite(zz) || !isfinite(rz);
      run = max_its > 0 && !(pn < c.min_err || pn < pn * c.rel_err) && !bad;
      __syncthreads();
      if (tid == 0) {
        c.pn0[0] = pn;
        c.rz[0] = rz;
        c.bad = bad;
      }
      __syncthreads();
    }
  }
  if (MG && run) {
    run = vcycle();
    if (run) run = !vcycle_scalars(true);
    if (run) {
      direction<NR>(true);
      run = barrier();
    }
  }
  while (run) {
    apply<NR>(kProduct, 0, 0, 0);
    __syncthreads();
    if (!reduce([&](int v, int w) { return make_double2(dot0<NR, SHARED>(c.P, c.AP, own_units(NR), v, w), 0.0); }, 1)) break;
    if (tid < NR) c.alpha[tid] = c.rdone[tid] ? 0.f : (float)(c.rz[tid] / c.tot[tid]);
    __syncthreads();
    if (!reduce([&](int v, int w) { return update<NR, MG>(v, w); }, MG ? 1 : 2)) break;
    its += 1;
    if (tid < NR && !c.rdone[tid]) {
      const double tot = c.tot[tid], pn = sqrt(tot);
      const bool met = pn < c.min_err || pn < c.pn0[tid] * c.rel_err;
      bool bad = !isfinite(tot);
      if (!MG) {
        const double rz = c.tot[NR + tid];
        c.beta[tid] = (float)(rz / c.rz[tid]);
        c.rz[tid] = rz;
        if (NR == 1) bad = bad || !isfinite(rz);
      }
      if (bad && NR == 1) c.bad = 1;
      c.rdone[tid] = !(its < max_its) || met || bad;
      if (NR == 1) {
        pnorm = pn;
        maxed = !(its < max_its) && !met;
      }
    }
    if (all_done()) break;
    if (MG) {
      if (!vcycle()) break;
      if (vcycle_scalars(false)) break;
    }
    direction<NR>(false);
    if (!barrier()) break;
  }
  if (tid == 0) {
    if (rank == 0) {
      if (NR == 1) {
        I.cg->done = 1;
        I.cg->its = its;
        I.cg->pnorm = pnorm;
        I.out->cg_its = its;
        I.out->cg_maxed = maxed;
        if (c.bad) I.out->nonfinite = 1;
      } else {
        c6s->all_done = 1;
        c6s->its = its;
        I.out->cg6_its = its;
      }
    }
    if (!ok)
      I.out->stalled = 1;  // a block of the group never arrived: reported to the host, which clears the counter
    else if (atomicAdd(c.ctr, 1u) == target + G - 1)
      *c.ctr = 0u;  // the last block to leave; the others have left every barrier
  }
}

Grid grid_of(const MeshDev &m) {
  Grid g{m.nx, m.ny, m.nz, m.nxny, m.nn, m.np, (m.nn + 31) / 32, m.nx - 2, m.ny - 2, 0, 0};
  g.inner = g.ix > 0 && g.iy > 0 && m.nz > 2 ? g.ix * g.iy * (m.nz - 2) : 0;
  g.iunits = (g.inner + 31) / 32;
  return g;
}

// The fraction of the matrix values that stays in L2 at the normal priority, the others being the first to go: what
// three fifths of it hold.  Streamed all alike, values that exceed the L2 push each other out before the next pass reads
// them, and the vectors with them: 8 x 30^3 damage 14.1 ms, and 13.6 so (13.75 with 0.85 of the L2), 60^3 14.4 and 14.0.
float keep_fraction(double bytes) {
  int dev = 0, l2 = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess) {
    cudaGetLastError();
    return 1.f;
  }
  const double f = 0.6 * l2 / bytes;
  return f < 1.0 ? (float)f : 1.f;
}

template <int NR, bool MG>
int launch(const Levels &lv, const Inst *insts, const int *list, int nlist, int G, int V, int idle,
           const double *rel_tols, double abs_tol, int max_its, int pairs, float keep, cudaStream_t s) {
  Levels l = lv;
  const size_t smem = kCtxBytes + kHeldFloats * sizeof(float);
  const void *f = G < V ? (const void *)k_coop_cg32<NR, MG, true> : (const void *)k_coop_cg32<NR, MG, false>;
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  void *args[] = {&l, &insts, &list, &G, &V, &idle, &rel_tols, &abs_tol, &max_its, &pairs, &keep};
  e = cudaLaunchCooperativeKernel(f, dim3(nlist * G), dim3(kThreads), args, smem, s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return -1;
  }
  return (int)e;
}

}  // namespace
}  // namespace mgb

using namespace mgb;

extern "C" {

int mgb_coop_cg32_pays(const MeshDev *m, int nlist, int mg, long long beside) {
  const long long nodes = (long long)m->nn * nlist;
  if (nlist <= 0 || nodes > kCoopNodes) return 0;
  if (!mg && beside > kCoopBeside) return 0;
  const int blocks = coop_sms() / nlist;
  return blocks >= kTailBlocks || (mg && blocks >= kTailBlocks / 2 && nodes <= kCoopNodesFew);
}

int mgb_launch_coop_cg32(const MeshDev *levels, int nlevels, const Inst *insts, const int *list, int nlist, int nr,
                         const double *rel_tols, double abs_tol, int max_its, int pairs, int parts, cudaStream_t s) {
  if (nlist <= 0) return 0;
  if (nlevels < 1 || nlevels > kMgMaxLevels || (nr != 1 && nr != 6)) return (int)cudaErrorInvalidValue;
  const int sms = coop_sms();
  int V = sms / nlist, tail = 0;  // blocks per instance, one per SM
  if (V < 1) return -1;
  Levels lv{};
  lv.n = lv.tail = nlevels;
  for (int l = 0; l < nlevels; ++l) lv.g[l] = grid_of(levels[l]);
  const int runs = (lv.g[0].units + own_units(nr) - 1) / own_units(nr);
  if (V >= kTailBlocks)
    for (int l = nlevels - 1; l >= 1; --l) {
      const int more = tail_floats(lv.g[l], nr);
      if (tail + more > kHeldFloats || lv.g[l].inner == 0) break;
      tail += more;
      lv.tail = l;
    }
  // no more workers than have a run (1 RHS) or a unit for each group of warps (6 RHS): the rest of the SMs is better
  // left to the solves of other handles
  const int per = nr == 1 ? 1 : kGroups / own_units(6), most = (runs + per - 1) / per + (lv.tail < nlevels ? 1 : 0);
  if (V > most) V = most;
  const int idle = lv.tail < nlevels ? 1 : 0;
  // with a share of the SMs: fewer blocks than parts of the sums
  int G = sms / (nlist * parts);
  G = G < 1 ? 1 : G < V ? G : V;
  if (G < V && G < kTailBlocks) lv.tail = nlevels;
  const bool mg = nlevels > 1;
  const float keep = keep_fraction((double)kEllPerNode * sizeof(float) * levels[0].np * nlist);
#define MGB_COOP(NR)                                                                                                  \
  (mg ? launch<NR, true>(lv, insts, list, nlist, G, V, idle, rel_tols, abs_tol, max_its, pairs, keep, s)            \
      : launch<NR, false>(lv, insts, list, nlist, G, V, idle, rel_tols, abs_tol, max_its, pairs, keep, s))
  return nr == 1 ? MGB_COOP(1) : MGB_COOP(6);
#undef MGB_COOP
}

}  // extern "C"
