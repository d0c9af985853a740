// cg_kernels.cu -- Jacobi-preconditioned CG on the stencil ELL matrix (sm_103a, FP64).
//
// The iteration is the reference's ell_solve_cgpd (ell.cpp:66-122) step for step:
//   k = 1/diag(A); x = 0; r = b; z = k r; p = z; rz = r.z; pnorm0 = ||z||
//   while its < max_its and not (pnorm < min_err or pnorm < pnorm0*rel_err):
//     Ap = A p; alpha = rz / p.Ap; x += alpha p; r -= alpha Ap; z = k r; pnorm = ||z||; rz' = r.z;
//     beta = rz'/rz; p = z + beta p; rz = rz'
// with the scalars kept on the device: each kernel's last block (reduce.cuh) derives alpha or beta and the
// stop flag, and every block of a finished instance returns at once.  The host only polls the number of
// unfinished instances every few iterations; no kernel waits on another.
//
// One thread owns one node (its 3 rows).  ELL entry (s, fi, fj) of node n is vals[(s*9+fi*3+fj)*np + n], so
// the 81 value streams of a warp are coalesced; the 27 neighbour columns are implicit (structured grid)
// and their x values come through L1/L2.  Boundary rows are identity rows.
#include <cuda_runtime.h>

#include "coop.cuh"
#include "device.cuh"
#include "launch.h"
#include "reduce.cuh"

namespace mgb {

constexpr int kUpdRows = 4;  // rows per thread of the vector update
// Largest batch (nodes of all its instances) solved by one cooperative launch: above, the two forms are equal (60^3 nodes)
// or the launches faster (damage, plain form, 8 x 30^3 179 ms against 186, 32 x 20^3 191 against 210).
// Handles at work at the same time count as one batch (each as large as the caller's), since their launches overlap: 16
// points of 30^3, a handle each, 338 ms with every solve in one launch on all SMs, 199 launched.  Below that they share
// the SMs (AtWork::parts): 16 J2 points of 20^3 3,430 ms on all SMs each, 1,580 so, 1,656 launched; 4 of them 848, 525, 702.
constexpr long long kSolveNodes = 150000;
// Microseconds of an iteration in one launch: a block's unit of 32 nodes (243 FP64 warp instructions of 64 cycles on
// four quarters), the shortest unit (its chain of dependent products), and the rest.
constexpr double kUnitUs = 2.0, kChainUs = 6.0, kPhasesUs = 9.0;

__device__ __forceinline__ bool node_boundary(const MeshDev &m, int n, int &i, int &j, int &k) {
  i = n % m.nx;
  j = (n / m.nx) % m.ny;
  k = n / m.nxny;
  return i == 0 || j == 0 || k == 0 || i == m.nx - 1 || j == m.ny - 1 || k == m.nz - 1;
}

__global__ void __launch_bounds__(kNodeBlock) k_cg_setup(MeshDev m, const Inst *insts, const int *list) {
  const Inst &I = insts[list[blockIdx.y]];
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[2] = {0.0, 0.0};  // r.z, z.z
  if (n < m.nn) {
    int i, j, k;
    const bool bnd = node_boundary(m, n, i, j, k);
    const double *__restrict__ vals = I.vals;
    const double *__restrict__ b = I.b;
    double *__restrict__ kinv = I.kinv;
    double *__restrict__ x = I.du;
    double *__restrict__ rv = I.r;
    double *__restrict__ zv = I.z;
    double *__restrict__ pv = I.p;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int row = n * 3 + d;
      const double kd = bnd ? 1.0 : 1 / vals[(size_t)(13 * 9 + d * 3 + d) * m.np + n];
      const double r = b[row];
      const double z = kd * r;
      kinv[row] = kd;
      x[row] = 0.0;
      rv[row] = r;
      zv[row] = z;
      pv[row] = z;
      acc[0] += r * z;
      acc[1] += z * z;
    }
  }
  double tot[2];
  if (grid_sum<2>(acc, I.red, I.ticket, gridDim.x, tot) && threadIdx.x == 0) {
    CgState *c = I.cg;
    c->rz = tot[0];
    c->pnorm0 = sqrt(tot[1]);
    c->pnorm = c->pnorm0;
    c->its = 0;
    c->beta = 0.0;
    c->done = !(c->its < c->max_its) || c->pnorm < c->min_err || c->pnorm < c->pnorm0 * c->rel_err;
    if (!isfinite(tot[0]) || !isfinite(tot[1])) {
      c->done = 1;
      I.out->nonfinite = 1;
    }
  }
}

// Ap = A p and p.Ap; the last block sets alpha = rz / p.Ap.
__global__ void __launch_bounds__(kNodeBlock) k_cg_spmv(MeshDev m, const Inst *insts, const int *list) {
  const Inst &I = insts[list[blockIdx.y]];
  if (I.cg->done) return;
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[1] = {0.0};
  if (n < m.nn) {
    int i, j, k;
    const double *__restrict__ p = I.p;
    double *__restrict__ Ap = I.Ap;
    if (node_boundary(m, n, i, j, k)) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double pv = p[n * 3 + d];
        Ap[n * 3 + d] = pv;
        acc[0] += pv * pv;
      }
    } else {
      const double *__restrict__ v = I.vals + n;
      const size_t np = m.np;
      double y0 = 0.0, y1 = 0.0, y2 = 0.0;
#pragma unroll
      for (int s = 0; s < 27; ++s) {
        const int nb = n + (s / 9 - 1) * m.nxny + ((s / 3) % 3 - 1) * m.nx + (s % 3 - 1);
        const double x0 = p[nb * 3 + 0], x1 = p[nb * 3 + 1], x2 = p[nb * 3 + 2];
        const double *vs = v + (size_t)(s * 9) * np;
        y0 += __ldcs(vs + 0 * np) * x0;
        y0 += __ldcs(vs + 1 * np) * x1;
        y0 += __ldcs(vs + 2 * np) * x2;
        y1 += __ldcs(vs + 3 * np) * x0;
        y1 += __ldcs(vs + 4 * np) * x1;
        y1 += __ldcs(vs + 5 * np) * x2;
        y2 += __ldcs(vs + 6 * np) * x0;
        y2 += __ldcs(vs + 7 * np) * x1;
        y2 += __ldcs(vs + 8 * np) * x2;
      }
      Ap[n * 3 + 0] = y0;
      Ap[n * 3 + 1] = y1;
      Ap[n * 3 + 2] = y2;
      acc[0] = p[n * 3 + 0] * y0 + p[n * 3 + 1] * y1 + p[n * 3 + 2] * y2;
    }
  }
  double tot[1];
  if (grid_sum<1>(acc, I.red, I.ticket, gridDim.x, tot) && threadIdx.x == 0) {
    CgState *c = I.cg;
    c->pAp = tot[0];
    c->alpha = c->rz / tot[0];
  }
}

// x += alpha p; r -= alpha Ap; z = k r; then ||z|| and r.z; the last block sets beta and the stop flag.
__global__ void __launch_bounds__(kNodeBlock) k_cg_update(MeshDev m, const Inst *insts, const int *list) {
  const Inst &I = insts[list[blockIdx.y]];
  const CgState *cs = I.cg;
  if (cs->done) return;
  const double alpha = cs->alpha;
  const int nrow = m.nn * 3;
  double *__restrict__ x = I.du;
  double *__restrict__ rv = I.r;
  double *__restrict__ zv = I.z;
  const double *__restrict__ p = I.p;
  const double *__restrict__ Ap = I.Ap;
  const double *__restrict__ kinv = I.kinv;
  double acc[2] = {0.0, 0.0};  // z.z, r.z
  // kUpdRows rows per thread, strided by the grid so that every load is coalesced; all loads first.
  const int stride = gridDim.x * blockDim.x;
  for (int row0 = blockIdx.x * blockDim.x + threadIdx.x; row0 < nrow; row0 += kUpdRows * stride) {
    double pv[kUpdRows], av[kUpdRows], rr[kUpdRows], xv[kUpdRows], kv[kUpdRows];
#pragma unroll
    for (int q = 0; q < kUpdRows; ++q) {
      const int row = row0 + q * stride;
      if (row < nrow) {
        pv[q] = p[row]; av[q] = Ap[row]; rr[q] = rv[row]; xv[q] = x[row]; kv[q] = kinv[row];
      }
    }
#pragma unroll
    for (int q = 0; q < kUpdRows; ++q) {
      const int row = row0 + q * stride;
      if (row < nrow) {
        x[row] = xv[q] + alpha * pv[q];
        const double r = rr[q] - alpha * av[q];
        const double z = kv[q] * r;
        rv[row] = r;
        zv[row] = z;
        acc[0] += z * z;
        acc[1] += r * z;
      }
    }
  }
  double tot[2];
  if (grid_sum<2>(acc, I.red, I.ticket, gridDim.x, tot) && threadIdx.x == 0) {
    CgState *c = I.cg;
    c->pnorm = sqrt(tot[0]);
    c->beta = tot[1] / c->rz;
    c->rz = tot[1];
    c->its += 1;
    c->done = !(c->its < c->max_its) || c->pnorm < c->min_err || c->pnorm < c->pnorm0 * c->rel_err;
    if (!isfinite(tot[0]) || !isfinite(tot[1])) {
      c->done = 1;
      I.out->nonfinite = 1;
    }
    if (c->done) {
      I.out->cg_its = c->its;
      I.out->cg_maxed = !(c->its < c->max_its) && !(c->pnorm < c->min_err || c->pnorm < c->pnorm0 * c->rel_err);
    }
  }
}

// p = z + beta p (skipped once the instance has stopped: p is not used again).
__global__ void __launch_bounds__(kNodeBlock) k_cg_pupdate(MeshDev m, const Inst *insts, const int *list,
                                                           unsigned int *active_count) {
  const Inst &I = insts[list[blockIdx.y]];
  const CgState *cs = I.cg;
  if (cs->done) return;
  const double beta = cs->beta;
  const int nrow = m.nn * 3;
  double *__restrict__ p = I.p;
  const double *__restrict__ z = I.z;
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < nrow; row += gridDim.x * blockDim.x)
    p[row] = z[row] + beta * p[row];
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(active_count, 1u);
}

// ---------------------------------------------------------------------------------------------------
// The whole solve in one cooperative launch, for batches whose iterations are shorter than three launches.
//
// A group of G blocks owns an instance and iterates on it alone: no lockstep with the other instances, no
// launch between the phases.  The phases of an iteration (SpMV, vector update, p-update) are separated by a
// barrier over the group's blocks; the cooperative launch keeps all blocks resident, and every wait is bounded.
// Each block forms the scalars for itself from the partial sums, so a barrier is the only exchange.
//
// The FP64 pipe (2 lanes per SM and cycle: a warp instruction holds its quarter of the SM for 64 cycles) bounds
// the work, so it is spread over as many SMs and schedulers as there are: a unit of the SpMV is 32 nodes x 3
// rows on 3 warps, one row of 81 products per thread (one node per thread, as k_cg_spmv has it, leaves most SMs
// idle on small grids and runs 243 products one after the other), and as few units per block as there are SMs for.
// Every sum keeps the order of the launches of one iteration (k_cg_spmv, k_cg_update, k_cg_pupdate): the products of a
// row, the lanes of a warp, the 8 warps of a 256-thread block, the blocks -- so the solve is the same bit for bit.
//
// A block's units are a run, dealt over its groups of 3 warps.  p and z are component-major here (32 neighbours' entries
// are two lines, not seven); the caller's buffers hold 3 np values for them.
//
// Microseconds per iteration of one instance, three launches against this kernel: 10^3 nodes 42 and 16, 30^3 57 and 30,
// 40^3 72 and 56, 50^3 100 and 97, 60^3 149 and 145, 80^3 283 and 314 (there the FP64 pipe is full either way and the
// launches need no barrier).  At 10^3 an iteration is 5 us of dependent FP64 products, 4 us of barriers and 5 us of
// reduction trees, division and square root; at 50^3 73 us of products (54 at the pipe's measured rate).

constexpr int kUnitThreads = 96;   // 32 nodes x 3 rows

// The sum over the blocks of a launch from its warp sums part[k * stride + w], as grid_finish<K> forms it; the
// result is in sums[k * 8 + f] for the 8 warps f of the finishing block (sum8 adds them).
template <int K>
__device__ __forceinline__ void tree_blocks(const double *part, int stride, int nwarps, double (*sums)[8]) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, nblocks = (nwarps + 7) / 8;
  for (int t = threadIdx.x >> 5; t < 8 * K; t += nw) {
    const int f = t & 7, k = t >> 3;
    double v = 0.0;
    if (f * 32 < nblocks) {
      for (int b = f * 32 + lane; b < nblocks; b += 512) {
        double w[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = (b + h * 256) * 8 + i;
            w[h][i] = e < nwarps ? __ldcg(part + (size_t)k * stride + e) : 0.0;
          }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (b + h * 256 < nblocks)
            v += ((w[h][0] + w[h][4]) + (w[h][2] + w[h][6])) + ((w[h][1] + w[h][5]) + (w[h][3] + w[h][7]));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    if (lane == 0) sums[k][f] = v;
  }
}

__device__ __forceinline__ double sum8(const double *s, int nblocks) {
  if (nblocks <= 32) return s[0];
  return ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
}

// KMAX: units a block works on at a time, at most; the fewer, the more of a row's loads are in registers ahead of its
// chain of products (20^3 nodes, two units: 18.4 us per iteration with a third of them, 18.0 with all).
template <int KMAX>
__global__ void __launch_bounds__(kUnitThreads *KMAX, 1)
    k_cg_solve(MeshDev m, const Inst *insts, const int *list, int nlist, int G) {
  __shared__ double sy[2][KMAX][2][32];
  __shared__ double sums[2][8];
  __shared__ double s_alpha, s_beta, s_rz;
  __shared__ int s_its, s_done, s_ok;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int group = blockIdx.x / G, rank = blockIdx.x - group * G, ngroups = gridDim.x / G;
  const int ug = wid / 3, fi = wid - ug * 3, K = nw / 3;
  const int nrow = m.nn * 3, units = (m.nn + 31) / 32;
  const int u0 = (int)((long long)units * rank / G), u1 = (int)((long long)units * (rank + 1) / G);
  const int ublocks = (nrow + kUpdRows * kNodeBlock - 1) / (kUpdRows * kNodeBlock), ustride = ublocks * kNodeBlock;
  const int uwarps = ublocks * (kNodeBlock / 32);
  const size_t np = m.np;
  for (int a = group; a < nlist; a += ngroups) {
    const Inst &I = insts[list[a]];
    CgState *cs = I.cg;
    if (cs->done) continue;
    double *part = I.red, *upart = I.red + units;
    unsigned int *ctr = I.ticket, target = 0;
    const double *vals = I.vals, *kinv = I.kinv;
    double *x = I.du, *r = I.r, *z = I.z, *p = I.p, *Ap = I.Ap;
    const double min_err = cs->min_err, rel_err = cs->rel_err, pnorm0 = cs->pnorm0;
    const int max_its = cs->max_its;
    const unsigned int polls = I.polls ? I.polls : kSpinLimit;
    if (threadIdx.x == 0) {
      s_rz = cs->rz;
      s_its = 0;
    }
    __syncthreads();
    // p = z (as the setup left it), component-major from here on, as z from the first update
    for (int u = u0 + ug; u < u1; u += K)
      if (u * 32 + lane < m.nn) p[fi * np + u * 32 + lane] = z[(u * 32 + lane) * 3 + fi];
    target += G;
    bool ok = group_barrier(ctr, target, &s_ok, polls);
    while (ok) {
      // Ap = A p and p.Ap
      for (int u = u0 + ug, turn = 0; u < u1; u += K, turn ^= 1) {
        const int n = u * 32 + lane;
        double y = 0.0;
        bool bn = true;
        if (n < m.nn) {
          int i, j, k;
          bn = node_boundary(m, n, i, j, k);
          if (bn) {
            y = p[fi * np + n];
          } else {
            const double *v = vals + (size_t)(fi * 3) * np + n;
#pragma unroll(KMAX > 4 ? 3 : 27)
            for (int s = 0; s < 27; ++s) {
              const int nb = n + (s / 9 - 1) * m.nxny + ((s / 3) % 3 - 1) * m.nx + (s % 3 - 1);
              const double *vs = v + (size_t)(s * 9) * np;
              y = fma(ld_value(vs), p[nb], y);
              y = fma(ld_value(vs + np), p[np + nb], y);
              y = fma(ld_value(vs + 2 * np), p[2 * np + nb], y);
            }
          }
          Ap[n * 3 + fi] = y;
        }
        if (fi > 0) sy[turn][ug][fi - 1][lane] = y;
        asm volatile("bar.sync %0, 96;" ::"r"(ug + 1) : "memory");  // the unit's 3 warps
        if (fi == 0) {
          double t = 0.0;
          if (n < m.nn) {
            const double y1 = sy[turn][ug][0][lane], y2 = sy[turn][ug][1][lane];
            if (bn)
              t = fma(y2, y2, fma(y1, y1, y * y));
            else
              t = p[n] * y + p[np + n] * y1 + p[2 * np + n] * y2;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
          if (lane == 0) part[u] = t;
        }
      }
      target += G;
      if (!(ok = group_barrier(ctr, target, &s_ok, polls))) break;
      tree_blocks<1>(part, 0, units, sums);
      __syncthreads();
      if (threadIdx.x == 0) s_alpha = s_rz / sum8(sums[0], (units + 7) / 8);
      __syncthreads();
      // x += alpha p; r -= alpha Ap; z = kinv r; z.z and r.z
      const double alpha = s_alpha;
      for (int w = wid * G + rank; w < uwarps; w += G * nw) {
        double pv[kUpdRows], av[kUpdRows], rr[kUpdRows], xv[kUpdRows], kv[kUpdRows];
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
          const int row = w * 32 + lane + q * ustride, n = row / 3;
          if (row < nrow) {
            pv[q] = p[(row - n * 3) * np + n]; av[q] = Ap[row]; rr[q] = r[row]; xv[q] = x[row]; kv[q] = kinv[row];
          }
        }
        double zz = 0.0, rz = 0.0;
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
          const int row = w * 32 + lane + q * ustride, n = row / 3;
          if (row < nrow) {
            x[row] = fma(alpha, pv[q], xv[q]);
            const double rn = fma(-alpha, av[q], rr[q]);
            const double zn = kv[q] * rn;
            r[row] = rn;
            z[(row - n * 3) * np + n] = zn;
            zz = fma(zn, zn, zz);
            rz = fma(rn, zn, rz);
          }
        }
        // both warp sums in one tree: lanes 0-15 add up zz, 16-31 rz (half the FP64 additions, in the same order)
        const bool upper = lane >= 16;
        const double give = __shfl_xor_sync(0xffffffffu, upper ? zz : rz, 16);
        double both = upper ? give + rz : zz + give;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) both += __shfl_down_sync(0xffffffffu, both, o, 16);
        if (lane == 0) upart[w] = both;
        if (lane == 16) upart[uwarps + w] = both;
      }
      target += G;
      if (!(ok = group_barrier(ctr, target, &s_ok, polls))) break;
      tree_blocks<2>(upart, uwarps, uwarps, sums);
      __syncthreads();
      if (threadIdx.x == 32) s_beta = sum8(sums[1], ublocks) / s_rz;
      if (threadIdx.x == 0) {
        const double tot = sum8(sums[0], ublocks), pnorm = sqrt(tot);
        const int its = s_its + 1;
        const bool met = pnorm < min_err || pnorm < pnorm0 * rel_err, bad = !isfinite(tot) || !isfinite(sum8(sums[1], ublocks));
        s_its = its;
        s_done = !(its < max_its) || met || bad;
        if (rank == 0 && s_done) {
          cs->pnorm = pnorm;
          cs->its = its;
          cs->done = 1;
          I.out->cg_its = its;
          I.out->cg_maxed = !(its < max_its) && !met;
          if (bad) I.out->nonfinite = 1;
        }
      }
      __syncthreads();
      if (s_done) break;
      if (threadIdx.x == 0) s_rz = sum8(sums[1], ublocks);
      const double beta = s_beta;
      for (int q = rank * blockDim.x + threadIdx.x; q < 3 * m.np; q += G * blockDim.x) p[q] = fma(beta, p[q], z[q]);
      target += G;
      if (!(ok = group_barrier(ctr, target, &s_ok, polls))) break;
    }
    if (threadIdx.x == 0) {
      if (!ok) {  // a block of the group never arrived: reported to the host, which clears the counter
        cs->done = 1;
        I.out->stalled = 1;
      } else if (atomicAdd(ctr, 1u) == target + G - 1) {
        *ctr = 0u;  // the last block to leave; the others have left every barrier
      }
    }
    __syncthreads();
  }
}

// Setup leaves out.cg_its = 0 for instances that stop before the first iteration.
__global__ void k_cg_init_out(const Inst *insts, const int *list, int nlist) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nlist) {
    const Inst &I = insts[list[t]];
    I.out->cg_its = 0;
    I.out->cg_maxed = 0;
  }
}

}  // namespace mgb

using namespace mgb;

static inline unsigned cdiv(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

extern "C" {

int mgb_launch_cg_setup(const MeshDev *m, const Inst *insts, const int *list, int nlist, cudaStream_t s) {
  if (nlist <= 0) return 0;
  k_cg_init_out<<<cdiv(nlist, 128), 128, 0, s>>>(insts, list, nlist);
  k_cg_setup<<<dim3(cdiv(m->nn, kNodeBlock), nlist), kNodeBlock, 0, s>>>(*m, insts, list);
  return (int)cudaGetLastError();
}

// One CG iteration = spmv (+ p.Ap, alpha), update (+ ||z||, r.z, beta, stop flag), p-update.
int mgb_launch_cg_spmv(const MeshDev *m, const Inst *insts, const int *list, int nlist, cudaStream_t s) {
  if (nlist <= 0) return 0;
  k_cg_spmv<<<dim3(cdiv(m->nn, kNodeBlock), nlist), kNodeBlock, 0, s>>>(*m, insts, list);
  return (int)cudaGetLastError();
}

int mgb_launch_cg_update(const MeshDev *m, const Inst *insts, const int *list, int nlist, cudaStream_t s) {
  if (nlist <= 0) return 0;
  k_cg_update<<<dim3(cdiv((size_t)m->nn * 3, (size_t)kUpdRows * kNodeBlock), nlist), kNodeBlock, 0, s>>>(*m, insts,
                                                                                                      list);
  return (int)cudaGetLastError();
}

// active_count receives +1 for every instance that is still iterating.
int mgb_launch_cg_pupdate(const MeshDev *m, const Inst *insts, const int *list, int nlist, unsigned int *active_count,
                          cudaStream_t s) {
  if (nlist <= 0) return 0;
  k_cg_pupdate<<<dim3(cdiv((size_t)m->nn * 3, kNodeBlock), nlist), kNodeBlock, 0, s>>>(*m, insts, list,
                                                                                         active_count);
  return (int)cudaGetLastError();
}

// The iterations of the listed instances after mgb_launch_cg_setup, to the end, in one cooperative launch.  Returns
// -1 without launching where the batch is too large for it to pay (see kSolveNodes) or the device cannot hold it.
int mgb_launch_cg_solve(const MeshDev *m, const Inst *insts, const int *list, int nlist, int at_work, int parts,
                        cudaStream_t s) {
  if (nlist <= 0) return 0;
  if ((long long)m->nn * nlist * (at_work > 1 ? at_work : 1) > kSolveNodes) return -1;
  const int all = coop_sms();
  if (!all) return -1;
  const int units = (int)cdiv(m->nn, 32);
  const int sms = all > parts ? all / parts : 1;
  // groups of blocks that each take one instance after the other: the number that the iterations' times ask for
  // (kUnitUs per unit of a block, at least kChainUs, and kPhasesUs of barriers and scalars)
  int groups = 1, G = sms;
  double least = 0.0;
  for (int g = 1; g <= nlist && g <= sms; ++g) {
    const int blocks = sms / g < units ? sms / g : units;
    const double work = kUnitUs * cdiv(units, blocks);
    const double t = cdiv(nlist, g) * ((work > kChainUs ? work : kChainUs) + kPhasesUs);
    if (g == 1 || t < least) {
      least = t;
      groups = g;
      G = blocks;
    }
  }
  const int K = cdiv(units, G) < 8 ? (int)cdiv(units, G) : 8;
  MeshDev mesh = *m;
  void *args[] = {&mesh, &insts, &list, &nlist, &G};
  const void *f = K > 4   ? (const void *)k_cg_solve<8>
                  : K > 2 ? (const void *)k_cg_solve<4>
                          : (const void *)k_cg_solve<2>;
  const cudaError_t e = cudaLaunchCooperativeKernel(f, dim3(groups * G), dim3(kUnitThreads * K), args, 0, s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return -1;
  }
  return (int)e;
}

}  // extern "C"
