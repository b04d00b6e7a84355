// The whole FP64 PCG solve of a chip-resident system in one cooperative
// launch, for the local preconditioners (none, Jacobi, block-Jacobi): every
// vector of the solve lives in registers, the matrix in shared memory (or, a
// little larger, in L2), and an iteration's grid-wide sum runs while its
// matrix product does.
//
// Form: Ghysels and Vanroose's pipelined PCG (2014), the recurrences and stop
// test of cgSolver.cpp:13-57 in exact arithmetic: u = M^-1 r, w = A u carried
// by recurrences, n = A M^-1 w formed every iteration, and the step lengths
// from the one set of dot products (r.u, w.u, r.r) that needs no n.
//
// What bounds it: latency.  A system of this size is a few hundred
// multiply-adds per thread and iteration; what an iteration waits for is the
// chip (a counting barrier over 152 CTAs takes about 1.1 us, a read of the
// other CTAs' partial sums 0.4 us, a chain of FP64 operations 65 cycles a
// link, an FP64 division 554).  So the CTA splits into
//
//   worker warps   one group of 10 block rows (30 DOFs, a lane each): the
//                  recurrences, the dot products, m = M^-1 w, the product;
//   a sync warp    publishes m (grid barrier) and releases the workers into
//                  the product;
//   a sum warp     adds the dot products of the CTA, publishes them, adds
//                  those of all CTAs and forms alpha and beta, all of it
//                  while the workers wait for m and multiply.
//
// In od_sparse.cu's persistent kernel (its pipelined form) one sync carries m
// and the sums one after the other and the product follows.  Per iteration,
// that kernel -> this one: 108 DOFs 13.2 -> 3.3 us, 2,160 DOFs 12.5 -> 5.0,
// 6,900 DOFs 12.9 -> 5.0, 55,488 DOFs 16.7 -> 10.1.
//
// A system that one CTA holds (kOneCta groups) needs no grid sync at all; its
// FP64 unit then does all the work, about 0.3 us per group and iteration,
// against about 3 us of grid syncs, so the line lies at 12 groups.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "od_internal.h"
#include "od_grid.cuh"

namespace od {

constexpr int kRgRows = 10;                    // block rows per group (one worker warp)
constexpr int kRgLanes = 3 * kRgRows;          // DOFs per group, a lane each
constexpr int kRgMaxWarps = 22;                // worker warps per CTA (two more serve)
constexpr int kRgStepBytes = kRgLanes * 3 * 8 + kRgRows * 4;   // one step of a group: 10 blocks and their columns
constexpr int kOneCta = 12;                    // groups a single CTA solves alone

struct ResidentArgs {
  int nb, ngroups, warps;       // block rows; groups; worker warps per CTA
  const int* rp;
  const int* col;
  const double* A;              // full BSR
  const double* b;
  double* x;
  double* u0;                   // A u of the start gathers it
  double* m[2];                 // M^-1 w by iteration parity
  const double* pinv;
  int pkind, x_zero, max_iter;
  double tol;
  double* part;                 // 2 x 3 x gridDim.x partial sums
  unsigned char* ell;           // matrix steps in global memory when they do not fit shared memory
  const int* ell_off;           // first step of every CTA there
  SolveScalars* sc;
  GridBarrier* gb;              // arrive: barriers; gen: sums
  unsigned long long* prof;
};

// named barriers of a CTA
enum { kBarM = 1, kBarDots = 2, kBarGo = 3, kBarStep = 4 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// One arrival of this CTA at a counter that only grows, then a bounded wait
// for all CTAs of the epoch-th round (as barrier_arrive_wait_count).
__device__ __forceinline__ bool arrive_wait(unsigned* ctr, int* timeout, unsigned epoch) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
  const unsigned target = epoch * gridDim.x;
  for (unsigned long long spins = 1;; spins++) {
    unsigned cur;
    asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(cur) : "l"(ctr) : "memory");
    if ((int)(cur - target) >= 0) return true;
    if ((spins & 31) == 0) {
      if (*(volatile int*)timeout) return false;
      if (spins > kSpinLimit) {
        atomicExch(timeout, 1);
        return false;
      }
    }
  }
}

struct ResidentShared {
  double ab[2];                 // alpha, beta
  double tot[3];                // the last grid-wide sums
  int stop, status, iter;
  int fail_sync, fail_sum;
  int seg[kRgMaxWarps];         // steps of every worker's group
};

// vals[j][thread] of the CTA's workers summed over the CTA, then over the
// grid, in a fixed order; every lane of the sum warp gets all NV sums.
// Returns false after a timeout.
template <int NV>
__device__ __forceinline__ bool sum_grid(const double* vals, int nt, double* part, unsigned* ctr, int* timeout,
                                         unsigned epoch, double (&t)[NV]) {
  const int lane = threadIdx.x & 31, G = gridDim.x;
#pragma unroll
  for (int j = 0; j < NV; j++) {
    double a0 = 0.0, a1 = 0.0;
    for (int i = lane; i < nt; i += 64) {
      a0 += vals[j * nt + i];
      if (i + 32 < nt) a1 += vals[j * nt + i + 32];
    }
    t[j] = a0 + a1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < NV; j++) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
  if (G == 1) return true;
  int ok = 1;
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < NV; j++) part[(size_t)j * G + blockIdx.x] = t[j];
    ok = arrive_wait(ctr, timeout, epoch);
  }
  __syncwarp();
  ok = __shfl_sync(0xffffffffu, ok, 0);
#pragma unroll
  for (int j = 0; j < NV; j++) t[j] = 0.0;
  constexpr int kLoads = 5;     // 5 x 32 covers one CTA per SM on 152 SMs in one pass
  for (int c0 = 0; c0 < G; c0 += 32 * kLoads) {
    double v[NV][kLoads];
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
      for (int q = 0; q < kLoads; q++) {
        const int c = c0 + lane + 32 * q;
        v[j][q] = c < G ? __ldcg(part + (size_t)j * G + c) : 0.0;
      }
#pragma unroll
    for (int j = 0; j < NV; j++) t[j] += ((v[j][0] + v[j][1]) + (v[j][2] + v[j][3])) + v[j][4];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < NV; j++) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
  return ok != 0;
}

template <bool SMEM>
__global__ void __launch_bounds__(32 * (kRgMaxWarps + 2), 1) pcg_resident_kernel(const ResidentArgs P) {
  extern __shared__ __align__(16) unsigned char rg_dsm[];
  __shared__ ResidentShared sh;
  const int G = gridDim.x, W = P.warps, nt = 32 * W;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gb0 = (int)((long long)blockIdx.x * P.ngroups / G);
  const int gb1 = (int)((long long)(blockIdx.x + 1) * P.ngroups / G);
  const bool worker = w < W;
  const int rsub = lane % 3;
  double* vals = reinterpret_cast<double*>(rg_dsm);   // [3][nt]
  unsigned* ctr_m = &P.gb->arrive;
  unsigned* ctr_s = &P.gb->gen;
  int* timeout = &P.gb->timeout;
  if (threadIdx.x == 0) {
    sh.fail_sync = sh.fail_sum = 0;
    sh.stop = 0;
    sh.status = OD_OK;
  }

  // ---- the group of this warp, its matrix steps: step j holds the j-th
  // blocks of its 10 block rows, 90 values [c][lane] (a lane's row r of its
  // block), then the 10 columns; short rows are padded with zeros
  const int g = gb0 + w;
  const bool has = worker && g < gb1;
  const int row = has && lane < kRgLanes ? g * kRgRows + lane / 3 : P.nb;
  const bool valid = row < P.nb;
  const int i = 3 * row + rsub;
  int kb = 0, ke = 0;
  if (valid) {
    kb = P.rp[row];
    ke = P.rp[row + 1];
  }
  const int steps = __reduce_max_sync(0xffffffffu, ke - kb);
  if (worker && lane == 0) sh.seg[w] = steps;
  __syncthreads();
  double* eA = nullptr;   // this lane's first value
  int* eC = nullptr;
  if (worker) {
    int off = 0;
    for (int q = 0; q < w; q++) off += sh.seg[q];
    unsigned char* base = SMEM ? rg_dsm + 3 * sizeof(double) * nt : P.ell + (size_t)P.ell_off[blockIdx.x] * kRgStepBytes;
    base += (size_t)off * kRgStepBytes;
    eA = reinterpret_cast<double*>(base) + min(lane, kRgLanes - 1);
    eC = reinterpret_cast<int*>(base + (size_t)steps * kRgLanes * 3 * 8) + min(lane / 3, kRgRows - 1);
    if (lane < kRgLanes)
      for (int j = 0; j < steps; j++) {
        const bool in = kb + j < ke;
        const double* a = P.A + 9 * (size_t)(kb + j) + 3 * rsub;
#pragma unroll
        for (int c = 0; c < 3; c++) eA[(3 * j + c) * kRgLanes] = in ? a[c] : 0.0;
        if (rsub == 0) eC[j * kRgRows] = in ? 3 * P.col[kb + j] : 3 * min(row, P.nb - 1);
      }
  }
  double pm0 = 1.0, pm1 = 0.0, pm2 = 0.0;
  if (valid) {
    if (P.pkind == OD_PRECOND_JACOBI) {
      pm0 = P.pinv[i];
    } else if (P.pkind == OD_PRECOND_BLOCK_JACOBI) {
      pm0 = P.pinv[3 * (size_t)i];
      pm1 = P.pinv[3 * (size_t)i + 1];
      pm2 = P.pinv[3 * (size_t)i + 2];
    }
  }
  const int l0 = min(lane - rsub, kRgLanes - 3);
  auto precond = [&](double v) -> double {
    if (P.pkind != OD_PRECOND_BLOCK_JACOBI) return pm0 * v;   // 1 without a preconditioner
    const double v0 = __shfl_sync(0xffffffffu, v, l0), v1 = __shfl_sync(0xffffffffu, v, l0 + 1),
                 v2 = __shfl_sync(0xffffffffu, v, l0 + 2);
    return pm0 * v0 + pm1 * v1 + pm2 * v2;
  };
  // row of A v; each lane of a group takes all of the group's steps
  auto product = [&](const double* v) -> double {
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;   // a chain per column: an FP64 operation takes 65 cycles
#pragma unroll 5
    for (int j = 0; j < steps; j++) {
      const double* xv = v + eC[j * kRgRows];
      y0 = fma(eA[(3 * j) * kRgLanes], xv[0], y0);
      y1 = fma(eA[(3 * j + 1) * kRgLanes], xv[1], y1);
      y2 = fma(eA[(3 * j + 2) * kRgLanes], xv[2], y2);
    }
    return (y0 + y1) + y2;
  };
  // one full sync of the grid: the stores before it visible after it, and
  // (sum warp) the sums of the workers' vals[0]; false after a timeout
  unsigned epoch = 0;     // rounds of both counters
  auto full_sync = [&]() -> bool {
    __syncthreads();
    epoch++;
    if (w == W) {
      if (G > 1 && lane == 0 && !arrive_wait(ctr_m, timeout, epoch)) sh.fail_sync = 1;
    } else if (w == W + 1) {
      double t[1];
      const bool ok = sum_grid<1>(vals, nt, P.part + (size_t)(epoch & 1) * 3 * G, ctr_s, timeout, epoch, t);
      if (lane == 0) {
        sh.tot[0] = t[0];
        if (!ok) sh.fail_sum = 1;
      }
    }
    __syncthreads();
    return !(sh.fail_sync | sh.fail_sum);
  };

  // ---- start: r = b - A x, u = M^-1 r, w = A u (cgSolver.cpp:20-30)
  double x = 0.0, r = 0.0, u = 0.0, wv = 0.0, bv = 0.0;
  if (worker) {
    if (valid) bv = r = P.b[i];
    if (!P.x_zero) {
      if (valid) x = P.x[i];
      const double y = product(P.x);
      if (valid) r = bv - y;
    }
    u = precond(r);
    if (valid) P.u0[i] = u;
    vals[threadIdx.x] = valid ? bv * bv : 0.0;
  }
  if (!full_sync()) return;
  const double bb = sh.tot[0], eps = bb * P.tol * P.tol;
  if (worker) wv = product(P.u0);
  if (!valid) r = u = wv = 0.0;   // idle lanes add nothing

  const bool timer = P.prof && blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long t_prev = 0;
  auto stamp = [&](int slot) {
    if (!timer) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (slot >= 0) P.prof[slot] += t - t_prev;
    t_prev = t;
  };
  stamp(-1);
  const int all = nt + 64;
  if (worker) {
    double p = 0.0, q = 0.0, s = 0.0, z = 0.0, alpha = 0.0;
    for (int par = 0;; par ^= 1) {
      __syncwarp();
      vals[threadIdx.x] = r * u;
      vals[nt + threadIdx.x] = wv * u;
      vals[2 * nt + threadIdx.x] = r * r;
      bar_arrive(kBarDots, nt + 32);
      const double m = precond(wv);
      if (valid) P.m[par][i] = m;
      __syncwarp();
      bar_arrive(kBarM, nt + 32);
      x = fma(alpha, p, x);      // the last iteration's, off the path to the sums
      stamp(2);
      bar_sync(kBarGo, nt + 32);
      const double n = product(P.m[par]);
      stamp(0);
      bar_sync(kBarStep, all);
      stamp(3);
      if (sh.stop) break;
      alpha = sh.ab[0];
      const double beta = sh.ab[1];
      z = fma(beta, z, n);
      q = fma(beta, q, m);
      s = fma(beta, s, wv);
      p = fma(beta, p, u);
      wv = fma(-alpha, z, wv);
      u = fma(-alpha, q, u);
      r = fma(-alpha, s, r);
      if (!valid) r = u = wv = 0.0;
      if (timer) P.prof[kPcgPhases] += 1;
    }
  } else if (w == W) {
    for (;;) {
      bar_sync(kBarM, nt + 32);
      epoch++;
      if (G > 1 && lane == 0 && !arrive_wait(ctr_m, timeout, epoch)) sh.fail_sync = 1;
      __syncwarp();
      bar_arrive(kBarGo, nt + 32);
      bar_sync(kBarStep, all);
      if (sh.stop) break;
    }
  } else {
    double gam_inv = 0.0, den_prev = 0.0;   // 1 / gamma and gamma / alpha of the last iteration
    for (int it = 0;; it++) {
      bar_sync(kBarDots, nt + 32);
      epoch++;
      double t[3];
      const bool ok = sum_grid<3>(vals, nt, P.part + (size_t)(epoch & 1) * 3 * G, ctr_s, timeout, epoch, t);
      // beta = gamma / gamma_prev, alpha = gamma / (delta - beta gamma / alpha_prev):
      // gamma / alpha_prev = beta den_prev, so one division is on the path
      const double gam = t[0], rr = t[2];
      const double beta = gam * gam_inv;
      const double den = fma(-beta * beta, den_prev, t[1]);
      const double alpha = gam / den;
      int stop = 0, status = OD_OK;
      if (!isfinite(rr)) {
        stop = 1;
        status = OD_ERR_NAN;
      } else if (!(rr > eps) || it >= P.max_iter) {
        stop = 1;
      } else if (!isfinite(alpha) || !isfinite(beta)) {
        stop = 1;
        status = OD_ERR_NAN;
      }
      if (!ok) sh.fail_sum = 1;
      // a barrier that timed out (seen here an iteration later at most)
      if (!ok || *(volatile int*)&sh.fail_sync) stop = 1;
      if (lane == 0) {
        sh.ab[0] = alpha;
        sh.ab[1] = beta;
        sh.stop = stop;
        if (stop) {
          sh.status = status;
          sh.iter = it;
          sh.tot[1] = gam;
          sh.tot[2] = rr;
        }
      }
      __syncwarp();
      bar_sync(kBarStep, all);
      if (stop) break;
      gam_inv = 1.0 / gam;
      den_prev = den;
    }
  }
  __syncthreads();
  if (sh.fail_sync | sh.fail_sum) return;

  // ---- write x, then the true residual ||b - A x||^2
  if (valid) P.x[i] = x;
  if (worker) vals[threadIdx.x] = 0.0;
  if (!full_sync()) return;
  if (worker) {
    const double d = bv - product(P.x);
    vals[threadIdx.x] = valid ? d * d : 0.0;
  }
  if (!full_sync()) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    SolveScalars* sc = P.sc;
    sc->rz[0] = sh.tot[1];
    sc->rr = sh.tot[2];
    sc->bb = bb;
    sc->eps = eps;
    sc->iter = sh.iter;
    sc->max_iter = P.max_iter;
    sc->status = sh.status;
    sc->tr_num = sh.tot[0];
    sc->tr_den = bb;
    sc->done = 1;
  }
}

static const void* resident_kernel(bool smem) {
  return smem ? (const void*)pcg_resident_kernel<true> : (const void*)pcg_resident_kernel<false>;
}

// The shape of a scene's resident solve: CTAs, worker warps, where the
// matrix lives.  Leaves warps = 0 when the system is too large for one group
// per worker warp (the persistent kernel of od_sparse.cu takes it).
od_status resident_plan(Scene* s) {
  ResidentPlan& R = s->pcg.res;
  R = ResidentPlan();
  const int nb = s->bsr.nb;
  if (s->pcg.coop_grid <= 0 || nb <= 0 || (int)s->hbsr_rp.size() != nb + 1) return OD_OK;
  const std::vector<int>& rp = s->hbsr_rp;
  const int ng = (nb + kRgRows - 1) / kRgRows;
  const int sms = std::max(1, s->ctx->num_sms);
  const char* env = std::getenv("OD_GB300_PCG_SMEM");   // 0: the matrix from L2 (the same operations)
  const bool allow_smem = !(env && env[0] == '0');
  int dev_max = 0;
  cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->ctx->device);
  const int grids[2] = {ng <= kOneCta ? 1 : 0, std::min(sms, ng)};
  for (int G : grids) {
    if (G <= 0 || R.warps > 0) continue;
    const int warps = (ng + G - 1) / G;
    if (warps > kRgMaxWarps) continue;
    std::vector<int> off((size_t)G + 1, 0);
    int most = 0;
    for (int c = 0; c < G; c++) {
      int steps = 0;
      for (int g = (int)((long long)c * ng / G); g < (int)((long long)(c + 1) * ng / G); g++) {
        int m = 0;
        for (int r = g * kRgRows; r < std::min(nb, (g + 1) * kRgRows); r++) m = std::max(m, rp[r + 1] - rp[r]);
        steps += m;
      }
      off[c + 1] = off[c] + steps;
      most = std::max(most, steps);
    }
    const long long vals = 3LL * sizeof(double) * 32 * warps;
    for (int smem = allow_smem ? 1 : 0; smem >= 0 && R.warps == 0; smem--) {
      // a system that one CTA's shared memory cannot hold goes to the grid
      if (!smem && allow_smem && G == 1 && grids[1] > 1) break;
      const long long bytes = vals + (smem ? (long long)most * kRgStepBytes : 0);
      const void* fn = resident_kernel(smem != 0);
      cudaFuncAttributes fa{};
      int bps = 0;
      // the attribute is per function, shared by every scene: set it to the
      // most the device allows, never to one scene's size
      const long long cap = (long long)dev_max - 1024;
      if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess && bytes + (long long)fa.sharedSizeBytes <= cap &&
          cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(cap - (long long)fa.sharedSizeBytes)) == cudaSuccess &&
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, 32 * (warps + 2), (size_t)bytes) == cudaSuccess &&
          bps >= 1) {
        R.grid = G;
        R.warps = warps;
        R.bytes = (int)bytes;
        R.smem = smem != 0;
        if (!R.smem) R.off = off;
      }
      cudaGetLastError();   // a refused attribute is not an error of the scene
    }
  }
  return OD_OK;
}

void resident_free(ResidentPlan* R) {
  cudaFree(R->ell);
  cudaFree(R->ell_off);
  *R = ResidentPlan();
}

od_status resident_solve(Scene* s, const double* d_b, double* d_x, int pkind, double tol, int max_iter, bool x_zero,
                         unsigned long long* prof) {
  Pcg& P = s->pcg;
  ResidentPlan& R = P.res;
  if (!R.smem && !R.ell) {   // kept with the scene from its first such solve on
    const size_t bytes = (size_t)std::max(1, R.off.back()) * kRgStepBytes;
    OD_CUDA(cudaMalloc(&R.ell_off, sizeof(int) * R.off.size()));
    OD_CUDA(cudaMemcpy(R.ell_off, R.off.data(), sizeof(int) * R.off.size(), cudaMemcpyHostToDevice));
    OD_CUDA(cudaMalloc(&R.ell, bytes));
    s->device_bytes += (long long)(bytes + sizeof(int) * R.off.size());
  }
  ResidentArgs a{};
  a.nb = s->bsr.nb;
  a.ngroups = (s->bsr.nb + kRgRows - 1) / kRgRows;
  a.warps = R.warps;
  a.rp = s->bsr.row_ptr;
  a.col = s->bsr.col;
  a.A = s->A64;
  a.b = d_b;
  a.x = d_x;
  a.u0 = P.p;
  a.m[0] = P.z;
  a.m[1] = P.q;
  a.pinv = P.pinv;
  a.pkind = pkind;
  a.x_zero = x_zero;
  a.max_iter = max_iter;
  a.tol = tol;
  a.part = P.partial;
  a.ell = R.ell;
  a.ell_off = R.ell_off;
  a.sc = P.sc;
  a.gb = (GridBarrier*)P.gbar;
  a.prof = prof;
  void* args[] = {(void*)&a};
  OD_KL(s);
  OD_CUDA(cudaLaunchCooperativeKernel(resident_kernel(R.smem), dim3(R.grid), dim3(32 * (R.warps + 2)), args,
                                      (size_t)R.bytes, s->ctx->stream));
  return OD_OK;
}

}  // namespace od
