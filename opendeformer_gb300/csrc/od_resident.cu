// The whole FP64 PCG solve of a chip-resident system in one launch, for the
// local preconditioners (none, Jacobi, block-Jacobi): every vector of the solve
// lives in registers, the matrix in shared memory (or, a little larger, in L2),
// and an iteration's sums run while its matrix product does.
//
// Form: Ghysels and Vanroose's pipelined PCG (2014), the recurrences and stop
// test of cgSolver.cpp:13-57 in exact arithmetic: u = M^-1 r, w = A u carried
// by recurrences, n = A M^-1 w formed every iteration, and the step lengths
// from the one set of dot products (r.u, w.u, r.r) that needs no n.
//
// What bounds it: latency, and the FP64 unit.  A system of this size is a few
// hundred multiply-adds per thread and iteration.  What an iteration waits for:
// a grid barrier 1.3-1.5 us over 152 CTAs (0.3 us inside a cluster), a read of
// the other CTAs' sums 0.4 us, FP64 operations at 64 cycles each on a warp's
// own unit (a division 554), and the instructions of single warps at some four
// cycles each.  So the CTA splits into
//
//   worker warps   one group of 10 block rows (30 DOFs, a lane each): the
//                  recurrences, the dot products, m = M^-1 w, the product;
//   a sync warp    publishes m (barrier) and releases the workers into the
//                  product;
//   three sum warps, one per dot product: add the CTA's values, publish them,
//                  add those of all CTAs; the first forms alpha and beta, all
//                  of it while the workers wait for m and multiply.
//
// Products and sums run on the integer units (od_fixed.cuh).  Systems of up to
// 192 groups run as one cluster, whose CTAs exchange m and the sums through
// each other's shared memory; larger ones as a cooperative grid over the chip.
//
// Microseconds per iteration, od_sparse.cu's persistent kernel (its pipelined
// form: barrier, sums and product one after the other) -> the split above with
// FP64 products -> this kernel: 108 DOFs 13.2 -> 3.3 -> 3.0, 2,160 DOFs 12.5 ->
// 5.0 -> 3.5, 6,900 DOFs 12.9 -> 5.0 -> 5.7, 55,488 DOFs 16.7 -> 10.1 -> 8.4
// (solves of 45 to 150 iterations, their start and end, 37 to 70 us, included).
// What is left is the dependent instructions of single warps (issue slots 21%
// used, FP64 units 24% on the largest) and the grid barrier.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "od_internal.h"
#include "od_grid.cuh"
#include "od_fixed.cuh"

namespace od {

constexpr int kRgRows = 10;                    // block rows per group (one worker warp)
constexpr int kRgLanes = 3 * kRgRows;          // DOFs per group, a lane each
constexpr int kRgMaxWarps = 20;                // worker warps per CTA
constexpr int kRgServe = 4;                    // warps that serve them: one syncs, three sum
constexpr int kRgMaxGrid = 160;                // CTAs (one per SM)
constexpr int kRgCluster = 16;                 // most CTAs of the cluster form, and
constexpr int kRgClusterWarps = 12;            // most worker warps of each
constexpr int kRgStepBytes = kRgLanes * 3 * 8 + kRgRows * 4;   // one step of a group: 10 blocks and their columns
constexpr int kRgRowBytes = 24;                // a block row's gathered entries: digits, or doubles
// Matrix steps whose gathered entries a lane loads together: all of a usual
// row's where 128 registers are left for them, else half (more warps per
// scheduler cover the second round trip).
constexpr int fx_pass(int max_warps) { return max_warps <= 12 ? 16 : 8; }
constexpr int kCtrStride = 1024;               // the counters are polled at once: words apart, not in one line

// The matrix steps of a group: step j holds the j-th blocks of its 10 block
// rows.  Four steps make a chunk (short rows padded with zeros): its values are
// [pair of steps][row r of a block][lane 3 t + c][step of the pair], so that a
// lane reads two steps' entries at once, and after all chunks' values come
// their column entries [t][step of the chunk].
__host__ __device__ constexpr int rg_padded(int steps) { return (steps + 3) & ~3; }
__device__ __forceinline__ int rg_value(int j, int r, int lane) {
  return (((j >> 1) * 3 + r) * kRgLanes + lane) * 2 + (j & 1);
}
__device__ __forceinline__ int rg_column(int j, int t) { return ((j >> 2) * kRgRows + t) * 4 + (j & 3); }

struct ResidentArgs {
  int nb, ngroups, warps;       // block rows; groups; worker warps per CTA
  const int* rp;
  const int* col;
  const int* diag;              // every block row's diagonal block
  const double* A;              // full BSR
  const double* b;
  double* x;
  double* u0;                   // A u of the start gathers it
  double* m[2];                 // M^-1 w by iteration parity (not the cluster form)
  int2* mx[2];                  // its digits
  const double* pinv;
  int pkind, x_zero, max_iter, patience;
  double tol;
  double* part;                 // 2 x 3 x gridDim.x partial sums
  int* epart;                   // 2 x gridDim.x largest exponents
  unsigned char* ell;           // matrix steps in global memory when they do not fit shared memory
  const int* ell_off;           // first step of every CTA there
  SolveScalars* sc;
  unsigned* ctr;                // counters of the barriers and of the three sums, kCtrStride apart
  int* timeout;
  unsigned long long* prof;
};

// named barriers of a CTA
enum { kBarM = 1, kBarDots = 2, kBarGo = 3, kBarStep = 4, kBarTot = 5 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// the same shared-memory address in CTA rank of the cluster
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ResidentShared {
  unsigned long long mbar[4];   // cluster form: barriers of m and of the three sums
  double cpart[2][3][kRgCluster];   // cluster form: every CTA's sums, by round parity
  int cep[2][kRgCluster];           // and largest exponents
  double ab[2];                 // alpha, beta
  double tot[3];                // the last grid-wide sums
  // by the parity of the round: the sync warp reads its round's word while the
  // first sum warp may be writing the next round's.  That one's next write of
  // the same word lies behind a kBarStep that the sync warp takes part in
  int stop[2];
  int status, iter, best;
  int emax;                     // the last vector's largest biased exponent
  int ew[kRgMaxWarps];          // its worker warps'
  int fail;                     // a wait ran out
  int seg[kRgMaxWarps];         // steps of every worker's group
  unsigned long long prof[kPcgProfSlots];   // phase times of worker 0, written out at the end
};

// A warp's arrival for its CTA at meeting point `which` and its wait for the
// arrivals of all CTAs in the epoch-th round; what the CTA wrote before (named
// barriers and __syncwarp in between) is visible after it.  Bounded; false,
// and the timeout flag set, when the wait ran out.
//   grid form: a counter that only grows (release reduction, relaxed polls,
//     one acquire load at the end: 0.1 us less than acquire polls);
//   cluster form: one mbarrier per CTA and meeting point, every CTA arriving
//     at every other's: 0.3 us instead of 1.4.
template <bool CL>
__device__ __forceinline__ bool meet(const ResidentArgs& P, ResidentShared& sh, int which, unsigned epoch) {
  const int lane = threadIdx.x & 31;
  if constexpr (CL) {
    const unsigned bar = smem_addr(&sh.mbar[which]);
    if (lane < (int)gridDim.x)
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(bar, lane)) : "memory");
    unsigned done = 0;
#pragma unroll 1
    for (int n = 0; n < (1 << 20) && !done; n++)
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(done) : "r"(bar), "r"((epoch - 1) & 1) : "memory");
    if (!done) *(volatile int*)P.timeout = 1;
    return __all_sync(0xffffffffu, done != 0);
  } else {
    int ok = 1;
    if (lane == 0) {
      unsigned* ctr = P.ctr + which * kCtrStride;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      const unsigned target = epoch * gridDim.x;
#pragma unroll 1
      for (unsigned spins = 1;; spins++) {
        unsigned cur;
        asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(cur) : "l"(ctr) : "memory");
        if ((int)(cur - target) >= 0) break;
        if ((spins & 31) == 0 && (*(volatile int*)P.timeout || spins > (unsigned)kSpinLimit)) {
          atomicExch(P.timeout, 1);
          ok = 0;
          break;
        }
      }
      unsigned last;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(last) : "l"(ctr) : "memory");
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
  }
}

// A sum warp's round for dot product j: the workers' values v[0..nt) summed
// over the CTA, published, then summed over the grid; every lane gets the sum,
// bitwise the same in every CTA.  slot: the round's parity.
template <bool CL>
__device__ __noinline__ double sum_grid(const ResidentArgs& P, ResidentShared& sh, const double* v, int nt, int j, int slot,
                                        unsigned epoch) {
  const int lane = threadIdx.x & 31, G = gridDim.x;
  constexpr int kUpCta = fx_up(kRgMaxWarps), kN = CL ? 1 : kRgMaxGrid / 32, kUpGrid = fx_up(kN);
  int e = 0;
#pragma unroll 4
  for (int i = lane; i < nt; i += 32) e = max(e, fx_biased_exp(v[i]));
  e = __reduce_max_sync(0xffffffffu, e);
  long long x = 0;
#pragma unroll 4
  for (int i = lane; i < nt; i += 32) x += fx_align<kUpCta>(v[i], e);
  const double t = fx_warp_total<kUpCta>(x, e);
  if (G == 1) return t;
  double* part = P.part + (size_t)(3 * slot + j) * G;
  if constexpr (CL) {
    if (lane < G)
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(smem_addr(&sh.cpart[slot][j][blockIdx.x]), lane)),
                   "d"(t) : "memory");
  } else {
    if (lane == 0) part[blockIdx.x] = t;
  }
  __syncwarp();
  if (!meet<CL>(P, sh, 1 + j, epoch)) sh.fail = 1;
  double in[kN];
  e = 0;
#pragma unroll
  for (int q = 0; q < kN; q++)
    in[q] = lane + 32 * q >= G ? 0.0 : CL ? sh.cpart[slot][j][lane] : __ldcg(part + lane + 32 * q);
#pragma unroll
  for (int q = 0; q < kN; q++) e = max(e, fx_biased_exp(in[q]));
  e = __reduce_max_sync(0xffffffffu, e);
  x = 0;
#pragma unroll
  for (int q = 0; q < kN; q++) x += fx_align<kUpGrid>(in[q], e);
  return fx_warp_total<kUpGrid>(x, e);
}

// The sync warp's round: the workers' writes published to every CTA, then the
// largest biased exponent of their vector over the grid.  go() releases the
// workers in between.
template <bool CL, class F>
__device__ __forceinline__ int sync_grid(const ResidentArgs& P, ResidentShared& sh, int slot, unsigned epoch, F go) {
  const int lane = threadIdx.x & 31, G = gridDim.x;
  int e = __reduce_max_sync(0xffffffffu, lane < P.warps ? sh.ew[lane] : 0);
  if (G == 1) {
    go();
    return e;
  }
  if constexpr (CL) {
    if (lane < G)
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(smem_addr(&sh.cep[slot][blockIdx.x]), lane)), "r"(e)
                   : "memory");
  } else {
    if (lane == 0) P.epart[slot * G + blockIdx.x] = e;
  }
  __syncwarp();
  if (!meet<CL>(P, sh, 0, epoch)) sh.fail = 1;
  go();
  e = 0;
  if constexpr (CL) {
    if (lane < G) e = sh.cep[slot][lane];
  } else {
#pragma unroll 1
    for (int c = lane; c < G; c += 32) e = max(e, __ldcg(P.epart + slot * G + c));
  }
  return __reduce_max_sync(0xffffffffu, e);
}

// Row r of block row [kb, ke) of A v in FP64: the start and the true residual.
// Out of line, like everything outside the iteration: the iteration's code is
// run by single warps and has to stay in the instruction caches.
__device__ __noinline__ double row_product64(const double* A, const int* col, int kb, int ke, int r, const double* v) {
  double y0 = 0.0, y1 = 0.0, y2 = 0.0;   // a chain per column: an FP64 operation takes 65 cycles
#pragma unroll 5
  for (int k = kb; k < ke; k++) {
    const double* a = A + 9 * (size_t)k + 3 * r;
    const double* xv = v + 3 * (size_t)col[k];
    y0 = fma(a[0], xv[0], y0);
    y1 = fma(a[1], xv[1], y1);
    y2 = fma(a[2], xv[2], y2);
  }
  return (y0 + y1) + y2;
}

// The same of an m whose digits do not fit: its doubles, gathered through the
// steps' column entries (m: byte offset of the doubles from the digits in the
// cluster form, the array else).
template <bool CL>
__device__ __noinline__ double row_product_m(const double* A, const unsigned* cols, int n, int t, int r, const double* m,
                                             unsigned m_off) {
  double y0 = 0.0, y1 = 0.0, y2 = 0.0;
#pragma unroll 1
  for (int k = 0; k < n; k++) {
    const double* a = A + 9 * (size_t)k + 3 * r;
    double x0, x1, x2;
    if constexpr (CL) {
      const unsigned at = cols[rg_column(k, t)] + m_off;
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x0) : "r"(at) : "memory");
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x1) : "r"(at + 8) : "memory");
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x2) : "r"(at + 16) : "memory");
    } else {
      const double* xv = reinterpret_cast<const double*>(reinterpret_cast<const char*>(m) + cols[rg_column(k, t)]);
      x0 = xv[0];
      x1 = xv[1];
      x2 = xv[2];
    }
    y0 = fma(a[0], x0, y0);
    y1 = fma(a[1], x1, y1);
    y2 = fma(a[2], x2, y2);
  }
  return (y0 + y1) + y2;
}

// One block row's matrix steps as digits, by its three lanes (r: this lane's
// row of the blocks, t: the block row's place in the group): the values over
// their columns' powers of two (fx_column_exp), then the scale of the row's sum of magnitudes (from the leading 21 bits of each,
// rounded up), then the digits in place.  A column entry is the gathered row's
// byte offset, in the cluster form its shared-memory address (mx: this CTA's
// first row).  Returns the scale, kFxNone for a row without one (its products
// stay in FP64).
template <bool CL>
__device__ __noinline__ int stage_rows(const ResidentArgs& P, double* raw, unsigned* cols, unsigned mx, int steps, int kb,
                                       int ke, int row, int t, int r) {
  int em = 0;
  constexpr int kAhead = 16;   // columns whose diagonal blocks are looked up together: two round trips for all
#pragma unroll 1
  for (int j0 = 0; j0 < steps; j0 += kAhead) {
    int dp[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++) dp[u] = kb + j0 + u < ke ? P.col[kb + j0 + u] : min(row, P.nb - 1);
#pragma unroll
    for (int u = 0; u < kAhead; u++) {
      if (r == 0 && j0 + u < steps) {
        unsigned at = kRgRowBytes * dp[u];
        if constexpr (CL) {
          const int g = dp[u] / kRgRows, G = gridDim.x, c = ((g + 1) * G - 1) / P.ngroups;
          at = cluster_addr(mx, c) + kRgRowBytes * (dp[u] - kRgRows * (c * P.ngroups / G));
        }
        cols[rg_column(j0 + u, t)] = at;
      }
      dp[u] = P.diag[dp[u]];
    }
#pragma unroll
    for (int q = 0; q < kAhead; q += 4) {   // steps come in fours
      if (j0 + q >= steps) break;
      double v[4][3], d[4][3];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = kb + j0 + q + u;
        const double *a = P.A + 9 * (size_t)k + 3 * r, *ad = P.A + 9 * (size_t)dp[q + u];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          v[u][c] = k < ke ? a[c] : 0.0;
          d[u][c] = ad[4 * c];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double x = fx_times_pow2(v[u][c], -fx_column_exp(d[u][c]));
          raw[rg_value(j0 + q + u, r, 3 * t + c)] = x;
          em = max(em, fx_biased_exp(x));
        }
    }
  }
  unsigned long long sum = 0;
#pragma unroll 2
  for (int j = 0; j < steps; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int hi = __double2hiint(raw[rg_value(j, r, 3 * t + c)]);
      const int d = em - ((hi >> 20) & 0x7ff);
      sum += (d < 31 ? ((unsigned)((hi & 0xfffff) | 0x100000) + 1u) >> d : 0u) + 1u;
    }
  const bool fits = row < P.nb && em >= kFxExpMin && em <= kFxExpMax;
  const int ea = (64 - __clzll((long long)sum)) + em - 1043;
  int2* dig = reinterpret_cast<int2*>(raw);
#pragma unroll 1
  for (int j = 0; j < steps; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int k = rg_value(j, r, 3 * t + c);
      const double v = raw[k];
      dig[k] = fits ? fx_digits(v, ea) : make_int2(0, 0);
    }
  return fits ? ea : kFxNone;
}

// One full sync of the grid outside the iteration: the stores before it are
// visible after it, and sh.tot[0] is the grid's sum of the workers' vals.
// False after a timeout.
template <bool CL>
__device__ __noinline__ bool full_sync(const ResidentArgs& P, ResidentShared& sh, const double* vals, unsigned epoch) {
  const int W = P.warps, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (w == W) {
    const int e = sync_grid<CL>(P, sh, epoch & 1, epoch, [] {});
    if (lane == 0) sh.emax = e;
  } else if (w == W + 1) {
    const double t = sum_grid<CL>(P, sh, vals, 32 * W, 0, epoch & 1, epoch);
    if (lane == 0) sh.tot[0] = t;
  }
  __syncthreads();
  return !sh.fail;
}

template <bool SMEM, int MAXW, bool CL>
__device__ __forceinline__ void resident_body(const ResidentArgs& P, unsigned char* rg_dsm, ResidentShared& sh) {
  const int G = gridDim.x, W = P.warps, nt = 32 * W;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gb0 = (int)((long long)blockIdx.x * P.ngroups / G);
  const int gb1 = (int)((long long)(blockIdx.x + 1) * P.ngroups / G);
  const bool worker = w < W;
  const int rsub = lane % 3;
  // dynamic shared memory: the workers' values [3][nt]; cluster form: m's
  // digits and doubles, two buffers of each; the matrix steps
  double* vals = reinterpret_cast<double*>(rg_dsm);
  const int mrow = W * kRgRows * kRgRowBytes;         // one buffer
  unsigned char* mdig = rg_dsm + 3 * sizeof(double) * nt;
  unsigned char* steps_at = mdig + (CL ? 4 * mrow : 0);

  // ---- the group of this warp and its matrix steps
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
  const int steps = rg_padded(__reduce_max_sync(0xffffffffu, ke - kb));
  if (worker && lane == 0) sh.seg[w] = steps;
  __syncthreads();
  const int t10 = min(lane / 3, kRgRows - 1);
  const int4* eA = nullptr;      // this lane's values, as digits at the row's scale ea
  unsigned* cols = nullptr;
  int ea = kFxNone;
  if (worker) {
    int off = 0;
#pragma unroll 1
    for (int q = 0; q < w; q++) off += sh.seg[q];
    unsigned char* base = SMEM ? steps_at : P.ell + (size_t)P.ell_off[blockIdx.x] * kRgStepBytes;
    base += (size_t)off * kRgStepBytes;
    eA = reinterpret_cast<const int4*>(base) + min(lane, kRgLanes - 1);
    cols = reinterpret_cast<unsigned*>(base + (size_t)steps * kRgLanes * 3 * 8);
    if (lane < kRgLanes)
      ea = stage_rows<CL>(P, reinterpret_cast<double*>(base), cols, CL ? smem_addr(mdig) : 0u, steps, kb, ke, row, t10, rsub);
    __syncwarp();
  }
  const bool row_fx = ea != kFxNone;
  const int kc = valid ? fx_column_exp(P.A[9 * (size_t)P.diag[row] + 4 * rsub]) : 0;   // of this lane's entry
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
  // This lane's row of A m from digits.  Lane 3 t + c takes column c of the
  // blocks of block row t: one gathered entry a step (a pass's all issued
  // together, so the round trip is paid once), three rows of products; the
  // three lanes' sums of a row are exchanged at the end.  Integer sums: the
  // order does not matter.
  auto product_fx = [&](int par, int E) -> double {
    constexpr int kPass = fx_pass(MAXW), kChunks = kPass / 4;
    FxAcc acc[3];
    const char* mg = reinterpret_cast<const char*>(P.mx[par]) + 8 * rsub;
    const unsigned ms = par * mrow + 8 * rsub;
    const int4* eC = reinterpret_cast<const int4*>(cols) + t10;
#pragma unroll 1
    for (int j0 = 0; j0 < steps; j0 += kPass) {
      int2 xv[kPass];
#pragma unroll
      for (int c = 0; c < kChunks; c++)
        if (j0 + 4 * c < steps) {
          const int4 at = eC[(j0 / 4 + c) * kRgRows];
          const unsigned a4[4] = {(unsigned)at.x, (unsigned)at.y, (unsigned)at.z, (unsigned)at.w};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            int2& v = xv[4 * c + q];
            if constexpr (CL)
              asm volatile("ld.shared::cluster.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a4[q] + ms) : "memory");
            else
              v = *reinterpret_cast<const int2*>(mg + a4[q]);
          }
        }
#pragma unroll
      for (int c = 0; c < kChunks; c++) {
        if (j0 + 4 * c < steps) {
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int r = 0; r < 3; r++) {
              const int4 a = eA[(((j0 + 4 * c) / 2 + h) * 3 + r) * kRgLanes];
              acc[r].add(make_int2(a.x, a.y), xv[4 * c + 2 * h]);
              acc[r].add(make_int2(a.z, a.w), xv[4 * c + 2 * h + 1]);
            }
        }
        if (c % 2 == 1) {
#pragma unroll
          for (int r = 0; r < 3; r++) acc[r].carry();
        }
      }
    }
    FxAcc own;
    own.hh = rsub == 0 ? acc[0].hh : rsub == 1 ? acc[1].hh : acc[2].hh;
    own.mid = rsub == 0 ? acc[0].mid : rsub == 1 ? acc[1].mid : acc[2].mid;
#pragma unroll
    for (int d = 1; d < 3; d++) {
      const int to = rsub + d < 3 ? rsub + d : rsub + d - 3;        // the row this lane gives away
      const int from = rsub >= d ? rsub - d : rsub - d + 3;         // the lane that gives this one its row
      const long long gh = to == 0 ? acc[0].hh : to == 1 ? acc[1].hh : acc[2].hh;
      const long long gm = to == 0 ? acc[0].mid : to == 1 ? acc[1].mid : acc[2].mid;
      own.hh += __shfl_sync(0xffffffffu, gh, l0 + from);
      own.mid += __shfl_sync(0xffffffffu, gm, l0 + from);
    }
    return own.value(ea, E);
  };

  // ---- start: r = b - A x, u = M^-1 r, w = A u (cgSolver.cpp:20-30)
  unsigned epoch = 1;     // rounds so far
  double x = 0.0, r = 0.0, u = 0.0, wv = 0.0, bv = 0.0;
  if (worker) {
    if (valid) bv = r = P.b[i];
    if (!P.x_zero) {
      if (valid) x = P.x[i];
      r -= row_product64(P.A, P.col, kb, ke, rsub, P.x);
    }
    u = precond(r);
    if (valid) P.u0[i] = u;
    vals[threadIdx.x] = valid ? bv * bv : 0.0;
    const int e = __reduce_max_sync(0xffffffffu, valid ? fx_biased_exp(u, kc) : 0);
    if (lane == 0) sh.ew[w] = e;
  }
  if (!full_sync<CL>(P, sh, vals, epoch)) return;
  const double bb = sh.tot[0], eps = bb * P.tol * P.tol;
  if (worker) wv = row_product64(P.A, P.col, kb, ke, rsub, P.u0);
  if (!valid) r = u = wv = 0.0;   // idle lanes add nothing

  const bool timer = P.prof && blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long t_prev = 0;
  auto stamp = [&](int slot) {
    if (!timer) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (slot >= 0) sh.prof[slot] += t - t_prev;
    t_prev = t;
  };
  stamp(-1);
  const int all = nt + 32 * kRgServe;
  // the scale of m's digits (of its entries times their columns' powers of two):
  // one place above the last vector's maximum, which shrinks by up to two places
  // an iteration and hardly grows; for the first m, which is like M^-1 A u, u's.
  // The second m is three places up: under loads on part of the body it grows by
  // 1 to 4 places over the first (a product in FP64 instead: 19 us on 98k tets)
  auto next_scale = [](int emax, int up) { return emax < kFxExpMin || emax > kFxExpMax ? kFxNone : emax - 1022 + up; };
  int E = next_scale(sh.emax, 1), up = kFxSlack;
  if (worker) {
    double p = 0.0, q = 0.0, s = 0.0, z = 0.0, u_old = 0.0, alpha = 0.0, beta = 0.0;
    const int m_own = kRgRowBytes * (kRgRows * w + lane / 3) + 8 * rsub;   // cluster form: this lane's entry
#pragma unroll 1
    for (int par = 0;; par ^= 1) {
      __syncwarp();
      vals[threadIdx.x] = r * u;
      vals[nt + threadIdx.x] = wv * u;
      vals[2 * nt + threadIdx.x] = r * r;
      bar_arrive(kBarDots, nt + 96);
      const double m = precond(wv);
      if (valid) {
        const int2 d = fx_digits(m, E - kc);
        if constexpr (CL) {
          *reinterpret_cast<int2*>(mdig + par * mrow + m_own) = d;
          *reinterpret_cast<double*>(mdig + (2 + par) * mrow + m_own) = m;
        } else {
          P.mx[par][i] = d;
          P.m[par][i] = m;
        }
      }
      const int e = __reduce_max_sync(0xffffffffu, valid ? fx_biased_exp(m, kc) : 0);
      if (lane == 0) sh.ew[w] = e;
      __syncwarp();
      bar_arrive(kBarM, nt + 32);
      stamp(2);
      bar_sync(kBarGo, nt + 32);
      double n = product_fx(par, E);
      stamp(0);
      // the last iteration's, off the path to the sums
      p = fma(beta, p, u_old);
      x = fma(alpha, p, x);
      bar_sync(kBarStep, all);
      stamp(3);
      if (sh.stop[par]) break;
      const int top = sh.emax - 1022;          // 2^top is above m's scaled entries
      if (valid && (top > E || top < E - kFxSlack || !row_fx))
        n = row_product_m<CL>(P.A + 9 * (size_t)kb, cols, ke - kb, t10, rsub, P.m[par], (2 + par) * mrow);
      E = next_scale(sh.emax, up);
      up = 1;
      alpha = sh.ab[0];
      beta = sh.ab[1];
      z = fma(beta, z, n);
      q = fma(beta, q, m);
      s = fma(beta, s, wv);
      u_old = u;
      wv = fma(-alpha, z, wv);
      u = fma(-alpha, q, u);
      r = fma(-alpha, s, r);
      if (!valid) r = u = wv = 0.0;
      if (timer) sh.prof[kPcgPhases] += 1;
    }
  } else if (w == W) {
#pragma unroll 1
    for (int par = 0;; par ^= 1) {
      bar_sync(kBarM, nt + 32);
      epoch++;
      const int e = sync_grid<CL>(P, sh, epoch & 1, epoch, [&] {
        __syncwarp();
        bar_arrive(kBarGo, nt + 32);
      });
      if (lane == 0) sh.emax = e;
      __syncwarp();
      bar_sync(kBarStep, all);
      if (sh.stop[par]) break;
    }
  } else {
    // sum warp j takes dot product j; the first forms the step lengths
    const int j = w - W - 1;
    double gam_inv = 0.0, den_k = 0.0;   // 1 / gamma and den / gamma^2 of the last iteration
    // the iteration at which r.r last had halved, and its upper half then, for the
    // next round's stop test.  Counted here, while the workers update (by the third sum
    // warp, which no round waits for, an iteration took 0.35 us more on 98k tets)
    int best = 0, best_hi = 0x7fffffff;
    bool stalled = false;
#pragma unroll 1
    for (int it = 0;; it++) {
      bar_sync(kBarDots, nt + 96);
      epoch++;
      // (the start's round met at the first sum's point only)
      const double t = sum_grid<CL>(P, sh, vals + j * nt, nt, j, epoch & 1, j == 0 ? epoch : epoch - 1);
      if (lane == 0) sh.tot[j] = t;
      __syncwarp();
      if (j > 0) {
        bar_arrive(kBarTot, 96);
        bar_sync(kBarStep, all);
        if (sh.stop[it & 1]) break;
        continue;
      }
      // beta = gamma / gamma_prev, alpha = gamma / den with den = delta -
      // beta gamma / alpha_prev, and gamma / alpha_prev = beta den_prev: one
      // division on the path
      const double beta = t * gam_inv, gg = t * t * den_k;
      bar_sync(kBarTot, 96);
      const double rr = sh.tot[2];
      const double den = sh.tot[1] - gg;
      const double alpha = t / den;
      int stop = 0, status = OD_OK;
      if (!isfinite(rr)) {
        stop = 1;
        status = OD_ERR_NAN;
      } else if (!(rr > eps) || it >= P.max_iter) {
        stop = 1;
      } else if (stalled) {
        stop = 1;
        status = OD_ERR_NOT_CONVERGED;
      } else if (!isfinite(alpha) || !isfinite(beta)) {
        stop = 1;
        status = OD_ERR_NAN;
      }
      // a wait that ran out (the barrier's is seen an iteration later at most)
      if (*(volatile int*)&sh.fail) stop = 1;
      if (lane == 0) {
        sh.ab[0] = alpha;
        sh.ab[1] = beta;
        sh.stop[it & 1] = stop;
        if (stop) {
          sh.status = status;
          sh.iter = it;
          sh.best = __double2hiint(rr) < best_hi - (1 << 20) ? it : best;
        }
      }
      __syncwarp();
      bar_sync(kBarStep, all);
      if (sh.stop[it & 1]) break;   // lane 0's word: the lanes' reads of fail may differ
      if (__double2hiint(rr) < best_hi - (1 << 20)) {
        best_hi = __double2hiint(rr);
        best = it;
      }
      stalled = P.patience > 0 && it + 1 - best > P.patience + (best >> 2);
      gam_inv = 1.0 / t;
      den_k = den * gam_inv * gam_inv;
    }
  }
  __syncthreads();
  if (sh.fail) return;
  epoch = 2 + (unsigned)sh.iter;   // the start's round and one per iteration and for the stop
  const double gam_end = sh.tot[0], rr_end = sh.tot[2];
  __syncthreads();

  // ---- write x, then the true residual ||b - A x||^2
  if (valid) P.x[i] = x;
  if (!full_sync<CL>(P, sh, vals, epoch + 1)) return;
  if (worker) {
    const double d = bv - row_product64(P.A, P.col, kb, ke, rsub, P.x);
    vals[threadIdx.x] = valid ? d * d : 0.0;
  }
  if (!full_sync<CL>(P, sh, vals, epoch + 2)) return;
  if (timer)
    for (int k = 0; k < kPcgProfSlots; k++) P.prof[k] += sh.prof[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    SolveScalars* sc = P.sc;
    sc->rz[0] = gam_end;
    sc->rr = rr_end;
    sc->bb = bb;
    sc->eps = eps;
    sc->iter = sh.iter;
    sc->max_iter = P.max_iter;
    sc->status = sh.status;
    sc->best = sh.best;
    sc->tr_num = sh.tot[0];
    sc->tr_den = bb;
    sc->done = 1;
  }
}

template <bool SMEM, int MAXW, bool CL>
__global__ void __launch_bounds__(32 * (MAXW + kRgServe), 1) pcg_resident_kernel(const ResidentArgs P) {
  extern __shared__ __align__(16) unsigned char rg_dsm[];
  __shared__ ResidentShared sh;
  if (threadIdx.x == 0) {
    sh.fail = 0;
    sh.stop[0] = sh.stop[1] = 0;
    sh.status = OD_OK;
    for (int k = 0; k < kPcgProfSlots; k++) sh.prof[k] = 0;
    if constexpr (CL)
      for (int k = 0; k < 4; k++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sh.mbar[k])), "r"(gridDim.x) : "memory");
  }
  if constexpr (CL) {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cluster_barrier();   // no CTA reaches for another's shared memory before it is there
  } else {
    __syncthreads();
  }
  resident_body<SMEM, MAXW, CL>(P, rg_dsm, sh);
  if constexpr (CL) {
    __syncwarp();
    cluster_barrier();   // nor after it is gone
  }
}

// 12, 16 and 20 worker warps leave 128, 96 and 80 registers a thread
template <int MAXW>
static const void* resident_kernel_of(bool smem, bool cluster) {
  if (cluster)
    return smem ? (const void*)pcg_resident_kernel<true, MAXW, true> : (const void*)pcg_resident_kernel<false, MAXW, true>;
  return smem ? (const void*)pcg_resident_kernel<true, MAXW, false> : (const void*)pcg_resident_kernel<false, MAXW, false>;
}
static const void* resident_kernel(bool smem, int warps, bool cluster) {
  return warps <= 12   ? resident_kernel_of<12>(smem, cluster)
         : warps <= 16 ? resident_kernel_of<16>(smem, cluster)
                       : resident_kernel_of<kRgMaxWarps>(smem, cluster);
}

static cudaError_t resident_launch(const ResidentPlan& R, const ResidentArgs& a, cudaStream_t st) {
  void* args[] = {(void*)&a};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(R.grid);
  cfg.blockDim = dim3(32 * (R.warps + kRgServe));
  cfg.dynamicSmemBytes = (size_t)R.bytes;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  if (R.cluster) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = R.grid;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, resident_kernel(R.smem, R.warps, R.cluster), args);
}

// The shape of a scene's resident solve: CTAs, worker warps, where the
// matrix lives.  Leaves warps = 0 when the system is too large for one group
// per worker warp (the persistent kernel of od_sparse.cu takes it).
od_status resident_plan(Scene* s) {
  ResidentPlan& R = s->pcg.res;
  R = ResidentPlan();
  const int nb = s->bsr.nb;
  const int sms = s->ctx->num_sms;
  if (s->pcg.coop_grid <= 0 || sms <= 0 || sms > kRgMaxGrid || nb <= 0 || (int)s->hbsr_rp.size() != nb + 1) return OD_OK;
  const std::vector<int>& rp = s->hbsr_rp;
  const int ng = (nb + kRgRows - 1) / kRgRows;
  const char* env = std::getenv("OD_GB300_PCG_SMEM");   // 0: the matrix from L2 (the same operations)
  const bool allow_smem = !(env && env[0] == '0');
  int dev_max = 0;
  cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->ctx->device);
  const long long cap = (long long)dev_max - 1024;
  std::vector<int> off;
  // matrix steps of every CTA: off[c], and the largest
  auto steps_of = [&](int G) {
    off.assign((size_t)G + 1, 0);
    int most = 0;
    for (int c = 0; c < G; c++) {
      int steps = 0;
      for (int g = (int)((long long)c * ng / G); g < (int)((long long)(c + 1) * ng / G); g++) {
        int m = 0;
        for (int r = g * kRgRows; r < std::min(nb, (g + 1) * kRgRows); r++) m = std::max(m, rp[r + 1] - rp[r]);
        steps += rg_padded(m);
      }
      off[c + 1] = off[c] + steps;
      most = std::max(most, steps);
    }
    return (long long)most;
  };
  auto try_shape = [&](int G, bool smem, bool cluster) {
    const int warps = (ng + G - 1) / G;
    if (warps > kRgMaxWarps) return false;
    const long long bytes = 3LL * sizeof(double) * 32 * warps + (cluster ? 4LL * warps * kRgRows * kRgRowBytes : 0) +
                            (smem ? steps_of(G) * kRgStepBytes : 0);
    const void* fn = resident_kernel(smem, warps, cluster);
    cudaFuncAttributes fa{};
    bool ok = cudaFuncGetAttributes(&fa, fn) == cudaSuccess && bytes + (long long)fa.sharedSizeBytes <= cap;
    // the attributes are per function, shared by every scene: set to the most
    // the device allows, never to one scene's size
    ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(cap - (long long)fa.sharedSizeBytes)) == cudaSuccess;
    if (ok && cluster && G > 8) ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ok && cluster) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(G);
      cfg.blockDim = dim3(32 * (warps + kRgServe));
      cfg.dynamicSmemBytes = (size_t)bytes;
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = G;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      int n = 0;
      ok = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= 1;
    } else if (ok) {
      int bps = 0;
      ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, 32 * (warps + kRgServe), (size_t)bytes) == cudaSuccess &&
           bps >= 1;
    }
    cudaGetLastError();   // a refused attribute is not an error of the scene
    if (!ok) return false;
    R.grid = G;
    R.warps = warps;
    R.bytes = (int)bytes;
    R.smem = smem;
    R.cluster = cluster;
    if (!smem) {
      steps_of(G);
      R.off = off;
    }
    return true;
  };
  // One cluster, of as few CTAs as leave each of the SM's four schedulers one
  // worker, up to kRgClusterWarps workers on 16 CTAs: an iteration of 2,160
  // DOFs takes 3.5 us there and 5.5 us on 72 CTAs of a grid; at 15 workers
  // (6,900 DOFs) it takes 6.0 us against 5.6, the FP64 units being the limit.
  bool found = false;
  for (int G = 1; G <= kRgCluster && !found; G *= 2)
    found = (ng <= 4 * G || G == kRgCluster) && ng >= G && ng <= kRgClusterWarps * G && try_shape(G, true, true);
  const int G = std::min(sms, ng);
  found = found || try_shape(G, true, false);
  // the same shape, so the same sums
  if (found && !allow_smem) found = try_shape(R.grid, false, R.cluster);
  if (!found) try_shape(G, false, false);
  return OD_OK;
}

void resident_free(ResidentPlan* R) {
  cudaFree(R->mx);
  cudaFree(R->ctr);
  cudaFree(R->ell);
  cudaFree(R->ell_off);
  *R = ResidentPlan();
}

// The plan's device memory, with the scene from its first such solve on; without
// room for it the plan is given up (warps 0) and the persistent kernel of
// od_sparse.cu takes the system.
od_status resident_ready(Scene* s) {
  ResidentPlan& R = s->pcg.res;
  const bool ell = !R.smem && !R.ell, grid = !R.cluster && !R.ctr;
  if (R.warps == 0 || !(ell || grid)) return OD_OK;
  const size_t b_off = sizeof(int) * R.off.size(), b_ell = ell ? (size_t)std::max(1, R.off.back()) * kRgStepBytes : 0,
               b_mx = 2 * 3 * sizeof(int2) * (size_t)s->bsr.nb, b_ctr = 4 * kCtrStride * sizeof(unsigned);
  cudaError_t e = cudaSuccess;
  if (ell) {
    e = plan_malloc(&R.ell_off, b_off);
    if (e == cudaSuccess) e = plan_malloc(&R.ell, b_ell);
    if (e == cudaSuccess) e = cudaMemcpy(R.ell_off, R.off.data(), b_off, cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess && grid) {
    e = plan_malloc(&R.mx, b_mx);
    if (e == cudaSuccess) e = plan_malloc(&R.ctr, b_ctr);
  }
  if (e != cudaSuccess) {
    resident_free(&R);
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "chip-resident PCG plan");
    cudaGetLastError();
    return OD_OK;
  }
  s->device_bytes += (long long)((ell ? b_off + b_ell : 0) + (grid ? b_mx + b_ctr : 0));
  return OD_OK;
}

od_status resident_solve(Scene* s, const double* d_b, double* d_x, int pkind, double tol, int max_iter, int patience,
                         bool x_zero, unsigned long long* prof) {
  Pcg& P = s->pcg;
  ResidentPlan& R = P.res;
  if (!R.cluster) OD_CUDA(cudaMemsetAsync(R.ctr, 0, 4 * kCtrStride * sizeof(unsigned), s->ctx->stream));
  ResidentArgs a{};
  a.nb = s->bsr.nb;
  a.ngroups = (s->bsr.nb + kRgRows - 1) / kRgRows;
  a.warps = R.warps;
  a.rp = s->bsr.row_ptr;
  a.col = s->bsr.col;
  a.diag = s->bsr.diag_pos;
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
  a.patience = patience;
  a.tol = tol;
  a.part = P.partial;
  a.epart = (int*)(P.partial + 6 * (size_t)R.grid);   // partial holds 8 per SM
  a.mx[0] = (int2*)R.mx;
  a.mx[1] = (int2*)R.mx + 3 * (size_t)s->bsr.nb;
  a.ell = R.ell;
  a.ell_off = R.ell_off;
  a.sc = P.sc;
  a.ctr = (unsigned*)R.ctr;
  a.timeout = &((GridBarrier*)P.gbar)->timeout;
  a.prof = prof;
  OD_KL(s);
  OD_CUDA(resident_launch(R, a, s->ctx->stream));
  return OD_OK;
}

}  // namespace od
