// FP64 PCG of systems beyond the chip-resident one (od_resident.cu): one
// cooperative launch, the recurrence form (q = A z + beta q, p = z + beta p:
// two grid syncs an iteration), products in fixed point (od_fixed.cuh), every
// vector in its CTA's shared memory.
//
// What bounds it: the matrix's bytes, from HBM and L2, once an iteration.  The
// FP64 products that this replaces held the FP64 unit for 27 of 43 us on
// 655k tets; as digits a product is three wide multiply-adds at a thirtieth
// of that.  So that nothing else is waited for:
// - a CTA's block rows are sorted by length before they are grouped in tens
//   (the five-tetrahedra cubes' rows have 7 and 19 blocks in turn), and all
//   its matrix steps are dealt to its warps evenly: the sums are integers, so a
//   group may be split between two warps without changing them;
// - x, p, q and p.q are done by the lanes that have just formed the product, in
//   the shadow of the other warps' loads.
//
// An iteration, FP64 products before and this: 237,600 DOFs (94 MB of digits)
// 42.5 -> 30.7 us, 424,320 (155 MB) 69.4 -> 46.4, 617,760 (300 MB) 87.0 ->
// 69.9; of the 46.4 the product takes 27, at 5.6 TB/s (a plain read of as many
// bytes: 21), its wait for the slowest CTA and the sum 8, the update 7.  The
// digits and the products with x, in FP64, cost a solve 0.2 ms at the first size
// and 0.3 at the second.  With the matrix loaded by the computing warps
// instead of through a ring in shared memory a product took 54 us.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "od_internal.h"
#include "od_grid.cuh"
#include "od_fixed.cuh"

namespace od {

constexpr int kWdWarps = 16;
constexpr int kWdThreads = 32 * kWdWarps;
constexpr int kWdRows = 10;                    // block rows per group, three lanes each
constexpr int kWdLanes = 3 * kWdRows;
constexpr int kWdMaxGrid = 160;
constexpr int kWdSteps = 4;                    // matrix steps of a record
constexpr int kWdRec = 16 * 6 * kWdLanes + 16 * kWdRows;   // bytes of a record: the steps' digits and their columns
// Bytes of the matrix that are left to L2's own order; the rest is marked to go
// first, so that these (and the vectors) stay.  At 155 MB all: 57.1 us an
// iteration, 120 MB: 57.5, 75: 52.5, 45: 50.8, 15: 50.7; at 300 MB 85, .., 40:
// 75.7, 30: 73.7.
constexpr long long kWdKeep = 45000000;
constexpr int kWdStagesMin = 2, kWdStagesMax = 4;          // records of a warp's ring
constexpr int kWdCtr = 1024;                   // counters lie words apart: they are polled at once
static_assert(kWdRec % 16 == 0, "bulk copies");

// One scene's plan (device arrays; built with the scene's first such solve)
struct WidePlan {
  int grid = 0, ngroups = 0, most = 0, records = 0;   // CTAs, groups, most groups of a CTA, records
  int stages = 0;
  bool staged = false;
  size_t smem = 0;
  int* ints = nullptr;
  const int *cg = nullptr, *goff = nullptr, *perm = nullptr, *slot = nullptr;
  unsigned char* rec = nullptr;
  int* ea = nullptr;         // row scales; one more: whether a row has none
  int* kx = nullptr;         // columns' powers of two, by places
  int2* zd = nullptr;
  double *zg = nullptr, *xg = nullptr, *pg = nullptr, *zv = nullptr, *inv = nullptr;
  unsigned* ctr = nullptr;
};

struct WideArgs {
  int nb, ngroups, most, pkind, max_iter, stages, x_zero, keep;   // keep: of 1,024 parts of the matrix those to stay in L2
 
  const int* cg;             // first group of every CTA
  const int* goff;           // first record of every group
  const int* perm;           // block row of every place (ten a group), -1: none
  const int* slot;           // place of every block row
  const int *rp, *col;
  const double *A, *b, *pinv;
  double* x;
  unsigned char* rec;        // per record [2][row of the block][30 lanes] digits of two steps (lane 3 t + c: column c of the group's row t), [10] the four columns, as byte offsets in zd
  int* ea;                   // [group][30] scales; then the flag
  const int* diag;           // every block row's diagonal block
  int* kx;                   // every place's power of two (fx_column_exp)
  int2* zd;                  // digits of the gathered vector, by places
  double* zg;                // the vector itself, where digits cannot be had; x at the start and the end
  double *xg, *pg, *zv, *inv;   // x, p, z; the preconditioner [3][entries]; by places
  double tol;
  double* part;              // [2][3][G] partial sums
  int* epart;                // [2][G] largest exponents
  unsigned* ctr;
  int* timeout;
  SolveScalars* sc;
  unsigned long long* prof;
};

struct WideShared {
  double vals[3][kWdThreads];
  long long head[kWdWarps][kWdLanes][2];   // sums of the groups that the next warp ends
  double tot[3];
  int ew[kWdWarps];
  int emax, fail;
  unsigned calls[3];                       // of each sum's counter
  unsigned long long full[kWdWarps][kWdStagesMax];
  int stage[kWdWarps], parity[kWdWarps];   // the rings between two products
  int from[kWdWarps], count[kWdWarps], group[kWdWarps], end[kWdWarps], inside[kWdWarps];   // the warps' shares: records, the first one's group and its end, whether it began before
  int c0, c1;                              // this CTA's groups
};

__global__ void __launch_bounds__(256) wide_scale_kernel(const __grid_constant__ WideArgs P) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= kWdLanes * P.ngroups) return;
  const int row = P.perm[i / 3];
  P.kx[i] = row >= 0 ? fx_column_exp(P.A[9 * (size_t)P.diag[row] + 4 * (i % 3)]) : 0;
}

// The matrix as digits, columns over their powers of two, a warp per group: the scale of every row's sum of
// magnitudes (from the leading 21 bits of each value, rounded up), then the
// digits.  Reads the matrix twice and writes it once: memory-bound.
__global__ void __launch_bounds__(256) wide_stage_kernel(const __grid_constant__ WideArgs P, int first) {
  const int g = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= P.ngroups || lane >= kWdLanes) return;
  const int t = lane / 3, r = lane % 3, row = P.perm[kWdRows * g + t];
  const int p0 = P.goff[g], np = P.goff[g + 1] - p0;
  const int kb = row >= 0 ? P.rp[row] : 0, n = row >= 0 ? P.rp[row + 1] - kb : 0;
  unsigned char* rec0 = P.rec + (size_t)p0 * kWdRec;
  const int4* at = reinterpret_cast<const int4*>(rec0 + 16 * 6 * kWdLanes) + t;   // a record's columns, kWdRec apart
  auto columns = [&](int p) { return at[(size_t)p * (kWdRec / 16)]; };
  if (first) {
    if (r == 0)
#pragma unroll 2
      for (int p = 0; p < np; p++) {
        int c[kWdSteps];
#pragma unroll
        for (int q = 0; q < kWdSteps; q++) {
          const int j = kWdSteps * p + q;
          c[q] = 24 * (j < n ? P.slot[P.col[kb + j]] : kWdRows * g + t);
        }
        reinterpret_cast<int4*>(rec0 + (size_t)p * kWdRec + 16 * 6 * kWdLanes)[t] = make_int4(c[0], c[1], c[2], c[3]);
      }
    __syncwarp((1u << kWdLanes) - 1);
  }
  int em = 0;
  unsigned long long sum = 0;
#pragma unroll 1
  for (int p = 0; p < np; p++) {
    const int4 c4 = columns(p);
    const int c[kWdSteps] = {c4.x / 8, c4.y / 8, c4.z / 8, c4.w / 8};
    double v[kWdSteps][3];
    int k[kWdSteps][3];
#pragma unroll
    for (int q = 0; q < kWdSteps; q++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        v[q][i] = kWdSteps * p + q < n ? P.A[9 * (size_t)(kb + kWdSteps * p + q) + 3 * r + i] : 0.0;
        k[q][i] = P.kx[c[q] + i];
      }
#pragma unroll
    for (int q = 0; q < kWdSteps; q++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const int hi = __double2hiint(v[q][i]), e = fx_biased_exp(v[q][i], -k[q][i]);
        if (e > em) {
          sum = (sum >> min(e - em, 63)) + 1;
          em = e;
        }
        const int d = em - e;
        sum += (d < 31 ? ((unsigned)((hi & 0xfffff) | 0x100000) + 1u) >> d : 0u) + 1u;
      }
  }
  const bool fits = em >= kFxExpMin && em <= kFxExpMax;
  const int ea = fits ? (64 - __clzll((long long)sum)) + em - 1043 : kFxNone;
  P.ea[kWdLanes * g + lane] = ea;
  if (row >= 0 && !fits) P.ea[kWdLanes * P.ngroups] = 1;
  const int ent = kWdLanes * g + lane, ne = kWdLanes * P.ngroups;
  if (P.pkind == OD_PRECOND_JACOBI) P.inv[ent] = row >= 0 ? P.pinv[3 * (size_t)row + r] : 0.0;
  if (P.pkind == OD_PRECOND_BLOCK_JACOBI)
    for (int c = 0; c < 3; c++) P.inv[(size_t)c * ne + ent] = row >= 0 ? P.pinv[9 * (size_t)row + 3 * r + c] : 0.0;
#pragma unroll 1
  for (int p = 0; p < np; p++) {
    int4* rec = reinterpret_cast<int4*>(rec0 + (size_t)p * kWdRec);
    const int4 c4 = columns(p);
    const int c[kWdSteps] = {c4.x / 8, c4.y / 8, c4.z / 8, c4.w / 8};
    int2 d[kWdSteps][3];
#pragma unroll
    for (int q = 0; q < kWdSteps; q++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const int j = kWdSteps * p + q;
        d[q][i] = fits && j < n ? fx_digits(P.A[9 * (size_t)(kb + j) + 3 * r + i], ea + P.kx[c[q] + i]) : make_int2(0, 0);
      }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < 3; i++)
        rec[(3 * h + r) * kWdLanes + 3 * t + i] = make_int4(d[2 * h][i].x, d[2 * h][i].y, d[2 * h + 1][i].x, d[2 * h + 1][i].y);
  }
}

// One lane's bounded wait for every CTA's epoch-th arrival at a counter
__device__ __forceinline__ void wide_poll(const WideArgs& P, WideShared& sh, const unsigned* ctr, unsigned epoch) {
  const unsigned target = epoch * gridDim.x;
#pragma unroll 1
  for (unsigned spins = 1;; spins++) {
    unsigned cur;
    asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(cur) : "l"(ctr) : "memory");
    if ((int)(cur - target) >= 0) break;
    if ((spins & 31) == 0 && (*(volatile int*)P.timeout || spins > (unsigned)kSpinLimit)) {
      atomicExch(P.timeout, 1);
      sh.fail = 1;
      break;
    }
  }
  [[maybe_unused]] unsigned last;   // what the arrivals released
  asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(last) : "l"(ctr) : "memory");
}

__device__ __forceinline__ unsigned wd_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// bounded wait for a stage; false when it ran out
__device__ __forceinline__ bool wide_full(unsigned long long* bar, unsigned parity) {
#pragma unroll 1
  for (int i = 0; i < 1 << 24; i++) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(wd_smem(bar)), "r"(parity)
                 : "memory");
    if (ok) return true;
  }
  return false;
}
// one record into a stage (lane 0)
__device__ __forceinline__ unsigned long long wide_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void wide_load(const WideArgs& P, unsigned char* dst, int record, unsigned long long* bar, bool keep) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(wd_smem(bar)), "r"(kWdRec) : "memory");
  if (keep)
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(wd_smem(dst)),
                 "l"(P.rec + (size_t)record * kWdRec), "r"(kWdRec), "r"(wd_smem(bar))
                 : "memory");
  else
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                     wd_smem(dst)),
                 "l"(P.rec + (size_t)record * kWdRec), "r"(kWdRec), "r"(wd_smem(bar)), "l"(wide_policy())
                 : "memory");
}
// a warp's share of its CTA's records
__device__ __forceinline__ int2 wide_share(const WideArgs& P) {
  const int w = threadIdx.x >> 5, f0 = P.goff[P.cg[blockIdx.x]], len = P.goff[P.cg[blockIdx.x + 1]] - f0;
  return make_int2(f0 + (int)((long long)len * w / kWdWarps), f0 + (int)((long long)len * (w + 1) / kWdWarps));
}

// sums over the grid of the threads' values in sh.tot and the largest of their
// exponents in sh.emax, also a barrier (what was written before it, vectors'
// digits too, is seen after it); false after a timeout.  epoch: calls so far
template <int NV>
__device__ __noinline__ bool wide_sums(const WideArgs& P, WideShared& sh, double v0, double v1, double v2, int e0, unsigned epoch) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
  constexpr int kUpCta = fx_up(kWdWarps), kN = kWdMaxGrid / 32, kUpGrid = fx_up(kN);
  sh.vals[0][threadIdx.x] = v0;
  if (NV > 1) sh.vals[1][threadIdx.x] = v1;
  if (NV > 2) sh.vals[2][threadIdx.x] = v2;
  e0 = __reduce_max_sync(0xffffffffu, e0);
  if (lane == 0) sh.ew[w] = e0;
  __syncthreads();
  if (w < NV) {
    double* part = P.part + (size_t)(3 * (epoch & 1) + w) * G;
    int e = 0;
    long long x = 0;
#pragma unroll
    for (int i = 0; i < kWdWarps; i++) e = max(e, fx_biased_exp(sh.vals[w][lane + 32 * i]));
    e = __reduce_max_sync(0xffffffffu, e);
#pragma unroll 4
    for (int i = 0; i < kWdWarps; i++) x += fx_align<kUpCta>(sh.vals[w][lane + 32 * i], e);
    const double t = fx_warp_total<kUpCta>(x, e);
    if (lane == 0) {
      unsigned* ctr = P.ctr + w * kWdCtr;
      __stcg(part + blockIdx.x, t);
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      wide_poll(P, sh, ctr, ++sh.calls[w]);
    }
    __syncwarp();
    double in[kN];
    e = 0;
    x = 0;
#pragma unroll
    for (int q = 0; q < kN; q++) in[q] = lane + 32 * q < G ? __ldcg(part + lane + 32 * q) : 0.0;
#pragma unroll
    for (int q = 0; q < kN; q++) e = max(e, fx_biased_exp(in[q]));
    e = __reduce_max_sync(0xffffffffu, e);
#pragma unroll
    for (int q = 0; q < kN; q++) x += fx_align<kUpGrid>(in[q], e);
    const double s = fx_warp_total<kUpGrid>(x, e);
    if (lane == 0) sh.tot[w] = s;
  } else if (w == 3) {
    int* part = P.epart + (epoch & 1) * G;
    int e = __reduce_max_sync(0xffffffffu, lane < kWdWarps ? sh.ew[lane] : 0);
    if (lane == 0) {
      unsigned* ctr = P.ctr + 3 * kWdCtr;
      __stcg(part + blockIdx.x, e);
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      wide_poll(P, sh, ctr, epoch);
    }
    __syncwarp();
    e = 0;
#pragma unroll
    for (int q = 0; q < kN; q++) e = max(e, lane + 32 * q < G ? __ldcg(part + lane + 32 * q) : 0);
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) sh.emax = e;
  }
  __syncthreads();
  return !sh.fail;
}

// one row of A v in FP64 (v by places): products with x, vectors and rows without a scale
__device__ __noinline__ double wide_row64(const WideArgs& P, int g, int t, int r) {
  const int row = P.perm[kWdRows * g + t];
  if (row < 0) return 0.0;
  const int kb = P.rp[row], n = P.rp[row + 1] - kb;
  double y0 = 0.0, y1 = 0.0, y2 = 0.0;
#pragma unroll 6
  for (int j = 0; j < n; j++) {
    const double* a = P.A + 9 * (size_t)(kb + j) + 3 * r;
    const double* v = P.zg + 3 * (size_t)P.slot[P.col[kb + j]];
    y0 = fma(a[0], __ldcg(v), y0);
    y1 = fma(a[1], __ldcg(v + 1), y1);
    y2 = fma(a[2], __ldcg(v + 2), y2);
  }
  return (y0 + y1) + y2;
}

enum { kWdIterate, kWdStart, kWdEnd };

// A v on this CTA's rows, v as digits at the scale E (fx) or in zg; then, an
// entry a lane:
//   kWdIterate  q = y + beta q, x += alpha p, p = z + beta p; returns the sum of p.q
//   kWdStart    r = r - y
//   kWdEnd      returns the sum of (b - y)^2
__device__ __noinline__ double wide_product(const WideArgs& P, WideShared& sh, double* dsm, int mode, double alpha, double beta,
                                            bool fx, int E) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = min(lane / 3, kWdRows - 1), rsub = lane % 3;
  const int c0 = sh.c0, c1 = sh.c1, n = kWdLanes * P.most;
  double *R = dsm, *Q = R + n;
  unsigned char* ring = reinterpret_cast<unsigned char*>(Q + n) + (size_t)w * P.stages * kWdRec;
  const int l30 = min(lane, kWdLanes - 1), l0 = min(lane - rsub, kWdLanes - 3);
  double sum = 0.0;
  // the vectors of an entry that memory holds, fetched as its group begins
  double xv = 0.0, pv = 0.0, zv = 0.0;
  auto fetch = [&](int g) {
    if (mode != kWdIterate || lane >= kWdLanes) return;
    const size_t i = kWdLanes * (size_t)g + lane;
    xv = P.xg[i];
    pv = P.pg[i];
    zv = P.zv[i];
  };
  auto put = [&](int g, double y) {
    if (lane >= kWdLanes) return;
    const int i = kWdLanes * (g - c0) + lane;
    if (mode == kWdIterate) {
      const size_t at = kWdLanes * (size_t)g + lane;
      const double q = fma(beta, Q[i], y), p = fma(beta, pv, zv);
      P.xg[at] = fma(alpha, pv, xv);
      Q[i] = q;
      P.pg[at] = p;
      sum = fma(p, q, sum);
    } else if (mode == kWdStart) {
      R[i] -= y;
    } else {
      const int row = P.perm[kWdRows * g + t];
      const double d = row >= 0 ? P.b[3 * (size_t)row + rsub] - y : 0.0;
      sum = fma(d, d, sum);
    }
  };
  if (!fx) {
#pragma unroll 1
    for (int g = c0 + w; g < c1; g += kWdWarps) {
      const double y = wide_row64(P, g, t, rsub);
      fetch(g);
      put(g, y);
    }
    return sum;
  }
  // this warp's share of the CTA's records streams through its ring: the first
  // of them are on their way since the last product, and a record's columns are
  // read and what they gather is asked for one record ahead
  const int S = P.stages, a = sh.from[w], N = sh.count[w], keep = (int)((long long)N * P.keep >> 10);
  int g = sh.group[w], ge = sh.end[w];
  bool from_start = !sh.inside[w], ok = true;
  FxAcc tail;
  int tail_g = -1;
  const char* zd = reinterpret_cast<const char*>(P.zd + rsub);
  int st = sh.stage[w], ahead = st;
  unsigned par = sh.parity[w], ahead_par = par;
  const unsigned char* next = ring + st * kWdRec;
  auto gather = [&](int2 (&x)[kWdSteps]) {   // of the stage `ahead`
    ok = wide_full(&sh.full[w][ahead], ahead_par) && ok;
    const int4 c = reinterpret_cast<const int4*>(next + 16 * 6 * kWdLanes)[t];
    x[0] = *reinterpret_cast<const int2*>(zd + (unsigned)c.x);
    x[1] = *reinterpret_cast<const int2*>(zd + (unsigned)c.y);
    x[2] = *reinterpret_cast<const int2*>(zd + (unsigned)c.z);
    x[3] = *reinterpret_cast<const int2*>(zd + (unsigned)c.w);
    next += kWdRec;
    if (++ahead == S) {
      ahead = 0;
      ahead_par ^= 1;
      next = ring;
    }
  };
  int2 xa[kWdSteps], xb[kWdSteps];
#pragma unroll
  for (int q = 0; q < kWdSteps; q++) xa[q] = xb[q] = make_int2(0, 0);
  if (N > 0) gather(xa);
  FxAcc acc[3];
  int ea = P.ea[kWdLanes * g + l30];
  fetch(g);
#pragma unroll 1
  for (int i = 0; i < N; i++) {
    if (i + 1 < N) gather(xb);
    const int4* v = reinterpret_cast<const int4*>(ring + st * kWdRec) + l30;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const int4 m = v[(3 * h + r) * kWdLanes];
        acc[r].add(make_int2(m.x, m.y), xa[2 * h]);
        acc[r].add(make_int2(m.z, m.w), xa[2 * h + 1]);
      }
    __syncwarp();
    if (lane == 0 && i + S < N) wide_load(P, ring + st * kWdRec, a + i + S, &sh.full[w][st], i + S < keep);
    if (++st == S) {
      st = 0;
      par ^= 1;
    }
#pragma unroll
    for (int q = 0; q < kWdSteps; q++) xa[q] = xb[q];
    const bool ends = a + i + 1 == ge;
    if ((i & 1) || ends || i + 1 == N) {   // FxAcc: at most 12 products between two carries
#pragma unroll
      for (int r = 0; r < 3; r++) acc[r].carry();
    }
    if (!ends && i + 1 < N) continue;
    // a row's three sums lie in its three lanes
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
#pragma unroll
    for (int r = 0; r < 3; r++) acc[r] = FxAcc();
    if (!ends) {                 // the next warp ends this group
      if (lane < kWdLanes) {
        sh.head[w][lane][0] = own.hh;
        sh.head[w][lane][1] = own.mid;
      }
    } else if (!from_start) {    // the warp before began it
      tail = own;
      tail_g = g;
    } else {
      put(g, own.value(ea, E));
    }
    from_start = true;
    if (i + 1 < N) {
      g++;
      ge = P.goff[g + 1];
      ea = P.ea[kWdLanes * g + l30];
      fetch(g);
    }
  }
  // the first records of the next product
  if (lane == 0) {
    sh.stage[w] = st;
    sh.parity[w] = par;
    for (int i = 0, k = st; i < min(S, N); i++) {
      wide_load(P, ring + k * kWdRec, a + i, &sh.full[w][k], true);
      if (++k == S) k = 0;
    }
  }
  if (!ok) {
    atomicExch(P.timeout, 1);
    sh.fail = 1;
  }
  __syncthreads();
  if (tail_g >= 0) {
    tail.hh += sh.head[w - 1][l30][0];
    tail.mid += sh.head[w - 1][l30][1];
    fetch(tail_g);
    put(tail_g, tail.value(P.ea[kWdLanes * tail_g + l30], E));
  }
  return sum;
}

__device__ __forceinline__ void wide_body(const WideArgs& P, WideShared& sh, double* wd_dsm) {
  const int c0 = P.cg[blockIdx.x], n = kWdLanes * P.most, own = kWdLanes * (P.cg[blockIdx.x + 1] - c0);
  // this CTA's entries, in the order of its places: r and q; x, p and z in memory
  double *R = wd_dsm, *Q = R + n, *X = P.xg + kWdLanes * (size_t)c0, *D = P.pg + kWdLanes * (size_t)c0,
         *Z = P.zv + kWdLanes * (size_t)c0;
  const size_t ne = kWdLanes * (size_t)P.ngroups;
  const double* I = P.inv + kWdLanes * (size_t)c0;
  const int* KX = P.kx + kWdLanes * (size_t)c0;
  auto dof = [&](int i) {
    const int row = P.perm[kWdRows * c0 + i / 3];
    return row >= 0 ? 3 * row + i % 3 : -1;
  };
  const bool any64 = P.ea[kWdLanes * P.ngroups] != 0;   // a row without a scale
  const bool block = P.pkind == OD_PRECOND_BLOCK_JACOBI, diag = P.pkind == OD_PRECOND_JACOBI;
  for (int i = threadIdx.x; i < own; i += kWdThreads) {
    const int d = dof(i);
    const double b = d >= 0 ? P.b[d] : 0.0, x = d >= 0 && !P.x_zero ? P.x[d] : 0.0;
    X[i] = x;
    R[i] = b;
    D[i] = Q[i] = 0.0;
    if (!P.x_zero) __stcg(P.zg + kWdLanes * (size_t)c0 + i, x);
  }
  __syncthreads();
  unsigned es = 0;   // syncs so far
  // z's digits (or z itself) for the next product; its largest exponent e is
  // known to every CTA.  True: as digits
  int E = 0;
  auto publish = [&](int e) {
    E = e - 1022;
    const bool fx = !any64 && e >= kFxExpMin && e <= kFxExpMax;
    for (int i = threadIdx.x; i < own; i += kWdThreads) {
      if (fx) P.zd[kWdLanes * (size_t)c0 + i] = fx_digits(Z[i], E - KX[i]);
      else __stcg(P.zg + kWdLanes * (size_t)c0 + i, Z[i]);
    }
    return fx;
  };
  // z = M^-1 r, r.z and r.r of this thread's entries; digits: z's at the scale E
  // too (not at the start, which has no scale yet).  A sync lies between the last
  // product, whose gathers read what P.zd holds, and this
  double rz = 0.0, rr = 0.0;
  int ez = 0;
  auto precondition = [&](bool digits) {
    rz = rr = 0.0;
    ez = 0;
#pragma unroll 3
    for (int i = threadIdx.x; i < own; i += kWdThreads) {
      const int k = KX[i];
      const double r = R[i];
      double z = r;
      if (block) {
        const int b0 = i - i % 3;
        z = I[i] * R[b0] + I[ne + i] * R[b0 + 1] + I[2 * ne + i] * R[b0 + 2];
      } else if (diag) {
        z = I[i] * r;
      }
      Z[i] = z;
      if (digits) P.zd[kWdLanes * (size_t)c0 + i] = fx_digits(z, E - k);
      ez = max(ez, fx_biased_exp(z, k));
      rz = fma(r, z, rz);
      rr = fma(r, r, rr);
    }
  };

  const bool timer = P.prof && blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long t_prev = 0;
  auto stamp = [&](int k) {
    if (!timer) return;
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (k >= 0) P.prof[k] += now - t_prev;
    t_prev = now;
  };

  // ---- r = b - A x (products with x in FP64), z = M^-1 r
  if (!P.x_zero) {
    if (!wide_sums<1>(P, sh, 0.0, 0.0, 0.0, 0, ++es)) return;
    wide_product(P, sh, wd_dsm, kWdStart, 0.0, 0.0, false, 0);
    __syncthreads();
  }
  double bb = 0.0;
  for (int i = threadIdx.x; i < own; i += kWdThreads) {
    const int d = dof(i);
    const double b = d >= 0 ? P.b[d] : 0.0;
    bb = fma(b, b, bb);
  }
  precondition(false);
  if (!wide_sums<3>(P, sh, rz, rr, bb, ez, ++es)) return;
  rz = sh.tot[0];
  rr = sh.tot[1];
  bb = sh.tot[2];
  const double eps = bb * P.tol * P.tol;
  double rz_old = rz, rr_now = rr, alpha = 0.0, beta = 0.0;
  bool ready = false;   // z's digits are those of the product to come
  int it = 0, status = isfinite(rr) ? OD_OK : OD_ERR_NAN;
#pragma unroll 1
  while (status == OD_OK && it < P.max_iter && rr_now > eps) {
    stamp(-1);
    // z's scale was set from the last z; one that does not fit is done again
    const int e = sh.emax;
    bool fx = true;
    if (!ready || any64 || e < kFxExpMin || e > kFxExpMax || e - 1022 > E || E - (e - 1022) > kFxSlack) {
      fx = publish(e);
      if (!wide_sums<1>(P, sh, 0.0, 0.0, 0.0, e, ++es)) return;
    }
    const double pq = wide_product(P, sh, wd_dsm, kWdIterate, alpha, beta, fx, E);
    stamp(0);
    if (!wide_sums<1>(P, sh, pq, 0.0, 0.0, 0, ++es)) return;
    stamp(1);
    alpha = rz_old / sh.tot[0];
    for (int i = threadIdx.x; i < own; i += kWdThreads) R[i] = fma(-alpha, Q[i], R[i]);
    __syncthreads();
    E = e - 1021;
    ready = true;
    precondition(true);
    stamp(2);
    if (!wide_sums<2>(P, sh, rz, rr, 0.0, ez, ++es)) return;
    stamp(3);
    beta = sh.tot[0] / rz_old;
    rz_old = sh.tot[0];
    rr_now = sh.tot[1];
    it++;
    if (timer) P.prof[6] += 1;
    if (!isfinite(rr_now) || !isfinite(beta)) status = OD_ERR_NAN;
  }

  // ---- the last x += alpha p, and the true residual ||b - A x||^2, in FP64
  for (int i = threadIdx.x; i < own; i += kWdThreads) {
    const int d = dof(i);
    const double x = fma(alpha, D[i], X[i]);
    X[i] = x;
    if (d >= 0) P.x[d] = x;
    __stcg(P.zg + kWdLanes * (size_t)c0 + i, x);
  }
  if (!wide_sums<1>(P, sh, 0.0, 0.0, 0.0, 0, ++es)) return;
  const double d2 = wide_product(P, sh, wd_dsm, kWdEnd, 0.0, 0.0, false, 0);
  if (!wide_sums<1>(P, sh, d2, 0.0, 0.0, 0, ++es)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    SolveScalars* sc = P.sc;
    sc->rz[0] = sc->rz[1] = rz_old;
    sc->rr = rr_now;
    sc->bb = bb;
    sc->eps = eps;
    sc->iter = it;
    sc->max_iter = P.max_iter;
    sc->status = status;
    sc->tr_num = sh.tot[0];
    sc->tr_den = bb;
    sc->done = 1;
  }
}

__global__ void __launch_bounds__(kWdThreads, 1) wide_pcg_kernel(const __grid_constant__ WideArgs P) {
  extern __shared__ __align__(16) double wd_dsm[];
  __shared__ WideShared sh;
  const int w = threadIdx.x >> 5;
  if (threadIdx.x == 0) sh.fail = 0;
  if (threadIdx.x < 3) sh.calls[threadIdx.x] = 0;
  // every warp's share, and its ring with the first records of it
  const int c0 = P.cg[blockIdx.x], c1 = P.cg[blockIdx.x + 1];
  const int2 share = wide_share(P);
  const int held = min(P.stages, share.y - share.x);
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < P.stages; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(wd_smem(&sh.full[w][k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sh.stage[w] = sh.parity[w] = 0;
    unsigned char* ring = reinterpret_cast<unsigned char*>(wd_dsm + 2 * kWdLanes * P.most) + (size_t)w * P.stages * kWdRec;
    for (int k = 0; k < held; k++) wide_load(P, ring + k * kWdRec, share.x + k, &sh.full[w][k], true);
    int g = c0;
    for (int step = 1 << 20; step; step >>= 1)   // the last group that starts at or before the share
      if (g + step < c1 && P.goff[g + step] <= share.x) g += step;
    sh.from[w] = share.x;
    sh.count[w] = share.y - share.x;
    sh.group[w] = g;
    sh.end[w] = P.goff[g + 1];
    sh.inside[w] = P.goff[g] < share.x;
    sh.c0 = c0;
    sh.c1 = c1;
  }
  __syncthreads();
  wide_body(P, sh, wd_dsm);
  // no CTA leaves with copies on their way
  int k = sh.stage[w];
  unsigned par = sh.parity[w];
  for (int i = 0; i < held; i++) {
    wide_full(&sh.full[w][k], par);
    if (++k == P.stages) {
      k = 0;
      par ^= 1;
    }
  }
}

// ------------------------------------------------------------------- host
void wide_free(WidePlan* W) {
  if (!W) return;
  cudaFree(W->ints);
  cudaFree(W->rec);
  cudaFree(W->ea);
  cudaFree(W->kx);
  cudaFree(W->zd);
  cudaFree(W->zg);
  cudaFree(W->xg);
  cudaFree(W->pg);
  cudaFree(W->zv);
  cudaFree(W->inv);
  cudaFree(W->ctr);
  delete W;
}

// *out stays null when the launch does not take the system: vectors that do
// not fit the CTAs' shared memory, or too few steps for a share of them to
// hold a whole group.
od_status wide_build(Scene* s, WidePlan** out) {
  *out = nullptr;
  const int nb = s->bsr.nb, sms = s->ctx->num_sms;
  const std::vector<int>& rp = s->hbsr_rp;
  if (s->pcg.coop_grid <= 0 || sms <= 0 || sms > kWdMaxGrid || nb <= 0 || (int)rp.size() != nb + 1) return OD_OK;
  auto records_of = [&](int row) { return (rp[row + 1] - rp[row] + kWdSteps - 1) / kWdSteps; };
  long long all = 0;
  int longest = 1;
  for (int r = 0; r < nb; r++) {
    all += records_of(r);
    longest = std::max(longest, records_of(r));
  }
  if (longest > 1 << 12 || all > 0x7fffffff) return OD_OK;
  // CTAs: contiguous block rows of even lengths' sums; within one, by length
  const int G = (int)std::min<long long>(sms, all / kWdRows / ((long long)kWdWarps * longest + longest));
  if (G < 1) return OD_OK;
  WidePlan W;
  W.grid = G;
  std::vector<int> cg(1, 0), goff(1, 0), perm, slot(nb);
  long long seen = 0;
  int row = 0;
  for (int c = 0; c < G; c++) {
    std::vector<int> rows;
    const long long upto = all * (c + 1) / G;
    while (row < nb && (seen < upto || c + 1 == G)) {
      seen += records_of(row);
      rows.push_back(row++);
    }
    std::stable_sort(rows.begin(), rows.end(), [&](int a, int b) { return records_of(a) > records_of(b); });
    for (size_t k = 0; k < rows.size(); k += kWdRows) {
      goff.push_back(goff.back() + records_of(rows[k]));
      for (size_t t = k; t < k + kWdRows; t++) {
        if (t < rows.size()) slot[rows[t]] = (int)perm.size();
        perm.push_back(t < rows.size() ? rows[t] : -1);
      }
    }
    const int ng = (int)perm.size() / kWdRows, share = (goff.back() - goff[cg.back()]) / kWdWarps;
    if (share < longest) return OD_OK;   // a group would span three warps
    W.most = std::max(W.most, ng - cg.back());
    cg.push_back(ng);
  }
  W.ngroups = (int)perm.size() / kWdRows;
  W.records = goff.back();
  if (24LL * kWdRows * W.ngroups > 0x7fffffffLL) return OD_OK;   // columns are byte offsets
  int dev_max = 0;
  cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->ctx->device);
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, wide_pcg_kernel) != cudaSuccess) return OD_OK;
  const size_t cap = (size_t)dev_max - 1024 - fa.sharedSizeBytes, vec = sizeof(double) * kWdLanes * (size_t)W.most;
  const size_t stage = (size_t)kWdWarps * kWdRec;
  if (2 * vec + kWdStagesMin * stage > cap) return OD_OK;
  W.stages = (int)std::min<size_t>(kWdStagesMax, (cap - 2 * vec) / stage);
  W.smem = 2 * vec + W.stages * stage;
  int n = 0;
  const bool ok = cudaFuncSetAttribute(wide_pcg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) == cudaSuccess &&
                  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wide_pcg_kernel, kWdThreads, W.smem) == cudaSuccess && n >= 1;
  cudaGetLastError();   // a refused attribute is not an error of the scene
  if (!ok) return OD_OK;
  std::vector<int> ints;
  const std::vector<int>* arrays[] = {&cg, &goff, &perm, &slot};
  const int** dst[] = {&W.cg, &W.goff, &W.perm, &W.slot};
  size_t offs[4];
  for (int k = 0; k < 4; k++) {
    offs[k] = ints.size();
    ints.insert(ints.end(), arrays[k]->begin(), arrays[k]->end());
  }
  const size_t b_rec = (size_t)kWdRec * W.records, b_inv = 3 * sizeof(double) * kWdLanes * (size_t)W.ngroups,
               b_ea = sizeof(int) * (kWdLanes * (size_t)W.ngroups + 1), b_vec = sizeof(double) * kWdLanes * (size_t)W.ngroups,
               b_ctr = sizeof(unsigned) * 4 * kWdCtr + sizeof(double) * 6 * G + sizeof(int) * 2 * G;
  cudaError_t e = plan_malloc(&W.ints, sizeof(int) * ints.size());
  if (e == cudaSuccess) e = plan_malloc(&W.rec, b_rec);
  if (e == cudaSuccess) e = plan_malloc(&W.ea, b_ea);
  if (e == cudaSuccess) e = plan_malloc(&W.kx, b_ea);
  if (e == cudaSuccess) e = plan_malloc(&W.zd, b_vec);
  if (e == cudaSuccess) e = plan_malloc(&W.zg, b_vec);
  if (e == cudaSuccess) e = plan_malloc(&W.xg, b_vec);
  if (e == cudaSuccess) e = plan_malloc(&W.pg, b_vec);
  if (e == cudaSuccess) e = plan_malloc(&W.zv, b_vec);
  if (e == cudaSuccess) e = plan_malloc(&W.inv, b_inv);
  if (e == cudaSuccess) e = plan_malloc(&W.ctr, b_ctr);
  if (e == cudaSuccess) e = cudaMemcpy(W.ints, ints.data(), sizeof(int) * ints.size(), cudaMemcpyHostToDevice);
  WidePlan* made = new WidePlan(W);
  if (e != cudaSuccess) {
    wide_free(made);
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "wide PCG plan");
    cudaGetLastError();   // no room for the digits: the persistent kernel goes without them
    return OD_OK;
  }
  for (int k = 0; k < 4; k++) *dst[k] = W.ints + offs[k];
  *made = W;
  s->device_bytes += (long long)(sizeof(int) * ints.size() + b_rec + b_inv + 2 * b_ea + 5 * b_vec + b_ctr);
  *out = made;
  return OD_OK;
}

od_status wide_solve(Scene* s, WidePlan* W, const double* d_b, double* d_x, int pkind, double tol, int max_iter, bool x_zero,
                     unsigned long long* prof) {
  Pcg& P = s->pcg;
  cudaStream_t st = s->ctx->stream;
  WideArgs a{};
  a.nb = s->bsr.nb;
  a.ngroups = W->ngroups;
  a.most = W->most;
  a.pkind = pkind;
  a.max_iter = max_iter;
  a.stages = W->stages;
  a.keep = (int)std::min<long long>(1024, 1024 * kWdKeep / ((long long)kWdRec * W->records));
  a.x_zero = x_zero;
  a.cg = W->cg;
  a.goff = W->goff;
  a.perm = W->perm;
  a.slot = W->slot;
  a.rp = s->bsr.row_ptr;
  a.col = s->bsr.col;
  a.A = s->A64;
  a.b = d_b;
  a.pinv = P.pinv;
  a.x = d_x;
  a.rec = W->rec;
  a.ea = W->ea;
  a.diag = s->bsr.diag_pos;
  a.kx = W->kx;
  a.zd = W->zd;
  a.zg = W->zg;
  a.xg = W->xg;
  a.pg = W->pg;
  a.zv = W->zv;
  a.inv = W->inv;
  a.tol = tol;
  a.part = (double*)(W->ctr + 4 * kWdCtr);
  a.epart = (int*)(a.part + 6 * W->grid);
  a.ctr = W->ctr;
  a.timeout = &((GridBarrier*)P.gbar)->timeout;
  a.sc = P.sc;
  a.prof = prof;
  OD_CUDA(cudaMemsetAsync(W->ctr, 0, sizeof(unsigned) * 4 * kWdCtr, st));
  OD_CUDA(cudaMemsetAsync(W->ea + kWdLanes * (size_t)W->ngroups, 0, sizeof(int), st));
  OD_KL(s);
  wide_scale_kernel<<<(kWdLanes * W->ngroups + 255) / 256, 256, 0, st>>>(a);
  OD_CUDA(cudaGetLastError());
  OD_KL(s);
  wide_stage_kernel<<<(W->ngroups + 7) / 8, 256, 0, st>>>(a, W->staged ? 0 : 1);
  OD_CUDA(cudaGetLastError());
  W->staged = true;
  void* args[] = {(void*)&a};
  OD_KL(s);
  OD_CUDA(cudaLaunchCooperativeKernel((void*)wide_pcg_kernel, dim3(W->grid), dim3(kWdThreads), args, W->smem, st));
  return OD_OK;
}

}  // namespace od
