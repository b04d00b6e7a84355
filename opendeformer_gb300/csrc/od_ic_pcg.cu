// FP64 PCG with the shifted IC(0) preconditioner in two launches: the
// factorisation with its shift retries, and the whole solve (iterations with
// both triangular solves, the true residual).
//
// The factor is taken in colour order (no two block rows of a colour are
// coupled): a row needs finished rows of earlier colours only, so the
// factorisation and each sweep are one barrier per colour.  In the solve three
// block rows form a warp's task, nine lanes each, one for every entry of the
// row's current block; a task's blocks of A and of L lie in rows of 27 values
// in the lanes' order (strictly lower blocks, and strictly upper ones
// transposed), padded with zeros that multiply a zero, so that a task's loads
// have no conditions, and are issued before the barrier it waits at.  L is kept
// scaled by its diagonal blocks (y_R = L_RR^-1 r_R - sum (L_RR^-1 L_RC) y_C, and
// likewise backward), so that the diagonal blocks' products too come before it.  Task T
// belongs to CTA T mod G, and so do its entries of every vector, in shared
// memory.
//
// What bounds it: an iteration passes 2 nc barriers (nc: 7-8 colours on the
// structured meshes), and between two lie the reads of other rows' values and
// about 10 dependent FP64 operations of 64 cycles.  A barrier inside a cluster
// takes 0.3 us and a read of another CTA's shared memory 0.1 us, a barrier
// over the whole chip 1.4 us and a read of L2 0.3 us.
//
// Newmark steps of two solves with IC(0) at 1e-8, before (the factorisation in
// one launch, then five an iteration, the sweeps' rows waiting on one
// another's values) and now: 96 tets 3.4 -> 0.91 ms, 1,152 5.9 -> 1.27, 12,288
// 6.5 -> 2.28, 34,560 7.3 -> 2.70, 98,304 12.8 -> 3.65, 590k 37 -> 14.0.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "od_internal.h"
#include "od_grid.cuh"
#include "od_fixed.cuh"

namespace od {

constexpr int kIpWarps = 12;                   // warps per CTA
constexpr int kIpThreads = 32 * kIpWarps;
constexpr int kIpRows = 3;                     // block rows per task
constexpr int kIpVals = 9 * kIpRows;           // values of a slot: one block of each row
constexpr int kIpEnts = 3 * kIpRows;           // entries of a task in a vector, columns of a slot
constexpr int kIpMaxGrid = 160;                // CTAs (one per SM)
constexpr int kIpCluster = 16;                 // CTAs of the cluster form
constexpr int kIpPad = 4;                      // a task's slots come in fours
constexpr int kIpPre = 16;                     // slots loaded at once (before the barrier)
static_assert(kIpPre == 16, "two ip_dot8");
constexpr int kIpCtr = 1024;                   // counters lie words apart: they are polled at once
constexpr int kIpShifts = 40;                  // attempts at a shift
constexpr int kIpMaxColours = 255;
constexpr int kIpSmem = 200 * 1024;            // most dynamic shared memory

// Structure and values of a scene's factor (device)
struct IcPcg {
  int nb = 0, nc = 0, nt = 0, nfs = 0, nbs = 0, max_low = 0, max_pairs = 0, max_rounds = 0;
  int grid = 0, own = 0, factor_grid = 0, factor_warps = 0;   // CTAs, tasks of a CTA; of the factorisation
  bool cluster = false;
  size_t smem = 0, factor_smem = 0;
  int* ints = nullptr;       // every index array
  double* vals = nullptr;    // AF, AB, AD, LF, LB, LD, LU, v, p
  unsigned* ctr = nullptr;   // counters, breakdown flags
  unsigned* adr = nullptr;   // cluster form: addresses of fidx, bidx
  const int *tbase, *sysd, *task, *row, *fidx, *bidx, *asrc, *ldst, *fdia, *pa, *pb, *rounds, *rlist;
};

struct IpArgs {
  int nc, nt, nfs, nbs, own, max_low, max_pairs, max_rounds, factor_warps, max_iter;
  const int* tbase;          // first task of every colour
  const int* sysd;           // the system's DOF of every entry, -1: none
  const int4* task;          // first lower slot, first upper slot, their numbers (16 bits each) with and without padding
  const int4* row;           // rows of the tasks: lower blocks (-1: no row), first pair, pairs, place of its first block in LF (in nines)
  const int *fidx, *bidx;    // entry of every column of every slot (cluster form: its CTA << 24 and the entry there)
  unsigned* adr;
  const int* asrc;           // block of A of every nine values of AF, AB, AD in turn, -1: none
  const int* ldst;           // place in LB of every block of LF (in nines)
  const int* fdia;           // place in LD of the column of every block of LF (in nines)
  const int *pa, *pb;        // pairs, by block (R, C) of a row: K common to both rows, as (number in row R, place in LU of row C's block)
  const int2* rounds;        // rows of the tasks: first entry in rlist and their number (three a round)
  const int* rlist;          // a round's blocks: number, first pair << 8, pairs << 22; -1: none
  const double *A, *b;
  double* x;
  double *AF, *AB, *AD, *LF, *LB, *LD, *LU;
  double *v, *p;             // grid form: y and then z; the direction, in the tasks' order
  double tol;
  double* part;              // 2 x 2 x gridDim.x partial sums
  unsigned* ctr;
  int* timeout;
  int* bad;                  // kIpShifts breakdown flags
  SolveScalars* sc;
};

struct IpShared {
  double tot[2];
  double part[2][2][kIpCluster];   // cluster form: every CTA's sums, by round parity
  int fail;
  int tbase[kIpMaxColours + 1];
};

// shared-memory address a in CTA rank of the cluster
__device__ __forceinline__ unsigned ip_cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double ip_ld_cluster(unsigned a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

// One lane's bounded wait for every CTA's epoch-th arrival at a counter
__device__ __forceinline__ void ip_poll(const IpArgs& P, IpShared& sh, const unsigned* ctr, unsigned epoch) {
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

// Barrier over all CTAs in two halves: every thread's writes before its
// arrival are seen after the wait (memory through L2: the readers bypass L1).
template <bool CL>
__device__ __forceinline__ void ip_arrive(unsigned* ctr) {
  if (CL) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  } else {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
  }
}
// epoch: barriers so far; false after a timeout
template <bool CL>
__device__ __forceinline__ bool ip_wait(const IpArgs& P, IpShared& sh, unsigned* ctr, unsigned epoch) {
  if (CL) {
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  if (threadIdx.x == 0) ip_poll(P, sh, ctr, epoch);
  __syncthreads();
  return !sh.fail;
}
template <bool CL>
__device__ __noinline__ bool ip_barrier(const IpArgs& P, IpShared& sh, unsigned* ctr, unsigned epoch) {
  ip_arrive<CL>(ctr);
  return ip_wait<CL>(P, sh, ctr, epoch);
}

// sums over all CTAs of the threads' values v0 and v1 in sh.tot (also a
// barrier); false after a timeout.  epoch: sums so far
template <bool CL>
__device__ __noinline__ bool ip_sums(const IpArgs& P, IpShared& sh, double (*vals)[kIpThreads], double v0, double v1,
                                     unsigned epoch) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
  constexpr int kUpCta = fx_up(kIpWarps), kN = CL ? 1 : kIpMaxGrid / 32, kUpGrid = fx_up(kN);
  double* part = P.part + (size_t)(2 * (epoch & 1) + (w & 1)) * G;
  vals[0][threadIdx.x] = v0;
  vals[1][threadIdx.x] = v1;
  __syncthreads();
  if (w < 2) {
    int e = 0;
    long long x = 0;
#pragma unroll
    for (int i = 0; i < kIpWarps; i++) e = max(e, fx_biased_exp(vals[w][lane + 32 * i]));
    e = __reduce_max_sync(0xffffffffu, e);
#pragma unroll 4
    for (int i = 0; i < kIpWarps; i++) x += fx_align<kUpCta>(vals[w][lane + 32 * i], e);
    const double t = fx_warp_total<kUpCta>(x, e);
    if (CL) {
      if (lane < G)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ip_cluster_addr(
                         (unsigned)__cvta_generic_to_shared(&sh.part[epoch & 1][w][blockIdx.x]), lane)),
                     "d"(t)
                     : "memory");
    } else if (lane == 0) {
      unsigned* ctr = P.ctr + (1 + w) * kIpCtr;
      __stcg(part + blockIdx.x, t);
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      ip_poll(P, sh, ctr, epoch);
    }
  }
  if (CL) {
    ip_arrive<CL>(nullptr);
    ip_wait<CL>(P, sh, nullptr, 0);
  }
  if (w < 2) {
    __syncwarp();
    double in[kN];
    int e = 0;
    long long x = 0;
#pragma unroll
    for (int q = 0; q < kN; q++)
      in[q] = lane + 32 * q < G ? (CL ? sh.part[epoch & 1][w][lane & (kIpCluster - 1)] : __ldcg(part + lane + 32 * q)) : 0.0;
#pragma unroll
    for (int q = 0; q < kN; q++) e = max(e, fx_biased_exp(in[q]));
    e = __reduce_max_sync(0xffffffffu, e);
#pragma unroll
    for (int q = 0; q < kN; q++) x += fx_align<kUpGrid>(in[q], e);
    const double s = fx_warp_total<kUpGrid>(x, e);
    if (lane == 0) sh.tot[w] = s;
  }
  __syncthreads();
  return !sh.fail;
}

// ---------------------------------------------------------- factorisation
//   L_RC = (A_RC - sum_K L_RK L_CK^T) L_CC^-T,  L_RR L_RR^T = (1 + shift) A_RR - sum_K L_RK L_RK^T
// into LU; LD holds L_RR^-1, LF L_RR^-1 L_RC and LB the transposes of
// L_RC L_CC^-1.  A warp per row, on the whole chip whatever the solve's form:
// what bounds it is a row's chain of FP64 operations, so its blocks go three at
// a time (nine lanes each) in rounds of columns of one colour, which do not
// depend on one another.  The row's blocks, the inverse diagonal blocks of
// their columns and the paired blocks of other rows are brought to shared
// memory at once.
__device__ __forceinline__ void ip_factor_row(const IpArgs& P, double* own, int* list, int q, int4 row, double shift, int* bad) {
  const int lane = threadIdx.x & 31, g = min(lane / 9, 2), e = lane % 9, rr = e / 3, cc = e % 3;
  const bool act = lane < 27;
  double* cinv = own + 9 * P.max_low;      // L_CC^-1 of the columns
  double* paired = cinv + 9 * P.max_low;
  int *from = list + P.max_pairs, *rounds = from + P.max_pairs;
  const int m = row.x, np = row.z, f9 = row.w;   // block k at f9 + kIpRows k
  const int2 rd = P.rounds[q];                   // first of its rounds' entries, their number
  __syncwarp();
#pragma unroll 4
  for (int i = lane; i < np; i += 32) {
    list[i] = P.pa[row.y + i];
    from[i] = P.pb[row.y + i];
  }
  for (int i = lane; i < rd.y; i += 32) rounds[i] = P.rlist[rd.x + i];
  if (act) {
#pragma unroll 5
    for (int k = g; k < m; k += 3) {
      own[9 * k + e] = __ldcg(P.AF + 9 * (size_t)(f9 + kIpRows * k) + e);
      cinv[9 * k + e] = __ldcg(P.LD + 9 * (size_t)P.fdia[f9 + kIpRows * k] + e);
    }
  }
  double d = lane < 9 ? __ldcg(P.AD + 9 * (size_t)q + e) : 0.0;
  if (rr == cc) d *= 1.0 + shift;
  double s = d;
  __syncwarp();
  if (act) {
#pragma unroll 8
    for (int i = g; i < np; i += 3) paired[9 * i + e] = __ldcg(P.LU + 9 * (size_t)from[i] + e);
  }
  __syncwarp();
  const int l9 = min(9 * g + 3 * rr, 29);
#pragma unroll 1
  for (int r = 0; r < rd.y; r += 3) {
    // block, its first pair and their number; -1: none
    const int ent = act ? rounds[r + g] : -1, k = ent & 255;
    double v = 0.0;
    if (ent >= 0) {
      v = own[9 * k + e];
      const int p1 = (ent >> 8 & 0x3fff) + (ent >> 22);
#pragma unroll 1
      for (int i = ent >> 8 & 0x3fff; i < p1; i++) {
        const double* a = own + 9 * list[i] + 3 * rr;
        const double* o = paired + 9 * i + 3 * cc;
        v = fma(-a[0], o[0], v);
        v = fma(-a[1], o[1], v);
        v = fma(-a[2], o[2], v);
      }
    }
    __syncwarp();
    const double s0 = __shfl_sync(0xffffffffu, v, l9), s1 = __shfl_sync(0xffffffffu, v, l9 + 1),
                 s2 = __shfl_sync(0xffffffffu, v, l9 + 2);
    if (ent >= 0) {
      const double* l = cinv + 9 * k + 3 * cc;
      v = fma(s2, l[2], fma(s1, l[1], s0 * l[0]));   // L_CC^-1 is zero above its diagonal
      own[9 * k + e] = v;
      __stcg(P.LU + 9 * (size_t)(f9 + kIpRows * k) + e, v);
    }
    __syncwarp();
  }
  if (act) {
#pragma unroll 1
    for (int k = g; k < m; k += 3) {
      const double* a = own + 9 * k;
      s = fma(-a[3 * rr], a[3 * cc], s);
      s = fma(-a[3 * rr + 1], a[3 * cc + 1], s);
      s = fma(-a[3 * rr + 2], a[3 * cc + 2], s);
    }
  }
  __syncwarp();
  s = s + __shfl_down_sync(0xffffffffu, s, 9) + __shfl_down_sync(0xffffffffu, s, 18);
  // the diagonal block's Cholesky factor, inverted (every lane alike)
  auto at = [&](double v, int k) { return __shfl_sync(0xffffffffu, v, k); };
  const double a00 = at(s, 0), a10 = at(s, 3), a20 = at(s, 6), a11 = at(s, 4), a21 = at(s, 7), a22 = at(s, 8);
  const double d0 = at(d, 0), d1 = at(d, 4), d2 = at(d, 8);
  auto pivot = [&](double v, double dg) {
    if (!(v > 1e-12 * dg)) {
      if (lane == 0) *bad = 1;
      v = dg > 0.0 ? dg : 1.0;
    }
    return rsqrt(v);
  };
  const double i0 = pivot(a00, d0);
  const double l10 = a10 * i0, l20 = a20 * i0;
  const double i1 = pivot(fma(-l10, l10, a11), d1);
  const double l21 = fma(-l20, l10, a21) * i1;
  const double i2 = pivot(fma(-l21, l21, fma(-l20, l20, a22)), d2);
  const double m10 = -l10 * i0 * i1, m21 = -l21 * i1 * i2, m20 = -(l20 * i0 + l21 * m10) * i2;
  // row rr of L_RR^-1
  const double n0 = rr == 0 ? i0 : rr == 1 ? m10 : m20, n1 = rr == 0 ? 0.0 : rr == 1 ? i1 : m21, n2 = rr == 2 ? i2 : 0.0;
  if (lane < 9) __stcg(P.LD + 9 * (size_t)q + e, cc == 0 ? n0 : cc == 1 ? n1 : n2);
  if (act) {
#pragma unroll 1
    for (int k = g; k < m; k += 3) {
      const double *a = own + 9 * k, *c = cinv + 9 * k;
      const int to = f9 + kIpRows * k;
      __stcg(P.LF + 9 * (size_t)to + e, fma(n2, a[6 + cc], fma(n1, a[3 + cc], n0 * a[cc])));
      __stcg(P.LB + 9 * (size_t)P.ldst[to] + 3 * cc + rr,
             fma(a[3 * rr + 2], c[6 + cc], fma(a[3 * rr + 1], c[3 + cc], a[3 * rr] * c[cc])));
    }
  }
}

__global__ void __launch_bounds__(kIpThreads, 1) ic_pcg_factor_kernel(const __grid_constant__ IpArgs P) {
  extern __shared__ double ip_dsm[];
  __shared__ IpShared sh;
  const int w = threadIdx.x >> 5, FW = P.factor_warps;
  if (threadIdx.x == 0) sh.fail = 0;
  for (int c = threadIdx.x; c <= P.nc; c += kIpThreads) sh.tbase[c] = P.tbase[c];
  unsigned* ctr = P.ctr + 3 * kIpCtr;
  unsigned eb = 0;
  // A in the tasks' order, zero where a task has no block
  const int na = 9 * kIpRows * (P.nfs + P.nbs + P.nt);
#pragma unroll 4
  for (int i = blockIdx.x * kIpThreads + threadIdx.x; i < na; i += gridDim.x * kIpThreads) {
    const int src = P.asrc[i / 9];
    __stcg(P.AF + i, src >= 0 ? P.A[9 * (size_t)src + i % 9] : 0.0);
  }
  if (!ip_barrier<false>(P, sh, ctr, ++eb)) return;
  const int row_vals = 9 * (2 * P.max_low + P.max_pairs);
  double* own = ip_dsm + (size_t)w * row_vals;
  int* list = reinterpret_cast<int*>(ip_dsm + (size_t)FW * row_vals) + w * (2 * P.max_pairs + P.max_rounds);
  double shift = 0.0;
#pragma unroll 1
  for (int a = 0; a < kIpShifts; a++) {
#pragma unroll 1
    for (int c = 0; c < P.nc; c++) {
      if (w < FW) {
        const int q1 = kIpRows * sh.tbase[c + 1];
#pragma unroll 1
        for (int q = kIpRows * sh.tbase[c] + w * gridDim.x + blockIdx.x; q < q1; q += FW * gridDim.x) {
          const int4 row = P.row[q];
          if (row.x >= 0) ip_factor_row(P, own, list, q, row, shift, P.bad + a);
        }
      }
      if (!ip_barrier<false>(P, sh, ctr, ++eb)) return;
    }
    if (!__ldcg(P.bad + a)) break;
    shift = shift == 0.0 ? 1e-3 : 2.0 * shift;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) P.sc->alpha = shift;
}

// ------------------------------------------------------------------ solve
// acc + the first n <= 8 of the products a[k] b[k], the last one first; n the
// same in a warp.  A jump into the chain: an FP64 instruction holds its unit
// for 64 cycles even when no lane's predicate is set, and predicates are what
// the compiler makes of short branches.
__device__ __forceinline__ double ip_dot8(const double* a, const double* b, int n, double acc) {
  asm volatile(
      "{\n\t"
      "ts: .branchtargets L0, L1, L2, L3, L4, L5, L6, L7, L8;\n\t"
      "brx.idx.uni %1, ts;\n\t"
      "L8: fma.rn.f64 %0, %16, %17, %0;\n\t"
      "L7: fma.rn.f64 %0, %14, %15, %0;\n\t"
      "L6: fma.rn.f64 %0, %12, %13, %0;\n\t"
      "L5: fma.rn.f64 %0, %10, %11, %0;\n\t"
      "L4: fma.rn.f64 %0, %8, %9, %0;\n\t"
      "L3: fma.rn.f64 %0, %6, %7, %0;\n\t"
      "L2: fma.rn.f64 %0, %4, %5, %0;\n\t"
      "L1: fma.rn.f64 %0, %2, %3, %0;\n\t"
      "L0:\n\t"
      "}"
      : "+d"(acc)
      : "r"(n), "d"(a[0]), "d"(b[0]), "d"(a[1]), "d"(b[1]), "d"(a[2]), "d"(b[2]), "d"(a[3]), "d"(b[3]),
        "d"(a[4]), "d"(b[4]), "d"(a[5]), "d"(b[5]), "d"(a[6]), "d"(b[6]), "d"(a[7]), "d"(b[7]));
  return acc;
}

template <bool CL>
__global__ void __launch_bounds__(kIpThreads, 1) ic_pcg_kernel(const __grid_constant__ IpArgs P) {
  // this CTA's entries: y and then z, the direction (each ends with the zero
  // that padding reads), the residual, q, x
  extern __shared__ double ip_dsm[];
  __shared__ double vals[2][kIpThreads];
  __shared__ IpShared sh;
  const int lane = threadIdx.x & 31, l27 = min(lane, kIpVals - 1), t9 = l27 / 9, e = l27 % 9, rr = e / 3, cc = e % 3;
  const int G = gridDim.x, NW = kIpWarps * G, first = (threadIdx.x >> 5) * G + blockIdx.x;   // this warp's tasks
  const int ents = kIpEnts * P.own + 1;
  double *V = ip_dsm, *D = V + ents, *Rv = D + ents, *Q = Rv + ents, *X = Q + ents;
  const unsigned p_off = 8u * (unsigned)ents;   // from V to D, in every CTA
  // entries of this CTA's tasks
  const int n_own = (int)blockIdx.x < P.nt ? kIpEnts * ((P.nt - 1 - (int)blockIdx.x) / G + 1) : 0;
  const int lcol = 3 * t9 + cc, lent = 3 * t9 + rr;
  const bool put = lane < kIpVals && cc == 0;   // the lane that has an entry's sum
  if (*(volatile int*)P.timeout) return;        // the factorisation gave up
  if (threadIdx.x == 0) sh.fail = 0;
  for (int c = threadIdx.x; c <= P.nc; c += kIpThreads) sh.tbase[c] = P.tbase[c];
  unsigned eb = 0, es = 0;   // barriers and sums so far
  unsigned* ctr = P.ctr;

  // an entry of this CTA in the tasks' order; its DOF of the system
  auto place = [&](int i) { return kIpEnts * ((int)blockIdx.x + G * (i / kIpEnts)) + i % kIpEnts; };
  auto set_direction = [&](int i, double v) {
    D[i] = v;
    if (!CL) __stcg(P.p + place(i), v);
  };
  for (int i = threadIdx.x; i < ents; i += kIpThreads) {
    const int dof = i < n_own ? P.sysd[place(i)] : -1;
    X[i] = dof >= 0 ? P.x[dof] : 0.0;
    V[i] = D[i] = Rv[i] = 0.0;
    if (i < n_own) set_direction(i, X[i]);
  }
  // cluster form: the addresses of what this warp's tasks read
  if (CL) {
    const unsigned v0 = (unsigned)__cvta_generic_to_shared(V);
    for (int T = first; T < P.nt; T += NW) {
      const int4 tk = P.task[T];
      auto convert = [&](const int* idx, unsigned* adr, int n) {
#pragma unroll 4
        for (int i = lane; i < kIpEnts * n; i += 32)
          adr[i] = ip_cluster_addr(v0, idx[i] >> 24) + 8u * (unsigned)(idx[i] & 0xffffff);
      };
      convert(P.fidx + kIpEnts * tk.x, P.adr + kIpEnts * tk.x, tk.z & 0xffff);
      convert(P.bidx + kIpEnts * tk.y, P.adr + kIpEnts * (P.nfs + tk.y), tk.z >> 16);
    }
  }
  const int* fsrc = CL ? (const int*)P.adr : P.fidx;
  const int* bsrc = CL ? (const int*)P.adr + kIpEnts * P.nfs : P.bidx;
  auto value = [&](int a, bool direction) {
    if (CL) return ip_ld_cluster((unsigned)a + (direction ? p_off : 0u));
    return __ldcg((direction ? P.p : P.v) + a);
  };
  if (!ip_barrier<CL>(P, sh, ctr, ++eb)) return;

  // a row's three partial sums, right in the lane that puts it
  auto row_sum = [&](double v) { return v + __shfl_down_sync(0xffffffffu, v, 1) + __shfl_down_sync(0xffffffffu, v, 2); };
  // f(entry of this CTA, A p there) over this warp's tasks, in the lanes that put
  auto product = [&](auto f) {
#pragma unroll 1
    for (int T = first, at = kIpEnts * (first / G); T < P.nt; T += NW, at += kIpEnts * kIpWarps) {
      const int4 tk = P.task[T];
      double acc = __ldcg(P.AD + kIpVals * (size_t)T + l27) * D[at + lcol];
      auto blocks = [&](const int* a, const double* m, int n) {
#pragma unroll 2
        for (int k = 0; k < n; k += kIpPad) {
          int c[kIpPad];
          double v[kIpPad];
#pragma unroll
          for (int u = 0; u < kIpPad; u++) c[u] = a[kIpEnts * (k + u)];
#pragma unroll
          for (int u = 0; u < kIpPad; u++) v[u] = value(c[u], true);
#pragma unroll
          for (int u = 0; u < kIpPad; u++) acc = fma(__ldcg(m + kIpVals * (k + u)), v[u], acc);
        }
      };
      blocks(fsrc + kIpEnts * tk.x + lcol, P.AF + kIpVals * (size_t)tk.x + l27, tk.z & 0xffff);
      blocks(bsrc + kIpEnts * tk.y + lcol, P.AB + kIpVals * (size_t)tk.y + l27, tk.z >> 16);
      const double y = row_sum(acc);
      if (put) f(at + lent, y);
      __syncwarp();
    }
  };

  // y = L^-1 r, z = L^-T y.  y and z share one vector: a row's y is read by its
  // own warp alone once z is written.  False after a timeout.
  double s0 = 0.0, s1 = 0.0;
  auto sweeps = [&]() -> bool {
    int col[kIpPre], w = 0, n = 0;   // slots with and without padding
    double l[kIpPre], rhs = 0.0;
    const int* cp = nullptr;
    const double* lp = nullptr;
    int T = first, at = kIpEnts * (first / G);
    auto fetch = [&](bool back) {
      const int4 tk = P.task[T];
      w = back ? tk.z >> 16 : tk.z & 0xffff;
      n = back ? tk.w >> 16 : tk.w & 0xffff;
      cp = (back ? bsrc + kIpEnts * tk.y : fsrc + kIpEnts * tk.x) + lcol;
      lp = (back ? P.LB + kIpVals * (size_t)tk.y : P.LF + kIpVals * (size_t)tk.x) + l27;
      const double ld = __ldcg(P.LD + kIpVals * (size_t)T + (back ? 9 * t9 + 3 * cc + rr : l27));
#pragma unroll
      for (int g = 0; g < kIpPre; g += kIpPad)
        if (g < w) {
#pragma unroll
          for (int u = g; u < g + kIpPad; u++) {
            col[u] = cp[kIpEnts * u];
            l[u] = __ldcg(lp + kIpVals * u);
          }
        }
      rhs = row_sum(ld * (back ? V : Rv)[at + lcol]);
    };
    if (T < P.nt) fetch(false);
    int s = 0;
#pragma unroll 1
    while (s < 2 * P.nc) {
      const bool back = s >= P.nc;
      const int c = back ? 2 * P.nc - 1 - s : s;
      const int lo = sh.tbase[c], hi = sh.tbase[c + 1];
      bool next = false;   // a task to fetch
      if (T >= lo && T < hi) {
        double v[kIpPre], acc = 0.0;
#pragma unroll
        for (int g = 0; g < kIpPre; g += kIpPad)
          if (g < w) {
#pragma unroll
            for (int u = g; u < g + kIpPad; u++) v[u] = value(col[u], false);
          }
        acc = ip_dot8(l + 8, v + 8, min(max(n - 8, 0), 8), acc);
        acc = ip_dot8(l, v, min(n, 8), acc);
#pragma unroll 4
        for (int u = kIpPre; u < n; u++) acc = fma(__ldcg(lp + kIpVals * u), value(cp[kIpEnts * u], false), acc);
        const double out = rhs - row_sum(acc);
        if (put) {
          V[at + lent] = out;
          if (!CL) __stcg(P.v + kIpEnts * (size_t)T + lent, out);
        }
        __syncwarp();
        T += back ? -NW : NW;
        at += back ? -kIpEnts * kIpWarps : kIpEnts * kIpWarps;
        next = true;
      }
      // no barrier between the forward and the backward sweep: the last
      // colour's rows wait for their own
      const bool done = T < lo || T >= hi, turn = done && s == P.nc - 1, sync = done && !turn && s + 1 < 2 * P.nc;
      if (sync) ip_arrive<CL>(ctr);
      if (turn) {
        T -= NW;
        at -= kIpEnts * kIpWarps;
      }
      if ((next || turn) && T >= 0 && T < P.nt) fetch(back || turn);
      if (sync && !ip_wait<CL>(P, sh, ctr, ++eb)) return false;
      if (done) s++;
    }
    __syncthreads();
    return true;
  };
  // r.z over this CTA's entries
  auto dot_rz = [&]() {
    double t = 0.0;
    for (int i = threadIdx.x; i < n_own; i += kIpThreads) t = fma(Rv[i], V[i], t);
    return t;
  };
  auto rhs_of = [&](int i) {
    const int dof = P.sysd[place(i)];
    return dof >= 0 ? P.b[dof] : 0.0;
  };

  // ---- r = b - A x, b.b, z = M^-1 r
  product([&](int i, double y) {
    const double b = rhs_of(i), r = b - y;
    Rv[i] = r;
    s0 = fma(b, b, s0);
    s1 = fma(r, r, s1);
  });
  if (!ip_sums<CL>(P, sh, vals, s0, s1, ++es)) return;
  const double bb = sh.tot[0], eps = bb * P.tol * P.tol;
  double rrn = sh.tot[1], rz = 0.0, beta = 0.0;
  int it = 0, status = isfinite(rrn) ? OD_OK : OD_ERR_NAN;
  if (!sweeps()) return;
  if (!ip_sums<CL>(P, sh, vals, dot_rz(), 0.0, ++es)) return;
  rz = sh.tot[0];
#pragma unroll 1
  while (status == OD_OK && it < P.max_iter && rrn > eps) {
    // p = z + beta p, q = A p, p.q
    for (int i = threadIdx.x; i < n_own; i += kIpThreads) set_direction(i, it ? fma(beta, D[i], V[i]) : V[i]);
    if (!ip_barrier<CL>(P, sh, ctr, ++eb)) return;
    s0 = 0.0;
    product([&](int i, double y) {
      Q[i] = y;
      s0 = fma(D[i], y, s0);
    });
    if (!ip_sums<CL>(P, sh, vals, s0, 0.0, ++es)) return;
    // x += alpha p, r -= alpha q, z = M^-1 r, r.z and r.r
    const double alpha = rz / sh.tot[0];
    s1 = 0.0;
    for (int i = threadIdx.x; i < n_own; i += kIpThreads) {
      const double r = fma(-alpha, Q[i], Rv[i]);
      Rv[i] = r;
      X[i] = fma(alpha, D[i], X[i]);
      s1 = fma(r, r, s1);
    }
    __syncthreads();
    if (!sweeps()) return;
    if (!ip_sums<CL>(P, sh, vals, dot_rz(), s1, ++es)) return;
    beta = sh.tot[0] / rz;
    rz = sh.tot[0];
    rrn = sh.tot[1];
    it++;
    if (!isfinite(rrn) || !isfinite(beta)) status = OD_ERR_NAN;
  }

  // ---- x, and its true residual ||b - A x||^2
  for (int i = threadIdx.x; i < n_own; i += kIpThreads) {
    const int dof = P.sysd[place(i)];
    if (dof >= 0) P.x[dof] = X[i];
    set_direction(i, X[i]);
  }
  if (!ip_barrier<CL>(P, sh, ctr, ++eb)) return;
  s0 = 0.0;
  product([&](int i, double y) {
    const double d = rhs_of(i) - y;
    s0 = fma(d, d, s0);
  });
  if (!ip_sums<CL>(P, sh, vals, s0, 0.0, ++es)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    SolveScalars* sc = P.sc;
    sc->rz[0] = sc->rz[1] = rz;
    sc->rr = rrn;
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

// ------------------------------------------------------------------- host
void ic_pcg_free(IcPcg* I) {
  if (!I) return;
  cudaFree(I->ints);
  cudaFree(I->vals);
  cudaFree(I->ctr);
  cudaFree(I->adr);
  delete I;
}

static const void* ic_pcg_fn(bool cluster) {
  return cluster ? (const void*)ic_pcg_kernel<true> : (const void*)ic_pcg_kernel<false>;
}

static void ic_pcg_config(int grid, size_t smem, bool cluster, cudaStream_t st, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(kIpThreads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  *at = cudaLaunchAttribute{};
  if (cluster) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = grid;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
  } else {
    at->id = cudaLaunchAttributeCooperative;
    at->val.cooperative = 1;
  }
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// The factor's structure from the colour order (order: the system's block row
// of every factor row; cstart: first factor row of every colour).  *out stays
// null when the launches do not take the system: too many colours, rows too
// long, vectors or a row's blocks and pairs that do not fit shared memory, no
// device memory for it.
od_status ic_pcg_build(Scene* s, const std::vector<int>& rp, const std::vector<int>& col, const std::vector<int>& order,
                       const std::vector<int>& cstart, IcPcg** out) {
  *out = nullptr;
  const int nb = s->bsr.nb, nc = (int)cstart.size() - 1, sms = s->ctx->num_sms;
  if (nb <= 0 || nb >= 1 << 28 || nc <= 0 || nc > kIpMaxColours || s->pcg.coop_grid <= 0 || sms > kIpMaxGrid) return OD_OK;
  std::vector<int> inv(nb), rfp(nb + 1, 0), rbp(nb + 1, 0), dsrc(nb, -1);
  for (int R = 0; R < nb; R++) inv[order[R]] = R;
  std::vector<std::pair<int, int>> low, up, blk;   // rows' blocks left and right of the diagonal: (factor column, block of A)
  for (int R = 0; R < nb; R++) {
    blk.clear();
    for (int k = rp[order[R]]; k < rp[order[R] + 1]; k++) blk.push_back({inv[col[k]], k});
    std::sort(blk.begin(), blk.end());
    for (const auto& b : blk) {
      if (b.first < R) low.push_back(b);
      else if (b.first > R) up.push_back(b);
      else dsrc[R] = b.second;
    }
    if (dsrc[R] < 0) return OD_OK;   // no diagonal block: never from a scene's pattern
    rfp[R + 1] = (int)low.size();
    rbp[R + 1] = (int)up.size();
  }
  // tasks: slots of kIpRows rows, as many as the longest of them has blocks,
  // in fours
  std::vector<int> tbase(nc + 1, 0), task, place(nb);   // place: a row among the tasks' rows
  std::vector<int> fcol, bcol, asrc_f, asrc_b, asrc;    // columns (rows of the factor), -1: padding; blocks of A
  std::vector<int> fat(low.size()), bat(up.size());     // blocks' places (in nines)
  int nt = 0;
  for (int c = 0; c < nc; c++) {
    for (int R0 = cstart[c]; R0 < cstart[c + 1]; R0 += kIpRows, nt++) {
      const int rows = std::min(kIpRows, cstart[c + 1] - R0);
      int w[2] = {0, 0};
      for (int i = 0; i < rows; i++) {
        place[R0 + i] = kIpRows * nt + i;
        w[0] = std::max(w[0], rfp[R0 + i + 1] - rfp[R0 + i]);
        w[1] = std::max(w[1], rbp[R0 + i + 1] - rbp[R0 + i]);
      }
      if (w[0] > 255 || w[1] > 0x7ff0) return OD_OK;
      auto lay = [&](int width, const std::vector<int>& ptr, const std::vector<std::pair<int, int>>& blocks,
                     std::vector<int>& at, std::vector<int>& cols, std::vector<int>& src) {
        const int first = (int)cols.size() / kIpRows;
        for (int k = 0; k < width; k++)
          for (int i = 0; i < kIpRows; i++) {
            const int q = i < rows ? ptr[R0 + i] + k : 0;
            const bool on = i < rows && q < ptr[R0 + i + 1];
            if (on) at[q] = (int)cols.size();
            cols.push_back(on ? blocks[q].first : -1);
            src.push_back(on ? blocks[q].second : -1);
          }
        return first;
      };
      const int n[2] = {w[0], w[1]};
      for (int& x : w) x = (x + kIpPad - 1) / kIpPad * kIpPad;
      const int f0 = lay(w[0], rfp, low, fat, fcol, asrc_f), b0 = lay(w[1], rbp, up, bat, bcol, asrc_b);
      task.insert(task.end(), {f0, b0, w[0] | w[1] << 16, n[0] | n[1] << 16});
      if (9LL * ((long long)fcol.size() + (long long)bcol.size() + kIpRows * (nt + 1LL)) > 0x70000000LL) return OD_OK;
    }
    tbase[c + 1] = nt;
  }
  const int nfs = (int)fcol.size() / kIpRows, nbs = (int)bcol.size() / kIpRows;
  std::vector<int> sysd((size_t)kIpEnts * nt, -1), row((size_t)4 * kIpRows * nt, 0), asrc_d((size_t)kIpRows * nt, -1);
  for (int q = 0; q < kIpRows * nt; q++) row[4 * (size_t)q] = -1;
  for (int R = 0; R < nb; R++) {
    asrc_d[place[R]] = dsrc[R];
    for (int r = 0; r < 3; r++) sysd[3 * (size_t)place[R] + r] = 3 * order[R] + r;
  }
  // the transposed places: column C's lower blocks are row C's upper ones, in
  // the same order
  std::vector<int> ldst(fcol.size(), 0), fdia(fcol.size(), 0), fill(rbp.begin(), rbp.end() - 1);
  for (int R = 0; R < nb; R++)
    for (int k = rfp[R]; k < rfp[R + 1]; k++) {
      const int C = low[k].first, q = fill[C]++;
      if (q >= rbp[C + 1] || up[q].first != R) return OD_OK;   // not symmetric: never from a scene's pattern
      ldst[fat[k]] = bat[q];
      fdia[fat[k]] = place[C];
    }
  // pairs of a row's blocks: K ascending for every block (R, C)
  std::vector<int> pa, pb, rounds((size_t)2 * kIpRows * nt, 0), rlist, colour(nb);
  for (int c = 0; c < nc; c++) std::fill(colour.begin() + cstart[c], colour.begin() + cstart[c + 1], c);
  int max_low = 1, max_pairs = 1, max_rounds = 3;
  for (int R = 0; R < nb; R++) {
    const int f0 = rfp[R];
    const size_t at = pa.size(), r0 = rlist.size();
    for (int q = f0; q < rfp[R + 1]; q++) {
      // a round ends after three blocks and with the columns' colour
      const bool more = q > f0 && colour[low[q].first] == colour[low[q - 1].first] && (rlist.size() - r0) % 3 != 0;
      if (!more)
        while ((rlist.size() - r0) % 3 != 0) rlist.push_back(-1);
      const size_t p0 = pa.size() - at;
      int a = f0, b = rfp[low[q].first];
      const int be = rfp[low[q].first + 1];
      while (a < q && b < be) {
        if (low[a].first == low[b].first) {
          pa.push_back(a - f0);
          pb.push_back(fat[b]);
          a++;
          b++;
        } else if (low[a].first < low[b].first) {
          a++;
        } else {
          b++;
        }
      }
      const size_t n = pa.size() - at - p0;
      if (p0 > 0x3fff || n > 255) return OD_OK;
      rlist.push_back((q - f0) | (int)p0 << 8 | (int)n << 22);
    }
    while ((rlist.size() - r0) % 3 != 0) rlist.push_back(-1);
    rounds[2 * (size_t)place[R]] = (int)r0;
    rounds[2 * (size_t)place[R] + 1] = (int)(rlist.size() - r0);
    max_rounds = std::max(max_rounds, (int)(rlist.size() - r0));
    if (pa.size() > 0x3fffffffull) return OD_OK;
    const int m = rfp[R + 1] - f0, np = (int)(pa.size() - at), T = place[R] / kIpRows;
    int* q = &row[4 * (size_t)place[R]];
    q[0] = m;
    q[1] = (int)at;
    q[2] = np;
    q[3] = kIpRows * task[4 * (size_t)T] + place[R] % kIpRows;
    max_low = std::max(max_low, m);
    max_pairs = std::max(max_pairs, np);
  }
  IcPcg I;
  I.nb = nb;
  I.nc = nc;
  I.nt = nt;
  I.nfs = nfs;
  I.nbs = nbs;
  I.max_low = max_low;
  I.max_pairs = max_pairs;
  I.max_rounds = max_rounds;
  const size_t per_warp = sizeof(double) * 9 * (2 * (size_t)max_low + max_pairs) +
                          sizeof(int) * (2 * (size_t)max_pairs + max_rounds);
  I.factor_warps = (int)std::min<size_t>(kIpWarps, kIpSmem / per_warp);
  if (I.factor_warps < 1) return OD_OK;
  I.factor_smem = (I.factor_warps * per_warp + 7) / 8 * 8;
  I.factor_grid = std::min(sms, kIpRows * nt);
  // One cluster while its 16 CTAs' FP64 units keep up with its barriers:
  // measured 2.24 against the grid's 2.38 ms a step at 864 tasks (7,776 DOFs),
  // 2.36 against 2.32 at 972, 2.47 against 2.24 at 1,080, 4.29 against 2.59 at
  // 2,253 (OD_GB300_IC0_PCG=cluster, =grid: either form at any size).
  constexpr int kClusterTasks = 896;
  const char* form = std::getenv("OD_GB300_IC0_PCG");
  const bool want_cluster = form ? form[0] == 'c' : nt <= kClusterTasks;
  auto try_form = [&](bool cluster) {
    I.cluster = cluster;
    I.grid = cluster ? std::min(kIpCluster, (nt + 3) / 4) : std::min(sms, nt);
    I.own = (nt + I.grid - 1) / I.grid;
    I.smem = 5 * sizeof(double) * ((size_t)kIpEnts * I.own + 1);
    if (I.smem > (size_t)kIpSmem || (cluster && kIpEnts * I.own >= 1 << 24)) return false;
    const void* fn = ic_pcg_fn(cluster);
    int n = 0;
    bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kIpSmem) == cudaSuccess;
    if (ok && cluster) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at;
      ic_pcg_config(I.grid, I.smem, true, s->ctx->stream, &cfg, &at);
      ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
           cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= 1;
    } else if (ok) {
      ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kIpThreads, I.smem) == cudaSuccess && n >= 1;
    }
    return ok;
  };
  int n = 0;
  const bool fits = cudaFuncSetAttribute((const void*)ic_pcg_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kIpSmem) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void*)ic_pcg_factor_kernel, kIpThreads,
                                                                  I.factor_smem) == cudaSuccess &&
                    n >= 1 && ((want_cluster && try_form(true)) || try_form(false));
  cudaGetLastError();   // a refused attribute is not an error of the scene
  if (!fits) return OD_OK;
  // the entries that slots read (the padding's: a zero of its own CTA, or
  // behind the vector)
  auto entries = [&](const std::vector<int>& cols, int b16) {
    std::vector<int> idx(3 * cols.size());
    int T = 0;
    for (size_t i = 0; i < cols.size(); i++) {
      while (T + 1 < nt && (size_t)kIpRows * task[4 * (size_t)(T + 1) + b16] <= i) T++;
      for (int c = 0; c < 3; c++) {
        int v = kIpEnts * nt;
        if (cols[i] >= 0) v = 3 * place[cols[i]] + c;
        if (I.cluster) {
          const int Tc = v / kIpEnts;
          v = cols[i] >= 0 ? (Tc % I.grid) << 24 | (kIpEnts * (Tc / I.grid) + v % kIpEnts)
                           : (T % I.grid) << 24 | kIpEnts * I.own;
        }
        idx[3 * i + c] = v;
      }
    }
    return idx;
  };
  const std::vector<int> fidx = entries(fcol, 0), bidx = entries(bcol, 1);
  asrc = asrc_f;
  asrc.insert(asrc.end(), asrc_b.begin(), asrc_b.end());
  asrc.insert(asrc.end(), asrc_d.begin(), asrc_d.end());
  const std::vector<int>* arrays[] = {&task, &row, &rounds, &tbase, &sysd, &fidx, &bidx, &asrc, &ldst, &fdia, &pa, &pb, &rlist};
  const int** dst[] = {&I.task, &I.row, &I.rounds, &I.tbase, &I.sysd, &I.fidx, &I.bidx, &I.asrc, &I.ldst, &I.fdia, &I.pa, &I.pb, &I.rlist};
  constexpr int kArrays = sizeof(dst) / sizeof(dst[0]);
  size_t offs[kArrays];
  std::vector<int> all;
  for (int k = 0; k < kArrays; k++) {
    offs[k] = all.size();
    all.insert(all.end(), arrays[k]->begin(), arrays[k]->end());
  }
  const size_t nv = 2 * (size_t)kIpVals * ((size_t)nfs + nbs + nt) + (size_t)kIpVals * nfs + 2 * ((size_t)kIpEnts * nt + 1);
  const size_t nctr = 4 * kIpCtr + kIpShifts, nadr = I.cluster ? (size_t)kIpEnts * (nfs + nbs) : 0;
  cudaError_t e = plan_malloc(&I.ints, sizeof(int) * all.size());
  if (e == cudaSuccess) e = plan_malloc(&I.vals, sizeof(double) * nv);
  if (e == cudaSuccess) e = plan_malloc(&I.ctr, sizeof(unsigned) * nctr);
  if (e == cudaSuccess && nadr) e = plan_malloc(&I.adr, sizeof(unsigned) * nadr);
  if (e == cudaSuccess) e = cudaMemcpy(I.ints, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice);
  // places no block has are never written: zero
  if (e == cudaSuccess) e = cudaMemsetAsync(I.vals, 0, sizeof(double) * nv, s->ctx->stream);
  if (e != cudaSuccess) {
    cudaFree(I.ints);
    cudaFree(I.vals);
    cudaFree(I.ctr);
    cudaFree(I.adr);
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "IC(0) structure");
    cudaGetLastError();   // no room for it: the separate launches need less
    return OD_OK;
  }
  for (int k = 0; k < kArrays; k++) *dst[k] = I.ints + offs[k];
  s->device_bytes += (long long)(sizeof(int) * all.size() + sizeof(double) * nv + sizeof(unsigned) * (nctr + nadr));
  *out = new IcPcg(I);
  return OD_OK;
}

// The solve; the factor's shift comes back in the scalars' alpha.
od_status ic_pcg_solve(Scene* s, IcPcg* I, const double* d_b, double* d_x, double tol, int max_iter) {
  Pcg& P = s->pcg;
  cudaStream_t st = s->ctx->stream;
  IpArgs a{};
  a.nc = I->nc;
  a.nt = I->nt;
  a.nfs = I->nfs;
  a.nbs = I->nbs;
  a.own = I->own;
  a.max_low = I->max_low;
  a.max_pairs = I->max_pairs;
  a.max_rounds = I->max_rounds;
  a.factor_warps = I->factor_warps;
  a.max_iter = max_iter;
  a.tbase = I->tbase;
  a.sysd = I->sysd;
  a.task = (const int4*)I->task;
  a.row = (const int4*)I->row;
  a.fidx = I->fidx;
  a.bidx = I->bidx;
  a.adr = I->adr;
  a.asrc = I->asrc;
  a.ldst = I->ldst;
  a.fdia = I->fdia;
  a.pa = I->pa;
  a.pb = I->pb;
  a.rounds = (const int2*)I->rounds;
  a.rlist = I->rlist;
  a.A = s->A64;
  a.b = d_b;
  a.x = d_x;
  const size_t nf = (size_t)kIpVals * I->nfs, nbk = (size_t)kIpVals * I->nbs, nd = (size_t)kIpVals * I->nt;
  a.AF = I->vals;
  a.AB = a.AF + nf;
  a.AD = a.AB + nbk;
  a.LF = a.AD + nd;
  a.LB = a.LF + nf;
  a.LD = a.LB + nbk;
  a.LU = a.LD + nd;
  a.v = a.LU + nf;
  a.p = a.v + (size_t)kIpEnts * I->nt + 1;
  a.tol = tol;
  a.part = P.partial;
  a.ctr = I->ctr;
  a.timeout = &((GridBarrier*)P.gbar)->timeout;
  a.bad = (int*)(I->ctr + 4 * kIpCtr);
  a.sc = P.sc;
  OD_CUDA(cudaMemsetAsync(P.gbar, 0, sizeof(GridBarrier), st));
  OD_CUDA(cudaMemsetAsync(I->ctr, 0, sizeof(unsigned) * (4 * kIpCtr + kIpShifts), st));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  s->ctx->sweep_levels = 2 * I->nc;
  void* args[] = {(void*)&a};
  ic_pcg_config(I->factor_grid, I->factor_smem, false, st, &cfg, &at);
  OD_KL(s);
  OD_CUDA(cudaLaunchKernelExC(&cfg, (const void*)ic_pcg_factor_kernel, args));
  ic_pcg_config(I->grid, I->smem, I->cluster, st, &cfg, &at);
  OD_KL(s);
  OD_CUDA(cudaLaunchKernelExC(&cfg, ic_pcg_fn(I->cluster), args));
  return OD_OK;
}

}  // namespace od
