// FP64 products on the integer units.
//
// The part's FP64 unit takes 16 cycles for a warp-wide multiply-add, its
// integer units half a cycle for a 32 x 32 -> 64-bit one.  So a dot product
// whose operands share an exponent each (a matrix row; a vector) runs in
// fixed point: an operand v with |v| < 2^E is X = round(v 2^(60 - E)), kept as
// two signed digits X = h 2^29 + l, and a product takes three wide
// multiply-adds (h h, h l, l h; l l is below the last place).  60 bits against
// a row's sum of magnitudes and a vector's maximum, where FP64 keeps 53 against
// every product: on the matrices and iterates of one-material solves the result
// is within 0.7-1.6e-16 of the exact product in the 2-norm, FP64 within
// 1.2-2.3e-16, as long as E is at most three binary places above the vector's
// maximum (the caller checks that, and multiplies in FP64 otherwise).
#pragma once

#include <cuda_runtime.h>

namespace od {

constexpr int kFxBits = 60;       // |X| < 2^60
constexpr int kFxLow = 29;        // bits of the low digit
constexpr int kFxSlack = 3;       // places E may lie above the operand's maximum
// biased exponents whose scales stay far from FP64's ends
constexpr int kFxExpMin = 600, kFxExpMax = 1446;
constexpr int kFxNone = -4096;    // an E that no operand fits: the caller's check fails

__device__ __forceinline__ int fx_biased_exp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// One exponent for a whole vector loses the small entries' places, and a matrix
// of high contrast multiplies just those by its large values.  So column c of a
// matrix is taken as a 2^-k_c and entry c of the vector as v 2^k_c, k_c the
// exponent of the matrix's diagonal entry: what the preconditioners of these
// solves have divided by.  With one exponent, stiffness contrasts from 1e6 on
// (two materials in a mesh, the stiff one 1e6 as stiff) left the pipelined
// recurrence's true residual at 2.6e-8 where 1e-8 was asked for, and at 1e8 at
// 2.7e-5; with k_c it follows FP64's (up to 1e8, none / Jacobi / block-Jacobi,
// 60-bit digits emulated on the CPU).  Half the exponent does too down to 1e-8,
// and ends at 1.5e-10 for 1e-10 at 1e8.
constexpr int kFxColumnExp = 400;   // most of it, so that zeros stay below kFxExpMin and NaN above kFxExpMax
__device__ __forceinline__ int fx_column_exp(double diag) {
  return min(max(fx_biased_exp(diag) - 1023, -kFxColumnExp), kFxColumnExp);
}
// v 2^k, on the integer units; zero below the normal range (subnormal v too), infinite above it
__device__ __forceinline__ double fx_times_pow2(double v, int k) {
  const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
  if (e == 0x7ff) return v;
  if (e == 0 || e + k <= 0) return 0.0;
  if (e + k >= 0x7ff) return __hiloint2double((hi & (int)0x80000000) | 0x7ff00000, 0);
  return __hiloint2double(hi + k * (1 << 20), __double2loint(v));
}
// the biased exponent of v 2^k, k a column's: outside kFxExpMin .. kFxExpMax for zero, infinities and NaN
__device__ __forceinline__ int fx_biased_exp(double v, int k) { return fx_biased_exp(v) + k; }

// digits of v at the scale E; a magnitude of 2^E and more is cut off (the
// caller's check has failed then), subnormal numbers are zero
__device__ __forceinline__ int2 fx_digits(double v, int E) {
  const int hi = __double2hiint(v);
  const int e = (hi >> 20) & 0x7ff;
  long long m = ((long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(v);
  if (e == 0) m = 0;
  const int s = e - (1075 - kFxBits) - E;
  long long X;
  if (s >= 0) {
    X = m << min(s, 7);
  } else {
    const int r = min(-s, 62);
    X = (m + (1LL << (r - 1))) >> r;
  }
  if (hi < 0) X = -X;
  const long long h = min((X + (1LL << (kFxLow - 1))) >> kFxLow, 0x7fffffffLL);
  return make_int2((int)h, (int)(X - (h << kFxLow)));
}

// x 2^s, rounded to FP64 on the integer units (FP64's own conversions run on
// its slow unit); results below the normal range are zero
__device__ __forceinline__ double fx_double(long long x, int s) {
  if (x == 0) return 0.0;
  unsigned long long a = x < 0 ? 0ull - (unsigned long long)x : (unsigned long long)x;
  const int lz = __clzll((long long)a);
  a <<= lz;
  const int e = 63 - lz + s + 1023;
  const unsigned long long m = (a >> 11) + ((a >> 10) & 1);   // 2^52 .. 2^53
  unsigned long long bits = ((unsigned long long)(e - 1) << 52) + m;
  if (e < 1) bits = 0;
  if (e > 2046) bits = 0x7ff0000000000000ull;
  return __longlong_as_double((long long)(bits | (x < 0 ? 0x8000000000000000ull : 0ull)));
}
// sum of products h 2^58 + mid 2^29: up to 12 products between two carries
// keep mid in range when the magnitudes of one operand's digits sum to 2^31
struct FxAcc {
  long long hh = 0, mid = 0;
  __device__ __forceinline__ void add(int2 a, int2 b) {
    hh += (long long)a.x * b.x;
    mid += (long long)a.x * b.y;
    mid += (long long)a.y * b.x;
  }
  __device__ __forceinline__ void carry() {
    hh += mid >> kFxLow;
    mid &= (1LL << kFxLow) - 1;
  }
  // the sum of products of operands at scales Ea and Eb
  __device__ __forceinline__ double value(int Ea, int Eb) const {
    // hi 2^29 + lo in 64 bits, as far down as the leading zeros allow
    const long long hi = hh + (mid >> kFxLow), lo = mid & ((1LL << kFxLow) - 1);
    const int up = min(kFxLow, __clzll(hi ^ (hi >> 63)) - 1);
    return fx_double((hi << up) | (lo >> (kFxLow - up)), Ea + Eb - (2 * kFxBits - kFxLow) + kFxLow - up);
  }
};

// A sum of products of operands at scales Ea and Eb as digits at the scale
// Ea + Eb + (sh - 2); sh >= 1.
__device__ __forceinline__ int2 fx_split(long long x) {
  const int h = (int)((x + (1LL << (kFxLow - 1))) >> kFxLow);
  return make_int2(h, (int)((unsigned)x - ((unsigned)h << kFxLow)));
}
__device__ __forceinline__ int2 fx_norm(const FxAcc& c, int sh) {
  return fx_split((c.hh + (c.mid >> kFxLow) + (1LL << (sh - 1))) >> sh);
}
// The same sum as FP64, to 2^-62 of its scale 2^E, E = Ea + Eb.
__device__ __forceinline__ double fx_out(const FxAcc& c, int E) {
  return fx_double(c.hh + (c.mid >> kFxLow), E - 2 * (kFxBits - kFxLow));
}

// An FP64 addition holds a warp's unit for 64 cycles, so sums across a warp
// are integer sums too: every addend aligned to the largest exponent em
// (a multiple of 2^(em - 1075 - up)), added as 64-bit integers.  A warp-wide
// sum of one double per lane: 300 cycles against 500 in FP64.
template <int UP>
__device__ __forceinline__ long long fx_align(double v, int em) {
  const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
  long long m = ((long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(v);
  if (e == 0) m = 0;
  m = (((m << (UP + 1)) >> min(em - e, 63)) + 1) >> 1;
  return hi < 0 ? -m : m;
}
template <int UP>
__device__ __forceinline__ double fx_warp_total(long long x, int em) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return em == 0x7ff ? __hiloint2double(0x7ff80000, 0) : fx_double(x, em - 1075 - UP);
}
// the places left above 53 bits when 32 n addends may carry
__host__ __device__ constexpr int fx_up(int n) { return n <= 1 ? 4 : n <= 2 ? 3 : n <= 4 ? 2 : n <= 8 ? 1 : 0; }

}  // namespace od
