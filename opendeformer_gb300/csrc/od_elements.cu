// Per-tetrahedron kernels: precomputes, mass, loads and the material
// kernels (corotational linear, invertible Neo-Hookean / StVK) producing the
// 78 packed stiffness values and 12 nodal forces of every element, scattered
// without atomics: elements are coloured so that one launch (one colour)
// never touches a matrix value or force entry twice.
//
// One thread per element; element data is structure-of-arrays in colour
// order (pre[k * ne + e], emap[k * ne + e]) so every per-element load and the
// map loads are coalesced.  The staged outputs (the gathered assembly's
// input) are element-major, grouped by local node block (c_kslot below).
#include "od_internal.h"
#include "od_fixed.cuh"
#include "od_math.cuh"

namespace od {

// packed position of (i, i) in the 78-entry upper triangle of the 12x12
// element matrix (tetelement.cpp:284)
__constant__ int c_diag12[12] = {0, 12, 23, 33, 42, 50, 57, 63, 68, 72, 75, 77};

// Staged element values (the assembly's input) are element-major: 78
// stiffness values per element with the entries of each local node block
// contiguous -- blocks (0,0), (0,1), (0,2), (0,3), (1,1), ..., (3,3), a
// diagonal block's 6 upper entries, an off-diagonal block's 9 row-major --
// so that the assembly threads of one matrix block read one contiguous run
// of each contributing element; then 12 forces per element in local DOF
// order.  c_kslot maps the packed entry k (row-major upper triangle, the
// reference's order) to its slot.
__constant__ int c_kslot[78] = {0,  1,  2,  6,  7,  8,  15, 16, 17, 24, 25, 26, 3,  4,  9,  10, 11, 18, 19, 20,
                                27, 28, 29, 5,  12, 13, 14, 21, 22, 23, 30, 31, 32, 33, 34, 35, 39, 40, 41, 48,
                                49, 50, 36, 37, 42, 43, 44, 51, 52, 53, 38, 45, 46, 47, 54, 55, 56, 57, 58, 59,
                                63, 64, 65, 60, 61, 66, 67, 68, 62, 69, 70, 71, 72, 73, 74, 75, 76, 77};
__device__ __forceinline__ size_t kst(int k, int e) { return (size_t)e * 78 + c_kslot[k]; }
__device__ __forceinline__ size_t fst(int k, int e) { return (size_t)e * 12 + k; }

__device__ __forceinline__ V3t<double> ld3(const double* p, int n) {
  return {p[3 * n], p[3 * n + 1], p[3 * n + 2]};
}

__device__ __forceinline__ double tet_vol(V3t<double> a, V3t<double> b, V3t<double> c, V3t<double> d) {
  V3t<double> ab = v_sub(b, a), ac = v_sub(c, a), ad = v_sub(d, a);
  return fabs(v_dot(ab, v_cross(ac, ad))) / 6.0;
}

// ------------------------------------------------------------ precomputes
// What every material's element kernel reads of the rest shape, per element
// (structure of arrays, element order): the inverse Dm^-1 of the edge matrix
// (9) and the volume V.  Row i - 1 of Dm^-1 is the gradient of node i's shape
// function and node 0's is minus their sum, so the shape derivatives of
// tetelement.cpp:18-48 (6 V times the gradients) and the corotational rest
// stiffness K0 (tetelement.cpp:501-544) follow from these ten numbers; storing
// K0 cost 720 more bytes an element and its rotation 540 multiply-adds.
constexpr int kPreVol = 9;
constexpr int kPreCount = 10;
int element_precomputes() { return kPreCount; }

__global__ void precompute_kernel(int ne, const int4* __restrict__ tets, const double* __restrict__ X,
                                  double* __restrict__ pre) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  int4 t = tets[e];
  V3t<double> p0 = ld3(X, t.x), p1 = ld3(X, t.y), p2 = ld3(X, t.z), p3 = ld3(X, t.w);
  V3t<double> ab = v_sub(p1, p0), ac = v_sub(p2, p0), ad = v_sub(p3, p0);
  double Dm[9] = {ab.x, ac.x, ad.x, ab.y, ac.y, ad.y, ab.z, ac.z, ad.z}, Di[9];
  double inv = 1.0 / det3(Dm);
  Di[0] = (Dm[4] * Dm[8] - Dm[5] * Dm[7]) * inv;
  Di[1] = (Dm[2] * Dm[7] - Dm[1] * Dm[8]) * inv;
  Di[2] = (Dm[1] * Dm[5] - Dm[2] * Dm[4]) * inv;
  Di[3] = (Dm[5] * Dm[6] - Dm[3] * Dm[8]) * inv;
  Di[4] = (Dm[0] * Dm[8] - Dm[2] * Dm[6]) * inv;
  Di[5] = (Dm[2] * Dm[3] - Dm[0] * Dm[5]) * inv;
  Di[6] = (Dm[3] * Dm[7] - Dm[4] * Dm[6]) * inv;
  Di[7] = (Dm[1] * Dm[6] - Dm[0] * Dm[7]) * inv;
  Di[8] = (Dm[0] * Dm[4] - Dm[1] * Dm[3]) * inv;
  for (int i = 0; i < 9; i++) pre[(size_t)i * ne + e] = Di[i];
  pre[(size_t)kPreVol * ne + e] = tet_vol(p0, p1, p2, p3);
}

// ------------------------------------------------------------ mass / loads
__device__ __forceinline__ int local12(int a, int b) { return a * 12 - ((a - 1) * a) / 2 + b - a; }

// consistent mass, rho V / 10 on the diagonal and rho V / 20 off it, same
// axis only (tetelement.cpp:51-66, mechMaterial.cpp:69-98); one colour
__global__ void mass_kernel(int e0, int e1, int ne, double rho, const double* __restrict__ pre,
                            const int* __restrict__ emap, double* __restrict__ M) {
  int e = e0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= e1) return;
  double vol = pre[(size_t)kPreVol * ne + e];
  double od = vol * 0.05, dg = vol * 0.1;
  for (int a = 0; a < 4; a++)
    for (int b = a; b < 4; b++) {
      double entry = rho * (a == b ? dg : od);
      for (int ax = 0; ax < 3; ax++) {
        int idx = emap[(size_t)local12(3 * a + ax, 3 * b + ax) * ne + e];
        if (idx >= 0) M[idx] += entry;
      }
    }
}

// V/4 per incident element, summed per node (body-force weights); one colour
__global__ void node_vol_kernel(int e0, int e1, int ne, const int4* __restrict__ tets,
                                const double* __restrict__ pre, double* __restrict__ nv) {
  int e = e0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= e1) return;
  int4 t = tets[e];
  double q = pre[(size_t)kPreVol * ne + e] / 4.0;
  nv[t.x] += q; nv[t.y] += q; nv[t.z] += q; nv[t.w] += q;
}

// external forces in one launch: per padded DOF its body force (nodal
// volume x force density, TetElement::getBodyVirtualWorks,
// tetelement.cpp:68-77), then its uniform traction entries over deformed
// facets, area / 3 per vertex (TetFacet::getSurfVirtualWorks,
// tetelement.cpp:79-89), added in the order the loads were given -- the
// order in which Forcer accumulates them (forcer.cpp:8-96)
__global__ void loads_kernel(int n, int dofs, const int* __restrict__ free_pos, const double* __restrict__ nv,
                             double bx, double by, double bz, const int* __restrict__ lptr,
                             const int* __restrict__ lsrc, const int* __restrict__ fids,
                             const double* __restrict__ tvec, double scale, const int* __restrict__ facets,
                             const double* __restrict__ X, const double* __restrict__ u,
                             double* __restrict__ fext) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc = 0.0;
  if (i < dofs) {
    const int p = free_pos[i];
    const int ax = p % 3;
    acc = nv[p / 3] * (ax == 0 ? bx : (ax == 1 ? by : bz));
    if (lptr) {
      for (int j = lptr[i]; j < lptr[i + 1]; j++) {
        const int k = lsrc[j];
        const int f = fids[k];
        const int nd[3] = {facets[3 * f], facets[3 * f + 1], facets[3 * f + 2]};
        V3t<double> q[3];
        for (int v = 0; v < 3; v++)
          q[v] = {X[3 * nd[v]] + u[3 * nd[v]], X[3 * nd[v] + 1] + u[3 * nd[v] + 1], X[3 * nd[v] + 2] + u[3 * nd[v] + 2]};
        const V3t<double> cr = v_cross(v_sub(q[1], q[0]), v_sub(q[2], q[0]));
        const double fac = (sqrt(v_len2(cr)) * 0.5) / 3.0;
        const double w = fac * (scale * tvec[3 * k + ax]);
        if (w != 0.0) acc += w;
      }
    }
  }
  fext[i] = acc;
}

// ------------------------------------------------------ element stiffness
// An element's outputs: MODE 1 the packed 12x12 upper triangle in the caller's
// element order, MODE 2 the colour-ordered staging arrays (node blocks
// contiguous, c_kslot).
template <int MODE>
struct ElemOut {
  double* k;
  double* f;
  __device__ __forceinline__ ElemOut(int e, double* out78, double* out12, const int* perm) {
    const size_t o = MODE == 1 ? (size_t)perm[e] : (size_t)e;
    k = out78 + o * 78;
    f = out12 + o * 12;
  }
  // block (a, b), a <= b, row-major; a diagonal block's upper triangle
  __device__ __forceinline__ void block(int a, int b, const double (&o)[9]) const {
    if constexpr (MODE == 1) {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
          if (a != b || j >= i) k[c_diag12[a * 3 + i] + (b - a) * 3 - i + j] = o[i * 3 + j];
    } else {
      // blocks before (a, b): rows 0..a-1 hold 6 + 9 (3 - row) values each
      const int base = a * 33 - 9 * (a * (a - 1)) / 2 + (b == a ? 0 : 6 + 9 * (b - a - 1));
      double* p = k + base;
      if (a == b) {
        p[0] = o[0];
        p[1] = o[1];
        p[2] = o[2];
        p[3] = o[4];
        p[4] = o[5];
        p[5] = o[8];
      } else if (base & 1) {   // 78 e is even: pairs of values at even places
        p[0] = o[0];
#pragma unroll
        for (int q = 1; q < 9; q += 2) *reinterpret_cast<double2*>(p + q) = make_double2(o[q], o[q + 1]);
      } else {
#pragma unroll
        for (int q = 0; q < 8; q += 2) *reinterpret_cast<double2*>(p + q) = make_double2(o[q], o[q + 1]);
        p[8] = o[8];
      }
    }
  }
  __device__ __forceinline__ void forces(const double (&v)[12]) const {
    double2* p = reinterpret_cast<double2*>(f);
#pragma unroll
    for (int q = 0; q < 6; q++) p[q] = make_double2(v[2 * q], v[2 * q + 1]);
  }
};

// The stiffness runs in fixed point (od_fixed.cuh): it is two thirds of an
// element's arithmetic, a warp-wide FP64 multiply-add holds the SM's FP64 unit
// for 16 cycles and the three wide integer multiply-adds in its place take 1.5.
// Every factor of an element has one scale, products keep 60 bits of theirs,
// and the scales grow by at most 2^7 over a result's own size, so a value
// carries 2^-53 of the element's largest, where FP64's sums of the same
// products carry several 2^-53 (assembled matrix of the beam against 64-bit
// linear algebra, 2-norm: Neo-Hookean 5.9e-16, 5.8e-16 in FP64; corotational
// 5.0e-16 both).  Exponents outside this window (and NaN and infinities among
// the factors) take the same sums in FP64.
// Elements and assembly together, FP64 contraction -> now: Neo-Hookean 98k
// tets 445 -> 256 us, 655k 2,463 -> 1,391; corotational 416 -> 180 and 2,172 ->
// 896.  The FP64 unit is 40% busy with the decompositions then (506
// instructions an element); what keeps it from more are instruction latency at
// 16 warps an SM, waits for constants and instructions, and the last wave of
// warps (98k tets: 1.26 waves).
constexpr int kElExpMin = 823, kElExpMax = 1223;   // biased: 2^-200 .. 2^200
constexpr int kHyperCtas = 8;   // 128 registers a thread: 16 warps on an SM

template <int N>
__device__ __forceinline__ int max_exp(const double (&v)[N], int e = 0) {
#pragma unroll
  for (int i = 0; i < N; i++) e = max(e, fx_biased_exp(v[i]));
  return e;
}
__device__ __forceinline__ bool exp_fits(int e) { return e >= kElExpMin && e <= kElExpMax; }

// Per-thread columns of a CTA's shared memory: rotated gradients as digits
// (component 3 n + i of node n); the hyperelastic stiffness keeps node 0's row
// of blocks there too, as sums over the others.
struct HyperShared {
  int2 g[12][kElThreads];
  long long row0[27][kElThreads];
};

// Gradients of the shape functions in a rotated frame, Q g_n, as digits in
// this thread's column of sa; returns their scale Ea, with |Q g_n| <
// 2^(Ea - 1).  q: Q's digits at the scale 1 (orthonormal, row-major); d: those
// of Di at the scale E, its rows g_1..g_3; node 0's gradient (if asked for) is
// minus their sum.
template <bool NODE0>
__device__ __forceinline__ int fx_gradients(const int2 (&q)[9], const int2 (&d)[9], int E, int2 (*sa)[kElThreads]) {
  // at the scale E + 1, where node 0's, below 6 2^E, stay under 2^62; then
  // moved to the scale that leaves the largest one place spare (each place a
  // factor wastes is lost twice in a stiffness value)
  long long x[4][3], top = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    x[0][i] = 0;
#pragma unroll
    for (int n = 1; n < 4; n++) {
      FxAcc c;
#pragma unroll
      for (int k = 0; k < 3; k++) c.add(q[i * 3 + k], d[(n - 1) * 3 + k]);
      x[n][i] = (c.hh + (c.mid >> kFxLow) + 2) >> 2;
      x[0][i] -= x[n][i];
    }
#pragma unroll
    for (int n = NODE0 ? 0 : 1; n < 4; n++) top |= x[n][i] ^ (x[n][i] >> 63);
  }
  const int r = max(1, 5 - __clzll(top));   // 1..3 for an orthonormal Q
  const long long half = 1LL << (r - 1);
#pragma unroll
  for (int n = NODE0 ? 0 : 1; n < 4; n++)
#pragma unroll
    for (int i = 0; i < 3; i++) sa[3 * n + i][threadIdx.x] = fx_split((x[n][i] + half) >> r);
  return E + 1 + r;
}

__device__ __forceinline__ void fx_digits9(const double (&v)[9], int E, int2 (&d)[9]) {
#pragma unroll
  for (int i = 0; i < 9; i++) d[i] = fx_digits(v[i], E);
}

// f_n = V Q sigma g_n (n > 0) and f_0 = -(f_1 + f_2 + f_3), Q orthonormal.  In
// FP64: in fixed point these 70 operations made the kernels 5% slower, the
// FP64 units being half idle beside the stiffness.
template <int MODE>
__device__ __forceinline__ void stress_forces(const double (&Q)[9], const double (&st)[9], const double (&Di)[9], double vol,
                                              const ElemOut<MODE>& out) {
  double P[9], f[12];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      P[i * 3 + j] = (Q[i * 3] * st[j] + Q[i * 3 + 1] * st[3 + j] + Q[i * 3 + 2] * st[6 + j]) * vol;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    f[i] = 0.0;
#pragma unroll
    for (int n = 0; n < 3; n++) {
      f[3 * (n + 1) + i] = P[i * 3] * Di[n * 3] + P[i * 3 + 1] * Di[n * 3 + 1] + P[i * 3 + 2] * Di[n * 3 + 2];
      f[i] -= f[3 * (n + 1) + i];
    }
  }
  out.forces(f);
}

// The corotational stiffness R K0_ab R^T = V (lambda h_a h_b^T + mu h_b h_a^T +
// mu (h_a . h_b) I), h = R g: K0 is isotropic, so rotating it is rotating the
// gradients (tetelement.cpp:501-544, 583-651).
template <int MODE>
__device__ __noinline__ void corot_stiffness64(const double* R, const double* Di, double lv, double mv, ElemOut<MODE> out) {
  double h[4][3];
  for (int i = 0; i < 3; i++) {
    h[0][i] = 0.0;
    for (int n = 0; n < 3; n++) {
      h[n + 1][i] = R[i * 3] * Di[n * 3] + R[i * 3 + 1] * Di[n * 3 + 1] + R[i * 3 + 2] * Di[n * 3 + 2];
      h[0][i] -= h[n + 1][i];
    }
  }
  for (int a = 0; a < 4; a++)
    for (int b = a; b < 4; b++) {
      const double dot = mv * (h[a][0] * h[b][0] + h[a][1] * h[b][1] + h[a][2] * h[b][2]);
      double o[9];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) o[i * 3 + j] = lv * h[a][i] * h[b][j] + mv * h[b][i] * h[a][j] + (i == j ? dot : 0.0);
      out.block(a, b, o);
    }
}

template <int MODE>
__device__ __forceinline__ void corot_stiffness(const double (&R)[9], const double (&Di)[9], double lv, double mv,
                                                int2 (*sa)[kElThreads], const ElemOut<MODE>& out) {
  const int eD = max_exp(Di), eL = max(fx_biased_exp(lv), fx_biased_exp(mv));
  if (!(max_exp(R) <= 1023 && exp_fits(eD) && exp_fits(eL))) {
    corot_stiffness64<MODE>(R, Di, lv, mv, out);
    return;
  }
  int2 dR[9], dD[9];
  fx_digits9(R, 1, dR);
  fx_digits9(Di, eD - 1022, dD);
  const int Ea = fx_gradients<true>(dR, dD, eD - 1022, sa), El = eL - 1022;
  const int2 dl = fx_digits(lv, El), dm = fx_digits(mv, El);
#pragma unroll 1
  for (int a = 0; a < 4; a++) {
    // V lambda h_a and V mu h_a at the scale El + Ea: one place spare, five
    // products of a diagonal value in one sum
    int2 ha[3], la[3], ma[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      ha[i] = sa[3 * a + i][threadIdx.x];
      FxAcc c, d;
      c.add(dl, ha[i]);
      d.add(dm, ha[i]);
      la[i] = fx_norm(c, 2);
      ma[i] = fx_norm(d, 2);
    }
#pragma unroll 1
    for (int b = a; b < 4; b++) {
      int2 hb[3];
#pragma unroll
      for (int i = 0; i < 3; i++) hb[i] = sa[3 * b + i][threadIdx.x];
      FxAcc dot;
#pragma unroll
      for (int i = 0; i < 3; i++) dot.add(ma[i], hb[i]);
      double o[9];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          FxAcc c;
          if (i == j) c = dot;
          c.add(la[i], hb[j]);
          c.add(ma[j], hb[i]);
          o[i * 3 + j] = fx_out(c, El + 2 * Ea);
        }
      out.block(a, b, o);
    }
  }
}

// -------------------------------------------------- corotational element
// F = [x1-x0, x2-x0, x3-x0] Dm^-1; R = polar(F), or the proper QR factor when
// the deformed volume is below threshold * rest volume
// (tetelement.cpp:546-573); S = R^T F.
__device__ __forceinline__ void corot_frame(int e, int ne, const int4* __restrict__ tets, const double* __restrict__ X,
                                            const double* __restrict__ u, const double* __restrict__ pre, double thr,
                                            double (&Di)[9], double& v0, double (&R)[9], double (&S)[9]) {
  int4 t = tets[e];
  const int nd[4] = {t.x, t.y, t.z, t.w};
  V3t<double> c[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    V3t<double> x = ld3(X, nd[i]), du = ld3(u, nd[i]);
    c[i] = {x.x + du.x, x.y + du.y, x.z + du.z};
  }
  double F[9];
#pragma unroll
  for (int i = 0; i < 9; i++) { Di[i] = pre[(size_t)i * ne + e]; F[i] = 0.0; }
#pragma unroll
  for (int i = 1; i < 4; i++) {
    double ax[3] = {c[i].x - c[0].x, c[i].y - c[0].y, c[i].z - c[0].z};
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int k = 0; k < 3; k++) F[j * 3 + k] += ax[j] * Di[(i - 1) * 3 + k];
  }
  v0 = pre[(size_t)kPreVol * ne + e];
  const double v1 = tet_vol(c[0], c[1], c[2], c[3]);
  if (v1 >= thr * v0) polar3<double>(F, R);
  else qr3<double>(F, R);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) S[i * 3 + j] = R[i] * F[j] + R[3 + i] * F[3 + j] + R[6 + i] * F[6 + j];
}

// Corotational linear element: f_a = sum_b (R K0_ab R^T x_b - R K0_ab X_b)
// (tetelement.cpp:583-651), which for the isotropic K0 is the stress of the
// strain sym(S) - I on the rotated gradients; K_ab = R K0_ab R^T.
template <int MODE>
__device__ __forceinline__ void corot_elem(int e, int ne, const int4* __restrict__ tets, const double* __restrict__ X,
                                           const double* __restrict__ u, const double* __restrict__ pre, double thr,
                                           double lambda, double mu, double* __restrict__ out78,
                                           double* __restrict__ out12, const int* __restrict__ perm,
                                           int2 (*sa)[kElThreads]) {
  double Di[9], R[9], S[9], v0, st[9];
  corot_frame(e, ne, tets, X, u, pre, thr, Di, v0, R, S);
  const ElemOut<MODE> out(e, out78, out12, perm);
  const double d0 = S[0] - 1.0, d1 = S[4] - 1.0, d2 = S[8] - 1.0, dg = lambda * (d0 + d1 + d2), mu2 = 2.0 * mu;
  st[0] = mu2 * d0 + dg;
  st[4] = mu2 * d1 + dg;
  st[8] = mu2 * d2 + dg;
  st[1] = st[3] = mu * (S[1] + S[3]);
  st[2] = st[6] = mu * (S[2] + S[6]);
  st[5] = st[7] = mu * (S[5] + S[7]);
  stress_forces<MODE>(R, st, Di, v0, out);
  corot_stiffness<MODE>(R, Di, lambda * v0, mu * v0, sa, out);
}

// ------------------------------------------- invertible hyperelastic element
// K_ab = V U [sum_kl dP_ikjl a_ak a_bl] U^T, a_n = V^T g_n (tetelement.cpp:282-342),
// dP/dF in the singular frame by its 21 structural non-zeros: T (the
// diagonal's), Al and Be (tetelement.cpp:357-499).
template <int MODE>
__device__ __noinline__ void hyper_stiffness64(const double* U, const double* VT, const double* Di, const double* T6,
                                               const double* al, const double* be, double vol, ElemOut<MODE> out) {
  double an[4][3], T[3][3] = {{T6[0], T6[1], T6[2]}, {T6[1], T6[3], T6[4]}, {T6[2], T6[4], T6[5]}};
  for (int i = 0; i < 3; i++) {
    an[0][i] = 0.0;
    for (int n = 0; n < 3; n++) {
      an[n + 1][i] = VT[i * 3] * Di[n * 3] + VT[i * 3 + 1] * Di[n * 3 + 1] + VT[i * 3 + 2] * Di[n * 3 + 2];
      an[0][i] -= an[n + 1][i];
    }
  }
  for (int a = 0; a < 4; a++)
    for (int b = a; b < 4; b++) {
      double sm[9], tmp[9], o[9];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
          double en = 0.0;
          if (i == j) {
            for (int k = 0; k < 3; k++) en += (k == i ? T[i][i] : al[i + k - 1]) * an[a][k] * an[b][k];
          } else {
            en = T[i][j] * an[a][i] * an[b][j] + be[i + j - 1] * an[a][j] * an[b][i];
          }
          sm[i * 3 + j] = en;
        }
      mul3(U, sm, tmp);
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
          o[i * 3 + j] = (tmp[i * 3] * U[j * 3] + tmp[i * 3 + 1] * U[j * 3 + 1] + tmp[i * 3 + 2] * U[j * 3 + 2]) * vol;
      out.block(a, b, o);
    }
}

// al, be: entries (0,1), (0,2), (1,2); the index of (i, k) is i + k - 1
template <int MODE>
__device__ __forceinline__ void hyper_stiffness(const double (&U)[9], const double (&VT)[9], const double (&Di)[9],
                                                const double (&T6)[6], const double (&al)[3], const double (&be)[3],
                                                double vol, HyperShared& sh, const ElemOut<MODE>& out) {
  const int eT = max_exp(T6, max_exp(al, max_exp(be))), eD = max_exp(Di), eV = fx_biased_exp(vol);
  if (!(max_exp(U, max_exp(VT)) <= 1023 && exp_fits(eT) && exp_fits(eD) && exp_fits(eV))) {
    hyper_stiffness64<MODE>(U, VT, Di, T6, al, be, vol, out);
    return;
  }
  const int2 dv = fx_digits(vol, eV - 1022);
  int2 dU[9], dD[9], dVT[9];
  fx_digits9(U, 1, dU);
  fx_digits9(Di, eD - 1022, dD);
  fx_digits9(VT, 1, dVT);
  const int Ea = fx_gradients<false>(dVT, dD, eD - 1022, sh.g);
  // V dP/dF at the scale Et
  auto times_vol = [&](double t) {
    FxAcc c;
    c.add(fx_digits(t, eT - 1022), dv);
    return fx_norm(c, 2);
  };
  int2 dT[6], dA[3], dB[3];
#pragma unroll
  for (int i = 0; i < 6; i++) dT[i] = times_vol(T6[i]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    dA[i] = times_vol(al[i]);
    dB[i] = times_vol(be[i]);
  }
  auto sym6 = [](int i, int j) { return i <= j ? i * 3 - (i * (i - 1)) / 2 + (j - i) : j * 3 - (j * (j - 1)) / 2 + (i - j); };
  const int Et = eT + eV - 2044;
  // Blocks of nodes 1..3 by products; a column of blocks sums to zero (the
  // gradients do), so node 0's follow by exact integer sums.
  const int Ek = Et + 2 * Ea + 2;
#pragma unroll
  for (int i = 0; i < 27; i++) sh.row0[i][threadIdx.x] = 0;
#pragma unroll 1
  for (int a = 1; a < 4; a++) {
    // dP/dF contracted with node a's gradient, at the scale Et + Ea - 1
    int2 ha[3], wd[3][3], wo[3][3], wb[3][3];   // diagonal values' terms by k; T_ij a_i; Be_ij a_j
#pragma unroll
    for (int i = 0; i < 3; i++) ha[i] = sh.g[3 * a + i][threadIdx.x];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        auto times = [&](int2 t, int2 h) {
          FxAcc c;
          c.add(t, h);
          return fx_norm(c, 1);
        };
        wd[i][j] = times(i == j ? dT[sym6(i, i)] : dA[i + j - 1], ha[j]);
        if (i != j) {
          wo[i][j] = times(dT[sym6(i, j)], ha[i]);
          wb[i][j] = times(dB[i + j - 1], ha[j]);
        }
      }
#pragma unroll 1
    for (int b = a; b < 4; b++) {
      int2 hb[3], sm[9], tmp[9];
#pragma unroll
      for (int i = 0; i < 3; i++) hb[i] = sh.g[3 * b + i][threadIdx.x];
      // at the scale Et + 2 Ea: three products, below 0.75 of it
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          FxAcc c;
          if (i == j) {
#pragma unroll
            for (int k = 0; k < 3; k++) c.add(wd[i][k], hb[k]);
          } else {
            c.add(wo[i][j], hb[j]);
            c.add(wb[i][j], hb[i]);
          }
          sm[i * 3 + j] = fx_norm(c, 3);
        }
      // U sm, at the scale Et + 2 Ea + 1
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          FxAcc c;
#pragma unroll
          for (int k = 0; k < 3; k++) c.add(sm[k * 3 + j], dU[i * 3 + k]);
          tmp[i * 3 + j] = fx_norm(c, 2);
        }
      // (U sm) U^T: below 0.57 2^62 in units of 2^(Ek - 62), so three of them
      // fit an integer
      double o[9];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          FxAcc c;
#pragma unroll
          for (int k = 0; k < 3; k++) c.add(tmp[i * 3 + k], dU[j * 3 + k]);
          const long long x = c.hh + (c.mid >> kFxLow);
          sh.row0[9 * (b - 1) + 3 * i + j][threadIdx.x] -= x;
          if (a != b) sh.row0[9 * (a - 1) + 3 * j + i][threadIdx.x] -= x;
          o[i * 3 + j] = fx_double(x, Ek - 2 * (kFxBits - kFxLow));
        }
      out.block(a, b, o);
    }
  }
  long long own[9];
#pragma unroll
  for (int i = 0; i < 9; i++) own[i] = 0;
#pragma unroll 1
  for (int b = 1; b < 4; b++) {
    double o[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
      const long long x = sh.row0[9 * (b - 1) + i][threadIdx.x];
      own[i] -= x >> 2;
      o[i] = fx_double(x, Ek - 2 * (kFxBits - kFxLow));
    }
    out.block(0, b, o);
  }
  double o[9];
#pragma unroll
  for (int i = 0; i < 9; i++) o[i] = fx_double(own[i], Ek + 2 - 2 * (kFxBits - kFxLow));
  out.block(0, 0, o);
}

// Invertible SVD of F, energy derivatives in the invariants I1 = sum s^2,
// I2 = sum s^4, I3 = prod s^2 (invertibleHyperelastic.h:22-30): Neo-Hookean
// (invertibleNeoHookean.cpp:11-20) or StVK (invertibleStVK.cpp:11-20);
// P = U diag(2 g1 s + 4 g2 s^3 + 2 g3 I3 / s) V^T (invertibleHyperelastic.cpp:
// 247-265); dP/dF in the singular-value frame projected to PSD
// (tetelement.cpp:357-499); f_n = V P g_n, f_0 = -(f_1 + f_2 + f_3)
// (tetelement.cpp:344-355).  I3 / s_i and I3 / (s_i s_j) are the products of
// the other factors: FP64 divisions are long instruction sequences.
template <int MODE>
__device__ __forceinline__ void invhyper_elem(int e, int ne, int stvk, const int4* __restrict__ tets,
                                              const double* __restrict__ X, const double* __restrict__ u,
                                              const double* __restrict__ pre, double thr, double lambda, double mu,
                                              double* __restrict__ out78, double* __restrict__ out12,
                                              const int* __restrict__ perm, bool refine, HyperShared& sh) {
  int4 t = tets[e];
  const int nd[4] = {t.x, t.y, t.z, t.w};
  V3t<double> c[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    V3t<double> x = ld3(X, nd[i]), du = ld3(u, nd[i]);
    c[i] = {x.x + du.x, x.y + du.y, x.z + du.z};
  }
  double F[9], Di[9];
#pragma unroll
  for (int i = 0; i < 9; i++) { Di[i] = pre[(size_t)i * ne + e]; F[i] = 0.0; }
#pragma unroll
  for (int i = 1; i < 4; i++) {
    double ax[3] = {c[i].x - c[0].x, c[i].y - c[0].y, c[i].z - c[0].z};
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int k = 0; k < 3; k++) F[j * 3 + k] += ax[j] * Di[(i - 1) * 3 + k];
  }
  double sig[3], U[9], VT[9];
  if (!invertible_svd<double, true, false>(F, thr, sig, U, VT)) {
    if (refine) invertible_svd_flat<true>(F, thr, sig, U, VT);
    else invertible_svd_flat<false>(F, thr, sig, U, VT);
  }
  const double s02 = sig[0] * sig[0], s12 = sig[1] * sig[1], s22 = sig[2] * sig[2];
  const double I1 = s02 + s12 + s22, I3 = s02 * s12 * s22;
  // dP/dF non-zeros (tetelement.cpp:357-437).  Neo-Hookean has no derivative
  // in I2 and one second derivative, in I3; StVK no derivative in I3 and one
  // second derivative, in I1.  d_ij = I3 g2 / (s_i s_j).
  const double sc01 = sig[0] * sig[1], sc02 = sig[0] * sig[2], sc12 = sig[1] * sig[2];
  // I3 / s_i
  const double qs[3] = {sig[0] * (s12 * s22), sig[1] * (s02 * s22), sig[2] * (s02 * s12)};
  double al[3], be[3], T[6], de[3];   // de: dE / ds_i
  if (!stvk) {
    const double lI3 = log(I3), rI3 = 1.0 / I3;
    const double g0 = 0.5 * mu, g2 = (-0.5 * mu + 0.25 * lambda * lI3) * rI3;
    const double h5 = (0.5 * mu + 0.25 * lambda * (1.0 - lI3)) * (rI3 * rI3);
    const double a = 2.0 * g0, h = 4.0 * h5, g = 2.0 * g2;
    const double d00 = g2 * (s12 * s22), d01 = g2 * (sc01 * s22), d02 = g2 * (sc02 * s12);
    const double d11 = g2 * (s02 * s22), d12 = g2 * (sc12 * s02), d22 = g2 * (s02 * s12);
    al[0] = al[1] = al[2] = a;
    be[0] = -2.0 * d01;
    be[1] = -2.0 * d02;
    be[2] = -2.0 * d12;
    const double h0 = h * qs[0], h1 = h * qs[1], h2 = h * qs[2];
    T[0] = fma(-2.0, d00, a) + fma(4.0, d00, qs[0] * h0);
    T[1] = fma(4.0, d01, qs[1] * h0);
    T[2] = fma(4.0, d02, qs[2] * h0);
    T[3] = fma(-2.0, d11, a) + fma(4.0, d11, qs[1] * h1);
    T[4] = fma(4.0, d12, qs[2] * h1);
    T[5] = fma(-2.0, d22, a) + fma(4.0, d22, qs[2] * h2);
#pragma unroll
    for (int i = 0; i < 3; i++) de[i] = fma(g, qs[i], a * sig[i]);
  } else {
    const double g0 = 0.25 * lambda * (I1 - 3.0) - 0.5 * mu, g1 = 0.25 * mu;
    const double a = 2.0 * g0, b = 4.0 * g1, h = lambda;   // h: 4 d2E / dI1^2
    al[0] = fma(s02 + s12, b, a);
    al[1] = fma(s02 + s22, b, a);
    al[2] = fma(s12 + s22, b, a);
    be[0] = sc01 * b;
    be[1] = sc02 * b;
    be[2] = sc12 * b;
    const double t0 = s02 * b, t1 = s12 * b, t2 = s22 * b, h0 = h * sig[0], h1 = h * sig[1], h2 = h * sig[2];
    T[0] = fma(2.0, t0, a) + t0 + sig[0] * h0;
    T[1] = sig[1] * h0;
    T[2] = sig[2] * h0;
    T[3] = fma(2.0, t1, a) + t1 + sig[1] * h1;
    T[4] = sig[2] * h1;
    T[5] = fma(2.0, t2, a) + t2 + sig[2] * h2;
    de[0] = sig[0] * (a + t0);
    de[1] = sig[1] * (a + t1);
    de[2] = sig[2] * (a + t2);
  }
  psd3<double>(T);
#pragma unroll
  for (int i = 0; i < 3; i++) psd2<double>(al[i], be[i]);
  const double vol = pre[(size_t)kPreVol * ne + e];
  const ElemOut<MODE> out(e, out78, out12, perm);
  double dvt[9];
#pragma unroll
  for (int i = 0; i < 3; i++) {
#pragma unroll
    for (int j = 0; j < 3; j++) dvt[i * 3 + j] = de[i] * VT[i * 3 + j];
  }
  stress_forces<MODE>(U, dvt, Di, vol, out);
  hyper_stiffness<MODE>(U, VT, Di, T, al, be, vol, sh, out);
}

template <int MODE>
__global__ void __launch_bounds__(kElThreads) corot_kernel(int ne, const int4* __restrict__ tets,
                                                           const double* __restrict__ X, const double* __restrict__ u,
                                                           const double* __restrict__ pre, double thr, double lambda,
                                                           double mu, double* __restrict__ out78,
                                                           double* __restrict__ out12, const int* __restrict__ perm) {
  __shared__ int2 sa[12][kElThreads];
  const int e = blockIdx.x * kElThreads + threadIdx.x;
  if (e < ne) corot_elem<MODE>(e, ne, tets, X, u, pre, thr, lambda, mu, out78, out12, perm, sa);
}

template <int MODE>
__global__ void __launch_bounds__(kElThreads, kHyperCtas) invhyper_kernel(int ne, int stvk, const int4* __restrict__ tets,
                                                              const double* __restrict__ X,
                                                              const double* __restrict__ u,
                                                              const double* __restrict__ pre, double thr, double lambda,
                                                              double mu, double* __restrict__ out78,
                                                              double* __restrict__ out12, const int* __restrict__ perm,
                                                              bool refine) {
  __shared__ HyperShared sh;
  const int e = blockIdx.x * kElThreads + threadIdx.x;
  if (e < ne) invhyper_elem<MODE>(e, ne, stvk, tets, X, u, pre, thr, lambda, mu, out78, out12, perm, refine, sh);
}

// ---- several scenes per launch: tile j of scene s (directory prefix) is
// its elements [kElThreads j, kElThreads (j + 1)); every scene's values land in its own
// staging arrays
__global__ void __launch_bounds__(kElThreads) corot_batch_kernel(int n_sc, const int* __restrict__ prefix,
                                                                 const SceneDev* __restrict__ sd) {
  __shared__ int2 sa[12][kElThreads];
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  const int e = (blockIdx.x - prefix[s]) * kElThreads + threadIdx.x;
  if (e >= D.n_tets) return;
  corot_elem<2>(e, D.n_tets, D.tets, D.X, D.u, D.pre, D.thr, D.lambda, D.mu, D.stage_k, D.stage_f, nullptr, sa);
}

__global__ void __launch_bounds__(kElThreads, kHyperCtas) invhyper_batch_kernel(int n_sc, const int* __restrict__ prefix,
                                                                    const SceneDev* __restrict__ sd) {
  __shared__ HyperShared sh;
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  const int e = (blockIdx.x - prefix[s]) * kElThreads + threadIdx.x;
  if (e >= D.n_tets) return;
  invhyper_elem<2>(e, D.n_tets, D.kind == OD_MATERIAL_STVK, D.tets, D.X, D.u, D.pre, D.thr, D.lambda, D.mu, D.stage_k,
                   D.stage_f, nullptr, true, sh);
}

// Corotational plastic element (corotationalPlastic.cpp:53-183,
// tetelement.cpp:654-729).  F = R S: polar decomposition (S = R^T F), or QR
// when the deformed volume falls below threshold x rest volume (S = Q^T F,
// the upper factor).  Elastic strain e = sym(S) - I - plastic strain; stress
// 2 mu e + lambda tr(e) I, rotated by R; forces f_a = (R stress) dN_a / 6
// (a < 3), f_3 = -(f_0 + f_1 + f_2); stiffness R K0_ab R^T.  Every
// evaluation updates the element's plastic strain (in place, as the
// reference does): when the strain norm exceeds the yield criterion it grows
// by creep (|e| - yield)/|e| e and is scaled back to the maximum.  Both
// norms follow the reference, which adds the squares of the first three
// entries three times (corotationalPlastic.cpp:156-160, 169-173).
// plastic: [9][ne].
template <int MODE>
__device__ __forceinline__ void plastic_elem(int e, int ne, const int4* __restrict__ tets,
                                             const double* __restrict__ X, const double* __restrict__ u,
                                             const double* __restrict__ pre, double thr, double lambda, double mu,
                                             double yield, double creep, double max_plastic,
                                             double* __restrict__ plastic, double* __restrict__ out78,
                                             double* __restrict__ out12, const int* __restrict__ perm,
                                             int2 (*sa)[kElThreads]) {
  double Di[9], R[9], S[9], v0;
  corot_frame(e, ne, tets, X, u, pre, thr, Di, v0, R, S);
  const ElemOut<MODE> out(e, out78, out12, perm);
  // elastic strain, stress, plastic update (computeElasticStress)
  double ep[9], es[9];
#pragma unroll
  for (int i = 0; i < 9; i++) ep[i] = plastic[(size_t)i * ne + e];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) es[i * 3 + j] = 0.5 * (S[i * 3 + j] + S[j * 3 + i]) - ep[i * 3 + j];
  es[0] -= 1.0;
  es[4] -= 1.0;
  es[8] -= 1.0;
  const double mu2 = 2.0 * mu;
  double st[9];
#pragma unroll
  for (int i = 0; i < 9; i++) st[i] = mu2 * es[i];
  const double dg = lambda * (es[0] + es[4] + es[8]);
  st[0] += dg;
  st[4] += dg;
  st[8] += dg;
  double en = 0.0;  // the reference's sum: each of the first three squares three times, in its order
#pragma unroll
  for (int i = 0; i < 3; i++) {
    en += es[i] * es[i];
    en += es[i] * es[i];
    en += es[i] * es[i];
  }
  en = sqrt(en);
  if (en > yield) {
    const double ratio = creep * (en - yield) / en;
#pragma unroll
    for (int i = 0; i < 9; i++) ep[i] += ratio * es[i];
    double pn = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      pn += ep[i] * ep[i];
      pn += ep[i] * ep[i];
      pn += ep[i] * ep[i];
    }
    pn = sqrt(pn);
    if (pn > max_plastic) {
      const double fac = max_plastic / pn;
#pragma unroll
      for (int i = 0; i < 9; i++) ep[i] *= fac;
    }
#pragma unroll
    for (int i = 0; i < 9; i++) plastic[(size_t)i * ne + e] = ep[i];
  }
  stress_forces<MODE>(R, st, Di, v0, out);
  corot_stiffness<MODE>(R, Di, lambda * v0, mu * v0, sa, out);
}

template <int MODE>
__global__ void __launch_bounds__(kElThreads) plastic_kernel(int ne, const int4* __restrict__ tets,
                                                      const double* __restrict__ X, const double* __restrict__ u,
                                                      const double* __restrict__ pre, double thr, double lambda,
                                                      double mu, double yield, double creep, double max_plastic,
                                                      double* __restrict__ plastic, double* __restrict__ out78,
                                                      double* __restrict__ out12, const int* __restrict__ perm) {
  __shared__ int2 sa[12][kElThreads];
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < ne)
    plastic_elem<MODE>(e, ne, tets, X, u, pre, thr, lambda, mu, yield, creep, max_plastic, plastic, out78, out12,
                       perm, sa);
}

__global__ void __launch_bounds__(kElThreads) plastic_batch_kernel(int n_sc, const int* __restrict__ prefix,
                                                                   const SceneDev* __restrict__ sd) {
  __shared__ int2 sa[12][kElThreads];
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  const int e = (blockIdx.x - prefix[s]) * kElThreads + threadIdx.x;
  if (e >= D.n_tets) return;
  plastic_elem<2>(e, D.n_tets, D.tets, D.X, D.u, D.pre, D.thr, D.lambda, D.mu, D.yield, D.creep, D.max_plastic,
                  D.plastic, D.stage_k, D.stage_f, nullptr, sa);
}

// atomic-free scatter of staged element values, one colour per launch
// (corotationalHyperelastic.cpp:100-120): no two elements of a colour share
// a matrix value or a force entry.  One thread per (element, entry): entries
// 0..77 are stiffness values, 78..89 forces; for a fixed entry consecutive
// threads read consecutive staged values and map entries.
__global__ void scatter_kernel(int e0, int cnt, int ne, const double* __restrict__ k78, const double* __restrict__ f12,
                               const int* __restrict__ emap, const int* __restrict__ gdof, double* __restrict__ K,
                               double* __restrict__ fint) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 90LL * cnt) return;
  const int k = (int)(t / cnt);
  const int e = e0 + (int)(t - (long long)k * cnt);
  if (k < 78) {
    const int idx = emap[(size_t)k * ne + e];
    if (idx >= 0) K[idx] += k78[kst(k, e)];
  } else {
    const int g = gdof[(size_t)(k - 78) * ne + e];
    if (g >= 0) fint[g] += f12[fst(k - 78, e)];
  }
}

// gathered assembly: value i of K (and entry i of the forces) is the sum of
// its element contributions in the reference's assembly order (element
// index, then the element's entry index; the loops of
// material/corotationalHyperelastic.cpp:67-97), started from zero, so the
// additions happen in the reference's sequence.  One thread per destination,
// no atomics, no colour passes.
__device__ __forceinline__ void gather_one(long long i, int nk, const int* __restrict__ kptr,
                                           const int* __restrict__ ksrc, const double* __restrict__ k78,
                                           double* __restrict__ K, int nf, const int* __restrict__ fptr,
                                           const int* __restrict__ fsrc, const double* __restrict__ f12,
                                           double* __restrict__ fint, int accumulate, double* host_k = nullptr,
                                           double* host_f = nullptr, int host_nf = 0) {
  const int* ptr = kptr;
  const int* src = ksrc;
  const double* val = k78;
  double* out = K;
  double* host = host_k;
  if (i >= nk) {
    i -= nk;
    if (i >= nf) return;
    ptr = fptr; src = fsrc; val = f12; out = fint;
    host = i < host_nf ? host_f : nullptr;
  }
  const int j1 = ptr[i + 1];
  double acc = accumulate ? out[i] : 0.0;
  for (int j = ptr[i]; j < j1; j++) acc += val[src[j]];
  out[i] = acc;
  if (host) host[i] = acc;
}

__global__ void __launch_bounds__(256) gather_kernel(int nk, const int* __restrict__ kptr,
                                                     const int* __restrict__ ksrc, const double* __restrict__ k78,
                                                     double* __restrict__ K, int nf, const int* __restrict__ fptr,
                                                     const int* __restrict__ fsrc, const double* __restrict__ f12,
                                                     double* __restrict__ fint, int accumulate, double* host_k = nullptr,
                                                     double* host_f = nullptr, int host_nf = 0) {
  gather_one((long long)blockIdx.x * blockDim.x + threadIdx.x, nk, kptr, ksrc, k78, K, nf, fptr, fsrc, f12, fint,
             accumulate, host_k, host_f, host_nf);
}

// multi-scene scatter of colour c: tile j of scene s covers the colour's
// threads [256 j, 256 j + 256) (90 per element: 78 stiffness values, 12
// forces)
__global__ void scatter_batch_kernel(int n_sc, const int* __restrict__ prefix, int c,
                                     const SceneDev* __restrict__ sd) {
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  const int e0 = D.color_off[c], cnt = D.color_off[c + 1] - e0;
  const int t = (blockIdx.x - prefix[s]) * 256 + threadIdx.x;
  if (t >= 90 * cnt) return;
  const int ne = D.n_tets;
  const int k = t / cnt;
  const int e = e0 + (t - k * cnt);
  if (k < 78) {
    const int idx = D.emap[(size_t)k * ne + e];
    if (idx >= 0) D.K[idx] += D.stage_k[kst(k, e)];
  } else {
    const int g = D.gdof[(size_t)(k - 78) * ne + e];
    if (g >= 0) D.fint[g] += D.stage_f[fst(k - 78, e)];
  }
}

// ---- the gather lists, built on the device once per scene: count the
// contributions of every destination, scan the counts into the list
// offsets, place every source with an atomic cursor, then sort each list
// by (original element index, entry index) -- the reference's assembly
// order, whatever order the atomics placed them in.
constexpr int kScanBlock = 1024;

__global__ void gl_count_kernel(long long n, const int* __restrict__ dest, int* __restrict__ cnt) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int d = dest[t];
    if (d >= 0) atomicAdd(&cnt[d + 1], 1);
  }
}

// inclusive scan of each 1024-entry block in place; the block's total to sums
__global__ void __launch_bounds__(kScanBlock) gl_scan_block_kernel(int n, int* __restrict__ data,
                                                                   int* __restrict__ sums) {
  __shared__ int warp_tot[kScanBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  int v = i < n ? data[i] : 0;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int w = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v += warp_tot[warp - 1];
  if (i < n) data[i] = v;
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = v;
}

__global__ void __launch_bounds__(kScanBlock) gl_add_kernel(int n, int* __restrict__ data,
                                                            const int* __restrict__ offs) {
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) data[i] += offs[blockIdx.x];
}

// map entry t = k * ne + e (e the element's staged position) -> its staged
// source: e * kk + slot (c_kslot for the 78 stiffness values, k for forces)
__global__ void gl_fill_kernel(long long n, const int* __restrict__ dest, int* __restrict__ cur,
                               int* __restrict__ src, int ne, int kk) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int d = dest[t];
    if (d >= 0) {
      const int k = (int)(t / ne), e = (int)(t - (long long)k * ne);
      src[atomicAdd(&cur[d], 1)] = e * kk + (kk == 78 ? c_kslot[k] : k);
    }
  }
}

// a list's sources (e * kk + slot) sort by perm[e] * kk + slot: an element
// contributes at most once to a destination, so this is the reference's
// order, by original element index
__global__ void gl_sort_kernel(int nd, const int* __restrict__ ptr, int* __restrict__ src,
                               const int* __restrict__ perm, int ne, int kk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  const int a = ptr[i], b = ptr[i + 1];
  for (int j = a + 1; j < b; j++) {
    const int v = src[j];
    const long long key = (long long)perm[v / kk] * kk + v % kk;
    int q = j - 1;
    while (q >= a) {
      const int w = src[q];
      if ((long long)perm[w / kk] * kk + w % kk <= key) break;
      src[q + 1] = w;
      q--;
    }
    src[q + 1] = v;
  }
}

static od_status gather_list(Scene* s, const int* dest, int kk, int nd, int** ptr_out, int** src_out) {
  const int ne = s->n_tets;
  cudaStream_t st = s->ctx->stream;
  const long long n = (long long)kk * ne;
  const int grid = std::max(1, (int)std::min<long long>((n + 255) / 256, 64LL * std::max(1, s->ctx->num_sms)));
  // every buffer is freed on an early error return; ptr and src are handed
  // over on success
  struct Bufs {
    int *ptr = nullptr, *sums = nullptr, *cur = nullptr, *src = nullptr;
    ~Bufs() {
      for (int* p : {ptr, sums, cur, src}) cudaFree(p);
    }
  } b;
  int*& ptr = b.ptr;
  int*& sums = b.sums;
  int*& cur = b.cur;
  int*& src = b.src;
  const int nscan = nd + 1, nb = (nscan + kScanBlock - 1) / kScanBlock;
  OD_CUDA(cudaMalloc(&ptr, sizeof(int) * (size_t)nscan));
  OD_CUDA(cudaMalloc(&sums, sizeof(int) * (size_t)nb));
  OD_CUDA(cudaMemsetAsync(ptr, 0, sizeof(int) * (size_t)nscan, st));
  gl_count_kernel<<<grid, 256, 0, st>>>(n, dest, ptr);
  gl_scan_block_kernel<<<nb, kScanBlock, 0, st>>>(nscan, ptr, sums);
  std::vector<int> hs(nb);
  OD_CUDA(cudaMemcpyAsync(hs.data(), sums, sizeof(int) * (size_t)nb, cudaMemcpyDeviceToHost, st));
  OD_TRY(sync_stream(s));
  long long run = 0;
  for (int b = 0; b < nb; b++) {
    const long long t = hs[b];
    hs[b] = (int)run;
    run += t;
  }
  const int total = (int)run;
  OD_CUDA(cudaMemcpyAsync(sums, hs.data(), sizeof(int) * (size_t)nb, cudaMemcpyHostToDevice, st));
  gl_add_kernel<<<nb, kScanBlock, 0, st>>>(nscan, ptr, sums);
  OD_CUDA(cudaMalloc(&src, sizeof(int) * (size_t)std::max(1, total)));
  OD_CUDA(cudaMalloc(&cur, sizeof(int) * (size_t)std::max(1, nd)));
  if (nd > 0) OD_CUDA(cudaMemcpyAsync(cur, ptr, sizeof(int) * (size_t)nd, cudaMemcpyDeviceToDevice, st));
  gl_fill_kernel<<<grid, 256, 0, st>>>(n, dest, cur, src, ne, kk);
  if (nd > 0) gl_sort_kernel<<<(nd + 255) / 256, 256, 0, st>>>(nd, ptr, src, s->perm, ne, kk);
  OD_CUDA(cudaGetLastError());
  OD_TRY(sync_stream(s));   // hs is read by the copy above; the temporaries go next
  s->device_bytes += (long long)sizeof(int) * ((long long)nscan + std::max(1, total));
  *ptr_out = ptr;
  *src_out = src;
  ptr = src = nullptr;
  return OD_OK;
}

od_status build_gather_lists(Scene* s, int n_pad) {
  if (s->n_tets <= 0 || 78LL * s->n_tets >= (long long)INT32_MAX) return OD_OK;
  OD_TRY(gather_list(s, s->emap, 78, s->nvals, &s->gat_kptr, &s->gat_ksrc));
  OD_TRY(gather_list(s, s->gdof, 12, n_pad, &s->gat_fptr, &s->gat_fsrc));
  return OD_OK;
}

// multi-scene gathered assembly: tile j of scene s covers its destinations
// [256 j, 256 j + 256) (K values, then the padded f_int entries)
__global__ void __launch_bounds__(256) gather_batch_kernel(int n_sc, const int* __restrict__ prefix,
                                                           const SceneDev* __restrict__ sd) {
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  gather_one((long long)(blockIdx.x - prefix[s]) * 256 + threadIdx.x, D.nvals, D.gat_kptr, D.gat_ksrc, D.stage_k,
             D.K, D.n_pad, D.gat_fptr, D.gat_fsrc, D.stage_f, D.fint, 0);
}

// zero 4096 K values (which 0) or padded f_int entries (which 1) per tile
__global__ void zero_batch_kernel(int n_sc, const int* __restrict__ prefix, int which,
                                  const SceneDev* __restrict__ sd) {
  const int s = dir_scene(prefix, n_sc, blockIdx.x);
  const SceneDev& D = sd[s];
  double* p = which == 0 ? D.K : D.fint;
  const int n = which == 0 ? D.nvals : D.n_pad;
  const int i0 = (blockIdx.x - prefix[s]) * kZeroTileValues, i1 = min(n, i0 + kZeroTileValues);
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) p[i] = 0.0;
}

// ---------------------------------------------------------------- launches
static inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

od_status launch_precompute(Scene* s) {
  const int T = 128;
  if (s->n_tets == 0) return OD_OK;
  OD_KL(s);
  precompute_kernel<<<nblk(s->n_tets, T), T, 0, s->ctx->stream>>>(s->n_tets, s->tets, s->X, s->pre);
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

// ------------------------------------------------------------ linear (Hooke)
// HookeMaterial::generateStiffnessMatrix (material/hooke.cpp:18-60): per
// element and node pair a <= b the block of LinearIsotropicTetElement::
// generateSubStiffnessMatrix (element/tetelement.cpp:98-116) with the Lame
// coefficients D = (lambda + 2 mu, lambda, mu) (hooke.cpp:6-16), written into
// the colour-ordered staging layout (78 values: the element's 12x12 upper
// triangle by rows) that the assembly sums in element order.
__global__ void hooke_stage_kernel(int ne, const int4* __restrict__ tets, const double* __restrict__ X, double D0,
                                   double D1, double D2, double* __restrict__ k78) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int4 t = tets[e];
  const V3t<double> p0 = ld3(X, t.x), p1 = ld3(X, t.y), p2 = ld3(X, t.z), p3 = ld3(X, t.w);
  // shape-function gradients scaled by 6V, oriented as the precomputes
  const V3t<double> da = v_sub(p0, p3), db = v_sub(p1, p3), dc = v_sub(p2, p3), ca = v_sub(p0, p2),
                    cb = v_sub(p1, p2);
  V3t<double> g[4];
  if (v_dot(da, v_cross(db, dc)) > 0.0) {
    g[0] = v_cross(db, dc); g[1] = v_cross(dc, da); g[2] = v_cross(da, db); g[3] = v_cross(cb, ca);
  } else {
    g[0] = v_cross(dc, db); g[1] = v_cross(da, dc); g[2] = v_cross(db, da); g[3] = v_cross(ca, cb);
  }
  const double f = 1.0 / (36.0 * tet_vol(p0, p1, p2, p3));
  for (int a = 0; a < 4; a++) {
    const double Ba[3] = {g[a].x, g[a].y, g[a].z};
    for (int b = a; b < 4; b++) {
      const double Bb[3] = {g[b].x, g[b].y, g[b].z};
      // K_ab(i, j), row i of node a, column j of node b
      double Kab[9];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
          double v;
          if (i == j) {
            const int j1 = (i + 1) % 3, j2 = (i + 2) % 3;
            const int lo = j1 < j2 ? j1 : j2, hi = j1 < j2 ? j2 : j1;
            v = D0 * Ba[i] * Bb[i] + D2 * (Ba[lo] * Bb[lo] + Ba[hi] * Bb[hi]);
          } else {
            v = D1 * Ba[i] * Bb[j] + D2 * Ba[j] * Bb[i];
          }
          Kab[3 * i + j] = v * f;
        }
      for (int i = 0; i < 3; i++) {
        const int p = 3 * a + i, dp = p * 12 - (p * (p - 1)) / 2;   // packed index of (p, p)
        if (a == b) {
          for (int j = i; j < 3; j++) k78[kst(dp + j - i, e)] = Kab[3 * i + j];
        } else {
          for (int j = 0; j < 3; j++) k78[kst(dp + 3 * b + j - p, e)] = Kab[3 * i + j];
        }
      }
    }
  }
}

od_status launch_hooke(Scene* s, double youngs, double poisson, double* Kh) {
  const int T = 128;
  cudaStream_t st = s->ctx->stream;
  const double lambda = poisson * youngs / ((1.0 + poisson) * (1.0 - 2.0 * poisson));
  const double mu = youngs / (2.0 * (1.0 + poisson));
  OD_CUDA(cudaMemsetAsync(Kh, 0, sizeof(double) * std::max(1, s->nvals), st));
  if (s->n_tets == 0) return OD_OK;
  OD_KL(s);
  hooke_stage_kernel<<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->tets, s->X, lambda + 2.0 * mu, lambda, mu,
                                                      s->stage_k);
  if (s->gat_kptr) {
    if (s->nvals > 0) {
      OD_KL(s);
      gather_kernel<<<nblk(s->nvals, 256), 256, 0, st>>>(s->nvals, s->gat_kptr, s->gat_ksrc, s->stage_k, Kh, 0,
                                                         nullptr, nullptr, nullptr, nullptr, 0);
    }
  } else {
    for (size_t c = 0; c + 1 < s->color_off.size(); c++) {
      const int e0 = s->color_off[c], e1 = s->color_off[c + 1];
      if (e1 <= e0) continue;
      OD_KL(s);
      scatter_kernel<<<nblk(78LL * (e1 - e0), 256), 256, 0, st>>>(e0, e1 - e0, s->n_tets, s->stage_k, nullptr,
                                                                   s->emap, s->gdof, Kh, nullptr);
    }
  }
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

od_status launch_mass(Scene* s) {
  const int T = 128;
  OD_CUDA(cudaMemsetAsync(s->M, 0, sizeof(double) * (size_t)s->nvals, s->ctx->stream));
  OD_CUDA(cudaMemsetAsync(s->node_vol4, 0, sizeof(double) * (size_t)s->n_nodes, s->ctx->stream));
  for (size_t c = 0; c + 1 < s->color_off.size(); c++) {
    int e0 = s->color_off[c], e1 = s->color_off[c + 1];
    if (e1 <= e0) continue;
    OD_KL(s);
    mass_kernel<<<nblk(e1 - e0, T), T, 0, s->ctx->stream>>>(e0, e1, s->n_tets, s->mat.density, s->pre,
                                                             s->emap, s->M);
    OD_KL(s);
    node_vol_kernel<<<nblk(e1 - e0, T), T, 0, s->ctx->stream>>>(e0, e1, s->n_tets, s->tets, s->pre,
                                                                 s->node_vol4);
  }
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

od_status launch_eval(Scene* s, bool zero_first, bool refine, double* host_k, double* host_f) {
  const int T = kElThreads;
  cudaStream_t st = s->ctx->stream;
  if (zero_first && (!s->gat_kptr || s->n_tets == 0)) {
    OD_CUDA(cudaMemsetAsync(s->K, 0, sizeof(double) * (size_t)s->nvals, st));
    OD_CUDA(cudaMemsetAsync(s->fint, 0, sizeof(double) * (size_t)s->pcg.n_pad, st));
  }
  if (s->n_tets == 0) return OD_OK;
  // 1) every element at full occupancy into the colour-ordered staging arrays
  OD_KL(s);
  if (s->mat.kind == OD_MATERIAL_COROTATIONAL_PLASTIC)
    plastic_kernel<2><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->tets, s->X, s->u, s->pre, s->mat.threshold,
                                                         s->lambda, s->mu, s->mat.yield_criterion,
                                                         s->mat.creep_ratio, s->mat.max_plastic_strain, s->plastic,
                                                         s->stage_k, s->stage_f, nullptr);
  else if (s->mat.kind == OD_MATERIAL_COROTATIONAL)
    corot_kernel<2><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->tets, s->X, s->u, s->pre, s->mat.threshold,
                                                      s->lambda, s->mu, s->stage_k, s->stage_f, nullptr);
  else
    invhyper_kernel<2><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->mat.kind == OD_MATERIAL_STVK, s->tets, s->X, s->u,
                                                          s->pre, s->mat.threshold, s->lambda, s->mu, s->stage_k,
                                                          s->stage_f, nullptr, refine);
  // 2) assembly: one gather launch; one scatter launch per colour for meshes
  //    whose gather lists do not fit 32-bit indices
  if (s->gat_kptr) {
    const long long nd = (long long)s->nvals + s->pcg.n_pad;
    if (nd == 0) return OD_OK;
    OD_KL(s);
    gather_kernel<<<nblk(nd, 256), 256, 0, st>>>(s->nvals, s->gat_kptr, s->gat_ksrc, s->stage_k, s->K, s->pcg.n_pad,
                                                 s->gat_fptr, s->gat_fsrc, s->stage_f, s->fint, zero_first ? 0 : 1, host_k, host_f, s->dofs);
    OD_CUDA(cudaGetLastError());
    return OD_OK;
  }
  for (size_t c = 0; c + 1 < s->color_off.size(); c++) {
    int e0 = s->color_off[c], e1 = s->color_off[c + 1];
    if (e1 <= e0) continue;
    OD_KL(s);
    scatter_kernel<<<nblk(90LL * (e1 - e0), 256), 256, 0, st>>>(e0, e1 - e0, s->n_tets, s->stage_k, s->stage_f,
                                                                 s->emap, s->gdof, s->K, s->fint);
  }
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

od_status launch_element_values(Scene* s, double* d_k78, double* d_f12) {
  const int T = kElThreads;
  cudaStream_t st = s->ctx->stream;
  if (s->n_tets == 0) return OD_OK;
  OD_KL(s);
  if (s->mat.kind == OD_MATERIAL_COROTATIONAL_PLASTIC)
    plastic_kernel<1><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->tets, s->X, s->u, s->pre, s->mat.threshold,
                                                         s->lambda, s->mu, s->mat.yield_criterion,
                                                         s->mat.creep_ratio, s->mat.max_plastic_strain, s->plastic,
                                                         d_k78, d_f12, s->perm);
  else if (s->mat.kind == OD_MATERIAL_COROTATIONAL)
    corot_kernel<1><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->tets, s->X, s->u, s->pre, s->mat.threshold,
                                                      s->lambda, s->mu, d_k78, d_f12, s->perm);
  else
    invhyper_kernel<1><<<nblk(s->n_tets, T), T, 0, st>>>(s->n_tets, s->mat.kind == OD_MATERIAL_STVK, s->tets, s->X, s->u,
                                                          s->pre, s->mat.threshold, s->lambda, s->mu, d_k78, d_f12,
                                                          s->perm, false);
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

// every (facet, traction) pair of the scene gets the same traction vector
__global__ void fill_traction_kernel(int n, double tx, double ty, double tz, double* __restrict__ tvec) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    tvec[3 * k] = tx;
    tvec[3 * k + 1] = ty;
    tvec[3 * k + 2] = tz;
  }
}

// New load values on the facet list of the scene's last od_scene_set_loads
// (one traction group): the traction vector is written on the device and
// the external forces re-evaluated, no copy and no synchronisation.
od_status scene_set_uniform_loads(Scene* s, const double* body, const double* traction) {
  if (traction && s->n_trac > 0) {
    OD_KL(s);
    fill_traction_kernel<<<nblk(s->n_trac, 128), 128, 0, s->ctx->stream>>>(s->n_trac, traction[0], traction[1],
                                                                            traction[2], s->trac_vec);
  }
  s->has_body = body != nullptr;
  if (body)
    for (int i = 0; i < 3; i++) s->load_body[i] = body[i];
  return launch_loads(s, body, traction ? s->n_trac : 0, 1.0);
}

// body part then traction colours; s->trac_* hold the colour-ordered facets
od_status launch_loads(Scene* s, const double* body, int n_facets_total, double traction_scale) {
  const int T = 128;
  cudaStream_t st = s->ctx->stream;
  const int n = s->pcg.n_pad;
  if (n <= 0) return OD_OK;
  double b[3] = {0, 0, 0};
  if (body) { b[0] = body[0]; b[1] = body[1]; b[2] = body[2]; }
  const bool trac = n_facets_total > 0 && s->load_ptr;
  OD_KL(s);
  loads_kernel<<<nblk(n, T), T, 0, st>>>(n, s->dofs, s->free_pos, s->node_vol4, b[0], b[1], b[2],
                                         trac ? s->load_ptr : nullptr, s->load_src, s->trac_facets, s->trac_vec,
                                         traction_scale, s->facets_dev, s->X, s->u, s->fext);
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

}  // namespace od

namespace od {

od_status launch_eval_batch(Ctx* ctx, int n_sc, const SceneDev* sd, const TileDir& zero_k, const TileDir& zero_f,
                            const TileDir& corot, const TileDir& inv, const TileDir& plastic,
                            const std::vector<TileDir>& scatter, const TileDir& gather) {
  cudaStream_t st = ctx->stream;
  const bool gathered = gather.tiles >= 0;  // every scene has gather lists
  if (!gathered && zero_k.tiles > 0) {
    ctx->launches++;
    zero_batch_kernel<<<zero_k.tiles, 256, 0, st>>>(n_sc, zero_k.prefix, 0, sd);
  }
  if (!gathered && zero_f.tiles > 0) {
    ctx->launches++;
    zero_batch_kernel<<<zero_f.tiles, 256, 0, st>>>(n_sc, zero_f.prefix, 1, sd);
  }
  if (corot.tiles > 0) {
    ctx->launches++;
    corot_batch_kernel<<<corot.tiles, kElThreads, 0, st>>>(n_sc, corot.prefix, sd);
  }
  if (inv.tiles > 0) {
    ctx->launches++;
    invhyper_batch_kernel<<<inv.tiles, kElThreads, 0, st>>>(n_sc, inv.prefix, sd);
  }
  if (plastic.tiles > 0) {
    ctx->launches++;
    plastic_batch_kernel<<<plastic.tiles, kElThreads, 0, st>>>(n_sc, plastic.prefix, sd);
  }
  if (gathered) {
    if (gather.tiles > 0) {
      ctx->launches++;
      gather_batch_kernel<<<gather.tiles, 256, 0, st>>>(n_sc, gather.prefix, sd);
    }
    OD_CUDA(cudaGetLastError());
    return OD_OK;
  }
  for (size_t c = 0; c < scatter.size(); c++) {
    if (scatter[c].tiles <= 0) continue;
    ctx->launches++;
    scatter_batch_kernel<<<scatter[c].tiles, 256, 0, st>>>(n_sc, scatter[c].prefix, (int)c, sd);
  }
  OD_CUDA(cudaGetLastError());
  return OD_OK;
}

}  // namespace od
