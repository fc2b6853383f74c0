// The TECE edge block (atomic_basis.type = uv_so2): kernels around the SO(2) linears.
//
// Reference: tace/models/_e3nn/archive/oam_2026_07_05.py:547-823 (OAM20260705Convolution), the edge frame of
// tace/models/o2/rotation_matrix.py:74-88, the recursive Wigner matrices of tace/models/o2/wigner.py:231-357 and the
// graph softmax of tace/models/softmax.py:80-114.  Per edge: rotate the features of both ends into the frame whose polar
// (y) axis is the edge, keep the orders |m| <= mmax, weight them with the radial MLP output, run SO(2) linears (GEMMs,
// launched by the engine), gate + edge cluster expansion, attention-weighted inverse rotation and sum per target atom.
//
// Layouts (channel fastest): node features x [N][D][C], D = (L+1)^2; Wigner rows Wg [E][NEP], packed (see below); NR rows in
// order-major layout (m = 0: l = 0..L | +1: l = 1..L | -1 | +2 | -2); Ks / Qt / Kp / Qp / down [E][NR][C]; Mw [E][NR][2C];
// radial weights W [E][NC][2C]; up [E][G + NF][Ca]; glu, U [E][NF][Ca] with NF = n + 2 n mmax, n = L + 1 (every order
// carries n rows there); coef [E][paths][n][Ca]; logit / alpha [E][H].  Edges are sorted by target (CSR rowptr).
//
// The derivative of the Wigner rows with respect to the edge vector runs backwards through the recursion and in forward mode
// (three directional derivatives) through the frame, so no hand-derived adjoint of the quaternion blend exists.
#include <cuda_runtime.h>

#include <type_traits>

#include "kernels.h"
#include "tace_common.cuh"
#include "tace_math.cuh"
#include "tp_gen.cuh"

namespace tace {

namespace {

// ---- forward-mode scalar: value and three partial derivatives ------------------------------------
template <typename T>
struct Dual3 {
  T v, d[3];
};
template <typename T> TACE_D TACE_INLINE Dual3<T> mk(T v) { return {v, {T(0), T(0), T(0)}}; }
template <typename T> TACE_D TACE_INLINE Dual3<T> operator+(Dual3<T> a, Dual3<T> b) { return {a.v + b.v, {a.d[0] + b.d[0], a.d[1] + b.d[1], a.d[2] + b.d[2]}}; }
template <typename T> TACE_D TACE_INLINE Dual3<T> operator-(Dual3<T> a, Dual3<T> b) { return {a.v - b.v, {a.d[0] - b.d[0], a.d[1] - b.d[1], a.d[2] - b.d[2]}}; }
template <typename T> TACE_D TACE_INLINE Dual3<T> operator-(Dual3<T> a) { return {-a.v, {-a.d[0], -a.d[1], -a.d[2]}}; }
template <typename T> TACE_D TACE_INLINE Dual3<T> operator*(Dual3<T> a, Dual3<T> b) {
  return {a.v * b.v, {a.d[0] * b.v + a.v * b.d[0], a.d[1] * b.v + a.v * b.d[1], a.d[2] * b.v + a.v * b.d[2]}};
}
template <typename T> TACE_D TACE_INLINE Dual3<T> operator*(T a, Dual3<T> b) { return {a * b.v, {a * b.d[0], a * b.d[1], a * b.d[2]}}; }
template <typename T> TACE_D TACE_INLINE Dual3<T> operator/(Dual3<T> a, Dual3<T> b) {
  const T inv = T(1) / b.v, q = a.v * inv;
  return {q, {(a.d[0] - q * b.d[0]) * inv, (a.d[1] - q * b.d[1]) * inv, (a.d[2] - q * b.d[2]) * inv}};
}
template <typename T> TACE_D TACE_INLINE Dual3<T> dsqrt(Dual3<T> a) {
  const T r = sqrt(a.v), h = T(0.5) / r;
  return {r, {a.d[0] * h, a.d[1] * h, a.d[2] * h}};
}
template <typename T> TACE_D TACE_INLINE Dual3<T> dexp(Dual3<T> a) {
  const T e = exp(a.v);
  return {e, {a.d[0] * e, a.d[1] * e, a.d[2] * e}};
}
// plain scalars take the same code path
template <typename T> TACE_D TACE_INLINE T mkS(T, T v) { return v; }
template <typename T> TACE_D TACE_INLINE Dual3<T> mkS(Dual3<T>, T v) { return mk<T>(v); }
template <typename T> TACE_D TACE_INLINE T val(T a) { return a; }
template <typename T> TACE_D TACE_INLINE T val(Dual3<T> a) { return a.v; }
TACE_D TACE_INLINE float dsqrt(float a) { return sqrtf(a); }
TACE_D TACE_INLINE double dsqrt(double a) { return sqrt(a); }
TACE_D TACE_INLINE float dexp(float a) { return expf(a); }
TACE_D TACE_INLINE double dexp(double a) { return exp(a); }

template <typename T> struct Eps;
template <> struct Eps<float> { static constexpr float v = 1.1920928955078125e-07f; };
template <> struct Eps<double> { static constexpr double v = 2.220446049250313e-16; };

// tace/models/o2/rotation_matrix.py:74-88: rotation R (row-major [9]) that puts the edge on the y axis.  S = T or Dual3<T>.
template <typename T, typename S>
TACE_D void edge_frame(S vx, S vy, S vz, S (&R)[9]) {
  const T e2 = T(1e-7) * T(1e-7);
  const S zero = mkS(vx, T(0)), one = mkS(vx, T(1)), eps2 = mkS(vx, e2);
  const S nv = dsqrt(vx * vx + vy * vy + vz * vz + eps2);
  const S x = vx / nv, y = vy / nv, z = vz / nv;
  S qp[4] = {one + y, -z, zero, x};
  S qn[4] = {-z, one - y, x, zero};
  const S np_ = dsqrt(qp[0] * qp[0] + qp[1] * qp[1] + qp[2] * qp[2] + qp[3] * qp[3] + eps2);
  const S nn = dsqrt(qn[0] * qn[0] + qn[1] * qn[1] + qn[2] * qn[2] + qn[3] * qn[3] + eps2);
  for (int k = 0; k < 4; ++k) { qp[k] = qp[k] / np_; qn[k] = qn[k] / nn; }
  // C-infinity step in t = (y + 1) / 2 (rotation_matrix.py:25-36); outside (0, 1) it is constant
  const S t = T(0.5) * (y + one);
  S blend;
  if (val(t) <= T(0)) blend = zero;
  else if (val(t) >= T(1)) blend = one;
  else {
    const T eps = Eps<T>::v;
    const S tl = val(t) < eps ? mkS(vx, eps) : t;
    const S tr = val(one - t) < eps ? mkS(vx, eps) : one - t;
    const S left = dexp(-(one / tl)), right = dexp(-(one / tr));
    blend = left / (left + right);
  }
  S dot = qn[0] * qp[0] + qn[1] * qp[1] + qn[2] * qp[2] + qn[3] * qp[3];
  const bool flip = val(dot) < T(0);
  S q[4];
  for (int k = 0; k < 4; ++k) q[k] = (one - blend) * qn[k] + blend * (flip ? -qp[k] : qp[k]);
  const S nq = dsqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3] + eps2);
  for (int k = 0; k < 4; ++k) q[k] = q[k] / nq;
  const S w = q[0], a = q[1], b = q[2], c = q[3];
  const S two = mkS(vx, T(2));
  R[0] = one - two * (b * b + c * c); R[1] = two * (a * b - w * c); R[2] = two * (a * c + w * b);
  R[3] = two * (a * b + w * c); R[4] = one - two * (a * a + c * c); R[5] = two * (b * c - w * a);
  R[6] = two * (a * c - w * b); R[7] = two * (b * c + w * a); R[8] = one - two * (a * a + b * b);
}

template <typename T>
TACE_D TACE_INLINE T act_eval(int kind, T x) { return kind == 0 ? T(1.8467055342154763) * sigmoid_(x) : T(1.6791767923989418) * silu_(x); }
template <typename T>
TACE_D TACE_INLINE T act_grad(int kind, T x) {
  if (kind == 0) { const T s = sigmoid_(x); return T(1.8467055342154763) * s * (T(1) - s); }
  return T(1.6791767923989418) * silu_grad_(x);
}

// ---- compile-time geometry of the order-major rows --------------------------------------------------------------
// Row r of the order-major layout belongs to order m, part (0: +m, 1: -m) and rank l.  The Wigner rows of one edge are kept
// packed: only the 2l + 1 entries of the row's own rank block, in the order (m, l, part) in which for_rows visits the rows,
// padded to a multiple of four entries (72 of them for L = 3, mmax = 2, where full rows would take 14 x 16).
TACE_HD constexpr int row_index(int L, int m, int part, int l) { return (m == 0 ? 0 : m == 1 ? L + 1 : L + 1 + 2 * L) + part * (L + 1 - m) + (l - m); }
TACE_HD constexpr int comp_base(int L, int m) { return m == 0 ? 0 : m == 1 ? L + 1 : 2 * L + 1; }
TACE_HD constexpr int packed_offset(int L, int MM, int m, int part, int l) {
  int k = 0;
  for (int mm = 0; mm <= MM; ++mm)
    for (int ll = mm; ll <= L; ++ll)
      for (int pp = 0; pp < (mm ? 2 : 1); ++pp) {
        if (mm == m && ll == l && pp == part) return k;
        k += 2 * ll + 1;
      }
  return k;  // past the last row: the number of entries
}
template <int L, int MM> struct Rows {
  static constexpr int D = (L + 1) * (L + 1);
  static constexpr int NR = row_index(L, MM, MM ? 1 : 0, L) + 1, NC = comp_base(L, MM) + L + 1 - MM;
  static constexpr int NE = packed_offset(L, MM, MM + 1, 0, 0), NEP = (NE + 3) / 4 * 4;
};
// f(row, rank, weight component, packed offset), every argument a constant after unrolling, so that the per-thread arrays of
// the kernels below are indexed statically and stay in registers
template <int L, int MM, typename F>
TACE_D TACE_INLINE void for_rows(F&& f) {
#pragma unroll
  for (int m = 0; m <= MM; ++m)
#pragma unroll
    for (int l = m; l <= L; ++l)
#pragma unroll
      for (int part = 0; part < (m ? 2 : 1); ++part)
        f(row_index(L, m, part, l), l, comp_base(L, m) + l - m, packed_offset(L, MM, m, part, l));
}

// ---- K0: Wigner rows of every edge ---------------------------------------------------------------
// The recursion of wigner.py:316-357 with the coupling tables folded in at compile time (only the non-zero terms are left:
// 11 of 45 and 23 of 105), one column of the block at a time: T[a][b] = sum_{c, d} cg[c][d][n] R[a][c] D[b][d], then
// D'[m][n] = (2l + 1) sum_{a, b} cg[a][b][m] T[a][b].
template <int LP, typename T>
TACE_D TACE_INLINE T coupling(int a, int b, int m) { return T(LP == 1 ? w3j_1_1_2[(a * 3 + b) * 5 + m] : w3j_1_2_3[(a * 5 + b) * 7 + m]); }
template <int LP, typename T>  // block of rank LP + 1 from the rotation and the block of rank LP
TACE_D TACE_INLINE void wigner_up(const T (&R)[9], const T* Dp, T* Dn) {
  constexpr int np = 2 * LP + 1, nn = 2 * LP + 3;
#pragma unroll
  for (int n = 0; n < nn; ++n) {
    T t[3 * np];
#pragma unroll
    for (int k = 0; k < 3 * np; ++k) t[k] = T(0);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = 0; d < np; ++d) {
        const T w = coupling<LP, T>(c, d, n);
        if (w != T(0)) {
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < np; ++b) t[a * np + b] += (w * R[a * 3 + c]) * Dp[b * np + d];
        }
      }
#pragma unroll
    for (int m = 0; m < nn; ++m) {
      T v = T(0);
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < np; ++b) {
          const T w = coupling<LP, T>(a, b, m);
          if (w != T(0)) v += w * t[a * np + b];
        }
      Dn[m * nn + n] = T(nn) * v;
    }
  }
}
// adjoint of wigner_up: gDn -> += gR, gDp
template <int LP, typename T>
TACE_D TACE_INLINE void wigner_up_bwd(const T (&R)[9], const T* Dp, const T* gDn, T (&gR)[9], T* gDp) {
  constexpr int np = 2 * LP + 1, nn = 2 * LP + 3;
#pragma unroll
  for (int n = 0; n < nn; ++n) {
    T u[3 * np];  // d / d T[a][b]
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < np; ++b) {
        T v = T(0);
#pragma unroll
        for (int m = 0; m < nn; ++m) {
          const T w = coupling<LP, T>(a, b, m);
          if (w != T(0)) v += w * gDn[m * nn + n];
        }
        u[a * np + b] = T(nn) * v;
      }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = 0; d < np; ++d) {
        const T w = coupling<LP, T>(c, d, n);
        if (w != T(0)) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            T v = T(0);
#pragma unroll
            for (int b = 0; b < np; ++b) {
              v += u[a * np + b] * Dp[b * np + d];
              gDp[b * np + d] += (w * R[a * 3 + c]) * u[a * np + b];
            }
            gR[a * 3 + c] += w * v;
          }
        }
      }
  }
}

// One thread per edge; the packed rows leave through shared memory as whole lines.  526 k edges, L = 3, mmax = 2: 0.04 ms,
// against 2.05 ms with run-time recursion loops over local arrays and rows stored entry by entry.
constexpr int kFrameThreads = 64;
template <typename T, int L, int MM>
__global__ void __launch_bounds__(kFrameThreads) tece_wigner_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  __shared__ T st[kFrameThreads * (RW::NEP + 1)];
  const long long e0 = blockIdx.x * (long long)kFrameThreads, e = e0 + threadIdx.x;
  if (e < a.E) {
    T R[9], D2[25], D3[49];
    edge_frame<T, T>(a.vec[3 * e], a.vec[3 * e + 1], a.vec[3 * e + 2], R);
    if (L >= 2) wigner_up<1, T>(R, R, D2);
    if (L >= 3) wigner_up<2, T>(R, D2, D3);
    T* o = st + threadIdx.x * (RW::NEP + 1);
#pragma unroll
    for (int m = 0; m <= MM; ++m)
#pragma unroll
      for (int l = m; l <= L; ++l)
#pragma unroll
        for (int part = 0; part < (m ? 2 : 1); ++part) {
          const int k = packed_offset(L, MM, m, part, l), row = l + (part ? -m : m);
#pragma unroll
          for (int j = 0; j < 2 * l + 1; ++j)
            o[k + j] = l == 0 ? T(1) : l == 1 ? R[(row * 3 + j) % 9] : l == 2 ? D2[(row * 5 + j) % 25] : D3[(row * 7 + j) % 49];
        }
#pragma unroll
    for (int k = RW::NE; k < RW::NEP; ++k) o[k] = T(0);
  }
  __syncthreads();
  const long long left = a.E - e0;
  const int n = (int)(left < kFrameThreads ? left : kFrameThreads) * RW::NEP;
  for (int k = threadIdx.x; k < n; k += kFrameThreads) a.Wg[e0 * RW::NEP + k] = st[k / RW::NEP * (RW::NEP + 1) + k % RW::NEP];
}
// gvec[e][k] (+)= sum over the packed entries of gWg dWg / dv_k: adjoint through the recursion down to the rotation matrix,
// then the three directional derivatives of the frame in forward mode.  gWg comes as one share per group of 32 channels.
// 526 k edges: 0.55 ms, against 1.76 ms with the whole recursion in forward mode.
template <typename T, int L, int MM>
__global__ void __launch_bounds__(kFrameThreads) tece_wigner_bwd_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  __shared__ T st[kFrameThreads * (RW::NEP + 1)];
  const long long e0 = blockIdx.x * (long long)kFrameThreads, e = e0 + threadIdx.x;
  const long long left = a.E - e0;
  const int n = (int)(left < kFrameThreads ? left : kFrameThreads) * RW::NEP, n_col = a.C / 32;
  // eight entries at a time, so that a block waits for one load in eight (8 k edges: 53 -> 30 us)
  constexpr int U = 8;
  for (int k0 = threadIdx.x; k0 < n; k0 += U * kFrameThreads) {
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = T(0);
    for (int q = 0; q < n_col; ++q) {
      const T* p = a.gWg + ((long long)q * a.E + e0) * RW::NEP;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u * kFrameThreads < n) v[u] += p[k0 + u * kFrameThreads];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * kFrameThreads;
      if (k < n) st[k / RW::NEP * (RW::NEP + 1) + k % RW::NEP] = v[u];
    }
  }
  __syncthreads();
  if (e >= a.E) return;
  typedef Dual3<T> S;
  S RD[9];
  const S vx = {a.vec[3 * e], {T(1), T(0), T(0)}}, vy = {a.vec[3 * e + 1], {T(0), T(1), T(0)}}, vz = {a.vec[3 * e + 2], {T(0), T(0), T(1)}};
  edge_frame<T, S>(vx, vy, vz, RD);
  T R[9], gR[9], D2[25], gD2[25], gD3[49];
#pragma unroll
  for (int k = 0; k < 9; ++k) { R[k] = RD[k].v; gR[k] = T(0); }
#pragma unroll
  for (int k = 0; k < 25; ++k) gD2[k] = T(0);
#pragma unroll
  for (int k = 0; k < 49; ++k) gD3[k] = T(0);
  const T* g = st + threadIdx.x * (RW::NEP + 1);
#pragma unroll
  for (int m = 0; m <= MM; ++m)
#pragma unroll
    for (int l = m; l <= L; ++l)
#pragma unroll
      for (int part = 0; part < (m ? 2 : 1); ++part) {
        const int k = packed_offset(L, MM, m, part, l), row = l + (part ? -m : m);
#pragma unroll
        for (int j = 0; j < 2 * l + 1; ++j) {
          if (l == 1) gR[(row * 3 + j) % 9] = g[k + j];
          if (l == 2) gD2[(row * 5 + j) % 25] = g[k + j];
          if (l == 3) gD3[(row * 7 + j) % 49] = g[k + j];
        }
      }
  if (L >= 3) {
    wigner_up<1, T>(R, R, D2);
    wigner_up_bwd<2, T>(R, D2, gD3, gR, gD2);
  }
  if (L >= 2) {
    T gRp[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) gRp[k] = T(0);
    wigner_up_bwd<1, T>(R, R, gD2, gR, gRp);
#pragma unroll
    for (int k = 0; k < 9; ++k) gR[k] += gRp[k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    T v = a.accumulate_gvec ? a.gvec[3 * e + k] : T(0);
#pragma unroll
    for (int q = 0; q < 9; ++q) v += gR[q] * RD[q].d[k];
    a.gvec[3 * e + k] = v;
  }
}

// ---- rotations in and out of the edge frames ---------------------------------------------------------------------
// All four kernels take one block of four warps per (target atom, 32 channels); lane = channel, and the warps share the
// edges into the atom.  What belongs to the target - its features, the gradient of its message, the sums over its edges -
// stays in registers over all of its edges, and the four partial sums meet in shared memory.  Each warp keeps the packed Wigner rows
// of its edge in shared memory, read as broadcasts, while the next edge's are on their way in one coalesced load.
// What bounds them is the memory traffic of the [E][rows][C] buffers.
constexpr int kRotWarps = 4;

template <typename T, int NEP>
struct WigRows {
  static constexpr int Q = NEP * (int)sizeof(T) / 16, PER = (Q + 31) / 32;
  uint4 q[PER];
  TACE_D TACE_INLINE void fetch(const T* __restrict__ Wg, long long e, int lane) {
    const uint4* p = reinterpret_cast<const uint4*>(Wg + e * NEP);
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i * 32 + lane < Q) q[i] = p[i * 32 + lane];
  }
  TACE_D TACE_INLINE void store(T* buf, int lane) const {
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i * 32 + lane < Q) reinterpret_cast<uint4*>(buf)[i * 32 + lane] = q[i];
  }
};
// Largest |element| of the rows that the linears read next, per edge, operand and order (TeceTop): the tensor-core GEMM scales its FP16
// parts by it.  A warp instruction each and one atomic of neighbouring lanes per (edge, 32 channels), beside some 56 stores per lane.
TACE_D TACE_INLINE float larger(float m, float v) { return fmaxf(m, fabsf(v)); }
TACE_D TACE_INLINE double larger(double m, double) { return m; }  // double precision has no use for it
TACE_HD constexpr int row_order(int L, int r) { return r < L + 1 ? 0 : r < L + 1 + 2 * L ? 1 : 2; }
// Where the stage's largest elements of edge e begin
template <int STAGE, typename T>
TACE_D TACE_INLINE unsigned* tops_of(const TeceArgs<T>& a, long long e) { return a.top + STAGE * a.E + e * kTeceTopWidth<STAGE>; }
template <int N>
TACE_D TACE_INLINE void note_tops(unsigned* top, const float (&m)[N]) {  // all lanes of a warp, one edge
  unsigned mine = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(m[j]));
    if ((threadIdx.x & 31) == j) mine = b;
  }
  if ((threadIdx.x & 31) < N) atomicMax(top + (threadIdx.x & 31), mine);
}
template <int N>
TACE_D TACE_INLINE void note_tops(unsigned*, const double (&)[N]) {}
TACE_D TACE_INLINE void note_top_lane(unsigned* top, float m) { atomicMax(top, __float_as_uint(m)); }
TACE_D TACE_INLINE void note_top_lane(unsigned*, double) {}
// where a block of the kernels below works (channel counts are multiples of 32)
struct RotSlot {
  int i, col, c, warp, lane;  // target, group of 32 channels, this lane's channel, warp = share of the edges
  TACE_D TACE_INLINE RotSlot(int C) {
    const int n_col = C / 32;
    i = blockIdx.x / n_col; col = blockIdx.x - i * n_col;
    warp = threadIdx.x >> 5; lane = threadIdx.x & 31;
    c = col * 32 + lane;
  }
};
// the D sums of the four warps added up and written (or added) to out[j * C]
template <typename T, int D>
TACE_D TACE_INLINE void reduce_warps(const T (&acc)[D], T (*red)[D][32], const RotSlot& s, T* out, int C) {
  if (s.warp > 0)
#pragma unroll
    for (int j = 0; j < D; ++j) red[s.warp - 1][j][s.lane] = acc[j];
  __syncthreads();
  if (s.warp == 0)
#pragma unroll
    for (int j = 0; j < D; ++j) out[(long long)j * C] = ((acc[j] + red[0][j][s.lane]) + red[1][j][s.lane]) + red[2][j][s.lane];
}

// Rows of an edge on their way into shared memory: ROWS rows of 32 channels, C apart, 16 bytes per lane (with one element per
// lane the copies fill the queue they share with the stores of the previous edge: 4.5 instead of 3.4 ms for tece_rotate_in_kernel,
// 8.7 instead of 5.8 ms for its backward, at the size below)
TACE_D TACE_INLINE void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <int ROWS, typename T>
TACE_D TACE_INLINE void copy_rows(T* dst, const T* src, int C, int lane) {
  constexpr int V = 16 / (int)sizeof(T), LR = 32 / V, RI = 32 / LR;  // elements per lane, lanes per row, rows per instruction
  const int r0 = lane / LR, v = lane % LR * V;
#pragma unroll
  for (int r = 0; r < ROWS; r += RI)
    if (r + RI <= ROWS || r + r0 < ROWS) copy_async16(dst + (r + r0) * 32 + v, src + (long long)(r + r0) * C + v);
}
TACE_D TACE_INLINE void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
TACE_D TACE_INLINE void copy_wait_all_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// K1: both ends into the frame, radial weighting.  The source's features and the radial weights of the next edge travel while
// this edge's rows are formed: loads placed between the 56 stores of an edge would each wait out their latency.  526 k edges, 128 channels: 3.4 ms
// (5.9 TB/s), against 4.5 ms with a thread per (edge, channel).
template <typename T, int L, int MM> struct RotIn { static constexpr int kRows = 2 * Rows<L, MM>::NC + Rows<L, MM>::D; };
template <typename T, int L, int MM>
__global__ void __launch_bounds__(kRotWarps * 32) tece_rotate_in_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  constexpr int D = RW::D, NR = RW::NR, NC = RW::NC, kRows = RotIn<T, L, MM>::kRows;
  extern __shared__ __align__(16) unsigned char rot_smem[];
  const RotSlot s(a.C);
  const int C = a.C, c = s.c, e1 = a.rowptr[s.i + 1];
  int e = a.rowptr[s.i] + s.warp;
  if (e >= e1) return;
  T* wbuf = reinterpret_cast<T*>(rot_smem) + s.warp * 2 * RW::NEP;
  T* stage = reinterpret_cast<T*>(rot_smem) + kRotWarps * 2 * RW::NEP + s.warp * 2 * kRows * 32;
  auto load = [&](int e, int src, T* st) {
    copy_rows<2 * NC>(st, a.W + (long long)e * NC * 2 * C + s.col * 32, C, s.lane);
    copy_rows<D>(st + 2 * NC * 32, a.x + (long long)src * D * C + s.col * 32, C, s.lane);
  };
  T vt[D], vs[D];
#pragma unroll
  for (int j = 0; j < D; ++j) vt[j] = a.x[((long long)s.i * D + j) * C + c];
  WigRows<T, RW::NEP> wq;
  load(e, a.e_src[e], stage);
  copy_commit();
  wq.fetch(a.Wg, e, s.lane);
  int src = e + kRotWarps < e1 ? a.e_src[e + kRotWarps] : 0;
  for (int b = 0; e < e1; e += kRotWarps, b ^= 1) {
    T* w = wbuf + b * RW::NEP;
    const T* st = stage + b * kRows * 32 + s.lane;
    wq.store(w, s.lane);
    __syncwarp();  // the other stage has been read by every lane
    if (e + kRotWarps < e1) {
      load(e + kRotWarps, src, stage + (b ^ 1) * kRows * 32);
      wq.fetch(a.Wg, e + kRotWarps, s.lane);
      if (e + 2 * kRotWarps < e1) src = a.e_src[e + 2 * kRotWarps];
    }
    copy_commit();
    copy_wait_all_but_last();
    __syncwarp();
#pragma unroll
    for (int j = 0; j < D; ++j) vs[j] = st[(2 * NC + j) * 32];
    T top[6] = {T(0), T(0), T(0), T(0), T(0), T(0)}, top_w[3] = {T(0), T(0), T(0)};
    for_rows<L, MM>([&](int r, int l, int comp, int k) {
      T ks = T(0), qt = T(0);
#pragma unroll
      for (int j = 0; j < 2 * l + 1; ++j) {
        ks += w[k + j] * vs[l * l + j];
        qt += w[k + j] * vt[l * l + j];
      }
      const T ws = st[comp * 2 * 32], wt = st[(comp * 2 + 1) * 32];
      const long long at = (long long)e * NR + r;
      a.Ks[at * C + c] = ks;
      a.Qt[at * C + c] = qt;
      a.Mw[at * 2 * C + c] = ws * ks;
      a.Mw[at * 2 * C + C + c] = wt * qt;
      const int m = row_order(L, r);
      top[m] = larger(top[m], ks);
      top[3 + m] = larger(top[3 + m], qt);
      top_w[m] = larger(larger(top_w[m], ws * ks), wt * qt);
    });
    if (a.top) {
      note_tops(tops_of<TECE_TOP_IN>(a, e), top);
      note_tops(tops_of<TECE_TOP_MW>(a, e), top_w);
    }
  }
}

// Backward of K1.  gKs / gQt hold the gradients that came through the key / query projections, gMw the one through the weighted
// features.  Writes dW (over W), the per-edge source rows dxe, the target's own gradient (to gx, before the source rows are
// added) and the gradient of the packed Wigner rows, one share per group of 32 channels:
//   gWg[row][j] = sum_c ( gKs_total x[source][j] + gQt_total x[target][j] + alpha scale gM[target][j] down[row] ).
// Ks and Qt are rotated again from x rather than read, and neither the totals nor per-edge target rows go to memory: 122
// rows of C per edge are left of the 238 that separate kernels for the rotation, the target sum and the Wigner gradient moved.
// All rows of the next edge (104 for L = 3, mmax = 2: 13 KB per warp) travel while this one is worked on; two blocks per SM keep 100 KB in flight.
// 526 k edges, L = 3, mmax = 2, 128 channels: 5.8 ms (6.5 TB/s), against 11.5 + 0.8 + 4.3 ms as those three kernels.
template <typename T, int L, int MM> struct RotInBwd { static constexpr int kRows = 5 * Rows<L, MM>::NR + 2 * Rows<L, MM>::NC + Rows<L, MM>::D; };
template <typename T, int L, int MM>
__global__ void __launch_bounds__(kRotWarps * 32, sizeof(T) == 4 ? 2 : 1) tece_rotate_in_bwd_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  constexpr int D = RW::D, NR = RW::NR, NC = RW::NC, NE = RW::NE, NEP = RW::NEP, kRows = RotInBwd<T, L, MM>::kRows;
  constexpr int kKs = 2 * NR, kQt = 3 * NR, kDn = 4 * NR, kW = 5 * NR, kX = 5 * NR + 2 * NC;  // first rows of a stage's parts (gMw first)
  extern __shared__ __align__(16) unsigned char rot_smem[];
  T* const smem = reinterpret_cast<T*>(rot_smem);
  const RotSlot s(a.C);
  const int C = a.C, c = s.c;
  const bool owned = s.i < a.n_local;  // ghost atoms have no incoming edges: their gradient starts at zero
  const int e1 = owned ? a.rowptr[s.i + 1] : 0;
  int e = owned ? a.rowptr[s.i] + s.warp : 0;
  T gt[D];
#pragma unroll
  for (int j = 0; j < D; ++j) gt[j] = T(0);
  if (e < e1) {
    const int h = c / (C / a.H);
    T* wbuf = smem + s.warp * 2 * NEP;
    T* stage = smem + kRotWarps * 2 * NEP + s.warp * 2 * kRows * 32;
      auto load = [&](int e, int src, T* st) {
      const long long at = (long long)e * NR * C + s.col * 32;
      copy_rows<2 * NR>(st, a.gMw + (long long)e * NR * 2 * C + s.col * 32, C, s.lane);
      copy_rows<NR>(st + kKs * 32, a.gKs + at, C, s.lane);
      copy_rows<NR>(st + kQt * 32, a.gQt + at, C, s.lane);
      copy_rows<NR>(st + kDn * 32, a.down + at, C, s.lane);
      copy_rows<2 * NC>(st + kW * 32, a.W + (long long)e * NC * 2 * C + s.col * 32, C, s.lane);
      copy_rows<D>(st + kX * 32, a.x + (long long)src * D * C + s.col * 32, C, s.lane);
    };
    T vt[D], vg[D], vs[D], gs[D];
#pragma unroll
    for (int j = 0; j < D; ++j) {
      vt[j] = a.x[((long long)s.i * D + j) * C + c];
      vg[j] = a.gM[((long long)s.i * D + j) * C + c];
    }
    WigRows<T, NEP> wq;
    load(e, a.e_src[e], stage);
    copy_commit();
    wq.fetch(a.Wg, e, s.lane);
    int src = e + kRotWarps < e1 ? a.e_src[e + kRotWarps] : 0;
    T al = a.alpha[(long long)e * a.H + h], al_next = al;
    for (int b = 0; e < e1; e += kRotWarps, b ^= 1, al = al_next) {
      T* w = wbuf + b * NEP;
      const T* st = stage + b * kRows * 32 + s.lane;
      wq.store(w, s.lane);
      __syncwarp();  // the other stage has been read by every lane
      if (e + kRotWarps < e1) {
        load(e + kRotWarps, src, stage + (b ^ 1) * kRows * 32);
        wq.fetch(a.Wg, e + kRotWarps, s.lane);
        al_next = a.alpha[(long long)(e + kRotWarps) * a.H + h];
        if (e + 2 * kRotWarps < e1) src = a.e_src[e + 2 * kRotWarps];
      }
      copy_commit();
      copy_wait_all_but_last();
      __syncwarp();
#pragma unroll
      for (int j = 0; j < D; ++j) { vs[j] = st[(kX + j) * 32]; gs[j] = T(0); }
      T* W = a.W + (long long)e * NC * 2 * C + c;
      T* gw = a.gWg + ((long long)s.col * a.E + e) * NEP;
      T buf[16];
      T ws = T(0), wt = T(0), dws = T(0), dwt = T(0);
      int comp_now = -1;
      for_rows<L, MM>([&](int r, int l, int comp, int k) {
        if (comp != comp_now) {
          if (comp_now >= 0) { W[comp_now * 2 * C] = dws; W[comp_now * 2 * C + C] = dwt; }
          comp_now = comp;
          ws = st[(kW + comp * 2) * 32]; wt = st[(kW + comp * 2 + 1) * 32]; dws = T(0); dwt = T(0);
        }
        const T gms = st[2 * r * 32], gmt = st[(2 * r + 1) * 32];
        const T gks = st[(kKs + r) * 32] + ws * gms, gqt = st[(kQt + r) * 32] + wt * gmt;
        const T dn = al * a.row_scale[r] * st[(kDn + r) * 32];
        T ks = T(0), qt = T(0);
#pragma unroll
        for (int j = 0; j < 2 * l + 1; ++j) {
          const int q = l * l + j;
          const T wv = w[k + j];
          ks += wv * vs[q];
          qt += wv * vt[q];
          gs[q] += wv * gks;
          gt[q] += wv * gqt;
          // sum over the lanes of 16 entries at a time: every exchange halves the entries a lane still carries
          buf[(k + j) & 15] = gks * vs[q] + gqt * vt[q] + dn * vg[q];
          if (((k + j) & 15) == 15 || k + j == NE - 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (i > ((k + j) & 15)) buf[i] = T(0);
#pragma unroll
            for (int o = 16, n = 8; o >= 2; o >>= 1, n >>= 1)
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (i < n) {
                  const bool up = s.lane & o;
                  const T send = up ? buf[i] : buf[i + n];
                  buf[i] = (up ? buf[i + n] : buf[i]) + __shfl_xor_sync(0xffffffffu, send, o);
                }
            buf[0] += __shfl_xor_sync(0xffffffffu, buf[0], 1);
            const int at0 = ((k + j) & ~15) + (s.lane >> 1);
            if (!(s.lane & 1) && at0 < NEP) gw[at0] = buf[0];
          }
        }
        dws += gms * ks;
        dwt += gmt * qt;
      });
      W[comp_now * 2 * C] = dws;
      W[comp_now * 2 * C + C] = dwt;
#pragma unroll
      for (int j = 0; j < D; ++j) a.dxe[((long long)e * D + j) * C + c] = gs[j];
    }
  }
  __syncthreads();  // every warp is done with its stages (no copy is in flight): the partial sums take their place
  reduce_warps<T, D>(gt, reinterpret_cast<T(*)[D][32]>(smem), s, a.gx + (long long)s.i * D * C + c, C);
}

// K6: attention-weighted inverse rotation and sum per target atom.  526 k edges, 128 channels: 0.66 ms (5.7 TB/s), against 2.0 ms
// with one thread walking all edges of its (target, channel); 8 k edges: 16 against 316 us.
template <typename T, int L, int MM>
__global__ void __launch_bounds__(kRotWarps * 32) tece_rotate_out_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  constexpr int D = RW::D, NR = RW::NR;
  __shared__ __align__(16) T wbuf[kRotWarps][2][RW::NEP];
  __shared__ T red[kRotWarps - 1][D][32];
  const RotSlot s(a.C);
  const int C = a.C, c = s.c, h = c / (C / a.H), e1 = a.rowptr[s.i + 1];
  int e = a.rowptr[s.i] + s.warp;
  const T* __restrict__ down = a.down;
  T acc[D];
#pragma unroll
  for (int j = 0; j < D; ++j) acc[j] = T(0);
  WigRows<T, RW::NEP> wq;
  if (e < e1) wq.fetch(a.Wg, e, s.lane);
  for (int b = 0; e < e1; e += kRotWarps, b ^= 1) {
    T* w = wbuf[s.warp][b];
    wq.store(w, s.lane);
    const T al = a.alpha[(long long)e * a.H + h];
    const T* dn = down + (long long)e * NR * C + c;
    T v[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = dn[(long long)r * C];
    __syncwarp();
    if (e + kRotWarps < e1) wq.fetch(a.Wg, e + kRotWarps, s.lane);
    for_rows<L, MM>([&](int r, int l, int, int k) {
      const T t = al * a.row_scale[r] * v[r];
#pragma unroll
      for (int j = 0; j < 2 * l + 1; ++j) acc[l * l + j] += w[k + j] * t;
    });
  }
  reduce_warps<T, D>(acc, red, s, a.M + (long long)s.i * D * C + c, C);
}
// gdown[e][r][c] = alpha scale_r sum_j Wg[r][j] gM[target][j][c] and galpha[e][h] = sum over the head's channels and the rows
// of down scale_r t.  Heads whose channels are a power of two of neighbouring lanes finish galpha with shuffles (FUSE); other
// heads leave it to tece_alpha_bwd_kernel, which gets the sums per channel in row 0 of the edge's gQp (written only later).  526 k edges, 128 channels:
// 1.2 ms (6.2 TB/s), against 5.2 ms with the target's rows read again for every edge.
template <typename T, int L, int MM, bool FUSE>
__global__ void __launch_bounds__(kRotWarps * 32) tece_rotate_out_bwd_kernel(const TeceArgs<T> a) {
  typedef Rows<L, MM> RW;
  constexpr int D = RW::D, NR = RW::NR;
  __shared__ __align__(16) T wbuf[kRotWarps][2][RW::NEP];
  const RotSlot s(a.C);
  const int C = a.C, c = s.c, Ch = C / a.H, h = c / Ch, e1 = a.rowptr[s.i + 1];
  int e = a.rowptr[s.i] + s.warp;
  if (e >= e1) return;
  const T* __restrict__ down = a.down;
  T vg[D];
#pragma unroll
  for (int j = 0; j < D; ++j) vg[j] = a.gM[((long long)s.i * D + j) * C + c];
  WigRows<T, RW::NEP> wq;
  wq.fetch(a.Wg, e, s.lane);
  for (int b = 0; e < e1; e += kRotWarps, b ^= 1) {
    T* w = wbuf[s.warp][b];
    wq.store(w, s.lane);
    const T al = a.alpha[(long long)e * a.H + h];
    const T* dn = down + (long long)e * NR * C + c;
    T v[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = dn[(long long)r * C];
    __syncwarp();
    if (e + kRotWarps < e1) wq.fetch(a.Wg, e + kRotWarps, s.lane);
    T part = T(0), top[3] = {T(0), T(0), T(0)};
    for_rows<L, MM>([&](int r, int l, int, int k) {
      T t = T(0);
#pragma unroll
      for (int j = 0; j < 2 * l + 1; ++j) t += w[k + j] * vg[l * l + j];
      t *= a.row_scale[r];
      a.gdown[((long long)e * NR + r) * C + c] = al * t;
      top[row_order(L, r)] = larger(top[row_order(L, r)], al * t);
      part += v[r] * t;
    });
    if (a.top) note_tops(tops_of<TECE_TOP_DOWN>(a, e), top);
    if (FUSE) {
      for (int o = Ch >> 1; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if (s.lane % Ch == 0) a.galpha[(long long)e * a.H + h] = part;
    } else {
      a.gQp[(long long)e * NR * C + c] = part;
    }
  }
}
// galpha[e][h] from the per-channel sums that tece_rotate_out_bwd_kernel left in row 0 of the edge's gQp
template <typename T>
__global__ void tece_alpha_bwd_kernel(const TeceArgs<T> a) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= a.E * a.H) return;
  const long long e = idx / a.H;
  const int h = (int)(idx - e * a.H), Ch = a.C / a.H;
  const T* p = a.gQp + e * a.NR * a.C + h * Ch;
  T acc = T(0);
  for (int u = 0; u < Ch; ++u) acc += p[u];
  a.galpha[idx] = acc;
}

// ---- K3: attention logits ---------------------------------------------------------------------------
template <typename T>
TACE_D void radial_projection(const TeceArgs<T>& a, T d, T* proj, T* dproj) {  // proj[2H], dproj = d proj / d d (or nullptr)
  T b[kNumBessel], db[kNumBessel];
  radial_eval<T>(d, a.rp, b, db);
  for (int j = 0; j < 2 * a.H; ++j) {
    T v = a.rproj_b[j], dv = T(0);
    for (int k = 0; k < kNumBessel; ++k) { v += b[k] * a.rproj_w[k * 2 * a.H + j]; dv += db[k] * a.rproj_w[k * 2 * a.H + j]; }
    proj[j] = v;
    if (dproj) dproj[j] = dv;
  }
}
template <typename T>
__global__ void tece_logit_kernel(const TeceArgs<T> a) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= a.E * a.H) return;
  const long long e = idx / a.H;
  const int h = (int)(idx - e * a.H), C = a.C, Ch = C / a.H, n0 = a.L + 1;
  T proj[32];
  radial_projection(a, a.dlen[e], proj, (T*)nullptr);
  const T phase = T(3.141592653589793) * tanh(proj[a.H + h]);
  const T* q = a.Qp + e * a.NR * C + h * Ch;
  const T* k = a.Kp + e * a.NR * C + h * Ch;
  T score = T(0);
  for (int r = 0; r < n0; ++r)
    for (int u = 0; u < Ch; ++u) score += q[r * C + u] * k[r * C + u];
  int off = n0;
  for (int m = 1; m <= a.mmax; ++m) {
    const int n = a.L + 1 - m;
    const T cs = cos(T(m) * phase), sn = sin(T(m) * phase);
    for (int r = 0; r < n; ++r)
      for (int u = 0; u < Ch; ++u) {
        const T kr = k[(off + r) * C + u], ki = k[(off + n + r) * C + u];
        score += q[(off + r) * C + u] * (cs * kr - sn * ki) + q[(off + n + r) * C + u] * (sn * kr + cs * ki);
      }
    off += 2 * n;
  }
  a.logit[idx] = score * a.temp[h] + proj[h];
}
// gQp / gKp from glogit; gproj[e][2H] = d E / d (radial projection)
template <typename T>
__global__ void tece_logit_bwd_kernel(const TeceArgs<T> a) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= a.E * a.H) return;
  const long long e = idx / a.H;
  const int h = (int)(idx - e * a.H), C = a.C, Ch = C / a.H, n0 = a.L + 1;
  T proj[32];
  radial_projection(a, a.dlen[e], proj, (T*)nullptr);
  const T th = tanh(proj[a.H + h]);
  const T phase = T(3.141592653589793) * th;
  const T gl = a.glogit[idx], gs = gl * a.temp[h];
  const T* q = a.Qp + e * a.NR * C + h * Ch;
  const T* k = a.Kp + e * a.NR * C + h * Ch;
  T* gq = a.gQp + e * a.NR * C + h * Ch;
  T* gk = a.gKp + e * a.NR * C + h * Ch;
  for (int r = 0; r < n0; ++r)
    for (int u = 0; u < Ch; ++u) { gq[r * C + u] = gs * k[r * C + u]; gk[r * C + u] = gs * q[r * C + u]; }
  int off = n0;
  T gphase = T(0), top_q = T(0), top_k = T(0);
  auto note = [&](int m) {
    if (!a.top) return;
    note_top_lane(tops_of<TECE_TOP_GPROJ>(a, e) + m, top_k);
    note_top_lane(tops_of<TECE_TOP_GPROJ>(a, e) + 3 + m, top_q);
    top_q = top_k = T(0);
  };
  for (int r = 0; r < n0; ++r)
    for (int u = 0; u < Ch; ++u) { top_q = larger(top_q, gq[r * C + u]); top_k = larger(top_k, gk[r * C + u]); }
  note(0);
  for (int m = 1; m <= a.mmax; ++m) {
    const int n = a.L + 1 - m;
    const T cs = cos(T(m) * phase), sn = sin(T(m) * phase);
    for (int r = 0; r < n; ++r)
      for (int u = 0; u < Ch; ++u) {
        const int ir = (off + r) * C + u, ii = (off + n + r) * C + u;
        const T kr = k[ir], ki = k[ii], qr = q[ir], qi = q[ii];
        gq[ir] = gs * (cs * kr - sn * ki);
        gq[ii] = gs * (sn * kr + cs * ki);
        gk[ir] = gs * (cs * qr + sn * qi);
        gk[ii] = gs * (-sn * qr + cs * qi);
        top_q = larger(larger(top_q, gq[ir]), gq[ii]);
        top_k = larger(larger(top_k, gk[ir]), gk[ii]);
        // d score / d (m phase) = qr (-sn kr - cs ki) + qi (cs kr - sn ki)
        gphase += gs * T(m) * (qr * (-sn * kr - cs * ki) + qi * (cs * kr - sn * ki));
      }
    note(m);
    off += 2 * n;
  }
  a.gproj[e * 2 * a.H + h] = gl;
  a.gproj[e * 2 * a.H + a.H + h] = gphase * T(3.141592653589793) * (T(1) - th * th);
}
// Lane-per-channel forms of the two kernels above, for head widths that are a power of two <= 32: thread (e, c) handles the
// channel's share of the dot products (contiguous loads), the head's lanes reduce with shuffles, the radial projection is
// read from proj [E][2H] (tece_proj_kernel).  Bound by memory: a thread has all its 2 NR elements in flight before it evaluates the
// rotation, whose two orders neighbouring lanes evaluate for each other.  526 k edges, L = 3, mmax = 2, 128 channels, both with loads
// inside run-time loops and every lane evaluating both orders before: forward 1.79 -> 1.29 ms (5.9 TB/s), backward 3.36 -> 2.22 (6.8 TB/s).
template <typename T>
__global__ void tece_proj_kernel(const TeceArgs<T> a) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= a.E) return;
  T proj[32];
  radial_projection(a, a.dlen[e], proj, (T*)nullptr);
  for (int j = 0; j < 2 * a.H; ++j) a.proj[e * 2 * a.H + j] = proj[j];
}
template <typename T, int L, int MM, bool BWD>
__global__ void __launch_bounds__(128) tece_logit_lane_kernel(const TeceArgs<T> a) {
  constexpr int NR = Rows<L, MM>::NR, N0 = L + 1;
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= a.E * a.C) return;
  const long long e = idx / a.C;
  const int c = (int)(idx - e * a.C), C = a.C, Ch = C / a.H, h = c / Ch;
  const T* __restrict__ q = a.Qp + e * NR * C + c;
  const T* __restrict__ k = a.Kp + e * NR * C + c;
  T qv[NR], kv[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) { qv[r] = q[r * C]; kv[r] = k[r * C]; }
  const T th = tanh(a.proj[e * 2 * a.H + a.H + h]);
  const T phase = T(3.141592653589793) * th;
  T cs[3], sn[3];
  if (MM == 2 && Ch > 1) {  // the lanes of a head have the same phase: one order each, the other from the neighbour
    const int odd = c & 1;
    const T own = T(1 + odd) * phase, cm = cos(own), sm = sin(own);
    const T co = __shfl_xor_sync(0xffffffffu, cm, 1), so = __shfl_xor_sync(0xffffffffu, sm, 1);
    cs[1] = odd ? co : cm; sn[1] = odd ? so : sm;
    cs[2] = odd ? cm : co; sn[2] = odd ? sm : so;
  } else {
#pragma unroll
    for (int m = 1; m <= MM; ++m) { cs[m] = cos(T(m) * phase); sn[m] = sin(T(m) * phase); }
  }
  T gs = T(0);
  T* gq = nullptr; T* gk = nullptr;
  if (BWD) { gs = a.glogit[e * a.H + h] * a.temp[h]; gq = a.gQp + e * NR * C + c; gk = a.gKp + e * NR * C + c; }
  T top[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
  T part = T(0);  // forward: the channel's share of the score; backward: of d score / d phase
#pragma unroll
  for (int r = 0; r < N0; ++r) {
    if (!BWD) part += qv[r] * kv[r];
    else { gq[r * C] = gs * kv[r]; gk[r * C] = gs * qv[r]; top[3] = larger(top[3], gs * kv[r]); top[0] = larger(top[0], gs * qv[r]); }
  }
#pragma unroll
  for (int m = 1; m <= MM; ++m) {
    const int n = N0 - m, off = N0 + (m - 1) * (2 * N0 - m);
#pragma unroll
    for (int r = 0; r < n; ++r) {
      const int ir = off + r, ii = off + n + r;
      const T kr = kv[ir], ki = kv[ii], qr = qv[ir], qi = qv[ii];
      if (!BWD) part += qr * (cs[m] * kr - sn[m] * ki) + qi * (sn[m] * kr + cs[m] * ki);
      else {
        const T g0 = gs * (cs[m] * kr - sn[m] * ki), g1 = gs * (sn[m] * kr + cs[m] * ki);
        const T g2 = gs * (cs[m] * qr + sn[m] * qi), g3 = gs * (-sn[m] * qr + cs[m] * qi);
        gq[ir * C] = g0;
        gq[ii * C] = g1;
        gk[ir * C] = g2;
        gk[ii * C] = g3;
        top[3 + m] = larger(larger(top[3 + m], g0), g1);
        top[m] = larger(larger(top[m], g2), g3);
        part += gs * T(m) * (qr * (-sn[m] * kr - cs[m] * ki) + qi * (cs[m] * kr - sn[m] * ki));
      }
    }
  }
  if (BWD && a.top) note_tops(tops_of<TECE_TOP_GPROJ>(a, e), top);
  for (int o = Ch >> 1; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (c % Ch == 0) {
    if (!BWD) a.logit[e * a.H + h] = part * a.temp[h] + a.proj[e * 2 * a.H + h];
    else {
      a.gproj[e * 2 * a.H + h] = a.glogit[e * a.H + h];
      a.gproj[e * 2 * a.H + a.H + h] = part * T(3.141592653589793) * (T(1) - th * th);
    }
  }
}
// ddlen_extra[e] = sum_j gproj[e][j] d proj_j / d d + gcut[e] d envelope / d d
template <typename T>
__global__ void tece_edge_scalar_bwd_kernel(const TeceArgs<T> a) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= a.E) return;
  T proj[32], dproj[32];
  radial_projection(a, a.dlen[e], proj, dproj);
  T acc = T(0);
  for (int j = 0; j < 2 * a.H; ++j) acc += a.gproj[e * 2 * a.H + j] * dproj[j];
  if (a.env) {
    T gc = T(0);
    for (int h = 0; h < a.H; ++h) gc += a.gcut[e * a.H + h];
    T u, du;
    envelope_eval<T>(a.dlen[e], a.rp, u, du);
    acc += gc * du;
  }
  a.ddlen_extra[e] = acc;
}

// ---- K4: softmax over the edges into one atom, per head (softmax.py:97-112) --------------------------
// One warp per atom: lane = (one of 32 / H groups of edges, head), so that a step reads consecutive scores of consecutive edges.  A
// thread per (atom, head) walked some 65 edges three or four times alone: 128 atoms 16.5 -> 8 us, backward 30 -> 16.
template <typename T>
struct SoftmaxLanes {
  int H, G, g, h;
  __device__ __forceinline__ SoftmaxLanes(int heads) : H(heads), G(32 / heads), g((threadIdx.x & 31) / heads), h((threadIdx.x & 31) - g * heads) {}
  // over the groups, in their order; every lane of a head gets the same value (the lanes past the last group one they do not use)
  __device__ __forceinline__ T sum(T v) const {
    T s = T(0);
    for (int k = 0; k < G; ++k) s += __shfl_sync(0xffffffffu, v, k * H + h);
    return s;
  }
  __device__ __forceinline__ T max(T v) const {
    T m = v;
    for (int k = 0; k < G; ++k) m = fmax(m, __shfl_sync(0xffffffffu, v, k * H + h));
    return m;
  }
};
template <typename T, bool BWD>
__global__ void tece_softmax_kernel(const TeceArgs<T> a) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  if (i >= a.n_local) return;  // whole warps
  const int e0 = a.rowptr[i], e1 = a.rowptr[i + 1];
  if (e0 == e1) return;
  const SoftmaxLanes<T> l(a.H);
  const int first = l.g < l.G ? e0 + l.g : e1;
  auto at = [&](int e) { return (long long)e * a.H + l.h; };
  auto cut = [&](int e) { return a.env ? a.env[e] : T(1); };
  T mx = T(-INFINITY);
  for (int e = first; e < e1; e += l.G) mx = fmax(mx, a.logit[at(e)]);
  mx = l.max(mx);
  T sum = T(0);
  for (int e = first; e < e1; e += l.G) sum += exp(a.logit[at(e)] - mx) * cut(e);
  const T inv = T(1) / (l.sum(sum) + T(1e-16));
  if constexpr (!BWD) {
    for (int e = first; e < e1; e += l.G) {
      const T u = cut(e);
      a.alpha[at(e)] = exp(a.logit[at(e)] - mx) * u * inv * u;
    }
  } else {  // galpha -> glogit, gcut.  alpha = s cut, s = p / (S + eps), p = exp(l - max) cut
    T dot = T(0);  // sum_k s_k g_k with g_k = galpha_k cut_k
    for (int e = first; e < e1; e += l.G) {
      const T u = cut(e);
      dot += exp(a.logit[at(e)] - mx) * u * inv * a.galpha[at(e)] * u;
    }
    dot = l.sum(dot);
    for (int e = first; e < e1; e += l.G) {
      const T u = cut(e), ex = exp(a.logit[at(e)] - mx) * inv, s = ex * u, g = a.galpha[at(e)] * u;  // ex: s / cut
      a.glogit[at(e)] = s * (g - dot);
      if (a.env) a.gcut[at(e)] = a.galpha[at(e)] * s + ex * (g - dot);
    }
  }
}

// ---- K5: gate + edge cluster expansion on the SO(2) features ------------------------------------------
// Rows of the full layout: order 0 rows [0, N); order m >= 1 real rows [N + (m-1) 2N, +N), imaginary rows the next N.  Row i of
// every order, its gate and its coefficients meet only one another (gate: oam_2026_07_05.py:301-309, channel-wise layout, order
// m row i scaled by act(gate[(m - start) N + i]); cluster expansion: :417-488, channel-wise products of the complex order
// components), so one thread takes (edge, i, channel): some 25 values in registers where a thread per (edge, channel) held
// 150 and left the machine a third full.  526 k edges, 32 channels: 1.0 + 1.9 ms, against 1.3 + 4.2 ms.
TACE_HD constexpr bool mix_path(int m3, int m1, int m2) { return m1 + m2 == m3 || m1 - m2 == m3; }
TACE_HD constexpr int mix_path_id(int mm, int m3, int m1, int m2) {  // position in the output-order-major list; past the end: their number
  int p = 0;
  for (int q3 = 0; q3 <= mm; ++q3)
    for (int q1 = 0; q1 <= mm; ++q1)
      for (int q2 = 0; q2 <= q1; ++q2) {
        if (!mix_path(q3, q1, q2)) continue;
        if (q3 == m3 && q1 == m1 && q2 == m2) return p;
        ++p;
      }
  return p;
}
template <typename T, int N, int MM, bool GATE_M0, bool BWD>
__global__ void __launch_bounds__(128) tece_mix_kernel(const TeceArgs<T> a) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= a.E * N * a.Ca) return;
  const int Ca = a.Ca;
  const long long ei = idx / Ca, e = ei / N;
  const int ca = (int)(idx - ei * Ca), i = (int)(ei - e * N);
  constexpr int NF = N + 2 * N * MM, G = N * (MM + (GATE_M0 ? 1 : 0)), M = 2 * MM + 1;
  constexpr int START = GATE_M0 ? 0 : 1, NG = MM + 1 - START, NPATH = mix_path_id(MM, MM + 1, 0, 0);
  // component q of the registers: order (q + 1) / 2, real (0, 1, 3) or imaginary (2, 4) part; its row is q N + i
  T x[M], y[M], gz[NG > 0 ? NG : 1], cz[NPATH], out[M], go[M], gx[M], gy[M];
  const long long up = e * (G + NF) * Ca + (long long)i * Ca + ca, full = e * NF * Ca + (long long)i * Ca + ca,
                  path = e * NPATH * N * Ca + (long long)i * Ca + ca;
  const int row = N * Ca;
  constexpr int STAGE = BWD ? TECE_TOP_GMIX : TECE_TOP_MIX, NTOP = kTeceTopWidth<STAGE>;
  T top[NTOP];
#pragma unroll
  for (int j = 0; j < NTOP; ++j) top[j] = T(0);
  // every input is in registers before the first store: the gradients overwrite their forward buffers
#pragma unroll
  for (int q = 0; q < NG; ++q) gz[q] = a.up[up + q * row];
#pragma unroll
  for (int q = 0; q < M; ++q) {
    x[q] = a.up[up + G * Ca + q * row];
    y[q] = a.glu[full + q * row];
    if (BWD) { go[q] = a.gU[full + q * row]; gx[q] = go[q]; gy[q] = T(0); }
    else out[q] = x[q];
  }
#pragma unroll
  for (int p = 0; p < NPATH; ++p) cz[p] = a.coefZ[path + p * row];
#pragma unroll
  for (int m = 0; m <= MM; ++m) {
    if (m < START) {
      if (BWD) gx[0] += go[0] * act_grad<T>(a.act, x[0]);
      else out[0] += act_eval<T>(a.act, x[0]);
    } else {
      const T ag = act_eval<T>(a.act, gz[m - START]);
      T gg = T(0);
#pragma unroll
      for (int q = (m ? 2 * m - 1 : 0); q <= 2 * m; ++q) {
        if (BWD) { gx[q] += go[q] * ag; gg += go[q] * x[q]; }
        else out[q] += ag * x[q];
      }
      if (BWD) {
        const T g = gg * act_grad<T>(a.act, gz[m - START]);
        a.gup[up + (m - START) * row] = g;
        top[0] = larger(top[0], g);
      }
    }
  }
#pragma unroll
  for (int m3 = 0; m3 <= MM; ++m3)
#pragma unroll
    for (int m1 = 0; m1 <= MM; ++m1)
#pragma unroll
      for (int m2 = 0; m2 <= m1; ++m2)
        if (mix_path(m3, m1, m2)) {
          constexpr int kLast = M - 1;
          const int p = mix_path_id(MM, m3, m1, m2);
          const bool sum_mode = (m1 + m2 == m3);
          const int xq = m1 ? 2 * m1 - 1 : 0, yq = m2 ? 2 * m2 - 1 : 0, oq = m3 ? 2 * m3 - 1 : 0;
          const int xi_ = m1 ? 2 * m1 : kLast, yi_ = m2 ? 2 * m2 : kLast, oi_ = m3 ? 2 * m3 : kLast;
          const T sc = a.p_scale[p], w = act_eval<T>(a.act, cz[p]) * sc;
          const T xr = x[xq], xi = m1 ? x[xi_] : T(0), yr = y[yq], yi = m2 ? y[yi_] : T(0);
          const T sg = sum_mode ? T(1) : T(-1);  // sum of the orders: product; difference: product with the conjugate of y
          const T zr = xr * yr - sg * xi * yi, zi = sum_mode ? xr * yi + xi * yr : xi * yr - xr * yi;
          if (!BWD) {
            out[oq] += w * zr;
            if (m3) out[oi_] += w * zi;
          } else {
            const T gr = go[oq], gi = m3 ? go[oi_] : T(0);
            const T g = (gr * zr + gi * zi) * sc * act_grad<T>(a.act, cz[p]);
            a.gcoefZ[path + p * row] = g;
            top[NTOP - 1] = larger(top[NTOP - 1], g);
            const T ar = w * gr, ai = w * gi;
            gx[xq] += ar * yr + sg * ai * yi;
            if (m1) gx[xi_] += -sg * ar * yi + ai * yr;
            gy[yq] += ar * xr + ai * xi;
            if (m2) gy[yi_] += sum_mode ? -ar * xi + ai * xr : ar * xi - ai * xr;
          }
        }
#pragma unroll
  for (int q = 0; q < M; ++q) {
    const int m = (q + 1) / 2;
    if constexpr (BWD) {
      a.gup[up + G * Ca + q * row] = gx[q];
      a.gglu[full + q * row] = gy[q];
      top[m] = larger(top[m], gx[q]);
      top[3 + m] = larger(top[3 + m], gy[q]);
    } else {
      a.U[full + q * row] = out[q];
      top[m] = larger(top[m], out[q]);
    }
  }
  if (a.top) {
    unsigned* at = tops_of<STAGE>(a, e);
    if (Ca % 32 == 0) note_tops(at, top);  // the lanes of a warp share their edge
    else
#pragma unroll
      for (int j = 0; j < NTOP; ++j) note_top_lane(at + j, top[j]);
  }
}

}  // namespace

// f<L, mmax>() for the ranks and orders a model can have (1 <= L <= 3, mmax <= min(L, 2))
template <typename F>
bool rank_dispatch(int L, int mmax, F&& f) {
  switch (L * 4 + mmax) {
    case 4: f(std::integral_constant<int, 1>(), std::integral_constant<int, 0>()); return true;
    case 5: f(std::integral_constant<int, 1>(), std::integral_constant<int, 1>()); return true;
    case 8: f(std::integral_constant<int, 2>(), std::integral_constant<int, 0>()); return true;
    case 9: f(std::integral_constant<int, 2>(), std::integral_constant<int, 1>()); return true;
    case 10: f(std::integral_constant<int, 2>(), std::integral_constant<int, 2>()); return true;
    case 12: f(std::integral_constant<int, 3>(), std::integral_constant<int, 0>()); return true;
    case 13: f(std::integral_constant<int, 3>(), std::integral_constant<int, 1>()); return true;
    case 14: f(std::integral_constant<int, 3>(), std::integral_constant<int, 2>()); return true;
  }
  return false;
}
template <typename K>
bool rot_smem_limit(K* kernel, int bytes) {  // a failure is left for the caller's cudaGetLastError
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}
int tece_wigner_stride(int L, int mmax) {
  int n = 0;
  rank_dispatch(L, mmax, [&](auto l, auto m) { n = Rows<decltype(l)::value, decltype(m)::value>::NEP; });
  return n;
}

template <typename T>
cudaError_t launch_tece(const TeceArgs<T>& a, int stage, cudaStream_t s) {
  if (a.H > 16 || a.C % a.H != 0 || a.C % 32 != 0) return cudaErrorInvalidValue;
  // nothing to launch: stages over atoms need atoms (one without edges still gets its zero message and gradient), every other
  // stage needs edges
  const bool per_atom = stage == TECE_SOFTMAX || stage == TECE_ROTATE_OUT || stage == TECE_SOFTMAX_BWD;
  if (stage == TECE_ROTATE_IN_BWD ? a.n_atoms <= 0 : per_atom ? a.n_local <= 0 : (a.E <= 0 || a.n_local <= 0)) return cudaSuccess;
  const int ch = a.C / a.H, n_col = a.C / 32;
  const bool fuse_alpha = ch <= 32 && (ch & (ch - 1)) == 0;
  auto grid = [](long long count, int block) { return (unsigned)((count + block - 1) / block); };
  const unsigned rot_grid = (unsigned)((long long)a.n_local * n_col);
  constexpr int kRot = kRotWarps * 32;
  bool known = true;
  switch (stage) {
    case TECE_WIGNER:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { tece_wigner_kernel<T, l(), m()><<<grid(a.E, kFrameThreads), kFrameThreads, 0, s>>>(a); });
      break;
    case TECE_ROTATE_IN:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { constexpr int Lc = decltype(l)::value, Mc = decltype(m)::value;
        constexpr int bytes = kRotWarps * 2 * (Rows<Lc, Mc>::NEP + RotIn<T, Lc, Mc>::kRows * 32) * (int)sizeof(T);
        if (rot_smem_limit(tece_rotate_in_kernel<T, Lc, Mc>, bytes)) tece_rotate_in_kernel<T, Lc, Mc><<<rot_grid, kRot, bytes, s>>>(a);
      });
      break;
    case TECE_LOGIT:
      if (fuse_alpha) {
        tece_proj_kernel<T><<<grid(a.E, 128), 128, 0, s>>>(a);
        known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { tece_logit_lane_kernel<T, l(), m(), false><<<grid(a.E * a.C, 128), 128, 0, s>>>(a); });
      } else {
        tece_logit_kernel<T><<<grid(a.E * a.H, 128), 128, 0, s>>>(a);
      }
      break;
    case TECE_SOFTMAX: tece_softmax_kernel<T, false><<<grid((long long)a.n_local * 32, 128), 128, 0, s>>>(a); break;
    case TECE_MIX:
    case TECE_MIX_BWD:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) {
        constexpr int N = decltype(l)::value + 1, MM = decltype(m)::value;
        const unsigned g = grid(a.E * N * a.Ca, 128);
        if (stage == TECE_MIX) {
          if (a.gate_m0) tece_mix_kernel<T, N, MM, true, false><<<g, 128, 0, s>>>(a);
          else tece_mix_kernel<T, N, MM, false, false><<<g, 128, 0, s>>>(a);
        } else {
          if (a.gate_m0) tece_mix_kernel<T, N, MM, true, true><<<g, 128, 0, s>>>(a);
          else tece_mix_kernel<T, N, MM, false, true><<<g, 128, 0, s>>>(a);
        }
      });
      break;
    case TECE_ROTATE_OUT:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { tece_rotate_out_kernel<T, l(), m()><<<rot_grid, kRot, 0, s>>>(a); });
      break;
    case TECE_ROTATE_OUT_BWD:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) {
        if (fuse_alpha) tece_rotate_out_bwd_kernel<T, l(), m(), true><<<rot_grid, kRot, 0, s>>>(a);
        else tece_rotate_out_bwd_kernel<T, l(), m(), false><<<rot_grid, kRot, 0, s>>>(a);
      });
      break;
    case TECE_ALPHA_BWD:  // already done by the fused kernel above when the head width allows it
      if (!fuse_alpha) tece_alpha_bwd_kernel<T><<<grid(a.E * a.H, 128), 128, 0, s>>>(a);
      break;
    case TECE_SOFTMAX_BWD: tece_softmax_kernel<T, true><<<grid((long long)a.n_local * 32, 128), 128, 0, s>>>(a); break;
    case TECE_LOGIT_BWD:
      if (fuse_alpha) known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { tece_logit_lane_kernel<T, l(), m(), true><<<grid(a.E * a.C, 128), 128, 0, s>>>(a); });
      else tece_logit_bwd_kernel<T><<<grid(a.E * a.H, 128), 128, 0, s>>>(a);
      break;
    case TECE_EDGE_SCALAR_BWD: tece_edge_scalar_bwd_kernel<T><<<grid(a.E, 128), 128, 0, s>>>(a); break;
    case TECE_ROTATE_IN_BWD:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) {
        constexpr int Lc = decltype(l)::value, Mc = decltype(m)::value;
        constexpr int bytes = kRotWarps * 2 * (Rows<Lc, Mc>::NEP + RotInBwd<T, Lc, Mc>::kRows * 32) * (int)sizeof(T);
        if (rot_smem_limit(tece_rotate_in_bwd_kernel<T, Lc, Mc>, bytes))
          tece_rotate_in_bwd_kernel<T, Lc, Mc><<<(unsigned)((long long)a.n_atoms * n_col), kRot, bytes, s>>>(a);
      });
      break;
    case TECE_WIGNER_BWD:
      known = rank_dispatch(a.L, a.mmax, [&](auto l, auto m) { tece_wigner_bwd_kernel<T, l(), m()><<<grid(a.E, kFrameThreads), kFrameThreads, 0, s>>>(a); });
      break;
    default: known = false;
  }
  return known ? cudaGetLastError() : cudaErrorInvalidValue;
}

template cudaError_t launch_tece<float>(const TeceArgs<float>&, int, cudaStream_t);
template cudaError_t launch_tece<double>(const TeceArgs<double>&, int, cudaStream_t);

}  // namespace tace
