// Split-axis Riemann fluxes and thermodynamics of the density-based path.
//
// T = double compiled without FMA contraction (kernels_exact.cu) rounds
// every operation in the order the reference evaluates it, so the face
// fluxes are bit-identical to the reference's:
//   work/FUNCTION.cpp:3-15            getP / getht (2D momentum only)
//   rhoSolver/SolverAusm.cpp:3-26, :53-63, :105-143   AUSM+
//   rhoSolver/SolverRoe.cpp:3-16, :70-111, :114-123   Roe, |A| = R|L|R^-1
// The same code compiled with FMA (kernels_fast.cu) gives the FP64 and
// FP32 production variants.
#pragma once
#include <cuda_runtime.h>

namespace mst {

template <class T>
struct Gas {
  // gamma = 1.4 is fixed by the reference (CONST.h:41)
  static __host__ __device__ __forceinline__ T gamma() { return T(1.4); }
  static __host__ __device__ __forceinline__ T gm1() { return T(1.4) - T(1); }
  static __host__ __device__ __forceinline__ T gp1() { return T(1.4) + T(1); }
};

// x / y of the exact path.  A zero numerator -- a velocity component that
// vanishes, as in the reference's initial field -- takes the slow path of the
// FP64 division (1,500 cycles a warp instead of 560); its quotient by a
// normal number is a zero of the quotient's sign.
template <class T>
__host__ __device__ __forceinline__ T ediv(T x, T y) {
  return x / y;
}
#ifdef __CUDA_ARCH__
template <>
__device__ __forceinline__ double ediv<double>(double x, double y) {
  const int hx = __double2hiint(x), hy = __double2hiint(y), ey = (hy >> 20) & 0x7ff;
  if (((hx & 0x7fffffff) | __double2loint(x)) == 0 && ey != 0 && ey != 0x7ff)
    return __hiloint2double((hx ^ hy) & (int)0x80000000, 0);
  return x / y;
}
#endif

template <class T>
__host__ __device__ __forceinline__ T th_p(const T q[4]) {
  T ke = ediv(T(0.5) * (q[1] * q[1] + q[2] * q[2]), q[0]);
  return (q[3] - ke) * Gas<T>::gm1();
}
template <class T>
__host__ __device__ __forceinline__ T th_ht(const T q[4]) {
  T p = th_p(q);
  return (q[3] + p) / q[0];
}

// Per-state quantities of the AUSM+ flux that do not depend on the axis
// (SolverAusm.cpp:6-25 set(), :107-113): pressure, total enthalpy, the
// critical-speed interface estimate a*^2/max(a*,|U|), the true sound speed,
// and the convected vector (rho, rho u, rho v, rho H).  Computing them once
// per face state and reusing them for both axes gives the same values as
// the reference's per-axis recomputation.
template <class T>
struct AusmSide {
  T p, a_face, a_true, fc[4];
};

template <class T>
__host__ __device__ __forceinline__ AusmSide<T> ausm_side(const T q[4]) {
  const T g = Gas<T>::gamma(), gm1 = Gas<T>::gm1(), gp1 = Gas<T>::gp1();
  AusmSide<T> s;
  s.p = th_p(q);
  const T h = (q[3] + s.p) / q[0];
  const T as = sqrt(T(2) * h * gm1 / gp1);
  const T U = sqrt(ediv(ediv(q[1] * q[1] + q[2] * q[2], q[0]), q[0]));
  s.a_face = as * as / (as < U ? U : as);
  s.a_true = sqrt(g * s.p / q[0]);
  s.fc[0] = q[0];
  s.fc[1] = q[1];
  s.fc[2] = q[2];
  s.fc[3] = q[3] + s.p;
  return s;
}

// AUSM+ flux along axis d (0 = x, 1 = y) from the two sides' quantities;
// ql, qr are the states themselves (for the Mach numbers).
template <class T>
__host__ __device__ __forceinline__ void ausm_axis(const T ql[4], const AusmSide<T>& L,
                                                   const T qr[4], const AusmSide<T>& R,
                                                   int d, T f[4]) {
  const T aF = (R.a_face < L.a_face) ? R.a_face : L.a_face;
  const T mL = ediv(ediv(ql[d + 1], ql[0]), aF);
  const T mR = ediv(ediv(qr[d + 1], qr[0]), aF);
  const T pL = L.p, pR = R.p, aL = L.a_true, aR = R.a_true;
  T mp, mm, pp, pm;
  // the reference's abs(mach <= 1) is the plain test mach <= 1
  if (mL <= T(1)) {
    mp = T(0.25) * (mL + T(1)) * (mL + T(1)) +
         T(0.125) * (mL * mL - T(1)) * (mL * mL - T(1));
    pp = pL * T(0.25) * (mL + T(1)) * (mL + T(1)) * (T(2) - mL) +
         T(0.1875) * mL * (mL * mL - T(1)) * (mL * mL - T(1));
  } else {
    mp = T(0.5) * (mL + fabs(mL));
    pp = pL * T(0.5) * (mL + fabs(mL)) / mL;
  }
  if (mR <= T(1)) {
    mm = T(-0.25) * (mR - T(1)) * (mR - T(1)) -
         T(0.125) * (mR * mR - T(1)) * (mR * mR - T(1));
    pm = pR * T(0.25) * (mR - T(1)) * (mR - T(1)) * (T(2) + mR) -
         T(0.1875) * mR * (mR * mR - T(1)) * (mR * mR - T(1));
  } else {
    mm = T(0.5) * (mR - fabs(mR));
    pm = pR * T(0.5) * (mR - fabs(mR)) / mR;
  }
  const T mF = mm + mp;
  const T pF = pm + pp;
  const T amF = fabs(mF);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    T a = mF * (aL * L.fc[k] + aR * R.fc[k]);
    T b = amF * (aR * R.fc[k] - aL * L.fc[k]);
    f[k] = T(0.5) * (a - b);
  }
  f[d + 1] += pF;
}

// 1/sqrt(x) of the production paths: the FP64 one costs 5.5 FP64-pipe
// instructions on this GPU against 9.3 for a square root and 8.8 for a
// division (measured: one FP64 instruction holds an SM sub-partition for 64
// cycles whatever the occupancy), the FP32 one is a single MUFU operation.
__device__ __forceinline__ double inv_sqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float inv_sqrt(float x) { return rsqrtf(x); }

// AUSM+ of both axes of a face for the production paths (FP64 and FP32): the
// formulas of ausm_side / ausm_axis (including the pressure polynomial whose
// second term is not scaled by p) up to rounding, arranged for few divisions
// and no divergence:
//   * per side one reciprocal (1/rho), one reciprocal square root for the
//     interface speed a*^2 / max(a*, |U|), one square root (sound speed);
//     one reciprocal of the common interface speed for both axes;
//   * the convected flux 1/2 (M (aL fL + aR fR) - |M| (aR fR - aL fL)) is the
//     upwind side's M a f;
//   * the side order of each axis (bit d of `flags`: c0 is the left state)
//     selects the operands, so a warp whose faces differ in it runs the axis
//     once.
template <class T>
struct AusmCell {
  T u[2], p, a_face, a_true, w[4];  // w = a_true (rho, rho u, rho v, rho H)
};
template <class T>
__device__ __forceinline__ AusmCell<T> ausm_cell(const T q[4]) {
  const T gm1 = Gas<T>::gm1();
  AusmCell<T> s;
  const T ir = T(1) / q[0];
  s.u[0] = q[1] * ir;
  s.u[1] = q[2] * ir;
  s.p = (q[3] - T(0.5) * (q[1] * s.u[0] + q[2] * s.u[1])) * gm1;
  const T rh = q[3] + s.p;
  const T as2 = rh * ir * (T(2) * gm1 / Gas<T>::gp1());
  const T U2 = s.u[0] * s.u[0] + s.u[1] * s.u[1];
  s.a_face = as2 * inv_sqrt(as2 < U2 ? U2 : as2);
  s.a_true = sqrt(Gas<T>::gamma() * s.p * ir);
  s.w[0] = s.a_true * q[0];
  s.w[1] = s.a_true * q[1];
  s.w[2] = s.a_true * q[2];
  s.w[3] = s.a_true * rh;
  return s;
}
template <class T>
__device__ __forceinline__ void ausm_face(const T qa[4], const T qb[4], int flags, T F[8]) {
  const AusmCell<T> A = ausm_cell(qa), B = ausm_cell(qb);
  // (the zero product hands a sound speed that is not a number -- a state
  // without positive pressure or density on either side -- to every flux)
  const T ia = T(1) / (B.a_face < A.a_face ? B.a_face : A.a_face) +
               T(0) * (A.a_true + B.a_true);
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const bool c0l = (flags >> d) & 1;  // c0 (qa) is the left state
    const T mL = (c0l ? A.u[d] : B.u[d]) * ia, mR = (c0l ? B.u[d] : A.u[d]) * ia;
    const T pL = c0l ? A.p : B.p, pR = c0l ? B.p : A.p;
    T mp = mL, pp = pL, mm = T(0), pm = T(0);
    if (!(mL > T(1))) {
      const T s = mL + T(1), h = T(0.25) * (s * s), t = mL * mL - T(1), b = t * t;
      mp = h + T(0.125) * b;
      pp = (pL * h) * (T(2) - mL) + (T(0.1875) * mL) * b;
    }
    if (!(mR > T(1))) {
      const T s = mR - T(1), h = T(0.25) * (s * s), t = mR * mR - T(1), b = t * t;
      mm = -h - T(0.125) * b;
      pm = (pR * h) * (T(2) + mR) - (T(0.1875) * mR) * b;
    }
    const T mF = mm + mp;
    const bool up = (mF >= T(0)) == c0l;  // the upwind side is c0
#pragma unroll
    for (int k = 0; k < 4; ++k) F[4 * d + k] = mF * (up ? A.w[k] : B.w[k]);
    F[5 * d + 1] += pp + pm;
  }
}

template <class T>
__host__ __device__ __forceinline__ T entropy_fix(T x) {
  const T e = T(0.125);
  if (x > e) return x;
  return (x * x + e * e) / T(2) / e;
}

template <class T>
__host__ __device__ __forceinline__ T det3(T a, T b, T c, T d, T e, T f, T g,
                                           T h, T i) {
  return a * (e * i - f * h) - b * (d * i - f * g) + c * (d * h - e * g);
}

// 4x4 inverse by the adjugate formula (row-major), the algorithm of the
// oracle's Eigen shim: cofactors from 3x3 minors by first-row expansion,
// det along row 0, inverse = adj^T * (1/det).
template <class T>
__host__ __device__ __forceinline__ void inv4(const T m[16], T inv[16]) {
  T cof[16];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r0 = (i == 0) ? 1 : 0, r1 = (i <= 1) ? 2 : 1, r2 = (i <= 2) ? 3 : 2;
      const int c0 = (j == 0) ? 1 : 0, c1 = (j <= 1) ? 2 : 1, c2 = (j <= 2) ? 3 : 2;
      T v = det3(m[4 * r0 + c0], m[4 * r0 + c1], m[4 * r0 + c2],
                 m[4 * r1 + c0], m[4 * r1 + c1], m[4 * r1 + c2],
                 m[4 * r2 + c0], m[4 * r2 + c1], m[4 * r2 + c2]);
      cof[4 * i + j] = ((i + j) & 1) ? -v : v;
    }
  }
  T det = m[0] * cof[0];
  det += m[1] * cof[1];
  det += m[2] * cof[2];
  det += m[3] * cof[3];
  const T id = T(1) / det;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) inv[4 * i + j] = cof[4 * j + i] * id;
}

// Roe flux along axis d.
template <class T>
__host__ __device__ __forceinline__ void roe_flux(const T ql[4], const T qr[4],
                                                  int d, T f[4]) {
  const T eor = T(1e-10);
  const T D = sqrt(fabs(qr[0] / ql[0]));
  T u[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
    u[k] = ediv(ediv(ql[k + 1], ql[0]) + ediv(D * qr[k + 1], qr[0]), T(1) + D);
  const T pL = th_p(ql), pR = th_p(qr);
  const T hL = (ql[3] + pL) / ql[0], hR = (qr[3] + pR) / qr[0];
  const T H = (hL + D * hR) / (T(1) + D);
  const T un = sqrt(u[0] * u[0] + u[1] * u[1]);
  const T a = sqrt(fabs(Gas<T>::gm1() * (H - T(0.5) * (un * un))));
  const T ud = u[d];
  T lam[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) lam[k] = T(0);
  lam[0] = entropy_fix(fabs(ud - a));
  lam[5] = entropy_fix(fabs(ud));
  lam[10] = entropy_fix(fabs(ud));
  lam[15] = entropy_fix(fabs(ud + a));
  const T ke = T(0.5) * (u[0] * u[0] + u[1] * u[1]);
  T R[16], FL[4], FR[4];
  if (d == 0) {
    R[0] = T(1); R[1] = T(1); R[2] = T(0); R[3] = T(1);
    R[4] = u[0] - a; R[5] = u[0]; R[6] = T(0); R[7] = u[0] + a;
    R[8] = u[1]; R[9] = u[1]; R[10] = T(1); R[11] = u[1];
    R[12] = H - u[0] * a; R[13] = ke; R[14] = u[1]; R[15] = H + u[0] * a;
    FL[0] = ql[1];
    FL[1] = ediv(ql[1] * ql[1], ql[0] + eor) + pL;
    FL[2] = ediv(ql[1] * ql[2], ql[0] + eor);
    FL[3] = hL * ql[1];
    FR[0] = qr[1];
    FR[1] = ediv(qr[1] * qr[1], qr[0] + eor) + pR;
    FR[2] = ediv(qr[1] * qr[2], qr[0] + eor);
    FR[3] = hR * qr[1];
  } else {
    R[0] = T(1); R[1] = T(1); R[2] = T(0); R[3] = T(1);
    R[4] = u[0]; R[5] = u[0]; R[6] = T(1); R[7] = u[0];
    R[8] = u[1] - a; R[9] = u[1]; R[10] = T(0); R[11] = u[1] + a;
    R[12] = H - u[1] * a; R[13] = ke; R[14] = u[0]; R[15] = H + u[1] * a;
    FL[0] = ql[2];
    FL[1] = ediv(ql[1] * ql[2], ql[0] + eor);
    FL[2] = ediv(ql[2] * ql[2], ql[0] + eor) + pL;
    FL[3] = hL * ql[2];
    FR[0] = qr[2];
    FR[1] = ediv(qr[1] * qr[2], qr[0] + eor);
    FR[2] = ediv(qr[2] * qr[2], qr[0] + eor) + pR;
    FR[3] = hR * qr[2];
  }
  T Ri[16];
  inv4(R, Ri);
  // (R * Lambda) * R^-1 with the shim's left-to-right sums
  T RL[16], A[16];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      T s = R[4 * i] * lam[j];
#pragma unroll
      for (int k = 1; k < 4; ++k) s += R[4 * i + k] * lam[4 * k + j];
      RL[4 * i + j] = s;
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      T s = RL[4 * i] * Ri[j];
#pragma unroll
      for (int k = 1; k < 4; ++k) s += RL[4 * i + k] * Ri[4 * k + j];
      A[4 * i + j] = s;
    }
  T dU[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) dU[k] = qr[k] - ql[k];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    T s = (T(0.5) * A[4 * k]) * dU[0];
#pragma unroll
    for (int j = 1; j < 4; ++j) s += (T(0.5) * A[4 * k + j]) * dU[j];
    f[k] = T(0.5) * (FL[k] + FR[k]) - s;
  }
}

// Roe of both axes of a face for the production paths (FP64 and FP32): the
// same physical fluxes, entropy-fixed eigenvalues and EOR denominators as
// roe_flux, with |A| dQ in closed form (the sum over the waves of
// |lambda_k| alpha_k r_k) and everything that does not depend on the axis
// formed once per face: the Roe average is symmetric in the two states and
// the jumps change sign with their order, so the dissipation of axis d only
// enters with the sign of the side order (bit d of `flags`: c0 is the left
// state).  One reciprocal square root gives a and 1/a^2.  Not used by the
// exact path.
template <class T>
__device__ __forceinline__ T entropy_fix_fast(T x) {
  const T ax = fabs(x), e = T(0.125);
  return ax > e ? ax : (x * x + e * e) * (T(0.5) / e);
}
// Products whose rounded values have to cancel: equal pressures and velocities
// of the two sides, the terms of mirrored states at a wall.  A fused
// multiply-add of one of them leaves the other's rounding error (at FP32 a mass
// flux of 1e-9 through walls).  sep: in FP32 only; in FP64 that error is below
// 1e-16 and the fused form saves an instruction of the busiest pipe.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float sep(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sep(double a, double b) { return a * b; }
// sqrt(R / L) of the Roe average: in FP32 the root itself, which gives 1 where
// the quotient of equal numbers is off by its rounding
__device__ __forceinline__ float roe_ratio(float x) { return sqrtf(x); }
__device__ __forceinline__ double roe_ratio(double x) { return x * inv_sqrt(x); }

template <class T>
__device__ __forceinline__ void roe_face(const T L[4], const T R[4], int flags, T F[8]) {
  const T eor = T(1e-10), gm1 = Gas<T>::gm1();
  const T irL = T(1) / L[0], irR = T(1) / R[0];
  const T uL[2] = {mul_rn(L[1], irL), mul_rn(L[2], irL)},
          uR[2] = {mul_rn(R[1], irR), mul_rn(R[2], irR)};
  const T pL = mul_rn(L[3] - T(0.5) * (L[1] * uL[0] + L[2] * uL[1]), gm1);
  const T pR = mul_rn(R[3] - T(0.5) * (R[1] * uR[0] + R[2] * uR[1]), gm1);
  const T hL = (L[3] + pL) * irL, hR = (R[3] + pR) * irR;
  const T D = roe_ratio(fabs(R[0] * irL));
  const T iD = T(1) / (T(1) + D);
  const T u[2] = {(uL[0] + D * uR[0]) * iD, (uL[1] + D * uR[1]) * iD};
  const T H = (hL + D * hR) * iD;
  const T ke = T(0.5) * (u[0] * u[0] + u[1] * u[1]);
  const T a2 = fabs(gm1 * (H - ke));
  const T ia = inv_sqrt(a2);
  const T a = a2 * ia, ia2 = ia * ia;
  const T rt = D * L[0];
  const T dp = pR - pL, du[2] = {uR[0] - uL[0], uR[1] - uL[1]};
  const T al2 = (R[0] - L[0]) - dp * ia2;
  const T hia2 = T(0.5) * ia2, rta = rt * a;
  const T iL = T(1) / (L[0] + eor), iR = T(1) / (R[0] + eor);
  // momentum / (rho + EOR), momentum fluxes' second factor
  const T vL[2] = {L[1] * iL, L[2] * iL}, vR[2] = {R[1] * iR, R[2] * iR};
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const int t = 1 - d;
    const T ud = u[d], ut = u[t];
    const T l1 = entropy_fix_fast(ud - a), l2 = entropy_fix_fast(ud),
            l4 = entropy_fix_fast(ud + a);
    const T rd = rta * du[d];
    const T w1 = sep(l1, (dp - rd) * hia2), w4 = sep(l4, (dp + rd) * hia2);
    const T w2 = sep(l2, al2), w3 = l2 * (rt * du[t]);
    const T ws = (w1 + w2) + w4, wd = (w4 - w1) * a;
    const T sg = ((flags >> d) & 1) ? T(-0.5) : T(0.5);
    const T mL = L[1 + d], mR = R[1 + d];
    F[4 * d] = T(0.5) * (mL + mR) + sg * ws;
    F[4 * d + 1 + d] = T(0.5) * ((sep(mL, vL[d]) + sep(mR, vR[d])) + (pL + pR)) + sg * (ws * ud + wd);
    F[4 * d + 1 + t] = T(0.5) * (sep(mL, vL[t]) + sep(mR, vR[t])) + sg * (ws * ut + w3);
    F[4 * d + 3] = T(0.5) * (sep(hL, mL) + sep(hR, mR)) +
                   sg * ((w1 + w4) * H + (wd * ud + (w2 * ke + w3 * ut)));
  }
}

}  // namespace mst
