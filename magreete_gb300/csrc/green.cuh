// Green's-function blocks, evaluated in FP64 (shared by assembly and the
// matrix-free propagate).
//
// Formulas (r = t - s, R = |r|, P = r r^T / R^2):
//   2D TE  (Transmission2D.py:63-91): (i/4)[(I-P) H0(kR) - (I-2P) H1(kR)/(kR)]
//   2D TM  (Transmission2D.py:595-618): (i/4) H0(kR)
//   3D vec (Transmission3D.py:47-77): [I - P - (I-3P)(1/(ikR) + 1/(kR)^2)] e^{ikR}/(4 pi R)
//   3D sca (Transmission3D.py:573-601): e^{ikR}/(4 pi R)
// with H_nu from hankel.cuh.  FP64 operations are what these cost (1.7 a clock
// and SM), so each block is formed from its two scalar coefficients -- the
// identity's and the projector's.
#pragma once
#include "common.cuh"
#include "hankel.cuh"

namespace mgt {

template <int KIND> struct Kind;
template <> struct Kind<MGT_2D_VECTOR> { static constexpr int dim = 2, d = 2; };
template <> struct Kind<MGT_2D_SCALAR> { static constexpr int dim = 2, d = 1; };
template <> struct Kind<MGT_3D_VECTOR> { static constexpr int dim = 3, d = 3; };
template <> struct Kind<MGT_3D_SCALAR> { static constexpr int dim = 3, d = 1; };

// Before a kernel that calls green_block<KIND>, on its stream.
template <int KIND>
static inline cudaError_t prepare_green(cudaStream_t s) {
  return Kind<KIND>::dim == 2 ? hk::ensure_table(s) : cudaSuccess;
}

// d x d Green's block for separation r (row-major in g).
// Returns false where the reference's value is NaN: R == 0, or R (k*R for the
// 2D TE kind) below `radius` when regularising.
template <int KIND>
__device__ __forceinline__ bool green_block(const double* r, double k0, bool regularize,
                                            double radius, double2* g) {
  constexpr double kPi = 3.14159265358979323846;
  if constexpr (KIND == MGT_2D_VECTOR) {
    const double R2 = r[0] * r[0] + r[1] * r[1];
    const double R = sqrt(R2);
    double kR = k0 * R;
    if (regularize && kR < radius) kR = 0.0;
    if (R2 == 0.0 || kR == 0.0) return false;
    const double ikR = __drcp_rn(kR), q = __drcp_rn(R2);
    double2 h0, h1;
    hk::hankel01<true>(kR, h0, h1);
    h1.x *= ikR;
    h1.y *= ikR;
    // t = (I - P) H0 - (I - 2 P) H1 / (kR) = I D - P F, times i / 4
    const double Dr = 0.25 * (h0.x - h1.x), Di = 0.25 * (h0.y - h1.y);
    const double Fr = 0.25 * fma(-2.0, h1.x, h0.x), Fi = 0.25 * fma(-2.0, h1.y, h0.y);
    const double xq = r[0] * q, yq = r[1] * q;
    const double xx = r[0] * xq, xy = r[1] * xq, yy = r[1] * yq;
    g[0] = make_double2(fma(xx, Fi, -Di), fma(-xx, Fr, Dr));
    g[3] = make_double2(fma(yy, Fi, -Di), fma(-yy, Fr, Dr));
    g[1] = g[2] = make_double2(xy * Fi, -xy * Fr);
    return true;
  } else if constexpr (KIND == MGT_2D_SCALAR) {
    double R = sqrt(r[0] * r[0] + r[1] * r[1]);
    if (regularize && R < radius) R = 0.0;
    if (R == 0.0) return false;
    double2 h0, h1;
    hk::hankel01<false>(k0 * R, h0, h1);
    g[0] = make_double2(-0.25 * h0.y, 0.25 * h0.x);
    return true;
  } else if constexpr (KIND == MGT_3D_VECTOR) {
    const double R2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    double R = sqrt(R2);
    if (regularize && R < radius) R = 0.0;
    if (R2 == 0.0 || R == 0.0) return false;
    const double kR = k0 * R, inv = __drcp_rn(kR), q = __drcp_rn(R2);
    double s, c;
    sincos(kR, &s, &c);
    const double amp = __drcp_rn(4.0 * kPi * R);
    const double er = c * amp, ei = s * amp;
    // f = 1/(ikR) + 1/(kR)^2 = inv^2 - i inv; identity 1 - f, projector -(1 - 3 f)
    const double fr = inv * inv, dr = 1.0 - fr, pr = fma(3.0, fr, -1.0), pi = -3.0 * inv;
    const double Dr = fma(dr, er, -inv * ei), Di = fma(dr, ei, inv * er);
    const double Pr = q * fma(pr, er, -pi * ei), Pi = q * fma(pr, ei, pi * er);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a; b < 3; ++b) {
        const double rr = r[a] * r[b];
        g[a * 3 + b] = a == b ? make_double2(fma(rr, Pr, Dr), fma(rr, Pi, Di)) : make_double2(rr * Pr, rr * Pi);
        if (b != a) g[b * 3 + a] = g[a * 3 + b];
      }
    return true;
  } else {
    double R = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    if (regularize && R < radius) R = 0.0;
    if (R == 0.0) return false;
    double s, c;
    sincos(k0 * R, &s, &c);
    const double amp = __drcp_rn(4.0 * kPi * R);
    g[0] = make_double2(c * amp, s * amp);
    return true;
  }
}

}  // namespace mgt
