// WENO7 face reconstruction shared by the stage kernels.
#pragma once

#include "common.cuh"

namespace cosenu {

// The face value of the cell whose right face (j+1/2) is reconstructed with
// left-biased weights (rflux of src/rhs_fv.hpp:37-71), from the six first
// differences dl[i] = u[i-2] - u[i-3] (i = 0..5) of its seven-point stencil
// u[-3..3]: smoothness indicators and candidate polynomials of the four
// 4-point sub-stencils, nonlinear weights gamma_r / (eps + beta_r)^2 with
// gamma = (4, 18, 12, 1)/35 and eps = 1e-6.  The mirrored stencil (the left
// face of a cell with downwind weights) has the same differences in reverse
// order with the opposite sign; every term below is then even (the
// indicators) or odd (the correction), so the caller passes them reversed and
// subtracts the correction.
//
// FP64 issue bounds the FV stages, so the indicators are written as the sums of
// squares they are, not as quadratic forms in the values: with the second,
// third and fourth differences D, T, F,
//     beta_r / 60 = y_r^2 + 13/3 D_r^2 + 781/180 T_r^2,
// where y_r and D_r are twice the first and second derivative of sub-stencil
// r's cubic at the centre (the constant 60 cancels in the weights), and
// neighbouring candidates differ by one fourth difference:
//     q0 = q1 + Fa,  q2 = q1 + Fb,  q3 = q2 - 3 Fc.
// 70 FP64 operations for a lone face, but D, T, F and the T^2 terms are those
// of the neighbouring faces too: 55 per face for four consecutive faces of one
// row evaluated by one thread (the compiler merges the equal expressions),
// against 75 in the quadratic form, which shares nothing.
constexpr double WENO_EPS = 1e-6 / 60.0;

template <class T> struct WenoB {
    T b0, b1, b2, b3;  // eps + beta_r, over 60
    T Fa, Fb, Fc;      // fourth differences about centre + 1, centre, centre - 1
    T q1;              // 12 x (candidate 1 - centre value)
};

template <class T> __device__ __forceinline__ WenoB<T> weno7_indicators(const T *dl)
{
    const T c13 = T(13.0 / 3.0), c781 = T(781.0 / 180.0), eps = T(WENO_EPS);
    const T D0 = dl[1] - dl[0], D1 = dl[2] - dl[1], D2 = dl[3] - dl[2], D3 = dl[4] - dl[3],
            D4 = dl[5] - dl[4];
    const T T0 = D1 - D0, T1 = D2 - D1, T2 = D3 - D2, T3 = D4 - D3;
    const T t0 = (c781 * T0) * T0 + eps, t1 = (c781 * T1) * T1 + eps, t2 = (c781 * T2) * T2 + eps,
            t3 = (c781 * T3) * T3 + eps;
    const T C2 = dl[2] + dl[3];       // u[1] - u[-1]
    const T dd = (c13 * D2) * D2;     // the inner sub-stencils' second difference
    const T y1 = C2 - T(1.0 / 3.0) * T2, y2 = C2 - T(1.0 / 3.0) * T1;
    const T e0 = D3 - T3, e3 = D1 + T0;  // the outer ones', continued to the centre
    const T y0 = (T(2) * dl[3] - D3) + T(2.0 / 3.0) * T3;
    const T y3 = (T(2) * dl[2] + D1) + T(2.0 / 3.0) * T0;
    WenoB<T> r;
    r.b0 = (c13 * e0) * e0 + (y0 * y0 + t3);
    r.b1 = (y1 * y1 + dd) + t2;
    r.b2 = (y2 * y2 + dd) + t1;
    r.b3 = (c13 * e3) * e3 + (y3 * y3 + t0);
    r.Fc = T1 - T0;
    r.Fb = T2 - T1;
    r.Fa = T3 - T2;
    r.q1 = T(6) * dl[3] + (dl[2] - dl[4]);
    return r;
}

// FP64: the weights brought to a common denominator; the face is
// centre + (q1 + num / den) / 12.
__device__ __forceinline__ void weno7_parts(const double *dl, double &q1, double &num, double &den)
{
    const WenoB<double> r = weno7_indicators<double>(dl);
    const double d0 = r.b0 * r.b0, d1 = r.b1 * r.b1, d2 = r.b2 * r.b2, d3 = r.b3 * r.b3;
    const double d01 = d0 * d1, d23 = d2 * d3;
    // gamma_r x prod_{k != r} d_k
    const double w0 = 4. * (d1 * d23), w1 = d0 * d23, w2 = 12. * (d01 * d3), w3 = d01 * d2;
    q1 = r.q1;
    num = w0 * r.Fa + w2 * r.Fb + w3 * (r.Fb - 3. * r.Fc);
    den = (18. * w1 + w0) + (w2 + w3);
}

// 12 x (face - centre), one face.
__device__ __forceinline__ double weno7_corr12(const double *dl)
{
    double q1, num, den;
    weno7_parts(dl, q1, num, den);
    return q1 + num / den;
}

// 1 / D0 .. 1 / D3 from one division: the product of the four, its
// reciprocal, then products of the others.  Denominators of weno7_parts lie
// in [7e-46, 1e21] where the stencil differences are at most 2 in magnitude
// (density-matrix entries of O(1)), so the product of four stays far inside
// the FP64 range.
__device__ __forceinline__ void recip4(double D0, double D1, double D2, double D3, double &i0,
                                       double &i1, double &i2, double &i3)
{
    const double p01 = D0 * D1, p23 = D2 * D3;
    const double r = 1.0 / (p01 * p23);
    const double r01 = r * p23, r23 = r * p01;
    i0 = r01 * D1;
    i1 = r01 * D0;
    i2 = r23 * D3;
    i3 = r23 * D2;
}

// 12 x (face - centre) of four consecutive faces from the nine differences of
// their ten cells.
__device__ __forceinline__ void weno7_quad(const double *dl, double *c12)
{
    double q1[4], num[4], den[4], inv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) weno7_parts(dl + k, q1[k], num[k], den[k]);
    recip4(den[0], den[1], den[2], den[3], inv[0], inv[1], inv[2], inv[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) c12[k] = num[k] * inv[k] + q1[k];
}

// FP32-bulk form: 12 x (face - centre) in FP32 from differences the caller
// takes in FP64, so that FP32 sees only the small differences and not the
// O(1) values.  Same indicators and candidates; the weights use fast
// reciprocals (a common denominator would leave the FP32 range).
__device__ __forceinline__ float weno7_corr12(const float *dl)
{
    const WenoB<float> r = weno7_indicators<float>(dl);
    const float w0 = __fdividef(4.f, r.b0 * r.b0), w1 = __fdividef(18.f, r.b1 * r.b1),
                w2 = __fdividef(12.f, r.b2 * r.b2), w3 = __fdividef(1.f, r.b3 * r.b3);
    const float num = w0 * r.Fa + w2 * r.Fb + w3 * (r.Fb - 3.f * r.Fc);
    return r.q1 + __fdividef(num, (w0 + w1) + (w2 + w3));
}

__device__ __forceinline__ void weno7_quad(const float *dl, float *c12)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) c12[k] = weno7_corr12(dl + k);
}

}  // namespace cosenu
