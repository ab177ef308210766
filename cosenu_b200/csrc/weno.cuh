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

struct WenoB {
    double b0, b1, b2, b3;  // eps + beta_r, over 60
    double Fa, Fb, Fc;      // fourth differences about centre + 1, centre, centre - 1
    double q1;              // 12 x (candidate 1 - centre value)
};

// (Multiply-adds are written out here and below, so that a face has the same bits
// whether it is evaluated alone or among its neighbours.)
__device__ __forceinline__ WenoB weno7_indicators(const double *dl)
{
    const double c13 = 13.0 / 3.0, c781 = 781.0 / 180.0, eps = WENO_EPS;
    const double D0 = dl[1] - dl[0], D1 = dl[2] - dl[1], D2 = dl[3] - dl[2], D3 = dl[4] - dl[3],
                 D4 = dl[5] - dl[4];
    const double T0 = D1 - D0, T1 = D2 - D1, T2 = D3 - D2, T3 = D4 - D3;
    const double t0 = __fma_rn(c781 * T0, T0, eps), t1 = __fma_rn(c781 * T1, T1, eps),
                 t2 = __fma_rn(c781 * T2, T2, eps), t3 = __fma_rn(c781 * T3, T3, eps);
    const double C2 = dl[2] + dl[3];                  // u[1] - u[-1]
    const double dd = __dmul_rn(c13 * D2, D2);        // the inner sub-stencils' second difference
    const double y1 = __fma_rn(-1.0 / 3.0, T2, C2), y2 = __fma_rn(-1.0 / 3.0, T1, C2);
    const double e0 = D3 - T3, e3 = D1 + T0;          // the outer ones', continued to the centre
    const double y0 = __fma_rn(2.0 / 3.0, T3, __fma_rn(2., dl[3], -D3));
    const double y3 = __fma_rn(2.0 / 3.0, T0, __fma_rn(2., dl[2], D1));
    WenoB r;
    r.b0 = __fma_rn(c13 * e0, e0, __fma_rn(y0, y0, t3));
    r.b1 = __fma_rn(y1, y1, dd) + t2;
    r.b2 = __fma_rn(y2, y2, dd) + t1;
    r.b3 = __fma_rn(c13 * e3, e3, __fma_rn(y3, y3, t0));
    r.Fc = T1 - T0;
    r.Fb = T2 - T1;
    r.Fa = T3 - T2;
    r.q1 = __fma_rn(6., dl[3], dl[2] - dl[4]);
    return r;
}

// FP64: the weights brought to a common denominator; the face is
// centre + (q1 + num / den) / 12.
__device__ __forceinline__ void weno7_parts(const double *dl, double &q1, double &num, double &den)
{
    const WenoB r = weno7_indicators(dl);
    const double d0 = r.b0 * r.b0, d1 = r.b1 * r.b1, d2 = r.b2 * r.b2, d3 = r.b3 * r.b3;
    const double d01 = d0 * d1, d23 = d2 * d3;
    // gamma_r x prod_{k != r} d_k
    const double w0 = __dmul_rn(4., d1 * d23), w1 = __dmul_rn(d0, d23),
                 w2 = __dmul_rn(12., d01 * d3), w3 = __dmul_rn(d01, d2);
    q1 = r.q1;
    num = __fma_rn(w3, __fma_rn(-3., r.Fc, r.Fb), __fma_rn(w0, r.Fa, __dmul_rn(w2, r.Fb)));
    den = __fma_rn(18., w1, w0) + __dadd_rn(w2, w3);
}

// 12 x (face - centre), one face.
__device__ __forceinline__ double weno7_corr12(const double *dl)
{
    double q1, num, den;
    weno7_parts(dl, q1, num, den);
    return __dadd_rn(q1, __ddiv_rn(num, den));
}

// 12 x (face - centre) of four consecutive faces from the nine differences of
// their ten cells, with one division: the reciprocal of the product of the four
// denominators, times the others.
//
// The last face is the one that a tile's neighbour also evaluates, by itself
// (its upwind edge), and a cell has to be left by what enters the next one: its
// quotient gets one residual step (Markstein 1990), which makes it that of the
// division, num / den rounded once, but for some 4e-15 of all faces.  Two of 240
// operations; without it fluxes across every 32nd face telescoped to rounding
// only.
//
// Denominators lie in [7e-46, 1e21] where the stencil differences are at most 2
// in magnitude (density-matrix entries of O(1)), so the product of four is far
// inside the FP64 range.  States in other units leave it (differences of 1e5 and
// more); then, and for non-finite cells, every face has its own division.
__device__ __forceinline__ void weno7_quad(const double *dl, double *c12)
{
    double q1[4], num[4], den[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) weno7_parts(dl + k, q1[k], num[k], den[k]);
    const double p01 = den[0] * den[1], p23 = den[2] * den[3], p = p01 * p23;
    // (denominators are positive: their high words order as the values do)
    const unsigned top = max(max((unsigned)__double2hiint(p01), (unsigned)__double2hiint(p23)),
                             (unsigned)__double2hiint(p));
    if (top < 0x7fb00000u) {  // 2^1020: the reciprocals are normal numbers
        const double r = 1.0 / p;
        const double r01 = r * p23, r23 = r * p01;
        c12[0] = __fma_rn(num[0], r01 * den[1], q1[0]);
        c12[1] = __fma_rn(num[1], r01 * den[0], q1[1]);
        c12[2] = __fma_rn(num[2], r23 * den[3], q1[2]);
        const double inv = r23 * den[2], q = __dmul_rn(num[3], inv);
        c12[3] = __dadd_rn(q1[3], __fma_rn(__fma_rn(-q, den[3], num[3]), inv, q));
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) c12[k] = __dadd_rn(q1[k], __ddiv_rn(num[k], den[k]));
    }
}

// FP32-bulk form: the face's increment, x0 + (face - centre), from the
// stencil's differences to its centre, A .. G = u[-3..3] - u[0] (skipping the
// centre), which the caller takes in FP64 so that FP32 sees only the small
// differences and not the O(1) values; x0 is the centre's own increment.  The
// indicators are the published quadratic forms; the weights use approximate
// reciprocals (a common denominator would leave the FP32 range).
//
// The forms' cancellation is this option's largest error: on noise of 2e-2 a
// face is within 1.2e-7, where the sums of squares above would give 8.5e-9.
// FP32-bulk results are these roundings, though (sums of squares moved a state
// by 6.5e-10 of its size in six rough steps), so every operation is written
// out: the bits do not depend on what surrounds the call.  LARGE: whether
// candidate 1 or 0 is the first product of the sum, the one that is rounded
// before it is added.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <bool LARGE>
__device__ __forceinline__ float weno7_inc(float A, float B, float Cc, float E, float F, float G,
                                           float x0)
{
    // a x + b y + c z, and eps + P (..) + Q (..) + k R R
    auto sum3 = [](float a, float x, float b, float y, float c, float z) {
        return __fmaf_rn(c, z, __fmaf_rn(a, x, __fmul_rn(b, y)));
    };
    auto beta = [](float P, float p, float Q, float q, float k, float R) {
        return __fadd_rn(1e-6f, __fmaf_rn(__fmul_rn(k, R), R, __fmaf_rn(P, p, __fmul_rn(Q, q))));
    };
    auto sum2 = [](float a, float x, float b, float y) { return __fmaf_rn(a, x, __fmul_rn(b, y)); };
    const float b0 = beta(E, sum3(11003.f, E, -17246.f, F, 4642.f, G), F,
                          sum2(7043.f, F, -3882.f, G), 547.f, G);
    const float b1 = beta(Cc, sum3(547.f, Cc, 1922.f, E, -494.f, F), E,
                          sum2(2843.f, E, -1642.f, F), 267.f, F);
    const float b2 = beta(B, sum3(267.f, B, -1642.f, Cc, -494.f, E), Cc,
                          sum2(2843.f, Cc, 1922.f, E), 547.f, E);
    const float b3 = beta(A, sum3(547.f, A, -3882.f, B, 4642.f, Cc), B,
                          sum2(7043.f, B, -17246.f, Cc), 11003.f, Cc);
    // 12 x (candidate - centre)
    const float q0 = __fadd_rn(__fmaf_rn(13.f, E, __fmul_rn(-5.f, F)), G);
    const float q1 = __fsub_rn(__fmaf_rn(7.f, E, -Cc), F);
    const float q2 = __fmaf_rn(3.f, E, __fmaf_rn(-5.f, Cc, B));
    const float q3 = __fmaf_rn(-23.f, Cc, __fmaf_rn(13.f, B, __fmul_rn(-3.f, A)));
    const float w0 = __fmul_rn(4.f, rcp_approx(__fmul_rn(b0, b0))),
                w1 = __fmul_rn(18.f, rcp_approx(__fmul_rn(b1, b1))),
                w2 = __fmul_rn(12.f, rcp_approx(__fmul_rn(b2, b2))),
                w3 = rcp_approx(__fmul_rn(b3, b3));
    const float n01 = LARGE ? __fmaf_rn(w1, q1, __fmul_rn(w0, q0))
                            : __fmaf_rn(w0, q0, __fmul_rn(w1, q1));
    const float num = __fmaf_rn(w3, q3, __fmaf_rn(w2, q2, n01));
    const float sum = __fadd_rn(__fadd_rn(__fadd_rn(w0, w1), w2), w3);
    return __fmaf_rn(num, rcp_approx(__fmul_rn(12.f, sum)), x0);
}

// The faces about cells 4 .. 7 of twelve, stencil direction dir: dif(i, j) is
// u[j] - u[i] in FP32.  The differences between the four centres serve two faces
// each (rounding is symmetric in sign).
template <bool LARGE, class DIF>
__device__ __forceinline__ void weno7_inc_quad(DIF dif, int dir, const float *x0, float *c)
{
    float in[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i + 1; j < 4; ++j) {
            in[i][j] = dif(i + 4, j + 4);
            in[j][i] = -in[i][j];
        }
    auto d = [&](int k, int n) {  // u[k + n] - u[k]
        return k + n >= 0 && k + n < 4 ? in[k][(k + n) & 3] : dif(k + 4, k + 4 + n);
    };
    const bool up = dir > 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float m3 = d(k, -3), m2 = d(k, -2), m1 = d(k, -1), p1 = d(k, 1), p2 = d(k, 2), p3 = d(k, 3);
        c[k] = weno7_inc<LARGE>(up ? m3 : p3, up ? m2 : p2, up ? m1 : p1, up ? p1 : m1, up ? p2 : m2, up ? p3 : m3, x0[k]);
    }
}

}  // namespace cosenu
