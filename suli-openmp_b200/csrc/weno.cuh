// weno.cuh — fifth-order WENO one-sided derivatives (Jiang–Shu) of a cell field along one
// axis, as the reference's pencil routine weno1 computes them (14_level_set.f90:511-610),
// re-expressed per cell so that a thread needs only the seven values phi(i-3..i+3).
//
// Ghost values outside 1..n are rebuilt from interior values with the pencil routine's own
// rules (ihs, :530-570): 0 periodic with phi(0) = phi(n-1) (the reference's offset),
// 1 one-sided extrapolation (1/5 rows at the low end, 1/11 rows at the high end),
// 2 the 1/11 "zero derivative" rows at both ends.  The arithmetic is the reference's with its
// divisions rearranged: the reciprocal of h formed once on the host, and in FP64 the nonlinear
// weights w_k/q_k^2 / sum_m w_m/q_m^2 formed over a common denominator (one division per side).
//
// The FP64 kernels are bound by the FP64 pipe (70 % busy at 150 instructions a one-sided pair), so
// FP64 forms the pair from the differences E of the divided differences D: the second differences
// and smoothness terms of the stencils that both sides share once, the smoothness indicators up to
// a common factor, and each candidate as the centre D plus a combination of E, which needs the
// weights' ratios only (about 100 instructions).  FP32 keeps the reference's expressions.
#pragma once

namespace suli {

// Fetch phi(m) of a pencil at position m in [i-3, i+3], applying the ghost rules.
// `at(m)` returns the stored interior value for m in 1..n.
template <typename T, typename F>
__device__ __forceinline__ void pencil7(F at, int i, int n, int ihs, T P[7]) {
    if (i >= 4 && i <= n - 3) {
#pragma unroll
        for (int m = 0; m < 7; ++m) P[m] = at(i - 3 + m);
        return;
    }
    // boundary neighbourhood: build the ghosts the reference builds for the whole pencil
    T g_lo[3], g_hi[3];   // g_lo[0] = phi(0), g_lo[1] = phi(-1), g_lo[2] = phi(-2); g_hi[0] = phi(n+1) ...
    if (ihs == 0) {
        g_lo[0] = at(n - 1); g_lo[1] = at(n - 2); g_lo[2] = at(n - 3);
        g_hi[0] = at(2); g_hi[1] = at(3); g_hi[2] = at(4);
    } else {
        const T p1 = at(1), p2 = at(2), p3 = at(3);
        const T qn = at(n), qn1 = at(n - 1), qn2 = at(n - 2);
        if (ihs == 1) {
            g_lo[0] = T(1. / 5.) * (T(12.) * p1 - T(9.) * p2 + T(2.) * p3);
            g_lo[1] = T(1. / 5.) * (T(12.) * g_lo[0] - T(9.) * p1 + T(2.) * p2);
            g_lo[2] = T(1. / 5.) * (T(12.) * g_lo[1] - T(9.) * g_lo[0] + T(2.) * p1);
        } else {
            g_lo[0] = T(1. / 11.) * (T(18.) * p1 - T(9.) * p2 + T(2.) * p3);
            g_lo[1] = T(1. / 11.) * (T(18.) * g_lo[0] - T(9.) * p1 + T(2.) * p2);
            g_lo[2] = T(1. / 11.) * (T(18.) * g_lo[1] - T(9.) * g_lo[0] + T(2.) * p1);
        }
        g_hi[0] = T(1. / 11.) * (T(18.) * qn - T(9.) * qn1 + T(2.) * qn2);
        g_hi[1] = T(1. / 11.) * (T(18.) * g_hi[0] - T(9.) * qn + T(2.) * qn1);
        g_hi[2] = T(1. / 11.) * (T(18.) * g_hi[1] - T(9.) * g_hi[0] + T(2.) * qn);
    }
#pragma unroll
    for (int m = 0; m < 7; ++m) {
        const int q = i - 3 + m;
        T val;
        if (q < 1) val = g_lo[-q];
        else if (q > n) val = g_hi[q - n - 1];
        else val = at(q);
        P[m] = val;
    }
}

// FP32 (the mixed path's arithmetic), the reference's expressions: the derivative at the middle of
// the five divided differences v0..v4 (left-biased; reversed, right-biased).  The weights
// omega_k = (w_k/q_k^2) / sum_m (w_m/q_m^2), q_k = eps + is_k, as three quotients and one
// reciprocal of their sum, each with the hardware reciprocal (__fdividef, 2 ulp; q^2 stays far below
// the 2^126 where it would flush, and a common denominator could underflow), since IEEE FP32
// divisions were a third of the WENO kernels' instructions.
__device__ __forceinline__ float weno_side(float v0, float v1, float v2, float v3, float v4) {
    using T = float;
    const T aux1 = T(13. / 12.), aux2 = T(1. / 4.), aux3 = T(1. / 6.), eps = T(0.00000001);
    const T w1 = T(0.1), w2 = T(0.6), w3 = T(0.3);
    T a, b;
    a = v0 - 2 * v1 + v2; b = v0 - 4 * v1 + 3 * v2;
    const T is1 = aux1 * a * a + aux2 * b * b;
    a = v1 - 2 * v2 + v3; b = v1 - v3;
    const T is2 = aux1 * a * a + aux2 * b * b;
    a = v2 - 2 * v3 + v4; b = 3 * v2 - 4 * v3 + v4;
    const T is3 = aux1 * a * a + aux2 * b * b;
    const T q1 = (eps + is1) * (eps + is1), q2 = (eps + is2) * (eps + is2), q3 = (eps + is3) * (eps + is3);
    const T al1 = __fdividef(w1, q1), al2 = __fdividef(w2, q2), al3 = __fdividef(w3, q3);
    const T inv = __fdividef(T(1), al1 + al2 + al3);
    const T o1 = al1 * inv, o2 = al2 * inv, o3 = al3 * inv;
    return aux3 * (o1 * (2 * v0 - 7 * v1 + 11 * v2) + o2 * (-v1 + 5 * v2 + 2 * v3) + o3 * (2 * v2 + 5 * v3 - v4));
}

// FP64: what the weighted candidates add to v2, from the differences e_m = v_{m+1} - v_m and
// x_k = 12/13 eps + (second difference of stencil k)^2.  q_k = x_k + 3/13 b_k^2 is 12/13 (eps + is_k);
// the factor and the weights' (0.1, 0.6, 0.3) = (1, 6, 3)/10 cancel in the ratios, formed over the
// common denominator q_1^2 q_2^2 q_3^2 (q >= 9e-9, so the products stay far inside the FP64 range).
// Odd in e: the reversed differences, which change sign, give the right-biased side's with -.
constexpr double kWenoEps = 12. / 13. * 0.00000001, kWenoB = 3. / 13.;
__device__ __forceinline__ double weno_blend(double e0, double e1, double e2, double e3, double x1, double x2,
                                             double x3) {
    const double b1 = 3. * e1 - e0, b2 = e1 + e2, b3 = e3 - 3. * e2;
    const double q1 = x1 + (kWenoB * b1) * b1, q2 = x2 + (kWenoB * b2) * b2, q3 = x3 + (kWenoB * b3) * b3;
    const double a = q1 * q1, b = q2 * q2, c = q3 * q3;
    const double n1 = b * c, n2 = 6. * (a * c), n3 = 3. * (a * b);
    const double num = n1 * (5. * e1 - 2. * e0) + n2 * (e1 + 2. * e2) + n3 * (4. * e2 - e3);
    return num * (1. / (6. * (n1 + n2 + n3)));
}
__device__ __forceinline__ double weno_side(double v0, double v1, double v2, double v3, double v4) {
    const double e0 = v1 - v0, e1 = v2 - v1, e2 = v3 - v2, e3 = v4 - v3;
    const double s1 = e1 - e0, s2 = e2 - e1, s3 = e3 - e2;
    return v2 + weno_blend(e0, e1, e2, e3, kWenoEps + s1 * s1, kWenoEps + s2 * s2, kWenoEps + s3 * s3);
}

// One-sided derivatives from the seven values P[0..6] = phi(i-3..i+3) and ih = 1/h (formed
// once on the host, in the compute type): dp = phi_x^+ (dphidxp, right-biased), dn = phi_x^-
// (dphidxn, left-biased).
template <typename T>
__device__ __forceinline__ void weno_pair(const T P[7], T ih, T& dp, T& dn) {
    // D[m] = (phi(i-2+m) - phi(i-3+m))/h; up(i-4..i) = D1..D5, un(i..i+4) = D0..D4
    T D[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) D[m] = (P[m + 1] - P[m]) * ih;
    if constexpr (sizeof(T) == 8) {
        const T e0 = D[1] - D[0], e1 = D[2] - D[1], e2 = D[3] - D[2], e3 = D[4] - D[3], e4 = D[5] - D[4];
        const T s1 = e1 - e0, s2 = e2 - e1, s3 = e3 - e2, s4 = e4 - e3;
        const T x1 = kWenoEps + s1 * s1, x2 = kWenoEps + s2 * s2, x3 = kWenoEps + s3 * s3, x4 = kWenoEps + s4 * s4;
        dn = D[2] + weno_blend(e0, e1, e2, e3, x1, x2, x3);
        dp = D[3] - weno_blend(e4, e3, e2, e1, x4, x3, x2);
    } else {
        dp = weno_side(D[5], D[4], D[3], D[2], D[1]);
        dn = weno_side(D[0], D[1], D[2], D[3], D[4]);
    }
}

// FP64: max(vel, 0) phi_x^- + min(vel, 0) phi_x^+ with the upwind side alone formed (the other has
// the factor 0; its outermost value still enters with that factor, so that one that is not finite
// is carried on).  A transport stage at 191x97x113: 79 -> 58 us; the reinitialisation's nine
// kernels, which need both sides: 612 -> 516 us.
__device__ __forceinline__ double weno_upwind(const double P[7], double ih, double vel) {
    const bool left = vel > 0.;
    double v[6];   // the values from the outermost upwind one on
#pragma unroll
    for (int m = 0; m < 6; ++m) v[m] = left ? P[m] : P[6 - m];
    const double h = left ? ih : -ih;
    const double d = weno_side((v[1] - v[0]) * h, (v[2] - v[1]) * h, (v[3] - v[2]) * h, (v[4] - v[3]) * h, (v[5] - v[4]) * h);
    return vel * (d + 0. * (left ? P[6] : P[0]));
}

}  // namespace suli
