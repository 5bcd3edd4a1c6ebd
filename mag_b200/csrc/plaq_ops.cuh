// plaq_ops.cuh -- stout smearing written on plaquettes and in the Lie algebra.
//
// One plaquette at site x in the plane p < q has the links
//   a = U_p(x), b = U_q(x+p), c = U_p(x+q), d = U_q(x),   P = a b c^dag d^dag,
// and holds a staple of each of them: the loops U stp^dag of its four links are
// P, P^dag and their transports along a and d.  So a sum over the six staples of
// every link (the stout exponent of field-multi.h:32-39, its chain rule
// hep-lat/0311018 eq. 75) is a sum over the six plaquettes of every site, each
// formed once instead of four times.
//
// Only the Lie-algebra part of the chain rule is carried: with the variation of
// a link written as dU = i eta U, a function's derivative is the Hermitian
// traceless x with dS = Tr(eta x) (i TA(U Z) of the matrix derivative Z, eight
// reals instead of eighteen).  One level U' = e^{iQ} U gives
//   dQ : Lambda = phi(-i ad_Q) x',  phi(z) = (e^z - 1) / z,  ad_Q y = [Q, y]
//   U  : x      = e^{-i ad_Q} x' + rho * (plaquette terms of Lambda),
// the projection of compute_Lambda (field-multi.h:180-269) and of Z' e^{iQ}.
#pragma once

#include "gauge_ops.cuh"

namespace magb {

// x / 3, the product with the rounded 1/3 corrected by its remainder (FP32's 1/3 is
// 3e-8 off, always to the same side)
template <typename T>
MAG_HD T third(T x) {
    const T t = x * T(1.0 / 3.0);
    return fmaT(fmaT(T(-3), t, x), T(1.0 / 3.0), t);
}

// i [A, B] of Hermitian traceless matrices (Hermitian traceless)
template <typename T>
MAG_HD herm8<T> comm_i(const herm8<T>& A, const herm8<T>& B) {
    const T a2 = -A.h[0] - A.h[1], b2 = -B.h[0] - B.h[1];
    // Im(A_ij conj(B_ij))
    const T t01 = fmaT(A.h[3], B.h[2], -A.h[2] * B.h[3]);
    const T t02 = fmaT(A.h[5], B.h[4], -A.h[4] * B.h[5]);
    const T t12 = fmaT(A.h[7], B.h[6], -A.h[6] * B.h[7]);
    herm8<T> r;
    r.h[0] = T(-2) * (t01 + t02);
    r.h[1] = T(2) * (t01 - t12);
    const T da01 = A.h[0] - A.h[1], db01 = B.h[0] - B.h[1];
    const T da02 = A.h[0] - a2, db02 = B.h[0] - b2;
    const T da12 = A.h[1] - a2, db12 = B.h[1] - b2;
    // [A, B]_01 = (A00 - A11) B01 - (B00 - B11) A01 + A02 conj(B12) - B02 conj(A12)
    T re = da01 * B.h[2], im = da01 * B.h[3];
    re = fmaT(-db01, A.h[2], re);        im = fmaT(-db01, A.h[3], im);
    re = fmaT(A.h[4], B.h[6], re);       im = fmaT(A.h[5], B.h[6], im);
    re = fmaT(A.h[5], B.h[7], re);       im = fmaT(-A.h[4], B.h[7], im);
    re = fmaT(-B.h[4], A.h[6], re);      im = fmaT(-B.h[5], A.h[6], im);
    re = fmaT(-B.h[5], A.h[7], re);      im = fmaT(B.h[4], A.h[7], im);
    r.h[2] = -im;
    r.h[3] = re;
    // [A, B]_02 = (A00 - A22) B02 - (B00 - B22) A02 + A01 B12 - B01 A12
    re = da02 * B.h[4];                  im = da02 * B.h[5];
    re = fmaT(-db02, A.h[4], re);        im = fmaT(-db02, A.h[5], im);
    re = fmaT(A.h[2], B.h[6], re);       im = fmaT(A.h[2], B.h[7], im);
    re = fmaT(-A.h[3], B.h[7], re);      im = fmaT(A.h[3], B.h[6], im);
    re = fmaT(-B.h[2], A.h[6], re);      im = fmaT(-B.h[2], A.h[7], im);
    re = fmaT(B.h[3], A.h[7], re);       im = fmaT(-B.h[3], A.h[6], im);
    r.h[4] = -im;
    r.h[5] = re;
    // [A, B]_12 = (A11 - A22) B12 - (B11 - B22) A12 + conj(A01) B02 - conj(B01) A02
    re = da12 * B.h[6];                  im = da12 * B.h[7];
    re = fmaT(-db12, A.h[6], re);        im = fmaT(-db12, A.h[7], im);
    re = fmaT(A.h[2], B.h[4], re);       im = fmaT(A.h[2], B.h[5], im);
    re = fmaT(A.h[3], B.h[5], re);       im = fmaT(-A.h[3], B.h[4], im);
    re = fmaT(-B.h[2], A.h[4], re);      im = fmaT(-B.h[2], A.h[5], im);
    re = fmaT(-B.h[3], A.h[5], re);      im = fmaT(B.h[3], A.h[4], im);
    r.h[6] = -im;
    r.h[7] = re;
    return r;
}

// a Hermitian matrix with a trace: diagonal d, off-diagonal z = re, im of 01, 02, 12
template <typename T>
struct herm9 {
    T d[3], z[6];
};
// traceless part of (C M + M C) / 2 for Hermitian C and Hermitian traceless M
template <typename T>
MAG_HD herm8<T> anticomm_half(const herm9<T>& C, const herm8<T>& M) {
    const T c0 = C.d[0], c1 = C.d[1], c2 = C.d[2];
    const T* z = C.z;
    const T m2 = -M.h[0] - M.h[1];
    const T r01 = fmaT(z[0], M.h[2], z[1] * M.h[3]);
    const T r02 = fmaT(z[2], M.h[4], z[3] * M.h[5]);
    const T r12 = fmaT(z[4], M.h[6], z[5] * M.h[7]);
    const T d0 = fmaT(c0, M.h[0], r01 + r02), d1 = fmaT(c1, M.h[1], r01 + r12), d2 = fmaT(c2, m2, r02 + r12);
    const T t = third(d0 + d1 + d2);
    herm8<T> r;
    r.h[0] = d0 - t;
    r.h[1] = d1 - t;
    // 01: [(C00 + C11) M01 + (M00 + M11) C01 + C02 conj(M12) + M02 conj(C12)] / 2
    T s = c0 + c1, re = s * M.h[2], im = s * M.h[3];
    re = fmaT(-m2, z[0], re);            im = fmaT(-m2, z[1], im);
    re = fmaT(z[2], M.h[6], re);         im = fmaT(z[3], M.h[6], im);
    re = fmaT(z[3], M.h[7], re);         im = fmaT(-z[2], M.h[7], im);
    re = fmaT(M.h[4], z[4], re);         im = fmaT(M.h[5], z[4], im);
    re = fmaT(M.h[5], z[5], re);         im = fmaT(-M.h[4], z[5], im);
    r.h[2] = T(0.5) * re;
    r.h[3] = T(0.5) * im;
    // 02: [(C00 + C22) M02 + (M00 + M22) C02 + C01 M12 + M01 C12] / 2
    s = c0 + c2;
    re = s * M.h[4];                     im = s * M.h[5];
    re = fmaT(-M.h[1], z[2], re);        im = fmaT(-M.h[1], z[3], im);
    re = fmaT(z[0], M.h[6], re);         im = fmaT(z[0], M.h[7], im);
    re = fmaT(-z[1], M.h[7], re);        im = fmaT(z[1], M.h[6], im);
    re = fmaT(M.h[2], z[4], re);         im = fmaT(M.h[2], z[5], im);
    re = fmaT(-M.h[3], z[5], re);        im = fmaT(M.h[3], z[4], im);
    r.h[4] = T(0.5) * re;
    r.h[5] = T(0.5) * im;
    // 12: [(C11 + C22) M12 + (M11 + M22) C12 + conj(C01) M02 + conj(M01) C02] / 2
    s = c1 + c2;
    re = s * M.h[6];                     im = s * M.h[7];
    re = fmaT(-M.h[0], z[4], re);        im = fmaT(-M.h[0], z[5], im);
    re = fmaT(z[0], M.h[4], re);         im = fmaT(z[0], M.h[5], im);
    re = fmaT(z[1], M.h[5], re);         im = fmaT(-z[1], M.h[4], im);
    re = fmaT(M.h[2], z[2], re);         im = fmaT(M.h[2], z[3], im);
    re = fmaT(M.h[3], z[3], re);         im = fmaT(-M.h[3], z[2], im);
    r.h[6] = T(0.5) * re;
    r.h[7] = T(0.5) * im;
    return r;
}

// t = (u0, u1, u2) H, a row times a Hermitian traceless matrix
template <typename T>
MAG_HD void row_times_herm(cplx<T> u0, cplx<T> u1, cplx<T> u2, const herm8<T>& H, cplx<T> t[3]) {
    const cplx<T> z01 = mk(H.h[2], H.h[3]), z02 = mk(H.h[4], H.h[5]), z12 = mk(H.h[6], H.h[7]);
    const T h2 = -H.h[0] - H.h[1];
    t[0] = mk(u0.re * H.h[0], u0.im * H.h[0]);
    cmac<false, true, false>(t[0], u1, z01);
    cmac<false, true, false>(t[0], u2, z02);
    t[1] = mk(u1.re * H.h[1], u1.im * H.h[1]);
    cmac<false, false, false>(t[1], u0, z01);
    cmac<false, true, false>(t[1], u2, z12);
    t[2] = mk(u2.re * h2, u2.im * h2);
    cmac<false, false, false>(t[2], u0, z02);
    cmac<false, false, false>(t[2], u1, z12);
}
// Re(t0 u0 + t1 u1 + t2 u2)
template <typename T>
MAG_HD T dot_re(const cplx<T> t[3], cplx<T> u0, cplx<T> u1, cplx<T> u2) {
    T s = t[0].re * u0.re;
    s = fmaT(-t[0].im, u0.im, s);
    s = fmaT(t[1].re, u1.re, s);
    s = fmaT(-t[1].im, u1.im, s);
    s = fmaT(t[2].re, u2.re, s);
    return fmaT(-t[2].im, u2.im, s);
}
template <typename T>
MAG_HD cplx<T> dot_c(const cplx<T> t[3], cplx<T> u0, cplx<T> u1, cplx<T> u2) {
    cplx<T> s = cmul<false, false>(t[0], u0);
    cmac<false, false, false>(s, t[1], u1);
    cmac<false, false, false>(s, t[2], u2);
    return s;
}
// U H U^dag and U^dag H U of a Hermitian traceless H and a unitary U: rows 0, 1 of
// the first product and the five independent elements of the second
template <typename T>
MAG_HD herm8<T> transport_nd(const mat3<T>& U, const herm8<T>& H) {
    cplx<T> t[3];
    herm8<T> r;
    row_times_herm(U.e[0][0], U.e[0][1], U.e[0][2], H, t);
    r.h[0] = dot_re(t, conj(U.e[0][0]), conj(U.e[0][1]), conj(U.e[0][2]));
    cplx<T> z = dot_c(t, conj(U.e[1][0]), conj(U.e[1][1]), conj(U.e[1][2]));
    r.h[2] = z.re;
    r.h[3] = z.im;
    z = dot_c(t, conj(U.e[2][0]), conj(U.e[2][1]), conj(U.e[2][2]));
    r.h[4] = z.re;
    r.h[5] = z.im;
    row_times_herm(U.e[1][0], U.e[1][1], U.e[1][2], H, t);
    r.h[1] = dot_re(t, conj(U.e[1][0]), conj(U.e[1][1]), conj(U.e[1][2]));
    z = dot_c(t, conj(U.e[2][0]), conj(U.e[2][1]), conj(U.e[2][2]));
    r.h[6] = z.re;
    r.h[7] = z.im;
    return r;
}
template <typename T>
MAG_HD herm8<T> transport_dn(const mat3<T>& U, const herm8<T>& H) {
    cplx<T> t[3];
    herm8<T> r;
    row_times_herm(conj(U.e[0][0]), conj(U.e[1][0]), conj(U.e[2][0]), H, t);
    r.h[0] = dot_re(t, U.e[0][0], U.e[1][0], U.e[2][0]);
    cplx<T> z = dot_c(t, U.e[0][1], U.e[1][1], U.e[2][1]);
    r.h[2] = z.re;
    r.h[3] = z.im;
    z = dot_c(t, U.e[0][2], U.e[1][2], U.e[2][2]);
    r.h[4] = z.re;
    r.h[5] = z.im;
    row_times_herm(conj(U.e[0][1]), conj(U.e[1][1]), conj(U.e[2][1]), H, t);
    r.h[1] = dot_re(t, U.e[0][1], U.e[1][1], U.e[2][1]);
    z = dot_c(t, U.e[0][2], U.e[1][2], U.e[2][2]);
    r.h[6] = z.re;
    r.h[7] = z.im;
    return r;
}

// r (+)= s y
template <typename T>
MAG_HD void herm_axpy(herm8<T>& r, T s, const herm8<T>& y) {
#pragma unroll
    for (int k = 0; k < 8; k++) r.h[k] = fmaT(s, y.h[k], r.h[k]);
}
template <typename T>
MAG_HD void herm_add(herm8<T>& r, const herm8<T>& y) {
#pragma unroll
    for (int k = 0; k < 8; k++) r.h[k] += y.h[k];
}
template <typename T>
MAG_HD void herm_sub(herm8<T>& r, const herm8<T>& y) {
#pragma unroll
    for (int k = 0; k < 8; k++) r.h[k] -= y.h[k];
}

// a b, rounded: not contracted with an addition that follows, so that kernels that add up the
// same terms agree to the bit whatever the compiler makes of each.  Also 1% faster in the FP64
// rectangle kernel (32^4: 1.304 -> 1.288 ms with k_plaq): the product that is needed by itself
// as well is not formed twice
MAG_HD double mul_rnT(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
MAG_HD float mul_rnT(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}

// Hermitian traceless part of (P - P^dag) / 2i, times s
template <typename T>
MAG_HD herm8<T> plaq_sin(const mat3<T>& P, T s) {
    const T t = third(P.e[0][0].im + P.e[1][1].im + P.e[2][2].im), h = T(0.5) * s;
    herm8<T> r;
    r.h[0] = mul_rnT(s, P.e[0][0].im - t);
    r.h[1] = mul_rnT(s, P.e[1][1].im - t);
    r.h[2] = mul_rnT(h, P.e[0][1].im + P.e[1][0].im);
    r.h[3] = mul_rnT(h, P.e[1][0].re - P.e[0][1].re);
    r.h[4] = mul_rnT(h, P.e[0][2].im + P.e[2][0].im);
    r.h[5] = mul_rnT(h, P.e[2][0].re - P.e[0][2].re);
    r.h[6] = mul_rnT(h, P.e[1][2].im + P.e[2][1].im);
    r.h[7] = mul_rnT(h, P.e[2][1].re - P.e[1][2].re);
    return r;
}

template <typename T>
MAG_HD herm8<T> herm_convert(const herm8<double>& a) {
    herm8<T> r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.h[k] = (T)a.h[k];
    return r;
}

// (P + P^dag) / 2, times s
template <typename T>
MAG_HD herm9<T> plaq_cos(const mat3<T>& P, T s) {
    const T h = T(0.5) * s;
    herm9<T> r;
#pragma unroll
    for (int i = 0; i < 3; i++) r.d[i] = s * P.e[i][i].re;
    r.z[0] = h * (P.e[0][1].re + P.e[1][0].re);
    r.z[1] = h * (P.e[0][1].im - P.e[1][0].im);
    r.z[2] = h * (P.e[0][2].re + P.e[2][0].re);
    r.z[3] = h * (P.e[0][2].im - P.e[2][0].im);
    r.z[4] = h * (P.e[1][2].re + P.e[2][1].re);
    r.z[5] = h * (P.e[1][2].im - P.e[2][1].im);
    return r;
}

// The plaquette P = a b c^dag d^dag (special unitary links: two rows multiplied)
template <typename T>
MAG_HD mat3<T> plaquette(const mat3<T>& a, const mat3<T>& b, const mat3<T>& c, const mat3<T>& d) {
    const mat3<T> x = mul_2r(a, b);
    const mat3<T> y = mul_su3(d, c);
    return mul_nd_su3(x, y);
}

// The same where its sine is a term of the force by itself: in single precision the two halves
// with all their rows and the last product in double, so that P carries their roundings only.
// A third row rebuilt from two rounded ones has twice their error, and the terms are weighted by
// c0 = 3.6.  Error of the thin Iwasaki force of hot links 1.52 -> 1.28e-7 with this and with the
// gather's sums in double (one thread per link: 1.31); the plaquette kernels 0.71 -> 0.73 ms at 32^4.
MAG_HD mat3<double> plaquette_wide(const LinkPlanes<double>& U, int g, int gp, int gq, int p, int q) {
    return plaquette(U.load_rows01(p, g), U.load(q, gp), U.load(p, gq), U.load_rows01(q, g));
}
MAG_HD mat3<double> plaquette_wide(const LinkPlanes<float>& U, int g, int gp, int gq, int p, int q) {
    const mat3<float> x = mul(U.load(p, g), U.load(q, gp));
    const mat3<float> y = mul(U.load(q, g), U.load(p, gq));
    return mul_nd(convert<double>(x), convert<double>(y));
}

// e^{iQ} U = (f0 + f1 Q + f2 Q^2) U of a special unitary U: rows 0, 1 of e^{iQ} and of
// the product, the third reconstructed; the coefficients are those of expiQ
MAG_HD mat3<double> exp_times(const herm8<double>& q, const mat3<double>& U) {
    const double h0 = q.h[0], h1 = q.h[1], h2 = -q.h[0] - q.h[1];
    const cplx<double> z01 = mk(q.h[2], q.h[3]), z02 = mk(q.h[4], q.h[5]), z12 = mk(q.h[6], q.h[7]);
    const double n01 = fmaT(z01.re, z01.re, z01.im * z01.im);
    const double n02 = fmaT(z02.re, z02.re, z02.im * z02.im);
    const double n12 = fmaT(z12.re, z12.re, z12.im * z12.im);
    // rows 0, 1 of Q^2 (Hermitian): 00, 11 and 01, 02, 12
    const double s00 = fmaT(h0, h0, n01 + n02), s11 = fmaT(h1, h1, n01 + n12), s22 = fmaT(h2, h2, n02 + n12);
    cplx<double> s01 = mk(-h2 * z01.re, -h2 * z01.im), s02 = mk(-h1 * z02.re, -h1 * z02.im),
            s12 = mk(-h0 * z12.re, -h0 * z12.im);
    cmac<false, true, false>(s01, z02, z12);
    cmac<false, false, false>(s02, z01, z12);
    cmac<true, false, false>(s12, z01, z02);
    const double c1 = 0.5 * (s00 + s11 + s22);
    if (c1 == 0.0) return U;  // the reference's c1 = 0 branch (field-hmc.h:95)
    // det Q = Tr Q^3 / 3
    const cplx<double> p = cmul<false, false>(z01, z12);
    double c0 = fmaT(p.re, z02.re, p.im * z02.im);
    c0 = fmaT(2.0, c0, h0 * h1 * h2);
    c0 = fmaT(-h0, n12, c0);
    c0 = fmaT(-h1, n02, c0);
    c0 = fmaT(-h2, n01, c0);
    double f[6];
    if (!ch_series_exp_d(c0, c1, f)) {
        const ch_coef c = ch_coefficients<false>(c0, c1);
        f[0] = c.f0r, f[1] = c.f0i;
        f[2] = c.f1r, f[3] = c.f1i;
        f[4] = c.f2r, f[5] = c.f2i;
    }
    const cplx<double> f0 = mk(f[0], f[1]), f1 = mk(f[2], f[3]), f2 = mk(f[4], f[5]);
    mat3<double> e;
    auto diag = [&](double x, double s) { return mk(fmaT(f2.re, s, fmaT(f1.re, x, f0.re)), fmaT(f2.im, s, fmaT(f1.im, x, f0.im))); };
    auto off = [&](cplx<double> x, cplx<double> s) {
        cplx<double> r = cmul<false, false>(f1, x);
        cmac<false, false, false>(r, f2, s);
        return r;
    };
    e.e[0][0] = diag(h0, s00);
    e.e[0][1] = off(z01, s01);
    e.e[0][2] = off(z02, s02);
    e.e[1][0] = off(conj(z01), conj(s01));
    e.e[1][1] = diag(h1, s11);
    e.e[1][2] = off(z12, s12);
    return mul_su3(e, U);
}

// y <- prod_{j=1..n} (1 + e^{-i ad_Q / 2^j}) / 2 y, so that phi(-i ad_Q) x =
// phi(-i ad_Q / 2^n) y from y = x (phi(2z) = phi(z) (1 + e^z) / 2).  Out of line: only
// |Q| beyond the series of lambda_adjoint comes here, and the exponential's registers
// would set the caller's.
template <typename T>
#if defined(__CUDACC__)
__host__ __device__ __noinline__
#endif
    void
    half_angles(const herm8<T>& q, int n, herm8<T>& y) {
    T s = T(1);
    for (int j = 0; j < n; j++) {
        s *= T(0.5);
        const herm8<T> r = transport_dn(expiQ(scaled(q, s)), y);
        for (int k = 0; k < 8; k++) y.h[k] = T(0.5) * (y.h[k] + r.h[k]);
    }
}

// Tr Q^2 / 2
template <typename T>
MAG_HD T herm_c1(const herm8<T>& q) {
    const T q2 = -q.h[0] - q.h[1];
    T n = q.h[2] * q.h[2];
#pragma unroll
    for (int k = 3; k < 8; k++) n = fmaT(q.h[k], q.h[k], n);
    return fmaT(T(0.5), q.h[0] * q.h[0] + q.h[1] * q.h[1] + q2 * q2, n);
}

// Lambda = phi(-i ad_Q) x and dir = e^{-i ad_Q} x = x - i [Q, Lambda].
// m = (-i ad_Q)^2 has the eigenvalues -(l_i - l_j)^2 and satisfies, on the range of
// ad_Q, m^3 + e1 m^2 + e2 m + e3 = 0 with e1 = 6 c1, e2 = 9 c1^2, e3 = 4 c1^3 -
// 27 c0^2 (c0 = det Q, c1 = Tr Q^2 / 2; the cubic of the squared eigenvalue
// differences).  So phi is a polynomial of degree six in -i ad_Q whose
// coefficients sum_k m^k / (2k + 2)! and / (2k + 3)! are summed from the power
// series reduced by that recursion: six commutators of eight reals, no
// transcendental function and no division by small differences.  The series stops
// once z^2k / (2k + 2)!, z = 2 sqrt(c1) >= |l_i - l_j|, is below the type's
// rounding; z > 3 is halved first (half_angles).  c1 = 0 gives Lambda = 0 as the
// reference returns (field-multi.h:190).
template <typename T>
MAG_HD void lambda_adjoint(herm8<T> q, const herm8<T>& x, herm8<T>& lam, herm8<T>& dir) {
    T c1 = herm_c1(q);
    if (c1 == T(0)) {
        lam = herm_zero<T>();
        dir = x;
        return;
    }
    herm8<T> r = x;
    T full = T(1);
    if (T(4) * c1 > T(9)) {
        int n = 0;
        for (; T(4) * c1 > T(9) && n < 64; n++) {
            c1 *= T(0.25);
            full *= T(2);
        }
        half_angles(q, n, r);
        q = scaled(q, T(1) / full);
    }
    const T w = T(4) * c1;
    const T q2 = -q.h[0] - q.h[1];
    const T n01 = fmaT(q.h[2], q.h[2], q.h[3] * q.h[3]);
    const T n02 = fmaT(q.h[4], q.h[4], q.h[5] * q.h[5]);
    const T n12 = fmaT(q.h[6], q.h[6], q.h[7] * q.h[7]);
    // det Q = h0 h1 h2 + 2 Re(z01 z12 conj(z02)) - h0 |z12|^2 - h1 |z02|^2 - h2 |z01|^2
    const T pr = q.h[2] * q.h[6] - q.h[3] * q.h[7], pi = q.h[2] * q.h[7] + q.h[3] * q.h[6];
    const T c0 = q.h[0] * q.h[1] * q2 + T(2) * (pr * q.h[4] + pi * q.h[5]) - q.h[0] * n12 - q.h[1] * n02 - q2 * n01;
    const T e1 = T(6) * c1, e2 = T(9) * c1 * c1, e3 = T(4) * c1 * c1 * c1 - T(27) * c0 * c0;
    // odd powers o[j] of -i ad_Q (1, 3, 5) and even ones s[j] (2, 4, 6)
    T o0 = T(1.0 / 2.0), o1 = T(1.0 / 24.0), o2 = T(1.0 / 720.0);
    T s0 = T(1.0 / 6.0), s1 = T(1.0 / 120.0), s2 = T(1.0 / 5040.0);
    T al = T(0), be = T(0), ga = T(1);  // m^2
    T fo = T(1.0 / 720.0), bound = w * w * T(1.0 / 720.0);
    const T eps = sizeof(T) == 8 ? T(1e-17) : T(1e-9);
#pragma unroll
    for (int k = 3; k < 16; k++) {
        if (bound < eps) break;
        const T na = -e3 * ga, nb_ = fmaT(-e2, ga, al), ng = fmaT(-e1, ga, be);
        al = na;
        be = nb_;
        ga = ng;
        fo *= T(1.0 / ((2 * k + 1) * (2 * k + 2)));
        bound *= w * T(1.0 / ((2 * k + 1) * (2 * k + 2)));
        const T fs = fo * T(1.0 / (2 * k + 3));
        o0 = fmaT(fo, al, o0);
        o1 = fmaT(fo, be, o1);
        o2 = fmaT(fo, ga, o2);
        s0 = fmaT(fs, al, s0);
        s1 = fmaT(fs, be, s1);
        s2 = fmaT(fs, ga, s2);
    }
    // t <- -i [Q, t] = i [t, Q]
    herm8<T> t = comm_i(r, q);
    herm_axpy(r, o0, t);
    t = comm_i(t, q);
    herm_axpy(r, s0, t);
    t = comm_i(t, q);
    herm_axpy(r, o1, t);
    t = comm_i(t, q);
    herm_axpy(r, s1, t);
    t = comm_i(t, q);
    herm_axpy(r, o2, t);
    t = comm_i(t, q);
    herm_axpy(r, s2, t);
    lam = r;
    dir = x;
    herm_axpy(dir, full, comm_i(r, q));
}

}  // namespace magb
