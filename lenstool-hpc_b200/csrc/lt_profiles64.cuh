/*
 * lt_profiles64.cuh -- FP64 per-pair Hessian arithmetic (one halo record, one pixel): the
 * reference's quotient form with reciprocals (the FP32C path's FP64 pairs), its exact rounding
 * sequence (LT_FP64), and the closed form of the FP32C recomputation.  The deflection, the
 * potential and LT_FP64_FAST's Hessian are in lt_closed64.cuh.
 *
 *   Hessian:     dPIE src/gradient2.cpp:92-205 with mdci05 :54-83; PIEMD = one mdci05
 *                term; SIS = derivative of the SIS deflection (restated)
 */
#pragma once
#include "lt_halo.h"

namespace lt {

/* Reciprocal and reciprocal square root for the per-pair denominators: the hardware
 * approximations (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64; ~20 correct bits) refined by one
 * third-order step: with e = 1 - x y, 1/x = y/(1 - e) = y (1 + e + e^2 + O(e^3)); with
 * h = 1 - x y^2, 1/sqrt(x) = y (1 - h)^(-1/2) = y (1 + h/2 + 3 h^2/8 + O(h^3)).  The
 * truncation is ~e^3 (~1e-18), so the result is within a few ulp of the correctly rounded
 * value for positive normal inputs (checked against 1/x and 1/sqrt(x) by the tests).
 * Three FP64 operations for a reciprocal and five for a reciprocal square root (two
 * Newton steps take four and eight), and one approximation, instead of the IEEE division
 * and square-root sequences. */
__device__ __forceinline__ double rcp64(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double rsqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = fma(-x * y, y, 1.0);
    return fma(y * h, fma(0.375, h, 0.5), y);
}

struct Frame64 {
    double u, v;
};

/* Offset from the halo centre rotated into the halo frame (x' = x cos + y sin,
 * y' = y cos - x sin; src/gradient.hpp:29-37). */
__device__ __forceinline__ Frame64 to_frame(const lt_rec64 &h, double px, double py)
{
    double tx = px - h.x0, ty = py - h.y0;
    Frame64 f;
    f.u = tx * h.cs + ty * h.sn;
    f.v = ty * h.cs - tx * h.sn;
    return f;
}

/* ------------------------------------------------------------------- Hessian ---- */

struct Hess64 {
    double xx, yy, xy;
};

/* The three bracketed terms of mdci05 (didxre, didyre, didyim without the factor ci).
 * With t1 = 2 sqrt(e) w - v/cx1 (the small factor of den1 near the removable singular
 * point u = 0, v = 2 r sqrt(e)), the numerators factor exactly:
 *   didxre: cx1 (2 sqrt(e) u^2/((1+e)^2 w) - t1)
 *   didyre: u (2 sqrt(e) v cx1/((1-e)^2 w) - 1)
 *   didyim: t1 (1/cx1 - 2 sqrt(e) v/((1-e)^2 w))
 * (for didyim, 4e = (2 sqrt(e))^2 turns the reference's four terms into the product), so
 * numerator and denominator share one rounded t1 and the numerators cancel no digits. */
__device__ __forceinline__ void mdci05_terms(const lt_rec64 &h, double u, double uu, double v, double vv,
                                             double vq, double rem2, double r2, double tsr, double &X, double &Y,
                                             double &Z)
{
    (void)vv;
    const double q = r2 + rem2;
    double iw = rsqrt64(q);
    double wrem = q * iw;
    double t1 = h.sqe2 * wrem - vq;
    double den1 = h.cx1 * h.cx1 * uu + t1 * t1;
    double num2 = tsr - v;
    double den2 = uu + num2 * num2;
    double i1 = rcp64(den1);
    double i2 = rcp64(den2);
    double sv = h.sqe2 * v * h.cyro_inv * iw;
    X = h.cx1 * (h.sqe2 * uu * h.cxro_inv * iw - t1) * i1 + num2 * i2;
    Y = u * (sv * h.cx1 - 1.0) * i1 + u * i2;
    Z = t1 * (h.cx1inv - sv) * i1 - num2 * i2;
}

/* H = R^T H' R for the symmetric halo-frame Hessian H' = [[a, b], [b, c]]; the
 * reference applies the same rotation in two steps (src/gradient2.cpp:146-156). */
__device__ __forceinline__ void rotate_acc(const lt_rec64 &h, double a, double b, double c, double w, Hess64 &acc)
{
    double cs = h.cs, sn = h.sn;
    double cc = cs * cs, ss = sn * sn, csn = cs * sn;
    acc.xx += w * (a * cc - 2. * b * csn + c * ss);
    acc.yy += w * (a * ss + 2. * b * csn + c * cc);
    acc.xy += w * ((a - c) * csn + b * (cc - ss));
}

template <int TYPE>
__device__ __forceinline__ void hess_pair(const lt_rec64 &h, double px, double py, double w, Hess64 &acc)
{
    Frame64 f = to_frame(h, px, py);
    double u = f.u, v = f.v;
    double uu = u * u, vv = v * v;
    if (TYPE == 5) {
        double q = uu * h.cx1 + vv * h.cx1inv;
        double rs = rsqrt64(q);
        double k = h.ci * (rs * rs * rs);
        rotate_acc(h, k * vv, -k * u * v, k * uu, w, acc);
    } else {
        double rem2 = uu * h.cxro_inv + vv * h.cyro_inv;
        double vq = v * h.cx1inv;
        double X, Y, Z;
        mdci05_terms(h, u, uu, v, vv, vq, rem2, h.rc2, h.tsr_c, X, Y, Z);
        if (TYPE == 81) {
            double X2, Y2, Z2;
            mdci05_terms(h, u, uu, v, vv, vq, rem2, h.rcut2, h.tsr_t, X2, Y2, Z2);
            X -= X2;
            Y -= Y2;
            Z -= Z2;
        }
        rotate_acc(h, h.pref_h * X, h.pref_h * Y, h.pref_h * Z, w, acc);
    }
}

} // namespace lt

/* ------------------------------------------------ reference-exact Hessian ---- */
/* The reference's Hessian arithmetic with its rounding sequence: every operation is a
 * separately rounded IEEE operation (no contraction into FMA, true division and square
 * root), in C's left-to-right evaluation order.  The results are bit-identical to the
 * reference FP64 CPU path (src/gradient2.cpp:54-205), whose formula is ill-conditioned
 * near each halo's removable singular points and near small-ellipticity cores: any other
 * rounding sequence differs there by up to ~1e-12 of the map scale. */
namespace lt {
namespace ex {
__device__ __forceinline__ double M(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double A(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double S(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double V(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double R(double a) { return __dsqrt_rn(a); }

struct Mat {
    double a, b, c, d;
};

/* mdci05_hpc, src/gradient2.cpp:54-83, by IEEE division and square root */
__device__ __forceinline__ Mat mdci05(double x, double y, double eps, double rc, double b0)
{
    const double sqe = R(eps);
    const double cx1 = V(S(1., eps), A(1., eps));
    const double cx1inv = V(1., cx1);
    const double cxro = M(A(1., eps), A(1., eps));
    const double cyro = M(S(1., eps), S(1., eps));
    const double ci = V(M(0.5, S(1., M(eps, eps))), sqe);
    const double wrem = R(A(A(M(rc, rc), V(M(x, x), cxro)), V(M(y, y), cyro)));
    const double sq2 = M(2., sqe);
    double den1 = S(M(sq2, wrem), M(y, cx1inv));
    den1 = A(M(M(M(cx1, cx1), x), x), M(den1, den1));
    const double num2 = S(M(M(2., rc), sqe), y);
    const double den2 = A(M(x, x), M(num2, num2));
    double t = A(S(V(V(M(M(sq2, x), x), cxro), wrem), M(sq2, wrem)), M(y, cx1inv));
    const double didxre = M(ci, A(V(M(cx1, t), den1), V(num2, den2)));
    t = S(V(V(M(M(M(sq2, x), y), cx1), cyro), wrem), x);
    const double didyre = M(ci, A(V(t, den1), V(x, den2)));
    t = S(M(M(sq2, wrem), cx1inv), M(M(y, cx1inv), cx1inv));
    t = S(t, V(M(M(4., eps), y), cyro));
    t = A(t, M(V(V(M(M(sq2, y), y), cyro), wrem), cx1inv));
    const double didyim = M(ci, S(V(t, den1), V(num2, den2)));
    Mat r;
    r.a = M(b0, didxre);
    r.b = r.d = M(b0, didyre);
    r.c = M(b0, didyim);
    return r;
}

/* Correctly rounded quotients that share a divisor (P. Markstein, "Computation of elementary
 * functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): with
 * y = RN(1/b), q = RN(a y) and the exact remainder r = a - q b, RN(q + r y) = RN(a/b).  Three
 * operations a division instead of an IEEE division sequence each; the reference form divides
 * three times by den1, three times by wrem and twice by den2 per radius.
 *   rcp_rn: rcp64 is within half an ulp and 2^-7; one more Newton step gives RN(1/b) unless
 *     b's significand is all ones.
 *   sqrt_rn: from y within an ulp of 1/sqrt(x), two remainder steps give w = RN(sqrt(x)) and
 *     RN(1/w), unless w's significand is all ones (x's then ends in 11..10 or 11..11).
 * tests/test_hess_exact.py repeats these steps on every operand of small precisions.  The
 * operands they do not cover (those, and values near the ends of the exponent range, where a
 * remainder is not exact) are found by `Odd` and go through mdci05. */
__device__ __forceinline__ double quot(double a, double b, double y)
{
    const double q = M(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}
__device__ __forceinline__ double rcp_rn(double b)
{
    const double y = rcp64(b);
    return __fma_rn(__fma_rn(-b, y, 1.), y, y);
}
/* y/2 for a normal y, off the FP64 pipe */
__device__ __forceinline__ double half_of(double y)
{
    return __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));
}
__device__ __forceinline__ void sqrt_rn(double x, double &w, double &iw)
{
    const double y = rsqrt64(x);
    const double g = M(x, y);
    const double g1 = __fma_rn(__fma_rn(-g, g, x), half_of(y), g);
    const double y1 = __fma_rn(__fma_rn(-g1, y, 1.), y, y);
    w = __fma_rn(__fma_rn(-g1, g1, x), half_of(y1), g1);
    iw = __fma_rn(__fma_rn(-w, y1, 1.), y1, y1);
}

/* Running extremes of the bit patterns that the steps above do not cover. */
struct Odd {
    uint32_t lo = 0, hi = 0, hn = 0xffffffffu;
    __device__ __forceinline__ void divisor(double b)
    {
        lo = max(lo, (uint32_t)__double2loint(b));
        const uint32_t h = (uint32_t)__double2hiint(b);
        hi = max(hi, h);
        hn = min(hn, h);
    }
    __device__ __forceinline__ void offset(double u) /* 0, or not below 2^-400 */
    {
        hn = min(hn, ((uint32_t)__double2hiint(u) & 0x7fffffffu) - 1u);
    }
    /* significand's low word 11..10 or 11..11, a divisor (positive) above 2^800 or not
     * finite, below 2^-400 */
    __device__ __forceinline__ bool any() const { return lo >= 0xfffffffeu || hi > 0x71f00000u || hn < 0x26f00000u; }
};

/* What the two radii of a pair share: the reference's sub-expressions in x, y and the halo's
 * constants (record lt_rec64, the same roundings). */
struct MdShared {
    double xx, xxc, yyc, X1, Y1, Z1, Z2, yc, ycc, cxx;
};
__device__ __forceinline__ MdShared md_shared(const lt_rec64 &h, double x, double y)
{
    MdShared s;
    s.xx = M(x, x);
    s.xxc = quot(s.xx, h.cxro, h.cxro_inv);
    s.yyc = quot(M(y, y), h.cyro, h.cyro_inv);
    const double sx = M(h.sqe2, x);
    s.X1 = quot(M(sx, x), h.cxro, h.cxro_inv);
    s.Y1 = quot(M(M(sx, y), h.cx1), h.cyro, h.cyro_inv);
    s.Z1 = quot(M(M(h.sqe2, y), y), h.cyro, h.cyro_inv);
    s.Z2 = quot(M(h.k4, y), h.cyro, h.cyro_inv);
    s.yc = M(y, h.cx1inv);
    s.ycc = M(s.yc, h.cx1inv);
    s.cxx = M(M(h.cx1sq, x), x);
    return s;
}
__device__ __forceinline__ Mat mdci05(const lt_rec64 &h, const MdShared &s, double x, double y, double r2, double tsr,
                                      Odd &odd)
{
    const double w2 = A(A(r2, s.xxc), s.yyc);
    double w, iw;
    sqrt_rn(w2, w, iw);
    const double sw = M(h.sqe2, w);
    const double d1 = S(sw, s.yc);
    const double den1 = A(s.cxx, M(d1, d1));
    const double num2 = S(tsr, y);
    const double den2 = A(s.xx, M(num2, num2));
    const double i1 = rcp_rn(den1), i2 = rcp_rn(den2);
    const double n2 = quot(num2, den2, i2);
    double t = A(S(quot(s.X1, w, iw), sw), s.yc);
    const double didxre = M(h.ci, A(quot(M(h.cx1, t), den1, i1), n2));
    t = S(quot(s.Y1, w, iw), x);
    const double didyre = M(h.ci, A(quot(t, den1, i1), quot(x, den2, i2)));
    t = S(S(M(sw, h.cx1inv), s.ycc), s.Z2);
    t = A(t, M(quot(s.Z1, w, iw), h.cx1inv));
    const double didyim = M(h.ci, S(quot(t, den1, i1), n2));
    odd.divisor(w2);
    odd.divisor(w);
    odd.divisor(den1);
    odd.divisor(den2);
    Mat r;
    r.a = M(h.b0, didxre);
    r.b = r.d = M(h.b0, didyre);
    r.c = M(h.b0, didyim);
    return r;
}

/* two-step rotation back to the sky frame, src/gradient2.cpp:146-156 */
__device__ __forceinline__ void rotate_acc(const Mat &h, double cs, double sn, Mat &acc)
{
    const double ma = A(M(h.a, cs), M(h.b, -sn));
    const double mb = A(M(h.a, sn), M(h.b, cs));
    const double mc = A(M(h.d, sn), M(h.c, cs));
    const double md = A(M(h.d, cs), M(h.c, -sn));
    acc.a = A(acc.a, S(M(cs, ma), M(sn, md)));
    acc.b = A(acc.b, S(M(cs, mb), M(sn, mc)));
    acc.c = A(acc.c, A(M(sn, mb), M(cs, mc)));
    acc.d = A(acc.d, A(M(sn, ma), M(cs, md)));
}

/* One halo's halo-frame Hessian by IEEE operations (dPIE src/gradient2.cpp:92-205, PIEMD = one
 * mdci05 term): the pairs with an odd operand, out of line. */
template <int TYPE>
__device__ __noinline__ void hess_ieee(const lt_rec64 &h, double u, double v, Mat &m)
{
    m = mdci05(u, v, h.eps, h.rc, h.b0);
    if (TYPE == 81) {
        const double t05 = V(h.rcut, S(h.rcut, h.rc));
        const Mat cut = mdci05(u, v, h.eps, h.rcut, h.b0);
        m.a = M(t05, S(m.a, cut.a));
        m.b = M(t05, S(m.b, cut.b));
        m.c = M(t05, S(m.c, cut.c));
        m.d = M(t05, S(m.d, cut.d));
    }
}

/* One halo's halo-frame Hessian at offset (u, v) with the reference's roundings; false where an
 * operand is odd (hess_ieee then gives it).  SIS restated with the same rounding discipline. */
template <int TYPE>
__device__ __forceinline__ bool hess_frame(const lt_rec64 &h, double u, double v, Mat &m)
{
    if (TYPE == 5) {
        const double e = h.eps;
        const double q = A(M(M(u, u), S(1., e)), M(M(v, v), A(1., e)));
        const double r = R(q);
        const double k = V(M(M(h.b0, S(1., e)), A(1., e)), M(q, r));
        m.a = M(M(k, v), v);
        m.c = M(M(k, u), u);
        m.b = m.d = M(M(-k, u), v);
        return true;
    }
    Odd odd;
    odd.offset(u);
    odd.offset(v);
    const MdShared s = md_shared(h, u, v);
    m = mdci05(h, s, u, v, h.rc2, h.tsr_c, odd);
    if (TYPE == 81) {
        const Mat cut = mdci05(h, s, u, v, h.rcut2, h.tsr_t, odd);
        m.a = M(h.t05, S(m.a, cut.a));
        m.b = m.d = M(h.t05, S(m.b, cut.b));
        m.c = M(h.t05, S(m.c, cut.c));
    }
    return !odd.any();
}

/* The Hessians of U records at P pixels of a row added, in their order, to the run accumulators.
 * 220 FP64 operations a dPIE pair; the odd operands' branch is taken once in ~10^9 pairs.  The
 * U P pairs are independent chains that interleave (U = 2 where a grid is too small to fill the
 * SMs with warps). */
template <int TYPE, int P, int U>
__device__ __forceinline__ void hess_pairs(const lt_rec64 *h, const double (&px)[P], double py, Mat (&acc)[P])
{
    double u[U][P], v[U][P];
    Mat m[U][P];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < U; i++) {
        const double ty = S(py, h[i].y0);
#pragma unroll
        for (int k = 0; k < P; k++) {
            const double tx = S(px[k], h[i].x0);
            u[i][k] = A(M(tx, h[i].cs), M(ty, h[i].sn));
            v[i][k] = S(M(ty, h[i].cs), M(tx, h[i].sn));
            ok &= hess_frame<TYPE>(h[i], u[i][k], v[i][k], m[i][k]);
        }
    }
    if (TYPE != 5 && !ok) {
#pragma unroll
        for (int i = 0; i < U; i++)
#pragma unroll
            for (int k = 0; k < P; k++) {
                Mat t;
                hess_ieee<TYPE>(h[i], u[i][k], v[i][k], t);
                m[i][k] = t;
            }
    }
#pragma unroll
    for (int i = 0; i < U; i++)
#pragma unroll
        for (int k = 0; k < P; k++) rotate_acc(m[i][k], h[i].cs, h[i].sn, acc[k]);
}
} // namespace ex

/* Convergence and sky-frame shear of one pair, unweighted, from the real-valued closed form
 * (lt_profiles32.cuh's forms in FP64, record lt_nie64): the FP32C path's recomputation of
 * pixels near critical curves.  About 70 FP64 operations for a dPIE pair against ~95 for
 * the reference's quotient form, and no 0/0 point; equal to it within ~1e-15 of the terms.
 * Every operation's rounding is pinned (explicit round-to-nearest multiply, add and fused
 * multiply-add), so the function can be inlined into any kernel, and interleaved over
 * several pixels, and still round each pair alike everywhere. */
struct Kg64 {
    double k, g1, g2;
};

template <int TYPE>
__device__ __forceinline__ Kg64 nie_kg64(const lt_nie64 &h, double px, double py)
{
    using ex::A;
    using ex::M;
    using ex::S;
    const double tx = S(px, h.x0), ty = S(py, h.y0);
    const double u = __fma_rn(tx, h.cs, M(ty, h.sn)), v = __fma_rn(ty, h.cs, -M(tx, h.sn));
    const double uu = M(u, u), vv = M(v, v), uv = M(u, v);
    double k, g1, g2;
    if (TYPE == 5) {
        const double ir = rsqrt64(__fma_rn(h.q2, uu, M(h.k, vv)));
        const double kk = M(M(h.K, ir), M(ir, ir));
        const double hk = M(0.5, kk);
        k = M(hk, A(uu, vv));
        g1 = M(hk, S(vv, uu));
        g2 = M(-kk, uv);
    } else {
        const double B = __fma_rn(h.q2, uu, vv), r2 = A(uu, vv);
        const double pc2 = A(B, h.q2sc2);
        const double ipc = rsqrt64(pc2), pc = M(pc2, ipc);
        const double Dc = __fma_rn(h.tsc, pc, A(h.opsc2, r2));
        if (TYPE == 8) {
            const double E = M(ipc, rcp64(Dc));
            k = M(h.K, ipc);
            g1 = __fma_rn(h.Kc1sc2, E, M(M(h.K, S(vv, uu)), E));
            g2 = M(M(-2. * h.K, uv), E);
        } else {
            const double pt2 = A(B, h.q2st2);
            const double ipt = rsqrt64(pt2), pt = M(pt2, ipt);
            const double Dt = __fma_rn(h.tst, pt, A(h.opst2, r2));
            const double dpsi = M(h.dq2s2, rcp64(A(pc, pt)));
            const double dD = __fma_rn(2., __fma_rn(pt, h.ds, M(h.sc, dpsi)), h.opds2);
            const double dpD = __fma_rn(dpsi, Dc, M(pt, dD));
            const double Ec = M(ipc, rcp64(Dc)), Et = M(ipt, rcp64(Dt));
            const double dEK = M(M(-h.K, M(dpD, Ec)), Et);
            k = M(M(-h.K, dpsi), M(ipc, ipt));
            g1 = __fma_rn(h.Kc1sc2, Ec, __fma_rn(-h.Kc1st2, Et, M(S(vv, uu), dEK)));
            g2 = M(-2., M(uv, dEK));
        }
    }
    return {k, __fma_rn(g1, h.c2t, -M(g2, h.s2t)), __fma_rn(g1, h.s2t, M(g2, h.c2t))};
}

/* The Hessian of one pair as an out-of-line function, for the FP32C path's FP64 pairs (its
 * cluster-scale halos and the near field of its galaxies).  Compiled once per profile type, it
 * rounds alike in every kernel that calls it, whatever else that kernel computes, so a map is
 * the same from the grid kernels and the work-queue tiles bit for bit; and its registers are
 * not the calling pair loop's. */
template <int TYPE>
__device__ __noinline__ Hess64 hess_term(const lt_rec64 &h, double px, double py, double w)
{
    Hess64 a = {0., 0., 0.};
    hess_pair<TYPE>(h, px, py, w, a);
    return a;
}

} // namespace lt
