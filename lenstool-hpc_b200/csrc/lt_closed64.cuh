/*
 * lt_closed64.cuh -- FP64 deflection, potential and Hessian of one halo record and one pixel
 * from the real-valued closed forms of the non-singular isothermal ellipse (lt_profiles32.cuh
 * states them; record lt_nie64).
 *
 * They equal the reference's complex-quotient forms (src/gradient.cpp:548-607, 744-811,
 * src/potential_GPU.cu:47-116, src/gradient2.cpp:54-83) and have no 0/0 point.  A cut dPIE's
 * deflection takes one arc tangent and one logarithm, where the complex form takes two complex
 * logarithms (2 log + 2 atan2), and its potential two logarithms more, where pi05 takes 6 log,
 * 4 atan2, 16 exp, asinh, asin and 2 sincos: the kernels built on them are FP64-pipe bound
 * (half the FP32 rate on this part), so the FP64 operation count is the time.
 *
 * Every operation is an explicit round-to-nearest multiply, add or fused multiply-add, so a
 * pair rounds alike in every kernel that inlines these functions.
 */
#pragma once
#include "lt_profiles64.cuh"

namespace lt {

/* atan(j/64), j = 0..64, then pi/2 - atan(j/64); log(1 + j/64), j = 0..63: correctly rounded
 * (tests/test_closed64.py recomputes them).  1.5 KB, read through L1: neighbouring pixels of a
 * warp mostly share an entry. */
__device__ const double kAtanTab[130] = {
    0x0.0p+0, 0x1.fff555bbb729bp-7, 0x1.ffd55bba97625p-6, 0x1.7fb818430da2ap-5,
    0x1.ff55bb72cfdeap-5, 0x1.3f59f0e7c559dp-4, 0x1.7ee182602f10fp-4, 0x1.be39ebe6f07c3p-4,
    0x1.fd5ba9aac2f6ep-4, 0x1.1e1fafb043727p-3, 0x1.3d6eee8c6626cp-3, 0x1.5c9811e3ec26ap-3,
    0x1.7b97b4bce5b02p-3, 0x1.9a6a8e96c8626p-3, 0x1.b90d7529260a2p-3, 0x1.d77d5df205736p-3,
    0x1.f5b75f92c80ddp-3, 0x1.09dc597d86362p-2, 0x1.18bf5a30bf178p-2, 0x1.278372057ef46p-2,
    0x1.362773707ebccp-2, 0x1.44aa436c2af0ap-2, 0x1.530ad9951cd4ap-2, 0x1.614840309cfe2p-2,
    0x1.6f61941e4def1p-2, 0x1.7d5604b63b3f7p-2, 0x1.8b24d394a1b25p-2, 0x1.98cd5454d6b18p-2,
    0x1.a64eec3cc23fdp-2, 0x1.b3a911da65c6cp-2, 0x1.c0db4c94ec9f0p-2, 0x1.cde53432c1351p-2,
    0x1.dac670561bb4fp-2, 0x1.e77eb7f175a34p-2, 0x1.f40dd0b541418p-2, 0x1.0039c73c1a40cp-1,
    0x1.0657e94db30d0p-1, 0x1.0c6145b5b43dap-1, 0x1.1255d9bfbd2a9p-1, 0x1.1835a88be7c13p-1,
    0x1.1e00babdefeb4p-1, 0x1.23b71e2cc9e6ap-1, 0x1.2958e59308e31p-1, 0x1.2ee628406cbcap-1,
    0x1.345f01cce37bbp-1, 0x1.39c391cd4171ap-1, 0x1.3f13fb89e96f4p-1, 0x1.445065b795b56p-1,
    0x1.4978fa3269ee1p-1, 0x1.4e8de5bb6ec04p-1, 0x1.538f57b89061fp-1, 0x1.587d81f732fbbp-1,
    0x1.5d58987169b18p-1, 0x1.6220d115d7b8ep-1, 0x1.66d663923e087p-1, 0x1.6b798920b3d99p-1,
    0x1.700a7c5784634p-1, 0x1.748978fba8e0fp-1, 0x1.78f6bbd5d315ep-1, 0x1.7d528289fa093p-1,
    0x1.819d0b7158a4dp-1, 0x1.85d69576cc2c5p-1, 0x1.89ff5ff57f1f8p-1, 0x1.8e17aa99cc05ep-1,
    0x1.921fb54442d18p-1, 0x1.921fb54442d18p+0, 0x1.8e1fca98cb633p+0, 0x1.8a205fd558740p+0,
    0x1.8621f4822a647p+0, 0x1.82250768ac529p+0, 0x1.7e2a1635c67bep+0, 0x1.7a319d1e3fe07p+0,
    0x1.763c1685d3c9cp+0, 0x1.7249faa996a21p+0, 0x1.6e5bbf4e3a633p+0, 0x1.6a71d772b60cbp+0,
    0x1.668cb307c54cbp+0, 0x1.62acbeaca61b8p+0, 0x1.5ed2637169c54p+0, 0x1.5afe069f1e104p+0,
    0x1.5730098602231p+0, 0x1.5368c951e9cfdp+0, 0x1.4fa89ee4e1440p+0, 0x1.4befdeb8130bap+0,
    0x1.483ed8c2e3147p+0, 0x1.4495d86823225p+0, 0x1.40f5246938156p+0, 0x1.3d5cfedefb9c6p+0,
    0x1.39cda5381b920p+0, 0x1.3647503caf55cp+0, 0x1.32ca3416b401ap+0, 0x1.2f56805f1a64fp+0,
    0x1.2bec602f0d252p+0, 0x1.288bfa3512419p+0, 0x1.253570cda95fdp+0, 0x1.21e8e21f07a9cp+0,
    0x1.1ea6683792844p+0, 0x1.1b6e192ebbe44p+0, 0x1.18400747e568bp+0, 0x1.151c4116f2812p+0,
    0x1.1202d1a635b12p+0, 0x1.0ef3c09d694b0p+0, 0x1.0bef126968b2bp+0, 0x1.08f4c864643c4p+0,
    0x1.0604e0fe4ef0fp+0, 0x1.031f57e54adbep+0, 0x1.0044262dddde3p+0, 0x1.fae684f57cc00p-1,
    0x1.f559424818e66p-1, 0x1.efe068bba2275p-1, 0x1.ea7bd8bb44317p-1, 0x1.e52b6efe9c33cp-1,
    0x1.dfef04d0efedbp-1, 0x1.dac670561bb4fp-1, 0x1.d5b184cd16e2cp-1, 0x1.d0b012cff5412p-1,
    0x1.cbc1e89152a76p-1, 0x1.c6e6d2171bf18p-1, 0x1.c21e9972adea3p-1, 0x1.bd6906f6479aap-1,
    0x1.b8c5e167d1c98p-1, 0x1.b434ee31013fdp-1, 0x1.afb5f18cdcc22p-1, 0x1.ab48aeb2b28d2p-1,
    0x1.a6ece7fe8b99dp-1, 0x1.a2a25f172cfe4p-1, 0x1.9e68d511b976bp-1, 0x1.9a400a9306839p-1,
    0x1.9627bfeeb99d3p-1, 0x1.921fb54442d18p-1};
__device__ const double kLogTab[64] = {
    0x0.0p+0, 0x1.fc0a8b0fc03e4p-7, 0x1.f829b0e783300p-6, 0x1.77458f632dcfcp-5,
    0x1.f0a30c01162a6p-5, 0x1.341d7961bd1d1p-4, 0x1.6f0d28ae56b4cp-4, 0x1.a926d3a4ad563p-4,
    0x1.e27076e2af2e6p-4, 0x1.0d77e7cd08e59p-3, 0x1.29552f81ff523p-3, 0x1.44d2b6ccb7d1ep-3,
    0x1.5ff3070a793d4p-3, 0x1.7ab890210d909p-3, 0x1.9525a9cf456b4p-3, 0x1.af3c94e80bff3p-3,
    0x1.c8ff7c79a9a22p-3, 0x1.e27076e2af2e6p-3, 0x1.fb9186d5e3e2bp-3, 0x1.0a324e27390e3p-2,
    0x1.1675cababa60ep-2, 0x1.22941fbcf7966p-2, 0x1.2e8e2bae11d31p-2, 0x1.3a64c556945eap-2,
    0x1.4618bc21c5ec2p-2, 0x1.51aad872df82dp-2, 0x1.5d1bdbf5809cap-2, 0x1.686c81e9b14afp-2,
    0x1.739d7f6bbd007p-2, 0x1.7eaf83b82afc3p-2, 0x1.89a3386c1425bp-2, 0x1.947941c2116fbp-2,
    0x1.9f323ecbf984cp-2, 0x1.a9cec9a9a084ap-2, 0x1.b44f77bcc8f63p-2, 0x1.beb4d9da71b7cp-2,
    0x1.c8ff7c79a9a22p-2, 0x1.d32fe7e00ebd5p-2, 0x1.dd46a04c1c4a1p-2, 0x1.e744261d68788p-2,
    0x1.f128f5faf06edp-2, 0x1.faf588f78f31fp-2, 0x1.02552a5a5d0ffp-1, 0x1.0723e5c1cdf40p-1,
    0x1.0be72e4252a83p-1, 0x1.109f39e2d4c97p-1, 0x1.154c3d2f4d5eap-1, 0x1.19ee6b467c96fp-1,
    0x1.1e85f5e7040d0p-1, 0x1.23130d7bebf43p-1, 0x1.2795e1289b11bp-1, 0x1.2c0e9ed448e8cp-1,
    0x1.307d7334f10bep-1, 0x1.34e289d9ce1d3p-1, 0x1.393e0d3562a1ap-1, 0x1.3d9026a7156fbp-1,
    0x1.41d8fe84672aep-1, 0x1.4618bc21c5ec2p-1, 0x1.4a4f85db03ebbp-1, 0x1.4e7d811b75bb1p-1,
    0x1.52a2d265bc5abp-1, 0x1.56bf9d5b3f399p-1, 0x1.5ad404c359f2dp-1, 0x1.5ee02a9241675p-1};

namespace c64 {
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
/* a, negated where b is negative */
__device__ __forceinline__ double flip(double a, double b)
{
    return __hiloint2double(__double2hiint(a) ^ (__double2hiint(b) & (int)0x80000000), __double2loint(a));
}
/* a positive normal float (or +0, as 2^-127) as a double, by its bits */
__device__ __forceinline__ double widen(int bits) { return __hiloint2double((bits >> 3) + 0x38000000, 0); }
} // namespace c64

/* atan(n/d) for d > 0, any n.  With a = min(|n|, d)/max(|n|, d) and c = j/64 the table point
 * next to a (chosen in FP32: any neighbouring point would do),
 *   atan a = atan c + atan t,  t = (min - c max)/(max + c min),  |t| <= 1/128,
 * and atan t = t - t^3/3 + t^5/5 - t^7/7 (truncation t^9/9 < 2e-18 of t).  One reciprocal,
 * 12 FP64 operations; within 2 ulp of atan(n/d) while the larger of |n| and d is within FP32's
 * range (pack_nie64 sees to it that radii far outside the field's scales do not leave it).  j = 0
 * leaves t = a exactly, so small quotients keep their relative accuracy. */
__device__ __forceinline__ double atan_quot(double n, double d)
{
    using namespace c64;
    const double an = fabs(n);
    const float nf = __double2float_rn(an), df = __double2float_rn(d);
    const bool swap = nf > df;
    const double mn = swap ? d : an, mx = swap ? an : d;
    const float af = fminf(__fmul_rn(fminf(nf, df), frcp(fmaxf(nf, df))), 1.f);
    const float jf = __fmaf_rn(af, 64.f, 12582912.f); /* 1.5 x 2^23 + j */
    const int j = __float_as_int(jf) & 127;
    const double c = j ? widen(__float_as_int(__fmul_rn(__fsub_rn(jf, 12582912.f), 0.015625f))) : 0.;
    const double base = kAtanTab[swap ? j + 65 : j];
    const double t = mul(fma(-c, mx, mn), rcp64(fma(c, mn, mx)));
    const double s = mul(t, t);
    const double p = fma(fma(-1. / 7., s, 0.2), s, -1. / 3.);
    const double r = fma(mul(t, s), p, t);
    return copysign(swap ? sub(base, r) : add(base, r), n);
}

/* log(1 + n/d) for n >= 0, d > 0.  With c = 2^e (1 + j/64) next to 1 + n/d (chosen in FP32),
 *   log(1 + n/d) = log c + 2 atanh t,  t = (n + (1 - c) d)/(n + (1 + c) d),  |t| <= 1/256,
 * and 2 atanh t = t (2 + 2/3 t^2 + 2/5 t^4 + 2/7 t^6) (truncation below 1e-20 of t).  One
 * reciprocal, 15 FP64 operations; within 2 ulp.  c = 1 leaves t = n/(n + 2 d): small quotients
 * keep their relative accuracy. */
__device__ __forceinline__ double log1p_quot(double n, double d)
{
    using namespace c64;
    const float m = fminf(__fmaf_rn(__double2float_rn(n), frcp(__double2float_rn(d)), 1.f), 0x1p126f);
    const int b = (__float_as_int(m) + 0x10000) & 0x7ffe0000;
    const double c = widen(b);
    const double e = sub(__hiloint2double(0x43300000, (b >> 23) - 127), 4503599627370496.);
    const double base = fma(e, 0.69314718055994530942, kLogTab[(b >> 17) & 63]);
    const double t = mul(fma(sub(1., c), d, n), rcp64(fma(add(1., c), d, n)));
    const double s = mul(t, t);
    const double p = fma(fma(fma(2. / 7., s, 0.4), s, 2. / 3.), s, 2.);
    return fma(t, p, base);
}

/* The radius-dependent quantities of one pair: halo-frame offset, u^2, v^2, psi of the core
 * (and cut) radius. */
struct Nie64 {
    double u, v, uu, vv, B, pc, ipc, pt, ipt;
};

template <int TYPE>
__device__ __forceinline__ Nie64 nie64(const lt_nie64 &h, double px, double py)
{
    using namespace c64;
    Nie64 n;
    const double tx = sub(px, h.x0), ty = sub(py, h.y0);
    n.u = fma(tx, h.cs, mul(ty, h.sn));
    n.v = fma(-tx, h.sn, mul(ty, h.cs));
    n.uu = mul(n.u, n.u);
    n.vv = mul(n.v, n.v);
    if (TYPE == 5) {
        n.B = fma(h.q2, n.uu, mul(h.k, n.vv)); /* R^2 = (1-e) u^2 + (1+e) v^2 */
        n.ipc = rsqrt64(n.B);
        n.pc = n.pt = n.ipt = 0.;
        return n;
    }
    n.B = fma(h.q2, n.uu, n.vv);
    const double pc2 = add(n.B, h.q2sc2);
    n.ipc = rsqrt64(pc2);
    n.pc = mul(pc2, n.ipc);
    n.pt = n.ipt = 0.;
    if (TYPE == 81) {
        const double pt2 = add(n.B, h.q2st2);
        n.ipt = rsqrt64(pt2);
        n.pt = mul(pt2, n.ipt);
    }
    return n;
}

/* Halo-frame deflection (alpha_u, alpha_v).  For the dPIE
 *   atan a_c - atan a_t = atan(nu/du),     atanh b_c - atanh b_t = atanh(nv/dv),
 * with the numerators and denominators of grad32 (no cancellation in the numerators, through
 * psi_c - psi_t = q^2 (s_c^2 - s_t^2)/(psi_c + psi_t)); atanh(y) = log(1 + 2 y/(1 - y))/2 for
 * y >= 0.  dv - |nv| = (1 - b_c)(1 + b_t) x the two denominators loses digits like 1/q^2: for
 * q^2 < 1/16 (ellipticity of the potential above 0.6) it is formed as that product, with
 *   psi_c + q^2 s_c - k|v| = q^2 (u^2 + v^2 + s_c^2)/(psi_c + k|v|) + q^2 s_c. */
template <int TYPE>
__device__ __forceinline__ void defl64(const lt_nie64 &h, const Nie64 &n, double &au, double &av)
{
    using namespace c64;
    if (TYPE == 5) { /* SIS: b0 ((1-e) u, (1+e) v)/R */
        au = mul(mul(h.Ak, h.q2), mul(n.u, n.ipc));
        av = mul(mul(h.Ak, h.k), mul(n.v, n.ipc));
        return;
    }
    const double ku = mul(h.k, n.u), kv = mul(h.k, fabs(n.v));
    const double pcs = add(n.pc, h.sc), pcq = add(n.pc, h.q2sc);
    double nu, du, nv, qv;
    if (TYPE == 8) {
        nu = ku;
        du = pcs;
        nv = kv;
        qv = sub(pcq, kv);
    } else {
        const double dpsi = mul(h.dq2s2, rcp64(add(n.pc, n.pt))); /* psi_c - psi_t < 0 */
        const double ptq = add(n.pt, h.q2st);
        nu = mul(-ku, add(dpsi, h.ds));
        du = fma(ku, ku, mul(pcs, add(n.pt, h.st)));
        nv = mul(-kv, add(dpsi, h.dsq2));
        qv = sub(fma(-kv, kv, mul(pcq, ptq)), nv);
    }
    if (h.q2 < 0.0625) {
        const double lo = fma(h.q2, mul(fma(h.sc, h.sc, add(n.uu, n.vv)), rcp64(add(n.pc, kv))), h.q2sc);
        qv = TYPE == 8 ? lo : mul(lo, add(add(n.pt, h.q2st), kv));
    }
    au = mul(h.Ak, atan_quot(nu, du));
    av = flip(mul(h.hAk, log1p_quot(add(nv, nv), qv)), n.v); /* hAk < 0: a halo of negative mass */
}

/* Adds one pair's deflection in the sky frame. */
template <int TYPE>
__device__ __forceinline__ void grad_nie(const lt_nie64 &h, const Nie64 &n, double &gx, double &gy)
{
    using namespace c64;
    double au, av;
    defl64<TYPE>(h, n, au, av);
    /* one rounding of the sum per pair */
    gx = add(gx, fma(au, h.cs, -mul(av, h.sn)));
    gy = add(gy, fma(au, h.sn, mul(av, h.cs)));
}

/* Adds one pair's potential:
 *   u alpha_u + v alpha_v - (A s_c/2) log(1 + t_c) [+ (A s_t/2) log(1 + t_t)],
 *   t_s = (r^2 (psi + q s) + 2 s B)/(4 r_s^2 (psi + q s)), terms of one sign;
 * at a centre pi05 is 0/0 (src/potential_GPU.cu:56-60): NaN, as there. */
template <int TYPE>
__device__ __forceinline__ void pot_nie(const lt_nie64 &h, const Nie64 &n, double &psi)
{
    using namespace c64;
    if (TYPE == 5) {
        psi = fma(h.Ak, __dsqrt_rn(n.B), psi);
        return;
    }
    double au, av;
    defl64<TYPE>(h, n, au, av);
    const double r2 = add(n.uu, n.vv);
    const double pcq = add(n.pc, h.qsc);
    double hs = mul(h.sc, log1p_quot(fma(r2, pcq, mul(h.tsc, n.B)), mul(h.frc2, pcq)));
    if (TYPE == 81) {
        const double ptq = add(n.pt, h.qst);
        hs = fma(-h.st, log1p_quot(fma(r2, ptq, mul(h.tst, n.B)), mul(h.frt2, ptq)), hs);
    }
    const double p = fma(-h.K, hs, fma(n.u, au, mul(n.v, av)));
    psi = r2 == 0. ? __longlong_as_double(0x7ff8000000000000ll) : add(psi, p);
}

/* Adds w x one pair's convergence and sky-frame shear.  In FP64 the core - cut differences are
 * taken directly: their rounding is a few 1e-17 of the core term, below the rounding of the sums. */
template <int TYPE>
__device__ __forceinline__ void kg_nie(const lt_nie64 &h, const Nie64 &n, double w, double &kap, double &g1, double &g2)
{
    using namespace c64;
    double k, a, b;
    if (TYPE == 5) {
        const double kk = mul(mul(h.K, n.ipc), mul(n.ipc, n.ipc)), hk = mul(0.5, kk);
        k = mul(hk, add(n.uu, n.vv));
        a = mul(hk, sub(n.vv, n.uu));
        b = mul(-kk, mul(n.u, n.v));
    } else {
        const double r2 = add(n.uu, n.vv);
        double E = mul(n.ipc, rcp64(fma(h.tsc, n.pc, add(h.opsc2, r2))));
        double i = n.ipc, c = mul(h.Kc1sc2, E);
        if (TYPE == 81) {
            const double Et = mul(n.ipt, rcp64(fma(h.tst, n.pt, add(h.opst2, r2))));
            i = sub(i, n.ipt);
            c = fma(-h.Kc1st2, Et, c);
            E = sub(E, Et);
        }
        E = mul(h.K, E);
        k = mul(h.K, i);
        a = fma(sub(n.vv, n.uu), E, c);
        b = mul(mul(n.u, n.v), mul(-2., E));
    }
    kap = fma(w, k, kap);
    g1 = fma(w, fma(a, h.c2t, -mul(b, h.s2t)), g1);
    g2 = fma(w, fma(a, h.s2t, mul(b, h.c2t)), g2);
}

/* The FP64 deflection and potential of one pair as out-of-line functions, for the FP32C path's
 * FP64 pairs (its cluster-scale halos and the near field of its galaxies): their registers are
 * not the calling pair loop's. */
template <int TYPE>
__device__ __noinline__ double pot_term(const lt_nie64 &h, double px, double py)
{
    double p = 0.;
    pot_nie<TYPE>(h, nie64<TYPE>(h, px, py), p);
    return p;
}

template <int TYPE>
__device__ __noinline__ double2 grad_term(const lt_nie64 &h, double px, double py)
{
    double gx = 0., gy = 0.;
    grad_nie<TYPE>(h, nie64<TYPE>(h, px, py), gx, gy);
    return make_double2(gx, gy);
}

} // namespace lt
