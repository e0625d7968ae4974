// Device-side characteristic functions and Gil-Pelaez integrand (FP64).
//
// Reference: heston.rs:101-127 (cf_integrand, stable_cf), heston.rs:155-175
// (fast_csqrt), heston.rs:220-227 (the [0,inf) -> [0,1] substitution),
// bates.rs:65-83 (bates_integrand, jump_cf).
//
// `node_cf` + `node_finish` evaluate gk_integrate's g(t) at one GK node:
// u = (1-t)/t, f(u)/t^2, non-finite -> 0.  The Albrecher stable CF is
// evaluated with its per-contract constants hoisted into CfConsts.  The
// three exponential factors the reference multiplies together per node
// (stable_cf's exp, the jump factor's outer exp and e^{iux}), the division
// by the P1 normaliser CF(-i) and the final division by iu are merged into
// ONE complex exponent Z:
//
//     Re[ e^{iux} * CF(phi) / CF(-i) / (iu) ] = e^{Re Z} * sin(Im Z) / u,
//     Z = i r phi T + C + D [+ J] + i u x - Log CF(-i)
//
// which is the same number up to rounding (exp(a)exp(b) = exp(a+b)), and
// trades four complex exponentials and two complex divisions per node for
// one real exp and one sin.  Log CF(-i) is computed once per integral from
// CF(-i) evaluated with the reference's own operation sequence, so the
// degenerate cases (CF(-i) = 0, inf or NaN) zero the P1 integrand exactly as
// the reference's division does.
//
// Of Z only the phase u x depends on the strike (x = ln(S/K)); the rest is a
// function of the node, the expiry, the rate, the parameters and the
// integral.  So the evaluation is split: node_cf gives the strike-free part
// (W and Im Z without u x), node_finish adds one strike's phase and
// forms the value.  Contracts of one surface that share
// an expiry and a rate share node_cf's values at every panel they both
// bisect (the run cache of quadrature.cuh).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace ope {

struct Cx {
    double re, im;
};

// Reciprocal and reciprocal square root: the hardware approximation
// (rcp/rsqrt.approx.ftz.f64, about 2^-22 relative error) refined by one
// third-order step (the series of 1/(1 - e) and of (1 - 2 e)^-1/2 to e^2):
// y <- y + y (e + e^2), e = 1 - x y, and y <- y + y (e + 3/2 e^2),
// e = (1 - x y^2)/2.  Each cubes the relative error, so the result is within
// an ulp or two of the correctly rounded value (checked against IEEE division
// and sqrt by ope_selftest_math) with one operation less than two Newton steps
// for the reciprocal and two less for the root.  Used for the complex reciprocals and the
// square root of the node evaluation; a zero or infinite argument gives a
// non-finite result, which zeroes the node exactly as the reference's
// division by zero does.
__device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    e = fma(e, e, e);
    return fma(y, e, y);
}
__device__ __forceinline__ double rsqrt_nr(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-0.5 * x * y, y, 0.5);
    return fma(y, fma(1.5 * e, e, e), y);
}

// atan2(y, x), branch-free (the node evaluation's own argument is arg_node; this
// one is what ope_selftest_atan2 compares).  Method (the classical argument reduction of
// Cody and Waite's elementary-function manual): octant symmetry reduces it
// to atan(q), q = min(|x|,|y|)/max(|x|,|y|) in [0, 1]; above tan(pi/8),
// atan(q) = pi/4 + atan((q - 1)/(q + 1)); on |t| <= tan(pi/8),
// atan(t) = t + t s P(s), s = t^2, with the degree-10 Chebyshev interpolant P
// of node_math_coeffs.py (5e-18 relative).  With q = mn/mx the reduced quotient
// is (mn - mx)/(mn + mx), so one rcp_nr serves either case.  At most
// 4 ulp from CUDA's atan2 over finite arguments whose larger magnitude is at
// least 2^-1022; outside that (a NaN or infinite argument, or both below
// 2^-1022) it returns NaN.
__device__ __forceinline__ double atan2_node(double y, double x) {
    const double ax = fabs(x), ay = fabs(y);
    const bool swap = ay > ax;
    const double mn = swap ? ax : ay, mx = swap ? ay : ax;
    const bool big = mn > 0.41421356237309503 * mx;  // tan(pi/8)
    const double t = (big ? mn - mx : mn) * rcp_nr(big ? mn + mx : mx);
    const double s = t * t;
    double p = -0.01917688711906226;
    p = fma(p, s, 0.03923165829558719);
    p = fma(p, s, -0.0508544973794026);
    p = fma(p, s, 0.0585814891280221);
    p = fma(p, s, -0.06664511447381948);
    p = fma(p, s, 0.07692183190826087);
    p = fma(p, s, -0.09090904578123903);
    p = fma(p, s, 0.11111111015256361);
    p = fma(p, s, -0.14285714284666542);
    p = fma(p, s, 0.1999999999999552);
    p = fma(p, s, -0.3333333333333333);
    double r = fma(t * s, p, t);                       // atan(t)
    r = big ? r + 0.78539816339744831 : r;            // atan(q)
    r = swap ? 1.5707963267948966 - r : r;            // first quadrant
    r = (x < 0.0) ? 3.1415926535897931 - r : r;       // upper half plane
    return copysign(r, y);
}

// arg(x + iy) for the node evaluation's Log A, by a rotation: the difference of
// the high words of |y| and |x| is log2 |y/x| to within 0.09, which with the
// two signs picks one of 84 directions K (bins half an octave wide, so K lies
// within 0.111 of the angle; K = 0 and pi/2 beyond 2^(+-4.75)); turned by -K,
// t = (y cos K - x sin K)/(x cos K + y sin K), arg = K + atan t, atan t =
// t + t s P(s), s = t^2, P the degree-5 Chebyshev interpolant (8.8e-19 absolute).  Without
// it (atan2_node's octant reduction) a node makes seven selects, three
// comparisons, three additions and five polynomial steps more.  x = y = 0 and
// non-finite arguments give NaN or a finite angle; in the node evaluation
// those come only with a 1/|N|^2 that is not finite and drops the node.
struct alignas(16) ArgDir {
    double c, s, k, pad;
};
static __device__ const ArgDir g_arg_tab[84] = {
    {1.0, 0.0, 0.0, 0.0},
    {0.9990248656871402, 0.044151078568834795, 0.04416543524608704, 0.0},
    {0.9980525784828885, 0.06237828615518053, 0.06241880999595735, 0.0},
    {0.9961164901835046, 0.08804509063256238, 0.08815924263434795, 0.0},
    {0.9922778767136676, 0.12403473458920845, 0.12435499454676144, 0.0},
    {0.9847319278346619, 0.17407765595569785, 0.17496904566568885, 0.0},
    {0.9701425001453319, 0.24253562503633297, 0.24497866312686414, 0.0},
    {0.9428090415820634, 0.3333333333333333, 0.3398369094541219, 0.0},
    {0.8944271909999159, 0.4472135954999579, 0.4636476090008061, 0.0},
    {0.816496580927726, 0.5773502691896257, 0.6154797086703873, 0.0},
    {0.7071067811865476, 0.7071067811865476, 0.7853981633974483, 0.0},
    {0.5773502691896257, 0.816496580927726, 0.9553166181245093, 0.0},
    {0.4472135954999579, 0.8944271909999159, 1.1071487177940904, 0.0},
    {0.3333333333333333, 0.9428090415820634, 1.2309594173407747, 0.0},
    {0.24253562503633297, 0.9701425001453319, 1.3258176636680326, 0.0},
    {0.17407765595569785, 0.9847319278346619, 1.3958272811292078, 0.0},
    {0.12403473458920845, 0.9922778767136676, 1.446441332248135, 0.0},
    {0.08804509063256238, 0.9961164901835046, 1.4826370841605487, 0.0},
    {0.06237828615518053, 0.9980525784828885, 1.5083775167989393, 0.0},
    {0.044151078568834795, 0.9990248656871402, 1.5266308915488096, 0.0},
    {0.0, 1.0, 1.5707963267948966, 0.0},
    {-1.0, 0.0, 3.141592653589793, 0.0},
    {-0.9990248656871402, 0.044151078568834795, 3.0974272183437064, 0.0},
    {-0.9980525784828885, 0.06237828615518053, 3.079173843593836, 0.0},
    {-0.9961164901835046, 0.08804509063256238, 3.0534334109554453, 0.0},
    {-0.9922778767136676, 0.12403473458920845, 3.017237659043032, 0.0},
    {-0.9847319278346619, 0.17407765595569785, 2.966623607924104, 0.0},
    {-0.9701425001453319, 0.24253562503633297, 2.896613990462929, 0.0},
    {-0.9428090415820634, 0.3333333333333333, 2.8017557441356713, 0.0},
    {-0.8944271909999159, 0.4472135954999579, 2.677945044588987, 0.0},
    {-0.816496580927726, 0.5773502691896257, 2.5261129449194057, 0.0},
    {-0.7071067811865476, 0.7071067811865476, 2.356194490192345, 0.0},
    {-0.5773502691896257, 0.816496580927726, 2.186276035465284, 0.0},
    {-0.4472135954999579, 0.8944271909999159, 2.0344439357957027, 0.0},
    {-0.3333333333333333, 0.9428090415820634, 1.9106332362490186, 0.0},
    {-0.24253562503633297, 0.9701425001453319, 1.8157749899217608, 0.0},
    {-0.17407765595569785, 0.9847319278346619, 1.7457653724605855, 0.0},
    {-0.12403473458920845, 0.9922778767136676, 1.695151321341658, 0.0},
    {-0.08804509063256238, 0.9961164901835046, 1.6589555694292446, 0.0},
    {-0.06237828615518053, 0.9980525784828885, 1.633215136790854, 0.0},
    {-0.044151078568834795, 0.9990248656871402, 1.6149617620409837, 0.0},
    {0.0, 1.0, 1.5707963267948966, 0.0},
    {1.0, -0.0, 0.0, 0.0},
    {0.9990248656871402, -0.044151078568834795, -0.04416543524608704, 0.0},
    {0.9980525784828885, -0.06237828615518053, -0.06241880999595735, 0.0},
    {0.9961164901835046, -0.08804509063256238, -0.08815924263434795, 0.0},
    {0.9922778767136676, -0.12403473458920845, -0.12435499454676144, 0.0},
    {0.9847319278346619, -0.17407765595569785, -0.17496904566568885, 0.0},
    {0.9701425001453319, -0.24253562503633297, -0.24497866312686414, 0.0},
    {0.9428090415820634, -0.3333333333333333, -0.3398369094541219, 0.0},
    {0.8944271909999159, -0.4472135954999579, -0.4636476090008061, 0.0},
    {0.816496580927726, -0.5773502691896257, -0.6154797086703873, 0.0},
    {0.7071067811865476, -0.7071067811865476, -0.7853981633974483, 0.0},
    {0.5773502691896257, -0.816496580927726, -0.9553166181245093, 0.0},
    {0.4472135954999579, -0.8944271909999159, -1.1071487177940904, 0.0},
    {0.3333333333333333, -0.9428090415820634, -1.2309594173407747, 0.0},
    {0.24253562503633297, -0.9701425001453319, -1.3258176636680326, 0.0},
    {0.17407765595569785, -0.9847319278346619, -1.3958272811292078, 0.0},
    {0.12403473458920845, -0.9922778767136676, -1.446441332248135, 0.0},
    {0.08804509063256238, -0.9961164901835046, -1.4826370841605487, 0.0},
    {0.06237828615518053, -0.9980525784828885, -1.5083775167989393, 0.0},
    {0.044151078568834795, -0.9990248656871402, -1.5266308915488096, 0.0},
    {0.0, -1.0, -1.5707963267948966, 0.0},
    {-1.0, -0.0, -3.141592653589793, 0.0},
    {-0.9990248656871402, -0.044151078568834795, -3.0974272183437064, 0.0},
    {-0.9980525784828885, -0.06237828615518053, -3.079173843593836, 0.0},
    {-0.9961164901835046, -0.08804509063256238, -3.0534334109554453, 0.0},
    {-0.9922778767136676, -0.12403473458920845, -3.017237659043032, 0.0},
    {-0.9847319278346619, -0.17407765595569785, -2.966623607924104, 0.0},
    {-0.9701425001453319, -0.24253562503633297, -2.896613990462929, 0.0},
    {-0.9428090415820634, -0.3333333333333333, -2.8017557441356713, 0.0},
    {-0.8944271909999159, -0.4472135954999579, -2.677945044588987, 0.0},
    {-0.816496580927726, -0.5773502691896257, -2.5261129449194057, 0.0},
    {-0.7071067811865476, -0.7071067811865476, -2.356194490192345, 0.0},
    {-0.5773502691896257, -0.816496580927726, -2.186276035465284, 0.0},
    {-0.4472135954999579, -0.8944271909999159, -2.0344439357957027, 0.0},
    {-0.3333333333333333, -0.9428090415820634, -1.9106332362490186, 0.0},
    {-0.24253562503633297, -0.9701425001453319, -1.8157749899217608, 0.0},
    {-0.17407765595569785, -0.9847319278346619, -1.7457653724605855, 0.0},
    {-0.12403473458920845, -0.9922778767136676, -1.695151321341658, 0.0},
    {-0.08804509063256238, -0.9961164901835046, -1.6589555694292446, 0.0},
    {-0.06237828615518053, -0.9980525784828885, -1.633215136790854, 0.0},
    {-0.044151078568834795, -0.9990248656871402, -1.6149617620409837, 0.0},
    {0.0, -1.0, -1.5707963267948966, 0.0}};
__device__ __forceinline__ double arg_node(double y, double x) {
    const int hy = __double2hiint(y), hx = __double2hiint(x);
    constexpr int kBin = 1 << 19, kTop = 19 * (1 << 18);  // half an octave, 4.75 octaves
    int d = (hy & 0x7fffffff) - (hx & 0x7fffffff);
    d = min(max(d, -kTop - kBin), kTop);
    const int at = ((d + kTop + kBin) >> 19) + 21 * (int)((unsigned)hx >> 31) + 42 * (int)((unsigned)hy >> 31);
    const ArgDir* e = g_arg_tab + at;
    const double2 cs = __ldg(reinterpret_cast<const double2*>(e));
    const double t = __dmul_rn(fma(y, cs.x, __dmul_rn(-x, cs.y)), rcp_nr(fma(y, cs.y, __dmul_rn(x, cs.x))));
    const double s = __dmul_rn(t, t);
    double p = 0.07444393634796143;
    p = fma(p, s, -0.0908733606338501);
    p = fma(p, s, 0.1111108660697937);
    p = fma(p, s, -0.14285714206116987);
    p = fma(p, s, 0.19999999999895343);
    p = fma(p, s, -0.33333333333333287);
    return __dadd_rn(__ldg(&e->k), fma(__dmul_rn(t, s), p, t));
}

// log(v) (the node evaluation's own logarithm is log_ratio, made the same way;
// this one is what ope_selftest_log compares).  Method (the atanh form of
// the logarithm of Cody and Waite's manual): v = 2^k m with m in
// [sqrt(1/2), sqrt 2), read off the IEEE exponent and mantissa bits;
// log v = k ln 2 + 2 atanh(s), s = (m - 1)/(m + 1) (m - 1 is exact, the
// quotient uses rcp_nr), 2 atanh(s) = 2 s + s w R(w), w = s^2, with the
// degree-6 Chebyshev interpolant R of node_math_coeffs.py (4.5e-18 relative),
// and k ln 2 added through two FMAs with ln 2 split into a double and its
// remainder.  At most 2 ulp from CUDA's log.  Arguments
// outside the normal range (0, subnormal, infinite, NaN) take CUDA's log.
__device__ __forceinline__ double log_node(double v) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int k = (hi - 0x3FE6A09E) >> 20;  // 0x3FE6A09E: high word of sqrt(1/2)
    const double m = __hiloint2double(hi - k * 0x100000, lo);
    const double f = m - 1.0;
    const double s = f * rcp_nr(2.0 + f);
    const double w = s * s;
    double r = 0.14616449685043406;
    r = fma(r, w, 0.15331721600556042);
    r = fma(r, w, 0.18182889125261723);
    r = fma(r, w, 0.2222221113479508);
    r = fma(r, w, 0.28571428625975487);
    r = fma(r, w, 0.39999999999899505);
    r = fma(r, w, 0.666666666666667);
    const double lm = fma(s * w, r, 2.0 * s);  // log m
    const double kd = (double)k;
    double out = fma(kd, 0.6931471805599453, fma(kd, 2.3190468138462996e-17, lm));
    if (!(v >= 0x1p-1022 && v <= 0x1.fffffffffffffp+1023)) out = log(v);
    return out;
}

// log(a / b) for the node evaluation's log|A|^2, and ia = 1 / a, through one
// reciprocal: a = 2^k a' with a'/b near 1 (k from the difference of the high
// words, so a'/b lies within 2^(+-0.59) of 1), then log(a / b) = k ln 2 +
// 2 atanh(s), s = (a' - b)/(a' + b), |s| <= 0.2, 2 atanh(s) = 2 s + s w R(w)
// as in log_node (degree 7, 1.3e-17 relative, from node_math_coeffs.py); both
// quotients share
// rcp(a (a' + b)).  A zero, infinite or NaN a gives a
// non-finite ia (its callers then drop the node).
__device__ __forceinline__ double log_ratio(double a, double b, double& ia) {
    const int ha = __double2hiint(a);
    const int k = (ha - __double2hiint(b) + 0x80000) >> 20;
    const double as = __hiloint2double(ha - k * 0x100000, __double2loint(a));
    const double sum = as + b;
    const double inv = rcp_nr(a * sum);
    ia = inv * sum;
    const double s = (as - b) * (inv * a);
    const double w = s * s;
    double r = 0.13636279106140137;
    r = fma(r, w, 0.13204848766326904);
    r = fma(r, w, 0.15389204025268555);
    r = fma(r, w, 0.18181729316711426);
    r = fma(r, w, 0.2222222299253829);
    r = fma(r, w, 0.2857142857209699);
    r = fma(r, w, 0.3999999999996081);
    r = fma(r, w, 0.6666666666666672);
    const double kd = (double)k;
    return fma(kd, 0.6931471824645996, fma(kd, -1.904654299957768e-09, fma(s * w, r, 2.0 * s)));
}

// Tables of the node evaluation's own exponential and sine/cosine: 2^(j/64),
// and (cos, sin) of j pi/32, correctly rounded.  Read by index through L1.
static __device__ const double g_exp2_tab[64] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951};
static __device__ const double2 g_cis_tab[64] = {
    {1.0, 0.0}, {0.9951847266721969, 0.0980171403295606},
    {0.9807852804032304, 0.19509032201612828}, {0.9569403357322088, 0.2902846772544624},
    {0.9238795325112867, 0.3826834323650898}, {0.881921264348355, 0.47139673682599764},
    {0.8314696123025452, 0.5555702330196022}, {0.773010453362737, 0.6343932841636455},
    {0.7071067811865476, 0.7071067811865476}, {0.6343932841636455, 0.773010453362737},
    {0.5555702330196022, 0.8314696123025452}, {0.47139673682599764, 0.881921264348355},
    {0.3826834323650898, 0.9238795325112867}, {0.2902846772544624, 0.9569403357322088},
    {0.19509032201612828, 0.9807852804032304}, {0.0980171403295606, 0.9951847266721969},
    {0.0, 1.0}, {-0.0980171403295606, 0.9951847266721969},
    {-0.19509032201612828, 0.9807852804032304}, {-0.2902846772544624, 0.9569403357322088},
    {-0.3826834323650898, 0.9238795325112867}, {-0.47139673682599764, 0.881921264348355},
    {-0.5555702330196022, 0.8314696123025452}, {-0.6343932841636455, 0.773010453362737},
    {-0.7071067811865476, 0.7071067811865476}, {-0.773010453362737, 0.6343932841636455},
    {-0.8314696123025452, 0.5555702330196022}, {-0.881921264348355, 0.47139673682599764},
    {-0.9238795325112867, 0.3826834323650898}, {-0.9569403357322088, 0.2902846772544624},
    {-0.9807852804032304, 0.19509032201612828}, {-0.9951847266721969, 0.0980171403295606},
    {-1.0, 0.0}, {-0.9951847266721969, -0.0980171403295606},
    {-0.9807852804032304, -0.19509032201612828}, {-0.9569403357322088, -0.2902846772544624},
    {-0.9238795325112867, -0.3826834323650898}, {-0.881921264348355, -0.47139673682599764},
    {-0.8314696123025452, -0.5555702330196022}, {-0.773010453362737, -0.6343932841636455},
    {-0.7071067811865476, -0.7071067811865476}, {-0.6343932841636455, -0.773010453362737},
    {-0.5555702330196022, -0.8314696123025452}, {-0.47139673682599764, -0.881921264348355},
    {-0.3826834323650898, -0.9238795325112867}, {-0.2902846772544624, -0.9569403357322088},
    {-0.19509032201612828, -0.9807852804032304}, {-0.0980171403295606, -0.9951847266721969},
    {0.0, -1.0}, {0.0980171403295606, -0.9951847266721969},
    {0.19509032201612828, -0.9807852804032304}, {0.2902846772544624, -0.9569403357322088},
    {0.3826834323650898, -0.9238795325112867}, {0.47139673682599764, -0.881921264348355},
    {0.5555702330196022, -0.8314696123025452}, {0.6343932841636455, -0.773010453362737},
    {0.7071067811865476, -0.7071067811865476}, {0.773010453362737, -0.6343932841636455},
    {0.8314696123025452, -0.5555702330196022}, {0.881921264348355, -0.47139673682599764},
    {0.9238795325112867, -0.3826834323650898}, {0.9569403357322088, -0.2902846772544624},
    {0.9807852804032304, -0.19509032201612828}, {0.9951847266721969, -0.0980171403295606}};

// Adding 1.5 2^52 rounds a double of magnitude below 2^51 to the nearest
// integer, left in the low word of the sum.
constexpr double kRound = 6755399441055744.0;

// The arguments exp_node, cis_node and sin_node take must lie below 2^44 in
// magnitude (node_range: the high word without its sign; kRangeEnd: 2^44).
// Beyond, where a phase's own ulp passes 2^-9, and for non-finite arguments,
// a node takes CUDA's functions (node_slow, sin_slow; the adjoint's own).
constexpr unsigned kRangeEnd = 2u * 0x42B00000u;
__device__ __forceinline__ unsigned node_range(double x) { return 2u * (unsigned)__double2hiint(x); }

// e^x, branch-free (table-driven after Tang, ACM TOMS 15, 1989): x = k ln2/64
// + r, |r| <= 1.03 ln2/128, e^x = 2^(k/64) (1 + r + r^2 P(r)), P of degree 3
// (9e-18 absolute, node_math_coeffs.py), ln2/64 split into 21 bits and the
// rest.  x is held between -708 and 710 by its high word (as unsigned a more
// negative double is larger, as signed a negative one is negative), so that k
// fits the low word: below, some 1e-308 instead of 0, above 709.777 (k = 2^16, past
// 2^1023) infinity or NaN; a NaN may come out as either end, its callers test x.  In place of CUDA's
// exp on the 262k-contract Bates batch: 11.05 -> 10.61 ms (after cis_node and
// sin_node); a degree-11 polynomial without the table: 10.96 ms.
__device__ __forceinline__ double exp_node(double x) {
    const unsigned hu = min((unsigned)__double2hiint(x), 0xC0862000u);
    x = __hiloint2double(min((int)hu, 0x40863000), __double2loint(x));
    const double t = fma(x, 92.33245849609375, kRound);  // 64/ln2
    const int k = __double2loint(t);
    const double kd = __dsub_rn(t, kRound);
    const double tab = __ldg(g_exp2_tab + (k & 63));
    double r = fma(kd, -0.010830424726009369, x);
    r = fma(kd, 2.9760223436840126e-11, r);
    double q = 0.008333340287208557;
    q = fma(q, r, 0.04166671633720398);
    q = fma(q, r, 0.1666666666666286);
    q = fma(q, r, 0.5);
    q = fma(q, __dmul_rn(r, r), r);
    const double sc = __hiloint2double(__double2hiint(tab) + ((k >> 6) << 20), __double2loint(tab));
    return fma(sc, q, sc);
}

// cos and sin of r + K from r and the table's (cos K, sin K).
__device__ __forceinline__ void cis_tail(double r, double2 cs, double& re, double& im) {
    const double w = __dmul_rn(r, r);
    double a = fma(-0.00019840255845338106, w, 0.008333333322977338);
    a = fma(a, w, -0.16666666666666413);
    const double sr = fma(__dmul_rn(a, w), r, r);  // sin r
    double b = fma(2.4800567189231515e-05, w, -0.00138888880610466);
    b = fma(b, w, 0.04166666666656595);
    b = fma(b, w, -0.5);
    const double cm = __dmul_rn(b, w);  // cos r - 1
    re = fma(-cs.y, sr, fma(cs.x, cm, cs.x));
    im = fma(cs.x, sr, fma(cs.y, cm, cs.y));
}

// cos x and sin x, branch-free: x = k pi/32 + r, |r| <= pi/64, pi/32 split into
// 21 bits and the rest, sin r and cos r - 1 from polynomials (3e-19 and 6e-19
// absolute, node_math_coeffs.py), then the angle sum with the table's
// (cos, sin) of k pi/32.  Error a rounding or two of 1 per component.  In place
// of CUDA's sincos, with sin_node: 11.98 -> 11.05 ms on the same batch; reduced
// by pi with two longer polynomials and no table: 11.46 ms.
__device__ __forceinline__ void cis_node(double x, double& re, double& im) {
    const double t = fma(x, 10.185916357881302, kRound);  // 32/pi
    const int k = __double2loint(t);
    const double kd = __dsub_rn(t, kRound);
    const double2 cs = __ldg(g_cis_tab + (k & 63));
    double r = fma(kd, -0.09817475080490112, x);
    r = fma(kd, -1.9619779915655082e-08, r);
    cis_tail(r, cs, re, im);
}

// The same for x + a, x taken as exact and reduced before a is added.
__device__ __forceinline__ void cis_node(double x, double a, double& re, double& im) {
    const double t = fma(__dadd_rn(x, a), 10.185916357881302, kRound);
    const int k = __double2loint(t);
    const double kd = __dsub_rn(t, kRound);
    const double2 cs = __ldg(g_cis_tab + (k & 63));
    double r = fma(kd, -0.09817477042468103, x);
    r = __dadd_rn(fma(kd, -3.827021247335479e-18, r), a);
    cis_tail(r, cs, re, im);
}

// sin(x + a) w, branch-free, x taken as exact and reduced before a is added:
// k the integer nearest (x + a)/pi, r = (x - k pi) + a, |r| <= pi/2 (the first
// subtraction is one FMA, so it rounds at the size of a, not of x), sin r =
// r + r s Q(s), s = r^2, Q of degree 7 (3.4e-17 relative), the sign (-1)^k put
// on w.
__device__ __forceinline__ double sin_node(double x, double a, double w) {
    const double t = fma(__dadd_rn(x, a), 0.3183098861837907, kRound);  // 1/pi
    const int k = __double2loint(t);
    const double kd = __dsub_rn(t, kRound);
    double r = fma(kd, -3.141592653589793, x);
    r = __dadd_rn(fma(kd, -1.2246467991473532e-16, r), a);
    const double s = __dmul_rn(r, r);
    double q = 2.7314440856698874e-15;
    q = fma(q, s, -7.643941903057172e-13);
    q = fma(q, s, 1.6058976370914024e-10);
    q = fma(q, s, -2.5052107629086277e-08);
    q = fma(q, s, 2.755731921990685e-06);
    q = fma(q, s, -0.00019841269841263388);
    q = fma(q, s, 0.008333333333333344);
    q = fma(q, s, -0.16666666666666666);
    const double sw = __hiloint2double(__double2hiint(w) ^ (k << 31), __double2loint(w));
    return __dmul_rn(fma(__dmul_rn(q, s), r, r), sw);
}

// Error-free transformations (Knuth's TwoSum, Dekker's Fast2Sum, the FMA
// product residual) and double-double arithmetic, for log_cr below.
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
    s = __dadd_rn(a, b);
    const double bb = __dsub_rn(s, a);
    e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}
__device__ __forceinline__ void fast_two_sum(double a, double b, double& s, double& e) {  // |a| >= |b|
    s = __dadd_rn(a, b);
    e = __dsub_rn(b, __dsub_rn(s, a));
}
struct DD {
    double hi, lo;
};
__device__ __forceinline__ DD dd_add(DD a, DD b) {
    double s, e;
    two_sum(a.hi, b.hi, s, e);
    e = __dadd_rn(e, __dadd_rn(a.lo, b.lo));
    DD r;
    fast_two_sum(s, e, r.hi, r.lo);
    return r;
}
__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = __dmul_rn(a.hi, b.hi);
    double e = fma(a.hi, b.hi, -p);
    e = fma(a.hi, b.lo, fma(a.lo, b.hi, e));
    DD r;
    fast_two_sum(p, e, r.hi, r.lo);
    return r;
}

// ln(v) correctly rounded (to nearest) for positive normal v, other arguments
// through CUDA's log.  Used once per integral for x = ln(S/K): the integrand's
// phase u x reaches 1e7 and beyond on short-dated deep-wing contracts, where
// one ulp of x moves a node value by 1e-9 relative, so x must be the value
// the reference's own libm log returns -- the correctly rounded one.  Method
// (the atanh series of the logarithm, in double-double): v = 2^k m with m in
// [sqrt(1/2), sqrt 2); s = (m - 1)/(m + 1) as a double-double;
// ln m = 2s + 2s^3/3 + 2s^5/5 + s^7 q(s^2), q(w) = sum_j 2 w^j/(2j + 7)
// (|s| <= 0.1716, the first three terms in double-double, q in double); plus
// k ln 2 with ln 2 as a double-double.  The sum carries about 2^-68 relative
// error, so the final rounding is correct unless ln v lies within that of a
// rounding midpoint.
__device__ __forceinline__ double log_cr(double v) {
    if (!(v >= 0x1p-1022 && v <= 0x1.fffffffffffffp+1023)) return log(v);
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int k = (hi - 0x3FE6A09E) >> 20;  // 0x3FE6A09E: high word of sqrt(1/2)
    const double m = __hiloint2double(hi - k * 0x100000, lo);
    const double f = __dsub_rn(m, 1.0);  // exact (Sterbenz)
    double dh, dl;
    fast_two_sum(2.0, f, dh, dl);  // m + 1 = 2 + f exactly
    const double sh = __ddiv_rn(f, dh);
    const double res = __dsub_rn(fma(-sh, dh, f), __dmul_rn(sh, dl));  // f - sh (dh + dl)
    DD S;
    fast_two_sum(sh, __ddiv_rn(res, dh), S.hi, S.lo);
    const DD W = dd_mul(S, S);
    const DD S3 = dd_mul(S, W);
    const DD S5 = dd_mul(S3, W);
    const double w = W.hi;
    double q = 0.07407407407407407;
    q = fma(q, w, 0.08);
    q = fma(q, w, 0.08695652173913043);
    q = fma(q, w, 0.09523809523809523);
    q = fma(q, w, 0.10526315789473684);
    q = fma(q, w, 0.11764705882352941);
    q = fma(q, w, 0.13333333333333333);
    q = fma(q, w, 0.15384615384615385);
    q = fma(q, w, 0.18181818181818182);
    q = fma(q, w, 0.2222222222222222);
    q = fma(q, w, 0.2857142857142857);
    const double rest = __dmul_rn(__dmul_rn(S5.hi, w), q);
    DD acc{__dmul_rn(2.0, S.hi), __dmul_rn(2.0, S.lo)};
    acc = dd_add(acc, dd_mul(S3, DD{0.6666666666666666, 3.700743415417188e-17}));  // 2/3
    acc = dd_add(acc, dd_mul(S5, DD{0.4, -2.2204460492503132e-17}));               // 2/5
    acc = dd_add(acc, DD{rest, 0.0});
    const double kd = (double)k;
    DD kl;
    kl.hi = __dmul_rn(kd, 0.6931471805599453);  // ln 2 = 0.6931471805599453 + 2.3190468138462996e-17
    kl.lo = fma(kd, 2.3190468138462996e-17, fma(kd, 0.6931471805599453, -kl.hi));
    acc = dd_add(kl, acc);
    return __dadd_rn(acc.hi, acc.lo);
}

__device__ __forceinline__ Cx cadd(Cx a, Cx b) { return Cx{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ Cx csub(Cx a, Cx b) { return Cx{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ Cx cmul(Cx a, Cx b) {
    return Cx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ Cx cscale(Cx a, double s) { return Cx{a.re * s, a.im * s}; }
// conj/|b|^2 division (the num-complex algorithm), with one reciprocal.
__device__ __forceinline__ Cx cdiv(Cx a, Cx b) {
    double inv = 1.0 / (b.re * b.re + b.im * b.im);
    return Cx{(a.re * b.re + a.im * b.im) * inv, (a.im * b.re - a.re * b.im) * inv};
}
__device__ __forceinline__ Cx cexp(Cx z) {
    double s, c;
    sincos(z.im, &s, &c);
    double e = exp(z.re);
    return Cx{e * c, e * s};
}
__device__ __forceinline__ Cx clog(Cx z) { return Cx{log(hypot(z.re, z.im)), atan2(z.im, z.re)}; }

// heston.rs:155-175 fast_csqrt, branch-free: the safe component is
// w = sqrt((|a| + r)/2); the other is b/(2w) (its magnitude when a < 0).
// Same values as the reference's two branches, including the b == 0 cases.
__device__ __forceinline__ Cx fast_csqrt(double a, double b) {
    double r = hypot(a, b);
    double w = sqrt(0.5 * (r + fabs(a)));
    double q = (w > 0.0) ? (0.5 * b) / w : b;
    return (a >= 0.0) ? Cx{w, q} : Cx{fabs(q), copysign(w, b)};
}

// Per-integral constants (everything that does not depend on the node),
// folded so that the node evaluation does as little as possible:
//   xi   = (xr, -rs u)                       xi = kappa - i rho sigma phi, phi = u + i phi_im
//   z    = xi^2 + sigma^2 phi(phi+i)         = (zr0 + zr2 u^2, zi1 u): zr0 = xr^2,
//                                            zr2 = sigma^2 (1 - rho^2), zi1 = sgn sigma^2 - 2 xr rs
//   C    = kts ((xi - d) T - 2 Log A)        d = sqrt z
//   D    = -v0 phi(phi+i) (1 - e)/(2 N)      phi(phi+i) = u^2 + i sgn u = sgn u (sgn u + i)
//   Re Z = Re C + Re D + r T + Re(-Log CF(-i)) for P1, Re C + Re D for P2
//   Im Z = Im C + Im D + rtl u + z0im + (x u mod 2 pi)    x = ln(S/K), rtl = r T [- lambda T comp]
//   Bates: jump = exp(jr0 - hs2 u^2 + i jmu u);  J = lt (jump - 1 - i phi comp)
// (kept: halves of xr, -rs, zr0, zr2, zi1; kts2 = 2 kts; z0re: every real term
// that is constant over the nodes; t...: with xi and d taken times T, which
// A and, with one T in the factor tnhv0 = -sgn v0 T/2, D are free of, the
// exponent d T and the term (xi - d) T take no product of their own)
// The C and D of heston.rs:120-124 are formed without g = (xi - d)/(xi + d):
// with m = (xi - d)/2, e = exp(-d T), o = 1 - e and N = d + m o (half of
// (xi + d) - (xi - d) e),
//   A = (g e - 1)/(g - 1) = N/d   and, since xi^2 - d^2 = -sigma^2 phi(phi+i),
//   (xi - d) o/(1 - g e) = (xi^2 - d^2) o/(2 N) = -sigma^2 phi(phi+i) o/(2 N),
// so sigma^2 cancels in D, |A|^2 = |N|^2/|z| needs no quotient of its own, and
// a node takes one complex reciprocal (of N) where the literal sequence takes
// four.
struct CfConsts {
    // the fast node evaluation's: xi, z, d, m and N times T (z times T^2)
    double thxr, tnhrs, thzr0, thzr2, thzi1, tnhv0, kts, kts2, rtl, z0re, z0im;
    double jr0, hs2, jmu, lt, x;
    int sgn_bit;
    unsigned u_span;  // u it applies to: high words in [kULow, kULow + u_span)
    // the same without the factor T, for the slow evaluation and the adjoint
    double hxr, nhrs, hzr0, hzr2, hzi1, t, sgn, phi_im, v0, rt, comp;
    double z0;  // z0re without the logarithm's constant
};
constexpr unsigned kULow = 0x3D71979Au;  // the first high word above that of 1e-12

// stable_cf at a general complex phi, following heston.rs:113-127's operation
// order (used once per integral for the P1 normaliser CF(-i)).
__device__ __forceinline__ Cx stable_cf_ref(Cx phi, double t, double r, double v0, double kappa,
                                            double theta, double sigma, double rho) {
    const Cx I{0.0, 1.0};
    Cx xi = csub(Cx{kappa, 0.0}, cmul(cscale(phi, rho * sigma), I));
    Cx z = cadd(cmul(xi, xi), cmul(cscale(phi, sigma * sigma), cadd(phi, I)));
    Cx d = fast_csqrt(z.re, z.im);
    Cx g = cdiv(csub(xi, d), cadd(xi, d));
    Cx edt = cexp(cscale(Cx{-d.re, -d.im}, t));
    Cx ge = cmul(g, edt);
    Cx a = cdiv(Cx{ge.re - 1.0, ge.im}, Cx{g.re - 1.0, g.im});
    Cx la = clog(a);
    Cx xmd = csub(xi, d);
    Cx c = cscale(Cx{xmd.re * t - 2.0 * la.re, xmd.im * t - 2.0 * la.im}, (kappa * theta) / (sigma * sigma));
    Cx num = cmul(cscale(xmd, v0), Cx{1.0 - edt.re, 0.0 - edt.im});
    Cx den = cscale(Cx{1.0 - ge.re, 0.0 - ge.im}, sigma * sigma);
    Cx dd = cdiv(num, den);
    Cx e = cadd(cadd(cscale(cmul(cscale(phi, r), I), t), c), dd);
    return cexp(e);
}

// bates.rs:77-83 jump_cf at a general complex phi (normaliser only).
__device__ __forceinline__ Cx jump_cf_ref(Cx phi, double t, double lambda, double mu_j, double sigma_j) {
    const Cx I{0.0, 1.0};
    double comp = exp(mu_j + (0.5 * sigma_j) * sigma_j) - 1.0;
    Cx a = cscale(cmul(phi, I), mu_j);
    Cx b = cscale(cscale(cmul(cscale(phi, 0.5), phi), sigma_j), sigma_j);
    Cx jump = cexp(csub(a, b));
    Cx inner = csub(Cx{jump.re - 1.0, jump.im}, cscale(cmul(I, phi), comp));
    return cexp(cscale(inner, lambda * t));
}

// Log CF(-i) by the reference's sequence; rare (make_consts), so a call.
static __device__ __noinline__ Cx log_cf_mi_ref(double t, double r, double v0, double kappa, double theta, double sigma,
                                                double rho, bool bates, double lambda, double mu_j, double sigma_j) {
    const Cx phi_mi{0.0, -1.0};
    Cx m = stable_cf_ref(phi_mi, t, r, v0, kappa, theta, sigma, rho);
    if (bates) m = cmul(m, jump_cf_ref(phi_mi, t, lambda, mu_j, sigma_j));
    return clog(m);
}

// Build the per-integral constants.  which: 0 = P1 (stock measure), 1 = P2.
__device__ __forceinline__ CfConsts make_consts(double s, double k, double t, double r, const double* p,
                                                bool bates, int which) {
    const double v0 = p[0], kappa = p[1], theta = p[2], sigma = p[3], rho = p[4];
    CfConsts C;
    const double rs = rho * sigma, sig2 = sigma * sigma;
    C.kts = (kappa * theta) / (sigma * sigma);
    C.v0 = v0;
    C.t = t;
    C.rt = r * t;
    C.x = log_cr(s / k);  // heston.rs:86, rounded as the platform libm rounds it
    C.phi_im = (which == 0) ? -1.0 : 0.0;
    C.sgn = (which == 0) ? -1.0 : 1.0;
    const double xr = kappa + rs * C.phi_im;
    C.hxr = 0.5 * xr;
    C.nhrs = -0.5 * rs;
    C.hzr0 = 0.5 * (xr * xr);
    C.hzr2 = 0.5 * (sig2 * ((1.0 - rho) * (1.0 + rho)));
    C.hzi1 = 0.5 * fma(-2.0 * xr, rs, sig2 * C.sgn);
    C.kts2 = 2.0 * C.kts;
    C.tnhv0 = -0.5 * v0 * C.sgn * t;
    // from the rounded xr T, rs T and sigma T, so that z stays the square (and xi
    // the root) of one xi and d cancels against it as without the factor
    const double tsg = sigma * t, ts2 = 0.5 * (tsg * tsg);
    C.thxr = C.hxr * t;
    C.tnhrs = C.nhrs * t;
    C.thzr0 = 2.0 * (C.thxr * C.thxr);
    C.thzr2 = ts2 * ((1.0 - rho) * (1.0 + rho));
    C.thzi1 = fma(4.0 * C.thxr, C.tnhrs, ts2 * C.sgn);
    C.sgn_bit = which == 0 ? (int)0x80000000 : 0;
    double lt = 0.0, mu_j = 0.0, hs2 = 0.0, comp = 0.0;
    if (bates) {
        lt = p[5] * t;
        mu_j = p[6];
        hs2 = 0.5 * p[7] * p[7];
        comp = exp(p[6] + (0.5 * p[7]) * p[7]) - 1.0;
    }
    C.lt = lt;
    C.hs2 = hs2;
    C.comp = comp;
    C.jr0 = -C.phi_im * mu_j + hs2 * (C.phi_im * C.phi_im);
    C.jmu = mu_j - 2.0 * hs2 * C.phi_im;
    C.rtl = C.rt - lt * comp;
    double lnm_re = 0.0, lnm_im = 0.0;
    if (which == 0) {
        // CF(-i) = e^{rT} in exact arithmetic (C = D = 0 there, jump factor 1),
        // and the reference's operation sequence reproduces that to the last
        // ulp or so whenever xi(-i) = kappa - rho sigma (C.xr) is a positive
        // normal number and the other terms are moderate: then Log CF(-i) is
        // rT.  Everywhere else -- xi(-i) <= 0, where xi + d = 0 makes the
        // reference's CF(-i) NaN and drops every P1 node, and any extreme or
        // non-finite parameter -- it is evaluated with the reference's own
        // sequence.  (The regular case skips two complex exponentials, three
        // complex divisions and two complex logarithms per P1 integral.)
        bool regular = xr > 1e-100 && xr < 1e100 && sig2 > 1e-100 && C.kts < 1e4 &&
                       v0 * xr < 1e4 * sig2 && fabs(C.rt) < 700.0 && t < 1e3;
        if (bates) regular = regular && fabs(p[6] + 0.5 * p[7] * p[7]) < 50.0 && fabs(lt) * (comp + 1.0) < 1e4;
        if (regular) {
            lnm_re = -C.rt;
        } else {
            const Cx lm = log_cf_mi_ref(t, r, v0, kappa, theta, sigma, rho, bates, bates ? p[5] : 0.0,
                                        bates ? p[6] : 0.0, bates ? p[7] : 0.0);
            lnm_re = -lm.re;
            lnm_im = -lm.im;
        }
    }
    C.z0 = (-C.rt * C.phi_im + lnm_re) + lt * (C.phi_im * comp - 1.0);
    C.z0re = fma(C.kts, 0.6931471805599453, C.z0);
    C.z0im = lnm_im;
    // Where the fast evaluation applies, as a range of u: T > 1e-9 and |rho| <= 1
    // (Re z >= 0), a finite normaliser, u >= 1e-12, and every argument of its
    // functions that a bound on u bounds below 2^43: |d| T <= T (|xr| + 2 r1 +
    // r2) max(u, 1) with r1^2 = |zi1|, r2^2 = zr2 (and 2 sqrt y <= 1 + y), |jmu| u,
    // |jr0| + hs2 u^2.
    const float tf = (float)t, h2 = (float)C.hs2;
    const float q = tf * (2.0f + (float)(fabs(xr) + fma(2.0, fabs(C.hzi1), C.hzr2))) + (float)(fabs(C.jmu) + fabs(C.jr0));
    const bool fast = tf > 1e-9f && C.hzr2 >= 0.0 && q < 8.796e12f && h2 < 8.796e12f && isfinite(C.z0re) && isfinite(C.z0im);
    const float top = fminf(__fdividef(8.79e12f, q), 2.9e6f * rsqrtf(h2));
    C.u_span = fast && top > 1e-3f ? (unsigned)__double2hiint((double)fminf(top, 1e30f)) - kULow : 0u;
    return C;
}

// u = (1 - t)/t of a node, rounded as heston.rs:223 rounds it (the IEEE
// quotient): at large u the phase u x makes every ulp of u count.  From
// y ~ 1/t (= (1 - t) itt with itt ~ 1/((1 - t) t), a few ulps) the quotient
// u0 = (1 - t) y is within a few ulps; one correction with the exact residual
// (1 - t) - u0 t (an FMA) lands within about 1e-15 ulp of the true quotient,
// so its rounding is the IEEE one short of a midpoint that close (checked
// against IEEE division by ope_selftest_node_u).
__device__ __forceinline__ double node_u(double omt, double tn, double itt) {
    const double yt = omt * itt;
    const double u0 = omt * yt;
    return fma(fma(-u0, tn, omt), yt, u0);
}

// The strike-free part of a node (heston.rs:221-227 with the merged-exponent
// integrand): W = e^{Re Z} / ((1 - t) t), A = Im Z - (u x mod 2 pi), and the
// node's u = (1 - t)/t (which node_geom computes alone, bit for bit).
struct NodeCf {
    double w, a, u;
};

__device__ __forceinline__ void node_geom(double tn, double& u, double& itt) {
    const double omt = 1.0 - tn;
    itt = rcp_nr(omt * tn);
    u = node_u(omt, tn, itt);
}

// u of a node alone (bit for bit node_geom's).
__device__ __forceinline__ double node_u_of(double tn) {
    double u, itt;
    node_geom(tn, u, itt);
    return u;
}

// FAST: branch-free, with the functions above; returns whether they applied: u
// in the integral's range (CfConsts::u_span) and Z below 2^43, its real part
// below 600: with 1e-12 <= u < 1e30 the factor 1/((1 - t) t) is below 2e30, so
// that W stays below 1e291 and the sums over 200 panels are finite.  Not FAST: CUDA's functions and the
// square root's other branch.
//
// What bounds it: register-file reads and issue slots (an FMA of three
// different registers takes 3 cycles of a scheduler's operand reads, of two
// registers and an immediate 2, an addition or a product 2).  So constants are
// immediates wherever 21 bits do (node_math_coeffs.py), products are folded
// into FMAs and per-integral constants, and selects are avoided.  On 262k
// contracts, Bates / Heston, ms:
//   12.99 / 11.45  with g = (xi - d)/(xi + d) and CUDA's functions
//   12.03 / 10.52  C and D without g, merged reciprocals
//   10.17 /  8.95  own exponential, sine and cosine, one range branch per node
//    9.79 /  8.64  (the bisection step's bookkeeping, quadrature.cuh)
//    9.66 /  8.45  21-bit leading coefficients and reductions
//    9.36 /  7.88  N and o as below, arg_node's rotation, integer clamps in
//                  exp_node (Heston at 72 registers; 8.12 at 64)
//    9.05 /  7.61  (the step's argmax)
//    8.45 /  7.43  everything times T, one test of u for the arguments, no
//                  tests on the value, the normaliser's general form a call
//                  (both at 72 registers)
// Two integrals per warp side by side (128 registers) issue 13 % fewer
// instructions and read as many registers: 9.61 / 8.60 ms against 9.74 / 8.60.
template <bool BATES, bool FAST>
__device__ __forceinline__ bool node_eval(const CfConsts& C, double tn, NodeCf& n) {
    double u, itt;  // (1 - t) / t and 1 / ((1 - t) t)
    node_geom(tn, u, itt);
    const double u2 = __dmul_rn(u, u);
    // xi/2 = (hxr, hxi); z/2, z = xi^2 + sigma^2 phi(phi+i) = (xr^2 + zr2 u^2, zi1 u)
    const double hxr = FAST ? C.thxr : C.hxr, hxi = __dmul_rn(FAST ? C.tnhrs : C.nhrs, u);
    const double zr = FAST ? fma(C.thzr2, u2, C.thzr0) : fma(C.hzr2, u2, C.hzr0);
    const double zi = __dmul_rn(FAST ? C.thzi1 : C.hzi1, u);
    // d = sqrt z: Re d = sqrt(|z/2| + Re z/2), Im d = (Im z/2) / Re d
    const double zz = fma(zr, zr, __dmul_rn(zi, zi));
    const double az = __dmul_rn(zz, rsqrt_nr(zz));  // |z| / 2
    const double s2 = __dadd_rn(FAST ? zr : fabs(zr), az);
    const double iw = rsqrt_nr(s2);
    double dre = __dmul_rn(s2, iw), dim = __dmul_rn(zi, iw);
    if (!FAST && zr < 0.0) {
        const double w = dre;
        dre = fabs(dim);
        dim = copysign(w, zi);
    }
    const double mr = fma(dre, -0.5, hxr), mi = fma(dim, -0.5, hxi);  // m = (xi - d) / 2
    // e = exp(-d T) = em (ec - i es), o = 1 - e
    double em, ec, es;
    if (FAST) {
        cis_node(dim, ec, es);
        em = exp_node(-dre);
    } else {
        sincos(dim * C.t, &es, &ec);
        em = exp(-dre * C.t);
    }
    const double omr = fma(-em, ec, 1.0), omi = __dmul_rn(em, es);
    // N = d + m o
    const double nr = fma(-mi, omi, fma(mr, omr, dre));
    const double ni = fma(mr, omi, fma(mi, omr, dim));
    const double nn = fma(nr, nr, __dmul_rn(ni, ni));
    // Log A, A = N / d: |A|^2 = nn / (2 az) (the 2 is in z0re), arg A = arg(N conj(d))
    double ia;
    const double la = log_ratio(nn, az, ia);
    const double li = arg_node(fma(ni, dre, __dmul_rn(-nr, dim)), fma(nr, dre, __dmul_rn(ni, dim)));
    // D = -(v0/2) phi(phi+i) o / N, phi(phi+i) = u (u + i sgn) = sgn u (sgn u + i)
    const double qr = fma(omr, nr, __dmul_rn(omi, ni)), qi = fma(omi, nr, __dmul_rn(-omr, ni));
    const double su = __hiloint2double(__double2hiint(u) | C.sgn_bit, __double2loint(u));
    const double s = __dmul_rn(__dmul_rn(FAST ? C.tnhv0 : -0.5 * C.v0 * C.sgn, u), ia);
    // Re, Im Z = kts ((xi - d) T - 2 Log A) + D + z0 + i (r T u)
    const double km = FAST ? C.kts2 : C.kts2 * C.t;
    double zre = fma(km, mr, fma(-C.kts, la, fma(s, fma(su, qr, -qi), C.z0re)));
    double zim = fma(km, mi, fma(-C.kts2, li, fma(s, fma(su, qi, qr), fma(C.rtl, u, C.z0im))));
    if (BATES) {
        const double tj = __dmul_rn(C.jmu, u), ej = fma(-C.hs2, u2, C.jr0);
        double jc, js, je;
        if (FAST) {
            cis_node(tj, jc, js);
            je = __dmul_rn(C.lt, exp_node(ej));
        } else {
            sincos(tj, &js, &jc);
            je = __dmul_rn(C.lt, exp(ej));
        }
        zre = fma(je, jc, zre);
        zim = fma(je, js, zim);
    }
    n.u = u;
    n.a = zim;
    n.w = __dmul_rn(FAST ? exp_node(zre) : exp(zre), itt);
    if (!FAST) return true;
    const int hz = __double2hiint(zre);
    return (unsigned)__double2hiint(u) - kULow < C.u_span && hz < 0x4082C000 && (unsigned)hz < 0xC2A00000u &&
           node_range(zim) < 2u * 0x42A00000u;
}

// The rare nodes the fast evaluation does not apply to (internal linkage:
// within the calling kernel's register budget): W = 0 where the reference's g(t)
// is 0 (t <= 0, u < 1e-12) or W or the phase is not finite, and a phase beyond
// 2^44, whose last place passes 2^-9, brought below 2 pi.
template <bool BATES>
static __device__ __noinline__ NodeCf node_slow(const CfConsts& C, double tn) {
    NodeCf n;
    node_eval<BATES, false>(C, tn, n);
    if (!(tn > 0.0 && n.u >= 1e-12 && isfinite(n.w) && isfinite(n.a))) return NodeCf{0.0, 0.0, 0.0};
    if (fabs(n.a) >= 0x1p44) n.a = fmod(n.a, 6.283185307179586);
    return n;
}

template <bool BATES>
__device__ __forceinline__ NodeCf node_cf(const CfConsts& C, double tn) {
    NodeCf n;
    if (!node_eval<BATES, true>(C, tn, n)) n = node_slow<BATES>(C, tn);
    return n;
}

// One strike's node value from the strike-free part: Im(e^Z) / u / t^2 =
// e^{Re Z} sin(Im Z) / ((1 - t) t) = sin(A + phase) W with W = E itt; 0
// where the reference's g(t) is 0 (t <= 0, u < 1e-12) or the value is not
// finite.  The phase of e^{iux} (heston.rs:107): u x rounded as the
// reference rounds it, reduced modulo 2 pi without loss (Cody and Waite's
// argument reduction, 2 pi split into two doubles and the products taken
// exactly by FMA: |u x - n 2 pi| < 4 makes the first step exact), so that
// adding the CF's own phase costs an ulp of a number below 4 however large
// u x is.  The reference adds the two phases exactly too, through the
// complex product e^{iux} CF (an unreduced sum would lose ulp(u x), 1e-9 at
// u x = 1e7, on short-dated deep-wing contracts).
// W is 0 where that value is to be 0 (node_slow), so only a phase u x that is
// out of sin_node's range or not finite needs a test.
static __device__ __noinline__ double sin_slow(double ux, double a, double w) {
    const double nq = rint(ux * 0.15915494309189535);  // 1 / (2 pi)
    const double uxr = fma(-nq, 2.4492935982947064e-16, fma(-nq, 6.283185307179586, ux));
    const double v = __dmul_rn(sin(__dadd_rn(a, uxr)), w);
    return isfinite(v) ? v : 0.0;
}
__device__ __forceinline__ double node_finish(double x, double u, double a, double w) {
    const double ux = __dmul_rn(u, x);
    double v = sin_node(ux, a, w);
    if (node_range(ux) >= kRangeEnd) v = sin_slow(ux, a, w);
    return v;
}

}  // namespace ope
