// Reverse-mode derivative of one Gil-Pelaez node with respect to the model
// parameters (v0, kappa, theta, sigma, rho[, lambda, mu_j, sigma_j]).
//
// Reference: ad.rs:609-731 (forward-mode Dual through stable_cf_dual,
// jump_factor and dual_integrand, integrated over the primal's adaptive
// panel set).  Same quantity, computed backwards: the node value is
//
//     g(t) = Im(W) / (u t^2),  W = exp(Z),  Z = kts*Ch + v0*D0 + i r phi T + i u x - Log CF(-i) [+ J]
//
// with the C and D of cf_device.cuh: m = (xi - d)/2, e = exp(-d T), o = 1 - e,
// N = d + m o, Ch = 2 (m T - Log(N/d)) and D0 = -phi(phi+i) o/(2 N) (neither
// has a sigma of its own).  Every intermediate is a holomorphic function of
// xi and d, so the backward pass is two complex partials.  With q = o/N,
// t = T e/N, n = N_d/N = 1/N - q/2 + m t (N_xi/N = q/2) and D = v0 D0:
//
//   Z_xi = kts (T - q) - D q/2
//   Z_d  = kts (2/d - T) - v0 phi(phi+i) t/2 - (2 kts + D) n
//
// and, through z = d^2 = xi^2 + sigma^2 phi(phi+i), X = Z_d/d and
// Y = Z_xi + xi X:
//
//   dZ/dv0    = D0
//   dZ/dkappa = Y + Ch * theta / sigma^2
//   dZ/dtheta = Ch * kappa / sigma^2
//   dZ/dsigma = rho Y s + sigma X phi(phi+i) - 2 kts Ch / sigma      s = phi_im - i u
//   dZ/drho   = sigma Y s
//
// and dg/dp = Im(W dZ/dp) / (u t^2).  The five Heston derivatives are linear,
// with coefficients constant over the integral, in D0, Ch, Y, Y s and
// X phi(phi+i): a node adds those five, and each chunk's sums are combined
// once.  The CF is recomputed here, nothing from the primal pass is stored.
//
// Log CF(-i) = r T whatever the parameters (C = D = J = 0 at phi = -i), so it
// contributes nothing to the derivatives; where the reference's evaluation of
// it is not finite (kappa <= rho sigma), every P1 node's value is not finite
// and every node is dropped (ad.rs:679-682), here through z0.
#pragma once

#include "cf_device.cuh"

namespace ope {

struct C2 {
    double re, im;
};
__device__ __forceinline__ C2 c2(double re, double im) { return C2{re, im}; }
__device__ __forceinline__ C2 operator+(C2 a, C2 b) { return C2{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ C2 operator-(C2 a, C2 b) { return C2{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ C2 operator*(C2 a, C2 b) {
    return C2{fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ C2 operator*(C2 a, double s) { return C2{a.re * s, a.im * s}; }
__device__ __forceinline__ C2 operator*(double s, C2 a) { return C2{a.re * s, a.im * s}; }
// a b + c
__device__ __forceinline__ C2 cfma(C2 a, C2 b, C2 c) {
    return C2{fma(-a.im, b.im, fma(a.re, b.re, c.re)), fma(a.im, b.re, fma(a.re, b.im, c.im))};
}
__device__ __forceinline__ C2 cfma(double a, C2 b, C2 c) { return C2{fma(a, b.re, c.re), fma(a, b.im, c.im)}; }

// Model parameters of the chain, and what they give once per integral.
struct GradParams {
    double sigma, rho, sigma_j;
    double tis2, kis2;  // theta / sigma^2, kappa / sigma^2
    double sk;          // 2 kts / sigma
};

__device__ __forceinline__ GradParams make_grad_params(const double* p, bool bates) {
    GradParams G;
    const double is2 = 1.0 / (p[3] * p[3]);
    G.sigma = p[3];
    G.rho = p[4];
    G.sigma_j = bates ? p[7] : 0.0;
    G.tis2 = p[2] * is2;
    G.kis2 = p[1] * is2;
    G.sk = 2.0 * ((p[1] * p[2]) * is2) / p[3];
    return G;
}

// A node's intermediates, and its W = exp(Z) / (u t^2).  node_parts' `ok`:
// the value belongs to the sum (0 where the reference's g(t) is: u < 1e-12, or
// a W that is not finite).
struct NodeParts {
    C2 d, id, m, e, iN, q, Ch, D0;
    double u, su, hs;  // su = sgn u, hs = -sgn u / 2
    C2 W;
    C2 jump;
};

// -(phi(phi+i)/2) a: phi(phi+i) = sgn u (sgn u + i)
__device__ __forceinline__ C2 half_wphi(const NodeParts& n, C2 a) {
    return c2(n.hs * fma(n.su, a.re, -a.im), n.hs * fma(n.su, a.im, a.re));
}

// FAST: the functions of cf_device.cuh, valid while `range` < kRangeEnd.
template <bool BATES, bool FAST>
__device__ __forceinline__ NodeParts node_parts(const CfConsts& C, double tn, bool& ok, unsigned& range) {
    NodeParts n;
    const double omt = 1.0 - tn;
    const double itt = rcp_nr(omt * tn);  // 1 / ((1 - t) t), as the pricing node evaluation
    const double u = node_u(omt, tn, itt);
    const double u2 = u * u, T = C.t;
    n.u = u;
    n.su = __hiloint2double(__double2hiint(u) | C.sgn_bit, __double2loint(u));
    n.hs = -0.5 * n.su;
    const double hxi = C.nhrs * u;
    const double zr = fma(C.hzr2, u2, C.hzr0), zi = C.hzi1 * u;  // z / 2
    const double zz = fma(zr, zr, zi * zi);
    const double iaz = rsqrt_nr(zz);  // 1 / |z/2|
    const double az = zz * iaz;
    const double s2 = (FAST ? zr : fabs(zr)) + az;
    const double iw = rsqrt_nr(s2);
    n.d = c2(s2 * iw, zi * iw);
    if (!FAST && zr < 0.0) n.d = c2(fabs(n.d.im), copysign(n.d.re, zi));
    n.id = c2(n.d.re * (0.5 * iaz), -n.d.im * (0.5 * iaz));
    n.m = c2(fma(n.d.re, -0.5, C.hxr), fma(n.d.im, -0.5, hxi));
    const double th = -n.d.im * T, et = -n.d.re * T;
    double em, ec, es;
    if (FAST) {
        cis_node(th, ec, es);
        em = exp_node(et);
    } else {
        sincos(th, &es, &ec);
        em = exp(et);
    }
    n.e = c2(em * ec, em * es);
    const C2 o = c2(fma(-em, ec, 1.0), -n.e.im);
    const C2 N = cfma(n.m, o, n.d);
    const double nn = fma(N.re, N.re, N.im * N.im);
    const double ar = fma(N.re, n.d.re, N.im * n.d.im), ai = fma(N.im, n.d.re, -N.re * n.d.im);  // N conj(d)
    double ia, la, li;
    if (FAST) {
        la = log_ratio(nn, az, ia) - 0.69314718055994529;  // |d|^2 = 2 az
        li = arg_node(ai, ar);
    } else {
        ia = 1.0 / nn;
        la = log(nn / (2.0 * az));
        li = atan2(ai, ar);
    }
    n.iN = c2(N.re * ia, -N.im * ia);
    n.q = o * n.iN;
    n.Ch = c2(fma(2.0 * T, n.m.re, -la), fma(2.0 * T, n.m.im, -2.0 * li));
    n.D0 = half_wphi(n, n.q);
    double zre = fma(C.kts, n.Ch.re, fma(C.v0, n.D0.re, C.z0));
    double zim = fma(C.kts, n.Ch.im, fma(C.v0, n.D0.im, fma(C.rtl, u, C.z0im)));
    if (FAST) range = max(node_range(et), (unsigned)__double2hiint(zr));
    if (BATES) {
        const double tj = C.jmu * u, ej = fma(-C.hs2, u2, C.jr0);
        double jc, js, je;
        if (FAST) {
            range = max(range, max(node_range(tj), node_range(ej)));
            cis_node(tj, jc, js);
            je = exp_node(ej);
        } else {
            sincos(tj, &js, &jc);
            je = exp(ej);
        }
        n.jump = c2(je * jc, je * js);
        zre = fma(C.lt, n.jump.re, zre);
        zim = fma(C.lt, n.jump.im, zim);
    }
    const double ux = __dmul_rn(u, C.x);
    double ez, wc, ws;
    if (FAST) {
        range = max(max(range, node_range(zre)), max(node_range(ux), node_range(zim)));
        cis_node(ux, zim, wc, ws);
        ez = exp_node(zre);
    } else {
        const double nq = rint(ux * 0.15915494309189535);  // 1 / (2 pi)
        sincos(zim + fma(-nq, 2.4492935982947064e-16, fma(-nq, 6.283185307179586, ux)), &ws, &wc);
        ez = exp(zre);
    }
    const double w = ez * itt;
    n.W = c2(w * wc, w * ws);
    ok = u >= 1e-12 && isfinite(n.W.im);
    return n;
}

// The five quantities the Heston derivatives are made of: D0, Ch, Y, Y s and
// X phi(phi+i).
__device__ __forceinline__ void heston_partials(const CfConsts& C, const NodeParts& n, C2* out) {
    const double T = C.t;
    const C2 D = n.D0 * C.v0;
    const C2 t = n.e * n.iN * T;
    const C2 nd = cfma(n.m, t, cfma(-0.5, n.q, n.iN));
    const C2 Zx = c2(C.kts * T, 0.0) - n.q * c2(fma(0.5, D.re, C.kts), 0.5 * D.im);
    const C2 Zd = cfma(C.v0, half_wphi(n, t), c2(fma(C.kts2, n.id.re, -C.kts * T), C.kts2 * n.id.im)) -
                  nd * c2(C.kts2 + D.re, D.im);
    const C2 X = Zd * n.id;
    const C2 Y = cfma(c2(2.0 * C.hxr, 2.0 * C.nhrs * n.u), X, Zx);
    out[0] = n.D0;
    out[1] = n.Ch;
    out[2] = Y;
    out[3] = c2(fma(Y.re, C.phi_im, Y.im * n.u), fma(Y.im, C.phi_im, -Y.re * n.u));
    out[4] = half_wphi(n, X) * -2.0;
}

// dZ/d(lambda, mu_j, sigma_j).
__device__ __forceinline__ void jump_partials(const CfConsts& C, const GradParams& G, const NodeParts& n, C2* out) {
    const C2 iphi = c2(-C.phi_im, n.u);
    const C2 phi2 = c2(n.u * n.u - C.phi_im * C.phi_im, 2.0 * n.u * C.phi_im);
    out[0] = (n.jump - c2(1.0, 0.0) - iphi * C.comp) * C.t;
    out[1] = iphi * (n.jump - c2(1.0 + C.comp, 0.0)) * C.lt;
    out[2] = (n.jump * phi2 + iphi * (1.0 + C.comp)) * (-C.lt * G.sigma_j);
}

// The parameter derivatives of an integral from its sums of the five Heston
// quantities (linear, see the top); the jump derivatives are sums already.
__device__ __forceinline__ void heston_chain(const GradParams& G, double* a) {
    const double d0 = a[0], ch = a[1], y = a[2], ys = a[3], xw = a[4];
    a[0] = d0;
    a[1] = fma(G.tis2, ch, y);
    a[2] = G.kis2 * ch;
    a[3] = fma(G.rho, ys, fma(G.sigma, xw, -G.sk * ch));
    a[4] = G.sigma * ys;
}

// One node's terms hw Im(W X) of the derivative sums, X the five Heston
// quantities, then the jump derivatives.  A node whose value or a derivative
// is not finite contributes zero, as in gk_integrate_dual (ad.rs:679-682).
// FAST adds to acc and returns false (nothing added) where its functions do
// not apply; it tests the value only, so that a derivative that is not finite
// shows in acc and the caller takes its nodes again one by one, not FAST
// (which writes the terms to acc, after testing the parameter derivatives that
// they make).
template <bool BATES, bool FAST>
__device__ __forceinline__ bool node_sums(const CfConsts& C, const GradParams& G, double tn, double hw, double* acc) {
    constexpr int DIM = BATES ? 8 : 5;
    bool ok;
    unsigned range = 0;
    const NodeParts n = node_parts<BATES, FAST>(C, tn, ok, range);
    if (FAST && range >= kRangeEnd) return false;
    C2 x[8];
    heston_partials(C, n, x);
    if (BATES) jump_partials(C, G, n, x + 5);
    if (FAST) {
        const C2 W = n.W * hw;
        if (ok) {
#pragma unroll
            for (int k = 0; k < DIM; ++k) acc[k] = fma(W.re, x[k].im, fma(W.im, x[k].re, acc[k]));
        }
    } else {
        double g[8], d[8];
#pragma unroll
        for (int k = 0; k < DIM; ++k) d[k] = g[k] = hw * (n.W * x[k]).im;
        heston_chain(G, d);
#pragma unroll
        for (int k = 0; k < DIM; ++k) ok = ok && isfinite(d[k]);
#pragma unroll
        for (int k = 0; k < DIM; ++k) acc[k] = ok ? g[k] : 0.0;
    }
    return true;
}

// Its terms in g[0..DIM), by CUDA's functions; p: the parameter set (read anew,
// so that the caller's copy of the chain need not lie in memory for this call).
template <bool BATES>
static __device__ __noinline__ void node_sums_slow(const CfConsts& C, const double* p, double tn, double hw,
                                                   double* g) {
    double pl[8];
#pragma unroll
    for (int i = 0; i < (BATES ? 8 : 5); ++i) pl[i] = __ldg(p + i);
    node_sums<BATES, false>(C, make_grad_params(pl, BATES), tn, hw, g);
}

// The exponent's derivatives for the analytic Greeks (x = ln(S/K) and r enter
// Z as i u x and i u r T -- the P1 normaliser's r T cancels the real part of
// i r phi T -- so their derivatives need nothing from here):
//   dZ/dv0 = D0
//   dZ/dT  = 2 kts (m - m h) - v0 phi(phi+i)/2 h (1 - m q) + i r u [+ lambda (jump - 1 - i phi comp)]
// with h = d e/N (e_T = -d e, o_T = d e, N_T = m d e); the normaliser's own
// T-dependence, r T, is already taken out (C, D and J vanish at phi = -i).
template <bool BATES>
__device__ __forceinline__ C2 d_expiry(const CfConsts& C, const NodeParts& n, double r, double lambda) {
    const C2 h = n.d * n.e * n.iN;
    const C2 mh = n.m * h;
    const C2 dD = half_wphi(n, h - mh * n.q);
    C2 ZT = c2(fma(C.kts2, n.m.re - mh.re, C.v0 * dD.re), fma(C.kts2, n.m.im - mh.im, fma(C.v0, dD.im, r * n.u)));
    if (BATES) ZT = cfma(lambda, n.jump - c2(1.0, 0.0) - c2(-C.phi_im, n.u) * C.comp, ZT);
    return ZT;
}

// Terms of the analytic-Greek integrands of one node: d/dx, d2/dx2, d/dr,
// d/dT, d/dv0, d2/dx dv0, d2/dv0^2 of g = Im(W) / (u t^2), weighted by hw; with
// Z linear in x (i u x) and in v0 (v0 D0) the second derivatives are
// Im(W Zp Zq) / (u t^2).  FAST and non-finite terms as in node_sums.
template <bool BATES, bool FAST>
__device__ __forceinline__ bool greek_sums(const CfConsts& C, double r, double lambda, double tn, double hw,
                                           double* acc) {
    bool ok;
    unsigned range = 0;
    const NodeParts n = node_parts<BATES, FAST>(C, tn, ok, range);
    if (FAST && range >= kRangeEnd) return false;
    const C2 ZT = d_expiry<BATES>(C, n, r, lambda);
    const double u = n.u;
    const C2 W = n.W * (FAST ? hw : 1.0);
    const C2 Wv = W * n.D0;
    double g[7];
    g[0] = u * W.re;        // Im(W i u)
    g[1] = -u * u * W.im;   // Im(W (i u)^2)
    g[2] = C.t * g[0];      // Im(W i u T)
    g[3] = (W * ZT).im;
    g[4] = Wv.im;
    g[5] = u * Wv.re;       // Im(W Zv i u)
    g[6] = (Wv * n.D0).im;
    if (FAST) {
        if (ok) {
#pragma unroll
            for (int k = 0; k < 7; ++k) acc[k] += g[k];
        }
    } else {
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            g[k] *= hw;
            ok = ok && isfinite(g[k]);
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) acc[k] = ok ? g[k] : 0.0;
    }
    return true;
}

template <bool BATES>
static __device__ __noinline__ void greek_sums_slow(const CfConsts& C, double r, double lambda, double tn, double hw,
                                                    double* g) {
    greek_sums<BATES, false>(C, r, lambda, tn, hw, g);
}

}  // namespace ope
