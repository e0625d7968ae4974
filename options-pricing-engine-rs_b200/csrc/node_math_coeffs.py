"""Coefficients of cf_device.cuh's own functions, computed in 60-digit arithmetic
(mpmath): first those of atan2_node and log_node, which its self-tests alone use.

atan2_node reduces atan2(y, x) to atan(t) with |t| <= tan(pi/8): first to
q = min(|x|,|y|) / max(|x|,|y|) in [0, 1] (octant symmetry), then, for
q > tan(pi/8), to t = (q - 1)/(q + 1) with atan(q) = pi/4 + atan(t).  There
atan(t) = t + t s P(s), s = t^2, where P is the degree-10 polynomial that
interpolates f(s) = (atan(sqrt s)/sqrt s - 1)/s at the 11 Chebyshev nodes of
[0, (sqrt 2 - 1)^2]: 5e-18 relative error on atan(t).

log_node writes v = 2^k m with m in [sqrt(1/2), sqrt(2)), so that
log v = k ln 2 + 2 atanh(s), s = (m - 1)/(m + 1), |s| <= 3 - 2 sqrt 2, and
2 atanh(s) = 2 s + s w R(w), w = s^2, where R is the degree-6 polynomial that
interpolates (2 atanh(s) - 2 s)/(s w) at the 7 Chebyshev nodes of
[0, (3 - 2 sqrt 2)^2]: 4.5e-18 relative error on log m.

The node evaluation is made of the functions below (log_ratio, exp_node,
cis_node, sin_node, arg_node).  Their leading coefficients have a zero low word
(at most 21 significant bits): an FP64 instruction takes such a constant as an
immediate, where a full double costs a load and a third 64-bit register operand
(measured on B200: 2.1 cycles per FMA instead of 3.1).  `fit` rounds the top
coefficients one after another and lets the lower ones interpolate what is left,
so the rounding costs nothing as long as the result stays near 1e-17:

  log_ratio: 2 atanh(s) = 2 s + s w R(w), |s| <= 0.2016, degree 7, 4 short;
  exp_node:  e^r = 1 + r + r^2 P(r), |r| <= 1.03 ln2/128, degree 3, P(0) = 1/2, 2 short;
  cis_node:  sin r = r + r^3 S(r^2), degree 2, 1 short, and cos r = 1 + r^2 C(r^2),
             degree 3, C(0) = -1/2, 2 short, |r| <= 1.01 pi/64;
  sin_node:  the same S form, |r| <= pi/2, degree 7, 3 short;
  arg_node:  atan t = t + t^3 P(t^2), |t| <= 0.1125, degree 5, 3 short.

All are far below the 1.1e-16 rounding unit; the evaluation in double
precision then adds a few ulps (checked on the device through
ope_selftest_atan2, ope_selftest_log and ope_selftest_node_function, and in
numpy by tests/test_node_math_cpu.py and tests/test_node_functions_cpu.py).

Run: python node_math_coeffs.py  (prints the coefficients, highest degree
first, as they appear in cf_device.cuh, and the approximation errors).
"""
import struct

import mpmath as mp

mp.mp.dps = 60
ATAN_DEG = 10
LOG_DEG = 6


def _chebyshev_interpolant(fn, hi, deg):
    n = deg + 1
    xs = [hi / 2 * (1 - mp.cos(mp.pi * (k + mp.mpf(1) / 2) / n)) for k in range(n)]
    a = mp.matrix([[x ** j for j in range(n)] for x in xs])
    b = mp.matrix([fn(x) for x in xs])
    c = mp.lu_solve(a, b)
    return [c[j] for j in range(n)]


def _atan_f(s):
    if s == 0:
        return mp.mpf(-1) / 3
    r = mp.sqrt(s)
    return (mp.atan(r) / r - 1) / s


def _log_r(w):
    if w == 0:
        return mp.mpf(2) / 3
    s = mp.sqrt(w)
    return (2 * mp.atanh(s) - 2 * s) / (s * w)


def atan_coefficients(deg=ATAN_DEG):
    """P(s), lowest degree first, and the interval end (sqrt 2 - 1)^2."""
    smax = (mp.sqrt(2) - 1) ** 2
    return _chebyshev_interpolant(_atan_f, smax, deg), smax


def log_coefficients(deg=LOG_DEG):
    """R(w), lowest degree first, and the interval end (3 - 2 sqrt 2)^2."""
    wmax = (3 - 2 * mp.sqrt(2)) ** 2
    return _chebyshev_interpolant(_log_r, wmax, deg), wmax


def short(v):
    """The nearest double with a zero low word."""
    b = struct.unpack("<Q", struct.pack("<d", float(v)))[0]
    return mp.mpf(struct.unpack("<d", struct.pack("<Q", (b + 0x80000000) & 0xFFFFFFFF00000000))[0])


def _solve(fn, xs, weights, degrees):
    a = mp.matrix([[w * x ** d for d in degrees] for x, w in zip(xs, weights)])
    return list(mp.lu_solve(a, mp.matrix([w * fn(x) for x, w in zip(xs, weights)])))


def fit(fn, lo, hi, deg, n_short, c0=None, weight=None):
    """Coefficients, lowest degree first: the top n_short with zero low words,
    c0 given or free, the others doubles interpolating fn at Chebyshev nodes of
    [lo, hi] (with `weight`: weighted least squares at 41 nodes)."""
    fixed = {} if c0 is None else {0: mp.mpf(c0)}
    free = [d for d in range(deg + 1) if d not in fixed]
    while True:
        n = len(free) if weight is None else 41
        xs = [(lo + hi) / 2 - (hi - lo) / 2 * mp.cos(mp.pi * (k + mp.mpf(1) / 2) / n) for k in range(n)]
        c = _solve(lambda x: fn(x) - sum(v * x ** d for d, v in fixed.items()), xs,
                   [weight(x) if weight else 1 for x in xs], free)
        if n_short == 0:
            fixed.update((d, mp.mpf(float(v))) for d, v in zip(free, c))
            return [fixed[d] for d in range(deg + 1)]
        fixed[free.pop()] = short(c[-1])
        n_short -= 1


def _near0(fn, at0):
    return lambda x: fn(x) if abs(x) > mp.mpf(10) ** -25 else at0


_EXP_P = _near0(lambda r: (mp.e ** r - 1 - r) / r ** 2, mp.mpf(1) / 2)
_SIN_S = _near0(lambda w: (mp.sin(mp.sqrt(w)) / mp.sqrt(w) - 1) / w, -mp.mpf(1) / 6)
_COS_C = _near0(lambda w: (mp.cos(mp.sqrt(w)) - 1) / w, -mp.mpf(1) / 2)


def exp_coefficients():
    h = mp.log(2) / 128 * mp.mpf("1.03")
    return fit(_EXP_P, -h, h, 3, 2, mp.mpf("0.5"), lambda r: r * r + mp.mpf(10) ** -9)


def cis_coefficients():
    hi = (mp.pi / 64 * mp.mpf("1.01")) ** 2
    return fit(_SIN_S, 0, hi, 2, 1), fit(_COS_C, 0, hi, 3, 2, mp.mpf("-0.5"))


def sin_coefficients():
    return fit(_SIN_S, 0, (mp.pi / 2) ** 2, 7, 3)


def log_ratio_coefficients():
    return fit(_log_r, 0, mp.mpf("0.2016") ** 2, 7, 4)


def arg_coefficients():
    return fit(_atan_f, 0, mp.mpf("0.1125") ** 2, 5, 3)


def exp_table():
    return [float(mp.mpf(2) ** (mp.mpf(j) / 64)) for j in range(64)]


def cis_table():
    zero = mp.mpf(10) ** -40
    return [tuple(0.0 if abs(v) < zero else float(v) for v in (mp.cos(mp.pi * j / 32), mp.sin(mp.pi * j / 32)))
            for j in range(64)]


def arg_table():
    """(cos K, sin K, K) of arg_node's directions: per quadrant (x, y > 0; x < 0;
    y < 0; both), K = 0, atan 2^c for c = -4.5, -4, ... 4.5, and pi/2, reflected."""
    zero = mp.mpf(10) ** -40
    ks = [mp.mpf(0)] + [mp.atan(mp.mpf(2) ** (mp.mpf(c) / 2)) for c in range(-9, 10)] + [mp.pi / 2]
    rows = []
    for sy in (1, -1):
        for negative_x in (False, True):
            for k in ks:
                k = mp.pi - k if negative_x else k
                c, s = (0.0 if abs(v) < zero else float(v) for v in (mp.cos(k), mp.sin(k)))
                # the angle of the rounded direction (of -1, 0: pi)
                a = mp.atan2(mp.mpf(s), mp.mpf(c))
                rows.append((c, sy * s, float(sy * a)))
    return rows


def _poly(c, x):
    return sum(c[j] * x ** j for j in range(len(c)))


def atan_error(c, smax, samples=2000):
    return max(abs((mp.sqrt(s) + mp.sqrt(s) * s * _poly(c, s)) / mp.atan(mp.sqrt(s)) - 1)
               for s in (smax * i / samples for i in range(1, samples + 1)))


def log_error(c, wmax, samples=2000):
    return max(abs((2 * mp.sqrt(w) + mp.sqrt(w) * w * _poly(c, w)) / (2 * mp.atanh(mp.sqrt(w))) - 1)
               for w in (wmax * i / samples for i in range(1, samples + 1)))


if __name__ == "__main__":
    for name, (c, hi), err in (("atan2_node P(s)", atan_coefficients(), atan_error),
                               ("log_node R(w)", log_coefficients(), log_error)):
        print(name)
        for j in reversed(range(len(c))):
            print(f"    {float(c[j])!r},  // ^{j}")
        print("  max relative error:", mp.nstr(err(c, hi), 3))
    for name, c in (("log_ratio R(w)", log_ratio_coefficients()), ("exp_node P(r)", exp_coefficients()),
                    ("cis_node S(w)", cis_coefficients()[0]), ("cis_node C(w)", cis_coefficients()[1]),
                    ("sin_node S(w)", sin_coefficients()), ("arg_node P(s)", arg_coefficients())):
        print(name)
        for j in reversed(range(len(c))):
            print(f"    {float(c[j])!r},  // ^{j}")
