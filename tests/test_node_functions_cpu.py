"""CPU checks of the node evaluation's own exponential, sine and cosine
(csrc/cf_device.cuh: exp_node, cis_node, sin_node), logarithm and argument
(log_ratio, arg_node): tables and coefficients are
what csrc/node_math_coeffs.py derives, and the algorithms, restated in numpy
without FMA (each product rounded once more than on the device), stay within
the bound their operation counts give."""
import os
import re
import sys

import mpmath as mp
import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "options-pricing-engine-rs_b200", "csrc")
SRC = open(os.path.join(CSRC, "cf_device.cuh")).read()
sys.path.insert(0, CSRC)
import node_math_coeffs as coeffs  # noqa: E402

EPS = 2.0 ** -53


def _floats(text):
    return [float(v) for v in re.findall(r"-?\d+\.\d+(?:e-?\d+)?", text)]


def _table(name):
    body = SRC[SRC.index(name + "["):]
    return np.array(_floats(body[body.index("= {"):body.index("};")]))


def _body(name):
    body = SRC[SRC.index(f"void {name}(" if name == "cis_tail" else f"double {name}("):]
    return body[:body.index("\n}\n")]


EXP2, CIS = _table("g_exp2_tab"), _table("g_cis_tab").reshape(64, 2)
ARG = _table("g_arg_tab").reshape(84, 4)[:, :3]


def test_tables_are_what_their_generator_derives():
    assert EXP2.tolist() == coeffs.exp_table()
    assert [tuple(r) for r in CIS] == coeffs.cis_table()
    assert [tuple(r) for r in ARG] == coeffs.arg_table()


def test_coefficients_match_their_generator():
    s, c = coeffs.cis_coefficients()
    for name, want in (("exp_node", coeffs.exp_coefficients()), ("cis_tail", s), ("cis_tail", c),
                       ("sin_node", coeffs.sin_coefficients()), ("log_ratio", coeffs.log_ratio_coefficients()),
                       ("arg_node", coeffs.arg_coefficients())):
        have = _floats(_body(name))
        assert set(float(v) for v in want) <= set(have), name


def _exp(x):
    k = np.rint(x * 92.33245849609375)
    r = (x - k * 0.010830424726009369) + k * 2.9760223436840126e-11
    q = np.zeros_like(r)
    for c in reversed(coeffs.exp_coefficients()):
        q = q * r + float(c)
    k = k.astype(np.int64)
    return np.ldexp(EXP2[k & 63] * (1.0 + (q * (r * r) + r)), (k >> 6).astype(np.int32))


def _cis(x):
    k = np.rint(x * 10.185916357881302)
    r = (x - k * 0.09817475080490112) - k * 1.9619779915655082e-08
    s, c = coeffs.cis_coefficients()
    w = r * r
    sr = r + r * (w * (float(s[0]) + w * (float(s[1]) + w * float(s[2]))))
    cm = w * (float(c[0]) + w * (float(c[1]) + w * (float(c[2]) + w * float(c[3]))))
    t = CIS[k.astype(np.int64) & 63]
    return (t[:, 0] + t[:, 0] * cm) - t[:, 1] * sr, (t[:, 1] + t[:, 1] * cm) + t[:, 0] * sr


def _sin(x, a):
    k = np.rint((x + a) * 0.3183098861837907)
    r = ((x - k * 3.141592653589793) - k * 1.2246467991473532e-16) + a
    s, q = r * r, 0.0
    for c in reversed(coeffs.sin_coefficients()):
        q = q * s + float(c)
    return np.where(k.astype(np.int64) & 1, -1.0, 1.0) * (r + r * (s * q))


def _hi(v):
    return (np.asarray(v).view(np.int64) >> 32).astype(np.int64)


def _log_ratio(a, b):
    k = (_hi(a) - _hi(b) + 0x80000) >> 20
    m = np.ldexp(a, -k.astype(np.int32))
    s = (m - b) / (m + b)
    w, r = s * s, 0.0
    for c in reversed(coeffs.log_ratio_coefficients()):
        r = r * w + float(c)
    return k * 0.6931471805599453 + (2.0 * s + (s * w) * r)


def _arg(y, x):
    d = (_hi(y) & 0x7FFFFFFF) - (_hi(x) & 0x7FFFFFFF)
    top, half_octave = 19 << 18, 1 << 19
    at = (np.minimum(np.maximum(d, -top - half_octave), top) + top + half_octave) >> 19
    c, s, k = ARG[at + 21 * np.signbit(x) + 42 * np.signbit(y)].T
    t = (y * c - x * s) / (x * c + y * s)
    assert np.max(np.abs(t)) <= 0.1125
    w, p = t * t, 0.0
    for q in reversed(coeffs.arg_coefficients()):
        p = p * w + float(q)
    return k + (t + (t * w) * p)


def _worst(got, want, scale):
    with mp.workprec(120):
        return max(abs(mp.mpf(float(g)) - w) / s for g, w, s in zip(got, want, scale)) / EPS


def test_restated_functions_stay_within_their_rounding_bounds():
    """Without FMA the reduction's product rounds at the size of x (|x| <= 8
    for e^x: at most 8 EPS of r, so 8 EPS of the result; the table, the sum and
    the product add 3); for the phases |x| <= 4: 4 EPS, plus 4 roundings of
    numbers below 1 (cis) or 2 roundings and a of size 1 (sin).  The argument:
    2 EPS for a K up to pi and its sum, 3 for t's two products and quotient;
    log(a/b): the quotient, s w R and the sum below 1, and the roundings of
    k ln 2 at its own size."""
    rng = np.random.default_rng(3)
    n = 4000
    x = rng.uniform(-8.0, 8.0, n)
    y, a = rng.uniform(-4.0, 4.0, n), rng.uniform(-1.0, 1.0, n)
    with mp.workprec(120):
        ex = [mp.exp(mp.mpf(float(v))) for v in x]
        co, si = [mp.cos(mp.mpf(float(v))) for v in y], [mp.sin(mp.mpf(float(v))) for v in y]
        sa = [mp.sin(mp.mpf(float(v)) + mp.mpf(float(b))) for v, b in zip(y, a)]
    one = [mp.mpf(1)] * n
    re, im = _cis(y)
    assert _worst(_exp(x), ex, ex) <= 11
    assert _worst(re, co, one) <= 8 and _worst(im, si, one) <= 8
    assert _worst(_sin(y, a), sa, one) <= 8
    rad, th = np.ldexp(1.0, rng.integers(-40, 40, n)), rng.uniform(-np.pi, np.pi, n)
    th[: n // 2] = np.sign(th[: n // 2]) * np.arctan(2.0 ** rng.uniform(-8, 8, n // 2))
    yy, xx = rad * np.sin(th), rad * np.cos(th)
    with mp.workprec(120):
        ar = [mp.atan2(mp.mpf(float(v)), mp.mpf(float(b))) for v, b in zip(yy, xx)]
        pa, pb = np.exp(rng.uniform(-30, 30, n)), np.exp(rng.uniform(-30, 30, n))
        pb[: n // 4] = pa[: n // 4] * rng.uniform(0.9, 1.1, n // 4)
        lr = [mp.log(mp.mpf(float(v)) / mp.mpf(float(b))) for v, b in zip(pa, pb)]
    assert _worst(_arg(yy, xx), ar, [max(mp.mpf(1), abs(v)) for v in ar]) <= 5
    assert _worst(_log_ratio(pa, pb), lr, [max(mp.mpf(1), abs(v)) for v in lr]) <= 4
