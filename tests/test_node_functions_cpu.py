"""CPU checks of the node evaluation's own exponential, sine and cosine
(csrc/cf_device.cuh: exp_node, cis_node, sin_node): tables and coefficients are
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
    body = SRC[SRC.index(f"void {name}(" if name == "cis_node" else f"double {name}("):]
    return body[:body.index("\n}\n")]


EXP2, CIS = _table("g_exp2_tab"), _table("g_cis_tab").reshape(64, 2)


def test_tables_are_correctly_rounded():
    with mp.workprec(120):
        assert [float(mp.mpf(2) ** (mp.mpf(j) / 64)) for j in range(64)] == EXP2.tolist()
        for j in range(64):
            for got, want in zip(CIS[j], (mp.cos(mp.pi * j / 32), mp.sin(mp.pi * j / 32))):
                assert got == (0.0 if abs(want) < mp.mpf(2) ** -60 else float(want))


def test_coefficients_match_their_generator():
    def descending(c):
        return [float(v) for v in reversed(c)]

    assert descending(coeffs.exp_coefficients()[0]) == [v for v in _floats(_body("exp_node")) if 0.008 < v < 0.5]
    s, c, _ = coeffs.cis_coefficients()
    cis = _floats(_body("cis_node"))
    assert set(descending(s) + descending(c)) <= set(cis)
    assert descending(coeffs.sin_coefficients()[0]) == _floats(_body("sin_node"))[-8:]


def _exp(x):
    k = np.rint(x * 92.33248261689366)
    r = (x - k * 0.010830424696249145) - k * 3.623510646634843e-19
    q = np.zeros_like(r)
    for c in reversed(coeffs.exp_coefficients()[0]):
        q = q * r + float(c)
    k = k.astype(np.int64)
    return np.ldexp(EXP2[k & 63] * (1.0 + (q * (r * r) + r)), (k >> 6).astype(np.int32))


def _cis(x):
    k = np.rint(x * 10.185916357881302)
    r = (x - k * 0.09817477042468103) - k * 3.827021247335479e-18
    s, c, _ = coeffs.cis_coefficients()
    w = r * r
    sr = r + r * (w * (float(s[0]) + w * (float(s[1]) + w * float(s[2]))))
    cm = w * (float(c[0]) + w * (float(c[1]) + w * float(c[2])))
    t = CIS[k.astype(np.int64) & 63]
    return (t[:, 0] + t[:, 0] * cm) - t[:, 1] * sr, (t[:, 1] + t[:, 1] * cm) + t[:, 0] * sr


def _sin(x, a):
    k = np.rint((x + a) * 0.3183098861837907)
    r = ((x - k * 3.141592653589793) - k * 1.2246467991473532e-16) + a
    s, q = r * r, 0.0
    for c in reversed(coeffs.sin_coefficients()[0]):
        q = q * s + float(c)
    return np.where(k.astype(np.int64) & 1, -1.0, 1.0) * (r + r * (s * q))


def _worst(got, want, scale):
    with mp.workprec(120):
        return max(abs(mp.mpf(float(g)) - w) / s for g, w, s in zip(got, want, scale)) / EPS


def test_restated_functions_stay_within_their_rounding_bounds():
    """Without FMA the reduction's product rounds at the size of x (|x| <= 8
    for e^x: at most 8 EPS of r, so 8 EPS of the result; the table, the sum and
    the product add 3); for the phases |x| <= 4: 4 EPS, plus 4 roundings of
    numbers below 1 (cis) or 2 roundings and a of size 1 (sin)."""
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
