"""The functions that the node evaluation of the pricing and gradient kernels is
made of (csrc/cf_device.cuh: exp_node, cis_node in both forms, sin_node,
log_ratio, arg_node), on the device, against mpmath at 200 bits: over their
whole ranges, at the edges of their clamps and in every bin of their tables.

Bars in units u = 2^-53, from each function's roundings:
* e^x, relative: the table 1, the final FMA 1, the polynomial's roundings at
  2^-7 of the result: 3 u;
* cos x, sin x: table and two FMAs 0.5 each, half of that from the small terms:
  3 u; the reduction's 53-bit second part is 2e-7 of pi/32, so its rounding
  adds 2e-7 u |x|: bar 4e-7 u |x|;
* cos, sin of x + a: x - k c and its remainder round at the size of a: 2 u |a|,
  bar 3 u (1 + |a|); sin_node the same, with |r| up to pi/2: 3 u (2 + |a|);
* log(a/b): six roundings of 2 s <= 0.41, the sum's own: 4 u max(1, |v|); 1/a
  beside it: reciprocal 2, product, scaling, product: 5 u relative;
* arg: the table's angle, the quotient's numerator, the sum: 4 u max(1, |v|)."""
import mpmath as mp
import numpy as np
import pytest

from ope_b200 import _lib

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
EXP, COS, SIN, COS_SUM, SIN_SUM, SIN_VALUE, LOG_RATIO, LOG_RCP, ARG = range(9)


def _eval(which, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = np.zeros_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
    out = np.empty_like(a)
    _lib.check(_lib.load().ope_selftest_node_function(which, a.ctypes.data, b.ctypes.data, a.size, out.ctypes.data))
    return out


def _m(v):
    return [mp.mpf(float(x)) for x in v]


def _check(got, want, bar):
    """|got - want| <= bar U, element by element."""
    with mp.workprec(200):
        ratio = np.array([float(abs(mp.mpf(float(g)) - w) / mp.mpf(float(b * U))) for g, w, b in zip(got, want, bar)])
    worst = int(np.argmax(ratio))
    print(f"worst {ratio[worst]:.3f} of the bar at {worst}")
    assert ratio[worst] <= 1.0, (worst, got[worst], want[worst])


def _phases(rng, n):
    """Signed phases: log-uniform up to 2^44, small ones, and neighbours of the
    table's points and of the points half way between them."""
    wide = rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(-30.0, 43.999, n))
    near = rng.integers(-200, 200, n) * (np.pi / 64.0) * (1.0 + rng.choice([-1e-15, 0.0, 1e-15], n))
    return np.concatenate([wide, rng.uniform(-8.0, 8.0, n), near, [0.0, -0.0]])


def test_exponential():
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-708.0, 709.77, 4000), rng.uniform(-1.0, 1.0, 2000),
                        np.arange(-800, 800) * (np.log(2.0) / 128.0), [0.0, -0.0, -708.0, 709.77, 1e-300]])
    with mp.workprec(200):
        want = [mp.exp(v) for v in _m(x)]
    _check(_eval(EXP, x), want, [3.0 * float(w) for w in want])


def test_exponential_beyond_its_clamps():
    """From 709.777 (the last table index of 2^1023) to ln of the largest double the
    value is right or not finite: 1/((1 - t) t) >= 4 makes a node's value infinite
    there, and an infinite jump factor is left to the careful evaluation."""
    low = np.concatenate([[-708.5, -709.0, -745.2, -1e4, -1e9, -1e100, -1.7e308, -np.inf],
                          -np.arange(1, 6) * 2.0 ** 32 * np.log(2.0) / 64.0 + 3.0])
    got = _eval(EXP, low)
    assert np.all((got >= 0.0) & (got <= 3.4e-308))
    last = np.linspace(709.771, 709.782, 40)
    got = _eval(EXP, last)
    assert np.all(~np.isfinite(got) | (np.abs(got / np.exp(last) - 1.0) <= 4.0 * U))
    assert not np.any(np.isfinite(_eval(EXP, [709.8, 710.0, 1e3, 1e9, 1e100, 1.7e308, np.inf])))


def test_cosine_and_sine():
    x = _phases(np.random.default_rng(2), 3000)
    with mp.workprec(200):
        co, si = [mp.cos(v) for v in _m(x)], [mp.sin(v) for v in _m(x)]
    bar = 3.0 + 4e-7 * np.abs(x)
    _check(_eval(COS, x), co, bar)
    _check(_eval(SIN, x), si, bar)


@pytest.mark.parametrize("which", [COS_SUM, SIN_SUM, SIN_VALUE])
def test_cosine_and_sine_of_a_sum(which):
    rng = np.random.default_rng(3)
    x = _phases(rng, 3000)
    a = rng.choice([-1.0, 1.0], x.size) * np.exp2(rng.uniform(-20.0, 12.0, x.size))
    a[:50] = -x[:50] + rng.uniform(-1.0, 1.0, 50)  # large phases that cancel
    a[50:60] = 0.0
    with mp.workprec(200):
        want = [(mp.cos if which == COS_SUM else mp.sin)(v + w) for v, w in zip(_m(x), _m(a))]
    _check(_eval(which, x, a), want, 3.0 * ((2.0 if which == SIN_VALUE else 1.0) + np.abs(a)))


def test_logarithm_of_a_quotient_and_reciprocal():
    rng = np.random.default_rng(4)
    n = 3000
    a, b = np.exp(rng.uniform(-300.0, 300.0, n)), np.exp(rng.uniform(-300.0, 300.0, n))
    b[:1000] = a[:1000] * rng.uniform(0.5, 2.0, 1000)
    # both sides of the exponent's turning points, a/b = 2^(+-1/2) and around, and a = b
    b[1000:1600] = a[1000:1600] * 2.0 ** (rng.integers(-3, 4, 600) + rng.choice([0.5, 0.58, 0.59, 0.42], 600))
    b[1600:1650] = a[1600:1650]
    with mp.workprec(200):
        want, rcp = [mp.log(v / w) for v, w in zip(_m(a), _m(b))], [1 / v for v in _m(a)]
    _check(_eval(LOG_RATIO, a, b), want, [4.0 * max(1.0, abs(float(v))) for v in want])
    _check(_eval(LOG_RCP, a, b), rcp, [5.0 * float(v) for v in rcp])


def test_argument_in_every_bin_and_quadrant():
    rng = np.random.default_rng(5)
    octaves = np.repeat(np.arange(-6.0, 6.001, 1.0 / 16.0), 16)  # log2 |y/x|, all bins and beyond both ends
    octaves = np.concatenate([octaves, rng.uniform(-90.0, 90.0, 512)])
    x = np.exp2(rng.uniform(-60.0, 60.0, octaves.size))
    y = x * np.exp2(octaves + rng.uniform(-1e-3, 1e-3, octaves.size))
    x, y = (np.concatenate([s * v for s in signs])
            for signs, v in (((1, 1, -1, -1), x), ((1, -1, 1, -1), y)))
    # on the axes
    x = np.concatenate([x, [1.0, 1.0, -1.0, -1.0, 0.0, 0.0, 3e150, -3e150]])
    y = np.concatenate([y, [0.0, -0.0, 0.0, -0.0, 2.0, -2.0, 3e150, 3e150]])
    with mp.workprec(200):
        want = [mp.atan2(v, w) for v, w in zip(_m(y), _m(x))]
    for i in np.flatnonzero((y == 0.0) & np.signbit(y)):
        want[i] = -want[i] if want[i] > 0 else want[i]  # mpmath has no -0
    _check(_eval(ARG, y, x), want, [4.0 * max(1.0, abs(float(v))) for v in want])


def test_refuses_unknown_functions_and_missing_arrays():
    L = _lib.load()
    a = np.zeros(1)
    assert L.ope_selftest_node_function(9, a.ctypes.data, a.ctypes.data, 1, a.ctypes.data) != 0
    assert L.ope_selftest_node_function(-1, a.ctypes.data, a.ctypes.data, 1, a.ctypes.data) != 0
    assert L.ope_selftest_node_function(0, None, a.ctypes.data, 1, a.ctypes.data) != 0
