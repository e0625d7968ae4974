"""Exponents whose e^{Re Z} is finite and whose node value e^{Re Z}/((1-t) t)
is not: the reference's node is 0 there (heston.rs:224-226).  A jump intensity
of -650/T to -700/T without diffusion puts Re Z at 650 to 700 on every node with
a large u."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("top", [590.0, 650.0, 690.0, 699.0, 699.9])
def test_values_beyond_the_largest_double_are_dropped(ope, oracle, top, which):
    """Panels that both sides bisect agree to 1e-11 of the panel's largest node
    (the bar of the corner traces) plus eight roundings of the phase r T u at the
    panel's largest u, where e^{Re Z} times the panel's largest 1/((1-t) t) is
    below 1e308 (beyond, the kernels drop a node by that product, the reference
    by its product with the sine)."""
    con = W.c1().contracts[37:38]
    T = float(con["expiry"][0])
    par = np.array((0.0, 1.5, 0.0, 0.5, -0.7, -top / T, -0.5 * 0.15 ** 2, 0.15))  # mean jump 0
    got, _ = ope.trace_integral(ope.MODEL_BATES, con, par, which, tol=1e-10)
    ref, _ = oracle.trace_integral(con, par, True, which, 1e-10)
    assert np.all(np.isfinite(ref[:, 9:])) and np.all(np.isfinite(got[:, 9:]))  # the nodes; their sums may overflow
    panels = {(r[0], r[1]): r[9:39] for r in ref[1:]}
    compared = 0
    for g in got[1:]:
        a, b = g[:2]
        r = panels.get((a, b))
        lowest = a + 0.002 * (b - a)  # below the left child's first node
        bar = 1e-11 + 8.0 * 2.0 ** -53 * 0.01 / lowest
        if r is None or bar > 0.1 or top - np.log(lowest) > 308.0 * np.log(10.0):
            continue
        for x, y in ((g[9:24], r[:15]), (g[24:39], r[15:])):
            assert np.max(np.abs(x - y)) <= bar * np.max(np.abs(y))
            compared += 1
    assert compared >= 4
