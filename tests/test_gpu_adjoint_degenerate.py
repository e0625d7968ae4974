"""Gradients of parameter sets that drop nodes: a node whose value or any
parameter derivative is not finite contributes zero (ad.rs:679-682), whatever
the coefficients its chunk's sums are combined with.  Against the oracle at the
gradient parity bar (1e-7 relative plus 1e-9 S), with a regular surface beside
each, whose gradient stays what it is alone, bit for bit."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu

BASE = [0.04, 2.0, 0.04, 0.3, -0.7, 0.5, -0.1, 0.15]
V0, KAPPA, THETA, SIGMA, RHO, LAMBDA, MU_J, SIGMA_J = range(8)
NOT_FINITE = [float("nan"), float("inf"), float("-inf")]
HESTON = ([(k, v) for k in range(5) for v in NOT_FINITE] + [(SIGMA, v) for v in (0.0, 1e-170, 1e-120, 1e300)]
          + [(k, 1e300) for k in (V0, KAPPA, THETA)])
JUMPS = [(k, v) for k in (LAMBDA, MU_J, SIGMA_J) for v in NOT_FINITE + [0.0]]


def _contracts():
    con = np.zeros(3, W.CONTRACT_DTYPE)
    con["spot"], con["strike"], con["expiry"] = 100.0, [90.0, 100.0, 120.0], [0.5, 1.0, 2.0]
    con["rate"], con["div_yield"], con["opt_type"] = 0.03, 0.01, [1, 0, 0]
    return con


@pytest.mark.parametrize("model,k,value", [("heston", *c) for c in HESTON] + [("bates", *c) for c in HESTON + JUMPS])
def test_dropped_nodes_leave_finite_gradients(ope, oracle, model, k, value):
    bates = model == "bates"
    m, dim = (ope.MODEL_BATES, 8) if bates else (ope.MODEL_HESTON, 5)
    con = _contracts()
    bad = np.array(BASE[:dim])
    bad[k] = value
    par = np.stack([bad, BASE[:dim]])
    both = np.concatenate([con, con])
    price, grad = ope.price_gradient_surfaces(m, both, [0, 3, 6], par, tol=1e-8)
    ref_price, ref = oracle.batch_price_gradient(con, par[:1], bates, 1e-8)
    assert np.all(np.isfinite(ref))
    assert np.all(np.abs(grad[:3] - ref) <= 1e-7 * np.abs(ref) + 1e-9 * 100.0), (grad[:3], ref)
    assert np.max(np.abs(price[:3] - ref_price)) <= 1e-9 * 100.0
    _, alone = ope.price_gradient_surfaces(m, con, [0, 3], par[1:], tol=1e-8)
    assert np.array_equal(grad[3:], alone)


@pytest.mark.parametrize("value", [0.0, 1e-170])
def test_ad_greeks_without_vol_of_vol(ope, oracle, value):
    """Vega and volga come from the gradient's v0 column: 0 where every node is dropped."""
    p = np.array(BASE[:5])
    p[SIGMA] = value
    res = ope.batch_greeks_ad(ope.MODEL_HESTON, _contracts(), p, tol=1e-8)
    assert np.all(res["vega"] == 0.0) and np.all(res["volga"] == 0.0)
