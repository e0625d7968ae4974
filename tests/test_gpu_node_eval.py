"""The node evaluation where its branches turn: correlations beyond +-1 (the
square root's argument crosses into the left half plane), a vol-of-vol near 0,
kappa below rho sigma (the P1 normaliser degenerates), jumps switched off and
one-sided, against the CPU oracle."""
import numpy as np
import pytest

from ope_b200 import workloads as W

PARAMS = [(0.04, 1.5, 0.04, 0.5, 1.0), (0.04, 1.5, 0.04, 0.5, -1.0), (0.09, 0.5, 0.06, 1e-3, -0.4),
          (0.04, 0.1, 0.04, 0.9, 0.5), (0.04, 4.0, 0.09, 0.3, 0.0)]
JUMPS = [None, (0.0, 0.0, 0.1), (1.2, -0.3, 0.05), (0.4, 0.1, 0.6)]


@pytest.mark.gpu
@pytest.mark.parametrize("jump", JUMPS)
@pytest.mark.parametrize("heston", PARAMS)
def test_prices_at_the_branches_of_the_node_evaluation(ope, oracle, heston, jump):
    """At the parity bar, 1e-9 S."""
    con = W.c1().contracts.copy()
    con["expiry"] *= np.where(np.arange(con.size) % 3 == 0, 0.02, 1.0)
    par = np.array(heston + (jump or ()))
    got = (ope.batch_heston if jump is None else ope.batch_bates)(con, par, tol=1e-10)
    ref = oracle.batch_price(con, par[None, :], jump is not None, 1e-10)
    assert np.max(np.abs(got - ref)) <= 1e-9 * 100.0


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("rho", [1.2, -1.3])
def test_nodes_beyond_correlation_one(ope, oracle, rho, which):
    """The integrals diverge there, so the 30 nodes of the first bisection are
    compared: 1e-11 of the largest, the bar of the corner traces."""
    con, par = W.c1().contracts[37:38], np.array((0.04, 1.5, 0.04, 0.5, rho))
    got, _ = ope.trace_integral(ope.MODEL_HESTON, con, par, which, tol=1e-10)
    ref, _ = oracle.trace_integral(con, par, False, which, 1e-10)
    a, b = got[0, 9:39], ref[0, 9:39]
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))


@pytest.mark.gpu
def test_nodes_beyond_the_fast_functions_range(ope, oracle):
    """A jump mean of -2^47: the jump factor's phase passes 2^45 on the nodes
    with u > 1/4, below which the fast functions apply (P2; both evaluate
    cos and sin of the same rounded phase).  Same bar as above."""
    con = W.c1().contracts[37:38]
    par = np.array((0.04, 1.5, 0.04, 0.5, -0.7, 0.8, -2.0 ** 47, 0.1))
    got, _ = ope.trace_integral(ope.MODEL_BATES, con, par, 1, tol=1e-10)
    ref, _ = oracle.trace_integral(con, par, True, 1, 1e-10)
    a, b = got[0, 9:39], ref[0, 9:39]
    assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
    # a phase of 2^47 u in the final sine: its last place alone moves it by
    # more than 1e-2, so only its magnitude is bounded, by the node weights
    big = con.copy()
    big["rate"] = 2.0 ** 47 / big["expiry"]
    ref0, _ = oracle.trace_integral(con, par[:5], False, 1, 1e-10)
    got, _ = ope.trace_integral(ope.MODEL_HESTON, big, par[:5], 1, tol=1e-10)
    assert np.all(np.isfinite(got[0])) and np.max(np.abs(got[0, 9:39])) <= 1e3 * np.max(np.abs(ref0[0, 9:39]))


@pytest.mark.gpu
@pytest.mark.parametrize("multiple", [1, 2, 3])
def test_nodes_far_below_the_jump_factors_underflow(ope, oracle, multiple):
    """A jump width that puts one node's jump exponent where 64/ln2 times it is a
    multiple of 2^32 away from a number the exponential does not flush: the
    factor is 0 there all the same (P2).  mu_j takes the mean jump to -1 exactly.
    Where the factor is not 0, u mu_j is up to 1.2e5: 1.3e-11 per rounding."""
    con = W.c1().contracts[37:38]
    ref0, _ = oracle.trace_integral(con, np.array((0.04, 1.5, 0.04, 0.5, -0.7)), False, 1, 1e-10)
    x = 0.5 + 0.5 * np.array([-0.9491079123427585, -0.7415311855993945, 0.0, 0.5860872354676911])
    for t in x:  # nodes of the first panel, [0, 1]
        u = (1.0 - t) / t
        half = (multiple * 2.0 ** 32 - 300.0) / 92.33248261689366 / u ** 2  # sigma_j^2 / 2
        par = np.array((0.04, 1.5, 0.04, 0.5, -0.7, 0.8, -1.5 * half, np.sqrt(2.0 * half)))
        got, _ = ope.trace_integral(ope.MODEL_BATES, con, par, 1, tol=1e-10)
        ref, _ = oracle.trace_integral(con, par, True, 1, 1e-10)
        a, b = got[0, 9:39], ref[0, 9:39]
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(ref0[0, 9:39]))
