"""Launches chosen by the size of the call.  Small calls take one block per
contract; automatic launches of several surfaces take their contracts deepest-first and
may keep fewer warps resident per SM (from 16 contracts per SM): the prices are
those of input order, bit for bit, on both sides of the size limits, and for
the launches that store panel lists (gradients)."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _in_input_order(ope, model, w, warps=4, bisections=None):
    """The same call through a table whose every class is input order, `warps` per block."""
    saved, _ = ope.tune_table(model)
    try:
        ope.set_tune_table(model, [dict(r, warps_per_block=warps, deepest_first=False, occupancy=1.0, per_unit=1)
                                   for r in saved])
        return ope.price_surfaces(model, w.contracts, w.surf_offsets, w.params, tol=w.tol, bisections=bisections)
    finally:
        ope.set_tune_table(model, saved)


@pytest.mark.parametrize("n", [1, 2, 3, 149, (48, 0), (48, 1)])
@pytest.mark.parametrize("model", ["heston", "bates"])
def test_one_block_per_contract_prices_as_the_persistent_grid(ope, model, n):
    m = ope.MODEL_BATES if model == "bates" else ope.MODEL_HESTON
    n = n if isinstance(n, int) else n[0] * ope.device_info()[0] + n[1]
    w = W.c3(n=n, per_surface=n, seed=n)
    if model == "heston":
        w.params = np.ascontiguousarray(w.params[:, :5])
    w.contracts["expiry"][0] = 1.0 / 3650.0
    nb, nb_grid = np.zeros(2 * n, np.int32), np.zeros(2 * n, np.int32)
    ope.set_autotune(False)
    try:
        got = ope.price_surfaces(m, w.contracts, w.surf_offsets, w.params, tol=w.tol, bisections=nb)
        plain = (ope.batch_bates if m == ope.MODEL_BATES else ope.batch_heston)(w.contracts, w.params[0], tol=w.tol)
        graded, _ = ope.price_gradient_surfaces(m, w.contracts, w.surf_offsets, w.params, tol=w.tol)
    finally:
        ope.set_autotune(True)
    grid = _in_input_order(ope, m, w, warps=2, bisections=nb_grid)  # 2 warps per block: the persistent grid
    assert np.array_equal(got, grid) and np.array_equal(nb, nb_grid)
    assert np.array_equal(plain, grid) and np.array_equal(graded, grid)


@pytest.mark.parametrize("contracts_per_sm", [(16, -1), (16, 0), (40, 3), (128, 0), (128, 1), (300, -7)])
@pytest.mark.parametrize("model", ["heston", "bates"])
def test_automatic_order_prices_as_input_order(ope, model, contracts_per_sm):
    m = ope.MODEL_BATES if model == "bates" else ope.MODEL_HESTON
    sms = ope.device_info()[0]
    n = contracts_per_sm[0] * sms + contracts_per_sm[1]
    w = W.c3(n=n, per_surface=157, seed=n)
    if model == "heston":
        w.params = np.ascontiguousarray(w.params[:, :5])
    w.contracts["expiry"][:3] = 1.0 / 3650.0  # chains at the panel cap
    ope.set_autotune(False)
    try:
        auto = ope.price_surfaces(m, w.contracts, w.surf_offsets, w.params, tol=w.tol)
        graded, _ = ope.price_gradient_surfaces(m, w.contracts, w.surf_offsets, w.params, tol=w.tol)
    finally:
        ope.set_autotune(True)
    assert np.array_equal(auto, _in_input_order(ope, m, w))
    assert np.array_equal(graded, auto)


@pytest.mark.parametrize("short", [1, 0])
@pytest.mark.parametrize("model", ["heston", "bates"])
def test_smallest_call_that_shares_runs(ope, model, short):
    """Runs of 32 equal expiries are shared from 576 contracts per SM: the same
    prices on both sides, bit for bit."""
    m = ope.MODEL_BATES if model == "bates" else ope.MODEL_HESTON
    n = 576 * ope.device_info()[0] - short
    w = W.c3(n=n, per_surface=4096, seed=3)
    if model == "heston":
        w.params = np.ascontiguousarray(w.params[:, :5])
    for f in ("expiry", "rate"):
        w.contracts[f] = w.contracts[f][np.arange(n) // 32 * 32]
    ope.set_autotune(False)
    try:
        got = ope.price_surfaces(m, w.contracts, w.surf_offsets, w.params, tol=w.tol)
        used = ope.last_per_unit()
    finally:
        ope.set_autotune(True)
    assert used == (1 if short else 4)
    assert np.array_equal(got, _in_input_order(ope, m, w))
