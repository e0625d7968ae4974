"""Automatic launches of several surfaces take their contracts deepest-first and
may keep fewer warps resident per SM (from 16 contracts per SM): the prices are
those of input order, bit for bit, on both sides of the size limits, and for
the launches that store panel lists (gradients)."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _in_input_order(ope, model, w):
    """The same call through a table whose every class is 4 warps, input order."""
    saved, _ = ope.tune_table(model)
    try:
        ope.set_tune_table(model, [dict(r, warps_per_block=4, deepest_first=False, occupancy=1.0, per_unit=1)
                                   for r in saved])
        return ope.price_surfaces(model, w.contracts, w.surf_offsets, w.params, tol=w.tol)
    finally:
        ope.set_tune_table(model, saved)


@pytest.mark.parametrize("contracts_per_sm", [(16, -1), (16, 0), (40, 3), (130, 1), (300, -7)])
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
