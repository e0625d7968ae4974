"""Host-pointer calls whose inputs and results pass through the thread's pinned
buffer, on both sides of its limits: the results are those of device pointers
(prices, Greeks) or of the oracle (implied vols), whatever mixture of pageable
and pinned buffers the caller brings."""
import ctypes

import numpy as np
import pytest

from ope_b200 import _lib
from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch

    t = torch.empty(a.nbytes, dtype=torch.uint8).pin_memory()
    v = t.numpy().view(a.dtype).reshape(a.shape)
    v[...] = a
    return t, v


@pytest.mark.parametrize("n", [1, 7, 16384, 16385])
@pytest.mark.parametrize("pin_in,pin_out", [(False, False), (True, False), (False, True), (True, True)])
def test_plain_prices_from_any_buffers(ope, n, pin_in, pin_out):
    import torch

    w = W.c3(n=n, per_surface=n, seed=n)
    con, out = w.contracts, np.empty(n)
    if pin_in:
        keep_c, con = _pinned(con)
    if pin_out:
        keep_o, out = _pinned(out)
    o = _lib.Options(tol=w.tol, flags=0, reserved=0, stream=None)
    _lib.check(_lib.load().ope_batch_price_ex(ope.MODEL_BATES, con.ctypes.data, n, w.params.ctypes.data,
                                              out.ctypes.data, ctypes.byref(o)))
    d_con, d_par = torch.from_numpy(w.contracts.view(np.uint8).copy()).cuda(), torch.from_numpy(w.params).cuda()
    d_out = torch.empty(n, dtype=torch.float64, device="cuda")
    ope.batch_price_device(ope.MODEL_BATES, d_con, n, d_par, d_out, tol=w.tol)
    assert np.array_equal(out, d_out.cpu().numpy())
    assert np.array_equal(out, ope.price_surfaces(ope.MODEL_BATES, w.contracts, w.surf_offsets, w.params, tol=w.tol))


@pytest.mark.parametrize("analytic", [False, True])
def test_greeks_on_both_sides_of_the_staging_limit(ope, analytic):
    """3 << 19 bytes of contracts and results (120 per contract): 13,100 pass
    through the pinned buffer, 13,120 do not; the shared contracts' Greeks agree."""
    w = W.c3(n=13120, per_surface=13120, seed=5)
    w.contracts["expiry"] = np.maximum(w.contracts["expiry"], 0.3)

    def greeks(con):
        if analytic:
            return ope.batch_greeks_ad(ope.MODEL_BATES, con, w.params[0], tol=1e-8, analytic=True)
        return ope.batch_bates_greeks(con, w.params[0])

    a, b = greeks(w.contracts[:13100]), greeks(w.contracts)
    assert np.array_equal(a, b[:13100])


@pytest.mark.parametrize("n", [1, 2, 3, 4097, 16385, 131073])
def test_implied_vols_in_two_parts(ope, oracle, n):
    """Up to 4,097 go in one part; 131,073 is past what the results' pinned buffer takes.  The solver stops
    within 1e-10 of the price; these quotes' vegas are S sqrt(T) phi(d1) >= 3
    (T >= 0.1, |d1| <= 1.5), so the vols lie within 1e-10 / 3 of the true ones;
    the bar is 1e-9."""
    rng = np.random.default_rng(n)
    con = np.zeros(n, W.CONTRACT_DTYPE)
    vol, T = rng.uniform(0.1, 0.6, n), rng.uniform(0.1, 2.0, n)
    con["spot"], con["expiry"], con["rate"], con["div_yield"] = 100.0, T, 0.02, 0.01
    con["strike"] = 100.0 * np.exp(0.01 * T + rng.uniform(-1.0, 1.0, n) * vol * np.sqrt(T))
    con["opt_type"] = con["strike"] < 100.0 * np.exp(0.01 * T)
    con["vol"] = vol
    from scipy.special import ndtr

    w = np.where(con["opt_type"] == 0, 1.0, -1.0)
    sq = vol * np.sqrt(T)
    d1 = (np.log(100.0 / con["strike"]) + (0.01 + 0.5 * vol * vol) * T) / sq
    px = w * (100.0 * np.exp(-0.01 * T) * ndtr(w * d1) - con["strike"] * np.exp(-0.02 * T) * ndtr(w * (d1 - sq)))
    iv, ok = ope.batch_implied_vol(con, px)
    assert ok.all() and np.max(np.abs(iv - vol)) <= 1e-9
    pick = rng.choice(n, min(n, 500), replace=False)
    ref, rok = oracle.batch_implied_vol(con[pick], px[pick])
    assert np.all(rok) and np.max(np.abs(iv[pick] - ref)) <= 1e-9
