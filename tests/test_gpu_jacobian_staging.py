"""The Jacobian call's inputs and results pass through the thread's pinned buffer
up to 3 << 19 bytes and are copied directly beyond: the same rows on both sides
of either limit, and a large call leaves no page-locked memory behind."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu

DIM = {"heston": 5, "bates": 8}


def _quotes(ope, n, bates, per_surface=256):
    w = W.c3(n=n, per_surface=per_surface, seed=11)
    if not bates:
        w.params = np.ascontiguousarray(w.params[:, :5])
    w.contracts["expiry"] = np.maximum(w.contracts["expiry"], 0.2)
    return w, np.full(n, 0.25)


# bytes in: 64 per quote (and the surfaces' offsets and parameters), out: 8 (dim + 1) per quote
@pytest.mark.parametrize("model,n", [("heston", 24000), ("heston", 24700), ("heston", 32768), ("heston", 32769),
                                     ("bates", 21845), ("bates", 21846), ("bates", 1), ("heston", 257)])
def test_rows_on_both_sides_of_the_staging_limits(ope, model, n):
    bates = model == "bates"
    m = ope.MODEL_BATES if bates else ope.MODEL_HESTON
    w, iv = _quotes(ope, n, bates)
    jac, res = ope.calib_jacobian(m, w.contracts, iv, w.surf_offsets, w.params, tol=1e-8)
    assert jac.shape == (n, DIM[model])
    k = min(n, 256)  # the last surface alone, small enough to be staged both ways
    a = int(w.surf_offsets[-2])
    tail_jac, tail_res = ope.calib_jacobian(m, w.contracts[a:], iv[a:], [0, n - a], w.params[-1:], tol=1e-8)
    assert np.array_equal(jac[a:], tail_jac) and np.array_equal(res[a:], tail_res)
    head_jac, head_res = ope.calib_jacobian(m, w.contracts[:k], iv[:k], [0, k], w.params[:1], tol=1e-8)
    assert np.array_equal(jac[:k], head_jac) and np.array_equal(res[:k], head_res)
    assert np.any(jac != 0.0)


def _address_space():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) * 1024 for line in f if line.startswith("VmSize"))


def test_a_large_call_pins_nothing(ope):
    """400,000 quotes would take 26 MB of page-locked memory for the inputs."""
    w, iv = _quotes(ope, 400_000, False)
    small, small_iv = _quotes(ope, 1024, False)
    # the device workspace of the large call and every kernel are there before
    ope.price_gradient_surfaces(ope.MODEL_HESTON, *(lambda b: (b.contracts, b.surf_offsets, b.params))(
        _quotes(ope, 1_000_000, False)[0]), tol=1e-6)
    ope.calib_jacobian(ope.MODEL_HESTON, small.contracts, small_iv, small.surf_offsets, small.params, tol=1e-8)
    before = _address_space()
    jac, res = ope.calib_jacobian(ope.MODEL_HESTON, w.contracts, iv, w.surf_offsets, w.params, tol=1e-8)
    grown = _address_space() - before - jac.nbytes - res.nbytes
    assert grown < 8 << 20, grown
