"""A tuned table's default rows (4 warps, input order, all blocks, contracts per
unit 0) launch as an untuned call does, and the tuner measures its shapes
against that launch.  Seen by the kernel launches of a call: a deepest-first
queue takes two more (bucket and scatter)."""
import numpy as np
import pytest

from ope_b200 import workloads as W

pytestmark = pytest.mark.gpu

DEFAULT = dict(warps_per_block=4, deepest_first=False, occupancy=1.0, per_unit=0)


def _launches(ope, model, w):
    ope.price_surfaces(model, w.contracts, w.surf_offsets, w.params, tol=w.tol)  # workspace, first-use work
    before = ope.kernel_launch_count()
    prices = ope.price_surfaces(model, w.contracts, w.surf_offsets, w.params, tol=w.tol)
    return ope.kernel_launch_count() - before, prices


def _workload(ope, per_sm, model):
    w = W.c3(n=per_sm * ope.device_info()[0], per_surface=157, seed=per_sm)
    if model == "heston":
        w.params = np.ascontiguousarray(w.params[:, :5])
    return w


def _untuned(ope, model, w):
    ope.set_autotune(False)
    try:
        return _launches(ope, model, w)
    finally:
        ope.set_autotune(True)


@pytest.mark.parametrize("per_sm", [8, 40, 200])
@pytest.mark.parametrize("model", ["heston", "bates"])
def test_default_rows_launch_as_untuned(ope, model, per_sm):
    m = ope.MODEL_BATES if model == "bates" else ope.MODEL_HESTON
    w = _workload(ope, per_sm, model)
    untuned, prices = _untuned(ope, m, w)
    assert untuned == (1 if per_sm < 16 else 3)
    saved, _ = ope.tune_table(m)
    try:
        ope.set_tune_table(m, [dict(r, **DEFAULT) for r in saved])
        launches, got = _launches(ope, m, w)
        assert launches == untuned and np.array_equal(got, prices)
        # a row that differs in any field is taken as it is
        for other in (dict(per_unit=1), dict(occupancy=0.5), dict(warps_per_block=2)):
            ope.set_tune_table(m, [dict(r, **dict(DEFAULT, **other)) for r in saved])
            launches, got = _launches(ope, m, w)
            assert launches == 1 and np.array_equal(got, prices)
        ope.set_tune_table(m, [dict(r, **dict(DEFAULT, deepest_first=True)) for r in saved])
        launches, got = _launches(ope, m, w)
        assert launches == 3 and np.array_equal(got, prices)
    finally:
        ope.set_tune_table(m, saved)


def test_the_tuner_measures_against_the_automatic_launch(ope):
    """Launches of a quick tuning: per class and repetition, the automatic launch
    (1, or 3 where it orders), 5 other shapes in input order (1 each) and 6
    deepest-first (3 each); 3 warm-up and 9 timed repetitions (5 from 11,585
    contracts)."""
    sms = ope.device_info()[0]
    expected = 0
    for n in (45, 91, 181, 362, 724, 1448, 2896, 5793, 11585, 23170, 46341, 92682):
        ordered = n > 256 and max(16 * sms, 256) <= n < 2400 * sms
        expected += (3 + (5 if n >= 11585 else 9)) * ((3 if ordered else 1) + 5 + 6 * 3)
    saved, _ = ope.tune_table(ope.MODEL_HESTON)
    try:
        before = ope.kernel_launch_count()
        rows = ope.autotune(ope.MODEL_HESTON, quick=True)
        assert ope.kernel_launch_count() - before == expected
        # every class that kept the default, measured or not, launches as untuned
        kept = [r["max_contracts"] or 1 << 21 for r in rows if all(r[k] == v for k, v in DEFAULT.items())]
        assert len(kept) >= 4  # the four that a quick tuning does not measure
        for top in kept:
            n = min(top, 1 << 18) - 3
            w = W.c3(n=n, per_surface=157, seed=1)
            w.params = np.ascontiguousarray(w.params[:, :5])
            launches, prices = _launches(ope, ope.MODEL_HESTON, w)
            untuned, want = _untuned(ope, ope.MODEL_HESTON, w)
            if top <= 1 << 18:
                assert launches == untuned
            assert np.array_equal(prices, want)
    finally:
        ope.set_tune_table(ope.MODEL_HESTON, saved)
