"""The shapes a batch picks by its size give what the former fixed shape gives, bit for
bit: batches on each side of the rule's limits (16, 30 and 100 sub-apertures per SM),
mixed sizes, and each value given on its own."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(sizes, prec):
    from aob200 import workloads as W

    inst = [W.mc_make(nx, npix, 0.12, k) for k, (nx, npix) in enumerate(sizes)]
    return W.build_mc_batch(inst, precision=prec)


@pytest.mark.parametrize("sizes,prec", [
    ([(8, 6)], "f32"), ([(40, 6), (30, 8), (31, 6)], "fp8"), ([(40, 6)] * 4, "bf16"),
    ([(40, 8)] * 12 + [(9, 6), (24, 8)], "bf16"),
])
def test_picked_shapes_equal_the_fixed_one(sizes, prec):
    outs = []
    for tuning in (None, dict(subaps_per_item=32, team_threads=32, mvm_kb=48, lag=2, ctas_per_sm=2),
                   dict(ctas_per_sm=3), dict(mvm_kb=24, lag=0), dict(lag=-1), dict(team_threads=64, ctas_per_sm=4)):
        loops, b = _batch(sizes, prec)
        if tuning is not None:
            b.set_tuning(**tuning)
        for _ in range(2):
            b.step(True)
        outs.append([[np.array(ls.buffer("voltage")), np.array(w.d_binimg)] for w, c, ls, loop in loops])
        assert b.status() == 0
    for other in outs[1:]:
        for x, y in zip(outs[0], other):
            np.testing.assert_array_equal(x[0], y[0])
            np.testing.assert_array_equal(x[1], y[1])


def test_lag_left_to_the_batch():
    """set_tuning leaves the lag to the batch unless it is given, and takes -1 for that; below -1 it
    is refused."""
    from aob200._lib import AobError

    loops, b = _batch([(24, 6)] * 6, "bf16")
    for kw in ({}, dict(ctas_per_sm=3), dict(lag=-1, mvm_kb=24)):
        b.set_tuning(**kw)
        b.step(True)
    assert b.status() == 0
    with pytest.raises(AobError, match="lag"):
        b.set_tuning(lag=-2)
