"""Device-resident steps as two overlapping kernels equal the fused kernel's and the
separate kernels', bit for bit, over the matrix precisions, delays (0.4 takes the fused
kernel in both), clipping and slope orders, also when steps with and without host
buffers alternate; configurations that the pair does not take still run."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loop(prec, delay, clip, order, mode, name="plain16"):
    from aob200 import workloads as W

    s = W.sh_loop_setup(name)
    w, c, ls, loop = W.build_sh_loop(s, precision=prec, graph=False)
    ls.set_delay(delay)
    if clip:
        ls.set_com_range(-0.01, 0.012)
    c.set_slope_order(order)
    loop.set_mode(mode)
    w.set_noise(0.5, 9)
    rng = np.random.default_rng(3)
    w.set_phase((0.1 * rng.standard_normal((w.npup, w.npup))).astype(np.float32))
    return s, w, c, ls, loop


@pytest.mark.parametrize("prec,delay,clip,order", [
    ("f32", 0.0, False, 0), ("f32", 1.0, True, 1), ("bf16", 2.0, True, 0), ("fp8", 0.0, True, 1), ("f32", 1.5, False, 0),
    ("f32", 0.4, False, 0)])
def test_pair_equals_fused(prec, delay, clip, order):
    a = _loop(prec, delay, clip, order, 0)
    b = _loop(prec, delay, clip, order, 2)
    va, vb = np.zeros(a[0].nactu, np.float32), np.zeros(a[0].nactu, np.float32)
    for k in range(7):
        host = k in (2, 5)
        a[4].step(None, va if host else None, noise=True)
        b[4].step(None, vb if host else None, noise=True)
        assert a[4].kernels_per_step() == (1 if host or 0 < delay < 1 else 2)
        assert b[4].kernels_per_step() == 1
        for n in ("centroids", "err", "com", "voltage"):
            np.testing.assert_array_equal(np.array(a[3].buffer(n)), np.array(b[3].buffer(n)), err_msg=f"{n} {k}")
        np.testing.assert_array_equal(np.array(a[1].d_binimg), np.array(b[1].d_binimg))
    np.testing.assert_array_equal(va, vb)
    assert a[1].frame == b[1].frame == 7 and a[3].status() == 0


def test_perturbed_and_open_loops_take_their_own_path():
    a = _loop("f32", 0.0, False, 0, 0)
    b = _loop("f32", 0.0, False, 0, 1)
    p = np.linspace(-0.1, 0.1, 2 * a[0].nactu).astype(np.float32).reshape(2, -1)
    for s, w, c, ls, loop in (a, b):
        ls.add_perturb("p", p, 2)
    for k in range(4):
        if k == 2:
            for x in (a, b):
                x[3].enable_perturb("p", False)
        for x in (a, b):
            x[4].step(None, None, noise=False)
        assert a[4].kernels_per_step() == (3 if k < 2 else 2)
        np.testing.assert_array_equal(np.array(a[3].buffer("voltage")), np.array(b[3].buffer("voltage")))
    for x in (a, b):
        x[3].set_open_loop(1, False)
        x[4].step(None, None, noise=False)
    np.testing.assert_array_equal(np.array(a[3].buffer("voltage")), np.array(b[3].buffer("voltage")))
