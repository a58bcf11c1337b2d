"""The generic controller's row products at widths around a warp and around the 512
values a warp has in flight, and camera frames from device memory at every alignment
(the frame copy's 16-byte path and its remainders)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nslope,nactu", [(2, 1), (7, 31), (64, 33), (130, 511), (96, 513), (33, 1100)])
def test_row_products(nslope, nactu):
    """polc slopes s - imat com_clipped and matE in the modal integrator; float32 sums
    of n terms err by at most n 2^-24 of the terms' absolute sum."""
    from aob200 import core

    rng = np.random.default_rng(nactu)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    ls = core.LsController(nslope, nactu, kind="generic")
    cmat, imat, matE, com, s = f(nactu, nslope), f(nslope, nactu), f(nactu, nactu), f(nactu), f(nslope)
    ls.set_commandlaw("modal_integrator")
    ls.set_cmat(cmat)
    ls.set_imat(imat)
    ls.set_matE(matE)
    ls.set_gain(0.3)
    ls.set_polc(True)
    ls.set_com(com)
    ls.comp_voltage()
    ls.set_centroids(s)
    ls.comp_com()
    d = np.float64
    ol = s.astype(d) - imat.astype(d) @ com
    b = -(cmat.astype(d) @ ol)
    want = np.float64(np.float32(0.3)) * (matE.astype(d) @ b) + (1 - np.float64(np.float32(0.3))) * com
    scale = np.abs(matE) @ (np.abs(cmat) @ (np.abs(s) + np.abs(imat) @ np.abs(com))) * 0.3 + np.abs(com)
    got = np.array(ls.buffer("com"))
    assert np.all(np.abs(got - want) <= (nactu + nslope + 8) * 2.0**-24 * scale)


@pytest.mark.parametrize("shape", [(1, 1), (5, 3), (16, 16), (33, 7), (240, 240)])
def test_device_frames(shape):
    import torch

    from aob200 import core

    n = shape[0] * shape[1]
    rng = np.random.default_rng(n)
    c = core.Centroider(1, 0.0, 1.0, "cog")
    for off in (0, 1, 3, 8):
        h = rng.integers(0, 65536, n + 16).astype(np.uint16)
        d = torch.from_numpy(h.astype(np.int32)).cuda().to(torch.uint16)
        view = core.DeviceArray(d.data_ptr() + 2 * off, n, np.uint16, shape, d)
        c.load_img(view)
        np.testing.assert_array_equal(np.array(c.buffer("img_raw", dtype=np.uint16)), h[off:off + n])
    raw = c.buffer("img_raw", dtype=np.uint16, shape=shape)
    c.load_img(raw)  # in place
    np.testing.assert_array_equal(np.array(raw).ravel(order="F"), h[8:8 + n])
