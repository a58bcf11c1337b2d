"""The batched interaction matrix against one poke after the other.

Both form every value with the same operations, so the matrices are equal bit
for bit.  The cases are where the batched form selects its work: patches that
hang over the DM screen's edge, fractional offsets, one patch that reaches more
sub-apertures than an actuator's list holds at a time, patches that reach none,
interleaved slopes, and reference slopes that are not finite (the entries of
sub-apertures a poke does not reach are then NaN, as poking them gives).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _poked(core, optics, w, c, dm, off, push, nact, nslope, out):
    imat = np.zeros((nslope, nact), np.float32)
    for a in range(nact):
        s = []
        for com_a in (push, -push):
            com = np.zeros(nact, np.float32)
            com[a] = com_a
            dm.set_com(com)
            dm.comp_shape()
            optics.raytrace(w.d_phase.ptr, w.npup, w.npup, [(dm.d_shape.ptr, dm.dim, off, off)])
            w.comp_image(noise=False)
            c.get_cog(out.ptr)
            s.append(np.array(out))
        imat[:, a] = (s[0] - s[1]) / np.float32(2 * push)
    return imat


@pytest.mark.parametrize("nxsub,pd,isz,off,order,ref", [
    (16, 6, 20, 8.0, 0, 0.0),
    (12, 5, 17, 7.25, 1, 0.1),
    (30, 4, 140, 4.5, 0, 0.0),   # one patch over every sub-aperture: 716 > the list's 512
    (10, 8, 9, 6.0, 0, np.inf),
])
def test_imat_equals_pokes(nxsub, pd, isz, off, order, ref):
    from aob200 import _lib, core, optics
    from aob200 import geometry as G

    g = G.sh_geometry(G.ShParams(nxsub=nxsub, npix=6, pixsize=0.36, wavelength_um=0.7), nxsub * pd)
    w = core.ShWfs.from_geometry(g)
    c = core.Centroider(g.nvalid, g.npix / 2 - 0.5, g.pixsize, "tcog")
    c.set_npix(g.npix)
    c.set_threshold(0.01 * g.nphotons / 36)
    c.set_slope_order(order)
    c.load_validpos(g.validsubsx, g.validsubsy)
    c.set_centroids_ref(np.full(2 * g.nvalid, ref, np.float32))
    c.attach(w)
    rng = np.random.default_rng(nxsub)
    dim, nact = g.tel.n + 2 * int(off) + 1, 7
    # around the screen's centre, over each edge, and far outside it
    at = np.array([dim // 2 - isz // 2, -isz // 2, dim - isz // 2, 3, dim - isz - 2, -2 * isz, dim + 5], np.int32)
    influ = rng.standard_normal((isz, isz, nact)).astype(np.float32)
    dm = optics.Dm(dim, influ, at, at[::-1].copy())
    nslope, push = 2 * g.nvalid, 0.03
    out = core.OwnedDeviceArray(nslope)
    imat = core.OwnedDeviceArray(nslope * nact)
    for chunk in (0, 3):
        imat.set(np.full(nslope * nact, 7.0, np.float32))
        _lib.call("aob_imat_build", w.h, c.h, dm.h, float(off), float(off), push, chunk, imat.ptr, None)
        got = np.array(imat).reshape(nslope, nact, order="F")
        np.testing.assert_array_equal(got, _poked(core, optics, w, c, dm, off, push, nact, nslope, out))
    assert np.isfinite(got).all() == np.isfinite(ref)


@pytest.mark.parametrize("nxsub,isz", [
    (19, 200),   # nvalid just above one round of 256 candidates, all reached
    (24, 78),    # more than 256 reached, fewer than the list's 512
    (40, 300),   # every one of about 1250
])
def test_pokes_that_reach_many(nxsub, isz):
    """A CTA lists its actuator's sub-apertures 256 candidates at a time and forms the
    listed ones when 512 places could run out.  With a whole round reached (tip-tilt and
    modal influence functions) the count stands at the limit, where every thread has to
    take the same branch: each of several calls equals the pokes bit for bit."""
    from aob200 import _lib, core, optics
    from aob200 import geometry as G

    pd = 4
    g = G.sh_geometry(G.ShParams(nxsub=nxsub, npix=6, pixsize=0.36, wavelength_um=0.7), nxsub * pd)
    w = core.ShWfs.from_geometry(g)
    c = core.Centroider(g.nvalid, g.npix / 2 - 0.5, g.pixsize, "cog")
    c.set_npix(g.npix)
    c.load_validpos(g.validsubsx, g.validsubsy)
    c.attach(w)
    assert g.nvalid > 256
    dim, nact, off = g.tel.n + 13, 5, 6.0
    x, y = (np.arange(isz) - isz / 2)[:, None], (np.arange(isz) - isz / 2)[None, :]
    modes = np.stack([x + 0 * y, y + 0 * x, x * y / isz, (x * x + y * y) / isz, (x * x - y * y) / isz], -1)
    at = np.full(nact, dim // 2 - isz // 2, np.int32)
    dm = optics.Dm(dim, (modes / isz).astype(np.float32), at, at)
    nslope, push = 2 * g.nvalid, 0.05
    out = core.OwnedDeviceArray(nslope)
    want = _poked(core, optics, w, c, dm, off, push, nact, nslope, out)
    assert (want != 0).any(axis=1).sum() > 2 * 256 - 16
    imat = core.OwnedDeviceArray(nslope * nact)
    for _ in range(8):
        imat.set(np.full(nslope * nact, 7.0, np.float32))
        _lib.call("aob_imat_build", w.h, c.h, dm.h, off, off, push, 0, imat.ptr, None)
        np.testing.assert_array_equal(np.array(imat).reshape(nslope, nact, order="F"), want)
