"""The pyramid's transforms at every size they are compiled for, against numpy.

Each nfft runs other passes (radix 8 with a last radix 2 or 4), other groups of
threads and other splits of the modulation points; the cases also vary the
binning, the phase grid (odd, up to nfft), weights, a field stop that is neither 0
nor 1, and the focal-plane image.

Tolerance: float32 transforms of length N err by about log2(N) 2^-24 relative rms
per transform; four of them, |.|^2 and the normalisation stay below 2e-6 (the
largest size, 11 passes x 4 x 6e-8).
"""

from types import SimpleNamespace

import numpy as np
import pytest

from helpers import rel_rms
from oracle import pyr as opyr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft,ntot,nrebin,npts", [
    (64, 21, 8, 3), (64, 64, 1, 13), (128, 50, 4, 5), (256, 72, 4, 1), (256, 131, 1, 17), (512, 104, 2, 9),
    (1024, 300, 2, 5), (2048, 333, 8, 3),
])
def test_pyramid_sizes(nfft, ntot, nrebin, npts):
    from aob200 import core

    rng = np.random.default_rng(nfft + npts)
    x = np.arange(nfft) - nfft / 2
    r = np.hypot(*np.meshgrid(x, x, indexing="ij"))
    face = 0.2 * np.minimum(np.abs(x[:, None] + 0.3 * x[None, :]), 9.0) / nrebin
    n = np.arange(ntot) - ntot / 2
    pup = (np.hypot(*np.meshgrid(n, n, indexing="ij")) < ntot / 2.2).astype(np.float32)
    ang = 2 * np.pi * np.arange(npts) / npts
    g = SimpleNamespace(
        nfft=nfft, nrebin=nrebin, halfxy=np.fft.fftshift(face).astype(np.float32),
        submask=np.fft.fftshift(np.clip(1.2 - r / nfft, 0, 1)).astype(np.float32),
        sincar=np.fft.fftshift(np.sinc(x[:, None] / nfft) * np.sinc(x[None, :] / nfft)).astype(np.float32),
        pyr_cx=(0.05 * np.sin(ang)).astype(np.float32), pyr_cy=(0.05 * np.cos(ang)).astype(np.float32))
    wts = rng.uniform(0.5, 1.5, npts).astype(np.float32)
    w = core.PyrWfs(4, 1, 2, 2, nrebin, nfft, ntot, npts, 1.0, 1000.0, lambda_um=0.7)
    w.load_arrays(g.halfxy, g.pyr_cx, g.pyr_cy, wts, g.sincar, g.submask, np.zeros(4), np.zeros(4))
    w.set_pupil(pup)
    ph = (0.08 * rng.standard_normal((ntot, ntot))).astype(np.float32)
    w.set_phase(ph)
    ref = opyr.comp_image(ph, pup, g, 0.7, 1000.0, weights=wts)
    for focal in (False, True):
        w.set_compute_focalplane(focal)
        w.comp_image(noise=False)
        assert rel_rms(np.array(w.d_binimg), ref) < 2e-6
        assert rel_rms(np.array(w.d_hrimg), opyr.hr_image(ph, pup, g, 0.7, weights=wts)) < 2e-6
    foc = w.buffer("pyrfocalplane", shape=(nfft, nfft))
    assert rel_rms(np.array(foc), opyr.focal_plane(ph, pup, g, 0.7, weights=wts)) < 2e-6


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n,batch", [(8, 3), (16, 130), (32, 1), (64, 5), (128, 2), (256, 3), (512, 1), (1024, 2),
                                     (2048, 1)])
def test_fft2d_sizes(n, batch, inverse):
    import torch

    from aob200 import optics

    rng = np.random.default_rng(n)
    x = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    d = torch.from_numpy(x).cuda()
    optics.fft2d(d.data_ptr(), n, batch, inverse)
    torch.cuda.synchronize()
    ref = np.fft.ifft2(x.astype(np.complex128)) * n * n if inverse else np.fft.fft2(x.astype(np.complex128))
    got = d.cpu().numpy()
    assert rel_rms(np.stack([got.real, got.imag]), np.stack([ref.real, ref.imag])) < 1e-6
