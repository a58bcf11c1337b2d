"""The target's short- and long-exposure images at every transform size, against numpy
(float32 transforms: 2 x log2(N) roundings of 6e-8, squared; 2e-6 holds at 2048)."""

import numpy as np
import pytest

from helpers import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npup,nfft", [(8, 8), (5, 16), (31, 32), (64, 64), (77, 128), (100, 256), (240, 512),
                                       (512, 1024), (601, 2048)])
def test_target_sizes(npup, nfft):
    from aob200 import core, optics

    rng = np.random.default_rng(npup)
    pup = (rng.random((npup, npup)) < 0.8).astype(np.float32)
    pup[0, 0] = 1.0
    t = optics.Target(pup, 1.65, nfft)
    le, n = np.zeros((nfft, nfft)), pup.sum()
    for k in range(3):
        ph = (0.1 * rng.standard_normal((npup, npup))).astype(np.float32)
        t.d_phase.set(ph)
        t.comp_image(None, k != 1)  # the second image stays out of the long exposure
        f = np.zeros((nfft, nfft), complex)
        f[:npup, :npup] = np.where(pup > 0, np.exp(1j * np.float32(2 * np.pi / 1.65) * ph.astype(np.float64)), 0)
        spec = np.fft.fft2(f)
        se = np.abs(spec / n) ** 2
        le += se if k != 1 else 0
        assert rel_rms(np.array(t.d_image_se), se) < 2e-6
        assert rel_rms(np.array(t.d_image_le), le) < 2e-6
        amp = t.buffer("amplipup")  # nfft^2 complex values
        a = np.array(core.DeviceArray(amp.ptr, nfft * nfft, np.complex64, (nfft, nfft), t))
        assert rel_rms(np.stack([a.real, a.imag]), np.stack([spec.real, spec.imag])) < 2e-6
        s = t.strehl()
        assert s[0] == np.array(t.d_image_se).max()
        assert abs(s[1] * (1 if k < 2 else 2) - np.array(t.d_image_le).max()) <= 1e-6 * s[1]
