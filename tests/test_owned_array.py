"""OwnedDeviceArray hands its zeros to the copy while they are still alive (CPU: the
library call is replaced by one that looks)."""

import weakref

import numpy as np

from aob200 import core


def test_zeros_outlive_the_copy(monkeypatch):
    made, seen = [], []
    real_zeros = np.zeros

    def zeros(*a, **k):
        z = real_zeros(*a, **k)
        made.append(weakref.ref(z))
        return z

    def call(name, *args):
        if name == "aob_memcpy_h2d":
            z = made[-1]()
            seen.append(z is not None and args[1] == z.ctypes.data and args[2] == z.nbytes)

    monkeypatch.setattr(core.np, "zeros", zeros)
    monkeypatch.setattr(core, "call", call)
    core.OwnedDeviceArray(1000, np.float32)
    assert seen == [True]
