"""What optics.raytrace takes as a source: any numbers that int() and float() take (NumPy scalars,
a whole float), and entries behind the four that it reads.  The library call is replaced by
a recorder, so no GPU is needed."""

import ctypes

import numpy as np
import pytest

from aob200 import optics


@pytest.mark.parametrize("sources", [
    [(4096, 17, 0.5, -1.25)],
    [(4096, np.int64(17), np.float64(0.5), np.float32(-1.25)), (8192, np.int32(9), 1, np.int64(2))],
    [(4096, 17.0, "0.5", np.array(-1.25))],
    [[4096, 17, 0.5, -1.25, "layer 0"]],
    [(None, 17, 0.5, -1.25)],
    [],
])
def test_raytrace_sources(monkeypatch, sources):
    seen = {}

    def record(name, out, nx, ny, n, ptrs, dims, xo, yo, reset, stream):
        def read(t, at):
            return list((t * n).from_address(at)) if n else []

        seen.update(name=name, n=n, ptrs=read(ctypes.c_void_p, ptrs), dims=read(ctypes.c_int, dims),
                    xo=read(ctypes.c_float, xo), yo=read(ctypes.c_float, yo))

    monkeypatch.setattr(optics, "call", record)
    optics.raytrace(64, 8, 8, sources)
    assert seen["name"] == "aob_raytrace" and seen["n"] == len(sources)
    assert seen["ptrs"] == [s[0] for s in sources]
    assert seen["dims"] == [int(s[1]) for s in sources]
    assert seen["xo"] == [float(s[2]) for s in sources] and seen["yo"] == [float(s[3]) for s in sources]
