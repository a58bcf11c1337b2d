"""Chains of kernels started while their predecessor runs give what a chain with a
host wait after every call gives, bit for bit: calls on one stream, on two streams
that take turns, and captured in a CUDA graph."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(seed=5):
    import torch

    from aob200 import core, workloads as W

    s = W.sh_loop_setup("plain16")
    wfs, c, ls, loop = W.build_sh_loop(s, graph=False)
    ls.set_delay(1.0)
    c.set_threshold(s.threshold)
    rng = np.random.default_rng(seed)
    wfs.set_phase((0.1 * rng.standard_normal((wfs.npup, wfs.npup))).astype(np.float32))
    slopes = ls.buffer("centroids").ptr

    def step(sp, wait):
        for f in (lambda: wfs.comp_image(True, sp), lambda: c.get_cog(slopes, sp), lambda: ls.comp_com(sp),
                  lambda: ls.comp_voltage(sp)):
            f()
            if wait:
                torch.cuda.synchronize()

    def state():
        torch.cuda.synchronize()
        return [np.array(x) for x in (wfs.d_binimg, ls.buffer("centroids"), ls.buffer("err"), ls.buffer("voltage"))]

    return step, state


def test_chain_equals_waiting_after_every_call():
    a, sa = _chain()
    b, sb = _chain()
    for _ in range(40):
        a(None, True)
        b(None, False)
    for x, y in zip(sa(), sb()):
        np.testing.assert_array_equal(x, y)


def test_chains_on_two_streams():
    import torch

    chains = [_chain(k) for k in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    a, sa = chains[0]
    for _ in range(30):
        a(None, True)
    want = sa()
    x, sx = _chain(0)
    for k in range(30):  # the same chain changes streams, another one runs beside it
        s, o = streams[k % 2], streams[1 - k % 2]
        s.wait_stream(o)
        x(s.cuda_stream, False)
        chains[1][0](o.cuda_stream, False)
    for p, q in zip(want, sx()):
        np.testing.assert_array_equal(p, q)


def test_chain_in_a_graph():
    import torch

    a, sa = _chain()
    b, sb = _chain()
    for f in (a, b):  # (first uses, and the ring of commands, outside the capture)
        f(None, True)
    g = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        for _ in range(3):  # (the delay ring of three returns to its start)
            b(torch.cuda.current_stream().cuda_stream, False)
    for _ in range(2):
        g.replay()
    got = sb()
    assert np.isfinite(got[0]).all()
    for _ in range(3):
        a(None, True)
    first = sa()
    # the noise frame is part of the captured launch, so the second replay repeats the first's images
    np.testing.assert_array_equal(got[0], first[0])
    np.testing.assert_array_equal(got[1], first[1])
