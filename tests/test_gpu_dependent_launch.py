"""Chains of kernels started while their predecessor runs give what a chain with a
host wait after every call gives, bit for bit: calls on one stream, on two streams
that take turns, and captured in a CUDA graph.  What a kernel
writes into a table whose address the library hands out is what the next image uses."""

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


def _writers(shape, values):
    """Ways of writing ``values`` (x fastest) to a device buffer by a kernel on a stream: the
    library's raytracing of a screen, whose grid lets its successor start early, and an
    operation of another library."""
    import torch

    from aob200 import core, optics

    nx, ny = shape
    d = max(nx, ny) + 1
    screen = core.OwnedDeviceArray(d * d)
    host = np.zeros((d, d), np.float32)
    host[:nx, :ny] = values.reshape(nx, ny, order="F")
    screen.set(host)
    src = torch.from_numpy(values.ravel(order="F").copy()).cuda()

    def traced(buf, sp):
        optics.raytrace(buf.ptr, nx, ny, [(screen.ptr, d, 0.0, 0.0)], True, sp)

    def copied(buf, sp):
        with torch.cuda.stream(torch.cuda.ExternalStream(sp)):
            torch.add(src, 0.0, out=torch.as_tensor(core.DeviceArray(buf.ptr, nx * ny, np.float32), device="cuda"))

    return traced, copied


def _check_table(buf, shape, image, result, rng):
    """image(stream) behind a kernel that writes the table, without a host wait in
    between, gives what it gives with one."""
    import torch

    stream = torch.cuda.Stream()
    sp = stream.cuda_stream
    old = np.array(buf).ravel(order="F")[: shape[0] * shape[1]]
    sets = [old, (old * rng.uniform(0.5, 1.5, old.size) + 0.01 * rng.standard_normal(old.size)).astype(np.float32)]
    want = []
    for v in sets:
        _writers(shape, v)[0](buf, sp)
        torch.cuda.synchronize()
        image(sp)
        torch.cuda.synchronize()
        want.append(result())
    assert not all(np.array_equal(a, b) for a, b in zip(*want))
    ways = [_writers(shape, v) for v in sets]
    torch.cuda.synchronize()
    for k in range(24):
        ways[k % 2][k // 2 % 2](buf, sp)
        image(sp)
        torch.cuda.synchronize()
        for a, b in zip(result(), want[k % 2]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("table", ["pupil", "offsets", "fluxPerSub", "centroids_ref", "weights", "gain"])
def test_sensor_tables_written_on_the_stream(table):
    from aob200 import workloads as W

    s = W.sh_loop_setup("plain16")
    s.centroider = "wcog" if table == "weights" else "cog"
    wfs, c, ls, loop = W.build_sh_loop(s, graph=False)
    rng = np.random.default_rng(3)
    wfs.set_phase((0.1 * rng.standard_normal((wfs.npup, wfs.npup))).astype(np.float32))
    buf = {"centroids_ref": c, "weights": c, "gain": ls}.get(table, wfs).buffer(table)
    n = {"pupil": wfs.npup, "offsets": s.geom.pdiam, "weights": wfs.npix}.get(table)
    shape = (n, n) if n else (buf.n, 1)
    com = np.zeros(ls.buffer("com").n, np.float32)

    def image(sp):
        ls.set_com(com)
        loop.step(None, None, False, sp)

    def result():
        return [np.array(x) for x in (wfs.d_bincube, ls.buffer("centroids"), ls.buffer("voltage"))]

    _check_table(buf, shape, image, result, rng)


@pytest.mark.parametrize("table", ["submask", "phalfxy", "sincar"])
def test_pyramid_tables_written_on_the_stream(table):
    from aob200 import core

    rng = np.random.default_rng(4)
    nfft, ntot, npts = 256, 72, 5
    x = np.arange(nfft) - nfft / 2
    ang = 2 * np.pi * np.arange(npts) / npts
    r = np.hypot(x[:, None], x[None, :])
    w = core.PyrWfs(4, 1, 2, 2, 4, nfft, ntot, npts, 1.0, 1000.0, lambda_um=0.7)
    w.load_arrays(np.fft.fftshift(0.05 * np.minimum(np.abs(x[:, None] + 0.3 * x[None, :]), 9.0)).astype(np.float32),
                  (0.05 * np.sin(ang)).astype(np.float32), (0.05 * np.cos(ang)).astype(np.float32),
                  np.ones(npts, np.float32),
                  np.fft.fftshift(np.sinc(x[:, None] / nfft) * np.sinc(x[None, :] / nfft)).astype(np.float32),
                  np.fft.fftshift(np.clip(1.2 - r / nfft, 0, 1)).astype(np.float32), np.zeros(4), np.zeros(4))
    w.set_pupil(np.ones((ntot, ntot), np.float32))
    w.set_phase((0.05 * rng.standard_normal((ntot, ntot))).astype(np.float32))
    buf = w.buffer(table)
    _check_table(buf, (nfft, nfft), lambda sp: w.comp_image(False, sp), lambda: [np.array(w.d_binimg)], rng)


def test_training_chain():
    """Forward, backward and Adam of several steps, with and without a host wait after each call:
    a step's epilogues read the biases that the step before has just written."""
    import torch

    from aob200 import mlp

    rng = np.random.default_rng(6)
    nin, h1, h2, nout, batch = 200, 96, 72, 50, 700
    x = torch.from_numpy(rng.standard_normal((batch, nin)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal((batch, nout)).astype(np.float32)).cuda()
    got = []
    for wait in (True, False):
        m = mlp.MlpReconstructor(nin, nout, h1, h2, seed=7)
        y = torch.empty((batch, nout), device="cuda")
        for _ in range(20):
            for f in (lambda: m.train_step(x.data_ptr(), t.data_ptr(), batch, 1e-2),
                      lambda: m.forward(x.data_ptr(), batch, y.data_ptr())):
                f()
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        got.append([y.cpu().numpy()] + [p for layer in m.get_params() for p in layer if p is not None])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_atmosphere_chain():
    """Moves that extrude several columns in a row: each reads the screen that the one before
    wrote."""
    import torch

    from aob200 import system as S

    got = []
    for wait in (True, False):
        sy = S.ShAoSystem(S.plain16(), 0)
        for _ in range(30):
            sy.atmos.move()
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        got.append([sy.atmos.screen_host(i) for i in range(len(sy.layer_params))])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
