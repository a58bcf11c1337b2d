"""What is timed when this framework's speed is judged: its control loops, sensors,
calibration and learned reconstructor, each through its public entry points.

A case is a dict of plain values; ``kind`` names the path:

* ``rtc``      one real-time iteration through ``core.Loop.step`` (sensor image with fused
               centroids, command matrix, integrator, voltages) on a device-resident phase
* ``calls``    the same iteration as separate calls, the order in which a supervisor script drives
               the drop-in objects: comp_image, get_cog, comp_com, comp_voltage
* ``camera``   a real-time controller fed by a uint16 camera frame: pixel calibration, centroids,
               the generic controller with pseudo-open-loop slopes, voltages
* ``learned``  one iteration with the learned reconstructor (``core.Loop.step_mlp``)
* ``closed``   one iteration of the closed-loop simulator (``system.ShAoSystem.next``): layers,
               raytracing, the real-time step, DM shape, target PSF
* ``imat``     the push-pull interaction matrix of a whole DM (calibration)
* ``pyr``      the pyramid sensor's image, its slopes and the command matrix
* ``batch``    Monte Carlo: many loops of uneven size advanced by one call
* ``train``    one training step of the learned reconstructor (forward, backward, Adam)
* ``forward``  batched inference of the learned reconstructor

Sizes are those of the named workloads (``aob200.workloads``, ``aob200.system``, the
benchmark's pyramid and learned rows) and of the tests; ``draw`` spreads over their ranges.
Screens, frames and samples are seeded; matrices and geometry are what a program keeps.
"""

import functools
import os
import sys

import numpy as np
import torch

for _p in (os.getcwd(), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))):
    _pkg = os.path.join(_p, "compass-saxoplus_b200")
    if os.path.isdir(_pkg):
        sys.path.insert(0, _pkg)
        break

from aob200 import core, dm_geometry, mlp, optics, system  # noqa: E402
from aob200 import geometry as G  # noqa: E402
from aob200 import workloads as W  # noqa: E402
from aob200._lib import call  # noqa: E402

DIAM, COBS, LAM = 8.0, 0.14, 0.7


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest loop: 16 x 16, plain CoG, no noise; its time is latency and launches
        dict(name="rtc_plain16", kind="rtc", nxsub=16, npix=8, pd=8, pixsize=0.3, nactu=241, centroider="cog",
             prec="f32", noise=False, delay=0.0),
        # the headline loop: 40 x 40, photon and readout noise, weighted CoG, FP32 command matrix
        dict(name="rtc_saxo40", kind="rtc", nxsub=40, npix=6, pd=6, pixsize=0.36, nactu=1377, centroider="wcog",
             prec="f32", noise=True, delay=0.0),
        # the same sensor driven call by call, as the drop-in modules are, with the BF16 matrix
        dict(name="calls_saxo40_bf16", kind="calls", nxsub=40, npix=6, pd=6, pixsize=0.36, nactu=1377,
             centroider="tcog", prec="bf16", noise=False, delay=1.0),
        # a real bench: frames of a 240 x 240 pixel camera, pseudo-open-loop control
        dict(name="camera_saxo40", kind="camera", nxsub=40, npix=6, nactu=1377, centroider="wcog"),
        # the learned reconstructor in the 40 x 40 loop
        dict(name="learned_saxo40", kind="learned", nxsub=40, npix=6, pd=6, pixsize=0.36, nactu=1377, hidden=1024,
             centroider="wcog", noise=False),
        # a simulated closed-loop iteration with the long-exposure PSF of the target
        dict(name="closed_saxo40", kind="closed", nxsub=40, npix=6, pixsize=0.36, pupdiam=240, nact=41, layers=3,
             centroider="wcog", noise=True),
        # calibration of the 41 x 41 DM on the 40 x 40 sensor
        dict(name="imat_saxo40", kind="imat", nxsub=40, npix=6, pixsize=0.36, pupdiam=240, nact=41, centroider="wcog"),
        # a small pyramid (the tests' size) with photon and readout noise
        dict(name="pyr16", kind="pyr", nxsub=16, pd=4, npts=8, nactu=200, method=1, noise=True),
        # the pyramid of the benchmark: 24 modulation points, 512 x 512 transforms
        dict(name="pyr50", kind="pyr", nxsub=50, pd=2, npts=24, nactu=1600, method=1, noise=False),
        # Monte Carlo campaign: 32 loops of 24 .. 40 sub-apertures across, BF16 matrices
        dict(name="batch_mc32", kind="batch", count=32, lo=24, hi=40, prec="bf16", mix=0),
        # training the learned reconstructor at its benchmark batch
        dict(name="train_b4096", kind="train", nin=2496, hidden=1024, nout=1377, batch=4096),
        # reconstructing a block of recorded slopes
        dict(name="forward_b1000", kind="forward", nin=2496, hidden=1024, nout=1352, batch=1000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["rtc", "rtc", "calls", "camera", "learned", "closed", "imat", "pyr", "pyr", "batch", "train",
                       "forward"])
    nx = rng.randint(8, 40)
    sh = dict(kind=kind, nxsub=nx, npix=rng.choice([4, 5, 6, 8]), pd=rng.choice([4, 5, 6, 8]),
              pixsize=rng.choice([0.3, 0.36]), nactu=int(round(1377 * ((nx + 1) / 41.0) ** 2)) - rng.randint(0, 9),
              centroider=rng.choice(["cog", "tcog", "wcog"]))
    if kind in ("rtc", "calls"):
        return dict(sh, prec=rng.choice(["f32", "f32", "bf16", "fp8"]), noise=rng.random() < 0.5,
                    delay=float(rng.choice([0, 0, 1, 2])))
    if kind == "camera":
        return {k: sh[k] for k in ("kind", "nxsub", "npix", "nactu", "centroider")}
    if kind == "learned":
        return dict(sh, hidden=_log_int(rng, 64, 1024), noise=rng.random() < 0.3)
    if kind in ("closed", "imat"):
        c = dict(kind=kind, nxsub=nx, npix=sh["npix"], pixsize=sh["pixsize"], pupdiam=nx * rng.choice([4, 6]),
                 nact=nx + 1, centroider=sh["centroider"])
        return dict(c, layers=rng.randint(1, 4), noise=rng.random() < 0.5) if kind == "closed" else c
    if kind == "pyr":
        pd = rng.choice([2, 4])
        return dict(kind=kind, nxsub=rng.randint(10, 50 if pd == 2 else 40), pd=pd, npts=rng.randint(4, 24),
                    nactu=rng.randint(50, 1600), method=rng.randint(0, 3), noise=rng.random() < 0.5)
    if kind == "batch":
        lo = rng.randint(10, 32)
        return dict(kind=kind, count=_log_int(rng, 2, 32), lo=lo, hi=min(40, lo + rng.randint(0, 16)),
                    prec=rng.choice(["f32", "bf16", "fp8"]), mix=rng.randint(1, 1 << 20))
    return dict(kind=kind, nin=rng.randint(200, 2600), hidden=_log_int(rng, 64, 1024), nout=rng.randint(100, 1600),
                batch=_log_int(rng, 32, 4096))


# ------------------------------------------------------------------ geometry and inputs
@functools.lru_cache(maxsize=None)
def _setup(nxsub, npix, pd, pixsize, nactu, centroider):
    """Geometry, command matrix and centroider settings of one SH loop (the plan a program keeps)."""
    p = G.ShParams(nxsub=nxsub, npix=npix, pixsize=pixsize, wavelength_um=LAM, fracsub=0.5, gsmag=8.0, noise=0.5)
    g = G.sh_geometry(p, pd * nxsub, diam=DIAM, cobs=COBS, ittime=0.001)
    return W.ShLoopSetup(f"sh{nxsub}", g, _cmat(nactu, 2 * g.nvalid), 0.02 * g.nphotons / npix**2, _wcog_map(npix), 0.5,
                         centroider)


@functools.lru_cache(maxsize=4)
def _cmat(nactu, nslope):
    rng = np.random.default_rng(nactu)
    return (rng.standard_normal((nactu, nslope), dtype=np.float32) / np.float32(np.sqrt(nslope))).astype(np.float32)


def _wcog_map(npix):
    x = np.arange(npix) - (npix - 1) / 2.0
    return np.exp(-(x[:, None] ** 2 + x[None, :] ** 2) / (2 * (npix / 2.35) ** 2)).astype(np.float32)


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + salt)


def _screen(n, rms, seed, salt=0):
    """A von Karman-like phase screen of the given rms (micron), n x n float32 on the GPU."""
    m = 2 * n
    f = torch.fft.fftfreq(m, device="cuda", dtype=torch.float32)
    psd = (f[:, None] ** 2 + f[None, :] ** 2 + (0.3 / n) ** 2) ** (-11.0 / 6.0)
    psd[0, 0] = 0.0
    z = torch.randn(2, m, m, device="cuda", generator=_gen(seed, salt))
    s = torch.fft.ifft2(torch.complex(z[0], z[1]) * psd.sqrt()).real[:n, :n]
    return (s - s.mean()) * (rms / s.std())


def _view(buf):
    """A device buffer of the library as a flat torch tensor (no copy)."""
    flat = core.DeviceArray(buf.ptr, buf.n, buf.dtype, (buf.n,), buf)
    return torch.as_tensor(flat, device="cuda")


def _vec(n, scale, seed, salt=1):
    return (torch.randn(n, device="cuda", generator=_gen(seed, salt)) * scale).cpu().numpy()


RESIDUAL_UM = 0.1  # rms of a closed loop's residual phase


def _sh_setup_of(c):
    return _setup(c["nxsub"], c["npix"], c["pd"], c["pixsize"], c["nactu"], c["centroider"])


def _sh_state(c, seed):
    s = _sh_setup_of(c)
    wfs, cen, ls, loop = W.build_sh_loop(s, precision=c.get("prec", "f32"))
    if c.get("delay"):
        ls.set_delay(c["delay"])
    _view(wfs.d_phase).copy_(_screen(wfs.npup, RESIDUAL_UM, seed).reshape(-1))
    ls.set_com(_vec(s.nactu, 0.1, seed))
    out = {"binimg": _view(wfs.d_binimg), "intensities": _view(wfs.d_intensities),
           "slopes": _view(ls.buffer("centroids")), "err": _view(ls.buffer("err")),
           "voltage": _view(ls.buffer("voltage"))}
    return dict(wfs=wfs, cen=cen, ls=ls, loop=loop, noise=bool(c["noise"]), out=out,
                slopes=ls.buffer("centroids").ptr)


# ------------------------------------------------------------------ float64 restatements
def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").double()


def _sh_images64(g, fields):
    """Normalised sub-aperture images [n, nvalid, npix^2] and raw sums of n phase screens
    [n, npup, npup] (row = y)."""
    pd, nfft = g.pdiam, g.nfft
    ar = torch.arange(pd, device="cuda")
    ix = torch.as_tensor(g.validpuppixx.astype(np.int64), device="cuda")[:, None, None] + ar[None, None, :]
    iy = torch.as_tensor(g.validpuppixy.astype(np.int64), device="cuda")[:, None, None] + ar[None, :, None]
    pup = _f64(np.asarray(g.tel.mpupil, np.float32).T)[iy, ix]
    ph = fields[:, iy, ix] * float(np.float32(2 * np.pi / g.wavelength_um)) - _f64(g.halfxy.T)
    e = torch.polar(pup.expand_as(ph).contiguous(), ph)
    n, nv = e.shape[0], e.shape[1]
    f = torch.exp(-2j * np.pi / nfft * (torch.arange(nfft, device="cuda").double()[:, None] * ar.double()[None, :]))
    hr = (f @ e @ f.T).abs().square().reshape(n, nv, nfft * nfft)
    bm = torch.as_tensor(g.binmap.astype(np.int64), device="cuda")
    if g.ntot != g.nfft:
        inv = torch.full((g.ntot * g.ntot,), -1, dtype=torch.int64, device="cuda")
        hm = torch.as_tensor(np.asarray(g.hrmap).ravel().astype(np.int64), device="cuda")
        inv[hm] = torch.arange(nfft * nfft, device="cuda")
        bm = inv[bm]
    sums = torch.zeros(n, nv, bm.shape[1], dtype=torch.float64, device="cuda")
    for r in range(bm.shape[0]):
        ok = (bm[r] >= 0).double()
        sums += hr[:, :, bm[r].clamp(min=0)] * ok
    tot = sums.sum(-1)
    flux = _f64(g.fluxPerSub) * float(np.float32(g.nphotons))
    return torch.where(tot[..., None] != 0, sums * (flux / tot)[..., None], sums), tot


def _cog64(cube, npix, kind, threshold, weights, scale, offset):
    """CoG-family slopes (x block, then y block) and intensities of images [..., nvalid, npix^2]."""
    d = cube
    if kind in ("tcog", "wcog"):
        t = float(np.float32(threshold))
        d = torch.where(d > t, d - t, torch.full_like(d, 1e-6))
    if kind == "wcog":
        d = d * _f64(weights.ravel(order="F"))
    x = torch.arange(npix, device="cuda").double()
    s = d.sum(-1)
    xs = (d * x.repeat(npix)).sum(-1) / (s + 1e-6)
    ys = (d * x.repeat_interleave(npix)).sum(-1) / (s + 1e-6)
    scale = float(np.float32(scale))
    return torch.cat([(xs - offset) * scale, (ys - offset) * scale], -1), s


def _image64(g, cube):
    size = g.npix * g.nxsub
    p = np.arange(g.npix**2)
    at = (g.validsubsx[:, None] + p % g.npix) + (g.validsubsy[:, None] + p // g.npix) * size
    img = torch.zeros(size * size, dtype=torch.float64, device="cuda")
    img[torch.as_tensor(at.astype(np.int64).ravel(), device="cuda")] = cube.reshape(-1)
    return img


def _com64(cmat, slopes, com0, gain):
    err = -(_f64(cmat) @ slopes)
    return err, _f64(com0) + float(np.float32(gain)) * err


def _sh_exact(c, seed):
    s = _sh_setup_of(c)
    g = s.geom
    ph = _screen(g.tel.n, RESIDUAL_UM, seed).double()
    cube, tot = _sh_images64(g, ph[None])
    if c["noise"]:  # the draws are the framework's own sampler's: only the sums before them have a value
        return {"binimg": None, "intensities": tot[0], "slopes": None, "err": None, "voltage": None}
    slopes, _ = _cog64(cube[0], g.npix, s.centroider, s.threshold, s.weights, g.pixsize, g.npix / 2 - 0.5)
    err, com = _com64(s.cmat, slopes, _vec(s.nactu, 0.1, seed), 0.4)
    if c.get("delay"):  # the voltages are those of earlier commands: zero on the first pass
        com = torch.zeros_like(com)
    img = cube[0]
    if c["kind"] == "calls" and s.centroider == "tcog":  # get_cog stores the thresholded pixels
        t = float(np.float32(s.threshold))
        img = torch.where(img > t, img - t, torch.full_like(img, 1e-6))
    return {"binimg": _image64(g, img), "intensities": tot[0], "slopes": slopes, "err": err, "voltage": com}


def _sh_work(c, matrix_bytes, matrix_flops):
    g = _sh_setup_of(c).geom
    used = g.nrebin * g.npix
    dft = 8 * g.nvalid * (g.pdiam**2 * used + g.pdiam * used**2)
    return {"bytes": 8 * g.nvalid * g.pdiam**2 + 8 * g.nvalid * g.npix**2 + 32 * g.nvalid + 20 * c["nactu"] + matrix_bytes,
            "flops": dft + matrix_flops}


# ------------------------------------------------------------------ rtc, calls
_PREC_BYTES = {"f32": 4, "bf16": 2, "fp8": 1}


def _run_rtc(st):
    st["loop"].step(None, None, st["noise"])
    return st["out"]


def _run_calls(st):
    st["wfs"].comp_image(st["noise"])
    st["cen"].get_cog(st["slopes"])
    st["ls"].comp_com()
    st["ls"].comp_voltage()
    return st["out"]


def _work_rtc(c):
    ns = 2 * _sh_setup_of(c).geom.nvalid
    return _sh_work(c, c["nactu"] * ns * _PREC_BYTES[c["prec"]], 2 * c["nactu"] * ns)


def _tol_sh(c):
    if c["noise"]:
        # a change of rounding moves a pixel's mean across a step of its Poisson draw now and then: one photon
        return {"rel": 2e-3, "max": 0.2}
    return {"rel": 2e-5, "max": 4e-4}


# ------------------------------------------------------------------ camera
@functools.lru_cache(maxsize=None)
def _camera_plan(nxsub, npix, nactu):
    g = _setup(nxsub, npix, 6, 0.36, nactu, "wcog").geom
    rng = np.random.default_rng(7)
    size = nxsub * npix
    dark = rng.uniform(20, 30, (size, size)).astype(np.float32)
    flat = rng.uniform(0.9, 1.1, (size, size)).astype(np.float32)
    imat = (rng.standard_normal((2 * g.nvalid, nactu), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    return g, size, dark, flat, imat


def _frame(g, size, seed):
    """Spots of about 2000 counts over a background of 25, moved by up to a pixel, with photon noise."""
    npix = g.npix
    r = _gen(seed, 3)
    nv = g.nvalid
    cx = npix / 2 - 0.5 + torch.randn(nv, 1, device="cuda", generator=r) * 0.4
    cy = npix / 2 - 0.5 + torch.randn(nv, 1, device="cuda", generator=r) * 0.4
    p = torch.arange(npix * npix, device="cuda")
    spot = torch.exp(-((p % npix - cx) ** 2 + (p // npix - cy) ** 2) / (2 * 0.8**2)) * 500
    img = torch.full((size * size,), 25.0, device="cuda")
    at = (g.validsubsx[:, None] + np.arange(npix**2) % npix) + (g.validsubsy[:, None] + np.arange(npix**2) // npix) * size
    img[torch.as_tensor(at.astype(np.int64).ravel(), device="cuda")] += spot.reshape(-1)
    img = img + torch.randn(size * size, device="cuda", generator=r) * img.sqrt()
    return img.clamp(0, 65535).round().to(torch.int32)


def _camera_state(c, seed):
    g, size, dark, flat, imat = _camera_plan(c["nxsub"], c["npix"], c["nactu"])
    cen = core.Centroider(g.nvalid, g.npix / 2 - 0.5, g.pixsize, c["centroider"])
    cen.set_npix(g.npix)
    cen.load_validpos(g.validsubsx, g.validsubsy)
    if c["centroider"] != "cog":
        cen.set_threshold(10.0)
    if c["centroider"] == "wcog":
        cen.load_weights(_wcog_map(g.npix))
    frame = core.OwnedDeviceArray(size * size, np.uint16, (size, size))
    h = _frame(g, size, seed).cpu().numpy().astype(np.uint16)
    frame.set(h)
    cen.load_img(frame)
    cen.set_dark(dark)
    cen.set_flat(flat)
    cen.calibrate_img_validpix()
    ls = core.LsController(2 * g.nvalid, c["nactu"], kind="generic")
    ls.set_cmat(_cmat(c["nactu"], 2 * g.nvalid))
    ls.set_imat(imat)
    ls.set_gain(0.3)
    ls.set_leaky_factor(0.99)
    ls.set_polc(True)
    ls.set_com(_vec(c["nactu"], 0.1, seed))
    ls.comp_voltage()
    out = {"img": _view(cen.buffer("img")), "intensities": _view(cen.buffer("intensities")),
           "slopes": _view(ls.buffer("centroids")), "err": _view(ls.buffer("err")),
           "voltage": _view(ls.buffer("voltage"))}
    return dict(cen=cen, ls=ls, frame=frame, slopes=ls.buffer("centroids").ptr, out=out)


def _run_camera(st):
    cen, ls = st["cen"], st["ls"]
    cen.load_img(st["frame"])
    cen.calibrate_img_validpix()
    cen.get_cog(st["slopes"])
    ls.comp_com()
    ls.comp_voltage()
    return st["out"]


def _exact_camera(c, seed):
    g, size, dark, flat, imat = _camera_plan(c["nxsub"], c["npix"], c["nactu"])
    img = (_frame(g, size, seed).double() - _f64(dark.ravel(order="F"))) * _f64(flat.ravel(order="F"))
    p = np.arange(g.npix**2)
    at = (g.validsubsx[:, None] + p % g.npix) + (g.validsubsy[:, None] + p // g.npix) * size
    cube = img[torch.as_tensor(at.astype(np.int64), device="cuda")]
    slopes, inten = _cog64(cube, g.npix, c["centroider"], 10.0, _wcog_map(g.npix), g.pixsize, g.npix / 2 - 0.5)
    com0 = _f64(_vec(c["nactu"], 0.1, seed))
    err = -(_f64(_cmat(c["nactu"], 2 * g.nvalid)) @ (slopes - _f64(imat) @ com0))
    gain = float(np.float32(0.3))
    com = (1 - gain) * float(np.float32(0.99)) * com0 + gain * err
    if c["centroider"] == "tcog":  # get_cog stores the thresholded pixels
        cube = torch.where(cube > 10.0, cube - 10.0, torch.full_like(cube, 1e-6))
    return {"img": _image64(g, cube), "intensities": inten, "slopes": slopes, "err": err, "voltage": com}


def _work_camera(c):
    g, size, *_ = _camera_plan(c["nxsub"], c["npix"], c["nactu"])
    ns = 2 * g.nvalid
    return {"bytes": 10 * g.nvalid * g.npix**2 + 8 * c["nactu"] * ns + 8 * ns + 20 * c["nactu"],
            "flops": 4 * c["nactu"] * ns + 8 * g.nvalid * g.npix**2}


# ------------------------------------------------------------------ learned reconstructor
@functools.lru_cache(maxsize=2)
def _mlp_params(nin, hidden, nout):
    r = _gen(11, nin + hidden)
    dims = [(hidden, nin, 1.0), (hidden, hidden, 1.0), (nout, hidden, 0.2), (nout, nin, 0.5)]
    out = []
    for i, (o, k, a) in enumerate(dims):
        w = torch.randn(o, k, device="cuda", generator=r) * (a / k**0.5)
        b = torch.randn(o, device="cuda", generator=r) * 0.02
        out.append((w.cpu().numpy(), b.cpu().numpy() if i < 3 else None))
    return out


IN_SCALE, OUT_SCALE = 8.0, 0.2


def _net(nin, hidden, nout):
    net = mlp.MlpReconstructor(nin, nout, hidden, hidden)
    net.set_params(_mlp_params(nin, hidden, nout))
    net.set_scales(IN_SCALE, OUT_SCALE)
    return net


def _mlp64(params, x):
    """Forward pass on scaled inputs; returns the pre-activations, activations and scaled outputs."""
    (w1, b1), (w2, b2), (w3, b3), (ws, _) = [(_f64(w), None if b is None else _f64(b)) for w, b in params]
    z1 = x @ w1.T + b1
    h1 = torch.nn.functional.gelu(z1)
    z2 = h1 @ w2.T + b2
    h2 = torch.nn.functional.gelu(z2)
    return z1, h1, z2, h2, h2 @ w3.T + b3 + x @ ws.T


def _learned_state(c, seed):
    st = _sh_state(dict(c, prec="f32"), seed)
    s = _sh_setup_of(c)
    st["net"] = _net(s.nslope, c["hidden"], c["nactu"])
    return st


def _run_learned(st):
    st["loop"].step_mlp(st["net"], 3e38, None, None, st["noise"])
    return st["out"]


def _exact_learned(c, seed):
    ex = _sh_exact(dict(c, prec="f32"), seed)
    if c["noise"]:
        return ex
    s = _sh_setup_of(c)
    y = _mlp64(_mlp_params(s.nslope, c["hidden"], c["nactu"]), ex["slopes"][None] * IN_SCALE)[4][0]
    err = -y * float(np.float32(OUT_SCALE))
    return dict(ex, err=err, voltage=_f64(_vec(s.nactu, 0.1, seed)) + float(np.float32(0.4)) * err)


def _mlp_params_count(nin, hidden, nout):
    return nin * hidden + hidden * hidden + hidden * nout + nin * nout


def _work_learned(c):
    n = _mlp_params_count(2 * _sh_setup_of(c).geom.nvalid, c["hidden"], c["nactu"])
    return _sh_work(c, 2 * n, 2 * n)


def _tol_learned(c):
    # bfloat16 activations: a last-bit change of a slope flips the rounding of a few of them
    return {"rel": 4e-3, "max": 0.3} if c["noise"] else {"rel": 1e-3, "max": 0.01}


def _samples(c, seed):
    r = _gen(seed, 5)
    x = torch.randn(c["batch"], c["nin"], device="cuda", generator=r) * 0.1
    return x, torch.randn(c["batch"], c["nout"], device="cuda", generator=r) * 0.2


def _train_state(c, seed):
    net = _net(c["nin"], c["hidden"], c["nout"])
    x, t = _samples(c, seed)
    net.forward(x.data_ptr(), c["batch"])  # the workspace of this batch size
    loss = torch.zeros(1, device="cuda")

    def buf(which):
        p, n = net.buffer(which)
        return _view(core.DeviceArray(p, n, np.float32, (n,), net))

    names = [f"{a}{i}" for a in ("dW", "db", "W", "b") for i in (1, 2, 3)] + ["dWs", "Ws"]
    return dict(net=net, x=x, t=t, loss=loss, batch=c["batch"], out=dict({k: buf(k) for k in names}, loss=loss))


def _run_train(st):
    st["net"].train_step(st["x"].data_ptr(), st["t"].data_ptr(), st["batch"], 1e-4, st["loss"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
    return st["out"]


def _pad8(a):
    r = [(-n) % 8 for n in a.shape]
    return torch.nn.functional.pad(a, (0, r[1], 0, r[0]) if a.dim() == 2 else (0, r[0])).reshape(-1)


def _exact_train(c, seed):
    params = _mlp_params(c["nin"], c["hidden"], c["nout"])
    x, t = _samples(c, seed)
    x = x.double() * IN_SCALE
    z1, h1, z2, h2, y = _mlp64(params, x)
    d = y - t.double() / float(np.float32(OUT_SCALE))
    dy = 2 * d / d.numel()

    def dgelu(z):
        return 0.5 * (1 + torch.erf(z / 2**0.5)) + z * torch.exp(-0.5 * z * z) / (2 * np.pi) ** 0.5

    w = [_f64(p[0]) for p in params]
    dz2 = dy @ w[2] * dgelu(z2)
    dz1 = dz2 @ w[1] * dgelu(z1)
    grads = {"dW1": dz1.T @ x, "dW2": dz2.T @ h1, "dW3": dy.T @ h2, "dWs": dy.T @ x, "db1": dz1.sum(0),
             "db2": dz2.sum(0), "db3": dy.sum(0)}
    out = {k: _pad8(v) for k, v in grads.items()}
    for i, k in enumerate(("1", "2", "3", "s")):  # Adam's first step moves a weight by lr g / (|g| + eps)
        out["W" + k] = _pad8(w[i] - 1e-4 * grads["dW" + k] / (grads["dW" + k].abs() + 1e-8))
        if k != "s":
            out["b" + k] = _pad8(_f64(params[i][1]) - 1e-4 * grads["db" + k] / (grads["db" + k].abs() + 1e-8))
    out["loss"] = (d * d).mean().reshape(1)
    return out


def _work_train(c):
    nin, h, nout, b = c["nin"], c["hidden"], c["nout"], c["batch"]
    n = _mlp_params_count(nin, h, nout)
    # x and t read, every parameter and both moments read and written, the gradients written
    return {"bytes": 4 * b * (nin + nout) + 28 * n, "flops": 2 * b * (2 * n + h * h + h * nout)}


def _forward_state(c, seed):
    net = _net(c["nin"], c["hidden"], c["nout"])
    x, _ = _samples(c, seed)
    y = torch.empty(c["batch"], c["nout"], device="cuda")
    net.forward(x.data_ptr(), c["batch"], y.data_ptr())
    return dict(net=net, x=x, y=y, batch=c["batch"])


def _run_forward(st):
    st["net"].forward(st["x"].data_ptr(), st["batch"], st["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return st["y"]


def _exact_forward(c, seed):
    x, _ = _samples(c, seed)
    y = _mlp64(_mlp_params(c["nin"], c["hidden"], c["nout"]), x.double() * IN_SCALE)[4]
    return y * float(np.float32(OUT_SCALE))


def _work_forward(c):
    n = _mlp_params_count(c["nin"], c["hidden"], c["nout"])
    return {"bytes": 4 * c["batch"] * (c["nin"] + c["nout"]) + 2 * n, "flops": 2 * c["batch"] * n}


# ------------------------------------------------------------------ closed loop, interaction matrix
_closed_cmat = {}


def _closed_config(c, seed):
    n = c["layers"]
    return system.AoConfig(nxsub=c["nxsub"], npix=c["npix"], pixsize=c["pixsize"], pupdiam=c["pupdiam"],
                           nact=c["nact"], centroider=c["centroider"], fracs=(0.5, 0.3, 0.2, 0.1)[:n],
                           alts=(0.0,) * n, winds=(8.0, 15.0, 25.0, 40.0)[:n], dirs=(0.0, 45.0, 90.0, 200.0)[:n],
                           seeds=tuple(int(seed) * 16 + i for i in range(n)))


def _closed_state(c, seed):
    s = system.ShAoSystem(_closed_config(c, seed))
    key = tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    if key not in _closed_cmat:
        s.calibrate()
        _closed_cmat[key] = s.cmat
    else:
        s.ls.set_cmat(_closed_cmat[key])
    s.close()
    for _ in range(5):  # the loop is running
        s.next(noise=c["noise"])
    out = {"phase": _view(s.wfs.d_phase), "slopes": _view(s.ls.buffer("centroids")),
           "voltage": _view(s.ls.buffer("voltage")), "shape": _view(s.dm.d_shape),
           "image_se": _view(s.target.d_image_se), "image_le": _view(s.target.d_image_le)}
    return dict(sys=s, noise=bool(c["noise"]), out=out)


def _run_closed(st):
    st["sys"].next(noise=st["noise"])
    return st["out"]


def _work_closed(c):
    n = c["pupdiam"] + 8
    nsl = 1.55 * c["nxsub"] ** 2
    nact = 0.8 * c["nact"] ** 2
    nt = 1 << int(np.ceil(np.log2(2 * c["pupdiam"] - 1)))  # the target's transform
    return {"bytes": int(c["layers"] * 4 * n * (5 * n) + 4 * nact * nsl + 24 * n * n + 12 * nt * nt + 4 * nact * 784),
            "flops": int(10 * nt * nt * np.log2(nt) + 2 * nact * nsl)}


def _tol_closed(c):
    # some layers' noise and the sensor's draws follow the rounding of earlier frames
    return {"rel": 4e-3, "max": 0.3} if c["noise"] else {"rel": 1e-4, "max": 4e-3}


@functools.lru_cache(maxsize=None)
def _imat_plan(nxsub, npix, pixsize, pupdiam, nact):
    p = G.ShParams(nxsub=nxsub, npix=npix, pixsize=pixsize, wavelength_um=LAM, fracsub=0.5, gsmag=8.0, noise=0.5)
    g = G.sh_geometry(p, pupdiam, diam=DIAM, cobs=COBS, ittime=0.001)
    t = g.tel
    return g, dm_geometry.pzt_dm_geometry(nact, t.pupdiam, t.cent, t.ssize, t.n, COBS, coupling=0.3, margin_out=1.0)


def _imat_plan_of(c):
    return _imat_plan(c["nxsub"], c["npix"], c["pixsize"], c["pupdiam"], c["nact"])


def _influence(c, seed):
    """The measured influence functions of one DM: its actuators' gains differ by a few per cent."""
    _, d = _imat_plan_of(c)
    return d.influ * np.float32(1.0 + 0.05 * _vec(d.ntotact, 1.0, seed, 9))


PUSH = 0.05


def _imat_state(c, seed):
    g, d = _imat_plan_of(c)
    wfs = core.ShWfs.from_geometry(g, noise=0.5)
    cen = core.Centroider(g.nvalid, g.npix / 2 - 0.5, g.pixsize, c["centroider"])
    cen.set_npix(g.npix)
    cen.load_validpos(g.validsubsx, g.validsubsy)
    if c["centroider"] != "cog":
        cen.set_threshold(0.02 * g.nphotons / g.npix**2)
    if c["centroider"] == "wcog":
        cen.load_weights(_wcog_map(g.npix))
    cen.attach(wfs)
    dm = optics.Dm(d.dim, _influence(c, seed), d.i1, d.j1)
    imat = core.OwnedDeviceArray(2 * g.nvalid * d.ntotact)
    return dict(wfs=wfs, cen=cen, dm=dm, imat=imat, off=(d.dim - g.tel.n) / 2.0, out=_view(imat))


def _run_imat(st):
    call("aob_imat_build", st["wfs"].h, st["cen"].h, st["dm"].h, st["off"], st["off"], PUSH, 0, st["imat"].ptr, None)
    return st["out"]


def _exact_imat(c, seed):
    g, d = _imat_plan_of(c)
    n, na = g.tel.n, d.ntotact
    infl = _f64(_influence(c, seed).transpose(2, 1, 0))  # actuator, y, x
    off = (d.dim - n) / 2.0
    lo, frac = int(off), off - int(off)
    push = float(np.float32(PUSH))
    thr = 0.02 * g.nphotons / g.npix**2
    out = torch.empty(na, 2 * g.nvalid, dtype=torch.float64, device="cuda")
    isz = d.influsize
    step = max(1, int(3e8 // (g.nvalid * g.nfft**2 * 8)))
    for a0 in range(0, na, step):
        m = min(step, na - a0)
        sh = torch.zeros(m, d.dim + 2 * isz, d.dim + 2 * isz, dtype=torch.float64, device="cuda")
        for k in range(m):
            y, x = int(d.j1[a0 + k]) + isz, int(d.i1[a0 + k]) + isz
            sh[k, y:y + isz, x:x + isz] = infl[a0 + k]
        sh = sh[:, isz:isz + d.dim, isz:isz + d.dim]
        if frac:
            w = sh[:, lo:lo + n + 1, lo:lo + n + 1]
            w = (1 - frac) * w[:, :, :-1] + frac * w[:, :, 1:]
            ph = (1 - frac) * w[:, :-1] + frac * w[:, 1:]
        else:
            ph = sh[:, lo:lo + n, lo:lo + n]
        s = []
        for sign in (push, -push):
            cube, _ = _sh_images64(g, ph * sign)
            s.append(_cog64(cube, g.npix, c["centroider"], thr, _wcog_map(g.npix), g.pixsize, g.npix / 2 - 0.5)[0])
            del cube
        out[a0:a0 + m] = (s[0] - s[1]) / (2 * push)
    return out.reshape(-1)


def _work_imat(c):
    g, d = _imat_plan_of(c)
    used = g.nrebin * g.npix
    # a poke moves the sub-apertures under its influence function only
    under = d.ntotact * (d.influsize / g.pdiam + 1) ** 2
    return {"bytes": 4 * d.ntotact * (d.influsize**2 + 2 * g.nvalid) + 8 * g.tel.n**2,
            "flops": int(2 * under * 8 * (g.pdiam**2 * used + g.pdiam * used**2))}


# ------------------------------------------------------------------ pyramid
@functools.lru_cache(maxsize=None)
def _pyr_geom(nxsub, pd, npts):
    sep = {16: 12, 50: 32}.get(nxsub, int(0.7 * nxsub))
    lam = 1.075 if nxsub == 50 else 0.7
    return G.pyr_geometry(G.PyrParams(nxsub=nxsub, wavelength_um=lam, ampl=3.0, npts=npts, pup_sep=sep, fssize=3.2),
                          nxsub * pd, diam=DIAM, cobs=COBS)


def _pyr_state(c, seed):
    g = _pyr_geom(c["nxsub"], c["pd"], c["npts"])
    w = core.PyrWfs.from_geometry(g, noise=0.3)
    _view(w.d_phase).copy_(_screen(w.ntot, RESIDUAL_UM, seed).reshape(-1))
    cen = core.Centroider(g.nvalid, 0.0, 1.0, "pyr")
    cen.load_validpos(g.validsubsx, g.validsubsy)
    cen.set_pyr_method(c["method"])
    cen.attach(w)
    ls = core.LsController(2 * g.nvalid, c["nactu"])
    ls.set_cmat(_cmat(c["nactu"], 2 * g.nvalid))
    ls.set_gain(0.4)
    ls.set_com(_vec(c["nactu"], 0.1, seed))
    out = {"binimg": _view(w.d_binimg), "slopes": _view(ls.buffer("centroids")), "err": _view(ls.buffer("err")),
           "voltage": _view(ls.buffer("voltage"))}
    return dict(wfs=w, cen=cen, ls=ls, slopes=ls.buffer("centroids").ptr, noise=bool(c["noise"]), out=out)


def _exact_pyr(c, seed):
    if c["noise"]:
        return None
    g = _pyr_geom(c["nxsub"], c["pd"], c["npts"])
    n, nf = g.ntot, g.nfft
    off = (nf - n) // 2
    ph = _screen(n, RESIDUAL_UM, seed).double() * float(np.float32(2 * np.pi / np.float32(g.wavelength_um)))
    xx = torch.arange(n, device="cuda").double() - n / 2.0
    pup = _f64(np.asarray(g.tel.mpupil, np.float32).T)
    mask = torch.polar(_f64(g.submask.T), _f64(g.halfxy))  # the geometry's array is passed on transposed
    hr = torch.zeros(nf, nf, dtype=torch.float64, device="cuda")
    for p in range(g.pyr_cx.size):
        f = torch.zeros(nf, nf, dtype=torch.complex128, device="cuda")
        f[off:off + n, off:off + n] = torch.polar(pup, ph + float(g.pyr_cx[p]) * xx[None, :] + float(g.pyr_cy[p]) * xx[:, None])
        hr += torch.fft.fft2(torch.fft.ifft2(f, norm="forward") * mask).abs().square()
    hr = torch.fft.fft2(torch.fft.ifft2(hr, norm="forward") * _f64(g.sincar.T)).real
    r = g.nrebin
    nb = nf // r
    b = hr.reshape(nb, r, nb, r).sum((1, 3))
    b = b * (float(np.float32(g.nphotons)) / b.sum())
    at = torch.as_tensor((g.validsubsx + g.validsubsy * nb).astype(np.int64), device="cuda")
    q = b.reshape(-1)[at].reshape(4, g.nvalid)
    flux = q.sum(0)
    den = flux if c["method"] > 1 else flux.mean().expand_as(flux)
    s = torch.cat([(q[0] + q[3] - q[1] - q[2]) / den, (q[0] + q[2] - q[1] - q[3]) / den])
    if c["method"] % 2 == 0:
        s = torch.sin(np.pi * s / 2)
    s = torch.where(torch.cat([den, den]) < 1e-4, torch.zeros_like(s), s)
    err, com = _com64(_cmat(c["nactu"], 2 * g.nvalid), s, _vec(c["nactu"], 0.1, seed), 0.4)
    return {"binimg": b.reshape(-1), "slopes": s, "err": err, "voltage": com}


def _work_pyr(c):
    g = _pyr_geom(c["nxsub"], c["pd"], c["npts"])
    nf, nb = g.nfft, g.nfft // g.nrebin
    ns = 2 * g.nvalid
    # per point: the pupil's rows, every column twice, every row; then the pixel transfer's four passes
    lines = c["npts"] * (g.ntot + 3 * nf) + 4 * nf
    return {"bytes": 8 * g.ntot**2 + 16 * nf * nf + 4 * nb * nb + 4 * c["nactu"] * ns,
            "flops": int(5 * lines * nf * np.log2(nf)) + 2 * c["nactu"] * ns}


def _tol_pyr(c):
    return {"rel": 2e-3, "max": 0.2} if c["noise"] else {"rel": 1e-5, "max": 4e-4}


# ------------------------------------------------------------------ batched Monte Carlo
@functools.lru_cache(maxsize=None)
def _mc_list(count, lo, hi, mix):
    rng = np.random.default_rng(mix)
    out = []
    for _ in range(count):
        nx = int(rng.integers(lo, hi + 1))
        out.append((nx, int(rng.choice([6, 8])), 6, 0.36, int(round(1377 * ((nx + 1) / 41.0) ** 2)), "wcog"))
    return out


def _batch_state(c, seed):
    loops, out = [], {}
    for i, key in enumerate(_mc_list(c["count"], c["lo"], c["hi"], c["mix"])):
        wfs, cen, ls, loop = W.build_sh_loop(_setup(*key), precision=c["prec"], seed=1234 + i)
        _view(wfs.d_phase).copy_(_screen(wfs.npup, RESIDUAL_UM, seed, 17 + i).reshape(-1))
        loops.append((wfs, cen, ls, loop))
        out[f"{i:02d}"] = [_view(ls.buffer("voltage")), _view(wfs.d_binimg)]
    batch = core.Batch([l[3] for l in loops])
    batch.step()
    return dict(loops=loops, batch=batch, out=out)


def _run_batch(st):
    st["batch"].step(True)
    return st["out"]


def _work_batch(c):
    total = {"bytes": 0, "flops": 0}
    for nx, npix, pd, _, nact, _ in _mc_list(c["count"], c["lo"], c["hi"], c["mix"]):
        g = _setup(nx, npix, pd, 0.36, nact, "wcog").geom
        used = g.nrebin * npix
        total["bytes"] += nact * 2 * g.nvalid * _PREC_BYTES[c["prec"]] + g.nvalid * (8 * pd * pd + 8 * npix * npix + 32) + 20 * nact
        total["flops"] += 4 * nact * g.nvalid + 8 * g.nvalid * (pd * pd * used + pd * used * used)
    return total


# ------------------------------------------------------------------ the interface
_KINDS = {
    "rtc": (_sh_state, _run_rtc, _work_rtc, _tol_sh, _sh_exact),
    "calls": (_sh_state, _run_calls, _work_rtc, _tol_sh, _sh_exact),
    "camera": (_camera_state, _run_camera, _work_camera, lambda c: {"rel": 4e-6, "max": 1e-4}, _exact_camera),
    "learned": (_learned_state, _run_learned, _work_learned, _tol_learned, _exact_learned),
    "closed": (_closed_state, _run_closed, _work_closed, _tol_closed, lambda c, seed: None),
    "imat": (_imat_state, _run_imat, _work_imat, lambda c: {"rel": 2e-5, "max": 4e-3}, _exact_imat),
    "pyr": (_pyr_state, lambda st: _run_calls(st), _work_pyr, _tol_pyr, _exact_pyr),
    "batch": (_batch_state, _run_batch, _work_batch, lambda c: {"rel": 2e-3, "max": 0.2}, lambda c, seed: None),
    "train": (_train_state, _run_train, _work_train, lambda c: {"rel": 2e-3, "max": 0.02}, _exact_train),
    "forward": (_forward_state, _run_forward, _work_forward, lambda c: {"rel": 1e-3, "max": 0.01}, _exact_forward),
}


def prepare(case, seed):
    st = _KINDS[case["kind"]][0](case, seed)
    st["run"] = _KINDS[case["kind"]][1]
    return st


def run(state):
    return state["run"](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


def tolerance(case):
    return _KINDS[case["kind"]][3](case)


def exact(case, seed):
    return _KINDS[case["kind"]][4](case, seed)
