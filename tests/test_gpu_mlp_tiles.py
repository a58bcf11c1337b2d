"""The tcgen05 products at the edges of their tiles, against the float64 oracle with
bfloat16 storage (tolerances as in test_gpu_mlp.py): fewer rows than one CTA of a
pair holds, one more than a pair's 256, widths around 64 and 256, K below one stage
and above the ring of stages, more tiles than pairs of SMs (each pair takes several,
with its two accumulators in turn), one sample; and the training step's gradients
and Adam update through train_step."""

import numpy as np
import pytest

from helpers import rel_rms
from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _skip_gradient(nin, nout, batch, seed):
    """The skip path's weight and the output bias's gradients of a network of zeros, with the
    same from float64 sums: its output is zero, so the bfloat16 operands of the
    product over the batch are known exactly."""
    import torch

    from aob200 import _lib, mlp

    def bf16(a):
        return torch.from_numpy(a).to(torch.bfloat16).double().numpy()

    net = mlp.MlpReconstructor(nin, nout, 16, 8)
    net.set_params([(np.zeros((16, nin)), np.zeros(16)), (np.zeros((8, 16)), np.zeros(8)),
                    (np.zeros((nout, 8)), np.zeros(nout)), (np.zeros((nout, nin)), None)])
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.5, 1.5, (batch, nin)).astype(np.float32)
    t = rng.uniform(0.5, 1.5, (batch, nout)).astype(np.float32)
    dx, dt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    net.forward(dx.data_ptr(), batch)
    net.backward(dt.data_ptr(), batch)
    torch.cuda.synchronize()
    assert net.gemm_status() == 0
    dy = bf16(np.float32(2) / (np.float32(batch) * np.float32(nout)) * -t)
    pin, _, _, pout = net.padded_dims()
    got = [_lib.d2h(*net.buffer(k), np.float32).astype(np.float64) for k in ("dWs", "db3")]
    return (got[0].reshape(pout, pin)[:nout, :nin], dy.T @ bf16(x)), (got[1][:nout], dy.sum(0))


@pytest.mark.parametrize("nin,nout,batch", [(40, 24, 511), (264, 300, 513), (520, 130, 1024), (264, 300, 4096),
                                            (40, 24, 20001), (8, 8, 4194369)])
def test_gradients_over_a_long_batch(nin, nout, batch):
    """A weight gradient sums the batch in slices of 512 samples.  A slice is 32 additions to
    an FP32 accumulator, each off by 2^-23 of the partial sum at most (half the slice's sum
    on average): 1.9e-6; the slices' own additions, rounded to nearest, add 2^-24 of half the sum
    each, with either sign.  In one run over the batch 4096 samples would be 256 additions.
    The bias gradients add their rows' 32 (or 64) at a time, then those sums in eight lanes.  The
    largest batch has more chunks of rows than a grid's second dimension holds."""
    (dw, want), (db, wantb) = _skip_gradient(nin, nout, batch, batch)
    slices = -(-batch // 512)
    assert np.abs(dw / want - 1).max() < 32 * 2.0**-24 + np.sqrt(slices) * 2.0**-23 + 2.0**-23
    assert np.abs(db / wantb - 1).max() < 64 * 2.0**-25 + np.sqrt(slices) * 2.0**-24


@pytest.mark.parametrize("dims,batch", [
    ((24, 16, 8, 9), 1), ((72, 65, 257, 64), 129), ((400, 264, 56, 520), 257), ((65, 1032, 513, 255), 640),
    ((328, 300, 200, 1000), 5000),
])
def test_products_at_tile_edges(dims, batch):
    import torch

    from aob200 import _lib, mlp

    nin, nh1, nh2, nout = dims
    net = mlp.MlpReconstructor(nin, nout, nh1, nh2, seed=3)
    rng = np.random.default_rng(batch)
    params = [(w, rng.standard_normal(w.shape[0]).astype(np.float32) * 0.1) for w, _ in net.get_params()[:3]]
    params.append((rng.standard_normal((nout, nin)).astype(np.float32) * 0.05, None))
    net.set_params(params)
    net.set_scales(0.5, 2.0)
    x = rng.standard_normal((batch, nin)).astype(np.float32)
    t = rng.standard_normal((batch, nout)).astype(np.float32)
    # (an odd element offset: rows that do not start on 16 bytes)
    buf = torch.zeros(batch * nin + 1, device="cuda")
    buf[1:] = torch.from_numpy(x.ravel()).cuda()
    dt = torch.from_numpy(t).cuda()
    dy = torch.zeros((batch, nout), device="cuda")
    loss = torch.zeros(1, device="cuda")
    net.forward(buf.data_ptr() + 4, batch, dy.data_ptr())
    torch.cuda.synchronize()
    y_ref, _ = omlp.forward(params, x, 0.5)
    assert rel_rms(dy.cpu().numpy(), 2.0 * y_ref) < 5e-3
    lr = 1e-3
    net.train_step(buf.data_ptr() + 4, dt.data_ptr(), batch, lr, loss.data_ptr())
    torch.cuda.synchronize()
    assert net.gemm_status() == 0
    loss_ref, g = omlp.backward(params, x, t, 0.5, 2.0)
    assert abs(float(loss.item()) / loss_ref - 1) < 5e-3
    pin, ph1, ph2, pout = net.padded_dims()
    shapes = {"1": (ph1, pin), "2": (ph2, ph1), "3": (pout, ph2), "s": (pout, pin)}
    real = {"1": (nh1, nin), "2": (nh2, nh1), "3": (nout, nh2), "s": (nout, nin)}
    new = net.get_params()
    for i, k in enumerate("123s"):
        ptr, n = net.buffer("dW" + k)
        full = _lib.d2h(ptr, n, np.float32).reshape(shapes[k])
        got = full[: real[k][0], : real[k][1]]
        assert rel_rms(got, g["dW" + k]) < 3e-2, k
        assert not full[real[k][0]:].any() and not full[:, real[k][1]:].any()
        # Adam's first step from the gradients the device holds
        got64 = got.astype(np.float64)
        want = params[i][0] - lr * got64 / (np.abs(got64) + 1e-8)
        assert np.abs(new[i][0] - want).max() < 1e-5 * lr + 2e-7 * np.abs(want).max() + 1e-3 * lr
        if k != "s":
            ptr, n = net.buffer("db" + k)
            assert rel_rms(_lib.d2h(ptr, n, np.float32)[: real[k][0]], g["db" + k]) < 3e-2, k
