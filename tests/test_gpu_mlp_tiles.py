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
