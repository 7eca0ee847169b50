"""Closure CNN on the tensor cores against the float64 oracle: forward
output and every parameter gradient (BF16 activations through five layers:
relative L2 tolerance 3e-2 on the output, 6e-2 on the gradients), and a
short Adam run that must reduce the loss."""

import numpy as np
import pytest
import torch

from oracle import closure_oracle as CO

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def test_cnn_forward_backward_vs_oracle():
    from pygsquig_b200.build import build

    build()
    from pygsquig_b200.closure.cnn import ClosureCNN

    H, W = 8, 128
    net = ClosureCNN(H=H, W=W, max_batch=2, seed=3)
    rng = np.random.default_rng(4)
    x = rng.standard_normal((2, H, W))
    t = rng.standard_normal((2, H, W)) * 0.1
    xt = torch.as_tensor(x, dtype=torch.float32, device="cuda")
    tt = torch.as_tensor(t, dtype=torch.float32, device="cuda")
    y = net.forward(xt)
    loss = net.mse(y, tt)
    net.backward(xt, net.gy[:2])
    torch.cuda.synchronize()
    assert net.errors() == 0
    p = {k: v.detach().double().cpu().numpy() for k, v in net.p.items()}
    yo, c = CO.forward(p, x)
    go = CO.backward(p, c, 2 * (yo - t) / yo.size)
    assert rel(y.double().cpu().numpy(), yo) < 3e-2
    assert abs(float(loss) - np.mean((yo - t) ** 2)) < 3e-2 * np.mean((yo - t) ** 2)
    for k in p:
        gk = net.g[k].double().cpu().numpy()
        assert rel(gk, go[k]) < 6e-2, (k, rel(gk, go[k]))


def test_cnn_training_reduces_loss():
    from pygsquig_b200.closure.cnn import ClosureCNN

    H, W = 16, 128
    net = ClosureCNN(H=H, W=W, max_batch=2, seed=1)
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(2, H, W, device="cuda", generator=g)
    t = torch.roll(x, 1, dims=2) - x  # a learnable local map
    l0 = float(net.train_step(x, t))
    for _ in range(60):
        l1 = float(net.train_step(x, t))
    assert net.errors() == 0
    assert l1 < 0.3 * l0, (l0, l1)


@pytest.mark.parametrize("off", [2, 4, 6])
def test_gradients_of_tensors_at_any_channel_pair(off):
    """Tensors of the first and last layers' gradients that start past a 16-byte
    boundary give the bits of aligned ones."""
    from pygsquig_b200 import _lib
    from pygsquig_b200.build import build

    build()
    L, B, H, W = _lib.load(), 2, 3, 64
    gen = torch.Generator(device="cuda").manual_seed(2)

    def bf(*shape):
        t = torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)
        s = torch.zeros(t.numel() + 8, dtype=torch.bfloat16, device="cuda")[off : off + t.numel()].view(shape)
        assert t.data_ptr() % 16 == 0 and s.data_ptr() % 16 == 2 * off
        s.copy_(t)
        return t, s

    pad, z = bf(B, H + 2, W + 2, 64), bf(B, H, W, 64)
    gy, x = torch.randn(B, H, W, generator=gen, device="cuda"), torch.randn(B, H, W, generator=gen, device="cuda")
    w6 = torch.randn(9, 64, generator=gen, device="cuda")
    red = torch.empty(296 * 640, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    got = []
    for i in range(2):
        outs = [torch.empty(640, device="cuda") for _ in range(3)]
        for mode, a, gz in ((0, pad[i].data_ptr(), None), (1, None, pad[i].data_ptr()), (2, None, pad[i].data_ptr())):
            assert L.closure_small_grad(mode, B, H, W, gy.data_ptr(), a, x.data_ptr(), gz, red.data_ptr(),
                                        outs[mode].data_ptr(), st) == 0
        g = bf(B, H + 2, W + 2, 64)[i]
        assert L.closure_conv_out_dgrad(B, H, W, gy.data_ptr(), w6.data_ptr(), z[i].data_ptr(), g.data_ptr(), st) == 0
        got.append(outs + [g.contiguous()])
    for a, b in zip(*got):
        assert torch.equal(a, b)
