"""The network's tiled kernels at the edges of their tiles: theta sizes that are not
multiples of the 64- and 128-point windows, dilations beyond a window (three
separate windows per row) and beyond theta itself, a grid large enough for the
128-point tiles, each channel count; against the float64 torch network.

Tolerances: FP32 path: sums of <= 9 * 32 and <= nb nrg ntg terms, as in the
existing gradient test (1e-4 of the norm).  Tensor cores, two layers: the
BF16-rounded float64 network up to FP32 accumulation order (5e-4); their
gradients stay within BF16 rounding of the FP32 path's (2^-8 per operand, a few
layers: 5e-2)."""
import numpy as np
import pytest

from conftest import rel
from dimspers_b200 import learned
pytestmark = pytest.mark.gpu

# nrg, ntg, channels, dilations, batch
FP32 = [(5, 15, 8, (1, 2, 1), 3), (7, 80, 16, (3, 1), 2), (70, 67, 32, (1, 65, 2), 1), (6, 130, 32, (5, 1), 2),
        (9, 7, 8, (8, 1), 2)]
TC = [(70, 208, 32, (1, 3), 8), (9, 80, 16, (2, 1), 1), (140, 272, 32, (130, 1), 1), (68, 144, 8, (64, 1), 2),
      (20, 16, 32, (17, 1), 2)]


def _network(params, x, C, dil, bf16):
    """float64 torch network (periodic index in theta, also beyond one turn); bf16:
    convolution operands rounded to BF16, activations to FP32."""
    import torch
    import torch.nn.functional as F

    def r16(a):
        return a.to(torch.float32).to(torch.bfloat16).to(torch.float64) if bf16 else a

    h = torch.tensor(x, dtype=torch.float64)
    ntg, off = h.shape[-1], 0
    for layer, d in enumerate(dil):
        cin = 4 if layer == 0 else C
        cout = 1 if layer == len(dil) - 1 else C
        W = params[off:off + cout * cin * 9].view(cout, cin, 3, 3)
        b = params[off + cout * cin * 9:off + cout * cin * 9 + cout]
        off += cout * cin * 9 + cout
        hp = F.pad(r16(h)[..., torch.arange(-d, ntg + d) % ntg], (0, 0, d, d))
        h = F.conv2d(hp, r16(W), b, dilation=d)
        h = h.to(torch.float32).to(torch.float64) if bf16 else h
        h = torch.relu(h) if layer < len(dil) - 1 else h
    return h


def _data(nrg, ntg, nb):
    import torch
    rng = np.random.default_rng(7)
    x = rng.standard_normal((nb, 4, nrg, ntg)).astype(np.float32)
    t = rng.standard_normal((nb, 1, nrg, ntg)).astype(np.float32)
    return x, t, torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()


@pytest.mark.parametrize("nrg,ntg,C,dil,nb", FP32)
def test_weight_gradient_tiles(nrg, ntg, C, dil, nb):
    net = learned.GuessNet(nrg, ntg, C, len(dil), dil, max_batch=nb)
    net.set_math(bf16=False)
    net.init_params(seed=1)
    x, t, xd, td = _data(nrg, ntg, nb)
    loss = net.gradients(xd, td)
    params, grads = net.get_params(grads=True)
    import torch
    p = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    loss_ref = ((_network(p, x, C, dil, False) - torch.tensor(t, dtype=torch.float64)) ** 2).mean()
    loss_ref.backward()
    assert abs(loss - float(loss_ref)) < 1e-5 * abs(float(loss_ref))
    assert rel(grads, p.grad.numpy()) < 1e-4
    net.close()


@pytest.mark.parametrize("nrg,ntg,C,dil,nb", TC)
def test_tensor_core_tiles(nrg, ntg, C, dil, nb):
    import torch
    net = learned.GuessNet(nrg, ntg, C, len(dil), dil, max_batch=nb)
    net.init_params(seed=2)
    x, t, xd, td = _data(nrg, ntg, nb)
    # an output that is not 16-byte aligned
    buf = torch.empty(nb * nrg * ntg + 1, dtype=torch.float32, device="cuda")
    y = buf[1:].view(nb, 1, nrg, ntg)
    net.forward(xd, y)
    ref = _network(torch.tensor(net.get_params(), dtype=torch.float64), x, C, dil, True)
    assert rel(y.cpu().numpy(), ref.numpy()) < 5e-4
    net.gradients(xd, td)
    g_tc = net.get_params(grads=True)[1]
    net.set_math(bf16=False)
    net.gradients(xd, td)
    assert rel(g_tc, net.get_params(grads=True)[1]) < 5e-2
    net.close()
