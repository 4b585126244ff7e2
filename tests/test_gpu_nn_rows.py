"""The row-wise weight gradient, the 16-channel cross entropy and the vectorised
ReLU mask at the edges of their rows, slots and vectors, against float64 sums of
the bf16 inputs; tolerances: fp32 sums of n products, 2^-24 sqrt(n) and a factor
of eight for their order."""
import numpy as np
import pytest
import torch

from biomedisa_gb300 import _native as nat
from biomedisa_gb300 import surrogate as S

pytestmark = pytest.mark.gpu


def _bf(shape, gen, scale=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(torch.bfloat16)


def _wgrad64(x, dy, d):
    """dW[tap][co][ci], db in float64, and the sums of magnitudes behind them."""
    xd, yd = x.double(), dy.double()
    p = torch.nn.functional.pad(xd, (0, 0, d, d, d, d, d, d))
    _, D, H, W, _ = x.shape
    out, mag = [], []
    for k in range(27):
        z, y, v = d * (k // 9), d * (k // 3 % 3), d * (k % 3)
        s = p[:, z:z + D, y:y + H, v:v + W].reshape(-1, 16)
        out.append(yd.reshape(-1, 16).T @ s)
        mag.append(yd.abs().reshape(-1, 16).T @ s.abs())
    return torch.stack(out), torch.stack(mag), yd.reshape(-1, 16).sum(0), yd.abs().reshape(-1, 16).sum(0)


@pytest.mark.parametrize("partials", [True, False], ids=["deterministic", "atomics"])
@pytest.mark.parametrize("shape,dil", [((1, 1, 1, 1), 1), ((2, 3, 4, 63), 1), ((1, 5, 6, 64), 8), ((1, 9, 20, 65), 4),
                                       ((3, 4, 5, 130), 2), ((1, 6, 5, 33), 9), ((1, 20, 40, 70), 1)], ids=str)
def test_weight_gradient_rows(shape, dil, partials, cuda):
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + dil)
    x, dy = _bf((*shape, 16), g), _bf((*shape, 16), g, 0.1)
    net = S.SurrogateNet(dilations=(1,))
    conv = net.convs[1]
    conv.dil = dil
    conv.gw.fill_(1.0)
    conv.gb.fill_(-2.0)
    for _ in range(2):  # gradients add up
        S.conv_wgrad(x, dy, conv, shape, deterministic=partials)
    w, wm, b, bm = _wgrad64(x, dy, dil)
    n = x.numel() // 16
    tol = 8 * 2.0 ** -24 * np.sqrt(n + 4)
    assert float(((conv.gw.double() - 1 - 2 * w).abs() / (2 * wm + 1)).max()) < tol
    assert float(((conv.gb.double() + 2 - 2 * b).abs() / (2 * bm + 2)).max()) < tol


@pytest.mark.parametrize("V", [1, 255, 256, 5000])
@pytest.mark.parametrize("nol", [1, 2, 13, 16])
def test_cross_entropy_16(V, nol, cuda):
    g = torch.Generator(device="cuda").manual_seed(V + nol)
    z = torch.randn((V, 16), generator=g, device="cuda") * 4
    p = torch.softmax(torch.randn((V, nol), generator=g, device="cuda"), -1)
    w = torch.rand(V, generator=g, device="cuda")
    net = S.SurrogateNet(dilations=(1,))
    loss, dl = net.loss_and_grad(z, p, w, nol, denom=V)
    zd, pd, wd = z.double()[:, :nol], p.double(), w.double()
    logq = torch.log_softmax(zd, -1)
    exp = -(pd * logq).sum(-1).mul(wd).sum() / V
    mag = (pd * logq.abs()).sum(-1).mul(wd).sum() / V + 1e-3
    assert abs(float(loss) - float(exp)) / float(mag) < 2e-6  # __expf and __logf of a voxel: about 2^-20
    ed = torch.zeros((V, 16), dtype=torch.float64, device="cuda")
    ed[:, :nol] = wd[:, None] * (logq.exp() - pd) / V
    assert float((dl.double() - ed).abs().max()) <= 2.0 ** -8 * float(ed.abs().max()) + 1e-6 / V
    # logits that start between two 16-byte boundaries take the general kernel
    buf = torch.empty(V * 16 + 1, device="cuda")
    off = buf[1:].view(V, 16)
    off.copy_(z)
    loss2, dl2 = net.loss_and_grad(off, p, w, nol, denom=V)
    assert torch.equal(dl, dl2) and abs(float(loss) - float(loss2)) / float(mag) < 4e-6


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4099])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("with_add", [False, True])
def test_relu_backward(n, shift, with_add, cuda):
    g = torch.Generator(device="cuda").manual_seed(n)
    t = [torch.empty(n + 8, dtype=torch.bfloat16, device="cuda")[shift:shift + n] for _ in range(3)]
    for v in t:
        v.copy_(torch.randn(n, generator=g, device="cuda").to(torch.bfloat16))
    t[1][::3] = 0.0
    exp = torch.where(t[1].float() > 0, t[0].float(), torch.zeros(n, device="cuda"))
    if with_add:
        exp = exp + t[2].float()
    S.relu_bwd(t[0], t[1], t[2] if with_add else None)
    assert torch.equal(t[0], exp.to(torch.bfloat16))
