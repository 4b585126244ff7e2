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


def _conv64(x, w, b, d):
    xd = torch.nn.functional.pad(x.double(), (0, 0, d, d, d, d, d, d))
    _, D, H, W, _ = x.shape
    out, mag = 0, 0
    for k in range(27):
        z, y, v = d * (k // 9), d * (k // 3 % 3), d * (k % 3)
        s = xd[:, z:z + D, y:y + H, v:v + W]
        out = out + s @ w[k].double().T
        mag = mag + s.abs() @ w[k].double().abs().T
    return out + b.double(), mag + b.double().abs()


@pytest.mark.parametrize("shape,dil", [
    ((1, 5, 4, 64), 1), ((2, 3, 9, 64), 8),    # two lines a tile, an odd last group
    ((1, 7, 3, 40), 2), ((1, 4, 3, 43), 4),    # three and two lines, not a multiple of eight voxels
    ((1, 130, 2, 1), 1), ((1, 40, 2, 3), 8),   # many lines; neighbours always outside the row
    ((2, 1, 5, 64), 1),                        # one line: the tile with a halo
    ((1, 2, 3, 65), 1), ((1, 3, 2, 128), 8), ((1, 2, 4, 129), 3),
    ((1, 3, 5, 70), 8),                        # fewer rows than the dilation
    ((1, 40, 90, 300), 1), ((3, 33, 70, 64), 2),  # whole columns and a split rest, rings that wrap
], ids=str)
def test_convolution_tiles(shape, dil, cuda):
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + dil)
    x, res = _bf((*shape, 16), g), _bf((*shape, 16), g)
    w, b = _bf((27, 16, 16), g, 0.1), torch.randn(16, generator=g, device="cuda")
    x[:, -1, -1, -1] = 1e4  # a stray neighbour would be seen
    st = torch.cuda.current_stream().cuda_stream
    exp, mag = _conv64(x, w, b, dil)
    tol = 16 * 2.0 ** -24 * np.sqrt(432)
    for shift in (0, 4):  # outputs at 32-byte boundaries and 16 bytes past them
        y = torch.empty(x.numel() + 8, device="cuda")[shift:shift + x.numel()].view(x.shape)
        nat.call("si_nn_conv16_tc", x.data_ptr(), w.data_ptr(), b.data_ptr(), None, y.data_ptr(), *shape, dil, 0, 1, st)
        assert float(((y.double() - exp).abs() / mag).max()) < tol
        r = torch.empty(x.numel() + 16, dtype=torch.bfloat16, device="cuda")[2 * shift:2 * shift + x.numel()].view(x.shape)
        nat.call("si_nn_conv16_tc", x.data_ptr(), w.data_ptr(), b.data_ptr(), res.data_ptr(), r.data_ptr(), *shape, dil,
                 1, 0, st)
        assert torch.equal(r, torch.relu(y + res.float()).to(torch.bfloat16))
    S.umma_check()


def test_convolution_infinite_neighbours(cuda):
    """An infinity at the end of a line reaches its own line only."""
    shape = (1, 4, 3, 64)
    x = torch.zeros((*shape, 16), dtype=torch.bfloat16, device="cuda")
    x[0, 1, 1, -1] = float("inf")
    w = torch.ones((27, 16, 16), dtype=torch.bfloat16, device="cuda")
    y = torch.empty((*shape, 16), device="cuda")
    nat.call("si_nn_conv16_tc", x.data_ptr(), w.data_ptr(), None, None, y.data_ptr(), *shape, 1, 0, 1,
             torch.cuda.current_stream().cuda_stream)
    exp = torch.zeros_like(y)
    exp[0, :3, :, -2:] = float("inf")
    assert torch.equal(y, exp)


@pytest.mark.parametrize("shape", [(1, 19, 64, 64), (1, 8, 152, 1), (1, 1, 1, 1), (2, 30, 50, 70)], ids=str)
def test_weight_gradient_stays_in_its_buffer(shape, cuda):
    import ctypes
    g = torch.Generator(device="cuda").manual_seed(1)
    x, dy = _bf((*shape, 16), g), _bf((*shape, 16), g)
    need = ctypes.c_uint64(0)
    nat.call("si_nn_wgrad_partial_bytes", *shape, 16, 16, ctypes.byref(need))
    guard = 1 << 18
    buf = torch.full(((need.value + guard) // 4,), 7.0, device="cuda")
    dw, db = torch.zeros(27 * 256, device="cuda"), torch.zeros(16, device="cuda")
    nat.call("si_nn_conv3d_wgrad", x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(), *shape, 16, 16, 1,
             buf.data_ptr(), need.value, torch.cuda.current_stream().cuda_stream)
    assert bool((buf[need.value // 4:] == 7.0).all())
    w, wm, b, bm = _wgrad64(x, dy, 1)
    assert float(((dw.double().view(27, 16, 16) - w).abs() / (wm + 1)).max()) < 1e-5


@pytest.mark.parametrize("shape,dil", [((2, 5, 4, 64), 1), ((1, 3, 9, 130), 2), ((1, 4, 5, 40), 8)], ids=str)
@pytest.mark.parametrize("with_residual", [False, True])
def test_masked_data_gradient(shape, dil, with_residual, cuda):
    """Equal to the convolution and the ReLU mask after it, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    dy, res, act = (_bf((*shape, 16), g) for _ in range(3))
    act = torch.relu(act)
    act[..., 3] = float("nan")
    act[..., 4] = -0.0
    net = S.SurrogateNet(dilations=(1,))
    conv = net.convs[1]
    conv.dil = dil
    kw = dict(residual=res if with_residual else None)
    for tc in (True, False):
        got = S.conv_dgrad(dy, conv, shape, tensor_core=tc, mask=act, **kw)
        exp = S.conv_dgrad(dy, conv, shape, tensor_core=tc, **kw)
        S.relu_bwd(exp, act)
        assert torch.equal(got, exp) and bool((got[..., 3:5] == 0).all()) and bool((got != 0).any())
    S.umma_check()
