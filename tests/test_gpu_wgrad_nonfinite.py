"""Infinities and NaN in the 16 x 16 weight and bias gradient: they reach the sums
that they are part of, as infinities and NaN, and no others."""
import pytest
import torch

from biomedisa_gb300 import surrogate as S

pytestmark = pytest.mark.gpu
INF = float("inf")


def _grads(x, dy, dil, partials):
    conv = S.SurrogateNet(dilations=(1,)).convs[1]
    conv.dil = dil
    S.conv_wgrad(x, dy, conv, tuple(x.shape[:4]), deterministic=partials)
    return conv.gw, conv.gb


def _bf(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("partials", [True, False], ids=["deterministic", "atomics"])
@pytest.mark.parametrize("shape", [(1, 8, 400, 64), (2, 9, 40, 70)], ids=str)
def test_infinite_bias_gradient(shape, partials, cuda):
    x, dy = _bf((*shape, 16), 1), _bf((*shape, 16), 2)
    dy[0, 1, 3:9, 5, 2] = INF  # rows that one warp adds up
    dy[0, 1, 2:8, 60, 11] = -INF
    dy[0, 1, 2, 7, 4], dy[0, 1, 3, 9, 4] = INF, -INF
    dy[0, 0, 0, 0, 5] = float("nan")
    _, gb = _grads(x, dy, 1, partials)
    assert gb[2] == INF and gb[11] == -INF and gb[4].isnan() and gb[5].isnan()
    rest = [c for c in range(16) if c not in (2, 4, 5, 11)]
    d = dy.double().reshape(-1, 16)[:, rest]
    # fp32 sums of n terms: 2^-24 sqrt(n) and a factor of eight for their order
    assert bool(((gb.double()[rest] - d.sum(0)).abs() <= 8 * 2.0 ** -24 * len(d) ** 0.5 * d.abs().sum(0)).all())


@pytest.mark.parametrize("partials", [True, False], ids=["deterministic", "atomics"])
@pytest.mark.parametrize("shape,dil", [((1, 3, 5, 70), 1), ((2, 3, 9, 63), 2), ((1, 2, 3, 129), 8),
                                       ((1, 4, 20, 112), 4)], ids=str)
def test_infinite_end_of_a_row(shape, dil, partials, cuda):
    """The tap to the left meets none of a row's last dil voxels: its sums are those
    of a row that ends in zeros, bit for bit (but for the atomics' order)."""
    x, dy = _bf((*shape, 16), 3), _bf((*shape, 16), 4)
    x[..., -dil:, 6] = 0.0
    exp, _ = _grads(x, dy, dil, partials)
    x[..., -dil:, 6] = torch.tensor([INF, -INF, float("nan")], device="cuda").repeat(8)[:dil].to(torch.bfloat16)
    got, _ = _grads(x, dy, dil, partials)
    left = [t for t in range(27) if t % 3 == 0]
    if partials:
        assert torch.equal(got[left], exp[left])
    else:
        assert torch.allclose(got[left], exp[left], rtol=1e-4, atol=1e-3)
    other = [c for c in range(16) if c != 6]
    assert bool(torch.isfinite(got[..., other]).all()) and not bool(torch.isfinite(got[13, :, 6]).any())
