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
