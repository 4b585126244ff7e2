"""The cross entropy's sum over many voxels: against float64, the same in every
run, and infinite where a term is."""
import numpy as np
import pytest
import torch

from biomedisa_gb300 import surrogate as S

pytestmark = pytest.mark.gpu


def _inputs(V, nol, seed=0):
    g = torch.Generator(device="cuda").manual_seed(V + nol + seed)
    z = torch.randn((V, 16), generator=g, device="cuda") * 2
    p = torch.softmax(torch.randn((V, nol), generator=g, device="cuda") * 2, -1)
    return z, p, torch.rand(V, generator=g, device="cuda")


@pytest.mark.parametrize("V,nol", [(1, 13), (256, 1), (257, 2), (40 ** 3, 13), (3 * 56 ** 3, 5), (8 * 64 ** 3, 13),
                                   (2 ** 20 + 31, 16)])
def test_loss_is_the_float64_sum(V, nol, cuda):
    """One rounding of the sum and one of its quotient, 2^-24 each; a voxel's own
    binary32 operations (below 2^-20 of its terms) are independent of the next's."""
    z, p, w = _inputs(V, nol)
    net = S.SurrogateNet(dilations=(1,))
    loss, dl = net.loss_and_grad(z, p, w, nol, denom=V)
    logq = torch.log_softmax(z.double()[:, :nol], -1)
    terms = (p.double() * -logq).sum(-1) * w.double()
    exp, mag = float(terms.sum()) / V, float(terms.abs().sum()) / V + 1e-12
    assert abs(float(loss) - exp) / mag <= 2.0 ** -23 + 2.0 ** -20 / np.sqrt(V)
    for _ in range(4):
        again, dl2 = net.loss_and_grad(z, p, w, nol, denom=V)
        assert torch.equal(loss, again) and torch.equal(dl, dl2)
    # the gradient is the general kernel's, which logits between two 16-byte boundaries take
    off = torch.empty(V * 16 + 1, device="cuda")[1:].view(V, 16).copy_(z)
    assert torch.equal(dl, net.loss_and_grad(off, p, w, nol, denom=V)[1])


def test_loss_of_sure_voxels(cuda):
    """Logits 20 to 2 apart: terms of 1e-8 to 0.1 that a rounded 1 + e would lose.
    Voxel by voxel: 2^-20 of the term."""
    V = 64
    z = torch.full((V, 16), -30.0, device="cuda")
    z[:, 0] = torch.linspace(2, 20, V, device="cuda")
    z[:, 1] = 0.0
    p = torch.zeros((V, 3), device="cuda")
    p[:, 0] = 1.0
    net = S.SurrogateNet(dilations=(1,))
    for v in range(V):
        w = torch.zeros(V, device="cuda")
        w[v] = 1.0
        loss, _ = net.loss_and_grad(z, p, w, 3, denom=1)
        exp = -float(torch.log_softmax(z.double()[v, :3], -1)[0])
        assert abs(float(loss) - exp) <= 2.0 ** -20 * exp


def test_infinite_terms(cuda):
    """Infinite terms, also several in the voxels that one thread takes, leave an
    infinite loss; NaN stays NaN."""
    V, nol = 1 << 20, 3
    z, p, w = _inputs(V, nol)
    net = S.SurrogateNet(dilations=(1,))
    z[5, 1] = z[V - 300, 2] = -float("inf")
    z[5 + torch.arange(1, 3, device="cuda") * 4 * 256 * torch.cuda.get_device_properties(0).multi_processor_count, 0] = \
        -float("inf")
    assert float(net.loss_and_grad(z, p, w, nol, denom=V)[0]) == float("inf")
    z[77, 0] = float("nan")
    assert np.isnan(float(net.loss_and_grad(z, p, w, nol, denom=V)[0]))
