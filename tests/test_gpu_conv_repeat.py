"""The tensor-core convolution gives the same bits however often it runs: rows of
the residual wait in a ring of slots, and a slot that is refilled under its readers
shows in a few voxels of one launch in thousands."""
import pytest
import torch

from biomedisa_gb300 import surrogate as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,dil", [((7, 48, 48, 48), 8), ((3, 64, 64, 64), 8), ((2, 40, 50, 130), 2)], ids=str)
@pytest.mark.parametrize("masked", [False, True])
def test_residual_layers_repeat(shape, dil, masked, cuda):
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + dil)
    x, res = (torch.randn((*shape, 16), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    conv = S.SurrogateNet(dilations=(1,)).convs[1]
    conv.dil = dil

    def run():
        if masked:
            return S.conv_dgrad(x, conv, shape, residual=res, tensor_core=True, mask=res)
        return S.conv_fwd(x, conv, shape, relu=True, residual=res, tensor_core=True)

    first, wrong = run(), torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(3000):
        wrong += (run() != first).any()
    S.umma_check()
    assert int(wrong) == 0
    # the same residual added to the convolution without one, one rounding later
    if not masked:
        y = S.conv_fwd(x, conv, shape, relu=False, out_f32=True, tensor_core=True)
        assert torch.equal(first, torch.relu(y + res.float()).to(torch.bfloat16))
