"""Label lists of device volumes that the histogram kernel does not take."""
import pytest
import torch

from biomedisa_gb300 import postprocess as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int8, torch.int16, torch.int32, torch.int64, torch.bool])
def test_label_types(dtype, cuda):
    t = torch.zeros((3, 5, 7), dtype=dtype, device=cuda)
    t[1, 2, 3] = 1
    t[2] = 100
    assert P.present_labels(t) == ([0, 1] if dtype == torch.bool else [0, 1, 100])
    if dtype in (torch.int16, torch.int32, torch.int64):
        t[0, 0, 0] = 300
        assert P.present_labels(t) == [0, 1, 100, 300]


def test_empty_volume(cuda):
    t = torch.zeros((0, 4, 5), dtype=torch.uint8, device=cuda)
    assert P.present_labels(t) == []
    assert P.fill(t).shape == t.shape
