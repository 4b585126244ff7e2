"""Counts of the check of a result on its labels, at the ends of its 16-voxel
steps and at pointers between 16-byte boundaries. Whole numbers: exact."""
import numpy as np
import pytest
import torch

from biomedisa_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4099, 1_200_005])
@pytest.mark.parametrize("dtype,code", [(np.uint8, nat.SI_U8), (np.int16, nat.SI_I16), (np.int32, nat.SI_I32)])
@pytest.mark.parametrize("shift", [(0, 0), (1, 0), (0, 3)], ids=str)
def test_counts(n, dtype, code, shift, cuda):
    rng = np.random.default_rng(n)
    lab = rng.integers(0, 4, n).astype(dtype)
    if dtype != np.uint8:
        lab[::5] = -1
        lab[::7] = 300
    res = rng.integers(0, 4, n).astype(np.uint8)
    res[::11] = 300 % 256
    a, b = shift
    tl = torch.zeros(n + a, dtype=torch.from_numpy(lab).dtype, device="cuda")[a:]
    tr = torch.zeros(n + b, dtype=torch.uint8, device="cuda")[b:]
    tl.copy_(torch.from_numpy(lab))
    tr.copy_(torch.from_numpy(res))
    counts = torch.ones(3, dtype=torch.int64, device="cuda")
    nat.call("si_label_agreement", tl.data_ptr(), code, tr.data_ptr(), n, counts.data_ptr(), nat.stream())
    pos = lab > 0
    exp = [pos.sum(), (pos & (res > 0)).sum(), (pos & (lab == res)).sum()]
    assert counts.tolist() == [1 + int(v) for v in exp]
