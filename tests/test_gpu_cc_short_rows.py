"""clean and fill of rows shorter than a word, several to a warp, and of one voxel a
row: on both sides of every power of two, rows that do not fill the last warp, ties
between the largest components. Against the oracle."""
import numpy as np
import pytest
import torch

import cc_oracle as C
from biomedisa_gb300 import postprocess as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 7, x) for x in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17)] +
                         [(1, 1, 1), (1, 1, 40), (1, 40, 1), (40, 1, 1), (33, 70, 1), (70, 1, 3), (1, 45, 2), (61, 53, 3)],
                         ids=str)
@pytest.mark.parametrize("p", [0.3, 0.7])
def test_short_rows(shape, p, cuda):
    rng = np.random.default_rng(sum(shape))
    for labels in (2, 4):
        vol = np.where(rng.random(shape) < p, rng.integers(1, labels, shape), 0).astype(np.uint8)
        t = torch.from_numpy(vol).to(cuda)
        for thr in (0.02, 0.5, 1.0):
            assert np.array_equal(P.clean(t, thr).cpu().numpy(), C.clean(vol, thr)), ("clean", thr)
            assert np.array_equal(P.fill(t, thr).cpu().numpy(), C.fill(vol, thr)), ("fill", thr)
