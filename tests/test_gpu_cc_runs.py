"""clean and fill on runs and 32-voxel words: row widths around a word, runs over
several words, checkerboards, boxes that begin and end inside a word, labels that
outweigh their complement, against the oracle."""
import numpy as np
import pytest
import torch

import cc_oracle as C
from biomedisa_gb300 import postprocess as P

pytestmark = pytest.mark.gpu


def _check(vol, cuda):
    t = torch.from_numpy(np.ascontiguousarray(vol)).to(cuda)
    for thr in (0.02, 0.5):
        assert np.array_equal(P.clean(t, thr).cpu().numpy(), C.clean(vol, thr)), ("clean", thr)
        assert np.array_equal(P.fill(t, thr).cpu().numpy(), C.fill(vol, thr)), ("fill", thr)


@pytest.mark.parametrize("X", [1, 2, 31, 32, 33, 63, 64, 65, 97, 200])
@pytest.mark.parametrize("p", [0.02, 0.4, 0.9])
def test_row_widths(X, p, cuda):
    rng = np.random.default_rng(X * 10 + int(p * 10))
    vol = np.where(rng.random((7, 9, X)) < p, rng.integers(1, 4, (7, 9, X)), 0).astype(np.uint8)
    _check(vol, cuda)


def test_long_runs_and_boxes_inside_words(cuda):
    vol = np.zeros((10, 12, 150), np.uint8)
    vol[2:8, 3:9, 37:131] = 1          # box from inside word 1 to inside word 4
    vol[4:6, 5:7, 60:100] = 0          # a cavity over two word borders
    vol[4, 5, 70] = 2
    vol[1:9, 2, 5:140:2] = 3           # a comb
    vol[9, 11, 149] = 2
    _check(vol, cuda)
    _check(vol + 4, cuda)              # no label 0


def test_checkerboard_and_stripes(cuda):
    z, y, x = np.indices((6, 7, 70))
    _check(((z + y + x) & 1).astype(np.uint8), cuda)
    _check((1 + (x // 3 + y) % 2).astype(np.uint8), cuda)
    _check((1 + (x % 32 == 31)).astype(np.uint8), cuda)


def test_large_components_and_islands(cuda):
    """Several blocks per pass, one component through the whole volume."""
    rng = np.random.default_rng(1)
    vol = np.zeros((70, 90, 110), np.uint8)
    vol[10:60, 10:80, 8:100] = 2
    vol[20:50, 30:60, 40:70] = 1
    noise = rng.random(vol.shape) < 0.03
    vol[noise] = rng.integers(0, 4, int(noise.sum()))
    _check(vol, cuda)


def test_present_labels(cuda):
    t = torch.tensor([[[3, 0, 255], [3, 7, 7]]], dtype=torch.uint8)
    assert P.present_labels(t) == P.present_labels(t.to(cuda)) == [0, 3, 7, 255]
    assert P.present_labels(t.to(cuda)[:, :, 1:2]) == [0, 7]
