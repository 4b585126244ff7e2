"""Slice flags and bounding box of volumes with short rows, several to a warp: equal
to those of the same labels in rows made longer by zeros, and to NumPy's."""
import numpy as np
import pytest
import torch

from biomedisa_gb300 import _native as nat

pytestmark = pytest.mark.gpu
CODES = {np.uint8: nat.SI_U8, np.int16: nat.SI_I16, np.int32: nat.SI_I32}


def _flags(lab, allaxis):
    Z, Y, X = lab.shape
    lut = np.ones(256, np.uint8)
    lut[0] = 0
    imax = np.iinfo(np.int32).max
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in
         (lab, lut, np.zeros(Z + 2, np.uint8), np.zeros(Y + 2, np.uint8), np.zeros(X + 2, np.uint8),
          np.array([imax, -1] * 3, np.int32))]
    nat.call("si_slice_flags", t[0].data_ptr(), CODES[lab.dtype.type], Z, Y, X, t[1].data_ptr(), allaxis,
             *[v.data_ptr() for v in t[2:]], nat.stream())
    return [v.cpu().numpy() for v in t[2:]]


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.int32])
@pytest.mark.parametrize("X", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 33, 130])
@pytest.mark.parametrize("allaxis", [0, 1, 2])
def test_short_rows(X, dtype, allaxis, cuda):
    rng = np.random.default_rng(X)
    for shape, p in (((9, 30, X), 0.02), ((31, 7, X), 0.5), ((300, 70, X), 0.001)):
        lab = (rng.random(shape) < p).astype(dtype) * dtype(3)
        lab[shape[0] // 2] = 1
        got = _flags(lab, allaxis)
        longer = _flags(np.pad(lab, ((0, 0), (0, 0), (0, 200))), allaxis)
        for k in (0, 1, 3):
            assert np.array_equal(got[k], longer[k]), (shape, k)
        assert np.array_equal(got[2], longer[2][:X + 2]) and not longer[2][X + 1:].any()
        at = np.nonzero(lab)
        assert got[3].tolist() == [f(a) + 1 for a in at for f in (np.min, np.max)]
        if not allaxis:
            assert np.array_equal(got[0][1:-1], (lab != 0).any((1, 2)))
