"""Smoothing with a narrow last column (8 or 32 wide): rows on both sides of the
rule and shorter than a column, rows of columns cut short, outermost layers that
hold values of their own (infinities and -0 among them), a support that lies in a
corner or on a face only. Bit-exact against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from biomedisa_gb300 import _native as nat
from biomedisa_gb300.interpolation import smooth_buffers, smooth_check

pytestmark = pytest.mark.gpu


def _smooth(maps, iters, pairs):
    nol, Zc, Yc, Xc = maps.shape
    nat.call("si_smooth_set_pairs", pairs)
    try:
        tmp0, tmp1 = smooth_buffers(Zc, Yc, Xc, "cuda")
        tmp0.fill_(-7.0)
        tmp1.fill_(123.0)
        t = torch.from_numpy(maps).cuda()
        nat.call("si_smooth_f32", t.data_ptr(), tmp0.data_ptr(), tmp1.data_ptr(), nol, Zc, Yc, Xc, iters, 0, nat.stream())
        smooth_check()
    finally:
        nat.call("si_smooth_set_pairs", 1)
    return t.cpu().numpy()


@pytest.mark.parametrize("pairs", [1, 2])
@pytest.mark.parametrize("kind", ["dense", "corner", "face"])
@pytest.mark.parametrize("shape", [(5, 10, 66), (4, 67, 130), (9, 34, 72), (6, 65, 73), (7, 17, 96), (4, 5, 97),
                                   (3, 3, 3), (5, 64, 8), (4, 16, 9), (3, 33, 32), (1, 9, 65), (6, 26, 258)], ids=str)
def test_narrow_columns(shape, kind, pairs, cuda):
    rng = np.random.default_rng(sum(shape))
    m = (rng.random((2,) + shape) * 50).astype(np.float32)
    if kind == "dense":
        m[0, 0, 0, 0], m[0, -1, -1, -1], m[1, 0, -1, shape[2] // 2] = np.inf, -0.0, -0.0
    elif kind == "corner":
        m[:, :, 2:] = 0.0
        m[:, :, :, :-2] = 0.0
    else:
        m[:, :, :, 1:] = 0.0
    for iters in (1, 2, 5):
        got, exp = _smooth(m.copy(), iters, pairs), O.smooth(m.copy(), iters, "f32")
        nan = np.isnan(exp)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], exp.view(np.uint32)[~nan])
