"""Smoothing steps with every column length (4, 8, 16 and 32 planes per CTA, the
last column cut short) and long chains of steps that start before the previous
one has drained: bit-exact against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from biomedisa_gb300 import _native as nat
from biomedisa_gb300.interpolation import smooth_buffers, smooth_check

pytestmark = pytest.mark.gpu


def _smooth(maps, iters):
    nol, Zc, Yc, Xc = maps.shape
    tmp0, tmp1 = smooth_buffers(Zc, Yc, Xc, "cuda")
    tmp0.fill_(-7.0)
    tmp1.fill_(123.0)
    t = torch.from_numpy(maps).cuda()
    nat.call("si_smooth_f32", t.data_ptr(), tmp0.data_ptr(), tmp1.data_ptr(), nol, Zc, Yc, Xc, iters, 0,
             torch.cuda.current_stream().cuda_stream)
    smooth_check()
    return t.cpu().numpy()


def _map(shape, nol, seed):
    rng = np.random.default_rng(seed)
    m = (rng.random((nol,) + shape) * 50).astype(np.float32)
    m[:, :, : shape[1] // 3] = 0.0
    return m


@pytest.mark.parametrize("shape", [(33, 60, 70), (71, 400, 386), (130, 400, 386), (213, 400, 386)],
                         ids=["4_planes", "8_planes", "16_planes", "32_planes"])
def test_column_lengths(shape, cuda):
    maps = _map(shape, 1, sum(shape))
    assert np.array_equal(_smooth(maps, 2).view(np.uint32), O.smooth(maps, 2, "f32").view(np.uint32))


@pytest.mark.parametrize("iters", [2, 45])
def test_chains_of_steps(iters, cuda):
    maps = _map((18, 40, 75), 3, iters)
    assert np.array_equal(_smooth(maps, iters).view(np.uint32), O.smooth(maps, iters, "f32").view(np.uint32))
