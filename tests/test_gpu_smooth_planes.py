"""Smoothing steps with every number of planes per CTA, the last column cut short:
bit-exact against the oracle. The planes are asked for, so that a change of their
rule shows here."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from biomedisa_gb300 import _native as nat
from biomedisa_gb300.interpolation import smooth_buffers, smooth_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,shape", [(2, (17, 40, 75)), (4, (66, 100, 130)), (8, (199, 200, 258)),
                                          (16, (199, 250, 386)), (32, (212, 400, 450))], ids=str)
def test_planes_equal_oracle(planes, shape, cuda):
    n = ctypes.c_int(0)
    nat.call("si_smooth_planes", *shape, ctypes.byref(n))
    assert n.value == planes
    rng = np.random.default_rng(planes)
    m = (rng.random((1,) + shape) * 50).astype(np.float32)
    m[:, :, : shape[1] // 3] = 0.0
    tmp0, tmp1 = smooth_buffers(*shape, "cuda")
    tmp0.fill_(-7.0)
    tmp1.fill_(123.0)
    t = torch.from_numpy(m).cuda()
    nat.call("si_smooth_f32", t.data_ptr(), tmp0.data_ptr(), tmp1.data_ptr(), 1, *shape, 2, 0, nat.stream())
    smooth_check()
    assert np.array_equal(t.cpu().numpy().view(np.uint32), O.smooth(m, 2, "f32").view(np.uint32))
