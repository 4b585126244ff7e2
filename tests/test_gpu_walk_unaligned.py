"""Walks and sweeps that are no multiple of four steps, with more walks than the SMs
hold threads: hit maps equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
from biomedisa_gb300 import smart_interpolation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32], ids=["u8", "u16", "f32"])
@pytest.mark.parametrize("sorw,sweep", [(33, 0), (50, 30), (36, 7), (3, 0), (32, 32)], ids=str)
def test_unaligned_walks_equal_oracle(sorw, sweep, dtype, cuda):
    rng = np.random.default_rng(sorw + sweep)
    shape = (34, 36, 38)
    lab = np.zeros(shape, np.int32)
    lab[::3] = 1 + (np.arange(36) > 17)[None, :, None]
    img = rng.normal(90, 30, shape).clip(0, 255).astype(dtype) * dtype(3 if dtype != np.uint8 else 1)
    kw = dict(nbrw=13, sorw=sorw, return_hits=True)  # 12 slices, 213 thousand walks
    got = smart_interpolation(img, lab, rng_seed=4, sweep_steps=sweep, **kw)
    exp = O.smart_interpolation(img, lab, key=4, **kw)
    assert np.array_equal(got["hits"], exp["hits"]) and np.array_equal(got["regular"], exp["regular"])
