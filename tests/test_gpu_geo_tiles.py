"""Tiled geodesic scan where its tiles and launches can go wrong: volumes below,
at and beyond one tile on each axis, thin volumes, start maps with infinities,
NaN, negative and equal values, a scan right behind the kernel that writes its
image, against the oracle's sequential scan."""
import numpy as np
import pytest
import torch

import geo_oracle as G
from biomedisa_gb300 import geodis

pytestmark = pytest.mark.gpu


def _maps(shape, nol, seed, kind):
    rng = np.random.default_rng(seed)
    img = rng.random(shape).astype(np.float32)
    if kind == "steps":  # many equal costs
        img = np.round(img * 3).astype(np.float32) / 4
    c = np.where(rng.random((nol,) + shape) < 0.03, 0.0, np.inf).astype(np.float32)
    if kind == "odd":
        c[rng.random(c.shape) < 0.02] = np.nan
        c[rng.random(c.shape) < 0.02] = -0.0
        c[rng.random(c.shape) < 0.02] = -1.5
        img[rng.random(shape) < 0.01] = np.nan
        img[rng.random(shape) < 0.01] = np.inf
    return img, c


@pytest.mark.parametrize("kind", ["noise", "steps", "odd"])
@pytest.mark.parametrize("shape", [(2, 3, 3), (2, 40, 5), (9, 34, 35), (8, 3, 90), (40, 33, 70), (17, 65, 33)], ids=str)
def test_tiles_equal_sequential_scan(shape, kind, cuda):
    img, c = _maps(shape, 2, sum(shape), kind)
    for mode in (geodis.SCAN_TILES, geodis.SCAN_TILE_GRAPH):
        got = torch.from_numpy(c.copy()).to(cuda)
        geodis.scan_device(got, torch.from_numpy(img).to(cuda), 1.0, 2, mode)
        got = got.cpu().numpy()
        for k in range(2):
            exp = c[k].copy()
            with np.errstate(all="ignore"):
                G.raster_scan(img, exp, 1.0, 2)
            assert np.array_equal(got[k].view(np.uint32), exp.view(np.uint32)) or (
                np.array_equal(np.isnan(got[k]), np.isnan(exp)) and
                np.array_equal(got[k][~np.isnan(exp)].view(np.uint32), exp[~np.isnan(exp)].view(np.uint32))), (mode, k)


def test_scans_behind_the_writer_of_their_image(cuda):
    """The first launch may not read the image before the kernel before it has
    ended; scans of two images follow one another without a wait."""
    shape = (30, 50, 60)
    img, c = _maps(shape, 1, 5, "noise")
    d = torch.from_numpy(img).to(cuda)
    big = torch.zeros(1 << 26, device=cuda)
    outs = []
    for k in range(6):
        buf = torch.zeros(shape, device=cuda)
        m = torch.from_numpy(c.copy()).to(cuda)
        big.add_(1.0)
        buf.copy_(d + float(k % 2))
        outs.append(geodis.scan_device(m, buf, 1.0, 1, geodis.SCAN_TILES))
    exp = [c[0].copy(), c[0].copy()]
    for k in range(2):
        G.raster_scan(img + np.float32(k), exp[k], 1.0, 1)
    for k, o in enumerate(outs):
        assert np.array_equal(o.cpu().numpy()[0], exp[k % 2]), k
