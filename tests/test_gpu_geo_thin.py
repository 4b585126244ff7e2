"""Tiled geodesic scan of volumes so thin that whole tile-wavefronts are launched
without a voxel: the wavefronts around them keep their order. Against the oracle's
sequential scan, launched directly and as a captured graph, both cost forms."""
import numpy as np
import pytest
import torch

import geo_oracle as G
from biomedisa_gb300 import geodis

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lamb", [1.0, 0.5])
@pytest.mark.parametrize("shape", [(12, 3, 3), (17, 3, 6), (100, 4, 4), (24, 4, 4), (28, 4, 3), (22, 3, 5),
                                   (50, 3, 38)], ids=str)
def test_thin_volumes_equal_sequential_scan(shape, lamb, cuda):
    rng = np.random.default_rng(sum(shape))
    img = rng.random(shape).astype(np.float32)
    c = np.full((3,) + shape, np.inf, np.float32)
    c[:, 0, 1:-1, 1:-1] = 0.0  # distances run through the whole volume, wavefront by wavefront
    c[1, -1] = 0.5
    c[2][rng.random(shape) < 0.05] = 0.25
    exp = [c[k].copy() for k in range(3)]
    with np.errstate(all="ignore"):
        for e in exp:
            G.raster_scan(img, e, lamb, 2)
    d = torch.from_numpy(img).to(cuda)
    for mode in (geodis.SCAN_TILES, geodis.SCAN_TILE_GRAPH):
        for _ in range(20):
            got = geodis.scan_device(torch.from_numpy(c.copy()).to(cuda), d, lamb, 2, mode).cpu().numpy()
            for k in range(3):
                assert np.array_equal(got[k].view(np.uint32), exp[k].view(np.uint32)), (mode, k)
