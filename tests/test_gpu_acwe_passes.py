"""The chamfer band's relaxation passes, bit for bit against ten passes of the
27-point form in NumPy, on crops that end inside, at and behind a 32 x 8 tile and
a 16-plane column; labels on the crop's own faces included."""
import numpy as np
import pytest
import torch

from biomedisa_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _jacobi(d, passes=10):
    w = [np.float32(v) for v in (1.0, 1.41421356, 1.73205081)]
    Z, Y, X = d.shape
    for _ in range(passes):
        p = np.pad(d, 1, constant_values=np.float32(np.inf))
        best = d.copy()
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    n = abs(dz) + abs(dy) + abs(dx)
                    if n:
                        best = np.minimum(best, p[1 + dz:1 + dz + Z, 1 + dy:1 + dy + Y, 1 + dx:1 + dx + X] + w[n - 1])
        best = np.minimum(best, np.float32(11.0))
        new = d.copy()
        new[:, 1:-1, 1:-1] = best[:, 1:-1, 1:-1]
        d = new
    return d


@pytest.mark.parametrize("shape", [(1, 3, 3), (2, 8, 32), (16, 9, 33), (17, 7, 31), (33, 24, 65), (5, 2, 40)], ids=str)
def test_chamfer_passes_bit_exact(shape, cuda):
    rng = np.random.default_rng(sum(shape))
    lab = (rng.random(shape) < 0.01).astype(np.uint8)
    lab[0, 0, 0] = 1
    n = lab.size
    L = torch.from_numpy(lab.ravel()).to(cuda)
    d, t = (torch.empty(n, dtype=torch.float32, device=cuda) for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    nat.call("si_acwe_dist_init", L.data_ptr(), n, d.data_ptr(), st)
    nat.call("si_acwe_chamfer_band", d.data_ptr(), t.data_ptr(), *shape, st)
    exp = _jacobi(np.where(lab == 0, np.float32(100.0), np.float32(0.0)).astype(np.float32))
    assert np.array_equal(d.cpu().numpy().reshape(shape).view(np.uint32), exp.view(np.uint32))
