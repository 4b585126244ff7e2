"""si_geo_scan_launches counts the tile-wavefronts that a scan launches: at least
those that hold voxels, and none whose rows of tiles are all empty."""
import ctypes

import numpy as np
import pytest

from biomedisa_gb300 import _native as nat

TP, TQ, TR = 32, 32, 8  # tile extents along p, q, r


def _count(shape):
    n = ctypes.c_longlong(0)
    nat.call("si_geo_scan_launches", *shape, 1.0, 1, 4, ctypes.byref(n))
    return n.value


def _waves(shape, fwd):
    """(wavefronts with voxels, wavefronts with a row of tiles whose p, q, r ranges
    meet 1 <= q - 2 r <= Y - 2 and 1 <= p - 2 q <= X - 2)."""
    Z, Y, X = shape
    z, y, x = np.meshgrid(np.arange(1, Z) if fwd else np.arange(Z - 1), np.arange(1, Y - 1), np.arange(1, X - 1),
                          indexing="ij")
    s = 1 if fwd else -1
    p, q, r = s * (x + 2 * y + 4 * z), s * (y + 2 * z), s * z
    p0, q0, r0 = p.min(), q.min(), r.min()
    full = set(np.unique((p - p0) // TP + (q - q0) // TQ + (r - r0) // TR).tolist())
    u, v = sorted((s, s * (Y - 2))), sorted((s, s * (X - 2)))
    cover = set()
    for i in range((r.max() - r0) // TR + 1):
        ra, rb = r0 + i * TR, min(r0 + i * TR + TR - 1, r.max())
        for j in range((q.max() - q0) // TQ + 1):
            qa, qb = q0 + j * TQ, q0 + j * TQ + TQ - 1
            if qb < 2 * ra + u[0] or qa > 2 * rb + u[1]:
                continue
            for k in range((p.max() - p0) // TP + 1):
                pa, pb = p0 + k * TP, p0 + k * TP + TP - 1
                if pb >= 2 * qa + v[0] and pa <= 2 * qb + v[1]:
                    cover.add(i + j + k)
    return full, cover


@pytest.mark.parametrize("shape", [(12, 3, 3), (24, 4, 4), (100, 4, 4), (28, 4, 3), (22, 3, 5), (50, 3, 38),
                                   (9, 40, 33), (60, 5, 90), (40, 70, 90), (3, 100, 4)], ids=str)
def test_launches_are_those_of_the_scan(shape):
    waves = [_waves(shape, fwd) for fwd in (1, 0)]
    assert all(full <= cover for full, cover in waves)
    assert _count(shape) == sum(len(cover) for _, cover in waves)
