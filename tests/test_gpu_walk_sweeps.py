"""Sorted sweeps where their kernels can go wrong: hits held back over two steps
(voxels next to the border, where moves are refused; sweeps longer than the
held counts' 16 bits; walks that are not multiples of four steps), the flush of
small weights (strong edges, variance one, values that are not numbers), the
one-launch and the three-launch scan at the edges of their ranges, few and many
walks. Hit maps equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
from biomedisa_gb300 import _native as nat
from biomedisa_gb300 import smart_interpolation, smart_interpolation_batch

pytestmark = pytest.mark.gpu


def _volume(shape, seed, every=3, noise=14.0):
    rng = np.random.default_rng(seed)
    truth = np.ones(shape, np.int32)
    truth[:, shape[1] // 2:] = 2
    img = rng.normal(70 + 60 * (truth == 2), noise).clip(0, 255).astype(np.uint8)
    lab = np.zeros(shape, np.int32)
    lab[::every] = truth[::every]
    return img, lab


@pytest.mark.parametrize("dtype", [np.uint8, np.float32], ids=["u8", "f32"])
@pytest.mark.parametrize("shape,nbrw,sorw,sweep", [
    ((3, 3, 3), 4, 37, 0),          # one interior voxel behind refused moves on every side
    ((1, 5, 9), 3, 64, 0),          # a crop of three planes
    ((14, 17, 19), 2, 1001, 0),     # a walk of 1001 steps: default sweeps of 128, unaligned second walk
    ((9, 12, 11), 1, 999, 5),       # short sweeps
    ((8, 9, 10), 1, 140_001, 140_001),  # one sweep, more steps than a held count holds
], ids=str)
def test_held_hits_equal_oracle(shape, nbrw, sorw, sweep, dtype, cuda):
    img, lab = _volume(shape, sum(shape))
    kw = dict(nbrw=nbrw, sorw=sorw, return_hits=True)
    got = smart_interpolation(img.astype(dtype), lab, rng_seed=23, sweep_steps=sweep, **kw)
    exp = O.smart_interpolation(img.astype(dtype), lab, key=23, **kw)
    assert np.array_equal(got["hits"], exp["hits"]) and np.array_equal(got["regular"], exp["regular"])


@pytest.mark.parametrize("noise", [0.0, 0.6, 40.0])
def test_small_weights_equal_oracle(noise, cuda):
    """Differences on both sides of the flush at d^2 c = 125."""
    img, lab = _volume((20, 24, 22), 3, 4, noise)
    img[:, ::3, ::5] = 255
    kw = dict(nbrw=6, sorw=130, return_hits=True)
    got = smart_interpolation(img, lab, rng_seed=2, **kw)
    exp = O.smart_interpolation(img, lab, key=2, **kw)
    assert np.array_equal(got["hits"], exp["hits"])


@pytest.mark.parametrize("edge,device_loop", [(1, 1), (1, 0), (2, 1), (3, 0)], ids=str)
def test_scans_of_few_and_many_buckets(edge, device_loop, cuda):
    """29,406 (three launches), 4,095 (one launch, its tile one short) and 1,350
    buckets of three labels over a 26 x 29 x 13 crop."""
    img, lab = _volume((24, 27, 11), 6, 4)
    kw = dict(nbrw=5, sorw=200, return_hits=True)
    nat.call("si_walk_sorted_set_loop", device_loop)
    try:
        got = smart_interpolation(img, lab, rng_seed=5, sort_edge=edge, **kw)
    finally:
        nat.call("si_walk_sorted_set_loop", 1)
    exp = O.smart_interpolation(img, lab, key=5, **kw)
    assert np.array_equal(got["hits"], exp["hits"])


def test_many_walks_in_one_sweep(cuda):
    """More walks than small launches take, single and batched."""
    img, lab = _volume((21, 60, 58), 8, 2)
    kw = dict(nbrw=16, sorw=60, return_hits=True)  # 11 slices, 562 thousand walks
    exp = O.smart_interpolation(img, lab, key=9, **kw)
    got = smart_interpolation(img, lab, rng_seed=9, **kw)
    both = smart_interpolation_batch([img, img.astype(np.uint16)], [lab, lab], rng_seed=9, autotune_params=False, **kw)
    assert np.array_equal(got["hits"], exp["hits"]) and np.array_equal(both[0]["hits"], exp["hits"])
    exp16 = O.smart_interpolation(img.astype(np.uint16), lab, key=9, **kw)
    assert np.array_equal(both[1]["hits"], exp16["hits"])


@pytest.mark.parametrize("shift", [0, 16, 32])
def test_float_records_aligned_to_16_bytes_only(shift, cuda):
    """A record buffer that starts between two 32-byte boundaries."""
    import torch

    from biomedisa_gb300 import interpolation as I

    img, lab = _volume((12, 15, 14), 4)
    img = img.astype(np.float32)
    ti, tl = I.upload(*I.normalize_host_dtypes(img, lab))
    job = I.DeviceJob(ti, nat.SI_F32, tl, nat.SI_I32, nbrw=3, sorw=150, rng_seed=6)
    assert job.analyze() is None
    job.prepare()
    cp = job.cplan
    n = cp.voxels * 32
    buf = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
    assert buf.data_ptr() % 64 == 0
    packed = buf[shift:shift + n]
    st = torch.cuda.current_stream().cuda_stream
    nat.call("si_pack_neighbours", job.work.data_ptr(), 1, cp.Zc, cp.Yc, cp.Xc, packed.data_ptr(), st)
    job.hits = torch.zeros((job.lplan.nol, cp.Zc, cp.Yc, cp.Xc), dtype=torch.int32, device="cuda")
    I.walk_sorted(packed, True, cp.Zc, cp.Yc, cp.Xc, job.seeds, job.n_seeds, job.seed_capacity, 3, 150, 6, job.hits,
                  job.lplan.nol)
    exp = O.smart_interpolation(img, lab, key=6, nbrw=3, sorw=150, return_hits=True)
    assert np.array_equal(job.hits_full().cpu().numpy(), exp["hits"])


def test_batch_of_many_volumes(cuda):
    """130 volumes (more than one per thread of a float CTA), some without a
    walker of a kind, each equal to its own call."""
    rng = np.random.default_rng(4)
    imgs, labs = [], []
    for k in range(130):
        shape = tuple(int(v) for v in rng.integers(4, 10, 3))
        img, lab = _volume(shape, k)
        imgs.append(img if k % 3 else img.astype(np.float32))
        labs.append(lab)
    kw = dict(nbrw=2, sorw=70, return_hits=True, rng_seed=12)
    got = smart_interpolation_batch(imgs, labs, autotune_params=False, **kw)
    for img, lab, g in zip(imgs, labs, got):
        one = smart_interpolation(img, lab, walker="packed", **kw)
        assert np.array_equal(g["hits"], one["hits"])


@pytest.mark.parametrize("nbrw", [3, 5, 7], ids=["105k", "174k", "244k"])
@pytest.mark.parametrize("dtype", [np.uint8, np.float32], ids=["u8", "f32"])
def test_one_walk_or_two_per_thread(nbrw, dtype, cuda):
    """Walks on both sides of one and two per resident thread (117 and 233
    thousand on 152 SMs), with more steps than the longest default sweep."""
    img, lab = _volume((21, 60, 58), 11, 2)  # 11 slices, 35 thousand seeds
    kw = dict(nbrw=nbrw, sorw=1003 if nbrw == 3 else 70, return_hits=True)
    exp = O.smart_interpolation(img.astype(dtype), lab, key=3, **kw)
    got = smart_interpolation(img.astype(dtype), lab, rng_seed=3, **kw)
    assert np.array_equal(got["hits"], exp["hits"])


@pytest.mark.parametrize("dense", [False, True])
def test_default_bricks_fit_the_scratch(dense, cuda):
    """The default sort edge follows the walks per voxel; a scratch sized for
    bricks of six voxels, or for any number of walks above the actual one, is
    enough for it, and the hits stay the oracle's."""
    import ctypes

    import torch

    from biomedisa_gb300 import interpolation as I

    img, lab = _volume((26, 40, 44), 7, 2 if dense else 13)
    nbrw = 12 if dense else 1
    ti, tl = I.upload(*I.normalize_host_dtypes(img, lab))
    job = I.DeviceJob(ti, nat.SI_U8, tl, nat.SI_I32, nbrw=nbrw, sorw=90, rng_seed=8)
    assert job.analyze() is None
    job.prepare()
    cp, nol = job.cplan, job.lplan.nol
    exp = O.smart_interpolation(img, lab, key=8, nbrw=nbrw, sorw=90, return_hits=True)["hits"]
    n = int(job.n_seeds.item())
    sizes = set()
    for edge, walks in ((6, n * nbrw), (0, n * nbrw), (0, 40 * n * nbrw)):
        need = ctypes.c_ulonglong(0)
        nat.call("si_walk_sorted_scratch", cp.Zc, cp.Yc, cp.Xc, walks, nol, edge, ctypes.byref(need))
        sizes.add(need.value)
        scratch = torch.full((need.value + 4096,), 99, dtype=torch.uint8, device="cuda")
        job.hits = torch.zeros((nol, cp.Zc, cp.Yc, cp.Xc), dtype=torch.int32, device="cuda")
        nat.call("si_walk_sorted", job.packed.data_ptr(), 0, cp.Zc, cp.Yc, cp.Xc, job.seeds.data_ptr(),
                 job.n_seeds.data_ptr(), n, nbrw, 90, 8, job.hits.data_ptr(), nol, 0, 0, scratch.data_ptr(), need.value,
                 None, nat.stream())
        assert bool((scratch[need.value:] == 99).all())
        assert np.array_equal(job.hits_full().cpu().numpy(), exp)
    assert len(sizes) == (3 if dense else 2)  # sparse walks take larger bricks in no less scratch
    nat.call("si_walk_sorted_scratch", cp.Zc, cp.Yc, cp.Xc, n * nbrw, nol, 6, ctypes.byref(need))
    with pytest.raises(nat.NativeError, match="scratch"):
        nat.call("si_walk_sorted", job.packed.data_ptr(), 0, cp.Zc, cp.Yc, cp.Xc, job.seeds.data_ptr(),
                 job.n_seeds.data_ptr(), n, nbrw, 90, 8, job.hits.data_ptr(), nol, 0, 0, scratch.data_ptr(),
                 need.value - 1, None, nat.stream())
