"""The row search (csrc/edt_search.cu) against the oracle's EDT, bit for bit, at the sizes where its tiles end:
segments of 16 rows times 8 warps (16, 128, 256, 384, 512), 4-candidate rounds, 32-z chunks, rows whose length is a
multiple of 4 (16-byte stores) and not, columns longer than 512 (the sweeps take the map), and scenes from a few
sites (long jumps between winners) to nearly full."""
import numpy as np
import pytest
import torch

import gvx
import oracle
from gpu_helpers import first_mismatch, oracle_edt, to_u32
from gvx.batch import Batch

SIDE = 0.01


def _points(dims, n, seed):
    rng = np.random.default_rng(seed)
    v = np.stack([rng.integers(0, d, n) for d in dims], 1)
    return ((v + rng.uniform(0.1, 0.9, v.shape)) * SIDE).astype(np.float32)


def _floor(dims, seed):
    """A rough floor and a far wall: every column has sites, winners jump between the two."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(dims[0]), np.arange(dims[1]), indexing="ij")
    z = np.clip(dims[2] // 8 + rng.integers(-1, 2, x.shape), 0, dims[2] - 1)
    p = np.stack([x, y, z], -1).reshape(-1, 3)
    wall = np.stack([np.full(dims[1], dims[0] - 1), np.arange(dims[1]), np.full(dims[1], dims[2] // 2)], 1)
    return ((np.concatenate([p, wall]) + 0.5) * SIDE).astype(np.float32)


DIMS = [(1, 1, 1), (15, 17, 31), (16, 16, 32), (33, 31, 33), (127, 129, 40), (128, 128, 64), (130, 20, 65),
        (255, 257, 9), (384, 12, 34), (13, 385, 32), (511, 10, 33), (12, 512, 31), (512, 512, 5), (513, 9, 40),
        (9, 513, 20), (20, 24, 600), (21, 9, 1023), (64, 48, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("scene", ["none", "one", "few", "some", "dense", "floor"])
def test_search_equals_oracle(dims, scene):
    n = dims[0] * dims[1] * dims[2]
    count = {"none": 0, "one": 1, "few": 7, "some": max(1, n // 100), "dense": max(1, n // 2), "floor": 0}[scene]
    pts = _floor(dims, n) if scene == "floor" else _points(dims, min(count, 400_000), n + count)
    _, want = oracle_edt(dims, SIDE, pts)
    m = gvx.DistanceVoxelMap(dims, SIDE)
    p = torch.as_tensor(pts)
    m.voxelize_edt(p)
    got = to_u32(m.data())
    assert np.array_equal(got, want), first_mismatch(got, want, dims)
    m.clearMap()
    m.insertPointCloud(p)
    m.parallelBanding3D()
    got = to_u32(m.data())
    assert np.array_equal(got, want), first_mismatch(got, want, dims)
    assert m.edt_check() == 0


@pytest.mark.gpu
def test_search_leaves_other_sites_to_the_sweeps():
    """A map transformed before holds other sites than its voxels' own: the second EDT equals the oracle's second."""
    dims = (70, 65, 50)
    pts = _points(dims, 300, 5)
    _, want = oracle_edt(dims, SIDE, pts)
    m = gvx.DistanceVoxelMap(dims, SIDE)
    m.insertPointCloud(torch.as_tensor(pts))
    for _ in range(2):
        m.parallelBanding3D()
        got = to_u32(m.data())
        assert np.array_equal(got, want), first_mismatch(got, want, dims)
        oracle.pba(want, dims)


@pytest.mark.gpu
@pytest.mark.parametrize("long_map", [False, True])
def test_batch_search_equals_oracle(long_map):
    """Uneven maps in one batch, one of them transformed before its turn; with a column above 512 rows in the batch
    the sweeps take every map."""
    dims = [(40, 33, 70), (129, 16, 31), (16, 200, 33), (1, 1, 1), (65, 64, 96)] + ([(520, 8, 9)] if long_map else [])
    clouds = [_points(d, max(1, d[0] * d[1] * d[2] // 200), i) for i, d in enumerate(dims)]
    maps = [gvx.DistanceVoxelMap(d, SIDE) for d in dims]
    b = Batch(maps)
    xyz = torch.as_tensor(np.concatenate(clouds)).cuda()
    offsets = torch.tensor(np.concatenate([[0], np.cumsum([len(c) for c in clouds])]), dtype=torch.int64).cuda()
    wants = [oracle_edt(d, SIDE, c)[1] for d, c in zip(dims, clouds)]
    b.voxelize_edt(xyz, offsets)
    for m, d, w in zip(maps, dims, wants):
        assert np.array_equal(to_u32(m.data()), w), first_mismatch(to_u32(m.data()), w, d)
    b.clear()
    b.insert(xyz, offsets)
    maps[0].parallelBanding3D()  # this one comes transformed
    oracle.pba(wants[0], dims[0])
    b.edt()
    for m, d, w in zip(maps, dims, wants):
        assert np.array_equal(to_u32(m.data()), w), first_mismatch(to_u32(m.data()), w, d)
    assert b.edt_check() == 0


@pytest.mark.gpu
def test_batch_of_more_maps_than_block_rows():
    """A launch has at most 65,535 block rows; a batch has no such limit."""
    n, dims = 65_540, (18, 18, 32)  # dims at which the row search takes the batch
    n_vox = dims[0] * dims[1] * dims[2]
    voxels = torch.full((n, n_vox), 0x3FFFFFFF, dtype=torch.int32, device="cuda")
    at = torch.as_tensor(np.random.default_rng(1).integers(0, n_vox, n)).cuda()
    site = (at % dims[0] | at // dims[0] % dims[1] << 10 | at // (dims[0] * dims[1]) << 20).to(torch.int32)[:, None]
    voxels.scatter_(1, at[:, None], site)
    maps = [gvx.DistanceVoxelMap(dims, 1.0, voxels=voxels[k]) for k in range(n)]
    b = Batch(maps)
    b.edt()
    assert b.edt_check() == 0
    assert all(bool((v == s).all()) for v, s in zip(voxels.split(4096), site.split(4096)))


@pytest.mark.gpu
@pytest.mark.parametrize("dims,n", [((12, 12, 12), 500), ((20, 20, 20), 100), ((64, 50, 4), 30), ((5, 3, 1), 300)])
def test_batches_of_small_maps_equal_oracle(dims, n):
    """Many small or flat maps, which the sweeps take, a third of them transformed before."""
    clouds = [_points(dims, 1 + i % 40, i) for i in range(n)]
    maps = [gvx.DistanceVoxelMap(dims, SIDE) for _ in range(n)]
    b = Batch(maps)
    xyz = torch.as_tensor(np.concatenate(clouds)).cuda()
    offsets = torch.tensor(np.concatenate([[0], np.cumsum([len(c) for c in clouds])]), dtype=torch.int64).cuda()
    wants = [oracle_edt(dims, SIDE, c)[1] for c in clouds]
    b.voxelize_edt(xyz, offsets)
    assert np.array_equal(np.stack([to_u32(m.data()) for m in maps]), np.stack(wants))
    b.clear()
    b.insert(xyz, offsets)
    for m, w in list(zip(maps, wants))[::3]:
        m.parallelBanding3D()
        oracle.pba(w, dims)
    b.edt()
    assert np.array_equal(np.stack([to_u32(m.data()) for m in maps]), np.stack(wants))
    assert b.edt_check() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dims,n", [((12, 12, 12), 2000), ((20, 20, 20), 300), ((100, 100, 8), 64), ((48, 48, 48), 100),
                                    ((96, 96, 96), 32), ((128, 128, 128), 2)])
def test_batches_take_the_faster_way(dims, n):
    """Whatever the maps' sizes, the batched EDT takes no longer than the sweeps (which the tuner times) by more than a
    fourth, a few launches' time apart.  Taken by the row search, 2000 maps of 12^3 took three times as long."""
    clouds = [_points(dims, max(10, dims[0] * dims[1] * dims[2] // 100), i) for i in range(n)]
    maps = [gvx.DistanceVoxelMap(dims, SIDE) for _ in range(n)]
    b = Batch(maps)
    xyz = torch.as_tensor(np.concatenate(clouds)).cuda()
    offsets = torch.tensor(np.concatenate([[0], np.cumsum([len(c) for c in clouds])]), dtype=torch.int64).cuda()
    b.clear()
    b.insert(xyz, offsets)
    sweeps = b.autotune(force=True)["ms"]
    best = 1e9
    for _ in range(6):
        b.clear()
        b.insert(xyz, offsets)
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        b.edt()
        t1.record()
        torch.cuda.synchronize()
        best = min(best, t0.elapsed_time(t1))
    assert best < 1.25 * sweeps + 0.02
