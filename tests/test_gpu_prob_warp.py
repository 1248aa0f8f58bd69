"""ProbVoxelMap inserts whose neighbouring points share voxels and 4-voxel words (one swap per word and warp) against
the oracle, which applies the points one by one."""
import numpy as np
import pytest
import torch

import gvx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 40_000])
@pytest.mark.parametrize("spread", [3, 60, 100_000])
def test_runs_of_points(n, spread):
    dims = (37, 29, 23)
    rng = np.random.default_rng(n + spread)
    g, o = gvx.ProbVoxelMap(dims, 1.0), oracle.pvm_empty(dims)
    for meaning in (1, 0, 129, 90, 254, 0, 4, 255, 2):
        ids = np.sort(rng.integers(0, min(spread, dims[0] * dims[1] * dims[2]), n))
        pts = np.stack([ids % dims[0], ids // dims[0] % dims[1], ids // (dims[0] * dims[1])], 1) + 0.5
        pts[rng.random(n) < 0.05] = -3e9  # the reference's saturating conversion puts these into voxel 0
        pts[rng.random(n) < 0.05] = 1e9  # outside
        pts = pts.astype(np.float32)
        g.insertPointCloud(torch.as_tensor(pts), meaning)
        oracle.pvm_insert(o, dims, 1.0, pts, meaning)
        assert np.array_equal(g.data().cpu().numpy(), o)


@pytest.mark.parametrize("meaning", [0, 1, 100, 129, 255])
def test_settled_voxels_beside_moving_ones(meaning):
    """Repeated inserts until every voxel of the cloud stands still, then the cloud with a few new voxels in it."""
    dims = (37, 29, 23)
    rng = np.random.default_rng(meaning)
    g, o = gvx.ProbVoxelMap(dims, 1.0), oracle.pvm_empty(dims)
    pts = (rng.random((20_000, 3)) * dims * [1, 1, 0.5]).astype(np.float32)
    for k in range(16):
        if k == 15:
            pts[::97] += np.float32([0, 0, 11])
        g.insertPointCloud(torch.as_tensor(pts), meaning)
        oracle.pvm_insert(o, dims, 1.0, pts, meaning)
        assert np.array_equal(g.data().cpu().numpy(), o)


def test_settled_map_is_only_read():
    """A cloud into a map that it no longer changes takes a third of the time it took when it did."""
    m = gvx.ProbVoxelMap((256, 256, 256), 1.0)
    pts = torch.rand(3_000_000, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(0)) * 256

    def insert_ms():
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        m.insertPointCloud(pts, 1)
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    fresh = []
    for _ in range(8):
        m.clearMap()
        fresh.append(insert_ms())
    for _ in range(4):
        m.insertPointCloud(pts, 1)
    assert min(insert_ms() for _ in range(8)) < 0.45 * min(fresh)
