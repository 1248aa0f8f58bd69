"""The sweeps (csrc/edt.cu) in every configuration, on the maps they take: maps that hold other sites than their
voxels' own (moved by the caller, or transformed before), maps longer than 512 in x or y, and batches with such maps.
On other maps the row search runs whatever the configuration is."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest
import torch

import gvx
import oracle
from gpu_helpers import first_mismatch, oracle_edt, to_u32

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CONFIGS = [(rows, fused) for rows in (16, 32) for fused in (0, 1)]
THIN = [(1, 40, 60), (5, 3, 100), (33, 1, 20), (70, 9, 2), (1, 1, 300), (31, 33, 17)]


def _points(dims, n, seed):
    return (np.random.default_rng(seed).random((n, 3)) * dims).astype(np.float32)


@pytest.mark.parametrize("rows,fused", CONFIGS)
@pytest.mark.parametrize("dims", THIN + [(96, 80, 64), (200, 70, 50), (130, 300, 20), (48, 48, 200)])
def test_maps_with_other_sites(dims, rows, fused):
    """One voxel holds a site of another voxel; then the EDT of the transformed map, of which every voxel may."""
    n = dims[0] * dims[1] * dims[2]
    want = oracle.dvm_empty(dims)
    oracle.dvm_insert(want, dims, 1.0, _points(dims, max(1, n // 50), n))
    x, y, z = (d - 1 for d in dims)
    want[n // 3] = x | y << 10 | z << 20
    m = gvx.DistanceVoxelMap(dims, 1.0)
    m.set_edt_config(rows, fused)
    m.data().copy_(torch.as_tensor(want.view(np.int32)).cuda())
    for _ in range(2):
        m.parallelBanding3D()
        oracle.pba(want, dims)
        assert m.edt_check() == 0
        got = to_u32(m.data())
        assert np.array_equal(got, want), first_mismatch(got, want, dims)


@pytest.mark.parametrize("rows,fused", CONFIGS)
@pytest.mark.parametrize("dims", [(513, 20, 9), (17, 600, 12), (1023, 33, 5), (520, 515, 2)])
def test_long_maps(dims, rows, fused):
    for n in (3, dims[0] * dims[1] * dims[2] // 100):
        pts = _points(dims, n, n)
        _, want = oracle_edt(dims, 1.0, pts)
        p = torch.as_tensor(pts).cuda()
        m = gvx.DistanceVoxelMap(dims, 1.0)
        m.set_edt_config(rows, fused)
        m.voxelize_edt(p)
        got = to_u32(m.data())
        assert np.array_equal(got, want), first_mismatch(got, want, dims)
        m.clearMap()
        m.insertPointCloud(p)
        m.parallelBanding3D()
        assert m.edt_check() == 0
        got = to_u32(m.data())
        assert np.array_equal(got, want), first_mismatch(got, want, dims)


@pytest.mark.parametrize("rows", ["16", "32"])
def test_batches(rows):
    """A batch has no configuration of its own but the tuner's: the library's default is set for a process.  A long map
    sends the whole batch to the sweeps; without it, the maps that were transformed before."""
    script = textwrap.dedent(f"""
        import sys
        sys.path[:0] = [{os.path.join(ROOT, 'gpu-voxels_b200')!r}, {os.path.join(ROOT, 'oracle')!r}, {os.path.join(ROOT, 'tests')!r}]
        import numpy as np, torch, gvx, oracle
        from gvx.batch import Batch
        from gpu_helpers import oracle_edt, to_u32
        for extra in ([], [(600, 12, 10)]):
            dims = {THIN!r} + [(96, 80, 64), (130, 70, 50), (64, 128, 33)] + extra
            rng = np.random.default_rng(3)
            clouds = [(rng.random((max(1, int(np.prod(d)) // 60), 3)) * d).astype(np.float32) for d in dims]
            maps = [gvx.DistanceVoxelMap(d, 1.0) for d in dims]
            b = Batch(maps)
            xyz = torch.as_tensor(np.concatenate(clouds)).cuda()
            off = torch.as_tensor(np.concatenate([[0], np.cumsum([len(c) for c in clouds])]).astype(np.int64)).cuda()
            wants = [oracle_edt(d, 1.0, c)[1] for d, c in zip(dims, clouds)]
            def check(what):
                assert b.edt_check() == 0
                for m, d, w in zip(maps, dims, wants):
                    assert np.array_equal(to_u32(m.data()), w), (what, d)
            b.voxelize_edt(xyz, off)
            check("voxelize")
            b.clear()
            b.insert(xyz, off)
            for m, d, w in list(zip(maps, dims, wants))[::2]:
                m.parallelBanding3D()
                oracle.pba(w, d)
            b.edt()
            check("some transformed before")
            b.edt()
            for d, w in zip(dims, wants):
                oracle.pba(w, d)
            check("all transformed before")
    """)
    r = subprocess.run([sys.executable, "-c", script], env=dict(os.environ, GVX_EDT_SWEEP_ROWS=rows), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
