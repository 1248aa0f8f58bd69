"""The arm kernels' packed corner reads over caller-written maps: every kind of
site word (near, far, empty, one field of 1023, bits above the fields), spheres
in and outside the map, at every position of an aligned 16-byte word, in the
map's last words and on one-voxel axes."""
import ctypes

import numpy as np
import pytest
import torch

import gvx
import oracle
from gvx import _abi

pytestmark = pytest.mark.gpu

SIDE = 0.05


def _words(rng, n, odd):
    v = rng.integers(0, 1023, n) | rng.integers(0, 1023, n) << 10 | rng.integers(0, 1023, n) << 20
    if odd:
        kind = rng.integers(0, 24, n)
        v = np.where(kind == 0, 0x3FFFFFFF, v)
        for f in range(3):
            v = np.where(kind == 1 + f, v | 0x3FF << 10 * f, v)
        v = np.where(kind == 4, v | 0x40000000, v)
        v = np.where(kind == 5, v & 0x3FF003FF | 1022 << 10, v)
    return v.astype(np.uint32)


def test_roots_and_lattice_coordinates_equal_the_general_forms():
    """Every root the arm kernels can take is sqrtf's, and their position divided by the side is the IEEE divide's, ties
    and cell faces included."""
    roots, coordinates = ctypes.c_uint64(1), ctypes.c_uint64(1)
    _abi.call("gvx_check_query_arithmetic", ctypes.byref(roots), ctypes.byref(coordinates))
    assert (roots.value, coordinates.value) == (0, 0)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 7, 5), (2, 3, 4), (5, 1, 3), (6, 5, 1), (33, 6, 7), (61, 33, 29), (1023, 5, 3)])
def test_single_sphere_anywhere(dims, odd):
    """Two joints swing one sphere through a ball around the map.  A corner, its
    three interpolation steps and the fractions round by at most 2^-24 of the
    largest corner's distance each: 2^-20 of it bounds the sum."""
    rng = np.random.default_rng(sum(dims) + odd)
    words = _words(rng, int(np.prod(dims)), odd)
    m = gvx.DistanceVoxelMap(dims, SIDE, voxels=torch.as_tensor(words.view(np.int32)).cuda())
    base = np.eye(4)
    base[:3, 3] = np.asarray(dims) * SIDE / 2
    largest = 2.0 ** 15.5 if odd else np.sqrt(3.0) * 1023  # an empty corner; a site's
    for reach in (0.04, 0.3, 0.7):
        a = reach * (SIDE + np.linalg.norm(dims) * SIDE)
        spec = {"n_joints": 2, "base": base.reshape(-1).tolist(), "theta": [0.1, 0.2], "d": [0.0, 0.0], "a": [0.0, float(a)],
                "alpha": [np.pi / 2, 0.0], "link": [1], "t": [1.0], "r": [0.0]}
        q = rng.uniform(-np.pi, np.pi, (3000, 2)).astype(np.float32)
        got = m.sphere_clearance(gvx.make_arm(spec), torch.as_tensor(q)).cpu().numpy().astype(np.float64)
        want = oracle.sphere_clearance64(words, dims, SIDE, spec, q)
        assert np.abs(got - want).max() / SIDE <= 2.0 ** -20 * largest
        cost = m.traj_cost(gvx.make_arm(spec), torch.as_tensor(q[:, None]), 1.0).cpu().numpy().astype(np.float64)
        assert np.abs(cost - oracle.traj_cost64(words, dims, SIDE, spec, q[:, None], 1.0)).max() / SIDE <= 2.0 ** -20 * largest
