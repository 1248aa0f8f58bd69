"""The arm kernels' blocks (configurations in groups of 8 to 64, joints rounded up to 8 or 16, lanes over spheres)
at their edges, against the FP64 oracle with the bounds of test_gpu_continuous.py."""
import numpy as np
import pytest
import torch

import gvx
import oracle
from gpu_helpers import gpu_edt

pytestmark = pytest.mark.gpu

DIMS, SIDE, MARGIN = (60, 52, 44), 0.02, 0.05


@pytest.fixture(scope="module")
def field():
    rng = np.random.default_rng(1)
    _, edt, dvm = gpu_edt(DIMS, SIDE, (rng.random((400, 3)) * DIMS * SIDE).astype(np.float32))
    return edt, dvm


def _spec(joints, spheres, seed):
    rng = np.random.default_rng(seed)
    base = np.eye(4)
    base[:3, 3] = [0.6, 0.52, 0.1]
    return {"n_joints": joints, "base": base.reshape(-1).tolist(), "theta": rng.uniform(-1, 1, joints).tolist(),
            "d": rng.uniform(0.0, 0.4 / joints, joints).tolist(), "a": rng.uniform(0.3 / joints, 0.7 / joints, joints).tolist(),
            "alpha": rng.choice([np.pi / 2, -np.pi / 2, 0.3], joints).tolist(),
            "link": rng.integers(0, joints, spheres).tolist(), "t": rng.random(spheres).tolist(),
            "r": rng.uniform(0.005, 0.04, spheres).tolist()}


@pytest.mark.parametrize("joints,spheres,n_traj,n_wp", [(1, 1, 1, 1), (7, 33, 3, 7), (8, 32, 2, 65), (9, 31, 5, 9),
                                                        (16, 256, 2, 70), (7, 56, 40, 8)])
def test_arm_kernels(field, joints, spheres, n_traj, n_wp):
    edt, dvm = field
    spec = _spec(joints, spheres, joints * 1000 + spheres)
    arm = gvx.make_arm(spec)
    rng = np.random.default_rng(n_traj * 100 + n_wp)
    q = rng.uniform(-np.pi, np.pi, (n_traj, n_wp, joints)).astype(np.float32)
    flat = q.reshape(-1, joints)
    got = dvm.sphere_clearance(arm, torch.as_tensor(flat)).cpu().numpy().astype(np.float64)
    assert np.abs(got - oracle.sphere_clearance64(edt, DIMS, SIDE, spec, flat)).max() / SIDE < 1e-5
    gcost = rng.uniform(0.5, 1.5, n_traj).astype(np.float32)
    want, scale, gap = oracle.traj_cost_grad64(edt, DIMS, SIDE, spec, q, MARGIN, gcost)
    cost = dvm.traj_cost(arm, torch.as_tensor(q), MARGIN).cpu().numpy().astype(np.float64)
    cost64 = oracle.traj_cost64(edt, DIMS, SIDE, spec, q, MARGIN)
    n = spheres * n_wp  # at most every term active, each 1e-5 voxel off, plus the float sum of n terms
    assert np.all(np.abs(cost - cost64) <= 1e-5 * SIDE * n + n * 2.0 ** -23 * cost64 + 1e-12)
    gq = dvm.traj_cost_backward(arm, torch.as_tensor(q), MARGIN, torch.as_tensor(gcost)).cpu().numpy().astype(np.float64)
    # no hinge flips within a rounding, no centre within 1e-6 voxel of a cell face (where the gradient jumps)
    u = oracle.sphere_centres64(spec, q) / np.float64(np.float32(SIDE)) - 0.5
    face = np.abs(u - np.round(u)).min(axis=(2, 3)) > 1e-6
    ok = ((gap > 1e-6) & face)[..., None] & np.ones_like(want, dtype=bool)
    assert ok.mean() > 0.9
    assert np.all(np.abs(gq - want)[ok] <= (1e-5 * scale + 2.0 ** -23 * np.abs(want))[ok] + 1e-12)
