"""Arms of different sizes on several host threads at once.  From 12 joints on the kernels' shared memory is above the
48 KB that need no leave, and differs by joints, spheres and waypoints; a kernel's limit is one for all threads."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import gvx
from gvx import _abi

pytestmark = pytest.mark.gpu


def _arm(joints, spheres, seed):
    rng = np.random.default_rng(seed)
    base = np.eye(4)
    base[:3, 3] = 0.3
    return gvx.make_arm({"n_joints": joints, "base": base.reshape(-1).tolist(), "theta": rng.uniform(-1, 1, joints).tolist(),
                         "d": [0.02] * joints, "a": [0.03] * joints, "alpha": rng.uniform(-1, 1, joints).tolist(),
                         "link": rng.integers(0, joints, spheres).tolist(), "t": rng.random(spheres).tolist(),
                         "r": [0.02] * spheres})


def test_large_arms_on_threads():
    """One trajectory of 64 waypoints (a block of 64 configurations), called as fast as the threads can."""
    m = gvx.DistanceVoxelMap((60, 60, 60), 0.01)
    m.insertPointCloud(torch.as_tensor((np.random.default_rng(0).random((200, 3)) * 0.6).astype(np.float32)))
    m.parallelBanding3D()
    fn = _abi.lib().gvx_traj_cost
    jobs = []
    for joints, spheres in ((16, 256), (12, 8), (13, 40), (16, 64), (12, 4), (15, 200)):
        q = torch.as_tensor(np.random.default_rng(joints).uniform(-3, 3, (1, 64, joints)).astype(np.float32)).cuda()
        out, stream = torch.empty(1, device="cuda"), torch.cuda.Stream()
        arm = _arm(joints, spheres, spheres)
        args = (m.handle, ctypes.byref(arm), ctypes.c_void_p(q.data_ptr()), 1, 64, 0.05, ctypes.c_void_p(out.data_ptr()),
                ctypes.c_void_p(stream.cuda_stream))
        jobs.append((args, m.traj_cost(arm, q, 0.05), out, (q, arm, stream)))
    torch.cuda.synchronize()
    failed = [0] * len(jobs)
    start = threading.Barrier(len(jobs))

    def loop(i):
        args = jobs[i][0]
        start.wait()
        for _ in range(8000):
            failed[i] += fn(*args) != 0

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == [0] * len(jobs)
    for _, want, out, _ in jobs:
        assert torch.equal(out, want)
