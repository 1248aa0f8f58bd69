"""Voxel lists built by the bitmap of the reference map against the oracle's sort, ids and voxels: maps that end
inside a bitmap word and inside a tile of 1024 words, empty and full lists, points outside, repeated inserts with
other meanings, and lists whose ids may lie outside the map (gvx_blist_set), which are sorted."""
import ctypes

import numpy as np
import pytest
import torch

import gvx
import oracle
from gvx import _abi, maps

pytestmark = pytest.mark.gpu


def _equal(lst, ids, vox):
    assert lst.getDimensions() == (0 if ids is None else ids.shape[0])
    if ids is not None:
        assert np.array_equal(lst.ids().cpu().numpy().view(np.uint32), ids)
        assert np.array_equal(lst.voxels().cpu().numpy(), vox)


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 2), (33, 31, 32), (32, 32, 32), (40, 41, 43), (64, 64, 8)])
def test_inserts_equal_oracle(dims):
    lst = gvx.BitVectorVoxelList(dims, 0.5)
    ids = vox = None
    n_vox = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(n_vox)
    for n, meaning in ((1, 7), (n_vox // 3 + 1, 4), (3, 255), (4 * n_vox, 0), (50, 33)):
        pts = ((rng.random((n, 3)) * 1.2 - 0.05) * dims * 0.5).astype(np.float32)
        lst.insertPointCloud(torch.as_tensor(pts), meaning)
        ids, vox = oracle.list_insert(ids, vox, dims, 0.5, pts, meaning)
        _equal(lst, ids, vox)
    lst.clearMap()
    lst.insertPointCloud(torch.as_tensor(np.full((4, 3), 1e6, np.float32)), 4)  # nothing inside
    assert lst.getDimensions() == 0
    lst.insertPointCloud(torch.as_tensor(pts), 9)
    _equal(lst, *oracle.list_insert(None, None, dims, 0.5, pts, 9))


def test_set_lists_are_sorted():
    """Ids beyond the map survive an insert, as they do in the sort."""
    dims = (20, 20, 20)
    ids = np.array([3, 77, 7999, 8000, 123_456], np.uint32)
    vox = np.zeros((5, 32), np.uint8)
    vox[:, 2] = 1
    lst = gvx.BitVectorVoxelList(dims, 1.0)
    lst.set(torch.as_tensor(ids.astype(np.int64)), torch.as_tensor(vox.reshape(-1)).cuda())
    pts = (np.random.default_rng(2).random((500, 3)) * 20).astype(np.float32)
    lst.insertPointCloud(torch.as_tensor(pts), 5)
    _equal(lst, *oracle.list_insert(ids, vox.reshape(-1), dims, 1.0, pts, 5))


def _written(ids, how):
    """What a caller may leave in a list's ids."""
    out = ids.copy()
    if how == "beyond":  # the swept volume moved by an offset, half of it past the map's end
        out += np.uint32(20 * 20 * 20 // 2)
    elif how == "far":
        out[1::7] = 0xFFFFFFF0
    elif how == "descending":
        out = out[::-1].copy()
    elif how == "repeated":
        out[5:40] = out[4]
    elif how == "last":  # the map's first id that is none
        out[-1] = 20 * 20 * 20
    else:  # moved inside the map: still ascending
        out -= np.uint32(1)
    return out


@pytest.mark.parametrize("how", ["beyond", "far", "descending", "repeated", "last", "inside"])
def test_ids_written_by_the_caller(how):
    """gvx_blist_data hands out the ids' storage; an insert after a caller wrote it merges as the sort does, the list
    and the entries' voxels with it, and so do the inserts after that."""
    dims = (20, 20, 20)
    rng = np.random.default_rng(11)
    lst = gvx.BitVectorVoxelList(dims, 1.0)
    lst.insertPointCloud(torch.as_tensor((rng.random((300, 3)) * 20).astype(np.float32)), 3)
    ids, vox = lst.ids().cpu().numpy().view(np.uint32), lst.voxels().cpu().numpy().reshape(-1, 32)
    assert ids[0] > 0
    ids = _written(ids, how)
    vox[:, 7] = rng.integers(1, 256, len(ids))  # tells the entries apart
    pi, pv = ctypes.c_void_p(), ctypes.c_void_p()
    _abi.call("gvx_blist_data", lst.handle, ctypes.byref(pi), ctypes.byref(pv))
    maps._device_view(pi.value, len(ids)).copy_(torch.as_tensor(ids.view(np.int32)))
    maps._device_view_u8(pv.value, len(ids) * 32).copy_(torch.as_tensor(vox.reshape(-1)))
    vox = vox.reshape(-1)
    for n, meaning in ((500, 5), (40, 9)):
        pts = (rng.random((n, 3)) * 20).astype(np.float32)
        lst.insertPointCloud(torch.as_tensor(pts), meaning)
        ids, vox = oracle.list_insert(ids, vox, dims, 1.0, pts, meaning)
        _equal(lst, ids, vox)


def test_long_list_waits_for_its_length():
    """More points than entries whose storage is taken at the upper bound."""
    dims = (128, 128, 128)
    pts = (np.random.default_rng(3).random((1_200_000, 3)) * dims).astype(np.float32)
    lst = gvx.BitVectorVoxelList(dims, 1.0)
    lst.insertPointCloud(torch.as_tensor(pts[:1_100_000]), 4)
    ids, vox = oracle.list_insert(None, None, dims, 1.0, pts[:1_100_000], 4)
    _equal(lst, ids, vox)
    lst.insertPointCloud(torch.as_tensor(pts[1_100_000:]), 6)
    _equal(lst, *oracle.list_insert(ids, vox, dims, 1.0, pts[1_100_000:], 6))
