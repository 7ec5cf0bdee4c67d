"""Partitions in workspaces that start on an 8-byte and on a 16-byte boundary, at the C entry, and a KD-tree whose tree does not fit the
kernel argument that usually brings it: labels as the Python layer, whose workspaces start on a 256-byte boundary, gives them."""

import ctypes

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from dynamis_b200 import _lib

pytestmark = pytest.mark.gpu

N = 30_011


def positions(cuda):
    return torch.as_tensor(np.random.default_rng(3).random((N, 3)).astype(np.float32) * 40.0, device=cuda)


def workspace(cuda, nbytes, off):
    ws = torch.empty((nbytes + 512,), dtype=torch.uint8, device=cuda)
    return ws, ws.data_ptr() + (-ws.data_ptr()) % 256 + off


@pytest.mark.parametrize("off", [0, 8, 16, 24])
@pytest.mark.parametrize("W", [2, 13, 64, 300])
@pytest.mark.parametrize("weighted, method", [(False, 0), (False, 1), (True, 0)])
def test_kdtree(cuda, off, W, weighted, method):
    pos = positions(cuda)
    weights = torch.arange(N, device=cuda) % 7 + 1 if weighted else None
    nbytes = ctypes.c_int64()
    _lib.check(_lib.lib().dynb_kdtree_workspace_bytes(N, W, ctypes.byref(nbytes)))
    ws, at = workspace(cuda, nbytes.value, off)
    labels = torch.full((N,), -1, dtype=torch.int64, device=cuda)
    _lib.check(_lib.lib().dynb_kdtree_partition(pos.data_ptr(), N, weights.data_ptr() if weighted else None, W, labels.data_ptr(), method,
                                                at, nbytes.value, _lib.stream_of(pos.device)))
    assert torch.equal(labels, D.kdtree_partition_labels(pos, weights, W, sorted_cuts=True))


@pytest.mark.parametrize("off", [8, 16])
@pytest.mark.parametrize("W", [2, 16, 200])
def test_curve(cuda, off, W):
    pos = positions(cuda)
    nbytes = ctypes.c_int64()
    _lib.check(_lib.lib().dynb_sfc_workspace_bytes(N, ctypes.byref(nbytes)))
    ws, at = workspace(cuda, nbytes.value, off)
    labels = torch.full((N,), -1, dtype=torch.int64, device=cuda)
    _lib.check(_lib.lib().dynb_sfc_partition(pos.data_ptr(), N, None, W, 0, labels.data_ptr(), None, at, nbytes.value, _lib.stream_of(pos.device)))
    assert torch.equal(labels, D.sfc_partition_labels(pos, None, W, return_perm=True)[0])


def test_workspace_off_every_boundary_is_refused(cuda):
    pos = positions(cuda)
    nbytes = ctypes.c_int64()
    _lib.check(_lib.lib().dynb_kdtree_workspace_bytes(N, 4, ctypes.byref(nbytes)))
    ws, at = workspace(cuda, nbytes.value, 4)
    labels = torch.empty((N,), dtype=torch.int64, device=cuda)
    with pytest.raises(RuntimeError, match="8-byte boundary"):
        _lib.check(_lib.lib().dynb_kdtree_partition(pos.data_ptr(), N, None, 4, labels.data_ptr(), 0, at, nbytes.value, _lib.stream_of(pos.device)))
