"""KD-tree labels by selection where its passes change form: one upload of the tree for numbers of ranks with uneven levels, boxes of
more segments than fit shared memory, segments of one atom, groups of equal coordinates that overflow the list of the early
finish.  Against the sorted cuts of the same library (method 1), which share none of these passes."""

import ctypes

import pytest
import torch

from dynamis_b200 import _lib

pytestmark = pytest.mark.gpu


def _labels(pos, W, method):
    n = pos.size(0)
    nbytes = ctypes.c_int64()
    _lib.check(_lib.lib().dynb_kdtree_workspace_bytes(n, W, ctypes.byref(nbytes)), "kdtree_workspace_bytes")
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device=pos.device)
    out = torch.full((n,), -1, dtype=torch.int64, device=pos.device)
    _lib.check(_lib.lib().dynb_kdtree_partition(pos.data_ptr(), n, None, W, out.data_ptr(), method, ws.data_ptr(), ws.numel(),
                                                torch.cuda.current_stream().cuda_stream), "kdtree_partition")
    return out


@pytest.mark.parametrize("n,W", [(2, 2), (5, 4), (7, 7), (1000, 2), (1023, 13), (4097, 5), (20_000, 300), (20_000, 1024), (200_003, 16)])
@pytest.mark.parametrize("kind", ["random", "planes", "one_point"])
def test_selection_equals_sorted_cuts(cuda, n, W, kind):
    pos = torch.rand(n, 3, generator=torch.Generator().manual_seed(n + W)) * torch.tensor([90.0, 50.0, 70.0])
    if kind == "planes":       # thousands of atoms share a coordinate
        pos = torch.floor(pos / 10.0) * 10.0
    elif kind == "one_point":
        pos[:] = pos[0].clone()
    pos = pos.to(cuda)
    assert torch.equal(_labels(pos, W, 0), _labels(pos, W, 1))
