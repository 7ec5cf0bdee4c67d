"""The plan's header reaches the host whatever kind of memory it is to be written to: aligned pinned memory (written by the plan's
last kernel), pinned memory at an odd address and pageable memory (copied)."""

import ctypes

import numpy as np
import pytest
import torch

from dynamis_b200 import _lib
from dynamis_b200.graph import plan_radius_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 20_000])
@pytest.mark.parametrize("bins_only", [False, True])
@pytest.mark.parametrize("memory", ["pinned", "pinned_odd", "pageable"])
def test_header(cuda, memory, bins_only, n):
    L = _lib.lib()
    length = (n / 0.1) ** (1.0 / 3.0) + 6.0
    pos = (torch.rand(n, 3, generator=torch.Generator().manual_seed(n)) * length).to(cuda)
    cell, pbc = np.eye(3, dtype=np.float32) * np.float32(length), np.ones(3, dtype=np.uint8)
    src, cells, nbytes = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_int64()
    _lib.check(L.dynb_rg_suggest_capacity(n, cell.ctypes.data, pbc.ctypes.data, 5.0, _lib.DYNB_F32, ctypes.byref(src), ctypes.byref(cells)))
    _lib.check(L.dynb_rg_workspace_bytes(n, n, src.value, cells.value, _lib.DYNB_F32, ctypes.byref(nbytes)))
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device=cuda)
    counts = torch.empty(n, dtype=torch.int32, device=cuda)
    host = torch.full((256,), 255, dtype=torch.uint8, pin_memory=memory != "pageable")
    at = host.data_ptr() + (8 if memory == "pinned_odd" else 0)
    stream = torch.cuda.current_stream()
    if bins_only:
        _lib.check(L.dynb_rg_bin(pos.data_ptr(), _lib.DYNB_F32, n, cell.ctypes.data, pbc.ctypes.data, 5.0, ws.data_ptr(), ws.numel(), src.value,
                                 cells.value, at, stream.cuda_stream))
    else:
        _lib.check(L.dynb_rg_plan(pos.data_ptr(), _lib.DYNB_F32, n, cell.ctypes.data, pbc.ctypes.data, 5.0, None, n, ws.data_ptr(), ws.numel(), src.value,
                                  cells.value, counts.data_ptr(), at, stream.cuda_stream))
    stream.synchronize()
    h = _lib.RgHeader.from_address(at)
    on_device = torch.zeros(64, dtype=torch.uint8)
    base = (-ws.data_ptr()) % 256   # the layout starts at the first 256-byte boundary
    on_device.copy_(ws[base:base + 64])
    assert bytes(on_device.numpy()) == ctypes.string_at(at, 64)
    assert h.status == 0 and h.M >= n and h.num_groups > 0
    assert h.E == (0 if bins_only else int(counts.sum()))
    before, behind = at - host.data_ptr(), at + 64 - host.data_ptr()
    assert (host[:before] == 255).all() and (host[behind:] == 255).all()


@pytest.mark.parametrize("n", [8192 * 2048 - 1, 8192 * 2048])
def test_header_of_the_largest_scans(cuda, n):
    """Up to 8192 tiles of degrees (one more than targets) the scan writes the header itself; beyond that it is copied."""
    gen = torch.Generator(device=cuda).manual_seed(1)
    length = (n / 0.02) ** (1.0 / 3.0)
    pos = torch.rand(n, 3, generator=gen, device=cuda) * length
    plan = plan_radius_graph(pos, torch.eye(3) * length, torch.tensor([True] * 3), 2.0)
    base = (-plan.ws.data_ptr()) % 256
    E, M = plan.ws[base:base + 16].view(torch.int64).tolist()
    assert plan.E == E == int(plan.counts.sum(dtype=torch.int64)) > 0 and plan.M == M >= n
    assert plan.max_degree == int(plan.counts.max())
