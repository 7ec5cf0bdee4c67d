"""Domain partitioners and halo-map construction — host side.

Mirrors the reference's partitioner classes (dynamis_state/include/dynamis_state/partitioner.hpp:6-78,
bound in dynamis_state/src/dynamis_state_bindings.cpp:75-115): ``SFCPartitioner(curve_type)`` and
``SimpleSpatialPartitioner`` with ``partition(state, env[, config])`` and
``build_halo_maps(info, global_state, env, config)`` (fills ``info`` in place).

The compute is in libdynb.so: Morton/"Hilbert" keys, a stable radix sort, the label assignment
(dynb_sfc_partition), bincount / stream compaction (dynb_bincount_i64, dynb_select_eq_i64), and
for the halo maps one cell-scan pass at cutoff + buffer that marks which rank needs which atom
(dynb_rg_halo_mark_rank) followed by the assembly of the lists (dynb_halo_lists_plan / _fill).  Unlike the
reference, no [N, W] bool matrix and no edge list are materialised.
"""

from __future__ import annotations

import ctypes
import enum
from typing import Optional

import numpy as np
import torch

from . import _lib
from .graph import BinnedAtoms, give_host_words, lose_host_words, radius_graph_pbc, radius_graph_pbc_ex, take_host_words
from .state import DistEnvironment, MolecularInfo, PartitionMessagePassingInfo, SimulationConfig

PARTITION_MAX_NUM_NEIGHBORS = 1000
HALO_MAX_NUM_NEIGHBORS = 1000
SELECT_HOST_COUNT = 8192 * 2048   # SELECT_FUSED_MAX_TILES tiles of SELECT_TILE values (csrc/halo.cu)

_SCRATCH: dict = {}


def scratch(device: torch.device, name: str, nbytes: int) -> torch.Tensor:
    """Grow-only named device scratch buffers (uint8), one set per (device, stream): work on different streams of
    a device never shares one."""
    key = (device.index, _lib.stream_of(device), name)
    buf = _SCRATCH.get(key)
    if buf is None or buf.numel() < nbytes:
        _SCRATCH.pop(key, None)
        buf = torch.empty(max(int(nbytes * 1.1) + 256, 256), dtype=torch.uint8, device=device)
        _SCRATCH[key] = buf
    return buf


_stream = _lib.stream_of


def _single(x) -> float:
    """x (a number, or a tensor of one element on any device) rounded to single precision."""
    return float(np.float32(float(x)))


class SFCCurveType(enum.IntEnum):
    Morton = 0
    Hilbert = 1


def launches_per_partition() -> int:
    """Kernels one Morton partition of a million atoms into 8 labels launches (labels only): bounds (2, the first
    clears them), keys (1), 6 digit levels (the first behind a launch that clears its table; histogram; its last block
    advances the split points; once the remaining atoms are few the last block settles the split points and the later
    levels return at once), labels (1).  With the curve-order permutation requested the sorted path runs instead: bounds,
    keys, 8 radix passes x (histogram + 2 scan kernels + scatter), assignment."""
    return 2 + 1 + 1 + 6 + 1


def sfc_partition_labels(pos: torch.Tensor, weights: Optional[torch.Tensor], W: int, curve_type: int = 0,
                         return_perm: bool = False):
    """Rank label in [0, W) per atom (reference: sfc_partition_cuda, partition/sfc.cpp:9-33)."""
    if not pos.is_cuda:
        raise RuntimeError("pos must be a CUDA tensor")
    if pos.dim() != 2 or pos.size(1) != 3:
        raise RuntimeError(f"pos must have shape [N, 3], got [{pos.size(0)}, {pos.size(1) if pos.dim() > 1 else ''}]")
    if pos.dtype != torch.float32:
        raise RuntimeError(f"pos must be float32, got {pos.dtype}")
    if W < 1:
        raise RuntimeError(f"W must be >= 1, got {W}")
    if curve_type not in (0, 1):
        raise RuntimeError(f"curve_type must be 0 (Morton) or 1 (Hilbert), got {curve_type}")
    pos = pos.contiguous()
    N = pos.size(0)
    dev = pos.device
    if weights is not None:
        if not weights.is_cuda:
            raise RuntimeError("weights must be a CUDA tensor")
        if weights.dim() != 1 or weights.size(0) != N:
            raise RuntimeError(f"weights must have shape [N], got [{weights.size(0)}]")
        weights = weights.to(torch.int64).contiguous()
    L = _lib.lib()
    with _lib.on_device(dev):
        labels = torch.empty((N,), dtype=torch.int64, device=dev)
        perm = torch.empty((N,), dtype=torch.int64, device=dev) if return_perm else None
        if N > 0:
            nbytes = ctypes.c_int64()
            _lib.check(L.dynb_sfc_workspace_bytes(N, ctypes.byref(nbytes)), "sfc_workspace_bytes")
            ws = scratch(dev, "sfc", nbytes.value)
            _lib.check(L.dynb_sfc_partition(pos.data_ptr(), N, weights.data_ptr() if weights is not None else None, int(W),
                                            int(curve_type), labels.data_ptr(), perm.data_ptr() if perm is not None else None,
                                            ws.data_ptr(), ws.numel(), _stream(dev)), "sfc_partition")
    return (labels, perm) if return_perm else labels


def sfc_keys(pos: torch.Tensor, curve_type: int = 0) -> torch.Tensor:
    """Curve keys in atom order, int64 (reference kernels: sfc_kernels.cu:32-109)."""
    pos = pos.contiguous()
    N, dev = pos.size(0), pos.device
    keys = torch.empty((N,), dtype=torch.int64, device=dev)
    if N:
        L = _lib.lib()
        with _lib.on_device(dev):
            nbytes = ctypes.c_int64()
            _lib.check(L.dynb_sfc_workspace_bytes(N, ctypes.byref(nbytes)), "sfc_workspace_bytes")
            ws = scratch(dev, "sfc", nbytes.value)
            _lib.check(L.dynb_sfc_keys(pos.data_ptr(), N, int(curve_type), keys.data_ptr(), ws.data_ptr(), ws.numel(),
                                       _stream(dev)), "sfc_keys")
    return keys


def bincount_labels(labels: torch.Tensor, W: int) -> torch.Tensor:
    dev = labels.device
    L = _lib.lib()
    with _lib.on_device(dev):
        counts = torch.empty((W,), dtype=torch.int64, device=dev)
        bad = scratch(dev, "bad", 256)
        _lib.check(L.dynb_bincount_i64(labels.data_ptr(), labels.numel(), W, counts.data_ptr(), bad.data_ptr(), _stream(dev)),
                   "bincount")
    return counts


def select_eq(values: torch.Tensor, value: int, gather_src: Optional[torch.Tensor] = None,
              count: Optional[int] = None) -> torch.Tensor:
    """``gather_src[nonzero(values == value)]`` (or the positions themselves), ascending.  One host sync, none when the
    caller knows how many there are (``count``; the buffer has room for every position all the same)."""
    dev = values.device
    n = values.numel()
    L = _lib.lib()
    with _lib.on_device(dev):
        out = torch.empty((n,), dtype=torch.int64, device=dev)
        # a count that is waited for is written to the host by the kernel (up to 16.7 M values: its tiles then need no prefix sum)
        waited = count is None and 0 < n <= SELECT_HOST_COUNT
        nbytes = ctypes.c_int64()
        _lib.check(L.dynb_select_workspace_bytes(n, ctypes.byref(nbytes)), "select_workspace_bytes")
        ws = scratch(dev, "select", nbytes.value)

        cnt = take_host_words(1) if waited else torch.empty((1,), dtype=torch.int64, device=dev)
        try:
            _lib.check(L.dynb_select_eq_i64(values.data_ptr(), n, int(value), gather_src.data_ptr() if gather_src is not None else None,
                                            out.data_ptr(), cnt.data_ptr(), ws.data_ptr(), ws.numel(), _stream(dev)), "select_eq")
            if waited:
                torch.cuda.current_stream(dev).synchronize()
        except BaseException:
            if waited:
                lose_host_words(cnt, dev)
            raise
        if waited:
            k = int(cnt[0])
            give_host_words(cnt)
        else:
            k = int(cnt.item()) if count is None else count
    return out[:k]


def _finish_partition(labels: torch.Tensor, state: MolecularInfo, env: DistEnvironment,
                      n_local: Optional[int] = None) -> PartitionMessagePassingInfo:
    """partition_indices / atom_counts / matrix from the labels (sfc_partitioner.cpp:164-178).  ``n_local``: the number of
    atoms with this rank's label where it is known beforehand (saves the wait for it)."""
    info = PartitionMessagePassingInfo()
    W, R = int(env.world_size), int(env.global_rank)
    dev = labels.device
    info.partition_id = labels
    info.atom_counts = bincount_labels(labels, W)
    vn = state.atom_vertex_numbers
    vn = vn.to(device=dev, dtype=torch.int64).contiguous() if vn is not None else None
    info.partition_indices = select_eq(labels, R, vn, n_local)
    m = torch.zeros((W, W), dtype=torch.int64, device=dev)
    m[R, R].fill_(info.partition_indices.numel())   # (an assignment copies the number from pageable memory)
    info.global_send_recv_matrix = m
    return info


class AbstractPartitioner:
    def build_halo_maps(self, info: PartitionMessagePassingInfo, global_state: MolecularInfo, env: DistEnvironment,
                        config: SimulationConfig) -> None:
        """Send/recv CSR, interior mask and matrix row for rank ``env.global_rank``
        (reference: dynamis_state/src/csrc/build_halo_maps.cpp:20-157)."""
        pos = global_state.atom_positions
        if not pos.is_cuda:
            raise RuntimeError("pos must be a CUDA tensor")
        dev = pos.device
        N, W, R = int(global_state.num_atoms), int(env.world_size), int(env.global_rank)
        # refused before anything is queued: the header and the list sizes are written to buffers of this call
        if not 0 <= R < W:
            raise RuntimeError(f"global_rank must be in [0, world_size), got {R} of {W}")
        if W > 4096:
            raise RuntimeError("world_size above 4096 is not supported")
        ghost_cutoff = _single(config.cutoff + config.ghost_cutoff_buffer)
        pos32 = pos.to(torch.float32).contiguous()
        cell = config.cell.to(torch.float32)
        pbc = config.pbc.to(torch.bool)
        pid = info.partition_id.to(device=dev, dtype=torch.int64).contiguous()
        L = _lib.lib()
        words = (W + 31) // 32
        with _lib.on_device(dev):
            needed = torch.empty((max(N, 1), words), dtype=torch.int32, device=dev)
            has_foreign = torch.empty((max(N, 1),), dtype=torch.uint8, device=dev)
            nbytes = ctypes.c_int64()
            _lib.check(L.dynb_halo_lists_workspace_bytes(N, W, ctypes.byref(nbytes)), "halo_lists_workspace_bytes")
            ws = scratch(dev, "halo_lists", nbytes.value)
            # send offsets, recv offsets, number of own atoms and, behind them, the error word of the marking
            offs = torch.empty((2 * (W + 1) + 2,), dtype=torch.int64, device=dev)
            # everything up to the list sizes is queued before the one wait; the header's status is looked at behind it
            bins = BinnedAtoms(pos32, cell, pbc, ghost_cutoff) if N > 0 else None
            offs_h = take_host_words(2 * (W + 1) + 2)
            try:
                while True:
                    if bins is not None:
                        bins.launch()
                        _lib.check(L.dynb_rg_halo_mark_rank(bins.ws.data_ptr(), bins.dtype_code, pid.data_ptr(), N, W, R, needed.data_ptr(),
                                                            has_foreign.data_ptr(), offs.data_ptr() + 8 * (2 * W + 3), _stream(dev)), "rg_halo_mark")
                    _lib.check(L.dynb_halo_lists_plan_words(needed.data_ptr(), None, pid.data_ptr(), N, R, W, offs.data_ptr(), ws.data_ptr(),
                                                            ws.numel(), offs_h.data_ptr(), 2 * (W + 1) + 2, _stream(dev)), "halo_lists_plan")
                    torch.cuda.current_stream(dev).synchronize()
                    if bins is None or bins.done():
                        break
            except BaseException:   # the header of the bins waits as well
                lose_host_words(offs_h, dev)
                raise
            sizes = offs_h[:2 * (W + 1) + 2].tolist()
            give_host_words(offs_h)
            if bins is not None and sizes[2 * W + 3] & 0xFFFFFFFF != 0:
                raise RuntimeError(f"build_halo_maps: partition_id has a label that is no rank's (world_size is {W})")
            total_send, total_recv, n_local = sizes[W], sizes[2 * W + 1], sizes[2 * W + 2]
            send_local = torch.empty((total_send,), dtype=torch.int64, device=dev)
            recv_atom = torch.empty((total_recv,), dtype=torch.int64, device=dev)
            recv_ghost = torch.empty((total_recv,), dtype=torch.int64, device=dev)
            interior = torch.empty((n_local,), dtype=torch.bool, device=dev)
            matrix = info.global_send_recv_matrix
            if matrix is None:
                matrix = info.global_send_recv_matrix = torch.zeros((W, W), dtype=torch.int64, device=dev)
            # row R is written by the list pass where the matrix is what the partitioner made; any other kind of tensor
            # (another device, type, shape or stride) and the empty system go through an assignment, which checks them
            in_place = (N > 0 and matrix.device == dev and matrix.dtype == torch.int64 and matrix.is_contiguous()
                        and tuple(matrix.shape) == (W, W))
            _lib.check(L.dynb_halo_lists_fill(needed.data_ptr(), None, pid.data_ptr(), N, R, W, None, has_foreign.data_ptr(),
                                              offs.data_ptr(), n_local, send_local.data_ptr(), recv_atom.data_ptr(),
                                              recv_ghost.data_ptr(), interior.data_ptr(), matrix[R].data_ptr() if in_place else None,
                                              ws.data_ptr(), _stream(dev)), "halo_lists_fill")
            info.send_offsets = offs[:W + 1]
            info.send_local_indices = send_local
            info.recv_offsets = offs[W + 1:2 * W + 2]
            info.recv_ghost_indices = recv_ghost
            info.recv_atom_global = recv_atom
            info.interior_mask = interior
            if not in_place:  # build_halo_maps.cpp:150-154
                matrix[R] = info.send_offsets[1:] - info.send_offsets[:-1]
                matrix[R, R] = n_local
        info.edge_index_halo = None
        info._edge_index_halo_fn = lambda: radius_graph_pbc(pos32, cell, pbc, ghost_cutoff, HALO_MAX_NUM_NEIGHBORS, False)[0]


class SFCPartitioner(AbstractPartitioner):
    """Cuts the Morton (or "Hilbert") order of the atoms into world_size contiguous runs of equal
    count, or of equal summed ``edge_counts`` (reference: partition/sfc_partitioner.cpp:97-238)."""

    def __init__(self, curve_type: SFCCurveType = SFCCurveType.Morton):
        self.curve_type = SFCCurveType(int(curve_type))

    def partition(self, state: MolecularInfo, env: DistEnvironment, config: Optional[SimulationConfig] = None):
        pos = state.atom_positions
        if not pos.is_cuda:
            raise RuntimeError("SFCPartitioner: atom_positions must be a CUDA tensor (this build has no CPU path)")
        W = int(env.world_size)
        pos32 = pos.to(torch.float32)
        if config is None:
            labels = sfc_partition_labels(pos32, state.edge_counts, W, int(self.curve_type))
            # equal counts: the first N % W ranks hold one atom more (sfc_kernels.cu:123-134)
            N, R, n_local = pos32.size(0), int(env.global_rank), None
            if state.edge_counts is None and 0 <= R < W:
                n_local = N // W + (1 if R < N % W else 0)
            return _finish_partition(labels, state, env, n_local)
        # mode 3: weights = in-degree at the cutoff; the graph is kept for downstream use
        cutoff = _single(config.cutoff)
        cell = config.cell.to(torch.float32)
        ei, _, _, counts = radius_graph_pbc_ex(pos32, cell, config.pbc.to(torch.bool), cutoff, PARTITION_MAX_NUM_NEIGHBORS, False)
        labels = sfc_partition_labels(pos32, counts.to(torch.int64), W, int(self.curve_type))
        info = _finish_partition(labels, state, env)
        info.edge_index = ei
        return info


def kdtree_partition_labels(pos: torch.Tensor, weights: Optional[torch.Tensor], W: int, sorted_cuts: bool = False) -> torch.Tensor:
    """Rank label in [0, W) per atom by recursive bisection along the widest axis
    (reference: kdtree_bisect_cuda, partition/kdtree.cpp:9-26).  ``sorted_cuts`` takes the sort-based
    route also for equal-count cuts (same labels)."""
    if not pos.is_cuda:
        raise RuntimeError("pos must be a CUDA tensor")
    if pos.dim() != 2 or pos.size(1) != 3:
        raise RuntimeError(f"pos must have shape [N, 3], got [{pos.size(0)}, {pos.size(1) if pos.dim() > 1 else ''}]")
    if pos.dtype != torch.float32:
        raise RuntimeError(f"pos must be float32, got {pos.dtype}")
    if W < 1:
        raise RuntimeError(f"W must be >= 1, got {W}")
    pos = pos.contiguous()
    N, dev = pos.size(0), pos.device
    if weights is not None:
        if not weights.is_cuda:
            raise RuntimeError("weights must be a CUDA tensor")
        if weights.dim() != 1 or weights.size(0) != N:
            raise RuntimeError(f"weights must have shape [N], got [{weights.size(0)}]")
        weights = weights.to(torch.int64).contiguous()
    L = _lib.lib()
    with _lib.on_device(dev):
        labels = torch.empty((N,), dtype=torch.int64, device=dev)
        if N > 0:
            nbytes = ctypes.c_int64()
            _lib.check(L.dynb_kdtree_workspace_bytes(N, int(W), ctypes.byref(nbytes)), "kdtree_workspace_bytes")
            ws = scratch(dev, "kdtree", nbytes.value)
            _lib.check(L.dynb_kdtree_partition(pos.data_ptr(), N, weights.data_ptr() if weights is not None else None, int(W),
                                               labels.data_ptr(), 1 if sorted_cuts else 0, ws.data_ptr(), ws.numel(), _stream(dev)),
                       "kdtree_partition")
    return labels


class KDTreePartitioner(AbstractPartitioner):
    """Recursive bisection along the widest axis into world_size parts of equal count, or of equal
    summed ``edge_counts``; with a SimulationConfig the weights are the in-degrees at the cutoff and the
    graph is kept (reference: partition/kdtree_partitioner.cpp:52-164)."""

    def partition(self, state: MolecularInfo, env: DistEnvironment, config: Optional[SimulationConfig] = None):
        pos = state.atom_positions
        if not pos.is_cuda:
            raise RuntimeError("KDTreePartitioner: atom_positions must be a CUDA tensor (this build has no CPU path)")
        W = int(env.world_size)
        pos32 = pos.to(torch.float32)
        if config is None:
            labels = kdtree_partition_labels(pos32, state.edge_counts, W)
            return _finish_partition(labels, state, env)
        cutoff = _single(config.cutoff)
        cell = config.cell.to(torch.float32)
        ei, _, _, counts = radius_graph_pbc_ex(pos32, cell, config.pbc.to(torch.bool), cutoff, PARTITION_MAX_NUM_NEIGHBORS, False)
        labels = kdtree_partition_labels(pos32, counts.to(torch.int64), W)
        info = _finish_partition(labels, state, env)
        info.edge_index = ei
        return info


class SimpleSpatialPartitioner(AbstractPartitioner):
    """Contiguous index split: rank r owns atoms [r*(N//W), (r+1)*(N//W)), the last rank the
    remainder (reference: partition/simple_spatial_partitioner.cpp:6-47)."""

    def partition(self, state: MolecularInfo, env: DistEnvironment):
        dev = state.atom_positions.device
        N, W, R = int(state.num_atoms), int(env.world_size), int(env.global_rank)
        per = N // W
        info = PartitionMessagePassingInfo()
        ar = torch.arange(N, dtype=torch.int64, device=dev)
        info.partition_id = torch.clamp(torch.div(ar, per, rounding_mode="trunc"), 0, W - 1) if per > 0 else \
            torch.full((N,), W - 1, dtype=torch.int64, device=dev)
        start = R * per
        end = N if R == W - 1 else start + per
        info.partition_indices = state.atom_vertex_numbers[start:end].contiguous()
        m = torch.zeros((W, W), dtype=torch.int64, device=dev)
        m[R, R] = end - start
        info.global_send_recv_matrix = m
        info.atom_counts = torch.bincount(info.partition_id, minlength=W)
        return info
