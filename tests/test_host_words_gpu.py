"""A call that raises behind a launch that writes to its pinned words: the stream has been waited for when the exception arrives."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from dynamis_b200 import _lib
from dynamis_b200.partition import select_eq

pytestmark = pytest.mark.gpu

CALLS = {"dynb_halo_lists_plan_words": ("maps", "lists"), "dynb_rg_halo_mark_rank": ("maps",), "dynb_filter_edges_plan": ("filter",), "dynb_select_eq_i64": ("select",)}


@pytest.mark.parametrize("entry, call", [(e, c) for e, cs in CALLS.items() for c in cs])
def test_the_stream_is_idle_when_the_exception_arrives(cuda, monkeypatch, entry, call):
    rng = np.random.default_rng(1)
    n = 3000
    pos = torch.as_tensor((rng.random((n, 3)) * 30.0).astype(np.float32), device=cuda)
    cell, pbc = torch.eye(3) * 30.0, torch.tensor([True] * 3)
    labels = D.sfc_partition_labels(pos, None, 2)
    edges, shifts, _, _ = D.radius_graph_pbc_ex(pos, cell, pbc, 4.0, 0, False)
    mine = select_eq(labels, 0)
    info, env, config, state = D.PartitionMessagePassingInfo(), D.DistEnvironment(), D.SimulationConfig(), D.MolecularInfo()
    info.partition_id, env.global_rank, env.world_size = labels, 0, 2
    config.cutoff, config.ghost_cutoff_buffer, config.cell, config.pbc = 4.0, 0.0, cell, pbc
    state.num_atoms, state.atom_positions = n, pos
    calls = {"maps": lambda: D.SFCPartitioner().build_halo_maps(info, state, env, config), "lists": lambda: D.extract_halo_info(edges, labels, mine, 0, 2, n),
             "filter": lambda: D.filter_edges_to_radius(edges, shifts, pos, cell, 3.0), "select": lambda: select_eq(labels, 1)}
    calls[call]()   # buffers are there
    real = _lib.lib()

    class Failing:
        def __getattr__(self, name):
            fn = getattr(real, name)
            return (lambda *a: (fn(*a), 1)[1]) if name == entry else fn

    torch.cuda.synchronize()
    monkeypatch.setattr(_lib, "lib", lambda: Failing())
    torch.cuda._sleep(50_000_000)   # some 25 ms in front of the launches
    with pytest.raises(RuntimeError):
        calls[call]()
    assert torch.cuda.current_stream().query()
