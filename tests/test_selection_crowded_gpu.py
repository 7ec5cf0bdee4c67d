"""Selection of split points from keys that crowd into few digits (an atom far from all others, clusters far from one another): labels
against the sorted paths, over the numbers of split points at which its passes change form, and the time of a call."""

import pytest
import torch

import dynamis_b200 as D

pytestmark = pytest.mark.gpu


def system(name, n, device):
    gen = torch.Generator(device=device).manual_seed(5)
    pos = torch.rand(n, 3, generator=gen, device=device) * 200.0
    if name == "outlier":
        pos[n // 3] = 1.0e6
    elif name == "two":
        pos = pos * 0.01 + 1.0e5 * (torch.rand(n, 1, generator=gen, device=device) < 0.5)
    elif name == "many":
        pos = pos * 0.001 + 1.0e4 * torch.randint(0, 40, (n, 1), generator=gen, device=device)
    elif name == "equal":
        pos = torch.floor(pos / 67.0) * 67.0
    return pos


@pytest.mark.parametrize("name", ["uniform", "outlier", "two", "many", "equal"])
@pytest.mark.parametrize("n, W", [(120_011, 2), (120_011, 16), (120_011, 32), (120_011, 34), (300_007, 8), (40_009, 700)])
def test_kdtree_labels(cuda, name, n, W):
    pos = system(name, n, cuda)
    assert torch.equal(D.kdtree_partition_labels(pos, None, W), D.kdtree_partition_labels(pos, None, W, sorted_cuts=True))


@pytest.mark.parametrize("name", ["uniform", "two"])
@pytest.mark.parametrize("n, W", [((65 << 14) - 1, 8), (65 << 14, 8), (2_200_003, 16), (4_300_007, 3)])
def test_kdtree_labels_with_finer_places(cuda, name, n, W):
    pos = system(name, n, cuda)
    assert torch.equal(D.kdtree_partition_labels(pos, None, W), D.kdtree_partition_labels(pos, None, W, sorted_cuts=True))


@pytest.mark.parametrize("name", ["uniform", "outlier", "two", "many", "equal"])
@pytest.mark.parametrize("n, W", [(120_011, 2), (120_011, 17), (120_011, 18), (120_011, 769), (120_011, 770), (300_007, 8)])
def test_curve_labels(cuda, name, n, W):
    pos = system(name, n, cuda)
    assert torch.equal(D.sfc_partition_labels(pos, None, W), D.sfc_partition_labels(pos, None, W, return_perm=True)[0])


@pytest.mark.parametrize("name", ["outlier", "two"])
def test_time(cuda, name):
    """The pass over crowded keys that is not needed for others is one more of two a level, and the counters of a block take what would
    be additions to one address: a call takes less than twice as long as for even keys (5.8 and 8.9 times when all were added in memory)."""
    best = {}
    for _ in range(6):
        for system_name in ("uniform", name):
            pos = system(system_name, 1_000_000, cuda)
            D.kdtree_partition_labels(pos, None, 8)
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(5):
                D.kdtree_partition_labels(pos, None, 8)
            end.record()
            torch.cuda.synchronize()
            best[system_name] = min(best.get(system_name, float("inf")), start.elapsed_time(end))
    assert best[name] < 2.0 * best["uniform"], {k: f"{v / 5 * 1e3:.0f} us" for k, v in best.items()}
