"""The selection of the KD-tree's cuts puts the place of a coordinate in its segment in front of the coordinate's bits; the sorted cuts
do not.  Labels of both, over coordinates whose places crowd, tie, overflow or cannot be computed."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(11)
N = 20_011
CASES = {
    "uniform": RNG.random((N, 3)) * 90.0 - 45.0,
    "lattice": np.stack(np.meshgrid(*[np.arange(28.0)] * 3), -1).reshape(-1, 3)[:N],
    "one_point": np.ones((N, 3)),
    "two_clusters": np.concatenate([RNG.normal(size=(N // 2, 3)) * 1e-3, 1e6 + RNG.normal(size=(N - N // 2, 3))]),
    "outlier": np.concatenate([RNG.random((N - 1, 3)), np.full((1, 3), 3e37)]),
    "denormal": RNG.random((N, 3)) * 1e-40,
    "overflowing_extent": (RNG.random((N, 3)) - 0.5) * 6.0e38,
    "signed_zeros": np.where(RNG.random((N, 3)) < 0.5, 0.0, -0.0) + (RNG.random((N, 3)) < 0.01),
    "infinite": np.where(RNG.random((N, 3)) < 0.001, np.inf, RNG.random((N, 3))),
}


@pytest.mark.parametrize("W", [2, 5, 16])
@pytest.mark.parametrize("name", sorted(CASES))
def test_labels_of_both_methods(cuda, name, W):
    pos = torch.as_tensor(CASES[name].astype(np.float32), device=cuda)
    by_places = D.kdtree_partition_labels(pos, None, W)
    by_sort = D.kdtree_partition_labels(pos, None, W, sorted_cuts=True)
    np.testing.assert_array_equal(by_places.cpu().numpy(), by_sort.cpu().numpy())
