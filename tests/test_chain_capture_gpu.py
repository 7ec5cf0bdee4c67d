"""Launches of a chain inside a CUDA graph: recorded behind one another, behind a kernel of the framework and behind a wait for
another stream, replayed, and compared with the same calls outside."""

import pytest
import torch

from dynamis_b200 import integrators as I
from dynamis_b200.partition import sfc_partition_labels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 200_001])
def test_recorded_and_replayed(cuda, n):
    gen = torch.Generator(device=cuda).manual_seed(n)
    start = [torch.randn(n, 3, generator=gen, device=cuda) for _ in range(2)]
    frc, noise, mass = torch.randn(n, 3, generator=gen, device=cuda), torch.randn(n, 3, generator=gen, device=cuda), torch.ones(n, device=cuda)
    step = I.Langevin(0.5, 0.01, 0.025)

    def work(pos, vel, side):
        step.halfstep1_(pos, vel, frc, mass, noise, 0.5)
        pos.mul_(0.5)
        step.halfstep2_(vel, frc, mass, noise, 0.5)
        here = torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            step.halfstep2_(vel, frc, mass, noise, 0.5)
        here.wait_stream(side)
        step.halfstep1_(pos, vel, frc, mass, noise, 0.5)
        return sfc_partition_labels(pos, None, 5)

    side = torch.cuda.Stream()
    expected = [t.clone() for t in start]
    labels = work(*expected, side)
    rounds = [labels.clone()]
    rounds.append(work(*expected, side).clone())
    main = torch.cuda.Stream()
    with torch.cuda.stream(main):
        got = [t.clone() for t in start]
        work(*[t.clone() for t in start], side)   # workspaces of the streams
        main.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            recorded = work(*got, side)
        for k in range(2):
            graph.replay()
            main.synchronize()
            assert torch.equal(recorded, rounds[k])
    assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])
    assert not torch.equal(got[0], start[0])
