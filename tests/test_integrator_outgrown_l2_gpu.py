"""Four atoms a thread against one where the arrays begin to outgrow L2: the same step on arrays that start on a 16-byte boundary and on
arrays that do not, with one to three atoms left over; the drift word too."""

import pytest
import torch

from dynamis_b200 import integrators as I

pytestmark = pytest.mark.gpu


def _at(t, offset):
    """A copy of t that starts `offset` floats behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=torch.float32, device=t.device)
    out = buf[offset:offset + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("drift", [False, True])
@pytest.mark.parametrize("kind", [I.EULER, I.VERLET1, I.VERLET2, I.LANGEVIN1, I.LANGEVIN2])
@pytest.mark.parametrize("extra", [-1, 0, 1, 2, 3])
def test_same_bits(cuda, kind, drift, extra):
    moves = kind in (I.EULER, I.VERLET1, I.LANGEVIN1)
    if drift and not moves:
        pytest.skip("the drift word rides on a step that moves the positions")
    arrays = 2 + moves + (kind >= I.LANGEVIN1) + 2 * drift
    n = -(-(126 << 20) // (12 * arrays + 4)) + extra
    gen = torch.Generator(device=cuda).manual_seed(n + kind)
    pos, vel, frc, noise = (torch.randn(n, 3, generator=gen, device=cuda) for _ in range(4))
    mass = torch.rand(n, generator=gen, device=cuda) * 60.0 + 1.0
    results = []
    for offset in (0, 1):
        p, v, f, z, m = (_at(t, offset) for t in (pos, vel, frc, noise, mass))
        watch = None
        if drift:
            watch = I.DriftWatch(pos, vel, 1e-3)
            watch.ref, watch.prev_vel = _at(pos, offset), _at(vel + 0.01, offset)
        I._launch(kind, p if moves else None, v, f, m, z if kind >= I.LANGEVIN1 else None, 0.5, 0.01, 0.025, watch)
        results.append([p, v] + ([watch.prev_vel, watch.flag, watch.state] if drift else []))
    assert not torch.equal(results[0][1], vel)
    for a, b in zip(*results):
        assert torch.equal(a, b)
