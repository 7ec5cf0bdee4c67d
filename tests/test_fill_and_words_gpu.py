"""C entries whose Python callers use one form only: bytes set by a launch, at every start and end within 16 bytes, and the words of a halo
plan that go to the host, from the kernel or by a copy."""

import ctypes

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from dynamis_b200 import _lib

pytestmark = pytest.mark.gpu


def stream(device):
    return _lib.stream_of(torch.device(device))


@pytest.mark.parametrize("byte", [0, 0xFF, 0x5A])
def test_fill_bytes(cuda, byte):
    pitch, size = 128, 16 * 41
    buf = torch.full((size, pitch), 7, dtype=torch.uint8, device=cuda)
    assert buf.data_ptr() % 16 == 0
    expected = np.full((size, pitch), 7, dtype=np.uint8)
    for off in range(16):
        for length in range(41):
            row = off * 41 + length
            _lib.check(_lib.lib().dynb_fill_bytes(buf.data_ptr() + row * pitch + 32 + off, length, byte, stream(cuda)))
            expected[row, 32 + off:32 + off + length] = byte
    np.testing.assert_array_equal(buf.cpu().numpy(), expected)


@pytest.mark.parametrize("off, length", [(0, 4097), (3, 1_000_003), (15, 16 * 148 * 4096 + 29)])
def test_fill_many_bytes(cuda, off, length):
    buf = torch.full((length + 64,), 7, dtype=torch.uint8, device=cuda)
    _lib.check(_lib.lib().dynb_fill_bytes(buf.data_ptr() + 16 + off, length, 0x5A, stream(cuda)))
    assert bool((buf[16 + off:16 + off + length] == 0x5A).all()) and bool((buf[:16 + off] == 7).all()) and bool((buf[16 + off + length:] == 7).all())


def test_fill_refuses(cuda):
    buf = torch.zeros(16, dtype=torch.uint8, device=cuda)
    for at, length in ((buf.data_ptr(), -1), (None, 1)):
        with pytest.raises(RuntimeError):
            _lib.check(_lib.lib().dynb_fill_bytes(at, length, 0, stream(cuda)))
    _lib.check(_lib.lib().dynb_fill_bytes(None, 0, 0, stream(cuda)))


class Plan:
    def __init__(self, cuda, n, W, R):
        gen = torch.Generator(device=cuda).manual_seed(n + W)
        self.n, self.W, self.R, self.dev = n, W, R, cuda
        self.masks = [torch.randint(0, 1 << W, (max(n, 1), 1), generator=gen, device=cuda, dtype=torch.int32) for _ in range(2)]
        nbytes = ctypes.c_int64()
        _lib.check(_lib.lib().dynb_halo_lists_workspace_bytes(n, W, ctypes.byref(nbytes)))
        self.ws = torch.empty(max(nbytes.value, 1), dtype=torch.uint8, device=cuda)
        self.offsets = torch.full((2 * (W + 1) + 2,), -5, dtype=torch.int64, device=cuda)   # the last word is the caller's

    def run(self, at, n_words):
        _lib.check(_lib.lib().dynb_halo_lists_plan_words(self.masks[0].data_ptr(), self.masks[1].data_ptr(), None, self.n, self.R, self.W,
                                                         self.offsets.data_ptr(), self.ws.data_ptr(), self.ws.numel(), at, n_words, stream(self.dev)))

    def expected(self):
        counts = [[int(((m[:self.n] >> p) & 1).sum()) for p in range(self.W)] for m in self.masks]   # the masks are counted as they are
        return [0, *np.cumsum(counts[0])], [0, *np.cumsum(counts[1])]


@pytest.mark.parametrize("n", [0, 1, 3000, 40_003])
@pytest.mark.parametrize("where", ["pinned", "pinned, 8 bytes on", "pageable"])
def test_words_of_a_halo_plan(cuda, n, where):
    plan = Plan(cuda, n, 5, 2)
    most = 2 * 6 + 2
    words = torch.full((most + 4,), -9, dtype=torch.int64, pin_memory=where != "pageable")
    first = 1 if where == "pinned, 8 bytes on" else 0
    for n_words in (0, 1, 6, most - 1, most):
        words.fill_(-9)
        plan.run(words.data_ptr() + 8 * first, n_words)
        torch.cuda.synchronize()
        got = plan.offsets.tolist()
        send, recv = plan.expected()
        assert got[:6] == send and got[6:12] == recv and got[-1] == -5
        assert words[first:first + n_words].tolist() == got[:n_words]
        assert bool((words[:first] == -9).all()) and bool((words[first + n_words:] == -9).all())


def test_words_out_of_range_are_refused(cuda):
    plan = Plan(cuda, 100, 5, 2)
    words = torch.zeros(64, dtype=torch.int64, pin_memory=True)
    for n_words in (-1, 2 * 6 + 3):
        with pytest.raises(RuntimeError, match="n_words"):
            plan.run(words.data_ptr(), n_words)


def test_recorded_and_replayed(cuda):
    """A KD-tree, which no copy sets up any more, and a halo plan behind bytes set by a launch, in a CUDA graph."""
    n = 30_011
    pos = torch.rand(n, 3, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1)) * 50.0
    expected = [D.kdtree_partition_labels(p, None, 5) for p in (pos, pos.flip(0).contiguous())]
    plan = Plan(cuda, n, 5, 2)
    words = torch.zeros(64, dtype=torch.int64, pin_memory=True)
    main = torch.cuda.Stream()
    main.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(main):
        D.kdtree_partition_labels(pos, None, 5)   # the stream's workspace
        main.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            labels = D.kdtree_partition_labels(pos, None, 5)
            _lib.check(_lib.lib().dynb_fill_bytes(plan.masks[0].data_ptr(), 4 * n - 4, 0, stream(cuda)))
            plan.run(words.data_ptr(), 14)
        for k in range(2):
            words.zero_()
            graph.replay()
            main.synchronize()
            assert torch.equal(labels, expected[k])
            assert words[:14].tolist() == plan.offsets.tolist() and words[5] <= 5 and not plan.masks[0][:n - 1].any()
            pos.copy_(pos.flip(0))
