"""Pinned words that a queued launch may still write are waited for before a call that raises lets them go."""

import pytest
import torch

from dynamis_b200 import graph as G


class Stream:
    def __init__(self, log, fails=False):
        self.log, self.fails = log, fails

    def synchronize(self):
        self.log.append("wait")
        if self.fails:
            raise RuntimeError("CUDA error")


@pytest.fixture
def log(monkeypatch):
    log = []
    words = torch.zeros(G.HOST_WORDS, dtype=torch.int64)
    monkeypatch.setattr(G, "take_host_words", lambda count: words)
    monkeypatch.setattr(G, "give_host_words", lambda w: log.append("given" if w is words else "others given"))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: Stream(log))
    monkeypatch.setattr(G.HostWords, "_LOST", [])
    return log


def test_given_back_behind_the_callers_own_wait(log):
    with G.HostWords(3, torch.device("cuda", 0)) as words:
        assert words.numel() >= 3
    assert log == ["given"]


def test_a_call_that_raises_waits_first(log):
    with pytest.raises(RuntimeError, match="behind the launch"):
        with G.HostWords(3, torch.device("cuda", 0)):
            raise RuntimeError("behind the launch")
    assert log == ["wait", "given"]


def test_words_that_cannot_be_waited_for_are_kept(log, monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: Stream(log, fails=True))
    with pytest.raises(ValueError, match="behind the launch"):
        with G.HostWords(3, torch.device("cuda", 0)):
            raise ValueError("behind the launch")
    assert log == ["wait"] and len(G.HostWords._LOST) == 1
