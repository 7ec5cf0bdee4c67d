"""Pinned words that a queued launch may still write are waited for before a call that raises lets them go."""

import pytest
import torch

from dynamis_b200 import graph as G


class Stream:
    def __init__(self, log, fails):
        self.log, self.fails = log, fails

    def synchronize(self):
        self.log.append("wait")
        if self.fails:
            raise RuntimeError("CUDA error")


@pytest.mark.parametrize("fails", [False, True])
def test_waited_for_and_given_back_or_kept(monkeypatch, fails):
    log, words = [], torch.zeros(G.HOST_WORDS, dtype=torch.int64)
    monkeypatch.setattr(G, "give_host_words", lambda w: log.append("given" if w is words else "others given"))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: Stream(log, fails))
    monkeypatch.setattr(G, "_LOST_WORDS", [])
    G.lose_host_words(words, torch.device("cuda", 0))
    assert log == (["wait"] if fails else ["wait", "given"])
    assert [w is words for w in G._LOST_WORDS] == ([True] if fails else [])
