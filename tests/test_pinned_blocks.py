"""Pinned host memory that kernels read and write by address: who owns it waits for them before it goes away.  (The host
allocator knows of copies in flight, not of kernels: it would hand the block out again at once.)"""
import gc

from allpaca_b200.engine.runner import ModelRunner, _DecodeGraph
from allpaca_b200.sampling.sampler import Sampler


class Event:
    def __init__(self):
        self.waited = 0

    def synchronize(self):
        self.waited += 1


def test_owners_wait_for_the_kernels_in_flight():
    events = [Event() for _ in range(4)]
    sampler, runner, graph = Sampler.__new__(Sampler), ModelRunner.__new__(ModelRunner), _DecodeGraph.__new__(_DecodeGraph)
    sampler._events, runner._copied, graph.copied = events[:2], events[2], events[3]
    del sampler, runner, graph
    gc.collect()
    assert [e.waited for e in events] == [1, 1, 1, 1]


def test_owners_that_were_never_set_up_go_quietly(capsys):
    for kind in (Sampler, ModelRunner, _DecodeGraph):
        kind.__new__(kind)
    gc.collect()
    assert "Exception" not in capsys.readouterr().err
