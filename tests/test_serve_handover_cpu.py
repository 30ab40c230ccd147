"""A graph that leaves the resident set before the converter that handed it over has noted
whose it is (it joined and converged in a step that other graphs had begun), on the fake
engine of tests/test_serve_cpu.py (CPU)."""
import threading

import numpy as np

import serve
from test_serve_cpu import FakeEngine


class QuickToLeave(FakeEngine):
    """The set's lane stays busy with a graph of 1000 records until `release`; the handover of
    one of 12 records (a single step) returns only when its graph has been taken from the set."""
    release, taken = threading.Event(), threading.Event()

    def resident_add(self, src):
        quick = 12 in src.graphs
        ids = super().resident_add(src)
        if quick:
            self.taken.wait(5)
        return ids

    def resident_step(self):
        for g in self.live.values():
            if g["records"] == 1000 and not self.release.is_set():
                g["need"] = g["iters"] + 2
        return super().resident_step()

    def resident_take(self):
        out = super().resident_take()
        if any(lab.shape[0] == 12 for _, _, _, lab in out):
            self.taken.set()
        return out


def test_graph_leaves_before_its_handover_returns():
    srv = serve.Server(converters=1, budget_bytes=1e12, max_batch=1, bytes_per_record=10, engine_factory=QuickToLeave)
    long = srv.submit(np.zeros((1000, 2), np.uint32))
    while not srv.lanes[0].in_set:   # iterating
        threading.Event().wait(0.001)
    quick = srv.submit(np.zeros((12, 2), np.uint32))
    assert quick.wait(10)[0]["records"] == 12
    QuickToLeave.release.set()
    assert long.wait(10)[0]["records"] == 1000
    srv.close()
    assert abs(srv._in_use) < 1e-6
