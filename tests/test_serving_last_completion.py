"""A request refused for memory while the last active one completes is tried again: its refusal was
made beside a request that has since given its memory back."""
from __future__ import annotations

import threading
import time

import numpy as np

from tomoj_gb300.serving import SIRT, Request, Server


class OneAtATime:
    """Refuses a second request, and answers only after the first one has gone."""

    n_lanes = 1

    def __init__(self):
        self.held = 0
        self.refused = 0
        self.gone = threading.Event()

    def create(self, req):
        if self.held:
            self.refused += 1
            assert self.gone.wait(10)
            time.sleep(0.1)  # the completion is booked after its handle is destroyed
            return None
        self.held += 1
        self.gone.clear()
        return ("h", req.rid)

    def set_members(self, handles, lane=0):
        pass

    def iterate(self, handles, reqs, iteration, lane=0):
        time.sleep(0.02)
        return np.zeros((len(handles), 5))

    def destroy(self, hd):
        self.held -= 1
        self.gone.set()


def test_refusal_during_the_last_completion():
    series = np.zeros((3, 4, 4), np.float32)
    reqs = [Request(i, 0.0, SIRT, series, np.linspace(-10.0, 10.0, 3), 4, 4, 4, 2) for i in range(3)]
    eng = OneAtATime()
    res = Server(eng, max_active=4).run(reqs)
    assert [r.rid for r in res] == [0, 1, 2] and eng.refused > 0 and eng.held == 0
