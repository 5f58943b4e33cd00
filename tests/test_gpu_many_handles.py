"""Handles beyond the 64 places that the library keeps for their small answers,
made, used and closed in any order and by several threads at once: the same
answers as alone."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _run(w, precision, steps=7):
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision)
    s.set_state(w.q, w.v)
    for _ in range(steps):
        s.calculate(1)
    return s


def test_more_handles_than_places():
    w = W.fcc_liquid(5, 0.6, 1.0, seed=2, jitter=0.05, rc=2.5, dt=0.005)
    alone = {p: _run(w, p) for p in (M.FP64, M.FP32_MIXED)}
    want = {p: (*s.state_by_id(), s.observe()) for p, s in alone.items()}
    held = [(p, _run(w, p)) for k in range(70) for p in (M.FP64 if k % 2 else M.FP32_MIXED,)]
    for p, s in held[::3]:  # some places come free and are taken again
        s.close()
    held = [x for k, x in enumerate(held) if k % 3] + [(M.FP64, _run(w, M.FP64)) for _ in range(30)]
    for p, s in held:
        q, v = s.state_by_id()
        assert np.array_equal(q, want[p][0]) and np.array_equal(v, want[p][1])
        assert s.observe() == want[p][2]
        s.close()


def test_threads_make_and_close_handles():
    w = W.fcc_liquid(5, 0.6, 1.0, seed=2, jitter=0.05, rc=2.5, dt=0.005)
    s = _run(w, M.FP64)
    want = s.observe()
    s.close()
    wrong = []

    def work():
        for _ in range(6):
            s = _run(w, M.FP64)
            if s.observe() != want:
                wrong.append(1)
            s.close()

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
