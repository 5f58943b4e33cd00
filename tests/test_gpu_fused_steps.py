"""The fused NVE step outside the persistent pass (FP32-mixed systems larger than
one wave run so): single steps, which skip the wait for the device's decision
and leave the coming step's positions in either packed copy, between graph
launches, which start from the first copy; and the same calls with the kept
status dropped before each step."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _system(w, precision, n):
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=n, precision=precision, step_mode=1)
    s.set_state(w.q[:n], w.v[:n])
    return s


@pytest.mark.parametrize("cut", [257, 3000])
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("chunks", [[1] * 65, [1, 1, 1, 21, 1, 40], [1, 40, 1, 23], [3, 20, 2, 20, 20], [45, 1, 1, 1, 17]])
def test_single_steps_between_graphs(cut, precision, chunks):
    w = W.fcc_liquid(5 if cut < 500 else 10, 0.6, 1.0, seed=cut, jitter=0.05, rc=2.5, dt=0.005)
    out = []
    for steps in ([65], chunks):
        s = _system(w, precision, cut)
        assert sum(steps) == 65
        for k in steps:
            s.calculate(k)
        info = s.info()
        assert info["persistent_steps"] == 0
        out.append((*s.state_by_id(), info["steps"], info["rebuilds"], info["displacement_checks"]))
        s.close()
    a, b = out
    assert a[3] > 1 and a[4] > 1
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_kept_status_between_other_calls(precision):
    w = W.fcc_liquid(6, 0.7, 1.0, seed=4, jitter=0.05, rc=2.5, dt=0.005)
    out = []
    for drop in (False, True):
        s = _system(w, precision, w.n)
        sums = []

        def steps(n, s=s, sums=sums, drop=drop):
            for _ in range(n):
                if drop:
                    s.set_control(M.NVE)
                s.calculate(1)
                sums.append(s.observe())

        steps(13)
        q, v = s.state_by_id()
        s.set_state(q, 3.0 * v)  # faster atoms, a stale list
        steps(9)
        _, v4, _ = s.state()
        s.set_velocities4(np.concatenate([0.5 * v4, np.zeros((w.n, 1))], axis=1))
        steps(5)
        s.make_pairlist()
        steps(3)
        s.calculate(21)
        steps(7)
        s.change_scale(1.01)
        steps(6)
        info = s.info()
        assert info["persistent_steps"] == 0
        out.append((sums, *s.state_by_id(), info["steps"], info["rebuilds"], info["displacement_checks"]))
        s.close()
    a, b = out
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2]) and a[3:] == b[3:]
