"""Steps through graphs and step by step, and ensembles with and without
conditional branches, give the same trajectories bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


# one block, a block and an atom, and several blocks of the drift's sums
@pytest.mark.parametrize("cut", [256, 257, 3000])
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("thermostat", [M.NVE, M.NOSE_HOOVER, M.LANGEVIN])
def test_graph_steps_equal_single_steps(cut, precision, thermostat):
    w = W.fcc_liquid(5 if cut < 500 else 10, 0.6, 1.0, seed=cut, jitter=0.05, rc=2.5, dt=0.005)
    out = []
    for chunks in ([63], [1] * 63):
        s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision, thermostat=thermostat,
                     aimed_temperature=1.2, seed=3)
        s.set_state(w.q[:cut], w.v[:cut])
        for k in chunks:
            s.calculate(k)
        info = s.info()
        out.append((*s.state_by_id(), s.zeta(), info["steps"], info["rebuilds"], info["displacement_checks"]))
        s.close()
    a, b = out
    assert a[4] > 1 and a[5] > 1  # the steps rebuilt and checked
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_few_replicas_equal_many(precision):
    # from eight replicas the check's and rebuild's kernels run every step
    reps = [W.fcc_liquid(4 + k % 3, 0.5 + 0.04 * k, 1.0, seed=k, jitter=0.05, rc=2.5, dt=0.005) for k in range(9)]
    out = []
    for n, chunks in ((9, [67]), (9, [20] + [1] * 47), (8, [67]), (7, [67]), (1, [67])):
        ens = M.Ensemble([(r.q, r.v, r.L) for r in reps[:n]], cutoff=2.5, time_step=0.005, precision=precision)
        for k in chunks:
            ens.calculate(k)
        out.append(ens.states_by_id())
        ens.close()
    for other in out[1:]:
        for (q, v), (q1, v1) in zip(out[0], other):
            assert np.array_equal(q, q1) and np.array_equal(v, v1)


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_single_steps_between_other_calls(precision):
    # the status kept from the last step is dropped by whatever may change it:
    # the same calls with it dropped before every step (set_control drops it)
    w = W.fcc_liquid(6, 0.7, 1.0, seed=4, jitter=0.05, rc=2.5, dt=0.005)
    out = []
    for drop in (False, True):
        s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision)
        sums = []

        def steps(n, s=s, sums=sums, drop=drop):
            for _ in range(n):
                if drop:
                    s.set_control(M.NVE)
                s.calculate(1)
                sums.append(s.observe())

        s.set_state(w.q, w.v)
        steps(12)
        q, v = s.state_by_id()
        s.set_state(q, 3.0 * v)  # faster atoms, a stale list
        steps(9)
        s.make_pairlist()
        steps(3)
        s.set_external(kind=M.EXTERNAL_GRAVITY, axis=1, strength=0.3, time_step=0.005)
        steps(5)
        s.set_external()
        s.calculate(21)
        steps(8)
        s.change_scale(1.01)
        steps(6)
        info = s.info()
        out.append((sums, *s.state_by_id(), info["steps"], info["rebuilds"], info["displacement_checks"]))
        s.close()
    a, b = out
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2]) and a[3:] == b[3:]


# lanes per atom change at 8,192 and 24,000 atoms; 148 multiprocessors hold
# the lanes of 75,776 atoms with the row's head in registers
@pytest.mark.parametrize("n", [2, 33, 257, 8191, 8192, 23999, 24000, 75776, 75777])
def test_persistent_steps_equal_graphs_at_the_edges(n):
    w = W.fcc_liquid(max(5, int(np.ceil((n / 3.6) ** (1 / 3)))), 0.7, 1.0, seed=n, jitter=0.05, rc=2.5, dt=0.005)
    keep = np.sort(np.random.Generator(np.random.Philox(n)).permutation(w.n)[:n])
    out = []
    for mode in (1, 2):  # graphs, persistent
        s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=n, precision=M.FP32_MIXED, step_mode=mode)
        s.set_state(w.q[keep], w.v[keep])
        s.calculate(45)
        info = s.info()
        out.append((*s.state_by_id(), info["rebuilds"], info["displacement_checks"], info["persistent_steps"]))
        s.close()
    a, b = out
    assert a[4] == 0 and b[4] > 0
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:4] == b[2:4]
