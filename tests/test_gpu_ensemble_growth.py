"""A replica whose rows outgrow their capacity in the middle of a run: its build is
made again with longer rows, and every replica, itself included, goes on bit for
bit as it would alone."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _collapsing(n, L, rate):
    """Atoms on a sparse lattice, all moving towards the middle of the box."""
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    q = (g + 0.5) / m * L
    return q, -rate * (q - 0.5 * L), L


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("liquids", [2, 9])  # with conditional branches, and without
@pytest.mark.parametrize("chunks", [[160], [1] * 160, [40, 1, 1, 118]])
def test_the_others_go_on(precision, liquids, chunks):
    reps = [_collapsing(512, np.array([30.0, 31.0, 32.0]), 1.0)]
    for k in range(liquids):
        w = W.fcc_liquid(5 + k % 3, 0.2 + 0.01 * k, 1.5, seed=k, jitter=0.05, rc=2.5, dt=0.005)
        reps.append((w.q, w.v, w.L))
    ens = M.Ensemble(reps, cutoff=2.5, time_step=0.005, precision=precision)
    capacity = 32 + 1.6 * max(len(q) / np.prod(L) for q, _, L in reps) * 4 / 3 * np.pi * 2.8 ** 3
    for k in chunks:
        ens.calculate(k)
    got, rebuilds = ens.states_by_id(), ens.rebuilds()[0]
    ens.close()
    longest = 0
    for (q, v, L), (gq, gv), r in zip(reps, got, rebuilds):
        s = M.System(L, cutoff=2.5, time_step=0.005, capacity=len(q), precision=precision)
        s.set_state(q, v)
        s.calculate(160)
        sq, sv = s.state_by_id()
        info = s.info()
        longest = max(longest, info["max_row"])
        s.close()
        assert info["rebuilds"] == r
        assert np.array_equal(sq, gq) and np.array_equal(sv, gv)
    assert longest > capacity  # the rows did outgrow it


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("first", ["observe", "list_stats"])
def test_sums_before_the_first_step(precision, first):
    # a dense drop in a wide box: the first build's rows outgrow the capacity
    # that the mean density gives, and a call that only reads builds them longer
    w = W.fcc_liquid(6, 0.95, 1.0, seed=4, jitter=0.05, rc=2.5, dt=0.005)
    L = np.array([40.0, 41.0, 42.0])
    q = w.q + (L - w.L) / 2
    gas = W.fcc_liquid(5, 0.2, 1.0, seed=5, jitter=0.05, rc=2.5, dt=0.005)
    ens = M.Ensemble([(gas.q, gas.v, gas.L), (q, w.v, L)], cutoff=2.5, time_step=0.005, precision=precision)
    getattr(ens, first)()
    sums, (entries, within) = ens.observe(), ens.list_stats()
    ens.calculate(10)
    got = ens.states_by_id()
    ens.close()
    total = pairs = 0
    for k, (x, v, box) in enumerate(((gas.q, gas.v, gas.L), (q, w.v, L))):
        s = M.System(box, cutoff=2.5, time_step=0.005, capacity=len(x), precision=precision)
        s.set_state(x, v)
        assert [a[k] for a in sums] == pytest.approx(s.observe(), rel=1e-12)
        n, e = s.pair_counts()
        total, pairs = total + e, pairs + n // 2
        s.calculate(10)
        sq, sv = s.state_by_id()
        s.close()
        assert np.array_equal(sq, got[k][0]) and np.array_equal(sv, got[k][1])
    assert (entries, within) == (total, pairs)
