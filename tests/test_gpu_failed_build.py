"""A list build that finds an atom outside the box by more than a box length
reports it and leaves the atoms as they are: none is moved to another slot or
given another atom's, or an earlier state's, values."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [6, 20])
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("how", ["make", "step", "steps"])
def test_state_stays(cells, precision, how):
    w = W.fcc_liquid(cells, 0.7, 1.0, seed=2, jitter=0.05, rc=2.5, dt=0.005)
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision)
    s.set_state(w.q, w.v)
    s.calculate(25)
    s.forces()
    q = w.q.copy()
    q[w.n // 2, 1] -= 2.5 * w.L[1]
    v = np.arange(3.0 * w.n).reshape(w.n, 3) * 1e-6
    s.set_state(q, v)
    with pytest.raises(M.MdgError) as e:
        s.make_pairlist() if how == "make" else s.calculate(1 if how == "step" else 40)
    assert e.value.status == -5  # invalid position
    gq, gv, ids = s.state()
    assert np.array_equal(ids, np.arange(w.n)) and np.array_equal(gv, v)
    d = (gq - q) / w.L  # wrapped into the box or as uploaded
    assert np.abs(d - np.round(d)).max() < 1e-12
    s.set_state(w.q, w.v)
    s.calculate(3)
    s.close()


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_replicas_stay(precision):
    ws = [W.fcc_liquid(c, 0.7, 1.0, seed=c, jitter=0.05, rc=2.5, dt=0.005) for c in (5, 6, 7)]
    bad = ws[1].q.copy()
    bad[7, 0] += 3.0 * ws[1].L[0]
    ens = M.Ensemble([(ws[0].q, ws[0].v, ws[0].L), (bad, ws[1].v, ws[1].L), (ws[2].q, ws[2].v, ws[2].L)], cutoff=2.5,
                     time_step=0.005, precision=precision)
    with pytest.raises(M.MdgError) as e:
        ens.calculate(5)
    assert e.value.status == -5
    for (q, v), w in zip(ens.states_by_id(), ws):
        assert np.array_equal(v, w.v)
        assert np.abs((q - w.q) / w.L - np.round((q - w.q) / w.L)).max() < 1e-12
    ens.close()
