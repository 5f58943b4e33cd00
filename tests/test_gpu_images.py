"""FP64 pair terms through the nearest image wherever the atoms are now: the
cells in which the list was built say nothing about that once an atom has gone
far, which the reference's skin check lets it do while no other atom moves
(src/pairlist.cc:86-121: the candidates are the atoms that moved more than
BufferLength minus the largest displacement, in magnitude)."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 8, 4 and 1 lanes an atom; four to fourteen cells an axis
@pytest.mark.parametrize("cells", [8, (20, 9, 21), 27])
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_atoms_a_box_length_away(cells, precision):
    w = W.fcc_liquid(cells, 0.8442, 1.0, seed=9, jitter=0.05, rc=2.5, dt=0.005)
    rng = np.random.Generator(np.random.Philox(3))
    # atoms whose partners lie on their side of every face: an image is searched one box length away
    inner = ((w.q > 2.8) & (w.q < w.L - 2.8)).all(axis=1)
    far = rng.integers(0, 2, (w.n, 3)) * (inner & (rng.uniform(size=w.n) < 0.2))[:, None]
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision)
    s.set_state(w.q, 2.0 * far * w.L / 0.005)  # half a step moves them by the box lengths
    s.make_pairlist()
    f0, (_, pe0, vir0), (within0, _) = s.forces_by_id(), s.observe(), s.pair_counts()
    s.update_position_half()
    f1, (_, pe1, vir1), (within1, _) = s.forces_by_id(), s.observe(), s.pair_counts()
    s.close()
    # coordinates up to two box lengths: 1e-14 off; pair forces change by up to
    # some 1e3 per unit.  Fixed-point copies: a unit is L / 2^32.
    assert np.abs(f1 - f0).max() <= (1e-9 if precision == M.FP64 else 1e-3)
    assert pe1 == pytest.approx(pe0, rel=1e-10) and vir1 == pytest.approx(vir0, rel=1e-10)
    assert within1 == within0


def test_a_fast_atom_meets_its_partner_from_behind():
    # 6 x 6 x 6 cells; an atom flies from its partner (2.7 away, listed, out of
    # the cut-off) once around the box.  The others rest out of reach in the
    # same row of inner cells, so that no atom of an outermost cell is near.
    L = np.array([17.0, 17.2, 17.4])
    q = np.array([[8.6, 8.6, 8.6], [11.3, 8.6, 8.6], [4.4, 6.1, 8.6], [4.4, 9.0, 10.9], [13.6, 6.1, 10.9],
                  [13.6, 9.6, 10.9], [8.6, 6.1, 10.9], [8.6, 11.0, 10.9]])
    v = np.zeros_like(q)
    v[0] = [-20.0, 0.0, 0.02]
    dt, steps = 0.005, 150

    def pair_force(d):
        d = d - L * np.round(d / L)
        r2 = d @ d
        if r2 > 6.25:
            return 0.0 * d
        s6 = 2.5 ** -6
        c2 = (6 * s6 * s6 - 3 * s6) / 6.25
        return ((48.0 - 24.0 * r2 ** 3) / r2 ** 7 - 8.0 * c2) * d

    x, u = q[:2].copy(), v[:2].copy()
    for _ in range(steps):
        x += u * (dt / 2)
        f = pair_force(x[0] - x[1])
        u += np.array([f, -f]) * dt
        x += u * (dt / 2)
    assert abs(u[1, 0]) > 1e-3  # they met
    s = M.System(L, cutoff=2.5, time_step=dt, capacity=len(q))
    s.set_state(q, v)
    s.calculate(steps)
    got = [s.state_by_id()]
    assert s.info()["rebuilds"] == 1
    s.close()
    ens = M.Ensemble([(q, v, L)], cutoff=2.5, time_step=dt)
    ens.calculate(steps)
    got += ens.states_by_id()
    ens.close()
    for gq, gv in got:
        assert np.abs(gq[:2] - x).max() <= 1e-9 and np.abs(gv[:2] - u).max() <= 1e-9
        assert np.array_equal(gq[2:], q[2:])
