"""The list build's rows at the edges of its work split: the warp walk (one
lane per atom) against the general walk (two lanes per atom), entry for entry,
and the all-pairs rows of small replicas against the same system's rows.

Edges: three cells an axis (runs that wrap at both ends), atom counts around a
multiple of 32, x-rows shorter than a warp (several rows in one), empty cells,
runs longer than the 128 staged candidates, atoms exactly on the faces."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _rows(q, L, rc, lanes):
    s = M.System(L, cutoff=rc, time_step=0.005, capacity=len(q), build_block=128, build_threads_per_atom=lanes)
    s.set_state(q, np.zeros_like(q))
    s.make_pairlist()
    rows, part = s.neighbor_list()
    ids = s.ids()
    s.close()
    return rows, part, ids


@pytest.mark.parametrize("n,L,rc", [
    (33, (8.5, 8.5, 8.5), 2.5),       # three cells an axis, one atom in the second warp
    (864, (8.4, 8.7, 11.19), 2.5),    # dense, runs that wrap at both ends
    (1601, (11.1, 11.1, 11.1), 2.5),  # three wide cells, more than 128 candidates a run
    (700, (60.0, 9.0, 9.0), 2.5),     # long rows
    (257, (9.0, 40.0, 40.0), 2.5),    # a few atoms a row, empty cells
    (2500, (23.1, 14.0, 17.3), 3.0),
    (6000, (11.1, 11.1, 11.1), 2.5),  # nine warps per 32 atoms, more words than fit
    (34001, (40.0, 35.0, 37.0), 2.5),  # three warps (from 33,700 atoms on 148 multiprocessors)
    (34001, (18.0, 18.0, 18.0), 2.5),  # the same, more words than fit
    (203001, (64.0, 63.0, 62.0), 2.5),  # one warp (from 202,100)
])
def test_rows_equal_the_general_walk(n, L, rc):
    rng = np.random.Generator(np.random.Philox(n))
    q = rng.uniform(0.0, 1.0, (n, 3)) * np.array(L)
    q[: n // 16, 0] = 0.0                       # on the low face
    q[n // 16: n // 8, 1] = np.nextafter(L[1], 0.0)
    a = _rows(q, L, rc, 1)
    for lanes in (2, 8):
        b = _rows(q, L, rc, lanes)
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("n,L", [(500, (8.2, 8.2, 8.2)), (37, (5.7, 30.0, 8.6)), (130, (6.0, 6.0, 90.0)),
                                 (4700, (8.2, 8.2, 8.2))])
def test_small_replica_sums(n, L):
    # an axis shorter than three cells: every pair through its minimum image
    rng = np.random.Generator(np.random.Philox(n))
    # sites of a jittered grid: no overlaps
    m = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    q = (g + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) / m * np.array(L)
    ens = M.Ensemble([(q, np.zeros_like(q), np.array(L))], cutoff=2.5, time_step=0.005)
    _, pe, vir = ens.observe()
    entries, within = ens.list_stats()
    ens.close()
    d = q[:, None] - q[None]
    d -= np.array(L) * np.round(d / np.array(L))
    r2 = (d * d).sum(2)[np.triu_indices(n, 1)]
    assert entries == 2 * int((r2 <= 2.8 ** 2).sum())
    assert within == int((r2 <= 2.5 ** 2).sum())
    x = r2[r2 <= 6.25]
    s6 = 2.5 ** -6
    c2 = (6 * s6 * s6 - 3 * s6) / 6.25
    c0 = -s6 * s6 + s6 - c2 * 6.25
    # sums of up to 2 x 10^4 positive and negative terms, each rounded a few times
    assert pe[0] == pytest.approx(np.sum(4 * (x ** -6 - x ** -3 + c2 * x + c0)), rel=1e-11)
    assert vir[0] == pytest.approx(np.sum(((24 * x ** 3 - 48) / x ** 7 + 8 * c2) * x) / 3, rel=1e-11)


@pytest.mark.parametrize("cells", [16, 45, 60])
def test_replica_rows_equal_a_systems(cells):
    # 33,000, 729,000 and 1,728,000 atoms in all: nine, three and one warp per
    # 32 atoms, all of whose replicas rebuild; one replica is all-pairs
    reps = [W.fcc_liquid((cells,) * 3, 0.8, 1.0, seed=1, jitter=0.05, rc=2.5, dt=0.005),
            W.fcc_liquid((4, 4, 4), 0.8, 1.0, seed=2, jitter=0.05, rc=2.5, dt=0.005),
            W.fcc_liquid((cells,) * 3, 0.7, 1.0, seed=3, jitter=0.05, rc=2.5, dt=0.005)]
    ens = M.Ensemble([(r.q, r.v, r.L) for r in reps], cutoff=2.5, time_step=0.005)
    ens.observe()  # builds the lists
    got = ens.list_stats()
    ens.close()
    entries = within = 0
    for r in reps:
        if min(r.L) < 3 * 2.8:
            d = r.q[:, None] - r.q[None]
            d -= np.array(r.L) * np.round(d / np.array(r.L))
            r2 = (d * d).sum(2)[np.triu_indices(r.n, 1)]
            entries += 2 * int((r2 <= 2.8 ** 2).sum())
            within += int((r2 <= 2.5 ** 2).sum())
            continue
        s = M.System(r.L, cutoff=2.5, time_step=0.005, capacity=r.n, build_block=128, build_threads_per_atom=2)
        s.set_state(r.q, r.v)
        s.make_pairlist()
        w, e = s.pair_counts()
        entries, within = entries + e, within + w // 2
        s.close()
    assert got == (entries, within)


def test_fp64_sums_do_not_depend_on_the_lane_count():
    # 864 atoms run with 8 lanes an atom, 11,664 with 4, the ensemble of all
    # of them with 1 (over 65,536 atoms): the same trajectories bit for bit,
    # rows short and long, with and without partners beyond a face
    reps = [W.fcc_liquid(c, rho, 1.0, seed=c, jitter=0.05, rc=2.5, dt=0.005)
            for c, rho in ((6, 0.3), (6, 0.8), ((18, 18, 9), 0.85), ((23, 24, 27), 0.6))]
    assert sum(r.n for r in reps) > 65536
    ens = M.Ensemble([(r.q, r.v, r.L) for r in reps], cutoff=2.5, time_step=0.005, precision=M.FP64)
    ens.calculate(23)
    got = ens.states_by_id()
    ens.close()
    for k, r in enumerate(reps):
        s = M.System(r.L, cutoff=2.5, time_step=0.005, capacity=r.n, precision=M.FP64)
        s.set_state(r.q, r.v)
        s.calculate(23)
        q, v = s.state_by_id()
        s.close()
        assert np.array_equal(got[k][0], q) and np.array_equal(got[k][1], v), f"replica {k}"
