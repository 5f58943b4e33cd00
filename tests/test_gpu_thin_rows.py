"""Rows of atoms that lie thin, where a warp's lanes walk alone instead of taking
turns (build_rows_warp): entry for entry the general walk's, at densities and
shapes on both sides of the rule, with one, three and nine warps per 32 atoms,
rows longer than their capacity, atoms on the faces, and replicas of an ensemble
that mix thin, dense and all-pairs systems; a dense drop in a thin gas has both
walks in one build."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M

pytestmark = pytest.mark.gpu


def _gas(n, L, seed):
    rng = np.random.Generator(np.random.Philox(seed))
    q = rng.uniform(0.0, 1.0, (n, 3)) * L
    q[: n // 50, 0] = 0.0
    q[n // 50: n // 25, 1] = np.nextafter(L[1], 0.0)
    q[n // 25: n // 20, 2] = 0.0
    return q


def _rows(q, L, lanes, **kw):
    s = M.System(L, cutoff=2.5, capacity=len(q), build_block=128, build_threads_per_atom=lanes, **kw)
    s.set_state(q, np.zeros_like(q))
    s.make_pairlist()
    out = (*s.neighbor_list(), s.ids())
    s.close()
    return out


@pytest.mark.parametrize("n,L", [
    (40, (30.0, 30.0, 30.0)),          # a few atoms a row, nine warps
    (3000, (9.0, 200.0, 200.0)),       # three cells a row
    (3000, (45.0, 45.0, 15.0)),        # 0.1: about the rule's line for nine warps
    (30001, (9.0, 182.0, 182.0)),      # 0.1, seven atoms a row
    (60001, (130.0, 130.0, 130.0)),    # 0.03: one warp instead of three
    (60001, (9.0, 260.0, 260.0)),
    (120001, (20.0, 141.0, 141.0)),    # 0.3: three warps in turns
    (250001, (9.0, 700.0, 400.0)),     # 0.1
    (250001, (45.0, 80.0, 170.0)),     # 0.4
])
def test_rows_equal_the_general_walk(n, L):
    L = np.array(L)
    q = _gas(n, L, n)
    a = _rows(q, L, 1)
    b = _rows(q, L, 2)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [20001, 60001, 220001])
def test_a_drop_in_a_gas(n):
    L = np.array([120.0, 130.0, 140.0])
    q = _gas(n, L, n)
    q[: n // 2] = 0.5 * L + (q[: n // 2] / L - 0.5) * (n / 2 / 0.8) ** (1.0 / 3.0)
    a = _rows(q, L, 1)  # grows the rows' capacity where the estimate falls short
    b = _rows(q, L, 8)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_rows_longer_than_their_capacity_grow():
    L = np.array([9.0, 300.0, 300.0])
    q = _gas(3000, L, 5)
    q[:60] = q[0] + np.linspace(0.0, 0.5, 60)[:, None]  # one bunch of 60 atoms
    q = np.clip(q, 0.0, np.nextafter(L, 0.0))
    a = _rows(q, L, 1, max_neighbors=8)
    b = _rows(q, L, 2)
    assert a[0].max() > 8
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_replicas_equal_systems(precision):
    # thin, flat, dense and all-pairs replicas in one build; the same
    # trajectories as alone, bit for bit
    shapes = [(500, (60.0, 60.0, 60.0)), (700, (9.0, 150.0, 150.0)), (864, (10.2, 10.2, 10.2)), (90, (6.0, 7.0, 40.0)),
              (33, (30.0, 9.0, 30.0)), (2048, (13.6, 13.6, 13.6)), (1000, (20.0, 100.0, 60.0)), (5, (12.0, 12.0, 12.0))]
    reps = []
    for k, (n, L) in enumerate(shapes):
        L = np.array(L)
        rng = np.random.Generator(np.random.Philox(k))
        m = np.ceil(L / (np.prod(L) / n) ** (1 / 3)).astype(int)
        g = np.stack(np.meshgrid(*[np.arange(i) for i in m], indexing="ij"), -1).reshape(-1, 3)
        g = g[np.sort(rng.permutation(len(g))[:n])]
        q = (g + 0.5 + rng.uniform(-0.05, 0.05, (n, 3))) * L / m
        reps.append((q, rng.normal(0.0, 0.5, (n, 3)), L))
    ens = M.Ensemble(reps, cutoff=2.5, time_step=0.002, precision=precision)
    ens.calculate(40)
    got = ens.states_by_id()
    ens.close()
    for (q, v, L), (gq, gv) in zip(reps, got):
        if min(L) < 3 * 2.8:
            continue
        s = M.System(L, cutoff=2.5, time_step=0.002, capacity=len(q), precision=precision, build_block=64,
                     build_threads_per_atom=4)
        s.set_state(q, v)
        s.calculate(40)
        sq, sv = s.state_by_id()
        s.close()
        assert np.array_equal(gq, sq) and np.array_equal(gv, sv)


def test_slabs_of_a_gas():
    L = np.array([60.0, 50.0, 120.0])
    q = _gas(4000, L, 2)
    # no two atoms closer than 0.9: a lattice's gaps
    m = np.array([18, 14, 18])
    g = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)[:4000]
    q = (g + 0.5) * L / m
    v = np.random.Generator(np.random.Philox(1)).normal(0.0, 1.0, q.shape)
    x = M.Slabs(L, 3, cutoff=2.5, time_step=0.004, capacity=len(q))
    x.set_state(q, v)
    x.calculate(60)
    a = x.state_by_id()
    x.close()
    s = M.System(L, cutoff=2.5, time_step=0.004, capacity=len(q), build_block=64, build_threads_per_atom=8)
    s.set_state(q, v)
    s.calculate(60)
    b = s.state_by_id()
    s.close()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
