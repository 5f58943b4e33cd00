"""Ensemble calls at the ends of their range: no atoms at all, and the list's
figures asked for before any step has built a list."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("nrep", [1, 9])
def test_replicas_without_atoms(precision, nrep):
    none = np.zeros((0, 3))
    ens = M.Ensemble([(none, none, np.array([9.0, 10.0, 11.0]))] * nrep, cutoff=2.5, precision=precision)
    for _ in range(2):
        ens.calculate(3)
        assert all(np.array_equal(x, np.zeros(nrep)) for x in ens.observe())
        assert ens.list_stats() == (0, 0)
    ens.close()


def test_list_figures_before_any_step():
    # rows that no build has written yet, and rows of an earlier upload, are not walked
    def system(seed, n, L):
        rng = np.random.Generator(np.random.Philox(seed))
        return rng.uniform(0.0, 1.0, (n, 3)) * L

    def counts(q, L, reach):
        d = q[:, None] - q[None]
        d -= L * np.round(d / L)
        return int(((d * d).sum(2)[np.triu_indices(len(q), 1)] <= reach * reach).sum())

    Ls = [np.array([9.0, 10.0, 11.0]), np.array([7.0, 8.0, 30.0])]
    sets = [[system(10 * k + m, 300 + 100 * m, L) for m, L in enumerate(Ls)] for k in range(2)]
    ens = M.Ensemble([(q, 0.0 * q, L) for q, L in zip(sets[0], Ls)], cutoff=2.5)
    for qs in sets:
        q4 = np.zeros((sum(map(len, qs)), 4))
        q4[:, :3] = np.concatenate(qs)
        v4 = np.zeros_like(q4)
        dp = [a.ctypes.data_as(M._DP) for a in (q4, v4)]
        assert ens.lib.mdg_ensemble_set_state(ens.h, *dp) == 0
        assert ens.list_stats() == (2 * sum(counts(q, L, 2.8) for q, L in zip(qs, Ls)),
                                    sum(counts(q, L, 2.5) for q, L in zip(qs, Ls)))
    ens.close()
