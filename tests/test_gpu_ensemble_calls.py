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
