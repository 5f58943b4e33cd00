"""A call that fails for want of device memory reports that once: other handles'
next calls do not report it again."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import adjoint as A
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def handle():
    w = W.fcc_liquid(6, 0.7, 1.0, seed=1, jitter=0.05, rc=2.5, dt=0.005)
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n)
    s.set_state(w.q, w.v)
    yield w, s
    s.close()


def test_a_handle_too_large(handle):
    w, s = handle
    f = s.forces()
    for _ in range(3):
        with pytest.raises(M.MdgError):  # rows of 2^31 entries: 275 GB
            M.System(w.L, cutoff=2.5, capacity=w.n, max_neighbors=2147483000)
        assert np.array_equal(s.forces(), f)
        s.calculate(1)
        s.observe()
        f = s.forces()


def test_an_adjoint_run_too_long(handle):
    w, s = handle
    f = s.forces()
    q = W.fcc_liquid(20, 0.8442, 1.0, seed=1, jitter=0.05, rc=2.5, dt=0.005)
    with pytest.raises(M.MdgError):  # a checkpoint at each of 10^6 steps: 1.5 TB
        A.trajectory_gradients(q.q, q.v, q.L, steps=1000000, checkpoint_every=1)
    assert np.array_equal(s.forces(), f)
    A.release()
