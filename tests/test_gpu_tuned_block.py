"""The list build's block size, chosen by timing, says what runs: where warps
share atoms' rows the block size is not used, and is not a timing's noise."""
from __future__ import annotations

import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_shared_rows_have_one_block_size():
    blocks = []
    for cut in range(14):  # the choice is kept per atom count: each is timed
        w = W.fcc_liquid(10, 0.8, 1.0, seed=1, jitter=0.05, rc=2.5, dt=0.005)
        s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, build_threads_per_atom=1)
        s.set_state(w.q[cut:], w.v[cut:])
        s.calculate(1)
        blocks.append(s.info()["build_block"])
        s.close()
    assert set(blocks) == {128}


@pytest.mark.parametrize("block", [64, 128, 256])
def test_a_given_block_stays(block):
    w = W.fcc_liquid(10, 0.8, 1.0, seed=1, jitter=0.05, rc=2.5, dt=0.005)
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, build_block=block)
    s.set_state(w.q, w.v)
    s.calculate(1)
    assert s.info()["build_block"] == block and s.info()["build_threads_per_atom"] in (1, 2, 4, 8)
    s.close()
