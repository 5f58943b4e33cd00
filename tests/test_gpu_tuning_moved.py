"""The first step's timing of list-build shapes leaves the list as it is when the
atoms have moved since it was built: after a step made piece by piece, and in a
process that goes on from a checkpoint."""
from __future__ import annotations

import pathlib
import subprocess
import sys

import numpy as np
import pytest

import mdacp_b200 as M
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("cells,cut", [(9, 17), (20, 23), (38, 29)])
def test_rows_stay(cells, cut, precision):
    # atom counts of their own: each is timed
    w = W.fcc_liquid(cells, 0.8, 1.0, seed=cells, jitter=0.05, rc=2.5, dt=0.005)
    n = w.n - cut - precision
    s = M.System(w.L, cutoff=2.5, time_step=0.01, capacity=n, precision=precision)
    s.set_state(w.q[:n], w.v[:n])
    s.make_pairlist()
    before = s.neighbor_list()
    for _ in range(3):
        s.update_position_half()
    s.calculate(1)
    info = s.info()
    assert info["build_block"] > 0 and info["rebuilds"] == 1
    after = s.neighbor_list()
    s.close()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])


GO_ON = """
import sys
import numpy as np
import mdacp_b200 as M
L = [float(x) for x in sys.argv[3:6]]
s = M.System(L, cutoff=2.5, time_step=0.005, capacity=int(sys.argv[2]), precision=int(sys.argv[6]))
s.load_checkpoint(sys.argv[1])
s.calculate(30)
q, v = s.state_by_id()
np.savez(sys.argv[7], q=q, v=v, rebuilds=s.info()["rebuilds"])
"""


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
def test_another_process_goes_on_bit_for_bit(precision, tmp_path):
    w = W.fcc_liquid(14, 0.8, 1.2, seed=3, jitter=0.05, rc=2.5, dt=0.005)
    s = M.System(w.L, cutoff=2.5, time_step=0.005, capacity=w.n, precision=precision)
    s.set_state(w.q, w.v)
    s.calculate(23)
    s.save_checkpoint(tmp_path / "c.ck")
    s.calculate(30)
    q, v = s.state_by_id()
    rebuilds = s.info()["rebuilds"]
    s.close()
    subprocess.run([sys.executable, "-c", GO_ON, str(tmp_path / "c.ck"), str(w.n), *[repr(float(x)) for x in w.L],
                    str(int(precision)), str(tmp_path / "o.npz")], check=True, cwd=ROOT, timeout=200)
    with np.load(tmp_path / "o.npz") as o:
        assert int(o["rebuilds"]) == rebuilds
        assert np.array_equal(o["q"], q) and np.array_equal(o["v"], v)
