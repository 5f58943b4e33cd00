"""Adjoint calls at the ends of their range, against the dense autograd oracle
with the bars of tests/test_adjoint.py."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import torch_lj_reference as R
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(q0, v0, L, steps, cut, **kw):
    from mdacp_b200 import adjoint as A
    loss, de, ds, dq = A.trajectory_gradients(q0, v0, L, steps=steps, checkpoint_every=4, cutoff=cut, **kw)
    q, v, box, e, s = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (q0, v0, L, 1.0, 1.0))
    for x in (q, e, s):
        x.requires_grad_(True)
    ref = R.trajectory_loss(q, v, box, e, s, steps=steps, sc=cut)
    gq, ge, gs = torch.autograd.grad(ref, (q, e, s))
    assert loss == pytest.approx(float(ref.detach()), rel=1e-11)
    assert de == pytest.approx(float(ge), rel=1e-8)
    assert ds == pytest.approx(float(gs), rel=1e-8)
    assert np.linalg.norm(dq - gq.cpu().numpy()) <= 1e-8 * np.linalg.norm(gq.cpu().numpy())


@pytest.mark.parametrize("length", [9.0, 1.4e4, 1.5e4, 6e5, 5e6])
def test_a_dense_block_in_a_long_box(length):
    # the FP32 search's margin grows with the longest edge (1.1 at 6e5, more than
    # the rows have room for): beyond some 1.47e4 FP64 decides
    st = W.fcc_liquid(5, 0.8442, 1.0, 12, jitter=0.05, rc=2.5, dt=0.005)
    _check(st.q, st.v, np.array([9.0, 9.0, length]), 6, 2.5)


@pytest.mark.parametrize("cells,cut,drop", [
    (8, 3.0, 0),   # rows of about 128, some on either side
    (8, 3.9, 1),   # two parts and a little more
    (9, 4.9, 2),   # four parts
    (11, 6.1, 0),  # eight parts: rows of about 925
])
def test_long_rows(cells, cut, drop):
    # rows longer than the 128 entries that a warp sorts at a time
    st = W.fcc_liquid(cells, 0.8442, 1.0, 20 + cells, jitter=0.05, rc=2.5, dt=0.005)
    _check(st.q[: st.n - drop], st.v[: st.n - drop], st.L, 3, cut)
