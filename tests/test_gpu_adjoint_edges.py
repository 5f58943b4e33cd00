"""The adjoint's passes where their split can go wrong, against the dense
autograd oracle with the bars of tests/test_adjoint.py: rows longer than the
128 entries that a warp sorts in registers, an odd atom count, a single
segment and segments that do not divide the steps, no skin (the narrowest box:
a rebuild at every evaluation), a shell too sharp for the one-exponential form,
epsilon and sigma other than 1, atoms outside the box."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import torch_lj_reference as R
from mdacp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,cut,steps,every,shell,eps,sigma,drop", [
    (7, 3.6, 12, 5, (1.0, 1.5, 0.05), 1.0, 1.0, 1),      # rows of about 200, 1,371 atoms
    (5, 2.5, 9, 20, (1.0, 1.5, 0.05), 1.1, 0.98, 3),     # one segment, 497 atoms
    (6, 2.5, 33, 4, (1.0, 1.5, 0.004), 0.9, 1.01, 0),    # sharp shell
    (5, 2.799, 6, 3, (1.0, 1.5, 0.05), 1.0, 1.0, 0),     # three cells of the cut-off, no skin
])
@pytest.mark.parametrize("lanes", [1, 4, 8])
def test_edges_match_dense_autograd(cells, cut, steps, every, shell, eps, sigma, drop, lanes):
    from mdacp_b200 import adjoint as A
    st = W.fcc_liquid(cells, 0.8442, 1.0, 55 + cells, jitter=0.05, rc=cut, dt=0.005)
    n = st.n - drop
    q0, v0 = st.q[:n].copy(), st.v[:n].copy()
    q0[::7] += np.array([1.0, -2.0, 0.0]) * st.L  # images of the same system
    loss, de, ds, dq = A.trajectory_gradients(q0, v0, st.L, steps=steps, checkpoint_every=every, cutoff=cut,
                                              shell=shell, epsilon=eps, sigma=sigma, threads_per_atom=lanes)
    q, v, L, e, s = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (q0, v0, st.L, eps, sigma))
    for x in (q, e, s):
        x.requires_grad_(True)
    ref = R.trajectory_loss(q, v, L, e, s, steps=steps, sc=cut, shell=shell)
    gq, ge, gs = torch.autograd.grad(ref, (q, e, s))
    assert loss == pytest.approx(float(ref.detach()), rel=1e-11)
    assert de == pytest.approx(float(ge), rel=1e-8)
    assert ds == pytest.approx(float(gs), rel=1e-8)
    assert np.linalg.norm(dq - gq.cpu().numpy()) <= 1e-8 * np.linalg.norm(gq.cpu().numpy())
    assert loss == A.trajectory_loss(q0, v0, st.L, steps=steps, cutoff=cut, shell=shell, epsilon=eps, sigma=sigma,
                                     threads_per_atom=lanes)
