"""The FP64 pair terms' division (a Newton step on the hardware's reciprocal and
a residual correction instead of the operator) against IEEE division, through
forces and observers of isolated pairs: for one pair every other operation is
rounded as NumPy rounds it, so results differ only where a quotient does.
Distances from 1e-12 (the shortest that coordinates of this size resolve) to the
cut-off.

The quotient before its last rounding is good to about 2^-80, so it is the
correctly rounded one or, for some 2^-80 / 2^-53 = 1e-8 of operands, its
neighbour: at most one in 1e6 may differ here, by a unit in the last place."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M

pytestmark = pytest.mark.gpu
RC = 2.5
S2 = 1.0 / (RC * RC)
S6 = S2 * S2 * S2
C2 = 6.0 * (S6 * S6 * S2) - 3.0 * (S6 * S2)
C0 = -(S6 * S6) + S6 - C2 / S2


def _distances(rng, n):
    r = np.where(rng.uniform(size=n) < 0.5, rng.uniform(0.6, RC, n), np.exp(rng.uniform(np.log(1e-12), np.log(RC), n)))
    r[:8] = [1.0, 2.0 ** (1.0 / 6.0), 2.0, RC, np.nextafter(RC, 0.0), 1e-12, 0.5, 1e-3]
    return r


def _r2(d):
    return d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]


@pytest.mark.parametrize("m", [12, 24, 34])  # 3,456, 27,648 and 78,608 atoms: 8, 4 and 1 lanes
def test_forces_of_pairs(m):
    rng = np.random.Generator(np.random.Philox(m))
    n = m ** 3
    site = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * 8.0  # pairs out of reach of one another
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1)[:, None]
    other = site + e * _distances(rng, n)[:, None]
    s = M.System([8.0 * m] * 3, cutoff=RC, time_step=0.005, capacity=2 * n, precision=M.FP64)
    s.set_state(np.concatenate([site, other]), np.zeros((2 * n, 3)))
    got = s.forces_by_id()
    s.close()
    for sign, f in ((1.0, got[:n]), (-1.0, got[n:])):
        d = sign * (other - site)
        r2 = _r2(d)
        r6 = (r2 * r2) * r2
        q = (24.0 * r6 - 48.0) / ((r6 * r6) * r2)
        df = q + C2 * 8.0
        want = np.where((r2 > RC * RC)[:, None] | (r2 == 0.0)[:, None], 0.0, df[:, None] * d)
        ok = r2 > 0.0
        differ = (f[ok] != want[ok]).any(axis=1)
        assert differ.sum() <= 1e-6 * n + 1
        assert (np.abs(f[ok] - want[ok]) <= 2.0 ** -51 * np.maximum(np.abs(q[ok, None] * d[ok]), np.abs(want[ok]))).all()


def test_sums_of_single_pairs():
    rng = np.random.Generator(np.random.Philox(5))
    r = _distances(rng, 1500)
    s = M.System([9.0] * 3, cutoff=RC, time_step=0.005, capacity=2, precision=M.FP64)
    at = np.array([4.4, 4.5, 4.6])
    differ = 0
    for k in range(len(r)):
        e = rng.normal(size=3)
        q = np.stack([at, at + e / np.linalg.norm(e) * r[k]])
        d = (q[0] - q[1])[None]
        r2 = _r2(d)[0]
        if r2 == 0.0 or r2 > RC * RC:
            continue
        s.set_state(q, np.zeros((2, 3)))
        _, pe, vir = s.observe()
        r4 = r2 * r2
        r6 = r4 * r2
        r12 = ((r6 * r2) * r2) * r2
        want = 4.0 * (((1.0 / r12 - 1.0 / r6) + C2 * r2) + C0)
        w = ((24.0 * r6 - 48.0) / ((r6 * r6) * r2) + C2 * 8.0) * r2 / 3.0
        differ += pe != want or vir != w
        assert abs(pe - want) <= 2.0 ** -51 * max(4.0 / r12, abs(want))
        assert abs(vir - w) <= 2.0 ** -51 * max(48.0 / r12, abs(w))
    s.close()
    assert differ <= 1
