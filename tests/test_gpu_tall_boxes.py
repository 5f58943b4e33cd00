"""Boxes of more than 512 cell layers along z, whose packed cell coordinates use
the sign bit: the general row walk (several lanes an atom; rows with stage
indices) against the one-lane walk, and against the pairs themselves."""
from __future__ import annotations

import numpy as np
import pytest

import mdacp_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [512, 513, 700, 1022])
def test_rows_of_tall_boxes(layers):
    L = np.array([8.5, 8.6, 2.8 * layers + 1.0])
    rng = np.random.Generator(np.random.Philox(layers))
    n = 3001
    # three bunches: at the lower face, around the layer where the sign bit sets in, at the upper face
    z = np.concatenate([rng.uniform(0, 12, 1000), rng.uniform(0, 30, 1001) + min(512 * 2.8 - 15, L[2] - 30),
                        L[2] - rng.uniform(0, 12, 1000)])
    q = np.stack([rng.uniform(0, L[0], n), rng.uniform(0, L[1], n), np.minimum(z, np.nextafter(L[2], 0))], 1)
    out = {}
    for name, kw in (("one", dict(build_threads_per_atom=1)), ("two", dict(build_threads_per_atom=2)),
                     ("eight", dict(build_threads_per_atom=8)),
                     ("stage", dict(precision=M.FP32_MIXED, stage_atoms=-1))):
        s = M.System(L, cutoff=2.5, capacity=n, **kw)
        s.set_state(q, np.zeros_like(q))
        s.make_pairlist()
        out[name] = (*s.neighbor_list(), s.ids())
        s.close()
    for name in ("two", "eight", "stage"):
        for a, b in zip(out["one"], out[name]):
            assert np.array_equal(a, b), name
    order = np.argsort(q[:, 2])
    entries = 0
    for i in range(0, n, 500):  # pairs within SearchLength, in blocks along z
        d = q[order[i:i + 500], None] - q[None]
        d -= L * np.round(d / L)
        entries += int(((d * d).sum(2) <= 2.8 ** 2).sum()) - len(d)
    assert int(out["one"][0].sum()) == entries
