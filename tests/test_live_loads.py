"""The persistent pass rewrites the packed copies that it reads (k_nve_persistent:
each step reads one and writes the other), so nothing on its path may read them
through the read-only cache, whose loads are undefined for data that the kernel
writes.  What the compiler makes of such a load differs from one version to the
next, so this is checked in the source."""
from __future__ import annotations

import pathlib
import re

SOURCE = (pathlib.Path(__file__).resolve().parents[1] / "mdacp_b200" / "csrc" / "mdg_device.cuh").read_text()


def _body(signature):
    """The braces that follow the one place where `signature` is defined."""
    start = SOURCE.index("{", SOURCE.index(signature))
    depth = 0
    for k in range(start, len(SOURCE)):
        depth += {"{": 1, "}": -1}.get(SOURCE[k], 0)
        if depth == 0:
            return SOURCE[start:k + 1]
    raise AssertionError(signature)


def test_persistent_pass_reads_its_copies_with_ordinary_loads():
    persistent = _body("k_nve_persistent(Arrays a")
    deep = _body("void fp32_row_deep(")
    groups = _body("struct GlobalGroups ")
    for name, body in (("k_nve_persistent", persistent), ("fp32_row_deep", deep), ("GlobalGroups", groups)):
        assert not re.search(r"__ldg\(\s*&?\s*\(?(qf|q0|q1)", body), f"{name} reads a packed copy with __ldg"
    # the shared helpers are asked for their ordinary-load form
    assert re.findall(r"GlobalGroups<([^>]*)>", persistent) == ["true, true"]
    assert set(re.findall(r"packed_at<(\w+)>", deep)) == {"true"}
    assert set(re.findall(r"packed_at<(\w+)>", groups)) == {"LIVE"}
