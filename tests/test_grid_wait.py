"""Every kernel waits for the kernel before it: kernels go out with programmatic stream serialization
(csrc/internal.cuh, launch), under which a grid may start before its predecessor's writes are
visible, so each must pass griddepcontrol.wait before it touches memory."""
import glob
import os
import re

import pytest

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "cylinder-fem-amr_b200", "csrc")
# the macro, the instruction itself, and the tile loops that hold the wait (tiled.cuh)
WAITS = ("CFA_GRID_DEP()", "griddepcontrol.wait", "tile_loop_dep")


def _strip(src):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def _body(src, at):
    """The braces' content that opens at or after `at`, None for a declaration."""
    brace, semi = src.find("{", at), src.find(";", at)
    if brace < 0 or 0 <= semi < brace:
        return None
    depth = 0
    for k in range(brace, len(src)):
        depth += (src[k] == "{") - (src[k] == "}")
        if depth == 0:
            return src[brace + 1:k]
    raise AssertionError("unbalanced braces")


def kernels():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = _strip(open(path).read())
        for m in re.finditer(r"\b__global__\b", src):
            name = re.search(r"\b(k_\w+)\s*\(", src[m.end():])
            body = _body(src, m.end())
            if name and body is not None:
                out.append((os.path.basename(path), name.group(1), body))
    return out


KERNELS = kernels()


def test_kernels_are_found():
    names = {k for _, k, _ in KERNELS}
    assert len(names) > 60 and {"k_momentum_rows", "k_vct", "k_ring", "k_elem_tiles"} <= names


@pytest.mark.parametrize("path,name,body", KERNELS, ids=[f"{p}:{k}" for p, k, _ in KERNELS])
def test_kernel_waits_for_its_predecessor(path, name, body):
    assert any(w in body for w in WAITS), f"{name} in {path} never waits for the kernel before it"


def test_element_tile_plan_waits_before_its_first_read():
    body = next(b for _, k, b in KERNELS if k == "k_elem_tiles")
    wait = body.find("CFA_GRID_DEP()")
    first = min(body.find(w) for w in ("inc_ptr[", "inc[", "pos[", "rp[") if w in body)
    assert 0 <= wait < first
