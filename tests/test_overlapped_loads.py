"""Kernels that start with grid_wait live while the kernel before them still writes, so
what that kernel writes must not be read through the non-coherent path: there __ldg
takes constant tables only (and, in the forward y pass, the state, which was complete
before the x pass in front of it began), and no pointer is __restrict__ (which would let
the compiler choose that path)."""

import glob
import os
import re

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
# tables of a handle, written when it is created
TABLES = r"a\.(lin\.)?(d1|d2|DD1|DD2|(inv_|d3_)?alpha_c|(d3_)?alpha_i)\b"
# the state in the epilogue of k_fwd_yl
COMPLETE = {"bld_ylines.cuh": r"S[0z] \+"}


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _function(code, name):
    """Text of the function `name`, from its name to its closing brace."""
    a = code.index(name + "(")
    i = code.index("{", a)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(code[j], 0)
        j += 1
        if depth == 0:
            return code[a:j]


def test_overlapped_kernels_read_written_data_coherently():
    files = [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cuh")))
             if os.path.basename(p) != "bld_tma.cuh" and "grid_wait();" in _code(p)]
    assert {os.path.basename(p) for p in files} == {"bld_xrows.cuh", "bld_ylines.cuh", "bld_project_tile.cuh"}
    texts = {os.path.basename(p): _code(p) for p in files}
    # what they call elsewhere to read the state
    texts["y2_term"] = _function(_code(os.path.join(CSRC, "bld_ypass2.cuh")), "y2_term")
    for name, text in texts.items():
        allowed = "|".join([TABLES, COMPLETE.get(name, TABLES)])
        bad = [m.group(1) for m in re.finditer(r"__ldg\(([^)]*)", text) if not re.match(allowed, m.group(1).strip())]
        assert not bad, (name, bad)
        assert "__restrict__" not in text, name
