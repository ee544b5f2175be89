"""After a fatal error the cell and leaf counts of a tree may be set while its
records are not: a kernel that walks them has to look at the error word first.
Checked in the source, since a kernel that does not may read out of range."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lsmps_vpm_v2_b200", "csrc")
COUNTS = re.compile(r"info->n_(?:cells|leaves)\b(?!\s*=[^=])")   # read, not set


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"__global__[^;{]*?\b(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
            yield os.path.basename(path), m.group(1), text[m.end():text.index("\n}", m.end())]


WALKERS = [(f, name, body) for f, name, body in kernels() if COUNTS.search(body)]


def test_walkers_found():
    assert {"l2l_leaves2d", "near2d_f64", "flat_link", "p2m3d"} <= {name for _, name, _ in WALKERS}


@pytest.mark.parametrize("file,name,body", WALKERS, ids=[f"{f}:{n}" for f, n, _ in WALKERS])
def test_error_word_before_loops(file, name, body):
    m = re.search(r"\bfatal\(|\bblock_fatal\(", body)
    assert m and m.start() < max(COUNTS.search(body).start(), body.find("for ("))   # before the loops over them
