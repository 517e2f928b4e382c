"""The one-block grid where its shared memory just passes 48 KB, the room that a block has
without asking (12288 words, of which the kernel's static arrays take 33): each size is the
first such grid of a process."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
import numpy as np
import freud_gb300 as freud
from oracle import oracle as O
n, L, kind = int(sys.argv[1]), [float(x) for x in sys.argv[2].split(",")], sys.argv[3]
box = freud.box.Box(*L)
pts = ((np.random.RandomState(n).random_sample((n, 3)) - 0.5) * np.array(L)).astype(np.float32)
if kind == "list":
    nl = freud.locality.LinkCell(box, pts, 1.0).query(pts, dict(r_max=1.0, exclude_ii=True)).toNeighborList()
    ij, d, v = O.query(box, pts, r_max=1.0, exclude_ii=True, arith=O.ARITH_WRAP)
    np.testing.assert_array_equal(np.asarray(nl[:]), ij)
    np.testing.assert_array_equal(np.asarray(nl.vectors), v)
else:
    rdf = freud.density.RDF(40, 1.0)
    rdf.compute((box, pts))
    np.testing.assert_array_equal(rdf.bin_counts_u64, O.rdf_counts_query(box, pts, 40, 1.0))
"""


# lists: cells in index order, 2 n + cells + 1 words (8^3 cells); RDF: n + cells + 1 (15 x 71 x 4 cells)
@pytest.mark.parametrize("n", [5870, 5871, 5880, 5886, 5887, 5888])
def test_list(n):
    run(n, "8.5,8.5,8.5", "list")


@pytest.mark.parametrize("n", [7993, 7994, 8010, 8026, 8027, 8028])
def test_rdf(n):
    run(n, "15.5,71.5,4.5", "rdf")


def run(n, box, kind):
    res = subprocess.run([sys.executable, "-c", SCRIPT, str(n), box, kind], cwd=ROOT, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
