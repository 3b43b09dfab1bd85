"""The mixed-precision path keeps the order of its single-precision sums: its tangent,
hierarchy and linear solutions against the values in golden/single_precision.npz
(golden/make_single_precision.py)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_single_precision as G  # noqa: E402

pytestmark = pytest.mark.gpu

# A sum in another order differs in more than a tenth of the entries; the same order may
# meet, rarely, a double on the other side of a rounding boundary.
RARE = 1e-3


@pytest.fixture(scope="module")
def kept():
    return np.load(G.PATH)


@pytest.mark.parametrize("i", range(len(G.TANGENTS)))
def test_tangent(kept, i):
    K = G.tangent(*G.TANGENTS[i])
    assert np.mean(K != kept["tangent_%d" % i]) <= RARE


def test_hierarchy(kept):
    P, A = G.hierarchy()
    assert np.mean((P != kept["prolongator"])[P != 0]) <= RARE
    assert np.mean((A != kept["galerkin"])[A != 0]) <= RARE


@pytest.mark.parametrize("i", range(len(G.SOLVES)))
def test_solution(kept, i):
    x, y = G.solution(*G.SOLVES[i]).astype(float), kept["solution_%d" % i].astype(float)
    # the bound for a single-precision result; the same order gives the same bits
    assert np.linalg.norm(x - y) <= 2e-5 * np.linalg.norm(y)
