"""The coarsest level's inverse with partial pivoting at the edges of its three variants (up
to 192, 224 and 300 unknowns): bit for bit the elimination restated on the host.  The
kernel compares 11 bits of a pivot; no two candidates here are nearer than that."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    """a b + c rounded once: the product and the sum with their errors (Dekker, Knuth)."""
    def split(x):
        t = 134217729.0 * x
        h = t - (t - x)
        return h, x - h

    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    s = p + c
    v = s - p
    return s + (((p - (s - v)) + (c - v)) + e)


def inverse(A):
    """In-place Gauss-Jordan without row exchanges; a row is divided by its pivot at the end."""
    n = len(A)
    a, used = A.copy(), np.zeros(n, bool)
    rows, ip = np.zeros(n, int), np.zeros(n)
    for s in range(n):
        f = a[:, s].copy()
        p = int(np.argmax(np.where(used, -1.0, np.abs(f))))
        used[p], rows[s], ip[p] = True, p, 1.0 / f[p]
        f[p] = 0.0
        x = a[p] * ip[p]
        a = fma(-f[:, None], x[None], a)
        a[:, s] = -f * ip[p]
        a[p, s] = 1.0
    out = np.empty_like(a)
    pos = np.empty(n, int)
    pos[rows] = np.arange(n)
    out[np.ix_(pos, rows)] = a * ip[:, None]
    return out


# boxes whose first aggregation leaves 48, 192, 198, 222, 228 and 300 unknowns
@pytest.mark.parametrize("n,unknowns", [((4, 4, 4), 48), ((11, 11, 5), 192), ((32, 8, 2), 198), ((110, 2, 2), 222),
                                        ((56, 5, 2), 228), ((14, 5, 14), 300)])
def test_bits(n, unknowns):
    m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, np.random.default_rng(1))
    M = P.Model(m, P.J2Material(**W.MAT))
    M.fix(P.on_face(m, "zmin"))
    M.prescribe(P.on_face(m, "zmax"), "z", -0.005 * n[2])
    _, R = M.residual(0.1)
    M.linear_solve(-R, rtol=0.1)
    A, Ai = M.amg_dense(1, 0), M.amg_dense(1, 2)
    assert A.shape == (unknowns, unknowns)
    nz = np.abs(A).sum(axis=1) > 0  # a row without entries has a unit diagonal in the inverse
    A[~nz, ~nz] = 1.0
    assert np.array_equal(Ai, inverse(A))
