"""The coarsest level's inverse with partial pivoting (up to 300 unknowns, one cluster
launch): sizes at the edges of its panels and of its two variants, both types."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


# boxes whose first aggregation leaves 6, 12, 48, 162, 180, 216 and 300 unknowns
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,unknowns", [((2, 2, 2), 6), ((5, 2, 2), 12), ((4, 4, 4), 48), ((8, 8, 8), 162), ((14, 8, 5), 180),
                                        ((17, 8, 5), 216), ((14, 5, 14), 300)])
def test_inverse_times_operator(n, unknowns, precision):
    m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, np.random.default_rng(1))
    M = P.Model(m, P.J2Material(**W.MAT))
    M.fix(P.on_face(m, "zmin"))
    M.prescribe(P.on_face(m, "zmax"), "z", -0.005 * n[2])
    _, R = M.residual(0.1, precision=precision)
    M.linear_solve(-R, rtol=0.1, precision=precision)
    A, Ai = M.amg_dense(1, 0), M.amg_dense(1, 2)
    assert A.shape == (unknowns, unknowns)
    nz = np.abs(A).sum(axis=1) > 0  # a row without entries has a unit diagonal in the inverse
    A[~nz, ~nz] = 1.0
    # elimination with pivoting is backward stable: growth times n eps times the condition
    # number, and the inverse is rounded to the path's type
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    tol = (100 * A.shape[0] * 2.0 ** -53 + A.shape[0] ** 0.5 * eps) * np.linalg.cond(A)
    assert np.abs(Ai @ A - np.eye(unknowns)).max() <= tol
