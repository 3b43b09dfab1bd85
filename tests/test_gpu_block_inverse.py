"""The blocked dense inverse of coarsest levels above 300 unknowns, at panel counts and
remainders where its tiles can go wrong, and with fewer column tiles than row shares."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,unknowns", [((8, 8, 17), 324), ((10, 9, 11), 384), ((13, 37, 2), 390), ((21, 17, 13), 1440)])
def test_inverse_to_rounding(n, unknowns, precision):
    m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, np.random.default_rng(3))
    M = P.Model(m, P.J2Material(**W.MAT))
    M.fix(P.on_face(m, "zmin"))
    M.prescribe(P.on_face(m, "zmax"), "z", -0.005 * n[2])
    _, R = M.residual(0.1, precision=precision)
    for _ in range(2):  # the second set-up runs on the first one's buffers
        M.linear_solve(-R, rtol=0.1, precision=precision)
    A, X = M.amg_dense(1, 0), M.amg_dense(1, 2)
    assert len(A) == unknowns
    nz = np.abs(A).sum(axis=1) > 0
    A[~nz, ~nz] = 1.0
    # elimination in double (A is exact in either precision), the result rounded to T
    eps, eps_t = 2.0 ** -53, 2.0 ** (-53 if precision == "fp64" else -24)
    cond = np.linalg.cond(A)
    assert np.linalg.norm(X @ A - np.eye(unknowns)) <= (unknowns * eps + eps_t) * np.sqrt(unknowns) * cond
