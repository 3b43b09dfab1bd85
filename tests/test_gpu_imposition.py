"""Boundary conditions imposed on the assembled tangent and residual, in one launch with
the norm in the next: sparse, dense and complete constraint sets, loads on constrained
dofs, new values and new loads on an old set, against the same steps in numpy."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(M, U, K, R0, lam, precision):
    rn, R = M.residual(lam, precision=precision)
    K = K.toarray()
    fn = np.zeros(M.ndof)
    np.add.at(fn, np.asarray(M.neu_dofs, np.int64) - 1, np.asarray(M.neu_vals, float))
    d = np.asarray(M.dir_dofs, np.int64) - 1
    dg = np.where(np.asarray(M.dir_ramp) != 0, lam, 1.0) * np.asarray(M.dir_vals) - U[d]
    ref = R0 - lam * fn + K[:, d] @ dg
    ref[d] = -dg
    scale = np.abs(R0) + np.abs(lam * fn) + np.abs(K[:, d]) @ np.abs(dg)
    scale[d] = np.abs(np.asarray(M.dir_vals)) + np.abs(U[d])
    # sums of up to 81 products and two more terms, in double in either precision
    assert np.all(np.abs(R - ref) <= 84 * 2.0 ** -53 * scale)
    assert abs(rn - np.linalg.norm(R)) <= M.ndof * 2.0 ** -53 * np.linalg.norm(R)
    try:
        M.linear_solve(R, rtol=0.9, precision=precision)
    except P.PfemError:
        pass  # only the level-0 operator that it leaves is looked at
    A = M.amg_dense(0, 0)
    K[d, :] = 0.0
    K[:, d] = 0.0
    K[d, d] = 1.0
    assert np.array_equal(A, K)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
def test_imposition(share, precision):
    rng = np.random.default_rng(int(100 * share))
    m = W.jitter_interior(P.box_mesh(6, 5, 4, 6, 5, 4), 1.0, 0.1, rng)
    M = P.Model(m, P.J2Material(**W.MAT))
    U = 1e-3 * rng.standard_normal(M.ndof)
    d = 1 + rng.permutation(M.ndof)[:max(2, int(share * M.ndof))]
    M.dir_dofs, M.dir_vals = d, 1e-3 * rng.standard_normal(len(d))
    M.dir_ramp = rng.integers(0, 2, len(d)).astype(np.uint8)
    M.load(1 + rng.permutation(m.nnodes)[:40], "all", 3.0)  # some of them on constrained dofs
    K, R0, _, _ = M.assemble(U, precision=precision)
    M.set_displacement(U)
    _check(M, U, K, R0, 0.7, precision)
    M.dir_vals = 1e-3 * rng.standard_normal(len(d))  # the same set, new values
    _check(M, U, K, R0, 0.4, precision)
    M.load(1 + rng.permutation(m.nnodes)[:10], "x", -2.0)  # new loads
    _check(M, U, K, R0, 1.0, precision)
    keep = rng.permutation(len(d))[:len(d) // 2 + 1]  # another set under the old loads
    r, v = M.dir_ramp, M.dir_vals
    M.dir_dofs, M.dir_vals, M.dir_ramp = d[keep], v[keep], r[keep]
    _check(M, U, K, R0, 0.2, precision)
