"""BiCGStab's loop in a device graph: true residuals for both types, smoother degrees and
odd sizes, the loop's edges (zero right-hand side, iteration caps) and CG in between."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _system(n, precision):
    rng = np.random.default_rng(7)
    m = W.jitter_interior(P.box_mesh(n[0], n[1], n[2], *n), 1.0, 0.1, rng)
    M = P.Model(m, P.J2Material(**W.MAT))
    M.fix(P.on_face(m, "zmin"), "all")
    X = m.nodes
    U = np.stack([0.001 * X[0], 0.001 * X[1], -0.004 * X[2]]).T.reshape(-1)
    fixed = np.asarray(M.dir_dofs) - 1
    U[fixed] = 0.0
    K, _, _, _ = M.assemble(U, precision=precision)
    free = np.ones(M.ndof)
    free[fixed] = 0.0
    M.set_displacement(U)
    M.residual(1.0, precision=precision)
    return M, K, free, rng.standard_normal(M.ndof) * free


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,degree", [((3, 3, 2), 2), ((7, 6, 5), 2), ((7, 6, 5), 3), ((33, 32, 31), 2)])
def test_true_residual(n, degree, precision):
    M, K, free, b = _system(n, precision)
    rtol = 1e-8 if precision == "fp64" else 1e-4
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    for method in ("bicgstab", "cg", "bicgstab"):
        x, its = M.linear_solve(b, rtol=rtol, precision=precision, linsolve=method, cheb_degree=degree)
        assert its >= 1
        r = free * (K @ (x * free)) - b
        scale = np.linalg.norm(abs(K) @ abs(x * free))
        # the recursion's tolerance and the rounding of its updates, two an iteration
        assert np.linalg.norm(r) <= 1.01 * rtol * np.linalg.norm(b) + 2 * (its + 8) * eps * scale


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_loop_edges(precision):
    M, K, free, b = _system((7, 6, 5), precision)
    kw = dict(precision=precision, linsolve="bicgstab")
    x, its = M.linear_solve(0 * b, rtol=1e-4, **kw)
    assert its == 0 and not x.any()
    for cap in (0, 1):
        with pytest.raises(P.PfemError):
            M.linear_solve(b, rtol=1e-4, cg_itmax=cap, **kw)
    x, its = M.linear_solve(b, rtol=1e-4, **kw)
    again, its2 = M.linear_solve(b, rtol=1e-4, rebuild=False, **kw)
    assert its == its2 > 1 and np.array_equal(x, again)  # the sums have a fixed order
