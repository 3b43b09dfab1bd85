"""Products that only some meshes reach, by linear solves checked against the assembled
matrix: the streamed 6 x 6 product in both types (4,096 aggregates or more), and a mesh
with rows of more than 32 blocks and so many rows that a product inside a CG iteration has
more CTAs than places for partial sums."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

from test_gpu_gather import star

pytestmark = pytest.mark.gpu


def check(m, element, precision, rtol):
    rng = np.random.default_rng(5)
    M = P.Model(m, P.J2Material(**W.MAT), element=element)
    M.fix(P.on_face(m, "zmin"), "all")
    X = m.nodes
    U = np.stack([0.001 * X[0], 0.001 * X[1], -0.004 * X[2]]).T.reshape(-1)
    fixed = np.asarray(M.dir_dofs) - 1
    U[fixed] = 0.0
    K, _, _, _ = M.assemble(U, precision=precision)
    free = np.ones(M.ndof)
    free[fixed] = 0.0
    b = rng.standard_normal(M.ndof) * free
    M.set_displacement(U)
    M.residual(1.0, precision=precision)
    x, its = M.linear_solve(b, rtol=rtol, precision=precision, cg_itmax=400)
    # true residual: the recursion's tolerance and the rounding of its updates
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    r = free * (K @ (x * free)) - b
    assert np.linalg.norm(r) <= 1.01 * rtol * np.linalg.norm(b) + (its + 8) * eps * np.linalg.norm(abs(K) @ abs(x * free))
    return M, free, eps, rng


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_coarse_product_streamed(precision):
    n = (47, 49, 50)  # 16 x 17 x 17 = 4,624 aggregates of 48 x 50 x 51 nodes
    m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, np.random.default_rng(1))
    M, free, eps, rng = check(m, "small", precision, 1e-8 if precision == "fp64" else 1e-4)
    # the cycle is symmetric to rounding: a lost or doubled block of a coarse product is not
    y, z = rng.standard_normal((2, M.ndof)) * free
    My, Mz = M.amg_apply(y), M.amg_apply(z)
    assert abs(z @ My - y @ Mz) <= 1e4 * eps * np.linalg.norm(y) * np.linalg.norm(Mz)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_long_rows(precision):
    # a box of 41 x 41 x 21 nodes and, apart from it, a star whose axis has rows of 33 blocks
    box, s = P.box_mesh(40.0, 40.0, 20.0, 40, 40, 20), star(5, 3)
    m = P.Mesh(np.concatenate([box.nodes, s.nodes + [[60.0], [0.0], [0.0]]], 1),
               np.concatenate([box.elements, s.elements + box.nnodes], 1))
    check(m, "small", precision, 1e-8 if precision == "fp64" else 1e-4)
