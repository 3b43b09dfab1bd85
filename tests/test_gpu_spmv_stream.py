"""The level-0 product streamed through shared memory: linear solves on meshes around
its row limit, with a partial last tile, 16- and 32-bit column ids and both types,
checked against the assembled matrix."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,shuffle", [((19, 19, 19), False), ((20, 20, 20), False), ((27, 19, 16), False),
                                       ((33, 32, 31), False), ((33, 32, 31), True)])
def test_linear_solve_residual(n, shuffle, precision):
    rng = np.random.default_rng(5)
    m = W.jitter_interior(P.box_mesh(n[0], n[1], n[2], *n), 1.0, 0.1, rng)
    if shuffle:  # node numbers without order: column offsets leave 16 bits
        perm = rng.permutation(m.nnodes)
        nodes = np.empty_like(m.nodes)
        nodes[:, perm] = m.nodes
        m = P.Mesh(nodes, perm[m.elements - 1] + 1)
    M = P.Model(m, P.J2Material(**W.MAT))
    assert M.tangent_index_bytes() == (4 if shuffle else 2)
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
    rtol = 1e-8 if precision == "fp64" else 1e-4
    x, its = M.linear_solve(b, rtol=rtol, precision=precision)
    # true residual: the recursion's tolerance and the rounding of its updates
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    r = free * (K @ (x * free)) - b
    scale = np.linalg.norm(abs(K) @ abs(x * free))
    assert np.linalg.norm(r) <= 1.01 * rtol * np.linalg.norm(b) + (its + 8) * eps * scale
