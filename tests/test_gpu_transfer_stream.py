"""Prolongation and restriction of the finest level streamed through shared memory:
solves and cycles on either side of their limits (32-node tiles with a remainder, ids
off a 16-byte boundary, both types)."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 8,000 and 8,820 nodes: either side of the prolongation's limit; 69,741 nodes: the FP64
# level (127 MB of matrix) is over the restriction's, the FP32 one under it; 274,625: both over
@pytest.mark.parametrize("n,precision", [((19, 19, 19), "mixed"), ((20, 20, 19), "fp64"), ((20, 20, 19), "mixed"),
                                         ((42, 40, 38), "fp64"), ((42, 40, 38), "mixed"), ((64, 64, 64), "mixed")])
def test_linear_solve_residual(n, precision):
    rng = np.random.default_rng(11)
    m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, rng)
    M = P.Model(m, P.J2Material(**W.MAT), element="small")  # its tangent is symmetric, F-bar's is not
    M.fix(P.on_face(m, "zmin"), "all")
    fixed = np.asarray(M.dir_dofs) - 1
    K, _, _, _ = M.assemble(np.zeros(M.ndof), precision=precision)
    free = np.ones(M.ndof)
    free[fixed] = 0.0
    M.residual(1.0, precision=precision)
    b = rng.standard_normal(M.ndof) * free
    rtol = 1e-8 if precision == "fp64" else 1e-4
    x, its = M.linear_solve(b, rtol=rtol, precision=precision)
    # a wrong transfer is a wrong coarse correction: the smoother alone needs hundreds of
    # iterations for this load, the cycle tens
    assert its <= 60
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    r = free * (K @ (x * free)) - b
    scale = np.linalg.norm(abs(K) @ abs(x * free))
    assert np.linalg.norm(r) <= 1.01 * rtol * np.linalg.norm(b) + (its + 8) * eps * scale
    # the cycle is symmetric when its restriction is the transpose of its prolongation
    u, w = (rng.standard_normal(M.ndof) * free for _ in range(2))
    Mu, Mw = M.amg_apply(u), M.amg_apply(w)
    uMw, wMu = u @ Mw, w @ Mu
    bound = np.linalg.norm(u) * np.linalg.norm(Mw) + np.linalg.norm(w) * np.linalg.norm(Mu)
    # rounding of about forty dependent steps over rows of up to 81 entries
    assert abs(uMw - wMu) <= 40 * 81 * eps * bound
