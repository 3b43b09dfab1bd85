"""The row gather against the colored in-place assembly: boxes down to one element, node
orders without structure, and a mesh whose axis nodes are in ten elements (rows of 33
blocks, which the streamed gather leaves to the general one)."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def star(sectors, layers):
    """Prisms of quadrilaterals (centre, rim, outer, next rim) around the z axis."""
    t = 2 * np.pi * np.arange(sectors) / sectors
    half = t + np.pi / sectors
    ring = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], 1), 1.4 * np.stack([np.cos(half), np.sin(half)], 1)])
    n = len(ring)
    nodes = np.concatenate([np.concatenate([ring, np.full((n, 1), 0.5 * k)], 1) for k in range(layers + 1)])
    quad = np.stack([[0, 1 + i, 1 + sectors + i, 1 + (i + 1) % sectors] for i in range(sectors)])
    els = np.concatenate([np.concatenate([quad + k * n, quad + (k + 1) * n], 1) for k in range(layers)]) + 1
    return P.Mesh(np.ascontiguousarray(nodes.T), np.ascontiguousarray(els.T.astype(np.int64)))


def shuffled(m, rng):
    perm = rng.permutation(m.nnodes)
    nodes = np.empty_like(m.nodes)
    nodes[:, perm] = m.nodes
    return P.Mesh(nodes, perm[m.elements - 1] + 1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh", ["1x1x1", "2x1x1", "5x3x2", "17x16x15", "shuffled", "star"])
def test_gather_matches_colored(mesh, precision, monkeypatch):
    rng = np.random.default_rng(2)
    if mesh == "star":
        m = star(5, 3)
    elif mesh == "shuffled":
        m = shuffled(W.jitter_interior(P.box_mesh(6, 5, 4, 6, 5, 4), 1.0, 0.1, rng), rng)
    else:
        n = [int(k) for k in mesh.split("x")]
        m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, rng)
    X = m.nodes
    U = np.stack([0.003 * X[0], 0.001 * X[1], -0.008 * X[2]]).T.reshape(-1) + 1e-4 * rng.standard_normal(3 * m.nnodes)
    out = []
    for mode in ("gathered", "colored"):
        monkeypatch.setenv("PFEM_ASSEMBLY", mode)
        M = P.Model(m, P.J2Material(**W.MAT))
        for _ in range(2):  # the second assembly writes over the first
            K, R, tau, fl = M.assemble(U, precision=precision)
        out.append((K, R, tau, fl))
    (K, R, tau, fl), (Kc, Rc, tauc, flc) = out
    # at most ten terms per entry, in another order
    eps = 2.0 ** (-53 if precision == "fp64" else -24)
    assert abs(K - Kc).max() <= 10 * eps * abs(Kc).max()
    assert np.abs(R - Rc).max() <= 10 * 2.0 ** -53 * np.abs(Rc).max() * 8
    assert np.array_equal(tau, tauc) and np.array_equal(fl, flc)
