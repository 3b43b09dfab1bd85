"""Cases of the mixed-precision path whose values are kept in single_precision.npz.

Their sums are rounded to 32 bits at every term, so another order of the same terms is
another value; a slender box clamped at one end multiplies that by hundreds in its
solution.  The kept values are those of the library at revision b8b1c70:
    python tests/golden/make_single_precision.py LIBRARY OUT.npz
"""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import plasticity_b200 as P  # noqa: E402
from plasticity_b200 import workloads as W  # noqa: E402

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "single_precision.npz")
HARD = {"linear": dict(Hiso=2000.0), "voce": dict(Hiso=130.0, sigsat=350.0, delta=17.0),
        "kin": dict(Hiso=500.0, Hkin=500.0)}

# element, hardening, field: with noise, or with two equal stretches at every point, whose
# eigenvectors are left to the rounding
TANGENTS = [("finite_fbar", "linear", "noise"), ("finite_fbar", "linear", "equal"), ("finite_fbar", "kin", "noise"),
            ("finite", "voce", "noise")]

# box, element, hardening, pulled along, method, every how many entries are kept: around
# the row limits of the streamed products (8192 block rows, 4096 of 6 x 6) and transfers, and
# with more coarse blocks (157,300 in the last) than eight lanes each are given
SOLVES = [((13, 7, 7), "finite_fbar", "linear", 0, "cg", 1), ((20, 8, 8), "small", "linear", 0, "cg", 3),
          ((30, 8, 6), "finite", "linear", 0, "cg", 3), ((35, 25, 40), "finite_fbar", "linear", 2, "cg", 19),
          ((41, 21, 30), "finite", "voce", 0, "cg", 19), ((50, 50, 50), "finite_fbar", "linear", 0, "cg", 97),
          ((14, 10, 9), "finite_fbar", "linear", 0, "bicgstab", 1), ((27, 20, 25), "small", "linear", 0, "bicgstab", 19),
          ((56, 54, 52), "finite", "linear", 2, "cg", 97)]


def model(n, element, hard, axis, seed=3):
    rng = np.random.default_rng(seed)
    h = 1.0 / n[2]
    m = W.jitter_interior(P.box_mesh(n[0] * h, n[1] * h, n[2] * h, *n), h, 0.1, rng)
    M = P.Model(m, P.J2Material(E=200e3, nu=0.3, sigy0=250.0, **HARD[hard]), element=element,
                sigy0_e=W.lognormal_sigy(m.nelem, 250.0, 0.05, rng))
    M.fix(P.on_face(m, "xyz"[axis] + "min"), "all")
    M.prescribe(P.on_face(m, "xyz"[axis] + "max"), "xyz"[axis], 0.008 * n[axis] * h)
    X = m.nodes
    U = np.stack([(0.008 if d == axis else -0.0036) * X[d] for d in range(3)]).T.reshape(-1)
    return M, U + 0.0008 * h * rng.standard_normal(U.shape)


def tangent(element, hard, field):
    rng = np.random.default_rng(7)
    m = W.jitter_interior(P.box_mesh(1.0, 1.0, 1.0, 3, 3, 3), 1.0 / 3.0, 0.1, rng)
    M = P.Model(m, P.J2Material(E=200e3, nu=0.3, sigy0=250.0, **HARD[hard]), element=element)
    X = m.nodes
    U = np.stack([0.008 * X[0], -0.0024 * X[1], -0.0024 * X[2]])
    if field == "noise":
        U = U + np.stack([0.004 * X[1], -0.002 * X[2], 0 * X[0]]) + 3e-4 * rng.standard_normal(X.shape)
    U = np.ascontiguousarray(U.T.reshape(-1))
    M.assemble(0.6 * U, commit=True)
    return M.assemble(U, precision="mixed")[0].data.astype(np.float32)


def hierarchy():
    """The prolongator of the tangent and its Galerkin operator."""
    M, U = model((8, 5, 3), "small", "linear", 0)
    M.set_displacement(U)
    _, R = M.residual(1.0, precision="mixed")
    M.linear_solve(-R, rtol=0.5, precision="mixed")
    return M.amg_dense(0, 1).astype(np.float32), M.amg_dense(1, 0).astype(np.float32)


def solution(n, element, hard, axis, method, every):
    M, U = model(n, element, hard, axis)
    M.assemble(0.6 * U, commit=True, want_K=False)
    M.set_displacement(U)
    _, R = M.residual(1.0, precision="mixed")
    x, _ = M.linear_solve(-R, rtol=1e-3, precision="mixed", linsolve=method, cg_itmax=400)
    return x.astype(np.float32)[::every]


if __name__ == "__main__":
    from plasticity_b200 import _lib
    _lib.LIB_PATH = os.path.abspath(sys.argv[1])
    out = {"tangent_%d" % i: tangent(*c) for i, c in enumerate(TANGENTS)}
    out["prolongator"], out["galerkin"] = hierarchy()
    out.update({"solution_%d" % i: solution(*c) for i, c in enumerate(SOLVES)})
    np.savez_compressed(sys.argv[2], **out)
