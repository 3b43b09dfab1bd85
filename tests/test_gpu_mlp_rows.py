"""Row memory of the predictor's calls: kept between them, grown by a larger one, a
temporary of the call above its limit (64 MB, 92 bytes a row)."""
import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _model(p=None):
    w = W.config0(n=4, nsteps=4)
    M = P.Model(w.mesh, P.J2Material(**w.material))
    w.apply(M)
    if p is not None:
        M.mlp_params(p)
    return M


def test_sizes_in_turn_match_single_calls():
    rng = np.random.default_rng(2)
    p = rng.normal(0, 0.1, P.Model.NPARAMS).astype(np.float32)
    F = rng.normal(0, 1, (800_000, 12)).astype(np.float32)
    T = rng.normal(0, 1, (800_000, 3)).astype(np.float32)
    M, whole = _model(p), _model(p)
    y = whole.mlp_forward(F)
    for n in (1, 129, 70_000, 128, 729_000, 800_000, 5, 729_500):
        # a row's output depends on that row alone
        assert np.array_equal(M.mlp_forward(F[:n]), y[:n]), n
        loss, g = M.mlp_loss_grad(F[:n], T[:n])
        l1, g1 = _model(p).mlp_loss_grad(F[:n], T[:n])
        # single-precision sums over 148 blocks in the order in which they arrive
        eps = 2.0 ** -24
        assert abs(loss - l1) <= 2 * 148 * eps * abs(l1), n
        assert np.linalg.norm(g - g1) <= 2 * 148 * eps * np.linalg.norm(g1) * np.sqrt(len(g)), n
