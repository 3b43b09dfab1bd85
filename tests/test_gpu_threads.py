"""Contexts of different sizes set up and solved at the same time, each by its own host
thread: a kernel's limits are the process's, so no launch may set them for its own size."""
import threading

import numpy as np
import pytest

import plasticity_b200 as P
from plasticity_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_set_ups_at_once():
    # coarsest levels of 180 and 6 unknowns: 66 KB and 96 bytes of one kernel's shared memory
    def start(n):
        m = W.jitter_interior(P.box_mesh(*n, *n), 1.0, 0.1, np.random.default_rng(1))
        M = P.Model(m, P.J2Material(**W.MAT))
        M.fix(P.on_face(m, "zmin"))
        M.prescribe(P.on_face(m, "zmax"), "z", -0.005 * n[2])
        _, R = M.residual(0.1)
        x, _ = M.linear_solve(-R, rtol=0.1)
        return M, R, x

    states = [start(n) for n in ((14, 8, 5), (2, 2, 2), (14, 8, 5), (2, 2, 2))]
    faults = []

    def work(M, R, x):
        try:
            for _ in range(1500):
                y, _ = M.linear_solve(-R, rtol=0.1)
                if not np.array_equal(x, y):
                    faults.append("another solution")
                    return
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            faults.append(repr(e))

    threads = [threading.Thread(target=work, args=s) for s in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults
