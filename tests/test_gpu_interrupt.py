"""Cancellation and deadlines of running requests whose solve is one launch (a
Helmholtz level that fits a thread-block cluster)."""
import numpy as np
import pytest

import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh, periodic_box_fourier_rhs

pytestmark = pytest.mark.gpu

SHAPE, N, LAM = (4, 4, 4), 8, 12.5


@pytest.mark.parametrize("how, status", [("deadline", "SSG_ERR_TIMEOUT"),
                                         ("cancel", "SSG_ERR_CANCELLED")])
def test_running_helmholtz_request_is_interrupted(how, status):
    """A deadline that passes, or a cancel that arrives, during the mesh set-up
    (many milliseconds) or the solve ends the request with its status; the
    next request on the mesh is not affected."""
    mesh = box_mesh(SHAPE)
    f = periodic_box_fourier_rhs(SHAPE, N, 5)
    warm = box_mesh((3, 3, 3))
    srv = S.Server(0, hbm_budget=20e9, max_active=1)
    try:
        # the worker is up and idle, so that the next request starts at once
        g = periodic_box_fourier_rhs((3, 3, 3), N, 5)
        assert srv.wait(srv.submit(warm, N, g, lam=LAM, precision="fp64"))[1] == "SSG_OK"
        rid = srv.submit(mesh, N, f, lam=LAM, precision="fp64",
                         deadline_ms=2.0 if how == "deadline" else 0.0)
        while srv.stats()["mesh_misses"] < 2:   # admitted
            pass
        if how == "cancel":
            srv.cancel(rid)
        assert srv.wait(rid)[1] == status
        u, st, info = srv.wait(srv.submit(mesh, N, f, lam=LAM, precision="fp64"))
        assert st == "SSG_OK" and info["residual"] <= 1e-10
        assert srv.stats()["mesh_hits"] == 1    # the interrupted request's context serves it
    finally:
        srv.close()
