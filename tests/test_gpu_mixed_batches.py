"""Shared-launch batches of a queue that mixes affine and deformed meshes: they
are batched apart, so a request's result does not depend on which kind it
queues with."""
import numpy as np
import pytest

import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh, periodic_box_fourier_rhs

pytestmark = pytest.mark.gpu

N = 6
BOXES = [(box_mesh((3, 3, 3)), (3, 3, 3), 4.0), (box_mesh((3, 4, 3)), (3, 4, 3), 30.0)]
DEFORMED = [(box_mesh((3, 3, 4), perturb=0.05, seed=3), (3, 3, 4), 11.0),
            (box_mesh((4, 3, 3), perturb=0.05, seed=4), (4, 3, 3), 2.5)]


def run(reqs, batching=True):
    """The requests queued behind one that holds the only slot, their meshes
    resident: the results and the batch statistics of the queue."""
    big = box_mesh((8, 8, 8))
    srv = S.Server(0, hbm_budget=20e9, max_active=1)
    try:
        if batching:
            srv.set_batching(8, 1 << 20)

        def submit(k):
            mesh, shape, lam = reqs[k]
            return srv.submit(mesh, N, periodic_box_fourier_rhs(shape, N, 40 + k), lam=lam,
                              precision="fp64")

        for k in range(len(reqs)):
            assert srv.wait(submit(k))[1] == "SSG_OK"
        hold = srv.submit(big, 8, periodic_box_fourier_rhs((8, 8, 8), 8, 1))
        out = [srv.wait(i) for i in [submit(k) for k in range(len(reqs))]]
        assert srv.wait(hold)[1] == "SSG_OK"
        assert all(o[1] == "SSG_OK" for o in out)
        return [o[0] for o in out], srv.stats()
    finally:
        srv.close()


def test_affine_and_deformed_meshes_batch_apart():
    alone, st = run(BOXES)
    assert st["batches"] == 1 and st["batched_requests"] == 2
    mixed, st = run(BOXES + DEFORMED)
    assert st["batches"] == 2 and st["batched_requests"] == 4
    for a, b in zip(alone, mixed):
        assert np.array_equal(a, b)
    solo, _ = run(BOXES + DEFORMED, batching=False)
    for a, b in zip(solo, mixed):
        assert np.abs(a - b).max() <= 1e-11 * np.abs(a).max()
