"""Small levels solved inside one thread-block cluster, against the oracle, at
the sizes where the split over the blocks can go wrong: one block and
sixteen, blocks with a remainder of elements or none, every order, walls,
the per-point and the constant metric, and the first size past the
cluster's limit.

Helmholtz solves stop where the oracle's do, with a residual under the oracle's
own operator of the solves' eps (and the two operators' difference on the
solution: the rounding noise of the metric, at most 4e-14 n^2); one V-cycle
agrees to 1e-9 in FP64, as the other solver tests state.
"""
import numpy as np
import pytest

import oracle as O
from conftest import same_stop
from ssenss_b200.mesh import box_mesh, channel_mesh

pytestmark = pytest.mark.gpu

CASES = [("box", (3, 3, 3), 3), ("box", (3, 3, 3), 4), ("box", (7, 5, 6), 5),
         ("box", (5, 5, 6), 6), ("box", (3, 4, 5), 7), ("box", (4, 4, 4), 8),
         ("box", (3, 3, 4), 9), ("box", (3, 3, 5), 10), ("box", (3, 3, 3), 11),
         ("box", (3, 3, 3), 12), ("channel", (4, 3, 3), 8), ("channel", (5, 3, 4), 6),
         ("channel", (8, 6, 6), 4), ("box", (11, 12, 13), 3), ("box", (9, 9, 9), 5)]


@pytest.mark.parametrize("kind, shape, n", CASES)
def test_small_levels_against_the_oracle(kind, shape, n, gpu_ctx_factory):
    m = box_mesh(shape) if kind == "box" else channel_mesh(shape, seed=7)
    lam = 50.0
    visc = 1.0
    dt = (11.0 / 6.0) / lam
    orc = O.Oracle(m, n)
    orc.set_params(0.0, dt, visc)
    ctx = gpu_ctx_factory(m, n, dt=dt, visc=visc)
    X, Y, Z = (orc.geometry(0, 7 + a) for a in range(3))
    g = np.cos(X + 0.3) * np.cos(2 * Y + 0.7) * np.cos(Z + 1.1) + 0.2 * np.cos(2 * Z + 0.4)
    f = orc.dss(ctx.level_data(0, 6) * g)
    _, h_o = orc.solve_helmholtz(O.X_VELOCITY, f.copy(), np.zeros_like(f))
    u_g, info = ctx.solve_helmholtz_cg(O.X_VELOCITY, f.copy(), np.zeros_like(f))
    assert info["status"] == "SSG_OK"
    w = ctx.level_data(0, 9)
    # the solution's residual under the oracle's own (masked) operator: the
    # solve's eps and the two operators' difference on the solution
    mask = ctx.level_data(0, 10)
    res = mask * f - orc.global_opeval(O.X_VELOCITY, u_g)
    assert np.sqrt((w * res * res).sum()) < 1.5e-10 + 4e-14 * n * n * np.sqrt((w * f * f).sum())
    same_stop(info["iterations"], info["history"], h_o)
    r = f - (w * f).sum() / w.sum()
    z = ctx.multigrid_preconditioner(r)
    ref = orc.mg_precon(r)
    assert np.abs(z - ref).max() <= 1e-9 * np.abs(ref).max()
    # graphs replay the same launches
    ctx.set_graphs(False)
    again = ctx.solve_helmholtz_cg(O.X_VELOCITY, f.copy(), np.zeros_like(f))[0]
    assert np.array_equal(again, u_g)
    ctx.close()
    orc.close()
