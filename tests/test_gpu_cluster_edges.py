"""Cases at the edge of the one-launch solves: the iteration cap reached inside
the launch, a right-hand side of zero (0 / 0, as in the reference: not a
number), and meshes whose neighbours meet turned or on the same side."""
import dataclasses

import numpy as np
import pytest

import oracle as O
import ssenss_b200 as S
from ssenss_b200.mesh import ALL_DIRS, box_mesh, channel_mesh

pytestmark = pytest.mark.gpu

LAM = 50.0


def pair(m, n, gpu_ctx_factory):
    orc = O.Oracle(m, n)
    orc.set_params(0.0, (11.0 / 6.0) / LAM, 1.0)
    return orc, gpu_ctx_factory(m, n, dt=(11.0 / 6.0) / LAM, visc=1.0)


def turned(m):
    """The box with element 0's own axes turned: its r runs along y, its s along
    -x, so its faces, edges and corners meet their neighbours' on other sides."""
    v = m.vertices.copy()
    nb = m.neigh.copy()
    for c in range(8):
        a, b, k = c & 1, (c >> 1) & 1, c >> 2   # new r, s, t side
        v[0, :, c] = m.vertices[0, :, (1 - b) + 2 * a + 4 * k]
    for s, (dr, ds, dt) in enumerate(ALL_DIRS):   # new local direction -> old
        nb[0, s] = m.neigh[0, ALL_DIRS.index((-ds, dr, dt))]
    return dataclasses.replace(m, vertices=v, neigh=nb)


@pytest.mark.parametrize("cap", [1, 2, 7])
def test_cap_inside_the_launch(cap, gpu_ctx_factory):
    m, n = box_mesh((3, 3, 4)), 7
    orc, ctx = pair(m, n, gpu_ctx_factory)
    f = orc.dss(ctx.level_data(0, 6) * np.random.default_rng(1).standard_normal((m.nel, n, n, n)))
    u_o, h_o = orc.solve_helmholtz(O.X_VELOCITY, f.copy(), np.zeros_like(f), max_iter=cap)
    u, info = ctx.solve_helmholtz_cg(O.X_VELOCITY, f, np.zeros_like(f), max_iter=cap)
    assert info["status"] == "SSG_MAXITER" and info["iterations"] == cap == len(h_o)
    assert np.all(np.abs(info["history"] - h_o) <= 1e-10 * h_o[0])
    assert np.abs(u - u_o).max() <= 1e-9 * np.abs(u_o).max()
    ctx.close()
    orc.close()


@pytest.mark.parametrize("shape, n", [((3, 3, 3), 6), ((9, 9, 9), 5)])
def test_zero_right_hand_side(shape, n, gpu_ctx_factory):
    """In one launch and in separate ones: the same status, after one iteration;
    the context solves again afterwards."""
    m = box_mesh(shape)
    orc, ctx = pair(m, n, gpu_ctx_factory)
    z = np.zeros((m.nel, n, n, n))
    with pytest.raises(S.SsgError) as e:
        ctx.solve_helmholtz_cg(O.X_VELOCITY, z, z.copy())
    assert "NONFINITE" in str(e.value) or "non-finite" in str(e.value)
    f = orc.dss(ctx.level_data(0, 6) * np.random.default_rng(1).standard_normal(z.shape))
    assert ctx.solve_helmholtz_cg(O.X_VELOCITY, f, z.copy())[1]["status"] == "SSG_OK"
    ctx.close()
    orc.close()


@pytest.mark.parametrize("name, n", [("turned", 4), ("turned", 6), ("turned", 8), ("same_side", 5),
                                     ("same_side", 6)])
def test_other_pairings(name, n, gpu_ctx_factory):
    """Element 0 turned a quarter, and boxes of two elements along a direction,
    whose faces the reference pairs on the same side: six Helmholtz iterations
    and the smoothed DSS against the oracle."""
    m = turned(channel_mesh((4, 4, 3), seed=7)) if name == "turned" else box_mesh((2, 3, 3))
    orc, ctx = pair(m, n, gpu_ctx_factory)
    r = np.random.default_rng(n).standard_normal((m.nel, n, n, n))
    assert np.array_equal(ctx.direct_stiffness_summation(r.copy()), orc.dss(r))
    f = orc.dss(ctx.level_data(0, 6) * r)
    u_o, h_o = orc.solve_helmholtz(O.X_VELOCITY, f.copy(), np.zeros_like(f), eps=0.0, max_iter=6)
    u, info = ctx.solve_helmholtz_cg(O.X_VELOCITY, f, np.zeros_like(f), eps=0.0, max_iter=6)
    assert np.all(np.abs(info["history"] - h_o) <= 1e-10 * h_o[0])
    assert np.abs(u - u_o).max() <= 1e-9 * np.abs(u_o).max()
    ctx.close()
    orc.close()
