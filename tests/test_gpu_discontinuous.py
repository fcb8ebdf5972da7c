"""FP64 solves and smoothers whose search direction differs between the element
copies of a node: a right-hand side that was not summed over the elements, and
walls that meet an element in an edge alone (its copies of that edge are not
masked).  The reference's alpha, (p w).ap with the assembled ap, is defined for
both.  A few iterations against the oracle: the residual norms to 1e-10 of the
first and the iterate to 1e-9 of its largest entry, some 1e4 times the
rounding of six iterations.
"""
import dataclasses

import numpy as np
import pytest

import oracle as O
import ssenss_b200 as S
from ssenss_b200.mesh import ALL_DIRS, box_mesh

pytestmark = pytest.mark.gpu

# in one thread-block cluster; as separate launches (line-run DSS); odd order;
# the tensor-core operator
SIZES = [((3, 3, 3), 6), ((9, 9, 9), 5), ((3, 3, 4), 7), ((7, 7, 7), 8)]


def without_column(m):
    """The box without its elements (0, 0, .): a re-entrant edge, which the
    elements (1, 1, .) touch in an edge alone."""
    nx, ny, nz = m.shape
    e = np.arange(m.nel)
    keep = (e % nx > 0) | ((e // nx) % ny > 0)
    new = np.where(keep, np.cumsum(keep) - 1, -1)
    nb = m.neigh[keep]
    nb = np.where(nb >= 0, new[np.maximum(nb, 0)], nb).astype(np.int32)
    return dataclasses.replace(m, vertices=m.vertices[keep], neigh=nb)


def edge_left_out(m):
    """Periodic box whose elements (0, 0, .) and (1, 1, .) do not name each other
    across the edge they share, as a table with one slot an edge has it where
    more than four elements meet: summing leaves the copies of that edge's
    nodes different."""
    nx, ny, _ = m.shape
    nb = m.neigh.copy()
    e = np.arange(m.nel)
    for at, d in ((0, (1, 1, 0)), (1, (-1, -1, 0))):
        nb[(e % nx == at) & ((e // nx) % ny == at), ALL_DIRS.index(d)] = -1
    return dataclasses.replace(m, neigh=nb)


def compare(ctx, orc, var, f, iters=6, plain=False):
    z = np.zeros_like(f)
    if var == O.PRESSURE and not plain:
        u_o, h_o = orc.mg_precon(f), None
        u_g = ctx.multigrid_preconditioner(f)
    else:
        u_o, h_o = orc.solve_helmholtz(var, f.copy(), z.copy(), eps=0.0, max_iter=iters)
        u_g, info = ctx.conjugate_gradient(var, f, z.copy(), eps=0.0, max_iter=iters)
        assert info["iterations"] == iters and len(h_o) == iters
        assert np.all(np.abs(info["history"] - h_o) <= 1e-10 * h_o[0])
    assert np.abs(u_g - u_o).max() <= 1e-9 * np.abs(u_o).max()


@pytest.mark.parametrize("shape, n", SIZES)
def test_right_hand_side_that_differs_between_copies(shape, n, gpu_ctx_factory):
    m = box_mesh(shape)
    lam = 50.0
    orc = O.Oracle(m, n)
    orc.set_params(0.0, (11.0 / 6.0) / lam, 1.0)
    ctx = gpu_ctx_factory(m, n, dt=(11.0 / 6.0) / lam, visc=1.0)
    f = ctx.level_data(0, 6) * np.random.default_rng(n).standard_normal((m.nel, n, n, n))
    compare(ctx, orc, O.X_VELOCITY, f)
    compare(ctx, orc, O.PRESSURE, f)
    ctx.close()
    orc.close()


@pytest.mark.parametrize("shape, n", SIZES)
def test_walls_that_meet_an_element_in_an_edge(shape, n, gpu_ctx_factory):
    m = without_column(box_mesh(shape, periodic=(False, False, True)))
    lam = 50.0
    orc = O.Oracle(m, n)
    orc.set_params(0.0, (11.0 / 6.0) / lam, 1.0)
    ctx = gpu_ctx_factory(m, n, dt=(11.0 / 6.0) / lam, visc=1.0)
    assert np.abs(orc.dss(ctx.level_data(0, 10)) - orc.dss(np.ones((m.nel, n, n, n))) *
                  ctx.level_data(0, 10)).max() > 0.5     # the mask differs between copies
    f = orc.dss(ctx.level_data(0, 6) * np.random.default_rng(n).standard_normal((m.nel, n, n, n)))
    compare(ctx, orc, O.X_VELOCITY, f)
    ctx.close()
    orc.close()


@pytest.mark.parametrize("shape, n", SIZES)
def test_tables_that_leave_an_element_out(shape, n, gpu_ctx_factory):
    """Also with a right-hand side that is zero on every face, so equal in all
    copies: the first A p is not.  Helmholtz and the plain CG of the pressure
    operator."""
    m = edge_left_out(box_mesh(shape))
    lam = 50.0
    orc = O.Oracle(m, n)
    orc.set_params(0.0, (11.0 / 6.0) / lam, 1.0)
    ctx = gpu_ctx_factory(m, n, dt=(11.0 / 6.0) / lam, visc=1.0)
    r = ctx.level_data(0, 6) * np.random.default_rng(n).standard_normal((m.nel, n, n, n))
    inside = np.zeros_like(r)
    inside[:, 1:-1, 1:-1, 1:-1] = r[:, 1:-1, 1:-1, 1:-1]
    for f in (orc.dss(r), inside):
        compare(ctx, orc, O.X_VELOCITY, f)
        compare(ctx, orc, O.PRESSURE, f, plain=True)
    ctx.close()
    orc.close()


@pytest.mark.parametrize("shape, n", [((9, 9, 9), 5), ((7, 7, 7), 8)])
def test_forms_alternate_on_one_context(shape, n, gpu_ctx_factory):
    """Solves that may gather and update at once (a right-hand side equal in all
    copies) and solves that may not, in turn through the same buffers and
    graphs: three iterations each against the oracle, and every repeat bitwise
    the first of its kind."""
    m = box_mesh(shape)
    lam = 50.0
    orc = O.Oracle(m, n)
    orc.set_params(0.0, (11.0 / 6.0) / lam, 1.0)
    ctx = gpu_ctx_factory(m, n, dt=(11.0 / 6.0) / lam, visc=1.0)
    rough = ctx.level_data(0, 6) * np.random.default_rng(n).standard_normal((m.nel, n, n, n))
    w = ctx.level_data(0, 9)
    fs = []
    for f in (orc.dss(rough), rough):
        f = f - (w * f).sum() / w.sum()
        fs.append(f)
    z = np.zeros_like(rough)
    ref = [[orc.solve_helmholtz(O.X_VELOCITY, f.copy(), z.copy(), eps=1e-300, max_iter=3),
            orc.solve_poisson(f.copy(), z.copy(), eps=1e-10, max_iter=3)] for f in fs]
    first = {}
    for k in (0, 1, 0, 0, 1, 1, 0, 1):
        got = [ctx.solve_helmholtz_cg(O.X_VELOCITY, fs[k], z.copy(), eps=1e-300, max_iter=3),
               ctx.solve_poisson_cg(fs[k], z.copy(), eps=1e-10, max_iter=3)]
        for s in range(2):
            u, info = got[s]
            u_o, h_o = ref[k][s]
            assert np.all(np.abs(info["history"] - h_o) <= 1e-9 * h_o[0])
            assert np.abs(u - u_o).max() <= 1e-8 * np.abs(u_o).max()
            assert np.array_equal(first.setdefault((k, s), u.copy()), u)
    ctx.close()
    orc.close()
