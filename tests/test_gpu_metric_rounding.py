"""The metric factors of the mixed-precision V-cycle are one rounding of their
FP64 value, whether they are stored per point or follow from an affine
element's constants: the V-cycle of an affine mesh is bitwise that of the same
mesh with one level-0 factor moved by less than it takes to change any FP32
value (which makes the level non-affine).
"""
import numpy as np
import pytest

import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh

pytestmark = pytest.mark.gpu


def gll(n):
    c = np.zeros(n)
    c[-1] = 1.0
    P = np.polynomial.legendre
    x = np.concatenate(([-1.0], P.legroots(P.legder(c)), [1.0])) if n > 2 else np.array([-1.0, 1.0])
    ln = P.legval(x, c)
    w = 2.0 / (n * (n - 1) * ln ** 2)
    D = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                D[i, j] = ln[i] / (ln[j] * (x[i] - x[j]))
    # exactly antisymmetric, so that the line form of the operator takes it
    D = 0.5 * (D - D[::-1, ::-1])
    return x, 0.5 * (w + w[::-1]), D - np.diag(D.sum(1))


def lagrange(xto, x):
    J = np.ones((len(xto), len(x)))
    for p in range(len(x)):
        for q in range(len(x)):
            if q != p:
                J[:, p] *= (xto - x[q]) / (x[p] - x[q])
    return J


# one thread-block cluster; separate launches
@pytest.mark.parametrize("shape, n", [((3, 3, 3), 6), ((3, 3, 3), 8), ((9, 9, 9), 5),
                                      ((7, 7, 7), 8)])
def test_mixed_v_cycle_rounds_each_factor_once(shape, n):
    m = box_mesh(shape)
    orders = [n]
    while orders[-1] > 2:
        orders.append((orders[-1] - 1) // 2 + 1)
    # G_ab det with det = 1: exact sums, so the constants are these numbers
    const = np.array([3.0, 0.5, -0.25, 2.5, 0.75, 3.5])
    x0, w0, _ = gll(n)
    rho = (w0[None, None, :] * w0[None, :, None]) * w0[:, None, None]
    z = []
    for moved in (False, True):
        ctx = S.Context(0)
        ctx.set_precision("mixed")
        ctx.setup_connectivity(m.neigh)
        for level, nl in enumerate(orders):
            x, w, D = gll(nl)
            geom = np.broadcast_to(const[:, None, None, None, None],
                                   (6, m.nel, nl, nl, nl)).copy()
            if moved and level == 0:
                v = geom[0, 2, 1, 1, 1] * (1.0 + 2e-10)
                assert np.float32(v * rho[1, 1, 1]) == np.float32(const[0] * rho[1, 1, 1])
                geom[0, 2, 1, 1, 1] = v
            interp = None if level == 0 else lagrange(xf, x).T
            ctx.setup_level(level, nl, np.ascontiguousarray(D.T), None, w, geom,
                            np.ones((m.nel, nl, nl, nl)),
                            None if interp is None else np.ascontiguousarray(interp))
            xf = x
        ctx.setup_finish()
        wt = ctx.level_data(0, 9)
        r = np.random.default_rng(n).standard_normal((m.nel, n, n, n))
        r = ctx.direct_stiffness_summation(r * wt)
        r -= (wt * r).sum() / wt.sum()
        z.append((ctx.multigrid_preconditioner(r), ctx.level_data(0, 7).astype(np.float32)))
        ctx.close()
    assert np.array_equal(z[0][1], z[1][1])   # the same FP32 Jacobi diagonal
    assert np.array_equal(z[0][0], z[1][0])
