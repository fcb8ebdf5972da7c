"""A caller's derivative matrix that is off the GLL points' antisymmetry by more
than the rounding of the points is taken as it is, by the operator and by
convection: their results are the definition's (1e-13)."""
import numpy as np
import pytest

import oracle as O
import ssenss_b200 as S
from ssenss_b200.mesh import box_mesh
from test_gpu_affine import conv_reference, rel
from test_gpu_metric_rounding import gll, lagrange

pytestmark = pytest.mark.gpu

AX = ("pi,ekji->ekjp", "pj,ekji->ekpi", "pk,ekji->epji")


def nearly(D, rng):
    """D with every entry moved by up to 4.5e-13 of the largest."""
    return D + 4.5e-13 * np.abs(D).max() * rng.uniform(-1.0, 1.0, D.shape)


@pytest.mark.parametrize("n", [5, 6, 9])
def test_nearly_antisymmetric_derivative(n):
    m = box_mesh((3, 3, 3))
    rng = np.random.default_rng(n)
    ctx = S.Context(0)
    ctx.setup_connectivity(m.neigh)
    orders = [n]
    while orders[-1] > 2:
        orders.append((orders[-1] - 1) // 2 + 1)
    xf = None
    for level, nl in enumerate(orders):
        x, w, D = gll(nl)
        D = nearly(D, rng)
        geom = rng.uniform(0.5, 1.5, (6, m.nel, nl, nl, nl))
        det = rng.uniform(0.5, 1.5, (m.nel, nl, nl, nl))
        interp = None if level == 0 else np.ascontiguousarray(lagrange(xf, x).T)
        ctx.setup_level(level, nl, np.ascontiguousarray(D.T), None, w, geom, det, interp)
        if level == 0:
            x0, D0, w0, g0, d0 = x, D, w, geom, det
        xf = x
    md = (3 * n) // 2
    xm, wm, Dm = gll(md)
    Dm = nearly(Dm, rng)
    J = lagrange(xm, x0)
    detm = rng.uniform(0.5, 1.5, (m.nel, md, md, md))
    tinv = rng.standard_normal((9, m.nel, md, md, md))
    ctx.setup_dealias(md, np.ascontiguousarray(Dm.T), wm, tinv, detm, np.ascontiguousarray(J.T))
    ctx.setup_finish()
    u = rng.standard_normal((m.nel, n, n, n))
    du = [np.einsum(AX[b], D0, u) for b in range(3)]
    rho = (w0[:, None, None] * w0[:, None] * w0) * d0
    sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
    ref = sum(np.einsum(AX[a], D0.T, sum(g0[sym[a][b]] * du[b] for b in range(3)) * rho)
              for a in range(3))
    assert rel(ctx.local_opeval(O.PRESSURE, u), ref) < 1e-13
    a, b = (rng.standard_normal((3, m.nel, n, n, n)) for _ in range(2))
    assert rel(ctx.convection_operator(a, b), conv_reference(a, b, J, Dm, wm, detm, tinv)) < 1e-13
    ctx.close()
