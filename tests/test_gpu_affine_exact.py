"""The operator and convection on affine elements against the exact constant
metric (the parallelepipeds' edges in closed form) instead of the oracle's
factors, which carry the rounding of differentiated coordinates: 1e-13 for the
operator as on any mesh, whose constants (means of the factors) are within
2.1e-14 of the exact ones on these boxes; 2e-13 for convection, whose are within
9.3e-14."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from ssenss_b200.mesh import box_mesh
from test_gpu_affine import SHEAR, conv_reference, rel
from test_gpu_metric_rounding import gll, lagrange

pytestmark = pytest.mark.gpu

AX = ("pi,ekji->ekjp", "pj,ekji->ekpi", "pk,ekji->epji")


@pytest.mark.parametrize("n", range(2, 13))
@pytest.mark.parametrize("kind", ["box", "sheared"])
def test_against_closed_form_metric(kind, n, gpu_ctx_factory):
    S = np.eye(3) if kind == "box" else SHEAR
    m = box_mesh((3, 3, 3))
    if kind == "sheared":
        m = dataclasses.replace(m, vertices=np.einsum("ab,ebv->eav", S, m.vertices))
    ctx = gpu_ctx_factory(m, n)
    rng = np.random.default_rng(n)
    jac = S * (np.pi / 3.0)            # dx_a/dr_b
    det, inv = np.linalg.det(jac), np.linalg.inv(jac)   # inv[a][b] = dr_a/dx_b
    x, w, D = gll(n)
    rho = w[:, None, None] * w[:, None] * w
    u = rng.standard_normal((m.nel, n, n, n))
    du = [np.einsum(AX[b], D, u) for b in range(3)]
    G = inv @ inv.T * det
    ref = sum(np.einsum(AX[a], D.T, rho * sum(G[a, b] * du[b] for b in range(3)))
              for a in range(3))
    assert rel(ctx.local_opeval(O.PRESSURE, u), ref) < 1e-13
    xm, wm, Dm = gll((3 * n) // 2)
    one = np.ones((m.nel,) + (len(xm),) * 3)
    tinv = [inv[b, a] * one for a in range(3) for b in range(3)]   # dr_b/dx_a
    a, b = (rng.standard_normal((3, m.nel, n, n, n)) for _ in range(2))
    ref = conv_reference(a, b, lagrange(xm, x), Dm, wm, det * one, tinv)
    assert rel(ctx.convection_operator(a, b), ref) < 2e-13
    ctx.close()
