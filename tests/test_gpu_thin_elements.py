"""Thin elements, whose metric factors differ by the square of the aspect
ratio: the constants of affine elements are only taken where every factor is
constant on its own scale, so no direction is lost and no deformation passes as
the rounding of the largest factor.  Against the oracle's per-point factors.
"""
import dataclasses

import numpy as np
import pytest

import oracle as O
from ssenss_b200.mesh import box_mesh

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("thin, n", [(1e-7, 2), (1e-6, 6), (1e-6, 8), (1e-6, 9), (1e-6, 12)])
def test_in_plane_directions_of_thin_elements(thin, n, gpu_ctx_factory):
    """A field that is constant across the thickness.  The thickness factor
    times the rounding of that zero derivative drowns the in-plane terms point
    by point, but the sum of A p across the thickness holds the in-plane terms
    alone: the columns of the derivative matrix sum to zero, so that direction
    enters it with the product of two roundings (below 1e-15 of the in-plane
    terms at aspect 1e6).  The remaining difference is that of the factors,
    4e-14 n^2 at most."""
    m = box_mesh((3, 3, 3), hi=(3.0, 3.0 * thin, 3.0))
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n)
    rng = np.random.default_rng(n)
    p = np.broadcast_to(rng.standard_normal((m.nel, n, 1, n)), (m.nel, n, n, n)).copy()
    got = ctx.local_opeval(O.PRESSURE, p).sum(axis=2)
    ref = orc.local_opeval(O.PRESSURE, p).sum(axis=2)
    assert rel(got, ref) < 4e-14 * n * n
    ctx.close()
    orc.close()


@pytest.mark.parametrize("n", [6, 8, 9, 12])
@pytest.mark.parametrize("axis, size", [(0, 2e-12), (1, 1e-9)])
def test_twisted_thin_elements(axis, size, n, gpu_ctx_factory):
    """Elements 1 x 1e-3 x 1 with every vertex moved by +-size along x or y so
    that the faces twist: the deformation is real on the scale of the factors
    it changes, so the per-point factors stay and agree to 1e-13, as on any
    deformed mesh."""
    m = box_mesh((4, 3, 4), hi=(4.0, 3e-3, 4.0))
    v = m.vertices.copy()
    idx = np.rint(v / np.array([1.0, 1e-3, 1.0])[None, :, None]).astype(int)
    odd = (idx[:, 1] + idx[:, 2]) if axis == 0 else (idx[:, 0] + idx[:, 2])
    v[:, axis] += size * (1 - 2 * (odd % 2))
    m = dataclasses.replace(m, vertices=v)
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n)
    rng = np.random.default_rng(n)
    p = rng.standard_normal((m.nel, n, n, n))
    for var in (O.PRESSURE, O.X_VELOCITY):
        assert rel(ctx.local_opeval(var, p), orc.local_opeval(var, p)) < 1e-13
    u = rng.standard_normal((3, m.nel, n, n, n))
    w = rng.standard_normal((3, m.nel, n, n, n))
    assert rel(ctx.convection_operator(u, w), orc.convection(u, w)) < 1e-13
    ctx.close()
    orc.close()
