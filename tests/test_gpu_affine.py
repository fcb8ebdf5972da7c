"""The operator on affine elements (parallelepipeds), where the library holds
six metric constants an element instead of six factors a point, against the
oracle's per-point factors; and the rule's other side, a mesh with a single
deformed element, which keeps the per-point factors.

The oracle differentiates node coordinates, so its factors of an affine
element carry rounding noise of about eps |x| n^2 / h, at most 4e-14 n^2 of
the largest factor (the bound the rule itself uses): the operators agree to
that, the deformed mesh to the 1e-13 of the per-point path.
"""
import dataclasses

import numpy as np
import pytest

import oracle as O
from ssenss_b200.mesh import box_mesh, channel_mesh

pytestmark = pytest.mark.gpu

SHEAR = np.array([[1.0, 0.3, -0.2], [0.1, 0.8, 0.25], [-0.15, 0.05, 1.2]])


def sheared(periodic=(True, True, True)):
    m = box_mesh((3, 4, 3), periodic=periodic)
    return dataclasses.replace(m, vertices=np.einsum("ab,ebv->eav", SHEAR, m.vertices))


def one_deformed():
    m = box_mesh((3, 3, 3))
    v = m.vertices.copy()
    v[5, 0, 3] += 1e-6
    return dataclasses.replace(m, vertices=v)


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("n", range(2, 13))
@pytest.mark.parametrize("mesh, tol", [
    ("box", None), ("sheared", None), ("sheared_walls", None), ("one_deformed", 1e-13)])
def test_operator_on_affine_and_deformed_elements(mesh, tol, n, gpu_ctx_factory):
    m = {"box": lambda: box_mesh((3, 3, 4)), "sheared": sheared,
         "sheared_walls": lambda: sheared((True, False, True)),
         "one_deformed": one_deformed}[mesh]()
    # (1e-13 is stated for factors of the same rounding: the per-point path)
    tol = 4e-14 * n * n if tol is None else tol
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n)
    p = np.random.default_rng(n).standard_normal((m.nel, n, n, n))
    for var in (O.PRESSURE, O.X_VELOCITY):
        assert rel(ctx.local_opeval(var, p), orc.local_opeval(var, p)) < tol
        assert rel(ctx.global_opeval(var, p), orc.global_opeval(var, p)) < tol
    ctx.close()
    orc.close()


@pytest.mark.parametrize("mesh, n", [("box", 8), ("sheared", 6), ("sheared", 8)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_poisson_on_affine_elements(mesh, n, precision, gpu_ctx_factory):
    """The solution's residual under the oracle's own operator: the solve's
    eps, plus the two operators' difference on the solution."""
    m = box_mesh((3, 3, 4)) if mesh == "box" else sheared()
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n, precision=precision)
    r = np.random.default_rng(3).standard_normal((m.nel, n, n, n))
    f = orc.dss(orc.dss(r) / n ** 3 * ctx.level_data(0, 9))
    w = ctx.level_data(0, 9)
    f -= (w * f).sum() / w.sum()
    u, info = ctx.solve_poisson_cg(f, np.zeros_like(f))
    assert info["status"] == "SSG_OK"
    res = f - orc.global_opeval(O.PRESSURE, u)
    res -= (w * res).sum() / w.sum()
    assert np.sqrt((w * res * res).sum()) < 1.5e-10 + 4e-14 * n * n * np.sqrt((w * f * f).sum())
    ctx.close()
    orc.close()
