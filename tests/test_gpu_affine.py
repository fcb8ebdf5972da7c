"""The operator and convection on affine elements (parallelepipeds), where the library holds
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


def conv_reference(u, v, J, D, w, det, tinv):
    """The operator's definition in numpy for given matrices: D on the m
    points, J (m, n), weights w, det and tinv[a][b] = dr_b/dx_a there."""
    rho = w[:, None, None] * w[:, None] * w
    ax = ("pi,ekji->ekjp", "pj,ekji->ekpi", "pk,ekji->epji")

    def to(A, x):
        for e in ax:
            x = np.einsum(e, A, x)
        return x

    ui = [to(J, u[a]) for a in range(3)]
    out = []
    for c in range(3):
        vi = to(J, v[c])
        s = 0.0
        for b in range(3):
            dv, dp = np.einsum(ax[b], D, vi), np.einsum(ax[b], D, ui[b] * vi)
            for a in range(3):
                s = s + tinv[3 * a + b] * (ui[a] * dv + dp)
        out.append(to(J.T, 0.5 * rho * det * s))
    return np.stack(out)


@pytest.mark.parametrize("n", range(2, 13))
@pytest.mark.parametrize("mesh", ["box", "sheared", "channel"])
def test_convection_at_every_order(mesh, n, gpu_ctx_factory):
    """Both forms (u advecting v, and itself) against the oracle: nine
    constants an element on the affine meshes (to the noise of the oracle's
    own factors), per-point weights on the channel (1e-13); then the same
    fields at addresses that are not 16-byte aligned, which take the
    runtime-order kernel (1e-13 of each other, plus that noise)."""
    import torch
    m = {"box": lambda: box_mesh((3, 3, 4)), "sheared": sheared,
         "channel": lambda: channel_mesh((4, 3, 3), seed=7)}[mesh]()
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n)
    md = (3 * n) // 2
    tol = 1e-13 if mesh == "channel" else 1e-13 + 4e-14 * md * md
    rng = np.random.default_rng(n)
    u = rng.standard_normal((3, m.nel, n, n, n))
    v = rng.standard_normal((3, m.nel, n, n, n))
    got = ctx.convection_operator(u, v)
    assert rel(got, orc.convection(u, v)) < tol
    assert rel(ctx.convection_operator(u, u), orc.convection(u, u)) < tol
    raw = torch.zeros(2 * u.size + 2, dtype=torch.float64, device="cuda")
    um, vm = raw[1:1 + u.size].view(u.shape), raw[1 + u.size:1 + 2 * u.size].view(u.shape)
    um.copy_(torch.from_numpy(u))
    vm.copy_(torch.from_numpy(v))
    torch.cuda.synchronize()
    out = ctx.convection_operator(um, vm, torch.empty_like(um))
    assert rel(out.cpu().numpy(), got) < tol
    ctx.close()
    orc.close()


@pytest.mark.parametrize("n", [5, 8])
def test_convection_with_matrices_that_are_not_symmetric(n, gpu_ctx_factory):
    """A caller's own interpolation matrix without the points' symmetry: the
    line kernel's even / odd split does not apply, the result is the
    definition's all the same."""
    m = box_mesh((3, 3, 3))
    orc = O.Oracle(m, n)
    ctx = gpu_ctx_factory(m, n)
    md = (3 * n) // 2
    rng = np.random.default_rng(5)
    J = rng.standard_normal((md, n))
    D = rng.standard_normal((md, md))
    w = rng.uniform(0.1, 1.0, md)
    det = rng.uniform(0.5, 1.5, (m.nel, md, md, md))
    tinv = rng.standard_normal((9, m.nel, md, md, md))
    # stored matrices: deriv d[j][i] = D_ij, interp n x m
    ctx.setup_dealias(md, np.ascontiguousarray(D.T), w, tinv, det, np.ascontiguousarray(J.T))
    u = rng.standard_normal((3, m.nel, n, n, n))
    v = rng.standard_normal((3, m.nel, n, n, n))
    assert rel(ctx.convection_operator(u, v), conv_reference(u, v, J, D, w, det, tinv)) < 1e-13
    ctx.close()
    orc.close()


@pytest.mark.parametrize("n", [3, 6, 7])
def test_operator_with_a_matrix_that_is_not_antisymmetric(n, gpu_ctx_factory):
    """A caller's own derivative matrix without the points' symmetry, through
    the drop-in set-up: the line kernel's even / odd split does not apply, the
    result is the definition's all the same (1e-13)."""
    import ssenss_b200 as S
    m = box_mesh((3, 3, 3))
    orc = O.Oracle(m, n)
    rng = np.random.default_rng(n)
    ctx = S.Context(0)
    ctx.setup_connectivity(m.neigh)
    for level, nl in enumerate(orc.orders):
        D = rng.standard_normal((nl, nl))
        w = rng.uniform(0.1, 1.0, nl)
        geom = rng.uniform(0.5, 1.5, (6, m.nel, nl, nl, nl))
        det = rng.uniform(0.5, 1.5, (m.nel, nl, nl, nl))
        interp = None if level == 0 else rng.standard_normal((nl, orc.orders[level - 1]))
        ctx.setup_level(level, nl, np.ascontiguousarray(D.T), None, w, geom, det, interp)
        if level == 0:
            D0, w0, g0, d0 = D, w, geom, det
    ctx.setup_finish()
    u = rng.standard_normal((m.nel, n, n, n))
    ax = ("pi,ekji->ekjp", "pj,ekji->ekpi", "pk,ekji->epji")
    du = [np.einsum(ax[b], D0, u) for b in range(3)]
    rho = (w0[:, None, None] * w0[:, None] * w0) * d0
    sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
    ref = sum(np.einsum(ax[a], D0.T, sum(g0[sym[a][b]] * du[b] for b in range(3)) * rho)
              for a in range(3))
    assert rel(ctx.local_opeval(O.PRESSURE, u), ref) < 1e-13
    ctx.close()
    orc.close()
