"""The work a user of this library has it do, as measurable cases.

A case is one call (or one burst of calls) through the public Python entry
points of ssenss_b200 on a mesh of the library's own generators: the element
operator with its direct stiffness summation, the pressure Poisson and the
Helmholtz solves, dealiased convection, the whole time step on resident
fields, the particle advance, and a burst of requests to the solve server.
n is the number of GLL points per direction (polynomial order n - 1); a
"box" is the triply periodic [0, 2 pi]^3 box of equal hexahedra, a "channel"
the stretched and perturbed channel with two walls.

listed() are fixed cases, draw(rng) gives more of the same ranges,
prepare / run are what a user's program does before and in a pass, work is
what a pass cannot do without, exact the result in plain 64-bit torch.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import ssenss_b200 as S
from ssenss_b200 import _lib
from ssenss_b200.mesh import box_mesh, channel_mesh, periodic_box_fourier_rhs

EPS = 1e-10           # the absolute residual every solve of the path stops at
DT, VISC = 1e-3, 1.0 / 1600.0    # the Taylor-Green configuration's step


def listed():
    return [
        # the smallest call: one operator application on the 4^3 Taylor-Green
        # box (32,768 points), where latency and launches count
        dict(name="opeval_box4_n8", kind="opeval", mesh="box", nx=4, ny=4, nz=4, n=8,
             var="pressure", lam=0.0),
        # the velocity operator with walls on a deformed mesh, odd order
        dict(name="opeval_channel_n9", kind="opeval", mesh="channel", nx=24, ny=12, nz=12, n=9,
             var="velocity", lam=2.9e6),
        # the headline solve: Taylor-Green pressure, 2.1 M points, FP64
        dict(name="poisson_box16_n8", kind="poisson", mesh="box", nx=16, ny=16, nz=16, n=8,
             precision="fp64"),
        # the deformed channel's pressure solve, mixed precision
        dict(name="poisson_channel_n10_mixed", kind="poisson", mesh="channel", nx=16, ny=8,
             nz=8, n=10, precision="mixed"),
        # a small ragged box at another order, as the solve server meets
        dict(name="poisson_box556_n6_mixed", kind="poisson", mesh="box", nx=5, ny=5, nz=6, n=6,
             precision="mixed"),
        # a Helmholtz request of the server's range at its highest order
        dict(name="helmholtz_box889_n12", kind="helmholtz", mesh="box", nx=8, ny=8, nz=9, n=12,
             lam=50.0),
        # convection of a field by another: a periodic box, and a deformed
        # channel at odd order
        dict(name="convection_box12_n10", kind="convection", mesh="box", nx=12, ny=12, nz=12,
             n=10),
        dict(name="convection_channel_n7", kind="convection", mesh="channel", nx=20, ny=10,
             nz=11, n=7),
        # one time step of the two Taylor-Green configurations
        dict(name="step_box4_n8", kind="step", mesh="box", nx=4, ny=4, nz=4, n=8,
             precision="fp64"),
        dict(name="step_box16_n8", kind="step", mesh="box", nx=16, ny=16, nz=16, n=8,
             precision="mixed"),
        # the particle configuration: 1 M particles in the 16^3 flow
        dict(name="particles_1m_box16_n8", kind="particles", mesh="box", nx=16, ny=16, nz=16,
             n=8, count=1000000),
        # a burst of requests of mixed orders and sizes to the solve server
        dict(name="serve_burst24", kind="serve", count=24, most=125, batching=True,
             precision="mixed"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _shape(rng, points, n, aspect=(1.0, 1.0, 1.0), least=3, most=32):
    """Elements per direction for about `points` local points: each side a
    little off the cube (or the given aspect), at least `least`."""
    nel = max(points / n ** 3, float(least ** 3))
    unit = (nel / (aspect[0] * aspect[1] * aspect[2])) ** (1.0 / 3.0)
    side = [int(round(unit * a * rng.uniform(0.85, 1.15))) for a in aspect]
    return [min(max(s, least), most) for s in side]


def draw(rng):
    kind = rng.choice(["opeval", "poisson", "helmholtz", "convection", "step", "particles",
                       "serve"])
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(8, 32), most=rng.randint(27, 150),
                    batching=rng.random() < 0.7, precision=rng.choice(["fp64", "mixed"]))
    mesh = "box"
    if kind in ("opeval", "poisson", "convection") and rng.random() < 0.4:
        mesh = "channel"
    n = rng.choice([6, 7, 8, 9] if kind in ("step", "particles")
                   else [5, 6, 7, 8, 8, 9, 10, 11, 12])
    top = {"opeval": 3e6, "poisson": 2e6 if mesh == "box" else 6e5, "helmholtz": 1.8e6,
           "convection": 1.7e6, "step": 1.5e6, "particles": 2e6}[kind]
    points = _log_uniform(rng, 2e4, top)
    nx, ny, nz = _shape(rng, points / 1.3, n, (2.0, 1.0, 1.0) if mesh == "channel" else
                        (1.0, 1.0, 1.0))
    case = dict(kind=kind, mesh=mesh, nx=nx, ny=ny, nz=nz, n=n)
    if kind == "opeval":
        case["var"] = rng.choice(["pressure", "velocity"])
        case["lam"] = 0.0 if case["var"] == "pressure" else _log_uniform(rng, 0.5, 3e6)
    elif kind in ("poisson", "step"):
        case["precision"] = rng.choice(["fp64", "mixed"])
    elif kind == "helmholtz":
        case["lam"] = rng.choice([_log_uniform(rng, 0.5, 100.0), 2.9e6])
    elif kind == "particles":
        case["count"] = int(_log_uniform(rng, 1e3, 1e6))
    return case


# -- what a user's program has in hand -----------------------------------------

@functools.lru_cache(maxsize=32)
def _mesh(kind, nx, ny, nz):
    return channel_mesh((nx, ny, nz)) if kind == "channel" else box_mesh((nx, ny, nz))


def _mesh_of(case):
    return _mesh(case["mesh"], case["nx"], case["ny"], case["nz"])


def _context(case, dealias=False, particles=False):
    ctx = S.Context(0)
    ctx.set_setup_options(no_dealias=not dealias, no_particles=not particles)
    lam = case.get("lam") or 0.0
    ctx.set_parameters((11.0 / 6.0) / lam / VISC if lam > 0.0 else DT, VISC, 1.0)
    if "precision" in case:
        ctx.set_precision(case["precision"])
    ctx.setup_mesh(_mesh_of(case), case["n"])
    return ctx


def _modes(case, seed, count=8, even_y=True):
    """(amplitude, kx, ky, kz, phase) of `count` seeded Fourier modes that are
    periodic on the mesh; on a channel the mean-free cos(pi ky (y + 1) / 2)
    profiles of a pressure right-hand side."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        k = rng.integers(-3, 4, 3)
        if not k.any():
            k[0] = 1
        kx = k[0] / 2.0 if case["mesh"] == "channel" else float(k[0])
        out.append((rng.standard_normal(), kx, float(abs(k[1]) if case["mesh"] == "channel"
                                                      else k[1]), float(k[2]),
                    rng.uniform(0.0, 2.0 * math.pi)))
    return out


def _field(case, seed, X):
    """The sum of the seeded modes at the nodes X (three tensors)."""
    x, y, z = X
    g = torch.zeros_like(x)
    for a, kx, ky, kz, phase in _modes(case, seed):
        if case["mesh"] == "channel":
            g += a * torch.cos(kx * x + kz * z + phase) * torch.cos(0.5 * math.pi * ky * (y + 1))
        else:
            g += a * torch.cos(kx * x + ky * y + kz * z + phase)
    return g


def _vector(case, seed, X):
    return torch.stack([_field(case, seed * 7 + c, X) for c in range(3)])


def _nodes(ctx):
    return [torch.from_numpy(ctx.level_data(0, 12 + a)).cuda() for a in range(3)]


def _stream(ctx):
    return torch.cuda.ExternalStream(ctx.stream)


def _serve_requests(case, seed):
    """Shapes, orders and coefficients of a burst: periodic boxes of 8 to
    `most` elements, half Poisson and half Helmholtz (lambda in (0, 100])."""
    rng = np.random.default_rng(1000 + seed % 100000)
    boxes = [(a, b, c) for a in range(2, 7) for b in (a, a + 1) for c in (b, b + 1)
             if c <= a + 1 and a * b * c <= case["most"]]
    fixed = np.random.default_rng(77 * case["count"] + case["most"])
    reqs = []
    for k in range(case["count"]):
        # the mix of sizes and orders belongs to the case, the data to the seed
        shape = boxes[int(fixed.integers(len(boxes)))]
        n = int(fixed.choice([6, 8, 8, 10, 12]))
        poisson = bool(fixed.integers(2))
        lam = 0.0 if poisson else float(fixed.uniform(0.5, 100.0))
        reqs.append((shape, n, lam, int(rng.integers(1 << 31))))
    return reqs


def _taylor_green(case, seed, ctx):
    """Taylor-Green state at a seeded phase and amplitude after two steps of
    the integrator, as device fields."""
    rng = np.random.default_rng(seed)
    amp = rng.uniform(0.9, 1.1)
    X, Y, Z = (x + p for x, p in zip(_nodes(ctx), rng.uniform(0.0, 2.0 * math.pi, 3)))
    u = amp * torch.stack([torch.sin(X) * torch.cos(Y) * torch.cos(Z),
                           -torch.cos(X) * torch.sin(Y) * torch.cos(Z), torch.zeros_like(X)])
    p = amp ** 2 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0) / 16.0
    torch.cuda.synchronize()
    conv = ctx.convection_operator(u, u, torch.empty_like(u))
    rot = ctx.stokes_operator(0, u, None, torch.empty_like(u))
    zero = torch.zeros_like(u)
    torch.cuda.synchronize()
    ctx.flow_set([u, u, u], [conv, conv, zero], [rot, rot, zero], [p, p, p], None, 0.0)
    for _ in range(2):
        ctx.navier_stokes_step(history=False)
    got = {k: [torch.empty_like(u) for _ in range(3)] for k in ("u", "conv", "rot")}
    got["p"] = [torch.empty_like(p) for _ in range(3)]
    got["t"] = _flow_get(ctx, got)
    return got


def _flow_get(ctx, into):
    """Copy the resident state's levels into the given device fields."""
    ff = _lib.FlowFields()
    for name in ("u", "conv", "rot", "p"):
        for level, x in enumerate(into.get(name, [])):
            getattr(ff, name)[level] = ctypes.c_void_p(x.data_ptr())
    t = ctypes.c_double()
    if ctx.lib.ssg_flow_get(ctx.h, ctypes.byref(ff), ctypes.byref(t)) != 0:
        raise RuntimeError("flow_get")
    return t.value


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "serve":
        srv = S.Server(0, hbm_budget=40e9, max_active=8)
        if case["batching"]:
            srv.set_batching(16, 1 << 16)
        reqs = []
        for shape, n, lam, s in _serve_requests(case, seed):
            mesh = _mesh("box", *shape)
            reqs.append((mesh, n, periodic_box_fourier_rhs(shape, n, s), lam,
                         S.mesh_key(mesh, n)))
        st.update(srv=srv, reqs=reqs)
        return st
    ctx = _context(case, dealias=kind in ("convection", "step"),
                   particles=kind in ("step", "particles"))
    st["ctx"] = ctx
    if kind == "step":
        st["flow"] = _taylor_green(case, seed, ctx)
        st["out"] = {"u": [torch.empty_like(st["flow"]["u"][0])],
                     "p": [torch.empty_like(st["flow"]["p"][0])]}
        return st
    X = _nodes(ctx)
    if kind == "opeval":
        st["var"] = S.PRESSURE if case["var"] == "pressure" else S.X_VELOCITY
        st["p"] = _field(case, seed, X)
        st["out"] = torch.empty_like(st["p"])
    elif kind in ("poisson", "helmholtz"):
        g = _field(case, seed, X)
        bj = torch.from_numpy(ctx.level_data(0, 6)).cuda()
        if kind == "poisson":
            g -= (bj * g).sum() / bj.sum()
        f = bj * g
        torch.cuda.synchronize()
        st["f"] = ctx.direct_stiffness_summation(f)
        st["u"] = torch.zeros_like(f)
    elif kind == "convection":
        st["u"], st["v"] = _vector(case, 2 * seed, X), _vector(case, 2 * seed + 1, X)
        st["out"] = torch.empty_like(st["u"])
    elif kind == "particles":
        # reference-domain velocity of a Taylor-Green field at three times,
        # particles anywhere, half in motion, response times 0.1 .. 1
        rng = np.random.default_rng(seed)
        h = [2.0 * math.pi / case[a] for a in ("nx", "ny", "nz")]
        x, y, z = (a + p for a, p in zip(X, rng.uniform(0.0, 2.0 * math.pi, 3)))
        u = torch.stack([torch.sin(x) * torch.cos(y) * torch.cos(z) * (2.0 / h[0]),
                         -torch.cos(x) * torch.sin(y) * torch.cos(z) * (2.0 / h[1]), 0 * x])
        ur = torch.stack([u * 0.98, u * 0.99, u])
        torch.cuda.synchronize()
        ctx.set_particle_velocity(ur)
        state = np.zeros((case["count"], 8))
        ints = np.zeros((case["count"], 3), np.int32)
        state[:, :3] = rng.uniform(-1.0, 1.0, (case["count"], 3))
        state[::2, 3:6] = rng.uniform(-5.0, 5.0, (len(state[::2]), 3))
        state[:, 7] = rng.uniform(0.1, 1.0, case["count"])
        ints[:, 0] = ints[:, 1] = rng.integers(0, ctx.nel, case["count"])
        st["state0"], st["ints0"] = torch.from_numpy(state).cuda(), torch.from_numpy(ints).cuda()
        st["state"], st["ints"] = torch.empty_like(st["state0"]), torch.empty_like(st["ints0"])
    st["stream"] = _stream(ctx)
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = st["srv"]
        ids = [srv.submit(mesh, n, f, lam=lam, eps=EPS, precision=case["precision"], key=key)
               for mesh, n, f, lam, key in st["reqs"]]
        out = []
        for i in ids:
            u, status, _ = srv.wait(i)
            if status != "SSG_OK":
                raise RuntimeError(status)
            out.append(u)
        return out
    ctx = st["ctx"]
    if kind == "opeval":
        return ctx.global_opeval(st["var"], st["p"], st["out"])
    if kind == "convection":
        return ctx.convection_operator(st["u"], st["v"], st["out"])
    if kind in ("poisson", "helmholtz"):
        with torch.cuda.stream(st["stream"]):
            st["u"].zero_()
        if kind == "poisson":
            return ctx.solve_poisson_cg(st["f"], st["u"], eps=EPS, history=False)[0]
        return ctx.solve_helmholtz_cg(S.X_VELOCITY, st["f"], st["u"], eps=EPS,
                                      history=False)[0]
    if kind == "step":
        s = st["flow"]
        ctx.flow_set(s["u"], s["conv"], s["rot"], s["p"], None, s["t"])
        ctx.navier_stokes_step(history=False)
        _flow_get(ctx, st["out"])
        return st["out"]
    with torch.cuda.stream(st["stream"]):
        st["state"].copy_(st["state0"])
        st["ints"].copy_(st["ints0"])
    ctx.integrate_particle_equations(st["state"], st["ints"], 2 * DT, DT)
    return [st["state"], st["ints"]]


def work(case):
    """Bytes: each input field read once, each output field written once; the
    geometry of a box follows from its element size, a channel's metric (six
    terms a point, nine on the dealiasing grid) is read.  Flops: one
    application of the operators the call cannot do without."""
    kind = case["kind"]
    if kind == "serve":
        pts = sum(s[0] * s[1] * s[2] * n ** 3 * 1.0 for s, n, _, _ in _serve_requests(case, 0))
        return {"bytes": 16.0 * pts, "flops": 130.0 * pts}
    n = case["n"]
    pts = float(case["nx"] * case["ny"] * case["nz"] * n ** 3)
    metric = 48.0 if case["mesh"] == "channel" else 0.0
    op = 12.0 * n + 21.0
    if kind == "convection":
        m = (3 * n) // 2
        dense = pts * (m / n) ** 3
        lines = 2.0 * n * m * (n * n + n * m + m * m) / n ** 3 * pts
        return {"bytes": 72.0 * pts + (72.0 * dense if metric else 0.0),
                "flops": 9.0 * lines + dense * 9 * 2 * (2.0 * m)}
    if kind == "step":
        return {"bytes": (38.0 + 4.0) * 8.0 * pts, "flops": 60.0 * op * pts}
    if kind == "particles":
        return {"bytes": 152.0 * case["count"] + 72.0 * pts, "flops": 4000.0 * case["count"]}
    return {"bytes": (16.0 + metric) * pts, "flops": op * pts}


# -- the same results in plain 64-bit torch -------------------------------------

def _gll(n):
    c = np.zeros(n)
    c[-1] = 1.0
    x = np.concatenate(([-1.0], np.polynomial.legendre.legroots(
        np.polynomial.legendre.legder(c)), [1.0])) if n > 2 else np.array([-1.0, 1.0])
    d1 = np.polynomial.legendre.legder(c)
    d2 = np.polynomial.legendre.legder(d1)
    for _ in range(3):
        if n > 2:
            x[1:-1] -= np.polynomial.legendre.legval(x[1:-1], d1) / \
                np.polynomial.legendre.legval(x[1:-1], d2)
    ln = np.polynomial.legendre.legval(x, c)
    w = 2.0 / (n * (n - 1) * ln ** 2)
    D = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                D[i, j] = ln[i] / (ln[j] * (x[i] - x[j]))
    D -= np.diag(D.sum(1))
    return x, w, D


def _lagrange(xto, x):
    J = np.ones((len(xto), len(x)))
    for p in range(len(x)):
        for q in range(len(x)):
            if q != p:
                J[:, p] *= (xto - x[q]) / (x[p] - x[q])
    return J


def _apply(A, u, axis):
    """A along axis 0 (x, fastest), 1 or 2 of u[..., k, j, i]."""
    return torch.einsum(("pi,...kji->...kjp", "pj,...kji->...kpi", "pk,...kji->...pji")[axis],
                        A, u)


class _Exact:
    """Geometry and operators of a structured mesh from its vertices."""

    def __init__(self, case, shape=None):
        shape = shape or (case["nx"], case["ny"], case["nz"])
        n = case["n"]
        self.case, self.n = case, n
        mesh = _mesh(case["mesh"], *shape)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.vert = torch.from_numpy(mesh.vertices).to(self.dev).reshape(-1, 3, 2, 2, 2)
        x, w, D = _gll(n)
        self.x, self.D = x, torch.from_numpy(D).to(self.dev)
        self.X, self.det, self.inv = self.geometry(x)
        wt = torch.from_numpy(w).to(self.dev)
        rho = wt[:, None, None] * wt[:, None] * wt
        self.bj = rho * self.det
        self.G = torch.einsum("acekji,bcekji->abekji", self.inv, self.inv) * self.bj
        walls = case["mesh"] == "channel"
        e = np.arange(shape[0] * shape[1] * shape[2])
        at = [e % shape[0], (e // shape[0]) % shape[1], e // (shape[0] * shape[1])]
        m, r = n - 1, np.arange(n)
        ids, cnt = [], []
        for a in range(3):
            idx = at[a][:, None] * m + r[None]
            wall = walls and a == 1
            cnt.append(shape[a] * m + (1 if wall else 0))
            ids.append(idx if wall else idx % cnt[a])
        gid = ids[0][:, None, None, :] + cnt[0] * (ids[1][:, None, :, None] +
                                                   cnt[1] * ids[2][:, :, None, None])
        self.gid = torch.from_numpy(gid).to(self.dev)
        self.count = cnt[0] * cnt[1] * cnt[2]
        self.mask = torch.ones_like(self.X[0])
        if walls:
            on = (ids[1] == 0) | (ids[1] == shape[1] * m)
            self.mask *= torch.from_numpy(~on).to(self.dev)[:, None, :, None]

    def geometry(self, x):
        """Node coordinates, det J and inv[a][b] = dr_a/dx_b at the points x."""
        L = torch.from_numpy(np.stack([(1 - x) / 2, (1 + x) / 2], 1)).to(self.dev)
        dL = torch.from_numpy(np.stack([-0.5 + 0 * x, 0.5 + 0 * x], 1)).to(self.dev)
        X, J = [], []
        for a in range(3):
            v = self.vert[:, a]
            X.append(_apply(L, _apply(L, _apply(L, v, 0), 1), 2))
            J.append([_apply(dL if b == 2 else L, _apply(dL if b == 1 else L, _apply(
                dL if b == 0 else L, v, 0), 1), 2) for b in range(3)])
        Jm = torch.stack([torch.stack(r, -1) for r in J], -2)
        return X, torch.linalg.det(Jm), torch.linalg.inv(Jm).movedim((-2, -1), (0, 1))

    def dss(self, u):
        tot = torch.zeros(self.count, dtype=torch.float64, device=self.dev)
        tot.index_add_(0, self.gid.reshape(-1), u.reshape(-1))
        return tot[self.gid]

    def operator(self, u, lam, masked):
        d = torch.stack([_apply(self.D, u, a) for a in range(3)])
        w = torch.einsum("abekji,bekji->aekji", self.G, d)
        out = sum(_apply(self.D.T.contiguous(), w[a], a) for a in range(3))
        if lam:
            out = out + lam * self.bj * u
        return self.dss(out * self.mask if masked else out)

    def solve(self, f, lam):
        """Jacobi CG on the assembled system to rounding; None if it is slow."""
        one = torch.ones_like(f)
        weight = 1.0 / self.dss(one)
        D2 = (self.D ** 2).T.contiguous()
        diag = sum(_apply(D2, self.G[a, a], a) for a in range(3))
        if self.case["mesh"] == "channel":
            dd = torch.diagonal(self.D)
            d = [dd.view(-1, *([1] * a)) for a in range(3)]
            diag = diag + 2 * (self.G[0, 1] * d[0] * d[1] + self.G[0, 2] * d[0] * d[2] +
                               self.G[1, 2] * d[1] * d[2])
        diag = self.dss(diag + lam * self.bj)
        dot = lambda a, b: (a * weight * b).sum()  # noqa: E731
        unique = weight.sum()
        if not lam:
            f = f - dot(f, one) / unique
        u, r = torch.zeros_like(f), f.clone()
        z = r / diag
        p, rz = z.clone(), dot(r, z)
        stop = 1e-14 * float(dot(f, f)) ** 0.5
        best, since = float("inf"), 0
        for it in range(3000):
            ap = self.operator(p, lam, False)
            alpha = rz / dot(p, ap)
            u = u + alpha * p
            r = r - alpha * ap
            z = r / diag
            rz, old = dot(r, z), rz
            p = z + (rz / old) * p
            if it % 20 == 19:
                err = float(dot(r, r)) ** 0.5
                since = 0 if err < 0.5 * best else since + 20
                best = min(best, err)
                if err < stop or (since >= 200 and best < 1e-12):
                    break
        return u if lam else u - dot(u, one) / unique


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "particles"):
        return None     # a whole step; a walk across element faces (bits are compared)
    if kind == "serve":
        out = []
        for shape, n, lam, s in _serve_requests(case, seed):
            ex = _Exact(dict(mesh="box", n=n), shape)
            f = torch.from_numpy(periodic_box_fourier_rhs(shape, n, s)).to(ex.dev)
            out.append(ex.solve(f, lam))
        return out
    pts = case["nx"] * case["ny"] * case["nz"] * case["n"] ** 3
    if kind == "poisson" and case["mesh"] == "channel" and pts > 3e5:
        return None     # thousands of plain CG iterations
    ex = _Exact(case)
    if kind == "opeval":
        return ex.operator(_field(case, seed, ex.X), case["lam"], case["var"] == "velocity")
    if kind in ("poisson", "helmholtz"):
        g = _field(case, seed, ex.X)
        if kind == "poisson":
            g = g - (ex.bj * g).sum() / ex.bj.sum()
        return ex.solve(ex.dss(ex.bj * g), case.get("lam") or 0.0)
    u, v = _vector(case, 2 * seed, ex.X), _vector(case, 2 * seed + 1, ex.X)
    x, w, D = _gll((3 * case["n"]) // 2)
    J = torch.from_numpy(_lagrange(x, ex.x)).to(ex.dev)
    D = torch.from_numpy(D).to(ex.dev)
    _, det, inv = ex.geometry(x)
    wt = torch.from_numpy(w).to(ex.dev)
    bj = wt[:, None, None] * wt[:, None] * wt * det
    up = lambda a: _apply(J, _apply(J, _apply(J, a, 0), 1), 2)  # noqa: E731
    JT = J.T.contiguous()
    ui = [up(u[a]) for a in range(3)]
    out = []
    for c in range(3):
        vi = up(v[c])
        acc = torch.zeros_like(vi)
        for b in range(3):
            dv, duv = _apply(D, vi, b), _apply(D, ui[b] * vi, b)
            for a in range(3):
                acc += inv[b, a] * (ui[a] * dv + duv)
        acc *= 0.5 * bj
        out.append(_apply(JT, _apply(JT, _apply(JT, acc, 0), 1), 2))
    return torch.stack(out)
