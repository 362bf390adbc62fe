"""Performance cases of the solver library: the calls that an elliptic driver or
a DNS time step makes, through the public Python entry points.

Every case is a dict of plain values with a "kind":

  direct     one Helmholtz solve of a field on factored systems (Field::solve):
             "plain" mode by mode on device planes, "batched" every mode in one
             call on device planes, "host" the batched call on pinned host arrays
  mixed      the batched solve in FP32 iterations inside FP64 refinement
  build      systems built, factored, used for one solve and dropped (a driver
             that solves once, a time step that changed)
  batch      several small meshes of uneven size and order solved in one call
  transform  z-direction Fourier transform of a field, there and back
  forcing    wave step, pressure forcing and projection of a DNS step
  fieldops   the three gradients of a field and the smoothing of one

``listed`` gives the measured cases, ``draw`` more of the same ranges.
``exact`` computes the same outputs in 64 bits with torch alone (a
Jacobi-preconditioned conjugate gradient with restarts from the true residual
for the solves).
"""
import functools
import math

import numpy as np
import torch

import semtex_b200 as sx
from semtex_b200.mesh import rect_mesh

DEV = "cuda"


def listed():
    return [
        # a 2-D elliptic run on a small mesh: one plane, the shortest call
        dict(name="direct_small", kind="direct", form="plain", nx=4, ny=4, np=9, nz=1, walls="D", periodic=False,
             jitter=0.0, lam="one", base=0),
        # the viscous or pressure solve of a periodic channel, 32 modes
        dict(name="direct_channel", kind="direct", form="batched", nx=32, ny=32, np=9, nz=64, walls="D",
             periodic=True, jitter=0.15, lam="spread", base=0),
        # a rank's few modes of a large mesh at high order: wide bands
        dict(name="direct_large", kind="direct", form="batched", nx=64, ny=64, np=11, nz=24, walls="D",
             periodic=True, jitter=0.2, lam="spread", base=0),
        # a pressure Poisson solve from host memory: natural walls, a singular
        # mean mode, ragged sizes, prescribed boundary fluxes
        dict(name="pressure_host", kind="direct", form="host", nx=37, ny=23, np=8, nz=40, walls="N",
             periodic=True, jitter=0.15, lam="zero", base=0),
        # the viscous solves of a DNS step at its usual time step (mass
        # dominated): the mixed-precision form
        dict(name="viscous_channel", kind="mixed", nx=32, ny=32, np=9, nz=64, walls="D", periodic=True,
             jitter=0.15, lam="1e6", base=0),
        # the same on the large DNS mesh, one rank's block of modes
        dict(name="viscous_large", kind="mixed", nx=128, ny=64, np=11, nz=16, walls="D", periodic=True,
             jitter=0.15, lam="4e6", base=8),
        # systems that are built for one solve
        dict(name="build_solve", kind="build", nx=33, ny=26, np=8, nz=20, walls="D", periodic=False, jitter=0.0,
             lam="spread", base=0),
        # many small meshes of uneven sizes and orders, in one call
        dict(name="batch_small", kind="batch", members=24, mesh_seed=9, most=12),
        # the transforms around the nonlinear terms: a power of two ...
        dict(name="transform_128", kind="transform", nx=64, ny=64, np=11, nz=128, pad=0),
        # ... and another length, with padded planes
        dict(name="transform_96", kind="transform", nx=32, ny=32, np=9, nz=96, pad=6),
        # one DNS step's forcing on the large mesh, second order in time
        dict(name="forcing_large", kind="forcing", nx=128, ny=64, np=11, nz=32, order=2, scalar=False, base=16),
        # velocity gradients and pressure smoothing, even order of points
        dict(name="fieldops_mid", kind="fieldops", nx=48, ny=40, np=8, nz=48, base=0),
    ]


def draw(rng):
    """One more case of the listed ranges, no larger than the listed ones."""
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    # direct solves are what the library is for: they are drawn most often
    kind = rng.choice(["direct", "direct", "direct", "mixed", "mixed", "build", "batch", "transform", "transform",
                       "forcing", "fieldops"])
    while True:
        nx, ny, n = log_int(2, 64), log_int(2, 64), rng.randint(5, 11)
        if kind in ("forcing", "mixed"):
            nx = log_int(4, 128)
        periodic = rng.random() < 0.6 and nx >= 3
        base = rng.choice([0, 0, rng.randint(1, 64)])
        mesh = dict(nx=nx, ny=ny, np=n, periodic=periodic, jitter=rng.choice([0.0, 0.15, 0.2]), base=base)
        if kind in ("direct", "build"):
            c = dict(kind=kind, nz=2 * log_int(1, 32), walls=rng.choice(["D", "D", "N", "DM"]), **mesh)
            c["lam"] = "zero" if c["walls"] == "N" else rng.choice(["spread", "zero", "one"])
            if kind == "direct":
                c["form"] = rng.choice(["batched", "batched", "plain", "host"])
            if c["lam"] == "one" and base == 0 and rng.random() < 0.5:
                c["nz"] = 1
        elif kind == "mixed":
            c = dict(kind=kind, nz=2 * log_int(1, 32), walls="D", lam=rng.choice(["1e5", "1e6", "4e6"]), **mesh)
        elif kind == "batch":
            c = dict(kind=kind, members=rng.randint(4, 24), mesh_seed=rng.randint(10, 10**6), most=rng.randint(6, 12))
        elif kind == "transform":
            nz = rng.choice([8, 16, 24, 32, 40, 48, 60, 64, 80, 96, 100, 120, 128, 144, 160, 192, 240, 256, 320, 512])
            c = dict(kind=kind, nx=nx, ny=ny, np=n, nz=nz, pad=rng.choice([0, 1, 6]))
        elif kind == "forcing":
            c = dict(kind=kind, nx=nx, ny=ny, np=n, nz=2 * log_int(4, 64), order=rng.randint(1, 3),
                     scalar=rng.random() < 0.3, base=base)
        else:
            c = dict(kind=kind, nx=nx, ny=ny, np=n, nz=2 * log_int(2, 32), base=base)
        if _size(c) <= max(_size(x) for x in listed() if x["kind"] == kind):
            return c


def _size(c):
    """A case's cost for draw: band storage where systems are factored, field points elsewhere."""
    if c["kind"] == "batch":
        return c["members"] * c["most"] ** 2
    points = c["nx"] * c["ny"] * c["np"] ** 2 * c["nz"]
    if c["kind"] == "forcing":
        return points * c["order"] * (4 if c["scalar"] else 3)
    if c["kind"] not in ("direct", "build"):
        return points
    m = _mesh(c["nx"], c["ny"], c["np"], c["walls"], c["periodic"], c["jitter"])
    return max(c["nz"] // 2, 1) * m.nsolve * m.nband


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _mesh(nx, ny, n, walls="D", periodic=True, jitter=0.15):
    """The host mesh (coordinates, numbering, boundary list) of a case."""
    if walls == "DM":  # essential below, mixed above
        bc = {"bottom": "D", "top": ("M", 2.0, 0.5)}
    else:
        bc = {"bottom": walls, "top": walls}
    if not periodic:
        bc.update(left="N" if walls == "N" else "D", right="N")
    return rect_mesh(nx, ny, n, 0.0, 2 * math.pi if periodic else 1.0, 0.0, 1.0, jitter=jitter, seed=3,
                     periodic_x=periodic, bc=bc)


def _case_mesh(c):
    return _mesh(c["nx"], c["ny"], c["np"], c.get("walls", "D"), c.get("periodic", True), c.get("jitter", 0.15))


@functools.lru_cache(maxsize=8)
def _batch_meshes(members, mesh_seed, most):
    """Straight-sided meshes of [0,1]^2, 2 to `most` elements a side, orders
    4 to 10, 1 to 12 modes, with a Helmholtz constant each."""
    rng = np.random.default_rng(mesh_seed)
    out = []
    for _ in range(members):
        ex, ey = (int(v) for v in rng.integers(2, most + 1, size=2))
        order, modes = int(rng.integers(4, 11)), int(rng.integers(1, 13))
        lam = float(np.exp(rng.uniform(np.log(1e3), np.log(1e5))))
        out.append((rect_mesh(ex, ey, order + 1), modes, lam))
    return out


def _stream():
    """One stream of the program's own, as a time-stepping program has."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


_STREAM = None


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _constants(c, seed):
    """Per-mode (lambda2, betak2) of a case."""
    nm = max(c["nz"] // 2, 1)
    k = np.arange(c["base"], c["base"] + nm, dtype=np.float64)
    lam = c["lam"]
    if lam == "spread":  # a time-step and a viscosity per mode are not known in advance: log-uniform
        lam2 = np.exp(np.random.default_rng(seed).uniform(np.log(1e-2), np.log(1e4), nm))
    else:
        lam2 = np.full(nm, {"zero": 0.0, "one": 1.0}.get(lam) if lam in ("zero", "one") else float(lam))
    return lam2, k ** 2


def _node_ids(m):
    """(nel, np, np) ids of the unique nodes: element-boundary nodes by the
    mesh's numbering, interior nodes after them."""
    n = m.np
    ring = [(0, j) for j in range(n - 1)] + [(i, n - 1) for i in range(n - 1)]
    ring += [(n - 1, n - 1 - j) for j in range(n - 1)] + [(n - 1 - i, 0) for i in range(n - 1)]
    ids = np.empty((m.nel, n, n), dtype=np.int64)
    for a, (i, j) in enumerate(ring):
        ids[:, i, j] = m.btog[:, a]
    ids[:, 1:-1, 1:-1] = m.nglobal + np.arange(m.nel * (n - 2) ** 2).reshape(m.nel, n - 2, n - 2)
    return ids


def _continuous(m, planes, base, gen, mean_free=False):
    """Random continuous Fourier planes whose modes decay, as a field's spectrum does."""
    ids = torch.from_numpy(_node_ids(m).reshape(-1)).to(DEV)
    k = (torch.arange(planes, device=DEV) // 2 + base).double()
    v = torch.randn(planes, m.n_unique, dtype=torch.float64, device=DEV, generator=gen)
    f = (v * torch.exp(-k / 8.0)[:, None])[:, ids]
    if mean_free and base == 0:  # a Poisson problem with natural walls has a solution only then
        w = _Sem(m).mass.reshape(-1)
        f[0] -= (f[0] * w).sum() / w.sum()
    if base == 0 and planes > 1:
        f[1] = 0.0  # the Nyquist datum is not solved for
    return f.contiguous()


def _boundary_lines(m, planes, rng, walls, base):
    """Boundary values (planes, nbound, np): essential values or fluxes,
    smooth along the walls and equal where two sides meet."""
    out = np.zeros((planes, max(len(m.boundaries), 1), m.np))
    for p in range(planes):
        a, b, ph = rng.standard_normal(3)
        amp = math.exp(-(p // 2 + base) / 8.0)
        if walls == "N":  # fluxes of the mean mode cancel between two walls only roughly: leave them out
            amp = 0.0 if (base == 0 and p == 0) else amp
        for i, bd in enumerate(m.boundaries):
            x, y = m.side_xy(bd)
            out[p, i] = amp * (a * np.cos(x + ph) + b * y)
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.as_tensor(a))
    return t


def _solve_inputs(c, seed):
    """mesh, constants, forcing (device) and boundary lines of a solve case."""
    m = _case_mesh(c)
    lam2, bk2 = _constants(c, seed)
    f = _continuous(m, c["nz"], c["base"], _gen(seed), mean_free=c["walls"] == "N")
    if c["kind"] == "mixed":  # a viscous solve's forcing is the velocity over (viscosity x time step)
        f *= -float(c["lam"])
    bc = _boundary_lines(m, c["nz"], np.random.default_rng(seed + 1), c["walls"], c["base"])
    return m, lam2, bk2, f, bc


def _batch_inputs(c, seed):
    g = _gen(seed)
    out = []
    for m, modes, lam in _batch_meshes(c["members"], c["mesh_seed"], c["most"]):
        nz = 1 if modes == 1 else 2 * modes
        out.append((m, np.full(modes, lam), np.arange(modes, dtype=np.float64) ** 2, _continuous(m, nz, 0, g)))
    return out


def _fields(count, m, nz, base, seed):
    g = _gen(seed)
    return [_continuous(m, nz, base, g) for _ in range(count)]


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c, stream=_stream())
    if kind in ("direct", "mixed", "build"):
        m, lam2, bk2, f, bc = _solve_inputs(c, seed)
        s.update(m=m, lam2=lam2, bk2=bk2, mesh=sx.Mesh(m))
        if kind != "build":
            s["S"] = sx.ModalMatrixSys(s["mesh"], base_mode=c["base"], num_modes=len(lam2),
                                       method=sx.DIRECT if kind == "direct" else sx.AUTO, lambda2_modes=lam2,
                                       betak2_modes=bk2)
        if c.get("form") == "host":
            s.update(f=_pinned(f), bc=bc, u=_pinned(torch.zeros_like(f)))
        else:
            s.update(f0=f, f=torch.empty_like(f), u=torch.zeros_like(f), bc=torch.from_numpy(bc).to(DEV))
    elif kind == "batch":
        s["members"] = []
        for m, lam2, bk2, f in _batch_inputs(c, seed):
            S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=len(lam2), method=sx.AUTO, lambda2_modes=lam2,
                                  betak2_modes=bk2)
            s["members"].append((S, f, torch.empty_like(f), torch.zeros_like(f), m))
        s["batch"] = sx.Batch()
    elif kind == "transform":
        m = _mesh(c["nx"], c["ny"], c["np"])
        n = m.nplane + c["pad"]
        x = torch.randn(c["nz"], n, dtype=torch.float64, device=DEV, generator=_gen(seed))
        s.update(m=m, x=x, xf=torch.empty_like(x), xr=torch.empty_like(x))
    elif kind == "forcing":
        m = _mesh(c["nx"], c["ny"], c["np"])
        nadv = 4 if c["scalar"] else 3
        fields = _fields(2 * c["order"] * nadv + 1, m, c["nz"], c["base"], seed)
        z = lambda: torch.zeros_like(fields[0])  # noqa: E731
        s.update(m=m, mesh=sx.Mesh(m), us=fields[:c["order"] * nadv], uf=fields[c["order"] * nadv:-1],
                 p=fields[-1], hat=[z() for _ in range(nadv)], div=z(), out=[z() for _ in range(nadv)], nadv=nadv)
    else:
        m = _mesh(c["nx"], c["ny"], c["np"])
        u, = _fields(1, m, c["nz"], c["base"], seed)
        s.update(m=m, mesh=sx.Mesh(m), u=u, g=[torch.empty_like(u) for _ in range(3)], q=torch.empty_like(u))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

DT, NU, BETA, PRANDTL = 2e-3, 5e-3, 1.0, 0.7


def run(state):
    s, c, st = state, state["case"], state["stream"]
    kind, sp = c["kind"], st.cuda_stream
    if c.get("form") == "host":
        u = s["u"].numpy()
        s["S"].solve_batched_host(s["f"].numpy(), bc=s["bc"], out=u)
        return u
    with torch.cuda.stream(st):
        if kind in ("direct", "mixed", "build"):
            f, u, nz, n = s["f"], s["u"], c["nz"], s["m"].nplane
            f.copy_(s["f0"])  # a solve overwrites its forcing
            ptrs = (u.data_ptr(), f.data_ptr(), s["bc"].data_ptr(), nz, n)
            if kind == "build":
                st.synchronize()  # systems are built on the device's default stream
                S = sx.ModalMatrixSys(s["mesh"], base_mode=c["base"], num_modes=len(s["lam2"]), method=sx.DIRECT,
                                      lambda2_modes=s["lam2"], betak2_modes=s["bk2"])
                S.solve_batched(*ptrs, stream=sp)
                st.synchronize()
                S.close()
            elif kind == "mixed":
                s["S"].solve_batched(*ptrs, precision=sx.MIXED_FP32, max_refine=20, stream=sp)
            elif c["form"] == "plain":
                s["S"].solve_device(*ptrs, stream=sp)
            else:
                s["S"].solve_batched(*ptrs, stream=sp)
            return u
        if kind == "batch":
            for _, f0, f, _, _ in s["members"]:
                f.copy_(f0)
            s["batch"].solve([(S, u.data_ptr(), f.data_ptr(), None, f.shape[0], m.nplane)
                              for S, _, f, u, m in s["members"]], sx.MIXED_FP32, max_refine=30, stream=sp)
            return [u for _, _, _, u, _ in s["members"]]
        if kind == "transform":
            n, np_ = s["x"].shape[1], s["m"].nplane
            s["xf"].copy_(s["x"])  # transforms are in place
            sx.transform_z(s["xf"].data_ptr(), c["nz"], n, np_, 1, stream=sp)
            s["xr"].copy_(s["xf"])
            sx.transform_z(s["xr"].data_ptr(), c["nz"], n, np_, -1, stream=sp)
            return {"forward": s["xf"][:, :np_], "back": s["xr"][:, :np_]}
        nz, n, base = c["nz"], s["m"].nplane, c["base"]
        if kind == "forcing":
            a = s["nadv"]
            lev = lambda v: [[x.data_ptr() for x in v[q * a:(q + 1) * a]] for q in range(c["order"])]  # noqa: E731
            hat, out = [x.data_ptr() for x in s["hat"]], [x.data_ptr() for x in s["out"]]
            sx.wave_prop(lev(s["us"]), lev(s["uf"]), hat, nz * n, DT, stream=sp)
            sx.pressure_forcing(s["mesh"], hat[:3], s["div"].data_ptr(), nz, n, DT, BETA, base, stream=sp)
            sx.project(s["mesh"], hat, s["p"].data_ptr(), out, nz, n, DT, NU, 3, 3, PRANDTL, BETA, base, stream=sp)
            return {"hat": s["hat"], "div": s["div"], "out": s["out"]}
        for d in range(3):
            s["g"][d].copy_(s["u"])  # gradients are in place
            sx.field_gradient(s["mesh"], s["g"][d].data_ptr(), nz, n, d, BETA, base, stream=sp)
        s["q"].copy_(s["g"][0])
        sx.field_smooth(s["mesh"], s["q"].data_ptr(), nz, n, stream=sp)
        return {"grad": s["g"], "smooth": s["q"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it may be off by
# ---------------------------------------------------------------------------

def _skyline(m):
    """Entries of the condensed factor's envelope: from each solve node's first
    coupled solve node to its diagonal."""
    solve = m.btog < m.nsolve
    lo = np.where(solve, m.btog, m.nsolve).min(axis=1)
    first = np.arange(m.nsolve)
    e, a = np.nonzero(solve)
    np.minimum.at(first, m.btog[e, a], lo[e])
    return float((np.arange(m.nsolve) - first + 1).sum()), float(((np.arange(m.nsolve) - first) ** 2.0).sum())


def _solve_work(m, nz, base, build):
    planes = 1 if nz == 1 else nz - (1 if base == 0 else 0)
    modes = max(nz // 2, 1)
    sky, sq = _skyline(m)
    elem = m.nel * float(m.next * m.nint + m.nint ** 2)
    field = 8.0 * planes * m.nplane
    flops = planes * (4 * sky + 2 * (elem + m.nel * m.next * m.nint))
    if build:  # factored and inverted blocks are made, not read: in and out of the solve
        return {"bytes": 2 * field + 8.0 * 6 * m.nplane,
                "flops": flops + modes * (sq + m.nel * (2.0 * m.nint ** 3 + 2.0 * m.next * m.nint * (m.nint + m.next)))}
    return {"bytes": 8.0 * modes * (sky + elem) + 2 * field, "flops": flops}


def _mixed_work(m, nz, base, lam2):
    """In and out, the geometry once, and the operator applied as often as
    conjugate gradients need for twelve digits."""
    planes = 1 if nz == 1 else nz - (1 if base == 0 else 0)
    h = (m.x[:, 0, 1] - m.x[:, 0, 0]) ** 2 + (m.y[:, 0, 1] - m.y[:, 0, 0]) ** 2
    v = (m.x[:, 1, 0] - m.x[:, 0, 0]) ** 2 + (m.y[:, 1, 0] - m.y[:, 0, 0]) ** 2
    kappa = 1.0 + 2.0 / max(min(h.min(), v.min()), 1e-30) / max(lam2, 1e-30)
    its = min(9.0 * math.sqrt(kappa), 1000.0)
    return {"bytes": 8.0 * (2 * planes + 4) * m.nplane, "flops": its * planes * m.nplane * (8.0 * m.np + 20.0)}


def work(case):
    c, kind = case, case["kind"]
    if kind in ("direct", "build"):
        return _solve_work(_case_mesh(c), c["nz"], c["base"], kind == "build")
    if kind == "mixed":
        return _mixed_work(_case_mesh(c), c["nz"], c["base"], float(c["lam"]))
    if kind == "batch":
        w = [_mixed_work(m, 1 if modes == 1 else 2 * modes, 0, lam)
             for m, modes, lam in _batch_meshes(c["members"], c["mesh_seed"], c["most"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    points = float(c["nx"] * c["ny"] * c["np"] ** 2 * c["nz"])
    if kind == "transform":  # read once; the transform and its inverse written
        return {"bytes": 8.0 * 3 * points, "flops": 2 * 2.5 * points * math.log2(c["nz"])}
    if kind == "forcing":  # levels and pressure in; u^, its divergence and u^^ out
        nadv = 4 if c["scalar"] else 3
        return {"bytes": 8.0 * points * (2 * c["order"] * nadv + 1 + 2 * nadv + 1),
                "flops": points * (4 * c["order"] * nadv + 16.0 * c["np"] + 20)}
    return {"bytes": 8.0 * points * 5, "flops": points * (8.0 * c["np"] + 10)}


def tolerance(case):
    # About four times what the present code differs from exact() over draws:
    # the solves by the conditioning of their systems (up to 2e-12), the mixed
    # form also by its stop at a relative residual of 1e-12, the derivatives
    # by cancellation in sums over random fields (3e-13).
    kind = case["kind"]
    if kind in ("direct", "build"):
        return {"rel": 8e-12, "max": 4e-10}
    if kind in ("mixed", "batch"):
        return {"rel": 1e-11, "max": 1e-9}
    if kind == "transform":
        return {"rel": 2.5e-15, "max": 1e-13}
    return {"rel": 1.2e-12, "max": 5e-11}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def _gll(n):
    """Gauss-Lobatto-Legendre points, weights and derivative matrix of n points."""
    N = n - 1

    def legendre(x):
        p0, p1 = np.ones_like(x), x
        for k in range(2, N + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        return p0, p1  # degrees N - 1, N

    x = -np.cos(np.pi * np.arange(n) / N).astype(np.longdouble)
    for _ in range(100):
        a, b = legendre(x)
        x = x - (x * b - a) / (n * b)
    L = legendre(x)[1]
    d = x[:, None] - x[None, :] + np.eye(n)
    D = L[:, None] / L[None, :] / d
    D[np.arange(n), np.arange(n)] = 0.0
    D[0, 0], D[-1, -1] = -N * (N + 1) / 4.0, N * (N + 1) / 4.0
    return (np.asarray(v, dtype=np.float64) for v in (x, 2.0 / (N * (N + 1) * L ** 2), D))


class _Sem:
    """Spectral-element derivatives, mass and Helmholtz operator of a mesh."""

    def __init__(self, m):
        self.m = m
        _, w, D = _gll(m.np)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
        self.D, self.w, x, y = t(D), t(w), t(m.x), t(m.y)
        xr, xs, yr, ys = x @ self.D.T, self.D @ x, y @ self.D.T, self.D @ y
        jac = xr * ys - xs * yr
        self.rx, self.ry, self.sx, self.sy = ys / jac, -xs / jac, -yr / jac, xr / jac
        self.mass = jac * self.w[:, None] * self.w[None, :]
        self.g11 = self.mass * (self.rx ** 2 + self.ry ** 2)
        self.g12 = self.mass * (self.rx * self.sx + self.ry * self.sy)
        self.g22 = self.mass * (self.sx ** 2 + self.sy ** 2)
        self.ids = torch.from_numpy(_node_ids(m)).to(DEV)

    def grad(self, u):
        """d/dx, d/dy of planes (P, nplane), element by element."""
        v = u.reshape(-1, self.m.nel, self.m.np, self.m.np)
        r, s = v @ self.D.T, self.D @ v
        return [(a * r + b * s).reshape(u.shape) for a, b in ((self.rx, self.sx), (self.ry, self.sy))]

    def gather(self, e):
        """Sum of element planes (P, nel, np, np) at the unique nodes."""
        out = torch.zeros(e.shape[0], self.m.n_unique, dtype=torch.float64, device=DEV)
        return out.index_add_(1, self.ids.reshape(-1), e.reshape(e.shape[0], -1))

    def helmholtz(self, v, h, robin):
        e = v[:, self.ids.reshape(-1)].reshape(-1, *self.ids.shape)
        r, s = e @ self.D.T, self.D @ e
        a = (self.g11 * r + self.g12 * s) @ self.D + self.D.T @ (self.g12 * r + self.g22 * s)
        return self.gather(a + h[:, None, None, None] * self.mass * e) + robin * v

    def diagonal(self, h):
        q = self.D ** 2
        d = self.g11 @ q + q.T @ self.g22
        dd = torch.diagonal(self.D)
        d = d + 2.0 * self.g12 * dd[None, :] * dd[:, None]
        return self.gather(d[None] + h[:, None, None, None] * self.mass)


def _side(m, b):
    n = m.np
    k = np.arange(n)
    i, j = [(0 * k, k), (k, 0 * k + n - 1), (0 * k + n - 1, n - 1 - k), (n - 1 - k, 0 * k)][b.side]
    return i, j


def _exact_solve(m, lam2, bk2, f, bc, base):
    """div grad u - (lambda2 + betak2) u = f on every solved plane, with
    essential values, fluxes and mixed conditions from the boundary lines."""
    sem = _Sem(m)
    nz = f.shape[0]
    planes = [p for p in range(nz) if not (p == 1 and nz > 1 and base == 0)]
    h = torch.tensor([lam2[p // 2] + bk2[p // 2] for p in planes], dtype=torch.float64, device=DEV)
    fp = f[planes].reshape(-1, m.nel, m.np, m.np)
    b = -sem.gather(sem.mass * fp)
    robin = torch.zeros(m.n_unique, dtype=torch.float64, device=DEV)
    free = torch.ones(len(planes), m.n_unique, dtype=torch.float64, device=DEV)
    free[:, m.nsolve:m.nglobal] = 0.0
    u = torch.zeros_like(b)
    ids = _node_ids(m)
    mixed = any(x.kind == 2 for x in m.boundaries)
    lines = None if bc is None else torch.as_tensor(bc, device=DEV)[planes]
    for k, x in enumerate(m.boundaries):
        i, j = _side(m, x)
        g = torch.from_numpy(ids[x.elmt, i, j]).to(DEV)
        if x.kind == 0:
            if lines is not None:
                u[:, g] = lines[:, k]
            continue
        px, py = (torch.as_tensor(v[x.elmt][i, j], device=DEV) for v in (m.x, m.y))
        area = torch.hypot(sem.D @ px, sem.D @ py) * sem.w
        if x.kind == 1:
            if lines is not None:
                b.index_add_(1, g, lines[:, k] * area)
        else:
            b.index_add_(1, g, (x.K * x.C * area).expand(len(planes), -1).contiguous())
            robin.index_add_(0, g, x.K * area)
    if m.nsolve == m.nglobal and not mixed:  # no essential node: the singular mode's last node is held at zero
        free[:, m.nsolve - 1] = torch.where(h < 6e-7, 0.0, 1.0)
    pc = free / (sem.diagonal(h) + robin)
    goal = None
    for _ in range(5):  # each pass starts from the true residual
        r = free * (b - sem.helmholtz(u, h, robin))
        rz = (r * pc * r).sum(1)
        start = rz.clone()
        goal = start if goal is None else goal
        d = torch.zeros_like(r)
        z = pc * r
        p = z.clone()
        for it in range(1, 40001):
            q = free * sem.helmholtz(p, h, robin)
            pq = (p * q).sum(1)
            a = torch.where(pq > 0, rz / pq, torch.zeros_like(pq))
            d += a[:, None] * p
            r -= a[:, None] * q
            z = pc * r
            new = (r * z).sum(1)
            p = z + torch.where(rz > 0, new / rz, torch.zeros_like(rz))[:, None] * p
            rz = new
            if it % 50 == 0 and bool((rz <= 1e-22 * start).all()):
                break
        u += d
        if bool((start <= 1e-27 * goal).all()):
            break
    out = torch.zeros(nz, m.nplane, dtype=torch.float64, device=DEV)
    out[planes] = u[:, sem.ids.reshape(-1)]
    return out


def _exact_size(m, nz, lam):
    """Rough seconds of _exact_solve."""
    its = 25.0 * m.np * math.sqrt(m.nel) if lam in ("zero", "spread", "one") else 1500.0
    return its * (3e-4 + nz * m.nplane * 1.2e-10)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("direct", "mixed", "build"):
        m, lam2, bk2, f, bc = _solve_inputs(c, seed)
        if _exact_size(m, c["nz"], c["lam"]) > 15.0:
            return None
        u = _exact_solve(m, lam2, bk2, f, bc, c["base"])
        return u.cpu().numpy() if c.get("form") == "host" else u
    if kind == "batch":
        return [_exact_solve(m, lam2, bk2, f, None, 0) for m, lam2, bk2, f in _batch_inputs(c, seed)]
    if kind == "transform":
        m = _mesh(c["nx"], c["ny"], c["np"])
        nz = c["nz"]
        x = torch.randn(nz, m.nplane + c["pad"], dtype=torch.float64, device=DEV, generator=_gen(seed))[:, :m.nplane]
        out = torch.empty_like(x)
        for p in range(0, m.nplane, 1 << 16):  # a direct transform, the angles reduced exactly
            q = slice(p, min(m.nplane, p + (1 << 16)))
            jk = (torch.arange(nz // 2 + 1, device=DEV)[:, None] * torch.arange(nz, device=DEV)[None, :]) % nz
            ang = jk.double() * (2.0 * math.pi / nz)
            re, im = torch.cos(ang) @ x[:, q] / nz, -torch.sin(ang) @ x[:, q] / nz
            out[0, q], out[1, q] = re[0], re[nz // 2]
            out[2::2, q], out[3::2, q] = re[1:nz // 2], im[1:nz // 2]
        return {"forward": out, "back": x}
    m = _mesh(c["nx"], c["ny"], c["np"])
    sem = _Sem(m)
    nz, base = c["nz"], c["base"]
    k = BETA * (torch.arange(nz, device=DEV) // 2 + base).double()
    if base == 0:
        k[:2] = 0.0

    def dz(v):
        w = v.reshape(nz // 2, 2, -1)
        return torch.stack((-k[::2, None] * w[:, 1], k[::2, None] * w[:, 0]), 1).reshape(v.shape)

    if kind == "fieldops":
        u, = _fields(1, m, nz, base, seed)
        g = sem.grad(u) + [dz(u)]
        e = g[0].reshape(nz, m.nel, m.np, m.np)
        avg = sem.gather(sem.mass * e) / sem.gather(sem.mass[None])
        return {"grad": g, "smooth": avg[:, sem.ids.reshape(-1)]}
    a = 4 if c["scalar"] else 3
    fields = _fields(2 * c["order"] * a + 1, m, nz, base, seed)
    us, uf, p = fields[:c["order"] * a], fields[c["order"] * a:-1], fields[-1]
    stiff = {1: [1.0], 2: [2.0, -0.5], 3: [3.0, -1.5, 1.0 / 3.0]}[c["order"]]
    extra = {1: [1.0], 2: [2.0, -1.0], 3: [3.0, -3.0, 1.0]}[c["order"]]
    hat = [sum(stiff[q] * us[q * a + i] + DT * extra[q] * uf[q * a + i] for q in range(c["order"]))
           for i in range(a)]
    div = (sem.grad(hat[0])[0] + sem.grad(hat[1])[1] + dz(hat[2])) / DT
    gp = sem.grad(p) + [dz(p)]
    out = [-hat[i] / (DT * NU) + gp[i] / NU for i in range(3)]
    if c["scalar"]:
        out.append(-hat[3] / (DT * NU) * PRANDTL)
    return {"hat": hat, "div": div, "out": out}
