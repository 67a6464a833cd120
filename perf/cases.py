"""The work that a user of this framework has it do, as timed cases.

Every case goes through the public entry points (the C ABI through
dvmpp_b200.native): the velocity sums a host program calls, the sheet solve,
whole steps of one simulation and of a batch, merging, remeshing, probing and
creating simulations.  Sizes are those of the repository's workloads
(dvmpp_b200/workloads.py, bench.py, tests/test_gpu_configs.py) and smaller ones.

A simulation in single precision (native.F32) carries single precision in
its velocities, sheet strengths and circulations, so a program that chose it
keeps what it reads back as float32; one in double precision keeps float64.
"""
import ctypes as C
import math

import numpy as np
import torch

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

RPI2 = 1.0 / (2.0 * math.pi)
_ctx = None


def _context():
    """The program's one context."""
    global _ctx
    if _ctx is None:
        _ctx = N.Context(0)
    return _ctx


# ---- the cases -----------------------------------------------------------------------------


def listed():
    return [
        # a host program's VelocityKernel plugin call on a young wake: host arrays in and out
        dict(name="velocity host f32 5k", kind="self_host", n=5003, prec="f32"),
        # the standalone N-body workload: a developed wake resident on the device
        dict(name="velocity f32 2^20", kind="self", n=1 << 20, prec="f32"),
        # the same call in double precision, at the size of a run that is checked against FP64
        dict(name="velocity f64 40k", kind="self", n=40009, prec="f64"),
        # the standalone workload's collocation targets (computeInducedAt)
        dict(name="at targets f32 256 x 2^20", kind="at", ns=1 << 20, nt=256, prec="f32"),
        # velocities at a grid of probe points, in double precision
        dict(name="probe f64 3k x 60k", kind="probe", ns=60013, nt=3001, np=200, prec="f64"),
        # right-hand side, solve and sheet velocity of a finely panelled ellipse
        dict(name="sheet f32 1024 x 131k", kind="sheet", n=131072, np=1024, prec="f32"),
        # the cylinder run in double precision with a host random stream: many short steps
        dict(name="cylinder f64 20 steps", kind="steps", n=2011, np=128, prec="f64", rk3=False,
             delete=False, inject=True, steps=20),
        # one RK3 step of the ellipse with a large wake, blobs inside the body deleted
        dict(name="ellipse f32 RK3 250k", kind="steps", n=250007, np=1024, prec="f32", rk3=True,
             delete=True, inject=False, steps=1),
        # the batched steps of a server's admitted simulations, uneven in size
        dict(name="batch f32 12 sims", kind="batch", sims=12, n=30000, np=256, prec="f32", steps=2),
        # vortex merging between steps
        dict(name="merge 20k", kind="merge", n=20011),
        # remeshing a large wake onto a background mesh
        dict(name="remesh 300k", kind="remesh", n=300007, kernel=0, cells=400),
        # admission of a group of requests: set-up, factorisation and first solve
        dict(name="create 4 bodies", kind="create", bodies=4, np=512),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["self_host", "self", "self", "at", "probe", "sheet", "steps", "steps",
                       "batch", "merge", "remesh", "create"])
    prec = rng.choice(["f32", "f64"])
    if kind == "self_host":
        return dict(kind=kind, n=_logint(rng, 500, 50000), prec=prec)
    if kind == "self":
        return dict(kind=kind, n=_logint(rng, 1000, 900000 if prec == "f32" else 100000),
                    prec=prec)
    if kind == "at":
        return dict(kind=kind, ns=_logint(rng, 10000, 1 << 20), nt=_logint(rng, 64, 4096), prec=prec)
    if kind == "probe":
        return dict(kind=kind, ns=_logint(rng, 5000, 150000), nt=_logint(rng, 100, 10000),
                    np=rng.randrange(64, 513), prec=prec)
    if kind == "sheet":
        return dict(kind=kind, n=_logint(rng, 5000, 200000), np=rng.randrange(64, 1025), prec=prec)
    if kind == "steps":
        big = 300000 if prec == "f32" else 40000
        return dict(kind=kind, n=_logint(rng, 1000, big), np=_logint(rng, 64, 512), prec=prec,
                    rk3=rng.random() < 0.5, delete=rng.random() < 0.5, inject=rng.random() < 0.5,
                    steps=1)
    if kind == "batch":
        return dict(kind=kind, sims=rng.randrange(3, 17), n=_logint(rng, 3000, 40000),
                    np=rng.randrange(96, 257), prec="f32", steps=rng.randrange(1, 3))
    if kind == "merge":
        return dict(kind=kind, n=_logint(rng, 1000, 40000))
    if kind == "remesh":
        return dict(kind=kind, n=_logint(rng, 5000, 500000), kernel=rng.randrange(0, 3),
                    cells=rng.randrange(60, 601))
    return dict(kind="create", bodies=rng.randrange(1, 7), np=rng.randrange(64, 513))


# ---- inputs --------------------------------------------------------------------------------


def _pin(a):
    """A pinned copy of a host array, as a program that exchanges it each step keeps it."""
    a = np.ascontiguousarray(a)
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:0]).dtype, pin_memory=torch.cuda.is_available())
    out = t.numpy()
    out[...] = a
    return out


def _zeros(n):
    """A pinned buffer that results are read into; the part past a count stays 0."""
    return torch.zeros(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _wake(n, seed, sigma, scale=1.0):
    """The repository's wake, its circulations those of a released sheet."""
    return W.wake(n, seed, sigma, scale)


def _between(lo, hi, k):
    """The k-th of a case's uneven sizes: hi first, then spread over [lo, hi] logarithmically."""
    return int(round(hi * (lo / hi) ** (k * 0.618034 % 1.0)))


def _body(case, k, rng):
    """The k-th body of a case: circle, ellipse at incidence or rounded square."""
    npan = _between(64, case["np"], k)
    kind = k % 3
    if kind == 0:
        return W.circle(npan)
    if kind == 1:
        return W.ellipse(npan, 0.5, 0.5 / float(rng.uniform(1.0, 4.0)), float(rng.uniform(0.0, 20.0)))
    return W.rounded_square(npan)


def _prec(case):
    return N.F64 if case["prec"] == "f64" else N.F32


def _params(case, seed, capacity, rng_capacity=1):
    fine = case["np"] >= 512  # the ellipse workload's time step and stream, else the cylinder's
    return N.Params(nu=1e-3, dt=0.002 if fine else 0.005, ux=1.0 if fine else 3.0,
                    scheme=N.RK3 if case.get("rk3") else N.EULER,
                    surface_cross=N.DELETE if case.get("delete") else N.REFLECT,
                    rng=N.RNG_INJECT if case.get("inject") else N.RNG_PHILOX,
                    precision=_prec(case), seed=seed + 1, capacity=capacity,
                    rng_capacity=rng_capacity)


def _one_body(case):
    return W.ellipse(case["np"], 0.5, 0.25, 20.0) if case["np"] >= 512 else W.circle(case["np"])


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    st = {"case": case, "ctx": _context()}
    if kind in ("self", "self_host", "at"):
        n = case.get("n") or case["ns"]
        sigma = W.core_size(*W.ellipse(1024, 0.5, 0.25, 20.0)) if n > 100000 else 0.0818804
        host = _wake(n, seed, sigma)
        if kind == "self_host":
            st["host"] = host
            return st
        st["src"] = [torch.from_numpy(a).cuda() for a in host]
        if kind == "at":
            t = W.collocation_circle(case["nt"], 0.5 + 0.01 * float(rng.uniform()))
            st["tgt"] = [torch.from_numpy(a).cuda() for a in t]
        m = n if kind == "self" else case["nt"]
        st["out"] = [torch.empty(m, dtype=torch.float64, device="cuda") for _ in range(2)]
        return st
    if kind == "probe":
        bx, bz = _one_body(case)
        sim = st["ctx"].sim(_params(case, seed, case["ns"]), bx, bz)
        sim.set_blobs(*_wake(case["ns"], seed, W.core_size(bx, bz)))
        th = 2.0 * np.pi * np.arange(case["np"]) / case["np"]
        st["gamma"] = 2.0 * np.sin(th) + 0.1 * rng.normal(size=case["np"])
        sim.set_gamma(st["gamma"])
        m = int(math.ceil(math.sqrt(case["nt"])))
        gx, gz = np.meshgrid(np.linspace(-1.5, 6.0, m), np.linspace(-1.5, 1.5, m))
        st["px"] = (gx + 0.01 * rng.uniform()).ravel()[:case["nt"]].copy()
        st["pz"] = (gz + 0.01 * rng.uniform()).ravel()[:case["nt"]].copy()
        st["sim"] = sim
        return st
    if kind == "sheet":
        bx, bz = _one_body(case)
        sim = st["ctx"].sim(_params(case, seed, case["n"]), bx, bz)
        sim.set_blobs(*_wake(case["n"], seed, W.core_size(bx, bz)))
        st["sim"], st["out"] = sim, [_zeros(case["n"]) for _ in range(2)]
        return st
    if kind == "steps":
        bx, bz = _one_body(case)
        room = case["n"] + 4 * case["np"] * case["steps"]
        draws = 2 * room * case["steps"] + 4 * case["np"] * case["steps"] if case["inject"] else 1
        sim = st["ctx"].sim(_params(case, seed, room, draws), bx, bz)
        st["blobs"] = [_pin(a) for a in _wake(case["n"], seed, W.core_size(bx, bz))]
        if case["inject"]:
            st["uniforms"] = _pin(rng.uniform(1e-12, 1.0, draws))
        st["sim"], st["out"] = sim, [_zeros(room) for _ in range(3)]
        return st
    if kind == "batch":
        sims, blobs, outs = [], [], [[], [], []]
        for k in range(case["sims"]):
            bx, bz = _body(case, k, rng)
            n = _between(1000, case["n"], k)
            room = n + 4 * (bx.size - 1) * case["steps"]
            sims.append(st["ctx"].sim(_params(dict(case, np=bx.size - 1), seed + k, room), bx, bz))
            blobs.append([_pin(a) for a in _wake(n, seed * 100 + k, W.core_size(bx, bz),
                                                 W.body_radius(bx, bz) / 0.5)])
            for o in outs:
                o.append(_zeros(room))
        st.update(sims=sims, blobs=blobs, out=outs)
        return st
    if kind == "merge":
        x, z, g, s = _wake(case["n"], seed, 0.0818804)
        st["blobs"] = [x, z, g, s] + list(rng.normal(0.0, 1.0, (4, case["n"])))
        st["out"] = [np.empty(case["n"]) for _ in range(8)] + [np.empty(case["n"], dtype=np.uint32)]
        return st
    if kind == "remesh":
        st["mesh"] = _mesh(case)
        nx, nz = N.remesh_grid(st["mesh"])
        st["host"] = np.ascontiguousarray(np.stack(_wake(case["n"], seed, 0.0169), axis=1))
        st["out"] = np.zeros((nx * nz + case["n"], 4))
        return st
    if kind == "create":
        st["bodies"] = [_body(case, k, rng) for k in range(case["bodies"])]
        st["params"] = [_params(dict(case, prec="f64", np=b[0].size - 1), seed + k, 4096)
                        for k, b in enumerate(st["bodies"])]
        return st
    raise ValueError(kind)


def _mesh(case):
    """A mesh over the near wake, as the remesh options describe one; blobs outside stay."""
    nx = case["cells"]
    dx = 16.0 / nx
    return N.RemeshParams(xmin=-2.0, xmax=14.0, zmin=-3.0, zmax=3.0, dx=dx, dz=dx, sigma=dx,
                          circ_threshold=1e-7, kernel=case["kernel"])


# ---- one pass ------------------------------------------------------------------------------


def _ok(rc):
    if rc != N.OK:
        raise N.DvmError(rc, N.load().dvm_last_error().decode())


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _kept(case, *arrays):
    """What the program keeps: single precision where it chose it."""
    if case["prec"] == "f64":
        return arrays
    return tuple(a.astype(np.float32) if isinstance(a, np.ndarray) else a.float() for a in arrays)


def _load(sim, blobs):
    """A simulation's start: its blobs and step counter."""
    sim.set_blobs(*blobs)
    _ok(sim.lib.dvm_sim_set_step(sim.h, 0))


def run(state):
    case, ctx, kind = state["case"], state["ctx"], state["case"]["kind"]
    lib = ctx.lib
    if kind == "self_host":
        return _kept(case, *ctx.biot_savart_self(*state["host"], _prec(case)))
    if kind == "self":
        u, w = state["out"]
        _ok(lib.dvm_biot_savart_self_device(ctx.h, *map(_ptr, state["src"]), case["n"], _ptr(u),
                                            _ptr(w), _prec(case)))
        ctx.sync()  # the context's stream is not torch's
        return _kept(case, u, w)
    if kind == "at":
        u, w = state["out"]
        _ok(lib.dvm_biot_savart_at_device(ctx.h, *map(_ptr, state["src"]), case["ns"],
                                          *map(_ptr, state["tgt"]), case["nt"], _ptr(u), _ptr(w),
                                          _prec(case), 1))
        ctx.sync()
        return _kept(case, u, w)
    if kind == "probe":
        return _kept(case, *state["sim"].probe(state["px"], state["pz"]))
    if kind == "sheet":
        sim = state["sim"]
        sim.phase(N.PHASE_SOLVE)
        sim.phase(N.PHASE_SHEETBC)
        uvs, wvs = state["out"]
        m = C.c_uint64()
        p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in state["out"]]
        _ok(lib.dvm_sim_get_blobs(sim.h, case["n"], C.byref(m), None, None, None, None, None, None,
                                  p[0], p[1], None))
        return _kept(case, sim.gamma(), uvs, wvs)
    if kind == "steps":
        sim = state["sim"]
        _load(sim, state["blobs"])
        if case["inject"]:
            _ok(lib.dvm_sim_clear_uniforms(sim.h))
            sim.push_uniforms(state["uniforms"])
        sim.step(case["steps"])
        sim.check()
        n = sim.get_state_into(*state["out"])  # what a written step holds
        return _kept(case, *state["out"], sim.gamma(), np.array(sim.loads())) + (n,)
    if kind == "batch":
        sims = state["sims"]
        for s, b in zip(sims, state["blobs"]):
            _load(s, b)
        ctx.step_batch(sims, case["steps"])
        if any(ctx.batch_status(sims)):
            raise RuntimeError("a simulation failed")
        counts, loads = ctx.batch_get_state(sims, *state["out"])
        return _kept(case, *[np.concatenate(o) for o in state["out"]], loads) + (np.array(counts),)
    if kind == "merge":
        out, m, count = state["out"], C.c_uint64(), C.c_uint64()
        for o, a in zip(out, state["blobs"]):
            np.copyto(o, a)
        out[8][:] = np.arange(case["n"], dtype=np.uint32)
        dp, up = C.POINTER(C.c_double), C.POINTER(C.c_uint32)
        _ok(lib.dvm_merge_blobs(ctx.h, *[o.ctypes.data_as(dp) for o in out[:8]],
                                out[8].ctypes.data_as(up), case["n"], 2e-6, C.byref(m),
                                C.byref(count)))
        return out, m.value, count.value
    if kind == "remesh":
        m, out = C.c_uint64(), state["out"]
        _ok(lib.dvm_remesh(ctx.h, C.c_void_p(state["host"].ctypes.data), case["n"],
                           C.byref(state["mesh"]), C.c_void_p(out.ctypes.data), out.shape[0],
                           C.byref(m)))
        return out, m.value
    sims = ctx.sims(state["params"], state["bodies"])
    out = []
    for s in sims:
        s.phase(N.PHASE_SOLVE)
        out.append((s.influence(), s.gamma()))
        s.close()
    return out


# ---- the least work ------------------------------------------------------------------------


def work(case):
    """Bytes: each input read once, each output written once.  Flops: what no
    method avoids, i.e. a few operations per input and output value; a velocity
    sum can be had without visiting every pair, so pairs are not counted."""
    kind = case["kind"]
    if kind in ("self", "self_host"):
        return {"bytes": 48.0 * case["n"], "flops": 100.0 * case["n"]}
    if kind == "at":
        return {"bytes": 32.0 * case["ns"] + 32.0 * case["nt"], "flops": 20.0 * case["ns"] + 100.0 * case["nt"]}
    if kind == "probe":
        return {"bytes": 32.0 * case["ns"] + 48.0 * case["nt"] + 80.0 * case["np"],
                "flops": 20.0 * case["ns"] + 100.0 * case["nt"]}
    if kind == "sheet":
        return {"bytes": 48.0 * case["n"] + 16.0 * case["np"] ** 2,
                "flops": 100.0 * case["n"] + 6.0 * case["np"] ** 2}
    if kind == "steps":
        stages = case["steps"] * (3 if case["rk3"] else 1)
        return {"bytes": stages * (64.0 * case["n"] + 16.0 * case["np"] ** 2),
                "flops": stages * (250.0 * case["n"] + 6.0 * case["np"] ** 2)}
    if kind == "batch":
        n = case["sims"] * 0.4 * case["n"]
        return {"bytes": 64.0 * n * case["steps"], "flops": 250.0 * n * case["steps"]}
    if kind == "merge":
        return {"bytes": 128.0 * case["n"], "flops": 20.0 * case["n"]}
    if kind == "remesh":
        nodes = 0.375 * case["cells"] ** 2
        return {"bytes": 32.0 * (2 * case["n"] + nodes), "flops": 200.0 * case["n"]}
    m = case["np"] * 0.6
    return {"bytes": case["bodies"] * 16.0 * m * m, "flops": case["bodies"] * 4.0 * m ** 3}


# ---- the same in 64 bits, by plain torch and numpy -------------------------------------------


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_dev())


def _induced(sx, sz, sg, ss, tx, tz, skip):
    """Velocities at targets by the direct sum; pairs with r^2 <= skip are left out."""
    sx, sz, sg, ss, tx, tz = map(_t, (sx, sz, sg, ss, tx, tz))
    s2 = ss * ss
    u, w = torch.empty_like(tx), torch.empty_like(tx)
    block = max(1, (1 << 23) // max(1, sx.numel()))
    for i in range(0, tx.numel(), block):
        dx = tx[i:i + block, None] - sx
        dz = tz[i:i + block, None] - sz
        r2 = dx * dx + dz * dz
        k = torch.where(r2 < 10.0 * s2, -torch.expm1(-r2 / s2), torch.ones((), dtype=r2.dtype, device=r2.device)) / r2
        k = torch.where(r2 > skip, k, torch.zeros((), dtype=r2.dtype, device=r2.device)) * sg
        u[i:i + block] = -(k * dz).sum(1)
        w[i:i + block] = (k * dx).sum(1)
    return u * RPI2, w * RPI2


def _panels(bx, bz):
    dx, dz = np.diff(bx), np.diff(bz)
    ds = np.hypot(dx, dz)
    return dict(xc=0.5 * (bx[:-1] + bx[1:]), zc=0.5 * (bz[:-1] + bz[1:]), ds=ds,
                th=np.arctan2(dz, dx), nx=dz / ds, nz=-dx / ds, x0=bx[:-1], z0=bz[:-1])


def _sheet_at(pan, gamma, tx, tz):
    """The panels' velocity at points (offsets from the collocation points)."""
    xc, zc, ds, th, g0 = map(_t, (pan["xc"], pan["zc"], pan["ds"], pan["th"], gamma))
    g1 = torch.roll(g0, -1)
    ct, st, c2, s2 = torch.cos(th), torch.sin(th), torch.cos(-2 * th), torch.sin(-2 * th)
    tx, tz = _t(tx), _t(tz)
    u, w = torch.empty_like(tx), torch.empty_like(tx)
    block = max(1, (1 << 23) // xc.numel())
    for i in range(0, tx.numel(), block):
        dx, dz = tx[i:i + block, None] - xc, tz[i:i + block, None] - zc
        c1 = -dx * ct - dz * st
        r2 = dx * dx + dz * dz
        c5 = dx * st - dz * ct
        c6 = torch.log1p(ds * (ds + 2 * c1) / r2)
        c7 = torch.atan2(c5 * ds, r2 + c1 * ds)
        c8, c9 = dx * s2 + dz * c2, dx * c2 - dz * s2
        qx = -st + 0.5 * c8 * c6 / ds + (c1 * ct + c5 * st) * c7 / ds
        px = -0.5 * c6 * st - c7 * ct - qx
        qz = ct + 0.5 * c9 * c6 / ds + (c1 * st - c5 * ct) * c7 / ds
        pz = 0.5 * c6 * ct - c7 * st - qz
        u[i:i + block] = (px * g0 + qx * g1).sum(1)
        w[i:i + block] = (pz * g0 + qz * g1).sum(1)
    return u * RPI2, w * RPI2


def _influence(pan):
    """The influence matrix with its closing row (total circulation)."""
    xc, zc, ds, th, x0, z0 = map(_t, (pan["xc"], pan["zc"], pan["ds"], pan["th"], pan["x0"], pan["z0"]))
    n = xc.numel()
    dx, dz = xc[:, None] - x0, zc[:, None] - z0
    ti, tj = th[:, None], th[None, :]
    c1 = -dx * torch.cos(tj) - dz * torch.sin(tj)
    r2 = dx * dx + dz * dz
    c3, c4 = torch.sin(ti - tj), torch.cos(ti - tj)
    c5 = dx * torch.sin(tj) - dz * torch.cos(tj)
    c6 = torch.log(1.0 + ds * ((ds + 2.0 * c1) / r2))
    c7 = torch.atan2(c5 * ds, r2 + c1 * ds)
    a2 = ti - 2.0 * tj
    c9 = dx * torch.cos(a2) - dz * torch.sin(a2)
    q = c4 + 0.5 * c9 * c6 / ds - (c1 * c3 + c4 * c5) * c7 / ds
    p = 0.5 * c4 * c6 + c3 * c7 - q
    eye = torch.eye(n, dtype=torch.bool, device=q.device)
    p, q = p.masked_fill(eye, -1.0), q.masked_fill(eye, 1.0)
    return torch.cat([-RPI2 * (p + torch.roll(q, 1, 1)), ds[None, :]], 0)


def _solve(A, b):
    q, r = torch.linalg.qr(A)
    g = torch.linalg.solve_triangular(r, q.T @ b[:, None], upper=True)
    res = b[:, None] - A @ g
    return (g + torch.linalg.solve_triangular(r, q.T @ res, upper=True))[:, 0]


def _remesh(host, mesh):
    """Remeshing of the wake, node sums by plain numpy."""
    x, z, g, s = host.T
    nx, nz = N.remesh_grid(mesh)
    kern = mesh.kernel
    S = 2 if kern == N.REMESH_M4PRIME else 3

    def weight(r):
        r = np.abs(r)
        if kern == N.REMESH_M4PRIME:
            return np.where(r < 1, 1 - 2.5 * r * r + 1.5 * r ** 3, np.where(r < 2, 0.5 * (2 - r) ** 2 * (1 - r), 0.0))
        if kern == N.REMESH_M6:
            p5 = lambda v: np.maximum(v, 0.0) ** 5  # noqa: E731
            return np.where(r < 3, (p5(3 - r) - 6 * p5(2 - r) + 15 * p5(1 - r)) / 120.0, 0.0)
        return np.where(r < 3, np.exp(-0.5 * r * r) / math.sqrt(2 * math.pi), 0.0)

    xi, ze = (x - mesh.xmin) / mesh.dx, (z - mesh.zmin) / mesh.dz
    fx, fz = np.floor(xi).astype(np.int64), np.floor(ze).astype(np.int64)
    inside = (fx - (S - 1) >= 0) & (fx + S <= nx - 1) & (fz - (S - 1) >= 0) & (fz + S <= nz - 1)
    a, b, fa, fb, ga = xi[inside], ze[inside], fx[inside], fz[inside], g[inside].copy()
    offs = range(-(S - 1), S + 1)
    wx, wz = [weight(a - (fa + o)) for o in offs], [weight(b - (fb + o)) for o in offs]
    if kern == N.REMESH_GAUSSIAN:
        ga = ga / (sum(wx) * sum(wz))
    node = np.zeros(nx * nz)
    for j, oz in enumerate(offs):
        for i, ox in enumerate(offs):
            node += np.bincount((fb + oz) * nx + fa + ox, weights=wx[i] * wz[j] * ga, minlength=nx * nz)
    keep = np.flatnonzero(np.abs(node) > mesh.circ_threshold)
    out = ~inside
    new = np.stack([mesh.xmin + (keep % nx) * mesh.dx, mesh.zmin + (keep // nx) * mesh.dz,
                    node[keep], np.full(keep.size, mesh.sigma)], axis=1)
    m = keep.size + int(out.sum())
    return np.concatenate([new, host[out], np.zeros((nx * nz + x.size - m, 4))]), m


def exact(case, seed):
    kind = case["kind"]
    if kind in ("steps", "batch", "merge"):
        return None  # a random walk's and a greedy merge's state has no closed value
    if kind == "self" and case["n"] > 400000:
        return None  # the direct sum takes too long
    st = prepare(case, seed)
    if kind in ("self", "self_host"):
        x, z, g, s = [a.cpu().numpy() for a in st["src"]] if kind == "self" else st["host"]
        return _induced(x, z, g, s, x, z, 0.0)
    if kind == "at":
        return _induced(*[a.cpu().numpy() for a in st["src"] + st["tgt"]], 1e-15)
    if kind == "probe":
        d = st["sim"].blobs()
        pan = _panels(*_one_body(case))
        u, w = _induced(d["x"], d["z"], d["circ"], d["sigma"], st["px"], st["pz"], 1e-15)
        us, ws = _sheet_at(pan, st["gamma"], st["px"], st["pz"])
        p = st["sim"].params
        return u + us + p.ux, w + ws + p.uz, us, ws
    if kind == "sheet":
        d, p = st["sim"].blobs(), st["sim"].params
        pan = _panels(*_one_body(case))
        u, w = _induced(d["x"], d["z"], d["circ"], d["sigma"], pan["xc"], pan["zc"], -1.0)
        b = torch.cat([(u + p.ux) * _t(pan["nx"]) + (w + p.uz) * _t(pan["nz"]), -_t(d["circ"]).sum()[None]])
        g = _solve(_influence(pan), b)
        return (g,) + _sheet_at(pan, g.cpu().numpy(), d["x"], d["z"])
    if kind == "remesh":
        return _remesh(st["host"], st["mesh"])
    out = []
    for (bx, bz), p in zip(st["bodies"], st["params"]):
        pan = _panels(bx, bz)
        A = _influence(pan)
        b = torch.cat([p.ux * _t(pan["nx"]) + p.uz * _t(pan["nz"]), torch.zeros(1, dtype=torch.float64, device=A.device)])
        out.append((A, _solve(A, b)))
    return out
