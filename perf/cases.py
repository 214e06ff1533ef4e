"""Performance cases of the solver: whole calls through the public Python
interface, over the range of sizes and options that it is used with.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (a device-resident state and a context), `run` makes one pass,
`work` says what a pass cannot do without, and `exact` computes the same
outputs in plain 64-bit torch."""
import math

import torch

from amrex_euler_allmach_explicit_imex_b200 import api, autograd, workloads
from amrex_euler_allmach_explicit_imex_b200.config import read_config

GAMMA = 1.4
PICARD = 4  # pressure solves of an IMEX step


def listed():
    return [
        # The reference driver's loop on its shock-tube grid: dt, step and
        # diagnostics one call at a time; launches and host waits are the cost.
        {"name": "loop_sod_400x4", "kind": "loop", "problem": "sod", "nx": 400, "ny": 4, "riemann": "hllc",
         "limiter": "minmod", "steps": 8},
        # The same grid through the device-resident time loop (a convergence
        # study runs hundreds of such short steps).
        {"name": "run_sod_400x4", "kind": "run", "problem": "sod", "nx": 400, "ny": 4, "riemann": "hllc",
         "limiter": "minmod", "steps": 256, "arith": "fast"},
        # Low-Mach vortex with the all-Mach flux: a grid that does not fill the GPU.
        {"name": "run_gresho_256_hllcp", "kind": "run", "problem": "gresho", "nx": 256, "ny": 256,
         "riemann": "xie_am_hllc_p", "limiter": "minmod", "mach": 0.01, "steps": 64, "arith": "fast"},
        # 2-D Riemann problem on an odd grid with the other limiter and flux.
        {"name": "run_quadrant_1021x509", "kind": "run", "problem": "quadrant", "nx": 1021, "ny": 509,
         "riemann": "lowmach_hllc", "limiter": "vanleer", "steps": 32, "arith": "fast"},
        # The headline workload: the shock-density bubble.
        {"name": "run_bubble_2560x640", "kind": "run", "problem": "bubble", "nx": 2560, "ny": 640, "riemann": "hllc",
         "limiter": "minmod", "steps": 32, "arith": "fast"},
        # Bit-exact arithmetic: runs that are compared with the reference's own output.
        {"name": "run_bubble_1280x320_exact", "kind": "run", "problem": "bubble", "nx": 1280, "ny": 320,
         "riemann": "hllc", "limiter": "minmod", "steps": 32, "arith": "exact"},
        # A step called by a driver that keeps its state in (pinned) host memory.
        {"name": "host_bubble_2560x640", "kind": "host", "problem": "bubble", "nx": 2560, "ny": 640,
         "riemann": "hllc", "limiter": "minmod", "steps": 1},
        # A parameter sweep: 64 Riemann problems on uneven grids, states read back at the end.
        {"name": "batch_64", "kind": "batch", "nsolve": 64, "scale": 1.0, "riemann": "hllc", "steps": 240},
        # Gradient of a rollout with respect to its initial state, forward and backward.
        {"name": "adjoint_blob_256", "kind": "adjoint", "problem": "blob", "nx": 256, "ny": 256, "riemann": "hllc",
         "limiter": "minmod", "steps": 20},
        # Pressure-implicit step of the low-Mach vortex, FP64 Krylov basis (about 36 iterations a solve;
        # at M = 0.01 some perturbed states end a hair above the solver's tolerance and leave no new state).
        {"name": "imex_gresho_256", "kind": "imex", "problem": "gresho", "nx": 256, "ny": 256, "mach": 0.02,
         "precision": "fp64"},
        # The same at a size whose Krylov basis streams from HBM, stored in FP32.
        {"name": "imex_gresho_768_mixed", "kind": "imex", "problem": "gresho", "nx": 768, "ny": 768, "mach": 0.02,
         "precision": "mixed"},
        # Pressure-implicit step of the bubble: short solves on a large grid.
        {"name": "imex_bubble_2560x640", "kind": "imex", "problem": "bubble", "nx": 2560, "ny": 640,
         "precision": "fp64"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["loop", "run", "run", "run", "host", "batch", "adjoint", "imex", "imex"])
    if kind == "batch":
        return {"kind": "batch", "nsolve": rng.randint(3, 48), "scale": rng.uniform(0.3, 1.0),
                "riemann": rng.choice(["hllc", "lowmach_hllc", "xie_am_hllc_p"]), "steps": rng.randint(24, 160)}
    limiter = rng.choice(["minmod", "mc", "vanleer"])
    if kind == "imex":
        if rng.random() < 0.5:
            nx = size(48, 800)
            return {"kind": "imex", "problem": "gresho", "nx": nx, "ny": nx + rng.randint(0, 3),
                    "mach": rng.choice([0.1, 0.03, 0.02]), "precision": rng.choice(["fp64", "mixed"])}
        return {"kind": "imex", "problem": "bubble", "nx": size(160, 2560), "ny": size(40, 640),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "adjoint":
        return {"kind": "adjoint", "problem": "blob", "nx": size(32, 320), "ny": size(32, 320),
                "riemann": rng.choice(["hllc", "lowmach_hllc", "rusanov"]), "limiter": limiter,
                "steps": rng.randint(2, 20)}
    problem = rng.choice(["sod", "gresho", "quadrant", "bubble"])
    riemann = rng.choice(["hllc", "xie_am_hllc_p"] if problem == "bubble" else
                         ["hllc", "lowmach_hllc", "xie_am_hllc_p", "rusanov"])
    c = {"kind": kind, "problem": problem, "riemann": riemann, "limiter": limiter}
    if problem == "sod":
        c["nx"], c["ny"] = size(100, 1600), rng.randint(4, 8)
    elif problem == "bubble":
        c["nx"], c["ny"] = size(160, 2560), size(40, 640)
    else:
        c["nx"], c["ny"] = size(48, 1024), size(48, 1024)
    if problem == "gresho":
        c["mach"] = rng.choice([0.1, 0.01])
    c["steps"] = {"loop": rng.randint(2, 16), "run": rng.randint(8, 64), "host": 1}[kind]
    if kind == "run":
        c["arith"] = rng.choice(["fast", "fast", "exact"])
    return c


# ---- configurations and initial states ---------------------------------------------


def _kv(c):
    p = c["problem"]
    kv = {"amr.n_cell": "%d %d" % (c["nx"], c["ny"]), "euler.problem": p, "euler.gamma": GAMMA, "stop_time": 1.0e9,
          "max_step": 100000000, "euler.spatial_order": 2}
    if p == "sod":
        kv.update({"euler.problem": "toro1", "prob.test": 1, "prob.x0": 0.5, "geometry.prob_hi": "1 %r" % (c["ny"] / c["nx"]),
                   "geometry.is_periodic": "0 1", "euler.field_boundary": "exact_dirichlet", "euler.cfl": 0.45})
    elif p == "gresho":
        m = c["mach"]
        kv.update({"euler.problem": "gresho_vortex", "geometry.is_periodic": "1 1", "euler.vortex_center": "0.5 0.5",
                   "euler.mach": m, "euler.pressure": repr(1.0 / (GAMMA * m * m)), "euler.cfl": 0.5})
    elif p == "quadrant":
        kv.update({"euler.problem": "riemann_quadrant", "geometry.is_periodic": "0 0", "euler.cfl": 0.45})
    elif p == "bubble":
        kv.update({"euler.problem": "shock_density_bubble_2d", "geometry.prob_hi": "2 0.5", "euler.cfl": 0.45})
    else:
        kv.update({"euler.problem": "advection_blob", "geometry.is_periodic": "1 1", "euler.cfl": 0.45})
    if c["kind"] == "imex":
        kv.update({"euler.method": "imex", "euler.imex_acoustic_startup": 0, "euler.imex_picard_iterations": PICARD,
                   "euler.imex_solver_tol": "1e-10", "euler.imex_solver_max_iter": 200,
                   "euler.imex_cfl": 0.45 if p == "bubble" else 0.4})
    else:
        kv.update({"euler.method": "explicit", "euler.riemann": c["riemann"], "euler.slope_limiter": c["limiter"]})
    return kv


def _settings(c):
    return read_config(_kv(c)).cfg


def _conserved(q):
    rho, u, v, p = q
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)])


def _waves(X, Y, gen, count=6):
    """A smooth random field of order one."""
    f = torch.zeros_like(X)
    for _ in range(count):
        k = torch.randint(1, 5, (2,), generator=gen).tolist()
        a, b, s = torch.rand(3, generator=gen, dtype=torch.float64).tolist()
        f += (0.5 + s) * torch.sin(2 * math.pi * (k[0] * X + a)) * torch.cos(2 * math.pi * (k[1] * Y + b))
    return f / count


def _state(c, seed):
    """Initial state of the case's problem with seeded smooth perturbations."""
    gen = torch.Generator().manual_seed(int(seed))
    nx, ny = c["nx"], c["ny"]
    dev = torch.device("cuda")
    x = (torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=dev) + 0.5) / ny
    X, Y = x.expand(ny, nx), y[:, None].expand(ny, nx)
    w = [_waves(X, Y, gen) for _ in range(4)]
    r = torch.rand(4, generator=gen, dtype=torch.float64).tolist()
    one = torch.ones_like(X)
    p = c["problem"]
    if p == "sod":
        left = X < 0.5
        bump = torch.exp(-((X - 0.5) / 0.06) ** 4) * 0.1  # the exact states reach the boundaries
        q = [torch.where(left, 1.0, 0.125) * (1 + bump * w[0]), bump * w[1], bump * w[2],
             torch.where(left, 1.0, 0.1) * (1 + bump * w[3])]
    elif p == "gresho":
        xc, yc = X - 0.5, Y - 0.5
        rr = torch.sqrt(xc * xc + yc * yc)
        mid = 2.0 - 5.0 * rr
        ut = torch.where(rr < 0.2, 5.0 * rr, torch.where(rr < 0.4, mid, 0.0 * rr))
        p0 = 1.0 / (GAMMA * c["mach"] ** 2)
        pin = p0 + 12.5 * rr * rr
        pmid = p0 + 12.5 * rr * rr + 4.0 * (1.0 - 5.0 * rr + torch.log(5.0 * rr.clamp_min(1e-3)))
        pp = torch.where(rr < 0.2, pin, torch.where(rr < 0.4, pmid, p0 - 2.0 + 4.0 * math.log(2.0) + 0 * rr))
        s = ut / rr.clamp_min(1e-12)
        # the density and a divergence-free velocity are perturbed
        kx = 2 * math.pi
        q = [one + 0.02 * w[0], -s * yc + 0.02 * (r[0] - 0.5) + 0.02 * torch.sin(kx * (Y + r[1])),
             s * xc + 0.02 * (r[2] - 0.5) + 0.02 * torch.sin(kx * (X + r[3])), pp]
    elif p == "quadrant":
        left, low = X < 0.8, Y < 0.8
        f = lambda a, b, d, e: torch.where(low, torch.where(left, d, e), torch.where(left, b, a))  # noqa: E731
        q = [f(1.5, 0.5323, 0.138, 0.5323) * (1 + 0.02 * w[0]), f(0.0, 1.206, 1.206, 0.0) + 0.02 * w[1],
             f(0.0, 0.0, 1.206, 1.206) + 0.02 * w[2], f(1.5, 0.3, 0.029, 0.3) * (1 + 0.02 * w[3])]
    elif p == "bubble":
        xs, ys = 2.0 * X, 0.5 * Y
        post = xs < 0.2
        rad = torch.sqrt((xs - 0.5 - 0.02 * r[0]) ** 2 + ys * ys)
        rho = 0.1 + 0.9 * torch.sigmoid((rad - 0.2) / 0.01)
        calm = torch.where(post, 0.0, 0.02)
        q = [torch.where(post, 2.8181818181818183, rho) * (1 + calm * w[0]),
             torch.where(post, 1.6064386578049976, 0.0) + calm * w[1], calm * w[2],
             torch.where(post, 5.0, 1.0) * (1 + calm * w[3])]
    else:
        rho = 1.0 + 0.5 * torch.exp(-((X - 0.35) ** 2 + (Y - 0.35) ** 2) / 0.01)
        q = [rho * (1 + 0.1 * w[0]), 1.0 + 0.1 * w[1], 0.5 + 0.1 * w[2], 1.0 + 0.1 * w[3]]
    return _conserved(q).contiguous()


BATCH_GRIDS = workloads.BATCH_GRIDS


def _batch(c, seed):
    """The case's solves: seeded Riemann problems on a fixed list of grids."""
    cfgs, states = [], []
    for k in range(c["nsolve"]):
        gx, gy = BATCH_GRIDS[k % len(BATCH_GRIDS)]
        grid = (max(16, int(gx * c["scale"])), max(16, int(gy * c["scale"])))
        a, b = workloads.riemann_batch(1, seed=1000 * int(seed) + k, grids=[grid], riemann=c["riemann"])
        cfgs += a
        states += b
    return cfgs, states


# ---- the cases ------------------------------------------------------------------------


def _dt(ctx, u, share=1.0):
    ctx.upload_device(u.data_ptr())
    return share * api.compute_euler_dt(ctx, 0.0)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        cfgs, states = _batch(c, seed)
        b = api.Batch(cfgs)
        for k, u in enumerate(states):
            b.upload(k, u)
        return {"kind": kind, "case": c, "batch": b}
    u = _state(c, seed)
    torch.cuda.current_stream().synchronize()  # the context has a stream of its own
    if kind == "adjoint":
        ctx = autograd.make_context(_settings(c))
    else:
        ctx = api.Context(_settings(c), arith=c.get("arith", "fast"), imex_precision=c.get("precision", "fp64"))
    s = {"kind": kind, "case": c, "ctx": ctx, "u": u, "out": torch.empty_like(u)}
    if kind == "host":
        s["dt"] = _dt(ctx, u)
        s["pinned"] = torch.empty(u.shape, dtype=u.dtype, pin_memory=True), torch.empty(u.shape, dtype=u.dtype, pin_memory=True)
        s["pinned"][0].copy_(u)
        s["u_in"], s["u_out"] = (t.numpy() for t in s["pinned"])
    if kind == "adjoint":
        s["dts"] = [_dt(ctx, u, 0.9)] * c["steps"]
        gen = torch.Generator().manual_seed(int(seed) + 7)
        s["g"] = torch.randn(u.shape, generator=gen, dtype=torch.float64).cuda()
        s["u"] = u.requires_grad_(True)
    return s


def run(state):
    s, c = state, state["case"]
    kind = s["kind"]
    if kind == "batch":
        b = s["batch"]
        b.run(c["steps"])
        return [b.download(k) for k in range(b.n)]
    ctx = s["ctx"]
    if kind == "host":
        deg = api.euler_fv_one_step_host(ctx, s["u_in"], s["u_out"], s["dt"])
        return {"state": s["u_out"], "degenerate": deg}
    if kind == "adjoint":
        un = autograd.explicit_rollout(ctx, s["u"], s["dts"])
        (g,) = torch.autograd.grad(un, s["u"], s["g"])
        return {"state": un.detach(), "gradient": g}
    ctx.upload_device(s["u"].data_ptr())
    if kind == "run":
        r = api.run(ctx, c["steps"], 1.0e9)
        ctx.download_device(s["out"].data_ptr())
        ctx.synchronize()
        return {"state": s["out"], "time": r.time, "rho_min": r.diagnostics.rho_min,
                "pressure_min": r.diagnostics.pressure_min, "steps": r.steps}
    t, rho_min, p_min = 0.0, 0.0, 0.0
    for _ in range(c.get("steps", 1)):
        if kind == "loop":
            dt = api.compute_euler_dt(ctx, t)
            api.euler_fv_one_step(ctx, dt, t)
            d = api.compute_diagnostics(ctx)
            rho_min, p_min = d.rho_min, d.pressure_min
        else:
            dt, _ = api.compute_imex_dt(ctx, t)
            d = api.euler_imex_bdltv20_o1_source_map_picard_one_step(ctx, dt)
            rho_min, p_min = d.rho_min, d.pressure_min
        t += dt
    ctx.download_device(s["out"].data_ptr())
    ctx.synchronize()
    return {"state": s["out"], "time": t, "rho_min": rho_min, "pressure_min": p_min}


# FP64 operations of one explicit cell update, by flux: counted from the formulas
FLOPS = {"rusanov": 250, "hllc": 330, "lowmach_hllc": 420, "xie_am_hllc_p": 700}


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        cells = sum(max(16, int(BATCH_GRIDS[k % 5][0] * c["scale"])) * max(16, int(BATCH_GRIDS[k % 5][1] * c["scale"]))
                    for k in range(c["nsolve"]))
        return {"bytes": 64 * cells, "flops": cells * c["steps"] * FLOPS[c["riemann"]]}
    cells = c["nx"] * c["ny"]
    if kind == "imex":
        # star update, assembly and closeout, and per solve the operator, one
        # dot product and one update per basis vector and iteration
        its = 6.5 if c["problem"] == "bubble" else (32.0 if c["mach"] < 0.05 else 12.5)
        return {"bytes": 64 * cells, "flops": cells * (400 + PICARD * (60 + 30 * its + 2 * its * (its + 1)))}
    if kind == "adjoint":  # the forward step and, backward, the face Jacobians applied to the cotangent
        return {"bytes": 128 * cells, "flops": cells * c["steps"] * 4 * FLOPS[c["riemann"]]}
    return {"bytes": 64 * cells, "flops": cells * c["steps"] * FLOPS[c["riemann"]]}


# ---- the same in 64-bit torch ------------------------------------------------------------


def _primitive(U):
    rho, mx, my, E = U.unbind(-3)
    u, v = mx / rho, my / rho
    return torch.stack([rho, u, v, (GAMMA - 1.0) * (E - 0.5 * rho * (u * u + v * v))], -3)


def _pad(U, problem, k=2):
    """`U` (..., 4, ny, nx), conserved, with k ghost cells on each side."""
    if problem in ("gresho", "blob"):
        U = torch.cat([U[..., -k:], U, U[..., :k]], -1)
        return torch.cat([U[..., -k:, :], U, U[..., :k, :]], -2)
    lo, hi = U[..., :1].expand(*U.shape[:-1], k), U[..., -1:].expand(*U.shape[:-1], k)
    fixed = {"sod": ((1.0, 0.0, 0.0, 1.0), (0.125, 0.0, 0.0, 0.1)),
             "bubble": ((2.8181818181818183, 1.6064386578049976, 0.0, 5.0), None)}.get(problem, (None, None))
    for n, q in enumerate(fixed):
        if q is not None:
            g = _conserved([torch.tensor(v, dtype=torch.float64, device=U.device) for v in q])
            g = g.view(4, 1, 1).expand(*U.shape[:-1], k)
            lo, hi = (g, hi) if n == 0 else (lo, g)
    U = torch.cat([lo, U, hi], -1)
    if problem in ("sod", "riemann"):
        return torch.cat([U[..., -k:, :], U, U[..., :k, :]], -2)
    top = U[..., -1:, :].expand(*U.shape[:-2], k, U.shape[-1])
    if problem == "bubble":  # a wall below
        low = U[..., :k, :].flip(-2) * torch.tensor([1.0, 1.0, -1.0, 1.0], dtype=torch.float64, device=U.device).view(4, 1, 1)
    else:
        low = U[..., :1, :].expand(*U.shape[:-2], k, U.shape[-1])
    return torch.cat([low, U, top], -2)


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _slope(a, b, limiter):
    if limiter == "mc":
        s = _minmod(_minmod(2 * a, 0.5 * (a + b)), 2 * b)
    elif limiter == "vanleer":
        d = a + b
        flat = d.abs() <= 1e-14
        s = torch.where(flat, torch.zeros_like(a), 2 * a * b / torch.where(flat, torch.ones_like(d), d))
    else:
        s = _minmod(a, b)
    return torch.where(a * b <= 0, torch.zeros_like(a), s)


def _faces(q, limiter):
    """States left and right of the faces between the inner cells of the last axis."""
    d = q[..., 1:] - q[..., :-1]
    s = _slope(d[..., :-1], d[..., 1:], limiter)
    return q[..., 1:-2] + 0.5 * s[..., :-1], q[..., 2:-1] - 0.5 * s[..., 1:]


def _normal(q):
    """(rho, normal velocity, tangential velocity, p) and conserved energy of x-states."""
    rho, u, v, p = q.unbind(-3)
    return rho, u, v, p, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)


def _physical(rho, u, v, p, E):
    return [rho * u, rho * u * u + p, rho * u * v, (E + p) * u]


def _rusanov(L, R, cl, cr):
    s = torch.maximum(L[1].abs() + cl, R[1].abs() + cr)
    fl, fr = _physical(*L), _physical(*R)
    ul, ur = ([q[0], q[0] * q[1], q[0] * q[2], q[4]] for q in (L, R))
    return [0.5 * (a + b) - 0.5 * s * (d - e) for a, b, e, d in zip(fl, fr, ul, ur)]


def _safe(x):
    return torch.where(x.abs() <= 1e-12, torch.ones_like(x), x)


def _flux(ql, qr, riemann, sensor=None):
    """Numerical flux along x of the states ql, qr (..., 4, h, w)."""
    if riemann == "lowmach_hllc":
        sp = [torch.sqrt(q[..., 1, :, :] ** 2 + q[..., 2, :, :] ** 2) /
              torch.sqrt(GAMMA * q[..., 3, :, :] / q[..., 0, :, :]).clamp_min(1e-12) for q in (ql, qr)]
        z = torch.maximum(*sp).clamp(0.0, 1.0).unsqueeze(-3)
        vl, vr = ql[..., 1:3, :, :], qr[..., 1:3, :, :]
        mean, half = 0.5 * (vl + vr), 0.5 * z * (vl - vr)
        ql = torch.cat([ql[..., :1, :, :], mean + half, ql[..., 3:, :, :]], -3)
        qr = torch.cat([qr[..., :1, :, :], mean - half, qr[..., 3:, :, :]], -3)
    L, R = _normal(ql), _normal(qr)
    cl, cr = torch.sqrt(GAMMA * L[3] / L[0]), torch.sqrt(GAMMA * R[3] / R[0])
    if riemann == "rusanov":
        return torch.stack(_rusanov(L, R, cl, cr), -3)
    sl, sr = torch.minimum(L[1] - cl, R[1] - cr), torch.maximum(L[1] + cl, R[1] + cr)
    al, ar = L[0] * (sl - L[1]), R[0] * (sr - R[1])
    den = al - ar
    sm = (R[3] - L[3] + al * L[1] - ar * R[1]) / _safe(den)
    left = torch.where(sl >= 0, torch.ones_like(sl, dtype=torch.bool), torch.where(sr <= 0, torch.zeros_like(sl, dtype=torch.bool), sm >= 0))
    K = [torch.where(left, a, b) for a, b in zip(L, R)]
    s, a = torch.where(left, sl, sr), torch.where(left, al, ar)
    sd = _safe(s - sm)
    F = _physical(*K)
    if riemann == "xie_am_hllc_p":
        ps = (ar * L[3] - al * R[3] - al * ar * (L[1] - R[1])) / _safe(ar - al)
        wl, wr = torch.sqrt(L[0]), torch.sqrt(R[0])
        uh, vh = (wl * L[1] + wr * R[1]) / (wl + wr), (wl * L[2] + wr * R[2]) / (wl + wr)
        hh = (wl * (L[4] + L[3]) / L[0] + wr * (R[4] + R[3]) / R[0]) / (wl + wr)
        c2 = (GAMMA - 1.0) * (hh - 0.5 * (uh * uh + vh * vh))
        mh = uh / torch.sqrt(c2)
        th = torch.maximum(torch.sqrt(L[1] ** 2 + L[2] ** 2) / cl, torch.sqrt(R[1] ** 2 + R[2] ** 2) / cr).clamp(0.0, 1.0)
        pss = th * ps + (1.0 - th) * 0.5 * (L[3] + R[3])
        psss = sensor * pss + (1.0 - sensor) * ps
        bp = (sensor - 1.0) * sl * sr / (sr - sl) * (R[3] - L[3]) / (c2 * (1.0 + mh.abs()))
        rs = a / sd
        es = K[4] / K[0] + (sm - K[1]) * (sm + K[3] / _safe(a))
        star = [rs * sm + bp, rs * sm * sm + psss + bp * uh, rs * sm * K[2] + bp * vh,
                sm * (rs * es + ps) + 0.5 * bp * (uh * uh + vh * vh)]
    else:
        ps = 0.5 * (L[3] + al * (sm - L[1]) + R[3] + ar * (sm - R[1]))
        rs = a / sd
        es = ((s - K[1]) * K[4] - K[3] * K[1] + ps * sm) / sd
        star = [f + s * (b - w) for f, b, w in zip(F, [rs, rs * sm, rs * K[2], es], [K[0], K[0] * K[1], K[0] * K[2], K[4]])]
    fast = (sl >= 0) | (sr <= 0)
    out = [torch.where(fast, f, g) for f, g in zip(F, star)]
    if riemann != "xie_am_hllc_p":
        bad = ~(sl < sr) | (~fast & ((den.abs() <= 1e-12) | ((sl - sm).abs() <= 1e-12) | ((sr - sm).abs() <= 1e-12)))
        out = [torch.where(bad, g, f) for f, g in zip(out, _rusanov(L, R, cl, cr))]
    return torch.stack(out, -3)


def _swap(q):
    """The state with x and y exchanged."""
    q = q.transpose(-1, -2)
    return torch.cat([q[..., :1, :, :], q[..., 2:3, :, :], q[..., 1:2, :, :], q[..., 3:, :, :]], -3)


def _ratio(ql, qr):
    pl, pr = ql[..., 3, :, :].clamp_min(1e-14), qr[..., 3, :, :].clamp_min(1e-14)
    return torch.minimum(pl / pr, pr / pl)


def _step(U, dt, dx, dy, problem, riemann, limiter):
    q = _primitive(_pad(U, problem))
    xl, xr = _faces(q, limiter)  # rows -2 .. ny+1, x-faces 0 .. nx
    yl, yr = _faces(_swap(q), limiter)  # columns -2 .. nx+1, y-faces 0 .. ny, x and y exchanged
    sx = sy = None
    if riemann == "xie_am_hllc_p":
        rx, ry = _ratio(xl, xr), _ratio(yl, yr).transpose(-1, -2)
        m = rx[..., 2:-2, :]
        for t in (ry[..., :-1, 1:-2], ry[..., 1:, 1:-2], ry[..., :-1, 2:-1], ry[..., 1:, 2:-1]):
            m = torch.minimum(m, t)
        sx = m.clamp(0.0, 1.0) ** 3
        m = ry[..., :, 2:-2]
        for t in (rx[..., 1:-2, :-1], rx[..., 1:-2, 1:], rx[..., 2:-1, :-1], rx[..., 2:-1, 1:]):
            m = torch.minimum(m, t)
        sy = (m.clamp(0.0, 1.0) ** 3).transpose(-1, -2)
    F = _flux(xl[..., 2:-2, :], xr[..., 2:-2, :], riemann, sx)
    G = _swap(_flux(yl[..., 2:-2, :], yr[..., 2:-2, :], riemann, sy))
    return U - dt * ((F[..., 1:] - F[..., :-1]) / dx + (G[..., 1:, :] - G[..., :-1, :]) / dy)


def _rate(U, dx, dy):
    rho, u, v, p = _primitive(U).unbind(-3)
    c = torch.sqrt(GAMMA * p / rho)
    return ((u.abs() + c) / dx + (v.abs() + c) / dy).amax((-1, -2))


def _march(U, steps, cfl, dx, dy, problem, riemann, limiter):
    t = torch.zeros(U.shape[:-3], dtype=torch.float64, device=U.device)
    for _ in range(steps):
        dt = cfl / _rate(U, dx, dy)
        U = _step(U, dt[..., None, None, None] if dt.dim() else dt, dx, dy, problem, riemann, limiter)
        t = t + dt
    return U, t


class _Imex:
    """One IMEX T1/S2 step: star update, Picard pressure solves, closeout."""

    def __init__(self, case, dx, dy):
        self.wall = case["problem"] == "bubble"
        self.problem, self.dx, self.dy = case["problem"], dx, dy
        self.post = (2.8181818181818183, 1.6064386578049976, 0.0, 5.0)

    def pressure(self, p, k, fixed):
        """Ghosted pressure: wrapped, or evenly reflected with `fixed` on the left."""
        if not self.wall:
            p = torch.cat([p[:, -k:], p, p[:, :k]], 1)
            return torch.cat([p[-k:], p, p[:k]], 0)
        p = torch.cat([torch.full_like(p[:, :k], fixed), p, p[:, -k:].flip(1)], 1)
        return torch.cat([p[:k].flip(0), p, p[-k:].flip(0)], 0)

    def momentum(self, K):
        if not self.wall:
            return _pad(torch.cat([K, K]), "gresho", 1)[:2]
        left = torch.tensor([self.post[0] * self.post[1], 0.0], dtype=torch.float64, device=K.device).view(2, 1, 1)
        K = torch.cat([left.expand(2, K.shape[1], 1), K, K[..., -1:]], 2)
        low = K[:, :1] * torch.tensor([1.0, -1.0], dtype=torch.float64, device=K.device).view(2, 1, 1)
        return torch.cat([low, K, K[:, -1:]], 1)

    def enthalpy(self, S, p, K):
        """Face enthalpies and the mean normal lagged momentum on x- and y-faces."""
        rho, K = _pad(S, self.problem, 1)[0], self.momentum(K)
        h = GAMMA * self.pressure(p, 1, self.post[3]) / ((GAMMA - 1.0) * rho)
        out = []
        for a, b, q in ((h[1:-1, :-1], h[1:-1, 1:], (K[0, 1:-1, :-1], K[0, 1:-1, 1:])),
                        (h[:-1, 1:-1], h[1:, 1:-1], (K[1, :-1, 1:-1], K[1, 1:, 1:-1]))):
            den = q[0] + q[1]
            guard = den.abs() <= 1e-14 * torch.maximum(q[0].abs(), q[1].abs()).clamp_min(1.0)
            mean = torch.where(guard, 0.5 * (a + b), (a * q[0] + b * q[1]) / torch.where(guard, torch.ones_like(den), den))
            out += [mean, 0.5 * den]
        return out

    def operator(self, p, hx, hy, dt, fixed=0.0):
        q = self.pressure(p, 2, fixed)
        xc, yc = 0.25 * (dt / self.dx) ** 2, 0.25 * (dt / self.dy) ** 2
        he, hw, hn, hs = hx[:, 1:], hx[:, :-1], hy[1:], hy[:-1]
        x, y = q[2:-2], q[:, 2:-2]
        return ((1.0 / (GAMMA - 1.0) + xc * (he + hw) + yc * (hn + hs)) * p
                - xc * (he * x[:, 4:] + (he - hw) * (x[:, 3:-1] - x[:, 1:-3]) + hw * x[:, :-4])
                - yc * (hn * y[4:] + (hn - hs) * (y[3:-1] - y[1:-3]) + hs * y[:-4]))

    @staticmethod
    def solve(A, b, x, cycles=3, m=120):
        shape, n = b.shape, b.numel()
        for _ in range(cycles):
            r = (b - A(x)).reshape(-1)
            beta = r.norm()
            if float(beta) <= 1e-15 * float(b.norm()):
                break
            V = torch.empty(m + 1, n, dtype=torch.float64, device=b.device)
            H = torch.zeros(m + 1, m, dtype=torch.float64, device=b.device)
            V[0] = r / beta
            k = m
            for j in range(m):
                w = A(V[j].view(shape)).reshape(-1)
                for _ in range(2):
                    d = V[: j + 1] @ w
                    w = w - d @ V[: j + 1]
                    H[: j + 1, j] += d
                H[j + 1, j] = w.norm()
                V[j + 1] = w / H[j + 1, j]
                if (j + 1) % 10 == 0:
                    e = torch.zeros(j + 2, 1, dtype=torch.float64, device=b.device)
                    e[0] = beta
                    y = torch.linalg.lstsq(H[: j + 2, : j + 1], e).solution
                    if float((H[: j + 2, : j + 1] @ y - e).norm()) <= 1e-13 * float(beta):
                        k = j + 1
                        break
            e = torch.zeros(k + 1, 1, dtype=torch.float64, device=b.device)
            e[0] = beta
            y = torch.linalg.lstsq(H[: k + 1, :k], e).solution.reshape(-1)
            x = x + (y @ V[:k]).view(shape)
            del V
        return x

    def step(self, U, dt):
        q = _pad(U, self.problem)

        def flux(q):
            d = q[..., 1:] - q[..., :-1]
            s = _minmod(d[..., :-1], d[..., 1:])
            L, R = (_normal(_primitive(t)) for t in (q[..., 1:-2] + 0.5 * s[..., :-1], q[..., 2:-1] - 0.5 * s[..., 1:]))
            sm = torch.maximum(L[1].abs(), R[1].abs())
            out = []
            for n in range(4):
                f = []
                for rho, u, v, p, E in (L, R):
                    c = [rho, rho * u, rho * v, E][n]
                    f.append((c, [rho * u, rho * u * u, rho * v * u, 0.5 * rho * (u * u + v * v) * u][n]))
                out.append(0.5 * (f[0][1] + f[1][1]) - 0.5 * sm * (f[1][0] - f[0][0]))
            return torch.stack(out, -3)

        F = flux(q[:, 2:-2, :])
        G = _swap(flux(_swap(q[:, :, 2:-2])))
        S = U - dt * ((F[..., 1:] - F[..., :-1]) / self.dx + (G[:, 1:, :] - G[:, :-1, :]) / self.dy)
        p, K = _primitive(U)[3], S[1:3]
        ghost = _pad(S, self.problem, 1)
        mx, my = ghost[1], ghost[2]
        for _ in range(PICARD):
            hx, _, hy, _ = self.enthalpy(S, p, K)
            he, hw, hn, hs = hx[:, 1:], hx[:, :-1], hy[1:], hy[:-1]
            b = S[3] - 0.5 * (K[0] ** 2 + K[1] ** 2) / S[0]
            b = b - 0.5 * dt / self.dx * (he * mx[1:-1, 2:] + (he - hw) * S[1] - hw * mx[1:-1, :-2])
            b = b - 0.5 * dt / self.dy * (hn * my[2:, 1:-1] + (hn - hs) * S[2] - hs * my[:-2, 1:-1])
            if self.wall:
                b = b - self.operator(torch.zeros_like(p), hx, hy, dt, self.post[3])
            p = self.solve(lambda v: self.operator(v, hx, hy, dt), b, p)
            g = self.pressure(p, 1, self.post[3])
            K = torch.stack([S[1] - dt * 0.5 * (g[1:-1, 2:] - g[1:-1, :-2]) / self.dx,
                             S[2] - dt * 0.5 * (g[2:, 1:-1] - g[:-2, 1:-1]) / self.dy])
        hx, kx, hy, ky = self.enthalpy(S, p, K)
        fx, fy = hx * kx, hy * ky
        E = S[3] - dt * ((fx[:, 1:] - fx[:, :-1]) / self.dx + (fy[1:] - fy[:-1]) / self.dy)
        return torch.stack([S[0], K[0], K[1], E])


def _minima(U):
    q = _primitive(U)
    return float(q[0].min()), float(q[3].min())


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        cfgs, states = _batch(c, seed)
        out, groups = [None] * len(states), {}
        for k, u in enumerate(states):
            groups.setdefault(u.shape, []).append(k)
        for shape, ks in groups.items():
            U = torch.stack([torch.from_numpy(states[k]) for k in ks]).cuda()
            cfg = cfgs[ks[0]].cfg
            dx, dy = cfg.prob_hi[0] / shape[2], cfg.prob_hi[1] / shape[1]
            U, _ = _march(U, c["steps"], cfg.cfl, dx, dy, "riemann", c["riemann"], "minmod")
            for k, v in zip(ks, U):
                out[k] = v.cpu().numpy()
        return out
    cfg = _settings(c)
    dx, dy = ((cfg.prob_hi[n] - cfg.prob_lo[n]) / cfg.n_cell[n] for n in (0, 1))
    U = _state(c, seed)
    args = (dx, dy, c["problem"], c.get("riemann"), c.get("limiter"))
    if kind == "imex":
        _, u, v, _ = _primitive(U)
        dt = cfg.imex_cfl / float((2.0 * torch.sqrt(u * u + v * v)).max() / min(dx, dy))
        U = _Imex(c, dx, dy).step(U, dt)
        rho, p = _minima(U)
        return {"state": U, "time": dt, "rho_min": rho, "pressure_min": p}
    if kind == "host":
        dt = cfg.cfl / float(_rate(U, dx, dy))
        return {"state": _step(U, dt, *args).cpu().numpy(), "degenerate": None}
    if kind == "adjoint":
        dt = 0.9 * cfg.cfl / float(_rate(U, dx, dy))
        gen = torch.Generator().manual_seed(int(seed) + 7)
        g = torch.randn(U.shape, generator=gen, dtype=torch.float64).cuda()
        states = [U]
        for _ in range(c["steps"]):
            states.append(_step(states[-1], dt, *args))
        for u in reversed(states[:-1]):
            u = u.detach().requires_grad_(True)
            (g,) = torch.autograd.grad(_step(u, dt, *args), u, g)
        return {"state": states[-1], "gradient": g}
    U, t = _march(U, c["steps"], cfg.cfl, *args)
    rho, p = _minima(U)
    out = {"state": U, "time": float(t), "rho_min": rho, "pressure_min": p}
    if kind == "run":
        out["steps"] = None
    return out
