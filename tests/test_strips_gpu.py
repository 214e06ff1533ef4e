"""The column strips against the tile kernels, and the device loop against
single steps.

Exact arithmetic: the strips evaluate the reference's expressions, so they must
equal the 32x16 tiles bit for bit.  Fast arithmetic: strips and 16x16 tiles
share their refined divisions but associate the fluxes differently; one step
moves a state by less than itself, and a few hundred roundings a cell stay
below 1e-13 of the field (3e-13 for the HLLC-P flux, as its older test holds).
Sizes: one cell, fewer columns than a strip owns, one either side of a strip
and of a block of two, rows fewer than and around a strip's; every ghost
policy, first and second order."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config
from tests.golden_io import state_rel_err

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (27, 5), (28, 8), (29, 9), (57, 33), (300, 97), (64, 1)]
PROBLEMS = {
    "periodic": "geometry.is_periodic=1 1\neuler.problem=advection_blob\n",
    "outflow": "geometry.is_periodic=0 0\neuler.problem=advection_blob\n",
    "mixed": "geometry.is_periodic=0 1\neuler.problem=toro1\n",
    "ring": "geometry.is_periodic=0 1\neuler.problem=toro1\neuler.field_boundary=exact_dirichlet\n",
    "ring_xy": "geometry.is_periodic=0 0\neuler.problem=riemann_quadrant\neuler.field_boundary=exact_dirichlet\n",
    "bubble": "euler.problem=shock_density_bubble_2d\ngeometry.prob_hi=2 0.5\n",
    "walls": "euler.problem=shock_bubble_mach122\ngeometry.prob_hi=4 1\n",
}


def _state(nx, ny, seed):
    rng = np.random.default_rng(seed)
    rho, p = 0.6 + 0.8 * rng.random((ny, nx)), 0.6 + 0.8 * rng.random((ny, nx))
    u, v = 1.5 * rng.standard_normal((ny, nx)), 0.7 * rng.standard_normal((ny, nx))
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


def _step(cfg, u, dt, **gpu):
    with api.Context(cfg, **gpu) as ctx:
        ctx.upload(u)
        deg = api.euler_fv_one_step(ctx, dt, 0.01)
        d = api.compute_diagnostics(ctx)
        return ctx.download(), deg, (d.rho_min, d.pressure_min, d.nonfinite_count), api.compute_euler_dt(ctx, 0.01)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("riemann,limiter", [("hllc", "minmod"), ("lowmach_hllc", "vanleer"), ("rusanov", "mc"),
                                             ("xie_am_hllc_p", "minmod")])
@pytest.mark.parametrize("problem", sorted(PROBLEMS))
def test_strips_equal_tiles(gpu, problem, riemann, limiter, order):
    if problem in ("bubble", "walls") and (order == 1 or riemann not in ("hllc", "xie_am_hllc_p")):
        pytest.skip("not a configuration of the bubble")
    for k, (nx, ny) in enumerate(SIZES):
        if problem in ("bubble", "walls") and (nx < 16 or ny < 4):
            continue
        cfg = read_config(f"amr.n_cell={nx} {ny}\neuler.spatial_order={order}\neuler.riemann={riemann}\n"
                          f"euler.slope_limiter={limiter}\nstop_time=10\nmax_step=1000\n" + PROBLEMS[problem]).cfg
        u = _state(nx, ny, 100 * k + order)
        dt = 0.1 * min((cfg.prob_hi[n] - cfg.prob_lo[n]) / cfg.n_cell[n] for n in (0, 1))
        a, b = _step(cfg, u, dt, arith="exact"), _step(cfg, u, dt, arith="exact", tile_y=16)
        assert np.array_equal(a[0], b[0]) and a[1:] == b[1:], (nx, ny)
        c, d = _step(cfg, u, dt), _step(cfg, u, dt, tile_y=1)
        assert state_rel_err(c[0], d[0]) <= (3e-13 if riemann == "xie_am_hllc_p" else 1e-13), (nx, ny)
        assert c[1] == d[1] and c[2][2] == d[2][2], (nx, ny)


@pytest.mark.parametrize("arith", ["fast", "exact"])
@pytest.mark.parametrize("steps", [0, 1, 31, 32, 33, 64, 70])
def test_run_equals_single_steps(gpu, steps, arith):
    """The device loop ends at its step limit, on a chunk's end or off it, with
    the state of that many steps taken one at a time."""
    cfg = read_config("amr.n_cell=75 40\ngeometry.is_periodic=0 1\neuler.problem=toro1\neuler.spatial_order=2\n"
                      "euler.field_boundary=exact_dirichlet\neuler.cfl=0.4\nstop_time=10\nmax_step=1000\n").cfg
    with api.Context(cfg, arith=arith) as ctx:
        api.initialize_state(ctx)
        u = ctx.download()
        r = api.run(ctx, steps, cfg.stop_time)
        got = ctx.download()
        assert r.steps == steps and not r.failed
        ctx.upload(u)
        t = 0.0
        for _ in range(steps):
            dt = api.compute_euler_dt(ctx, t)
            api.euler_fv_one_step(ctx, dt, t)
            t += dt
        assert r.time == t and np.array_equal(got, ctx.download())


def test_run_stops_at_the_time_limit_and_on_a_bad_state(gpu):
    kv = "amr.n_cell=75 40\ngeometry.is_periodic=1 1\neuler.problem=advection_blob\neuler.cfl=0.4\nstop_time=10\n"
    cfg = read_config(kv).cfg
    with api.Context(cfg) as ctx:
        api.initialize_state(ctx)
        u = ctx.download()
        r = api.run(ctx, 32, cfg.stop_time)
        t = r.time
        ctx.upload(u)
        r = api.run(ctx, 1000, t)  # the time limit falls on the chunk's last step
        assert r.steps == 32 and r.time == t and r.failure_code == 0
        u[0, 3, 5] = np.nan
        ctx.upload(u)
        r = api.run(ctx, 32, cfg.stop_time)
        assert r.failed and r.steps == 0
