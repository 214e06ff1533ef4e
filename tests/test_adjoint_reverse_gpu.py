"""The step's vector-Jacobian product against torch's own reverse mode.

The step is restated in float64 torch (perf/cases.py) and differentiated by
autograd, on states whose one-sided differences, wave speeds and middle speeds
are generic (no limiter tie or upwind switch sits at a rounding error), so the
two take the same branches.  Sizes: one cell row and column, fewer rows than a
tile, one past a tile edge, and several ragged tiles; every boundary policy of
the adjoint.  Both sides round each of a few hundred operations a face, so they
agree to a small multiple of 1e-13 of the largest gradient entry."""
import ctypes as C

import pytest

from amrex_euler_allmach_explicit_imex_b200 import _lib, api

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 2), (32, 8), (33, 9), (47, 70), (100, 31)]


def _setup(problem, nx, ny, riemann, limiter):
    import torch

    from perf import cases

    c = {"kind": "adjoint", "problem": problem, "nx": nx, "ny": ny, "riemann": riemann, "limiter": limiter, "steps": 1}
    gen = torch.Generator().manual_seed(nx * 1000 + ny)
    x = (torch.arange(nx, dtype=torch.float64) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64) + 0.5) / ny
    X, Y = x.expand(ny, nx), y[:, None].expand(ny, nx)
    w = [cases._waves(X, Y, gen) + 0.05 * torch.rand(ny, nx, generator=gen, dtype=torch.float64) for _ in range(4)]
    u = cases._conserved([1.0 + 0.3 * w[0], 0.3 + 0.4 * w[1], -0.2 + 0.4 * w[2], 1.0 + 0.3 * w[3]]).cuda().contiguous()
    g = torch.randn(u.shape, generator=gen, dtype=torch.float64).cuda()
    settings = cases._settings(c)
    dx, dy = ((settings.prob_hi[n] - settings.prob_lo[n]) / settings.n_cell[n] for n in (0, 1))
    dt = 0.2 * min(dx, dy)

    def step(v):
        return cases._step(v, dt, dx, dy, problem, riemann, limiter)

    return torch, settings, u, g, dt, step


def _vjp(ctx, u, dt, g, out):
    _lib.check(_lib.load().ecg_explicit_step_vjp_device(ctx.handle, C.c_void_p(u.data_ptr()), dt,
                                                        C.c_void_p(g.data_ptr()), C.c_void_p(out.data_ptr())),
               "vjp", ctx.handle)
    ctx.synchronize()


@pytest.mark.parametrize("limiter", ["minmod", "mc", "vanleer"])
@pytest.mark.parametrize("riemann", ["hllc", "lowmach_hllc", "rusanov"])
@pytest.mark.parametrize("problem", ["blob", "quadrant", "bubble"])
def test_vjp_matches_autograd(gpu, problem, riemann, limiter):
    if problem == "bubble" and riemann != "hllc":
        pytest.skip("the bubble is configured with hllc")
    for nx, ny in SIZES:
        if problem == "bubble" and (nx < 16 or ny < 4):
            continue  # refused by the configuration
        if problem == "blob" and min(nx, ny) < 2:
            continue  # the torch step wraps two cells of a periodic axis
        torch, settings, u, g, dt, step = _setup(problem, nx, ny, riemann, limiter)
        v = u.clone().requires_grad_(True)
        (want,) = torch.autograd.grad(step(v), v, g)
        got = torch.empty_like(u)
        torch.cuda.synchronize()
        with api.Context(settings) as ctx:
            _vjp(ctx, u, dt, g, got)
            again = torch.empty_like(u)
            _vjp(ctx, u, dt, g, again)
        assert torch.equal(got, again)  # gathered in a fixed order
        err = float((got - want).abs().max() / want.abs().max())
        assert err <= 2.0e-12, (nx, ny, err)


def test_vjp_result_on_the_state(gpu):
    """g_u0 may be u0's own array: the result goes through the scratch."""
    torch, settings, u, g, dt, _ = _setup("blob", 70, 45, "hllc", "minmod")
    want = torch.empty_like(u)
    torch.cuda.synchronize()
    with api.Context(settings) as ctx:
        _vjp(ctx, u, dt, g, want)
        _vjp(ctx, u, dt, g, u)
    assert torch.equal(u, want)
