"""Supersonic faces at the ends of the number range, strips and 16x16 tiles
against the 32x8 tiles, which take every branch as the reference does.

A supersonic face's flux is the upwind side's physical flux.  Extreme scales:
densities whose product leaves the double range while g p rho stays inside it
(the Roe averages of the HLLC-P flux overflow or underflow there).  Cold flow:
the acoustic speed is below half a unit in the last place of the velocity, so
that the wave speed equals the flow's, with a faster stream ahead; such a
pressure is the residue of E - rho u^2 / 2 on rows built for it."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config
from tests.golden_io import state_rel_err

pytestmark = pytest.mark.gpu


def _step(u, riemann, order, gamma, dt, tile):
    ny, nx = u.shape[1:]
    cfg = read_config(f"amr.n_cell={nx} {ny}\neuler.spatial_order={order}\neuler.riemann={riemann}\neuler.gamma={gamma}\n"
                      "geometry.is_periodic=1 1\neuler.problem=advection_blob\nstop_time=10\nmax_step=10\n").cfg
    with api.Context(cfg, tile_y=tile) as ctx:
        ctx.upload(u)
        api.euler_fv_one_step(ctx, dt, 0.0)
        return ctx.download()


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("riemann", ["hllc", "lowmach_hllc", "xie_am_hllc_p"])
@pytest.mark.parametrize("rho,p,speed", [(1e-155, 1e-150, 1e3), (1e155, 1e143, 1.0), (1.0, 1.0, 4.0)])
def test_extreme_densities(gpu, rho, p, speed, riemann, tile):
    rng = np.random.default_rng(5)
    s = [1.0 + 0.1 * rng.random((40, 70)) for _ in range(4)]
    r, u, v, q = rho * s[0], speed * s[1], 0.9 * speed * s[2], p * s[3]
    w = np.stack([r, r * u, r * v, q / 0.4 + 0.5 * r * (u * u + v * v)])
    dt = 0.1 / (70 * 3.0 * speed)
    want = _step(w, riemann, 2, 1.4, dt, 8)
    assert np.isfinite(want).all()
    got = _step(w, riemann, 2, 1.4, dt, tile)
    # a few hundred roundings a cell, the pressure's cancelling against the kinetic energy's square
    assert state_rel_err(got / np.abs(want).max(axis=(1, 2), keepdims=True),
                         want / np.abs(want).max(axis=(1, 2), keepdims=True)) <= 1e-12


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("riemann", ["hllc", "lowmach_hllc", "xie_am_hllc_p"])
def test_cold_flow(gpu, riemann, tile):
    """rho = 1 + a 2^-52, rho u = 1: E = rho u^2 / 2 to working precision leaves
    a residue of about a^2 2^-105, three rows to a state: the middle row's
    y-faces are one and the same, so its update is its x-faces' alone."""
    ulp, nx = 2.0 ** -52, 33
    rows = []
    for a in range(1, 25):
        for b in range(-2, 3):
            rows += [(1.0 + a * ulp, 1.0, 0.0, 0.5 * (1.0 - a * ulp) + 0.25 * b * ulp)] * 3
    w = np.repeat(np.array(rows).T[:, :, None], nx, axis=2)
    w[:, :, 16:] = np.array([1.0, 2.0, 0.0, 0.1 / 0.001 + 2.0])[:, None, None]
    want, got = (_step(w, riemann, 1, 1.001, 1e-4, t) for t in (8, tile))
    w, want, got = w[:, 1::3], want[:, 1::3], got[:, 1::3]
    fine = np.isfinite(want)
    assert fine.any()
    assert np.isfinite(got)[fine].all()
    # the bound of the strips against the tiles, over each field's largest value
    scale = np.broadcast_to(np.abs(w).max(axis=(1, 2), keepdims=True) + 1.0, w.shape)
    assert (np.abs(got - want) / scale)[fine].max() <= (3e-13 if riemann == "xie_am_hllc_p" else 1e-13)
