"""Column strips of several rows against the tile kernels.

A warp carries the y-face below a row, the face state above it and, for the
HLLC-P flux, pressure ratios from row to row; its rows live in a ring of eight
conserved and four primitive rows.  With one row a strip none of that is used
twice, so the rows a warp takes are given here (tile_x): fewer than the rings
hold, as many, one more, the counts the library itself takes on large grids, and
more than the grid has; on heights they do not divide.  Exact arithmetic: bit for
bit the 32x16 tiles.  Fast arithmetic: the bound of the strips against the 16x16
tiles (a few hundred roundings a cell below 1e-13 of the field, 3e-13 for the
HLLC-P flux, whose tiles and strips are the same up to association).  The last
test does both at full size with the library's own choice of rows."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200.config import read_config
from tests.golden_io import state_rel_err
from tests.test_strips_gpu import PROBLEMS, _state, _step

pytestmark = pytest.mark.gpu

ROWS = [1, 2, 3, 5, 8, 9, 26, 100]
SIZES = [(57, 33), (30, 70)]


def _cfg(problem, nx, ny, riemann, limiter, order=2):
    return read_config(f"amr.n_cell={nx} {ny}\neuler.spatial_order={order}\neuler.riemann={riemann}\n"
                       f"euler.slope_limiter={limiter}\nstop_time=10\nmax_step=1000\n" + PROBLEMS[problem]).cfg


def _dt(cfg):
    return 0.1 * min((cfg.prob_hi[n] - cfg.prob_lo[n]) / cfg.n_cell[n] for n in (0, 1))


def _same(a, b):
    return np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("riemann,limiter", [("hllc", "minmod"), ("lowmach_hllc", "vanleer"), ("rusanov", "mc"),
                                             ("xie_am_hllc_p", "minmod")])
@pytest.mark.parametrize("problem", sorted(PROBLEMS))
def test_rows_a_strip(gpu, problem, riemann, limiter):
    if problem in ("bubble", "walls") and riemann not in ("hllc", "xie_am_hllc_p"):
        pytest.skip("not a configuration of the bubble")
    for k, (nx, ny) in enumerate(SIZES):
        cfg = _cfg(problem, nx, ny, riemann, limiter)
        u, dt = _state(nx, ny, 40 + k), _dt(cfg)
        exact, tiles = _step(cfg, u, dt, arith="exact", tile_y=16), _step(cfg, u, dt, tile_y=1)
        for rows in ROWS:
            assert _same(_step(cfg, u, dt, arith="exact", tile_x=rows), exact), (nx, ny, rows)
            f = _step(cfg, u, dt, tile_x=rows)
            assert state_rel_err(f[0], tiles[0]) <= (3e-13 if riemann == "xie_am_hllc_p" else 1e-13), (nx, ny, rows)
            assert f[1] == tiles[1] and f[2][2] == tiles[2][2], (nx, ny, rows)


@pytest.mark.parametrize("rows", [1, 3, 8, 26, 100])
def test_degenerate_faces_count_once_a_cell(gpu, rows):
    """A state of rest and vacuum-thin columns: degenerate star states in the
    middle of strips, on their edges and on the rows between strips."""
    cfg = _cfg("outflow", 57, 33, "hllc", "minmod")
    u = _state(57, 33, 3)
    u[:, ::3, :] = np.array([1e-14, 0.0, 0.0, 1e-14])[:, None, None]
    u[:, :, 26:31] = np.array([1e-14, 0.0, 0.0, 1e-14])[:, None, None]
    dt = 1e-3 * _dt(cfg)
    want = _step(cfg, u, dt, arith="exact", tile_y=16)
    assert want[1] > 100
    assert _step(cfg, u, dt, arith="exact", tile_x=rows)[1] == want[1]
    assert _step(cfg, u, dt, tile_x=rows)[1] == _step(cfg, u, dt, tile_y=1)[1]


@pytest.mark.parametrize("riemann", ["hllc", "lowmach_hllc", "rusanov", "xie_am_hllc_p"])
def test_full_size(gpu, riemann):
    problem = "bubble" if riemann in ("hllc", "xie_am_hllc_p") else "mixed"
    cfg = _cfg(problem, 2560, 640, riemann, "minmod")
    u = _state(2560, 640, 8)
    dt = _dt(cfg)
    exact = _step(cfg, u, dt, arith="exact", tile_y=16)
    assert _same(_step(cfg, u, dt, arith="exact"), exact)
    # the fast build's bound on one step against the reference's arithmetic
    assert state_rel_err(_step(cfg, u, dt)[0], exact[0]) <= 1e-12
