"""The device loop with every explicit kernel, against single steps.

The loop's launches overlap (programmatic serialisation): a step is resident
while its predecessor still writes the state, the ghost ring and the records it
will read.  Each kernel, flux and ghost policy must give the state and time of
as many single steps, bit for bit.  35 steps: a chunk of 32 and a tail of 3.
75x40 has fewer than one 16x16 tile an SM; 230x190 has between one and three, where the
fast build takes the tile kernel for the HLLC-P flux."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config

pytestmark = pytest.mark.gpu

KERNELS = [("fast", t) for t in (0, 1, 2, 3, 8, 16)] + [("exact", t) for t in (0, 8, 16)]
PROBLEMS = {
    "ring": "geometry.is_periodic=0 1\neuler.problem=toro1\neuler.field_boundary=exact_dirichlet\n",
    "periodic": "geometry.is_periodic=1 1\neuler.problem=advection_blob\n",
}
STEPS = 35


@pytest.mark.parametrize("arith,tile", KERNELS, ids=[f"{a}-{t}" for a, t in KERNELS])
@pytest.mark.parametrize("riemann", ["hllc", "lowmach_hllc", "rusanov", "xie_am_hllc_p"])
@pytest.mark.parametrize("problem", sorted(PROBLEMS))
def test_run_equals_single_steps(gpu, problem, riemann, arith, tile):
    for n in ((75, 40), (230, 190)):
        cfg = read_config(f"amr.n_cell={n[0]} {n[1]}\neuler.spatial_order=2\neuler.riemann={riemann}\n"
                          "euler.cfl=0.4\nstop_time=10\nmax_step=1000\n" + PROBLEMS[problem]).cfg
        with api.Context(cfg, arith=arith, tile_y=tile) as ctx:
            api.initialize_state(ctx)
            u = ctx.download()
            r = api.run(ctx, STEPS, cfg.stop_time)
            got = ctx.download()
            assert r.steps == STEPS and not r.failed
            ctx.upload(u)
            t = 0.0
            for _ in range(STEPS):
                dt = api.compute_euler_dt(ctx, t)
                api.euler_fv_one_step(ctx, dt, t)
                t += dt
            assert r.time == t and np.array_equal(got, ctx.download()), n
