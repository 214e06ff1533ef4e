"""The device loop's captured graphs do not pile up.

A driver that advances a context to one output time after another gives ecg_run
a new stop time, or a new step limit, on every call.  The graphs of a run depend
on neither, so the device memory they hold stops growing; and a limit given to a
graph that an earlier run captured is the limit that counts."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config

pytestmark = pytest.mark.gpu

KV = ("amr.n_cell=48 20\ngeometry.is_periodic=1 1\neuler.problem=advection_blob\neuler.cfl=0.4\n"
      "stop_time=1000\nmax_step=1000\n")


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def test_successive_output_times_hold_no_more_memory(gpu):
    cfg = read_config(KV).cfg
    with api.Context(cfg) as ctx:
        api.initialize_state(ctx)
        api.run(ctx, 3, cfg.stop_time)
        free = []
        for call in range(1200):
            r = api.run(ctx, 2 + call % 2, 900.0 + 1.0e-3 * call)
            assert r.steps == 2 + call % 2
            if call in (100, 1199):
                free.append(_free())
    assert free[0] - free[1] <= 4 << 20


@pytest.mark.parametrize("arith", ["fast", "exact"])
def test_limits_of_later_runs(gpu, arith):
    cfg = read_config(KV).cfg
    with api.Context(cfg, arith=arith) as ctx, api.Context(cfg, arith=arith) as one:
        api.initialize_state(ctx)
        u = ctx.download()
        # each call replays graphs of the ones before with its own limits
        t36 = None
        for steps, stop in [(70, 1000.0), (40, 1000.0), (64, 1000.0), (36, 1000.0), (64, "t36"), (8, 1000.0),
                            (100, "t36"), (70, 0.02), (3, 0.02), (100, 0.0)]:
            stop = t36 if stop == "t36" else stop
            ctx.upload(u)
            r = api.run(ctx, steps, stop)
            one.upload(u)
            t, n = 0.0, 0
            while n < steps and t < stop - 1.0e-14:
                dt = min(api.compute_euler_dt(one, t), stop - t)
                api.euler_fv_one_step(one, dt, t)
                t += dt
                n += 1
            assert (r.steps, r.time, r.failed) == (n, t, 0), (steps, stop)
            assert np.array_equal(ctx.download(), one.download())
            if steps == 36:
                t36 = t
