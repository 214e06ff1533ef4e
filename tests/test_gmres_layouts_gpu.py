"""The pressure solve's shared-memory layouts at their edges: accumulator
entries apart up to 512 rows a block and packed above (75776 rows are 512 on 148
blocks, 75924 are 514), w in shared memory where no basis vector is resident (FP64
from some 120000 rows, the FP32 basis at 512 x 512; odd sizes take the one-row
sweeps), each with the default and the fixed-order sums.

One IMEX step of the Gresho vortex at M = 0.1 is held to the oracle's, at the
bound of the other large-grid tests; fixed-order solves repeat bit for bit."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config
from tests import golden_io

pytestmark = pytest.mark.gpu


def _step(cfg, u0, dt, prec, deterministic):
    with api.Context(cfg, imex_precision=prec, deterministic=deterministic) as ctx:
        ctx.upload(u0)
        d = api.euler_imex_bdltv20_o1_source_map_picard_one_step(ctx, dt)
        assert d.solver_status in (1, 2), api.solver_status_str(d.solver_status)
        assert min(d.pressure_linear_residual_relative_linf, d.pressure_linear_residual_linf) <= cfg.imex_solver_tol
        return ctx.download()


@pytest.mark.parametrize("grid", [(256, 296), (228, 333), (384, 352), (512, 512), (513, 511)])
def test_layouts_against_oracle(gpu, oracle, grid):
    c = golden_io.imex_case("gresho_m0p1")
    kv = dict(l.split("=", 1) for l in golden_io.kv_of(c["kv"]).split("\n"))
    kv["amr.n_cell"] = f"{grid[0]} {grid[1]}"
    kv["geometry.prob_hi"] = f"1 {grid[1] / grid[0]!r}"
    cfg = read_config(kv).cfg
    u0 = oracle.initialize(cfg)
    dt, _ = oracle.imex_dt(cfg, u0, 0.0)
    want, d = oracle.imex_step(cfg, u0, dt)
    assert d.solver_status in (1, 2)
    for prec in ("fp64", "mixed"):
        for deterministic in (0, 1):
            got = _step(cfg, u0, dt, prec, deterministic)
            assert golden_io.state_rel_err(got, want) <= 1e-9, (prec, deterministic)
            if deterministic:
                assert np.array_equal(got, _step(cfg, u0, dt, prec, 1)), prec
