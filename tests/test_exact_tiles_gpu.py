"""The exact build's 32x8 and 32x16 tiles against the reference's outputs, bit for
bit (the default exact step runs on column strips, the HLLC-P flux's apart)."""
import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import api
from amrex_euler_allmach_explicit_imex_b200.config import read_config
from tests import golden_io

pytestmark = pytest.mark.gpu

CASES = list(golden_io.explicit_cases())


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("key,case", CASES, ids=[k for k, _ in CASES])
def test_tiles_equal_the_reference(gpu, key, case, tile):
    cfg = read_config(golden_io.kv_of(case["kv"])).cfg
    with api.Context(cfg, arith="exact", tile_y=tile) as ctx:
        ctx.upload(case["u0"])
        deg = api.euler_fv_one_step(ctx, float(case["dt"]), float(case["t"]))
        assert np.array_equal(ctx.download(), case["u1"])
        assert api.compute_euler_dt(ctx, float(case["t"])) == float(case["edt"])
        d = api.compute_diagnostics(ctx)
    assert deg == int(case["deg"])
    assert [d.rho_min, d.pressure_min, d.nonfinite_count] == list(case["diag"])
