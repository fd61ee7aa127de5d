"""Staged tiles with halo capacities that leave the local lists behind arrays of odd length, against
gathers from global memory, bit for bit (the offsets themselves are asserted when the library is
compiled)."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [701, 702, 703, 1001, 2047])
def test_staged_tiles_of_any_capacity(cap):
    sc = S.jc_compression(R=0.006, H=0.012)
    opts = {"return_map": 1, "thermal": 1, "taylor_quinney": 0.9, "rebuild_every": 5,
            "rebuild_current_positions": 1, "rebuild_after_yield": 0, "precision": 1}
    runs = []
    for staging in (1, 0):
        d = S.load(Domain_d(sc["n"]), sc, dict(opts, tile_staging=staging, tile_cap_max=cap))
        d.step(12)
        runs.append({f: d.get_field(f) for f in ("x", "v", "shearstress", "pl_strain", "T", "rho")})
        if staging:
            assert d.get_scalar("tiles_staged") > 0
    for f in runs[0]:
        assert np.array_equal(runs[0][f], runs[1][f]), f
