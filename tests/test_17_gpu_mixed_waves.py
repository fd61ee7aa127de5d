"""The mixed passes' two compilations, for grids of one wave and larger ones, on both sides of the
lines between them: 38,912 particles for the acceleration pass (two lanes each, four blocks per
SM on 152 SMs) and 77,824 for the others, against plain FP64."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

OPTS = {"return_map": 1, "thermal": 1, "taylor_quinney": 0.9, "rebuild_every": 5,
        "rebuild_current_positions": 1, "rebuild_after_yield": 0, "energy_mode": 1}


# lattice cylinders of 38,883 and 39,880, 77,766 and 78,763 particles; network on or off
@pytest.mark.parametrize("R,layers", [(0.0089, 39), (0.0089, 40), (0.0089, 78), (0.0089, 79)])
@pytest.mark.parametrize("network", [0, 1])
def test_mixed_passes_around_the_wave_lines(R, layers, network):
    from weldformgpu_gb300 import mlp
    sc = S.jc_compression(R=R, H=layers * 0.0005, vz_top=-10.0)
    z = sc["x"][:, 2] / sc["x"][:, 2].max()
    out = []
    for precision in (0, 1):
        d = S.load(Domain_d(sc["n"]), sc, dict(OPTS, precision=precision))
        if precision and network:
            d.set_mlp_weights(mlp.init_params(2))
            d.set_option("mlp", 1)
        d.step(1)
        d.set_field("v", np.outer(z, (0.0, 0.0, -10.0)))        # straining everywhere, part of it
        d.set_field("pl_strain", 0.02 * z)                      # yielding
        d.set_field("shearstress", np.outer(z, np.array([1, 1, -2, 0, 0, 0]) * 1.1e8))
        d.step(6)
        out.append({f: d.get_field(f) for f in ("u", "v", "rho", "sigma", "pl_strain", "T")})
    for f, a in out[0].items():
        b = out[1][f]
        off = 20.0 if f == "T" else 0.0
        assert np.linalg.norm(b - a) <= 1e-3 * np.linalg.norm(a - off), f
