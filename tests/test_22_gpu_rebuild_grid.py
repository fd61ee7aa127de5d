"""Rebuilds inside the step loop, whose grid is sized on the device, against rebuilds that the host
sizes (graph 0) and against the oracle, bit for bit: bodies that grow past the cells allocated
between two rebuilds, by a little and by much, and bodies that shrink."""
import numpy as np
import pytest

from oracle import oracle as O
from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "rho", "sigma", "pl_strain")


# top layers that move away by 0, ~2, ~10 and ~100 cells a rebuild, and into the body
@pytest.mark.parametrize("cells", [0.0, 2.0, 10.0, 100.0, -0.3])
@pytest.mark.parametrize("precision", [0, 1])
def test_grid_follows_the_body(cells, precision):
    sc = S.compression_cylinder(R=0.0024, H=0.0045, generator="lattice", jitter=0.02, vz_top=-60.0)
    v = cells * 2.0 * sc["h"] / (3 * sc["dt"])
    sc["bcs"] = [(z, tuple(v if k == 2 and w[2] != 0.0 else w[k] for k in range(3)))
                 for z, w in sc["bcs"]]
    opts = {"precision": precision, "rebuild_every": 3, "rebuild_after_yield": 0,
            "rebuild_current_positions": 1}
    g = S.load(Domain_d(sc["n"]), sc, opts)
    w = S.load(Domain_d(sc["n"]), sc, dict(opts, graph=0))
    other = [w]
    if precision == 0:
        o = S.load(O.OracleDomain(sc["n"]), sc, {k: x for k, x in opts.items() if k != "precision"})
        other.append(o)
    for steps in (7, 5):
        g.step(steps)
        for r in other:
            r.step(steps)
            for f in FIELDS:
                assert np.array_equal(g.get_field(f), r.get_field(f), equal_nan=True), (f, steps)
    c, l = g.get_neighbors()
    cw, lw = w.get_neighbors()
    assert np.array_equal(c, cw) and np.array_equal(l, lw)
    if cells >= 2.0:
        z = g.get_field("x")[:, 2]
        assert z.max() - z.min() > 0.0045 + 3 * cells * 2.0 * sc["h"]
