"""Positions whose search grid has more cells than 64 bits count are refused like any grid of more
than 2e9 cells: by the search, by a solve's first rebuild and by one inside the step loop."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S
from weldformgpu_gb300.domain import WeldformError

pytestmark = pytest.mark.gpu


# 2^22 cells an axis are 2^66; 2^20 are 2^60, which 64 bits hold
@pytest.mark.parametrize("cells", [2.0**20, 2.0**22 - 4, 2.0**22, 3.0e6, 1.0e8])
@pytest.mark.parametrize("graph", [0, 1])
def test_refused(cells, graph):
    sc = S.compression_cylinder(R=0.0024, H=0.0045, generator="lattice")
    far = np.array(sc["x"])
    far[0] = far[1] + cells * 2.0 * sc["h"]
    d = S.load(Domain_d(sc["n"]), dict(sc, x=far), {"graph": graph, "rebuild_after_yield": 0})
    for call in (d.find_neighbors, lambda: d.step(3)):
        with pytest.raises(WeldformError, match="grid too large"):
            call()
    d.set_positions(sc["x"])
    d.step(5)
    d.set_positions(far)
    with pytest.raises(WeldformError, match="grid too large"):
        d.step(5)
    assert d.get_scalar("step") == 5
