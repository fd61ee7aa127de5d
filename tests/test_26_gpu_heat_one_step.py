"""A mixed heat solve of one step computes the pairs as it goes: nothing would be kept for a second
one, so it takes no work arrays from the device."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S
from weldformgpu_gb300.domain import release_cache

pytestmark = pytest.mark.gpu


def test_one_step_takes_no_work_arrays():
    torch = pytest.importorskip("torch")
    release_cache()
    sc = S.heat_box(n_side=47)
    d = S.load_heat(Domain_d(sc["n"]), sc)
    d.set_option("precision", 1)
    d.find_neighbors()                       # the cells are allocated
    free = torch.cuda.mem_get_info()[0]
    d.thermal_solve(0.5 * sc["dt"])
    assert torch.cuda.mem_get_info()[0] == free
    one = [d.get_field(f) for f in ("T", "Ta", "Tb", "dTdt")]
    d.thermal_solve(1.5 * sc["dt"])          # two steps take them
    assert torch.cuda.mem_get_info()[0] < free
    e = S.load_heat(Domain_d(sc["n"]), sc)
    e.set_option("precision", 1)
    e.set_option("pair_cache", 0)
    e.thermal_solve(0.5 * sc["dt"])
    for a, f in zip(one, ("T", "Ta", "Tb", "dTdt")):
        assert np.array_equal(a, e.get_field(f)), f
