"""A rebuild that is refused (a grid of more than 2e9 cells) leaves the domain as it was before the
step that asked for it, with rebuilds that the host sees only behind the captured steps (graph 1)
as with those it waits for (graph 0)."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S
from weldformgpu_gb300.domain import WeldformError

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "rho", "sigma", "pl_strain", "T")
SCALARS = ("time", "step", "isfirst", "is_yielding", "rebuilds")


def _domain(precision, graph, far=None):
    sc = S.compression_cylinder(R=0.0024, H=0.0045, generator="lattice", jitter=0.02, vz_top=-60.0)
    sc["k"], sc["cp"] = 167.0, 896.0
    if far:                                  # one particle off the body, a zone of its own
        sc["x"], sc["ids"] = np.array(sc["x"]), np.array(sc["ids"])
        sc["x"][0] = sc["x"].max(axis=0) + 0.02
        sc["ids"][0] = 9
        sc["bcs"] = list(sc["bcs"]) + [(9, (far, far, far))]
    return S.load(Domain_d(sc["n"]), sc, {"precision": precision, "graph": graph, "thermal": 1,
                                          "rebuild_every": 3, "rebuild_after_yield": 0,
                                          "rebuild_current_positions": 1}), sc


def _refused(d, call):
    with pytest.raises(WeldformError, match="grid too large"):
        call(d)


def _same(a, b):
    for s in SCALARS:
        assert a.get_scalar(s) == b.get_scalar(s), s
    for f in FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f), equal_nan=True), f


@pytest.mark.parametrize("precision", [0, 1])
def test_positions_that_no_grid_covers(precision):
    (g, _), (w, _) = _domain(precision, 1), _domain(precision, 0)
    for d in (g, w):
        d.step(3)
    x = g.get_field("x")
    far = x.copy()
    far[0] = 100.0
    for d in (g, w):
        d.set_positions(far)
    for _ in range(2):                       # refused again and again
        for d in (g, w):
            _refused(d, lambda d: d.step(4))
        assert g.get_scalar("step") == 3
        _same(g, w)
    for d in (g, w):
        d.set_positions(x)
        d.step(5)
    _same(g, w)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("solve", [False, True])
def test_a_body_that_outgrows_every_grid_inside_a_call(precision, solve):
    """A particle that moves away: more than 2e9 cells at the second rebuild, three steps on."""
    sc = _domain(0, 0)[1]
    h, dt = sc["h"], sc["dt"]
    far = 3000.0 * 2.0 * h / (3.0 * dt)
    (g, _), (w, _) = _domain(precision, 1, far), _domain(precision, 0, far)
    for d in (g, w):
        _refused(d, lambda d: d.mech_fraser_solve(11.5 * dt, 2.0 * dt) if solve else d.step(12))
    assert g.get_scalar("step") == 3
    _same(g, w)
    a, b = g.get_output_series(), w.get_output_series()
    assert np.array_equal(a, b, equal_nan=True) and len(a) == (1 if solve else 0)
