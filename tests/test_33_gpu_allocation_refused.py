"""Allocations for which the device has no memory (refused on the host by an option): the domain
gives its pair work arrays back and goes on with the same results, also where the refusal is noticed
behind captured steps; and when that is not enough the call fails with the state of the last step."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S
from weldformgpu_gb300.domain import WeldformError, release_cache

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "rho", "sigma", "pl_strain", "T", "dTdt")
SCALARS = ("time", "step", "rebuilds", "is_yielding")


def _domain(**opts):
    """A body whose top layer moves ~100 cells away from one rebuild to the next: the cells grow."""
    sc = S.compression_cylinder(R=0.0024, H=0.0045, generator="lattice", jitter=0.02, vz_top=-60.0)
    v = 100.0 * 2.0 * sc["h"] / (3 * sc["dt"])
    sc["bcs"] = [(z, tuple(v if k == 2 and w[2] != 0.0 else w[k] for k in range(3)))
                 for z, w in sc["bcs"]]
    sc["k"], sc["cp"] = 167.0, 896.0
    release_cache()                          # no cells of an earlier, larger domain
    return S.load(Domain_d(sc["n"]), sc, dict(
        {"thermal": 1, "rebuild_every": 3, "rebuild_after_yield": 0, "rebuild_current_positions": 1,
         "output_every_step": 1}, **opts)), sc


def _same(a, b):
    for s in SCALARS:
        assert a.get_scalar(s) == b.get_scalar(s), s
    for f in FIELDS:
        assert np.array_equal(a.get_field(f), b.get_field(f), equal_nan=True), f
    assert np.array_equal(a.get_output_series(), b.get_output_series(), equal_nan=True)


def _call(d, kind, steps, dt):
    if kind == "step":
        d.step(steps)
    elif kind == "time_steps":
        d.time_steps(steps)
    else:
        d.set_option("resume", 1)
        d.mech_fraser_solve(d.get_scalar("time") + (steps - 0.5) * dt, 1.0)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["step", "time_steps", "mech_fraser_solve"])
def test_one_refusal_is_met_by_the_work_arrays(graph, precision, kind):
    a, sc = _domain(graph=graph, precision=precision)
    b, _ = _domain(graph=graph, precision=precision)
    for d in (a, b):
        d.step(2)
    release_cache()
    if precision == 0:
        a.set_option("debug_refuse_allocations", 1)
    for steps in (8, 5):
        for d in (a, b):
            _call(d, kind, steps, sc["dt"])
    _same(a, b)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_more_refusals_end_the_call_at_a_step(graph, precision):
    a, sc = _domain(graph=graph, precision=precision)
    b, _ = _domain(graph=graph, precision=precision)
    for d in (a, b):
        d.step(2)
    a.set_option("debug_refuse_allocations", 100)
    with pytest.raises(WeldformError, match="out of memory"):
        a.step(8)
    done = int(a.get_scalar("step"))
    assert 3 <= done < 10 and done % 3 == 0      # a rebuild's step
    assert a.get_scalar("time") == sum([sc["dt"]] * done)
    with pytest.raises(WeldformError, match="out of memory"):
        a.step(8)
    assert a.get_scalar("step") == done
    a.set_option("debug_refuse_allocations", 0)
    a.step(10 - done)
    b.step(8)
    _same(a, b)


def test_logs_and_meshes_get_the_work_arrays_memory():
    sc = S.jc_compression(R=0.0010, H=0.0015, vz_top=-2.0)
    a = S.load(Domain_d(sc["n"]), sc, {"return_map": 1})
    b = S.load(Domain_d(sc["n"]), sc, {"return_map": 1})
    for d in (a, b):
        d.step(3)
    release_cache()
    a.set_option("debug_refuse_allocations", 1)
    for d in (a, b):
        d.set_option("log_return_map", 100)
        d.step(3)
    for f in ("x", "v", "sigma"):
        assert np.array_equal(a.get_field(f), b.get_field(f)), f
