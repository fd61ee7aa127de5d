"""Contact law 1 in the mixed form: the fused acceleration + integration pass with a warp per slot
near the tool, the zone filter left out and the running maximum of the strain increments, against
the general paths (separate passes, one-step calls), bit for bit."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "u", "a", "rho", "sigma", "pl_strain", "int_energy", "T", "contforce", "fric_heat")


def _block(omega=0.0, level=3, rebuild=0.02):
    sc = S.indent_block(L=(0.006, 0.006, 0.002), R=0.003, level=level, v_tool=-40.0, omega=omega,
                        rebuild_increment=rebuild)
    sc["mesh"]["nodes"] = sc["mesh"]["nodes"] - np.array([0.0, 0.0, 2.0e-5])
    return sc


def _run(sc, calls, **opts):
    d = S.load(Domain_d(sc["n"]), sc, dict({"precision": 1, "energy_mode": 1}, **opts))
    for k in calls:
        d.step(k)
    out = {f: d.get_field(f) for f in FIELDS}
    out["rebuilds"] = d.get_scalar("rebuilds")
    out["tests"] = (d.get_scalar("contact_tests32"), d.get_scalar("contact_tests64"))
    out["contacts"] = d.get_field_i32("cont_count")
    return out


def _same(a, b):
    for f in a:
        assert np.array_equal(a[f], b[f]), f


# tools of 40 triangles (fewer than a warp has lanes in any cell), 656 and 2,600 (several rounds of
# 32 in a cell); spinning tools are binned on the GPU in an order that changes from run to run
@pytest.mark.parametrize("omega", [0.0, 2000.0])
@pytest.mark.parametrize("level", [1, 3, 5])
def test_fused_contact_equals_separate_passes(level, omega):
    sc = _block(omega, level)
    a = _run(sc, (40,))
    assert a["contacts"].sum() > 0 and a["tests"][1] > 0
    _same(a, _run(sc, (40,), fuse_integrate=0))


def test_running_strain_maximum_rebuilds_when_the_full_one_does():
    """Every step of a one-step call reduces all strains; a long call keeps the maximum up.  (No heat:
    a call's last heat pass is a kernel of its own, whose temperatures differ in the last bit.)"""
    sc = _block(rebuild=0.001)
    a, b = _run(sc, (120,), thermal=0), _run(sc, (1,) * 120, thermal=0)
    assert a["rebuilds"] >= 3
    _same(a, b)


def test_zone_filter_still_acts_on_massive_particles_of_the_zone():
    """Solid particles that carry the mesh's zone id take no part in the pair sums of the others:
    the mixed form follows the plain one, whose filter is pinned by the oracle."""
    sc = _block()
    ids = np.array(sc["ids"])
    inner = (np.abs(sc["x"][:sc["n_solid"], 2] - 0.0010) < 0.0002) & (sc["x"][:sc["n_solid"], 0] > 0.004)
    ids[:sc["n_solid"]][inner] = sc["mesh"]["zone"]
    assert inner.sum() > 20
    sc["ids"] = ids
    m = _run(sc, (30,))
    p = _run(sc, (30,), precision=0)
    for f in ("u", "v", "rho", "sigma", "contforce"):
        assert np.linalg.norm(m[f] - p[f]) <= 1e-3 * np.linalg.norm(p[f]), f
    # and it is not the unfiltered answer
    free = _run(_block(), (30,))
    assert np.linalg.norm(free["sigma"] - p["sigma"]) > 1e-2 * np.linalg.norm(p["sigma"])
