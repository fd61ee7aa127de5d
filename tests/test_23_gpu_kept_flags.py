"""What a stepping call notes for its own steps (no massive particle in a tool's zone, the largest
strain increment) does not enter the next call: `mech_fraser_solve` behind another call against the
same calls with an empty `step(0)` between them, which drops all of it."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "u", "rho", "sigma", "pl_strain", "T", "contforce")


def _block(rebuild=0.02):
    sc = S.indent_block(L=(0.006, 0.006, 0.002), R=0.003, v_tool=-40.0, rebuild_increment=rebuild)
    sc["mesh"]["nodes"] = sc["mesh"]["nodes"] - np.array([0.0, 0.0, 2.0e-5])
    return sc


def _state(d):
    out = {f: d.get_field(f) for f in FIELDS}
    out["rebuilds"] = d.get_scalar("rebuilds")
    return out


def _same(a, b):
    for f in a:
        assert np.array_equal(a[f], b[f]), f


def _zone_ids(sc):
    """Solid particles inside the block carry the tool's zone id."""
    ids = np.array(sc["ids"])
    x = sc["x"][:sc["n_solid"]]
    inner = (np.abs(x[:, 2] - 0.0010) < 0.0002) & (x[:, 0] > 0.004)
    ids[:sc["n_solid"]][inner] = sc["mesh"]["zone"]
    assert inner.sum() > 20
    return ids


@pytest.mark.parametrize("first", ["step", "mech_fraser_solve"])
def test_zone_filter_after_ids_changed_between_two_calls(first):
    sc = _block()
    tf = 19.5 * sc["dt"]

    def run(ids, drop):
        d = S.load(Domain_d(sc["n"]), sc, {"precision": 1, "energy_mode": 1})
        if first == "step":
            d.step(4)
        else:
            d.mech_fraser_solve(3.5 * sc["dt"], 1.0)
        d.set_id(ids)
        if drop:
            d.step(0)
        d.mech_fraser_solve(tf, 1.0)
        return _state(d)

    ids = _zone_ids(sc)
    a = run(ids, False)
    _same(a, run(ids, True))
    free = run(sc["ids"], False)
    assert np.linalg.norm(free["sigma"] - a["sigma"]) > 1e-2 * np.linalg.norm(a["sigma"])


def test_strain_maximum_is_not_the_last_calls():
    """A call that ends with strains above the increment: the next solve starts from new lists."""
    sc = _block(rebuild=1.0)

    def run(drop):
        d = S.load(Domain_d(sc["n"]), sc, {"precision": 1, "energy_mode": 1, "thermal": 0})
        d.step(120)
        assert d.get_scalar("rebuilds") == 0 and d.get_field("pl_strain").max() > 0.002
        d.set_option("rebuild_strain_increment", 0.002)
        if drop:
            d.step(0)
        d.mech_fraser_solve(2.5 * sc["dt"], 1.0)
        return _state(d)

    a = run(False)
    assert a["rebuilds"] == 0
    _same(a, run(True))


def test_strain_maximum_of_the_mixed_form_is_not_the_plain_forms():
    """Adaptive rebuilds of the plain form behind a mixed call follow the plain form's strains."""
    sc = _block(rebuild=0.001)

    def run(drop):
        d = S.load(Domain_d(sc["n"]), sc, {"precision": 1, "energy_mode": 1, "thermal": 0})
        d.step(60)
        r0 = d.get_scalar("rebuilds")
        d.set_option("precision", 0)
        d.set_option("resume", 1)
        if drop:
            d.step(0)
        d.mech_fraser_solve(179.5 * sc["dt"], 1.0)
        return _state(d), d.get_scalar("rebuilds") - r0

    (a, ra), (b, rb) = run(False), run(True)
    assert 2 <= rb < 120                     # not at every step
    assert ra == rb
    _same(a, b)
