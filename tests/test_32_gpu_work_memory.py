"""The pair work arrays of the plain form (1.2 KB a particle) stay in the cache behind a destroyed
domain and go to the next one only when it asks for them; option pair_cache 0 frees them."""
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S
from weldformgpu_gb300.domain import release_cache

pytestmark = pytest.mark.gpu


def _free():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_mixed_domain_does_not_hold_the_last_domains_work_arrays():
    _free()
    release_cache()
    sc = S.compression_cylinder(R=0.0107, H=0.0214, generator="lattice")
    n = sc["n"]
    a = S.load(Domain_d(n), sc, {"precision": 0})
    a.step(1)
    a.close()
    before = _free()
    b = S.load(Domain_d(n), sc, {"precision": 1})
    b.step(2)
    held = _free()
    assert before - held < 400 * n           # arena and cells come from the cache (not the series)
    release_cache()
    assert _free() - held > 1150 * n         # the work arrays were still there to be freed
    b.close()


def test_a_plain_domain_takes_the_last_domains_work_arrays():
    _free()
    release_cache()
    sc = S.compression_cylinder(R=0.0107, H=0.0214, generator="lattice")
    a = S.load(Domain_d(sc["n"]), sc, {"precision": 0})
    a.step(1)
    x = a.get_field("a")
    a.close()
    before = _free()
    b = S.load(Domain_d(sc["n"]), sc, {"precision": 0})
    b.step(1)
    held = _free()
    assert before - held < 400 * sc["n"]
    assert (b.get_field("a") == x).all()
    release_cache()
    assert _free() == held                   # b holds all of it
    b.close()


def test_work_arrays_outlast_a_mixed_domain_in_between():
    _free()
    release_cache()
    sc = S.compression_cylinder(R=0.0107, H=0.0214, generator="lattice")
    for precision in (0, 1):
        d = S.load(Domain_d(sc["n"]), sc, {"precision": precision})
        d.step(1)
        d.close()
    before = _free()
    d = S.load(Domain_d(sc["n"]), sc, {"precision": 0})
    d.step(1)
    assert before - _free() < 400 * sc["n"]
    d.close()
    before = _free()
    release_cache()
    assert _free() - before > 1150 * sc["n"]     # one block, and it goes with the cache


def test_the_option_frees_the_work_arrays():
    _free()
    release_cache()
    sc = S.compression_cylinder(R=0.0107, H=0.0214, generator="lattice")
    a = S.load(Domain_d(sc["n"]), sc, {"precision": 0})
    b = S.load(Domain_d(sc["n"]), sc, {"precision": 0})
    for d in (a, b):
        d.step(2)
    held = _free()
    a.set_option("pair_cache", 0)
    assert _free() - held > 1150 * sc["n"]
    a.step(1)
    a.set_option("pair_cache", 1)
    for d, k in ((a, 2), (b, 3)):
        d.step(k)
    assert abs(_free() - held) < 100 * sc["n"]
    for f in ("x", "v", "sigma"):
        assert (a.get_field(f) == b.get_field(f)).all(), f
    a.close()
    b.close()
