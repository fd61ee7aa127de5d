"""The scalar `launches` counts the kernels of a contact step: the same steps with every kernel of a
step listed by hand."""
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def _launches(sc, opts, a, b):
    """Kernels of a step, from calls of a and b steps without a rebuild."""
    d = S.load(Domain_d(sc["n"]), sc, opts)
    d.step(1)
    d.step(a)
    l0 = d.get_scalar("launches")
    d.step(a)
    l1 = d.get_scalar("launches")
    d.step(b)
    l2 = d.get_scalar("launches")
    assert d.get_scalar("rebuilds") == 0
    per = ((l2 - l1) - (l1 - l0)) / (b - a)
    return per, (l1 - l0) - a * per


# mixed law 1: density, stress, acceleration with integration, listed contacts, node motion, elements;
# a spinning tool's bins are counted, scanned (one kernel up to 1,024 cells, else three) and filled.
# Separate passes: contact over all slots, and integration with the node motion.  A mixed call
# begins with the zone test and the largest strain increment.  Plain form: density, rates and stress
# point (several lanes a particle), acceleration, contact, integration with the node motion,
# elements, and the strains' maximum in every step.
@pytest.mark.parametrize("precision,omega,fuse,per,call", [
    (1, 0.0, 1, (6,), 2), (1, 0.0, 0, (6,), 2), (1, 2000.0, 1, (9, 11), 2), (0, 0.0, 1, (8,), 0)])
def test_law1(precision, omega, fuse, per, call):
    sc = S.indent_block(L=(0.006, 0.006, 0.002), R=0.003, v_tool=-40.0, omega=omega, thermal=False,
                        rebuild_increment=10.0)
    got = _launches(sc, {"precision": precision, "fuse_integrate": fuse}, 3, 8)
    assert sc["n"] < 64000 and got[0] in per and got[1] == call


def test_law0():
    """The plain form's law 0: the contact list at every fifth step only."""
    sc = S.contact_cylinder(gap=-2.0e-6)
    d = S.load(Domain_d(sc["n"]), sc, {"precision": 0, "rebuild_after_yield": 1})
    d.step(5)
    l0 = d.get_scalar("launches")
    r0 = d.get_scalar("rebuilds")
    d.step(5)
    assert d.get_scalar("rebuilds") == r0
    # density, rates, point, acceleration, surface, force, integration, elements; one list
    assert d.get_scalar("launches") - l0 == 5 * 8 + 1
