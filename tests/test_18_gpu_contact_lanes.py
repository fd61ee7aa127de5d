"""Contact law 0 with 1, 8, 16 and 32 lanes a particle against the oracle, bit for bit: surface
normals, contact lists and the sequence of contact forces, under a moving and a rotating plane."""
import numpy as np
import pytest

from oracle import oracle as O
from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "a", "rho", "sigma", "contforce", "normal")


# 644 slots take 32 lanes, 3,080 16, 10,536 eight, 65,644 one; dens sets the triangles, so
# how many contacts a particle tests (coarse: a few, fine: up to the limit of 20)
@pytest.mark.parametrize("R,H,dens,steps", [(0.0026, 0.0050, 4, 12), (0.0042, 0.0075, 14, 12),
                                            (0.0060, 0.0120, 24, 10), (0.0112, 0.0216, 20, 3),
                                            (0.0112, 0.0216, 20, 10)])
@pytest.mark.parametrize("mu", [(0.0, 0.0), (0.2, 0.1)])
def test_contact_bit_exact_vs_oracle(R, H, dens, steps, mu):
    sc = S.contact_cylinder(R=R, H=H, dens=dens, gap=-2.0e-6, mu=mu)
    if mu[0] > 0.0:
        sc["mesh"]["angvel"] = (3.0, -2.0, 40.0)
    o = S.load(O.OracleDomain(sc["n"]), sc)
    g = S.load(Domain_d(sc["n"]), sc)
    for k in (1, steps - 1):
        o.step(k)
        g.step(k)
        for f in FIELDS:
            assert np.array_equal(g.get_field(f), o.get_field(f), equal_nan=True), f
    if steps > 3:                        # three steps end before the first contact
        assert np.abs(g.get_field("contforce")).max() > 0.0
