"""Fields read back straight into page-locked memory against fields read back through the staging
buffer, at sizes around a block of the gather, at unaligned places of a larger allocation, and in
host memory that the caller registered."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = {"u": 3, "v": 3, "rho": 1, "sigma": 6, "shearstress": 6, "pl_strain": 1, "T": 1, "p": 1}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("R,H", [(0.0010, 0.0015), (0.0041, 0.0073)])
def test_read_back_into_page_locked_memory(precision, R, H):
    torch = pytest.importorskip("torch")
    sc = S.jc_compression(R=R, H=H, vz_top=-2.0)
    d = S.load(Domain_d(sc["n"]), sc, {"precision": precision, "return_map": 1})
    n = sc["n"]
    pinned = torch.full((6 * n + 37,), -7.0, dtype=torch.float64, pin_memory=True).numpy()
    own = np.full(6 * n + 37, -7.0)
    assert int(torch.cuda.cudart().cudaHostRegister(own.ctypes.data, own.nbytes, 0)) == 0
    try:
        for k in (0, 3):                 # before the first step and after some
            if k:
                d.step(k)
            for f, c in FIELDS.items():
                want = d.get_field(f).ravel()
                for buf in (pinned, own):
                    for at in (0, 5):
                        buf[:] = -7.0
                        d.get_field(f, out=buf[at:at + c * n])
                        assert np.array_equal(buf[at:at + c * n], want), f
                        assert (buf[:at] == -7.0).all() and (buf[at + c * n:] == -7.0).all(), f
    finally:
        torch.cuda.cudart().cudaHostUnregister(own.ctypes.data)
