"""Fields read back into page-locked memory at any byte address: an array that does not start on a
whole double goes through the staging buffer, as one in pageable memory does."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_read_back_at_every_byte_offset(precision):
    torch = pytest.importorskip("torch")
    sc = S.jc_compression(R=0.0010, H=0.0015, vz_top=-2.0)
    n = sc["n"]
    d = S.load(Domain_d(n), sc, {"precision": precision, "return_map": 1})
    d.step(2)
    raw = torch.zeros(8 * 6 * n + 64, dtype=torch.uint8, pin_memory=True).numpy()
    for f, c in (("sigma", 6), ("u", 3), ("rho", 1)):
        want = d.get_field(f).ravel()
        for at in range(17):
            raw[:] = 0xa5
            out = np.frombuffer(raw.data, dtype=np.float64, count=c * n, offset=at)
            assert out.flags.c_contiguous and out.flags.aligned == ((raw.ctypes.data + at) % 8 == 0)
            d.get_field(f, out=out)
            end = at + 8 * c * n
            assert raw[at:end].tobytes() == want.tobytes(), (f, at)
            assert (raw[:at] == 0xa5).all() and (raw[end:] == 0xa5).all(), (f, at)
