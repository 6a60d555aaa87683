"""The sketch as the RSVD draws it (pg::omega_device) is the reference's, bit for bit: every value
against the sequential std:: fill."""
import ctypes

import numpy as np
import pytest

import pcaone_b200 as pb
from oracle import pcaone_oracle as O

pytestmark = pytest.mark.gpu


def drawn(gpu, seed, rand, N, l):
    torch = pytest.importorskip("torch")
    npad = (N + 255) // 256 * 256
    d = torch.full((npad, l), float("nan"), dtype=torch.float64, device="cuda")
    f = torch.full((npad, l), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    fn = getattr(pb.lib(), "_ZN2pg12omega_deviceEP10pcaone_ctxiimimPdPf")
    fn.restype = None
    fn(gpu._h, ctypes.c_int(seed), ctypes.c_int(rand), ctypes.c_uint64(N), ctypes.c_int(l), ctypes.c_uint64(npad),
       ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(f.data_ptr()))
    torch.cuda.synchronize()
    return d.cpu().numpy(), f.cpu().numpy()


# one value, the largest fill of the host and the next, odd counts, several CTAs, above the size at which
# pcaone_omega itself draws in parallel
@pytest.mark.parametrize("N,l", [(1, 1), (64, 64), (241, 17), (1001, 21), (4099, 16), (20000, 40)])
@pytest.mark.parametrize("seed", [101, 0, 2147483647, -5])
@pytest.mark.parametrize("rand", [1, 0])
def test_sketch_is_the_sequential_fill(gpu, N, l, seed, rand):
    ref = O.omega(seed, N, l, rand)
    d, f = drawn(gpu, seed, rand, N, l)
    np.testing.assert_array_equal(d[:N], ref)
    assert not np.signbit(d[:N][ref == 0]).any()
    np.testing.assert_array_equal(f[:N], ref.astype(np.float32))
    assert not d[N:].any() and not f[N:].any()
    np.testing.assert_array_equal(pb.omega(seed, N, l, rand), ref)
