"""Device memory that a set-up holds at its peak (GPU)."""
import ctypes as C

import pytest

import mgcfd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

USED_CURRENT, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh


@pytest.fixture(scope="module")
def pool():
    """(get, set) of an attribute of the device's default memory pool."""
    torch.zeros(1, device="cuda")
    path = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line)
    rt = C.CDLL(path)
    handle = C.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(handle), 0) == 0

    def get(attr):
        v = C.c_uint64()
        assert rt.cudaMemPoolGetAttribute(handle, attr, C.byref(v)) == 0
        return v.value

    def reset_high():
        assert rt.cudaMemPoolSetAttribute(handle, USED_HIGH, C.byref(C.c_uint64(0))) == 0

    return get, reset_high


# One stream, two streams (from 8192 level-0 nodes), and one with the lists of the fused stage.
@pytest.mark.parametrize("n,nl", [(8, 3), (21, 3), (40, 4)])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "dw"])
def test_scratch_of_two_streams_is_little_more_than_one_chunk(pool, n, nl, precision):
    """Beyond what the solver keeps, a set-up holds one chunk of 64 MiB and what its
    coarse levels need: on a lattice (three edges a node) at most 69 + 3 * 180 and
    up to 60 bytes for each of the surface's entries, so 900 bytes for each of the
    n^3 / 7 coarse nodes (a little more of odd extents: n^3 / 5), and 1 MiB of
    rounding."""
    get, reset_high = pool
    mesh = mgcfd.HostMesh.generate(n, nl, 5)
    torch.cuda.synchronize()
    before = get(USED_CURRENT)
    reset_high()
    s = mgcfd.Solver(mesh, 0.5, 3.0, precision=precision)
    peak, kept = get(USED_HIGH) - before, s.stats().device_bytes
    s.close()
    assert peak - kept < (64 << 20) + 900 * n ** 3 // 5 + (1 << 20), (peak, kept)
