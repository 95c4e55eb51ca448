"""Device arrays that end before the field does: refused on the host, before a
kernel or a copy could run past their allocation."""
import ctypes

import numpy as np
import pytest

from gpe_b200 import GpeError, GpeParams, GpeSolver
from gpe_b200._lib import check, lib

pytestmark = pytest.mark.gpu

runtime = pytest.importorskip("cuda.bindings.runtime")


class Allocation:
    """An allocation of its own (torch's tensors share larger ones)."""

    def __init__(self, nbytes):
        err, self.ptr = runtime.cudaMalloc(nbytes)
        assert err == runtime.cudaError_t.cudaSuccess

    def __enter__(self):
        return int(self.ptr)

    def __exit__(self, *a):
        runtime.cudaFree(self.ptr)


@pytest.mark.parametrize("precision,elem", [(8, 8), (16, 16), (8, 16)])
def test_array_that_ends_beyond_its_allocation(precision, elem):
    n = 48
    prm = GpeParams(nx=n, ny=n, nz=n, xr=3.0, yr=3.0, zr=3.0, precision=precision)
    a = np.ones((n, n, n), dtype=np.complex128)
    need = a.size * elem
    with GpeSolver(prm, dt=0.01) as s:
        s.set_state(a)
        # not a multiple of any granule, so that nothing starts where it ends
        with Allocation(need // 2 + 4) as p:
            for call in (lib().gpe_gpu_set_state_device, lib().gpe_gpu_get_state_device):
                with pytest.raises(GpeError, match="ends beyond its allocation"):
                    check(call(s.handle, ctypes.c_void_p(p), elem), s.handle)
        assert np.array_equal(s.get_state(), a)
        # a whole one is taken, at its start and at an offset that still fits
        with Allocation(need + elem) as p:
            for at in (p, p + elem):
                check(lib().gpe_gpu_get_state_device(s.handle, ctypes.c_void_p(at), elem), s.handle)
                s.set_state(0.0 * a)
                check(lib().gpe_gpu_set_state_device(s.handle, ctypes.c_void_p(at), elem), s.handle)
                assert np.array_equal(s.get_state(), a)
            with pytest.raises(GpeError, match="ends beyond its allocation"):
                check(lib().gpe_gpu_set_state_device(s.handle, ctypes.c_void_p(p + 2 * elem), elem),
                      s.handle)
