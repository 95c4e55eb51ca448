"""Device arrays read and written directly by the row kernels: every pairing of
array and field precision, rows of odd and even length, and arrays that start
one element past a 16-byte boundary, against the host-array calls (which go
through the staging buffer).  Conversions round once, so results are equal bit
for bit."""
import numpy as np
import pytest

from gpe_b200 import GpeParams, GpeSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [8, 16])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", [(6, 7, 8), (33, 6, 9), (64, 10, 6), (66, 9, 7)])
@pytest.mark.parametrize("offset", [0, 1])
def test_device_arrays_equal_host_arrays(precision, dtype, n, offset):
    import torch
    rng = np.random.default_rng(sum(n))
    a = (rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1])).astype(dtype)
    td = getattr(torch, dtype)
    flat = torch.zeros(a.size + 2, dtype=td, device="cuda")
    view = flat[offset:offset + a.size].view(n[::-1])
    view.copy_(torch.from_numpy(a))
    for bcs in (1, 2):
        prm = GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=3.0, yr=3.0, zr=3.0, order=4, bcs=bcs,
                        precision=precision)
        with GpeSolver(prm, dt=0.01) as s, GpeSolver(prm, dt=0.01) as h:
            s.set_state(view)
            h.set_state(a)
            assert np.array_equal(s.get_state(dtype), h.get_state(dtype))
            # ghosts too: a step reads them all
            s.solver()
            h.solver()
            out = torch.zeros_like(flat)
            ov = out[offset:offset + a.size].view(n[::-1])
            s.get_state_device(ov)
            assert np.array_equal(ov.cpu().numpy(), h.get_state(dtype))
            # nothing outside the array is written
            assert float(out[:offset].abs().sum() + out[offset + a.size:].abs().sum()) == 0.0
