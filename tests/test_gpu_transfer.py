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


@pytest.mark.parametrize("scheme", ["euler", "rk2", "rk4", "rk45"])
@pytest.mark.parametrize("precision", [8, 16])
def test_norm_follows_every_change_of_the_state(scheme, precision):
    """The norm a step hands back with its status is the one a fresh reduction
    of the same state gives, and no later call returns it for another state."""
    rng = np.random.default_rng(5)
    prm = GpeParams(nx=20, ny=9, nz=11, xr=3.0, yr=3.0, zr=3.0, order=4, bcs=1, scheme=scheme,
                    precision=precision)
    a = 1.0 + 0.1 * (rng.normal(size=(11, 9, 20)) + 1j * rng.normal(size=(11, 9, 20)))
    # 1980 terms, each rounded once in the field's precision
    rel = 1e-12 if precision == 16 else 1e-5

    def fresh(s):
        with GpeSolver(prm, dt=1e-4) as o:
            o.set_state(s.get_state())
            return o.get_norm()

    with GpeSolver(prm, dt=1e-4) as s:
        s.set_state(a)
        for change in (s.solver, s.solver, lambda: s.renormalise(7.0), s.solver,
                       lambda: s.advance(3), s.solver, lambda: s.set_state(2.0 * a), s.solver):
            change()
            assert s.get_norm() == pytest.approx(fresh(s), rel=rel)
            assert s.get_norm() == pytest.approx(fresh(s), rel=rel)


@pytest.mark.parametrize("precision", [8, 16])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_batch_states_equal_member_states(precision, dtype):
    import torch
    from gpe_b200.batch import GpeBatch
    from gpe_b200.solver import GpeError
    rng = np.random.default_rng(7)
    shapes = [(20, 9, 11), (33, 8, 7), (16, 16, 8)]
    prms = [GpeParams(nx=x, ny=y, nz=z, xr=3.0, yr=3.0, zr=3.0, order=4, bcs=1,
                      precision=precision) for x, y, z in shapes]
    host = [(rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1])).astype(dtype)
            for n in shapes]
    dev = [torch.from_numpy(a).cuda() for a in host]
    with GpeBatch(prms, dt=0.01) as b:
        b.set_states(dev)
        got = [m.get_state(dtype) for m in b.members]
        b.set_states(host)
        for g, m in zip(got, b.members):
            assert np.array_equal(g, m.get_state(dtype))
        b.set_states([dev[0], host[1], dev[2]])         # mixed: one by one
        b.set_states(dev[:2])                           # a shorter list loads those
        for g, m in zip(got, b.members):
            assert np.array_equal(g, m.get_state(dtype))
        # a wrong shape or type is refused
        with pytest.raises(GpeError):
            b.set_states([dev[1], dev[0], dev[2]])
        with pytest.raises(GpeError):
            b.set_states([d.real.contiguous() for d in dev])
