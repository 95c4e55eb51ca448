"""Ghost layers of the fields: four where a step evaluates two stages at a time,
two where it never does."""
import numpy as np
import pytest

from gpe_b200 import GpeBatch, GpeParams, GpeSolver
from gpe_b200._lib import check, lib

pytestmark = pytest.mark.gpu

N = 112
FIELDS = {"euler": 2, "rk45": 9, "rk4": 4, "rk2": 3}


def rounded(n):
    return (n + 3) // 4 * 4


@pytest.mark.parametrize("layers,scheme,kw", [
    (2, "euler", dict(precision=16)), (2, "rk45", dict(precision=16, bcs=2)),
    (2, "rk4", dict(precision=8, bcs=1)),              # a grid a network can correct
    (2, "rk4", dict(precision=16, eqn_to_solve=3)),
    (4, "rk4", dict(precision=8, bcs=2)), (4, "rk4", dict(precision=16)),
    (4, "rk2", dict(precision=8, bcs=1))])
def test_fields_hold_the_ghosts_their_steps_need(layers, scheme, kw):
    prm = GpeParams(nx=N, ny=N, nz=N, xr=3.0, yr=3.0, zr=3.0, order=4, scheme=scheme, **kw)
    with GpeSolver(prm, dt=1e-3) as s:
        got = lib().gpe_gpu_device_bytes(s.handle)
    m = N + 2 * layers
    fields = FIELDS[scheme] * kw["precision"] * rounded(m) * m * m
    # besides them the staging buffer and, below 1 MB, partial sums and tables
    rest = got - fields - 16 * N ** 3
    assert 0 <= rest < 1 << 20


def place(s, nz, z_offset):
    check(lib().gpe_gpu_set_slab(s.handle, nz, z_offset), s.handle)


@pytest.mark.parametrize("scheme,precision,kahan", [("rk4", 8, True), ("rk4", 16, False),
                                                    ("rk2", 8, True), ("rk45", 8, True)])
def test_a_slab_has_two_layers_and_keeps_its_state(scheme, precision, kahan):
    """Placing a context as a slab narrows its fields: the state, and with it the
    compensation that the next step takes, are what they were."""
    n = (30, 21, 12)
    kw = dict(nx=n[0], ny=n[1], nz=n[2], xr=3.0, yr=3.0, zr=3.0, order=4, bcs=1, scheme=scheme,
              precision=precision, kahan=kahan)
    rng = np.random.default_rng(3)
    a = 1.0 + 0.2 * (rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1]))
    dtype = np.complex64 if precision == 8 else np.complex128
    with GpeSolver(GpeParams(**kw), dt=1e-3) as s, GpeSolver(GpeParams(**kw), dt=1e-3) as t:
        for x in (s, t):
            x.set_state(a.astype(dtype))
            x.advance(3)
        before = s.get_state(dtype)
        at = lib().gpe_gpu_device_bytes(s.handle)
        place(s, 2 * n[2], 0)
        fields = {"rk4": 4, "rk2": 3, "rk45": 9}[scheme] + (2 if scheme == "rk45" else 1) * kahan
        wide = 4 if scheme != "rk45" else 2
        sites = lambda g: rounded(n[0] + 2 * g) * (n[1] + 2 * g) * (n[2] + 2 * g)  # noqa: E731
        assert at - lib().gpe_gpu_device_bytes(s.handle) == fields * precision * (sites(wide) - sites(2))
        assert np.array_equal(s.get_state(dtype), before)
        # back in a box of its own, it goes on as the one that never left
        place(s, n[2], 0)
        s.advance(3)
        t.set_timing(scheme != "rk45")  # one stage per launch, as s has room for
        t.advance(3)
        assert np.array_equal(s.get_state(dtype), t.get_state(dtype))


@pytest.mark.parametrize("scheme,precision,kahan", [("rk4", 8, True), ("rk2", 16, False)])
def test_a_rank_has_two_layers(scheme, precision, kahan):
    """Ranks exchange whole padded planes, whose size follows from the layers: all
    have two."""
    from gpe_b200.dist import SlabSolver
    n = (30, 21, 12)
    prm = GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=3.0, yr=3.0, zr=3.0, order=4, bcs=1,
                    scheme=scheme, precision=precision, kahan=kahan)
    fields = {"rk4": 4, "rk2": 3}[scheme] + kahan
    sites = lambda g: rounded(n[0] + 2 * g) * (n[1] + 2 * g) * (n[2] + 2 * g)  # noqa: E731
    with GpeSolver(prm, dt=1e-3) as s, SlabSolver(prm, rank=0, nranks=1, dist=None, dt=1e-3) as r:
        saved = lib().gpe_gpu_device_bytes(s.handle) - lib().gpe_gpu_device_bytes(r._ctx)
        assert saved == fields * precision * (sites(4) - sites(2))


def test_a_batch_follows_a_member_that_is_placed():
    """Placing a member moves its tables and fields: the batch steps on the new
    ones, one stage per launch from then on."""
    n = (30, 21, 12)
    prms = [GpeParams(nx=n[0], ny=n[1], nz=n[2] + 2 * r, xr=3.0, yr=3.0, zr=3.0, order=2, bcs=2,
                      scheme="rk4", precision=16, omx=0.3, omy=0.3, omz=0.3) for r in range(2)]
    rng = np.random.default_rng(4)
    psi = [1.0 + 0.2 * rng.normal(size=(p.nz, p.ny, p.nx)) + 0j for p in prms]
    with GpeBatch(prms, 1e-3) as b, GpeSolver(prms[0], dt=1e-3) as s, GpeSolver(prms[1], dt=1e-3) as t:
        b.set_states(psi)
        b.advance(3)
        place(b.members[0], 2 * n[2], 3)
        b.advance(3)
        for x, a in ((s, psi[0]), (t, psi[1])):
            x.set_state(a)
            x.advance(3)
        place(s, 2 * n[2], 3)
        for x, m in ((s, b.members[0]), (t, b.members[1])):
            x.advance(3)
            assert np.array_equal(m.get_state(), x.get_state())
