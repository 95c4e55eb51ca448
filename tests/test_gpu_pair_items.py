"""CTAs of the pair kernels that take several work items one after another: what
is carried over from one to the next (ring slots and their phases, the planes of
first-stage values, the pointwise tiles, the planes handed back at an item's
end).  Short chunks give a grid of 3 x 5 (complex64) or 3 x 9 tiles more items
than there are SMs; states are compared bit for bit with one stage per launch."""
import numpy as np
import pytest

from gpe_b200 import BatchOpts, GpeBatch, GpeParams, GpeSolver

pytestmark = pytest.mark.gpu

N = (130, 70, 31)


def field(n, seed, precision):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1])
    return a.astype(np.complex64) if precision == 8 else a


def run(n, psi, timed, steps=3, dt=0.002, **kw):
    """State, norms and launches per step (4 and 5 for rk4 in pairs and in
    stages, 2 and 3 for rk2)."""
    prm = GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=4.0, yr=3.0, zr=3.5, g=1.3, mu=0.9, **kw)
    with GpeSolver(prm, dt=dt) as s:
        s.set_timing(timed)
        s.set_state(psi)
        before = s.launch_count()
        norms = s.advance(steps)
        launches = (s.launch_count() - before) / steps
        return s.get_state(), norms, launches


STEPS = {("rk4", False): 4, ("rk4", True): 5, ("rk2", False): 2, ("rk2", True): 3}


def compare(n, psi, scheme, **kw):
    got, norms, launches = run(n, psi, False, scheme=scheme, **kw)
    exp, exp_norms, exp_launches = run(n, psi, True, scheme=scheme, **kw)
    assert (launches, exp_launches) == (STEPS[scheme, False], STEPS[scheme, True])
    assert np.array_equal(got, exp, equal_nan=True)
    np.testing.assert_allclose(norms, exp_norms, rtol=1e-12)


@pytest.mark.parametrize("zchunk", [1, 2, 3])
@pytest.mark.parametrize("scheme,order,bcs,precision,kahan,trap", [
    ("rk4", 4, 2, 8, True, False), ("rk4", 4, 1, 8, False, True), ("rk4", 2, 1, 8, True, True),
    ("rk4", 2, 2, 8, False, False), ("rk4", 4, 1, 16, False, True), ("rk4", 2, 2, 16, False, False),
    ("rk2", 4, 2, 8, True, False), ("rk2", 2, 1, 8, False, True), ("rk2", 4, 1, 16, False, False),
    ("rk2", 2, 2, 16, False, True)])
def test_many_items_per_cta(zchunk, scheme, order, bcs, precision, kahan, trap):
    om = dict(omx=0.3, omy=0.2, omz=0.4) if trap else {}
    compare(N, field(N, 10 * zchunk + order, precision), scheme, order=order, bcs=bcs,
            precision=precision, kahan=kahan, zchunk=zchunk, **om)


@pytest.mark.parametrize("order,eqn,dt", [(2, 1, 1e-5), (2, 1, 0.002), (2, 4, 0.002),
                                          (4, 4, 0.002)])
@pytest.mark.parametrize("zchunk", [0, 2])
def test_periodic_complex64_rows_of_whole_tiles(order, eqn, dt, zchunk):
    """Rows of 192 sites, three whole tiles: wider than a network's grid, so rk4
    steps in pairs there.  (Equation 1 diffuses: at the longer time step its state
    overflows, in both forms at the same sites.)"""
    n = (192, 33, 24)
    kw = dict(Urhs=0.3, diss_amp=0.4) if eqn == 1 else {}
    compare(n, field(n, order + eqn, 8), "rk4", order=order, bcs=1, precision=8, kahan=eqn == 4,
            eqn_to_solve=eqn, dt=dt, zchunk=zchunk, **kw)


@pytest.mark.parametrize("order,precision,kahan", [(4, 8, True), (2, 8, False), (4, 16, False),
                                                   (2, 16, False)])
@pytest.mark.parametrize("opts", [BatchOpts(zchunk=1), BatchOpts(zchunk=2, tile_y=4)])
def test_batch_lists_of_many_items(order, precision, kahan, opts):
    """Batched pairs whose lists hold items of several runs each."""
    import torch
    sizes = [(130, 70, 31), (33, 40, 21), (70, 33, 40)]
    prms = [GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=4.0, yr=3.0, zr=3.5, scheme="rk4", order=order,
                      bcs=2, precision=precision, kahan=kahan, omx=0.3, omy=0.2, omz=0.4)
            for n in sizes]
    psi = [field(n, sum(n), precision) for n in sizes]
    with GpeBatch(prms, 0.002, opts=opts) as b:
        b.set_states(psi)
        b.advance(3)
        assert b.info()["items"] > 2 * torch.cuda.get_device_properties(0).multi_processor_count
        got = [m.get_state() for m in b.members]
    for p, a, g in zip(prms, psi, got):
        with GpeSolver(p, dt=0.002) as s:
            s.set_timing(True)
            s.set_state(a)
            s.advance(3)
            assert np.array_equal(g, s.get_state())


def test_batch_with_a_member_on_a_network_grid():
    """A periodic complex64 grid that a network can correct keeps its summation
    order, and with it every member of its batch steps one stage per launch."""
    sizes = [(64, 20, 12), (70, 20, 12)]
    prms = [GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=4.0, yr=3.0, zr=3.5, scheme="rk4", order=4,
                      bcs=1, precision=8, kahan=True) for n in sizes]
    psi = [field(n, sum(n), 8) for n in sizes]
    with GpeBatch(prms, 0.002) as b:
        b.set_states(psi)
        b.advance(4)
        got = [m.get_state() for m in b.members]
    for p, a, g in zip(prms, psi, got):
        with GpeSolver(p, dt=0.002) as s:
            s.set_state(a)
            s.advance(4)
            assert np.array_equal(g, s.get_state())
