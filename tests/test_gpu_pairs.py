"""Two Runge-Kutta stages per launch against one stage per launch and the
oracle, on B200: grids at the edges of the pair kernel's tiles (64 x 16
complex64, 64 x 8 complex128), with remainders, a last chunk, and the ghost
sites that the first stage of a pair is evaluated on."""
import numpy as np
import pytest

import oracle
from gpe_b200 import GpeParams, GpeSolver

pytestmark = pytest.mark.gpu

SIZES = [(6, 6, 6), (63, 15, 7), (64, 16, 9), (65, 17, 13), (66, 33, 24), (130, 8, 31)]


def field(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1])


def params(n, scheme, order, bcs, precision, kahan, trap, **kw):
    om = dict(omx=0.3, omy=0.2, omz=0.4) if trap else {}
    return dict(nx=n[0], ny=n[1], nz=n[2], xr=4.0, yr=3.0, zr=3.5, scheme=scheme, order=order,
                bcs=bcs, g=1.3, mu=0.9, **om, **kw), dict(precision=precision, kahan=kahan)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("scheme,order,bcs,precision,kahan,trap,eqn", [
    ("rk4", 4, 1, 8, True, False, 4), ("rk4", 4, 2, 8, False, True, 4),
    ("rk4", 2, 2, 8, True, True, 4), ("rk4", 2, 1, 8, False, False, 1),
    ("rk4", 4, 2, 16, False, False, 4), ("rk4", 2, 1, 16, False, True, 4),
    ("rk2", 4, 1, 8, True, False, 4), ("rk2", 2, 2, 8, False, False, 2),
    ("rk2", 4, 2, 16, False, True, 4)])
def test_pairs_equal_single_stages_bitwise(n, scheme, order, bcs, precision, kahan, trap, eqn):
    """Per-launch timing steps one stage per launch: the same bits, and the
    norm to rounding (its sum is grouped by tiles).  complex128 also follows
    the oracle to 1e-12, the bound of the one-stage parity tests."""
    kw, st = params(n, scheme, order, bcs, precision, kahan, trap, eqn_to_solve=eqn,
                    Urhs=0.3 if eqn != 4 else 0.0, diss_amp=0.4 if eqn == 1 else 0.0)
    psi = field(n, seed=sum(n) + order)
    if precision == 8:
        psi = psi.astype(np.complex64)
    dt, out = 0.002, []
    for timed in (False, True):
        with GpeSolver(GpeParams(**kw, **st), dt=dt) as s:
            s.set_timing(timed)
            s.set_state(psi)
            norms = s.advance(3)
            out.append((s.get_state(), norms))
    assert np.array_equal(out[0][0], out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
    if precision == 16:
        o = oracle.Oracle(oracle.OracleParams(**kw))
        tm, q = oracle.OraTime(0.0, 0.0, dt, 0.0, 0), psi
        for _ in range(3):
            q, _, _ = o.solver(q, tm)
        assert np.linalg.norm(out[0][0] - q) <= 1e-12 * np.linalg.norm(q)
        assert out[0][1][-1] == pytest.approx(o.get_norm(q), rel=1e-12)


def test_ghosts_follow_whoever_wrote_psi():
    """Pairs after single stages and the other way round: the deep ghosts are
    rebuilt when the last writer filled only the inner ones."""
    n = (66, 17, 13)
    kw, st = params(n, "rk4", 4, 2, 8, True, True)
    psi = field(n, seed=9).astype(np.complex64)
    out = []
    for modes in ((False, False, False, False), (True, False, False, True), (False, True, False, False)):
        with GpeSolver(GpeParams(**kw, **st), dt=0.002) as s:
            s.set_state(psi)
            for timed in modes:
                s.set_timing(timed)
                s.solver()
            out.append(s.get_state(np.complex64))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("n", [(6, 6, 6), (33, 20, 17), (64, 64, 64), (130, 70, 31)])
@pytest.mark.parametrize("scheme,order,precision,eqn", [
    ("euler", 2, 16, 4), ("rk2", 2, 16, 4), ("rk4", 2, 8, 4), ("rk4", 4, 16, 4), ("rk4", 2, 16, 1)])
def test_overlapped_launches_change_nothing(n, scheme, order, precision, eqn):
    """Launches whose blocks are set up while the kernel before them ends (off
    while per-launch timing is on): 200 steps, enqueued together and one by
    one, give the same bits either way."""
    kw, st = params(n, scheme, order, 1, precision, False, False, eqn_to_solve=eqn,
                    Urhs=0.3 if eqn != 4 else 0.0, diss_amp=0.4 if eqn == 1 else 0.0)
    psi = 1.0 + 0.1 * field(n, seed=sum(n))
    if precision == 8:
        psi = psi.astype(np.complex64)
    out = []
    for timed in (False, True):
        with GpeSolver(GpeParams(**kw, **st), dt=1e-4) as s:
            s.set_timing(timed)
            s.set_state(psi)
            s.advance(150)
            for _ in range(50):
                s.solver()
            out.append(s.get_state())
    assert np.array_equal(*out)
