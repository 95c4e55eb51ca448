"""Several contexts alive at once, whose launches of one kernel need different
amounts of shared memory: each steps as it does alone."""
import threading

import numpy as np
import pytest

from gpe_b200 import GpeParams, GpeSolver
from gpe_b200.batch import BatchOpts, GpeBatch

pytestmark = pytest.mark.gpu


def field(n, seed, precision):
    rng = np.random.default_rng(seed)
    a = 1.0 + 0.2 * (rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1]))
    return a.astype(np.complex64) if precision == 8 else a


def params(n, **kw):
    return GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=4.0, yr=3.0, zr=3.5, bcs=2, **kw)


def steps(s, n):
    for _ in range(n):
        s.solver()
    return s.get_state()


@pytest.mark.parametrize("scheme,order,precision,kahan,tiles", [
    # rows per tile of a pair: 16, and 8 where the grid has no more
    ("rk4", 4, 8, True, (0, 0)), ("rk4", 2, 8, False, (0, 0)), ("rk2", 4, 8, False, (0, 0)),
    ("rk4", 4, 16, False, (8, 4)), ("rk45", 4, 16, False, (8, 4)), ("euler", 2, 8, False, (8, 4))])
def test_contexts_of_different_tile_heights(scheme, order, precision, kahan, tiles):
    sizes = [(70, 20, 12), (70, 8, 12)]
    prms = [params(n, scheme=scheme, order=order, precision=precision, kahan=kahan, tile_y=t)
            for n, t in zip(sizes, tiles)]
    psi = [field(n, 3, precision) for n in sizes]
    alone = []
    for p, a in zip(prms, psi):
        with GpeSolver(p, dt=1e-3) as s:
            s.set_state(a)
            alone.append(steps(s, 3))
    with GpeSolver(prms[0], dt=1e-3) as s, GpeSolver(prms[1], dt=1e-3) as t:
        s.set_state(psi[0])
        t.set_state(psi[1])
        for _ in range(3):  # in turn: the larger need after the smaller one
            s.solver()
            t.solver()
        assert np.array_equal(s.get_state(), alone[0])
        assert np.array_equal(t.get_state(), alone[1])


def test_batches_of_different_tile_heights():
    n = (70, 20, 12)
    prms = [params(n, scheme="rk4", order=4, precision=8)] * 2
    psi = [field(n, 4 + r, 8) for r in range(2)]
    got = []
    with GpeBatch(prms, 1e-3, opts=BatchOpts(use_graph=False)) as a, \
            GpeBatch(prms, 1e-3, opts=BatchOpts(tile_y=4, use_graph=False)) as b:
        for x in (a, b):
            x.set_states(psi)
        for _ in range(2):
            for x in (a, b):
                x.advance(1)
        got = [[m.get_state() for m in x.members] for x in (a, b)]
    for p, q in zip(*got):
        assert np.array_equal(p, q)


def test_line_length_in_two_threads():
    """Rows of 30 and of 1000 sites: 9 and 2 kB of sign bits a block."""
    sizes = [(30, 40, 20), (1000, 12, 10)]
    solvers = [GpeSolver(params(n, scheme="euler", order=2, precision=16), dt=1e-3) for n in sizes]
    try:
        for s, n in zip(solvers, sizes):
            s.set_state(field(n, 5, 16) - 1.0)
        want = [s.linelength() for s in solvers]
        bad = []

        def work(k):
            try:
                for _ in range(300):
                    if solvers[k].linelength() != want[k]:
                        bad.append((k, "another length"))
                        return
            except Exception as e:  # noqa: BLE001 - reported below
                bad.append((k, repr(e)))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
    finally:
        for s in solvers:
            s.close()
