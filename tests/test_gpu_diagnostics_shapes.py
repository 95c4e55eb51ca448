"""Shapes at the edges of the diagnostics' launches on B200: rows of cells that
share a scan step, fill one, need several or are too long for shared memory
(line length), and tiles of 32 x 8 with remainders (mass and momentum), against
the oracle within the bounds of the tests of those calls (1e-12, both sum the
same terms in another order)."""
import numpy as np
import pytest

import oracle
from gpe_b200 import GpeParams, GpeSolver

pytestmark = pytest.mark.gpu


def solver(n, order=2, precision=16):
    return GpeSolver(GpeParams(nx=n[0], ny=n[1], nz=n[2], xr=0.25 * (n[0] - 1), yr=0.25 * (n[1] - 1),
                               zr=0.25 * (n[2] - 1), order=order, bcs=1, precision=precision), dt=0.01)


def field(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=n[::-1]) + 1j * rng.normal(size=n[::-1])


@pytest.mark.parametrize("n", [(6, 40, 9), (66, 11, 9), (258, 7, 8), (259, 7, 8), (600, 8, 7),
                               (33000, 6, 6)])
def test_line_length_of_short_and_long_rows(n):
    psi = field(n, sum(n))
    with solver(n) as s:
        s.set_state(psi)
        got = s.linelength()
    exp, _ = oracle.linelength(psi, 0.5)
    assert got == pytest.approx(exp, rel=1e-12)


@pytest.mark.parametrize("n", [(6, 6, 6), (31, 7, 40), (33, 9, 6), (256, 64, 20)])
@pytest.mark.parametrize("order,precision", [(2, 16), (4, 16), (4, 8)])
def test_mass_and_momentum_tiles(n, order, precision):
    psi = field(n, sum(n) + order)
    if precision == 8:
        psi = psi.astype(np.complex64).astype(np.complex128)
    with solver(n, order, precision) as s:
        s.set_state(psi)
        m, mom = s.diagnostics()
    o = oracle.Oracle(oracle.OracleParams(nx=n[0], ny=n[1], nz=n[2], xr=0.25 * (n[0] - 1),
                                          yr=0.25 * (n[1] - 1), zr=0.25 * (n[2] - 1), scheme="rk4",
                                          order=order, bcs=1))
    exp = np.array(o.momentum(psi))
    assert m == pytest.approx(o.mass(psi), rel=1e-12)
    # the signed sums are bounded by their terms' magnitudes, about mass / h
    assert np.abs(mom - exp).max() <= 1e-12 * m / 0.5


def odd_near(rng, top, shape):
    """Odd integers of 2^top plus a few thousands."""
    return 2 ** top + 2 * rng.integers(0, 2000, size=shape) + 1


def total(terms):
    """The exact sum of an int64 array below 2^62, as a Python integer."""
    return (int((terms >> 24).sum()) << 24) + int((terms & (2 ** 24 - 1)).sum())


@pytest.mark.parametrize("n", [(40, 20, 24), (640, 150, 60)])
def test_mass_and_momentum_of_integers_are_exact(n):
    """Fields of integers, whose terms and whose sums over eight planes are
    exact in 64 bits (below 2^52) while the sums of a block are not (2^56 and
    more): the totals are the correctly rounded ones, times dx dy dz = 1/8.  The
    second grid has more than two runs of planes to a block."""
    rng = np.random.default_rng(n[0])
    shape = n[::-1]
    with solver(n) as s:
        a, b = odd_near(rng, 23, shape), odd_near(rng, 23, shape)
        s.set_state(a + 1j * b)
        mass, _ = s.diagnostics()
        assert mass == float(total(a * a + b * b)) * 0.125
        # psi = 1 in the outer layers, whose weights are no integers: no term there
        inner = np.zeros(shape, dtype=bool)
        inner[3:-3, 3:-3, 3:-3] = True
        for axis in range(3):
            x = np.moveaxis(np.broadcast_to(np.arange(shape[axis]), np.moveaxis(a, axis, -1).shape), -1, axis)
            re1 = np.where(inner, odd_near(rng, 23, shape), 0)
            im = np.where(inner, odd_near(rng, 22, shape) * (x % 4), 0)
            s.set_state((re1 + 1) + 1j * im)
            _, mom = s.diagnostics()
            # h = 1/2: a first derivative is the difference of the two neighbours
            di = np.roll(im, -1, axis) - np.roll(im, 1, axis)
            dr = np.roll(re1, -1, axis) - np.roll(re1, 1, axis)
            assert mom[2 - axis] == float(total(-re1 * di - im * dr)) * 0.125
