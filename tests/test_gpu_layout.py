"""Ghost layers of the fields: four where a step evaluates two stages at a time,
two where it never does."""
import pytest

from gpe_b200 import GpeParams, GpeSolver
from gpe_b200._lib import lib

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
