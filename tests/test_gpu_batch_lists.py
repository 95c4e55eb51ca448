"""Batched pairs: the work is dealt to as many lists as there are CTAs running at
once, however many CTAs per SM are asked for."""
import pytest

from gpe_b200 import BatchOpts, GpeBatch, GpeParams

pytestmark = pytest.mark.gpu

# at four rows per tile two rings of complex64 fit the 227 KB of an SM at order 2,
# and one of the others; at the default height one of any kind
@pytest.mark.parametrize("order,precision,kahan,tile_y,ctas,most", [
    (2, 8, False, 4, 0, 2), (4, 8, True, 4, 0, 1), (2, 16, False, 4, 0, 1), (4, 16, False, 4, 0, 1),
    (2, 8, False, 0, 2, 1), (2, 16, False, 0, 2, 1), (2, 8, False, 4, 1, 1)])
def test_no_more_lists_than_ctas_run_at_once(order, precision, kahan, tile_y, ctas, most):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    prms = [GpeParams(nx=n, ny=n, nz=n, xr=4.0, yr=4.0, zr=4.0, scheme="rk4", order=order, bcs=2,
                      precision=precision, kahan=kahan) for n in (130, 96)]
    with GpeBatch(prms, 0.002, opts=BatchOpts(tile_y=tile_y, zchunk=4, ctas_per_sm=ctas)) as b:
        b.advance(1)
        info = b.info()
        assert info["items"] > 2 * sms
        assert info["grid"] == most * sms
