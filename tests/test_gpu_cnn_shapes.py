"""The convolution kernels where a slab of output rows ends early or late, a
half of it is empty, rows fill a few of an MMA's lanes or all, and z chunks are
of unequal length.  Oracle and tolerances as in tests/test_gpu_cnn.py, except
the loss: over a few hundred sites delta's rounding does not average out, so it
is compared with the mean of |u + delta - target|^2 over the kernel's own delta
(sums of up to 3e4 terms in 64 bits: 1e-12).  The ghosts an application writes are checked through a step that reads them, bit
for bit against the same state loaded afresh."""
import numpy as np
import pytest

from gpe_b200.cnn import CoarseCorrector
from oracle import cnn_ref as R
from tests.conftest import random_field, rel_l2
from tests.test_gpu_cnn import solver, weights

pytestmark = pytest.mark.gpu

SHAPES = [(16, 6, 6), (48, 11, 7), (128, 13, 8), (64, 15, 6), (112, 8, 33)]


@pytest.mark.parametrize("n", SHAPES)
def test_delta_and_gradients(n):
    import torch
    rng = np.random.default_rng(n[1])
    u = random_field((n[2], n[1], n[0]), seed=11).astype(np.complex64)
    tgt = (u + 0.02 * (rng.normal(size=u.shape) + 1j * rng.normal(size=u.shape))).astype(np.complex64)
    w, b = weights(3)
    with solver(n) as s, CoarseCorrector(*n, train=True, out_scale=0.05) as net:
        s.set_state(u)
        net.set_weights(w, b)
        d = net.delta(s).cpu().numpy().astype(np.float64)
        loss, dw, db = net.grad(s, torch.from_numpy(tgt).cuda())
    exp, _ = R.forward(u.astype(np.complex128), w, b, 0.05, emulate=True)
    assert rel_l2(d[..., 0] + 1j * d[..., 1], exp[..., 0] + 1j * exp[..., 1]) < 3e-3
    e = u.astype(np.complex128) + d[..., 0] + 1j * d[..., 1] - tgt
    assert loss == pytest.approx((np.abs(e) ** 2).mean(), rel=1e-12)
    _, dw_ref, db_ref = R.loss_and_grad(u.astype(np.complex128), tgt.astype(np.complex128),
                                            w, b, 0.05, emulate=True)
    for l in range(4):
        assert rel_l2(dw[l], dw_ref[l]) < 2e-2, l
        assert rel_l2(db[l], db_ref[l]) < 2e-2, l


@pytest.mark.parametrize("n", SHAPES)
def test_apply_writes_every_ghost(n):
    w, b = weights(1)
    psi = random_field((n[2], n[1], n[0]), seed=5).astype(np.complex64)
    with solver(n) as s, solver(n) as f, CoarseCorrector(*n, out_scale=0.05) as net:
        net.set_weights(w, b)
        s.set_state(psi)
        net.apply(s)
        f.set_state(s.get_state(np.complex64))
        s.solver()
        f.solver()
        assert np.array_equal(s.get_state(np.complex64), f.get_state(np.complex64))
