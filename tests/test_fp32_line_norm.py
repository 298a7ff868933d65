"""Generic FP32 line transforms do not let the norm drift: the constants of a
butterfly are rounded to FP32, which scales the line's norm by the same small
amount at every transform, so that the deviations of a plan's stages have to
offset each other.

One free 1-D propagation step is a forward and an inverse transform of length
n, a factor of modulus one and the normalisation 1/n (whose own rounding is
known and taken out).  Bounds: the change of the norm per transform, emulated
in FP32 on the CPU with every constant and every twiddle product rounded by
itself (radices 16 x 15, 16 x 10, 16 x 5, 8 x 15): 1.60e-8, 4.7e-9, 2.9e-9 and
1.6e-9, plus four standard deviations of the measured mean (a transform's own
rounding changes the norm of one line by about 2.2e-7 / sqrt(n))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 1600


@pytest.mark.parametrize("n,bias", [(240, 1.60e-8), (160, 4.7e-9), (80, 2.9e-9), (120, 1.6e-9)])
def test_norm_change_per_transform(gpu, n, bias):
    G = gpu
    G.set_precision(G.FP32)
    try:
        rng = np.random.default_rng(n)
        psi = (rng.standard_normal((1, 1, n)) + 1j * rng.standard_normal((1, 1, n))).astype(np.complex64)
        w, V = G.Wf((1, 1, n), 0.8), G.CGrid((1, 1, n), 0.8)
        w.set(psi.astype(np.complex128))
        V.zero()
        n0 = np.sum(np.abs(w.get()) ** 2)
        for _ in range(STEPS):
            w.propagate(V, 41.3 + 0.0j)
        n1 = np.sum(np.abs(w.get()) ** 2)
        V.free()
        w.free()
    finally:
        G.set_precision(G.FP64)
    inv_n = 2 * np.log(float(np.float32(1.0 / n)) * n)            # of the norm, per step
    per_transform = (np.log(n1 / n0) / STEPS - inv_n) / 2
    assert abs(per_transform) <= bias + 4 * 2.2e-7 / np.sqrt(n) / np.sqrt(2 * STEPS), per_transform
