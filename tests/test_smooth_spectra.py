"""Real transforms of smooth fields by the generic lines: the element of a pair
(k, n - k) at high k is small there, and must not take rounding errors of the
large one at low k.

A line f = (1 + 0.1 cos(2 pi x / L + phi)) (1 + 1e-3 noise); error of the
elements k > 1 against their own norm.  Bounds: the same transform emulated on
the CPU with every product rounded by itself and both elements of a pair formed
from the same sums (FP32 n = 16, 32, 60, 64: 6.1e-5, 6.6e-5, 6.3e-5, 7.8e-5; FP64
n = 32, 64: 1.32e-13, 1.45e-13), plus 7 % (three standard deviations of the
mean over the lines are below 5 %)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(1, 16, 6.1e-5), (1, 32, 6.6e-5), (1, 60, 6.3e-5), (1, 64, 7.8e-5), (0, 32, 1.32e-13), (0, 64, 1.45e-13)]


@pytest.mark.parametrize("prec,n,bound", CASES)
def test_high_k_of_a_smooth_line(gpu, prec, n, bound):
    G, N = gpu, 2 * n
    rng = np.random.default_rng(n)
    LD = np.longdouble
    x, k = np.arange(N), np.arange(n + 1)
    turn = (np.outer(x, k) % N).astype(LD) / N * (8 * np.arctan(LD(1)))
    c, s = np.cos(turn), np.sin(turn)
    G.set_precision(prec)
    err = norm = 0
    try:
        g = G.RGrid((1, 1, N), 0.8)
        for _ in range(8000 // n):
            f = (1 + 0.1 * np.cos(2 * np.pi * x / N + rng.standard_normal())) * (1 + 1e-3 * rng.standard_normal(N))
            if prec:
                f = f.astype(np.float32).astype(np.float64)
            g.set(f.reshape(1, 1, N))
            got = g.spectrum().ravel()
            re, im = f.astype(LD) @ c, -(f.astype(LD) @ s)
            err += float((((got.real - re) ** 2 + (got.imag - im) ** 2))[2:].sum())
            norm += float((re ** 2 + im ** 2)[2:].sum())
        g.free()
    finally:
        G.set_precision(G.FP64)
    assert np.sqrt(err / norm) <= 1.07 * bound, np.sqrt(err / norm)


@pytest.mark.parametrize("n,bound", [(64, 1.010e-7), (128, 1.075e-7), (256, 1.193e-7)])
def test_round_trip_of_a_smooth_line(gpu, n, bound):
    """A propagation over no time, forward and back, of a smooth complex line in FP32.  Bounds: emulated with every
    product rounded before the sums, plus 2.5 % (three standard deviations of the mean are below 1.5 %)."""
    G = gpu
    rng = np.random.default_rng(n)
    G.set_precision(G.FP32)
    err = norm = 0
    try:
        w, V = G.Wf((1, 1, n), 0.8), G.CGrid((1, 1, n), 0.8)
        V.zero()
        inv = float(np.float32(1.0 / n)) * n
        for _ in range(200000 // n):
            f = (1 + 0.1 * np.cos(2 * np.pi * np.arange(n) / n + rng.standard_normal())) * (1 + 1e-3 * rng.standard_normal(n))
            x = (f * (1 + 0.3j)).astype(np.complex64).astype(np.complex128).reshape(1, 1, n)
            w.set(x)
            w.propagate(V, 0j)
            err += np.sum(np.abs(w.get() / inv - x) ** 2)
            norm += np.sum(np.abs(x) ** 2)
        V.free()
        w.free()
    finally:
        G.set_precision(G.FP64)
    assert np.sqrt(err / norm) <= 1.025 * bound, np.sqrt(err / norm)
