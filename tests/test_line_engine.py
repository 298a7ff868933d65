"""The generic line transforms (any 2^a 3^b 5^c length, FP64 and FP32) at the
edges of their tiles: one to five stages, partial tiles, single lines, lengths
1 and 2, the longest line.  Reference: numpy's FP64 FFT.

Tolerance: a transform of N points by butterflies in precision eps has an rms
error of about 0.6 eps sqrt(log2 N) of the result's 2-norm; 4 eps log2 N holds
it with room for the FP32 tables."""
import numpy as np
import pytest

SHAPES = [(1, 1, 2), (1, 1, 4096), (1, 1, 3000), (2, 3, 2), (3, 5, 4), (9, 25, 6), (135, 6, 90), (25, 2, 250), (45, 27, 16),
          (243, 3, 10), (125, 18, 54), (8, 375, 30), (16, 20, 500), (1000, 2, 8), (5, 1024, 4), (64, 60, 128), (75, 81, 1000)]


def eps(prec):
    return 2.0 ** -53 if prec == 0 else 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_real_spectrum(shape, prec):
    import libdft_gb300 as G
    G.check(G.lib().dftgpu_init(0), "init")
    G.set_precision(prec)
    try:
        f = np.random.default_rng(3).standard_normal(shape)
        if prec:
            f = f.astype(np.float32).astype(np.float64)
        g = G.RGrid(shape, 0.8)
        g.set(f)
        got, ref = g.spectrum(), np.fft.rfftn(f)
        g.free()
    finally:
        G.set_precision(G.FP64)
    assert np.linalg.norm(got - ref) <= 4 * eps(prec) * max(1.0, np.log2(f.size)) * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("cn", [False, True], ids=["fft", "cn"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_propagation(shape, cn, prec):
    """exp(-iV dt/2) F^-1 K F exp(-iV dt/2): six complex line passes of every axis, two phase factors and the kinetic
    factor; each phase factor and the kinetic one add a few eps of their own."""
    import libdft_gb300 as G
    G.check(G.lib().dftgpu_init(0), "init")
    G.set_precision(prec)
    h, dt, k0 = 0.8, 12.0 - 5.0j, (0.03, -0.02, 0.05)
    rng = np.random.default_rng(5)
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    V = 1e-2 * (rng.standard_normal(shape) + 0.1j * rng.standard_normal(shape))
    if prec:
        psi, V = (x.astype(np.complex64).astype(np.complex128) for x in (psi, V))
    try:
        w = G.Wf(shape, h, propagator=G.WF_2ND_ORDER_CN if cn else G.WF_2ND_ORDER_FFT)
        P = G.CGrid(shape, h)
        w.set(psi)
        w.set_momentum(*k0)
        P.set(V)
        w.propagate(P, dt)
        got = w.get()
        P.free()
        w.free()
    finally:
        G.set_precision(G.FP64)
    half = np.exp(-0.5j * dt * V)
    f = np.fft.fftn(half * psi)
    for a, n in enumerate(shape):
        k = (2 * np.pi * np.fft.fftfreq(n, h) - k0[a]).reshape([-1 if b == a else 1 for b in range(3)])
        if cn:
            q = -0.5j * dt / G.HELIUM_MASS * (2 * np.sin(0.5 * h * k) / h) ** 2
            f = f * ((1 + 0.5 * q) / (1 - 0.5 * q))
        else:
            f = f * np.exp(-0.5j * dt / G.HELIUM_MASS * k ** 2)
    ref = half * np.fft.ifftn(f)
    assert np.linalg.norm(got - ref) <= (8 * np.log2(psi.size) + 16) * eps(prec) * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(1, 1, 256), (27, 25, 16), (125, 9, 10), (60, 135, 18), (256, 6, 20), (300, 3, 8)],
                         ids=lambda s: "x".join(map(str, s)))
def test_convolutions(shape, prec):
    """The x pass at lengths of one to four stages and with partial tiles: the potential of a shifted wave function is
    the shifted potential (its values against the oracle: test_gpu_parity.py)."""
    import libdft_gb300 as G
    G.check(G.lib().dftgpu_init(0), "init")
    G.set_precision(prec)
    rng = np.random.default_rng(7)
    psi = np.sqrt(0.00323) * (1 + 0.02 * rng.standard_normal(shape)) * np.exp(0.05j * rng.standard_normal(shape))
    shift = tuple(n // 3 for n in shape)
    try:
        w = G.Wf(shape, 0.8)
        ot = G.OT(G.DFT_OT_KC | G.DFT_OT_BACKFLOW, w)
        P = G.CGrid(shape, 0.8)
        out = []
        for s in (psi, np.roll(psi, shift, axis=(0, 1, 2))):
            w.set(s)
            P.zero()
            ot.potential(P, w)
            out.append(P.get())
        for x in (P, ot, w):
            x.free()
    finally:
        G.set_precision(G.FP64)
    ref = np.roll(out[0], shift, axis=(0, 1, 2))
    # the terms of the potential are up to 1e3 times its own size at this noise
    assert np.linalg.norm(out[1] - ref) <= 1e3 * 4 * eps(prec) * np.log2(psi.size) * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(1, 1, 500), (1, 1, 512), (1, 1, 1000), (1, 1, 1024), (1, 1, 2160), (1, 1, 4096), (2, 2, 1024)],
                         ids=lambda s: "x".join(map(str, s)))
def test_long_lines(shape, prec):
    """Lines around the length from which a 1-D grid's line is transformed in parts: plain potential
    V = LJ*rho + c2/2 rb^2 + c3/3 rb^3 + w*((c2 rb + c3 rb^2) rho), rb = w*rho, from the library's own kernel spectra
    with numpy's transforms, and one complex step there and back.  The four convolutions' terms are up to a few
    times the potential: 16 eps log2 N; a step forwards and backwards: two propagations' tolerance."""
    import libdft_gb300 as G
    G.check(G.lib().dftgpu_init(0), "init")
    G.set_precision(prec)
    h = 0.4
    rng = np.random.default_rng(11)
    psi = np.sqrt(0.00323) * (1 + 0.05 * rng.standard_normal(shape)) * np.exp(0.3j * rng.standard_normal(shape))
    if prec:
        psi = psi.astype(np.complex64).astype(np.complex128)
    try:
        w = G.Wf(shape, h)
        ot = G.OT(G.DFT_OT_PLAIN, w)
        P = G.CGrid(shape, h)
        w.set(psi)
        P.zero()
        ot.potential(P, w)
        got = P.get().real
        ker = [ot.kernel(k) for k in (0, 1)]
        c2, c3 = ot.params.c2, ot.params.c3
        P.zero()
        w.propagate(P, 9.0 + 0j)
        w.propagate(P, -9.0 + 0j)
        back = w.get()
        for x in (P, ot, w):
            x.free()
    finally:
        G.set_precision(G.FP64)
    nx, ny, nz = shape
    ix, iy = np.minimum(np.arange(nx), nx - np.arange(nx)), np.minimum(np.arange(ny), ny - np.arange(ny))
    full = [np.transpose(k[:, ix][:, :, iy], (1, 2, 0)) for k in ker]      # [kx][ky][kz], scaled by step^3 / N
    def conv(k, f):
        return np.fft.irfftn(k * np.fft.rfftn(f), s=shape, axes=(0, 1, 2)) * f.size
    rho = np.abs(psi) ** 2
    rb = conv(full[1], rho)
    ref = conv(full[0], rho) + c2 / 2 * rb ** 2 + c3 / 3 * rb ** 3 + conv(full[1], (c2 * rb + c3 * rb ** 2) * rho)
    e = eps(prec) * np.log2(psi.size)
    assert np.linalg.norm(got - ref) <= 16 * e * np.linalg.norm(ref)
    assert np.linalg.norm(back - psi) <= 2 * (8 * e + 16 * eps(prec)) * np.linalg.norm(psi)
