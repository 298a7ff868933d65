"""Paths that a size or a stream selects: the gradient on a 1-D grid whose FP64
line is transformed in parts, work of a caller's stream before and after the
library's launches, and the x pass of a convolution at lengths of one to four
stages with partial tiles, against numpy."""
import ctypes as C

import numpy as np
import pytest

from conftest import liquid_psi

pytestmark = pytest.mark.gpu


def rdot(a, b):
    return float(np.sum(a.real * b.real + a.imag * b.imag))


@pytest.mark.parametrize("model", [0, 1, 9])
@pytest.mark.parametrize("nz", [1000, 1024, 2160])
def test_gradient_on_a_split_line(gpu, model, nz):
    """nz = 1000 (real transforms of 500) stays in one launch, 1024 and 2160 are split.  A central difference of step t
    along d has the error t^2 / 6 of the third derivative: the smaller of two steps' deviations below 1e-6, as for 3-D
    grids."""
    G, shape, step = gpu, (1, 1, nz), 0.4
    G.set_precision(G.FP64)
    rng = np.random.default_rng(nz + model)
    psi = liquid_psi(shape, step, 7)
    gam = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    d = 0.1 * np.abs(psi) * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    w = G.Wf(shape, step)
    ot = G.OT(model, w)
    P, cot, g = G.CGrid(shape, step), G.CGrid(shape, step), G.CGrid(shape, step)

    def J(x):
        w.set(x)
        P.zero()
        ot.potential(P, w)
        return rdot(gam, P.get())

    w.set(psi)
    cot.set(gam)
    g.zero()
    ot.potential_vjp(w, cot, g)
    an = rdot(g.get(), d)
    errs = [abs((J(psi + h * d) - J(psi - h * d)) / (2 * h) - an) / abs(an) for h in (1e-3, 3e-4)]
    assert min(errs) < 1e-6, errs
    for o in (g, cot, P, ot, w):
        o.free()


class _Memory:
    def __init__(self, grid, shape, prec):
        address = C.cast(grid, C.POINTER(C.c_void_p))[0]
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<c8" if prec else "<c16", "data": (address, False),
                                         "version": 3, "strides": None}


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (60, 54, 48), (1, 1, 2048), (192, 192, 192)], ids=lambda s: "x".join(map(str, s)))
def test_work_of_the_callers_stream(gpu, prec, shape):
    """psi is written by the caller's kernels on the library's stream, behind some milliseconds of other work, and P and
    psi are copied by the caller's kernels right after the library's: the values of the same calls with a wait between."""
    import torch
    G, L = gpu, gpu.lib()
    if shape == (192, 192, 192) and prec == 0:
        pytest.skip("branches are for FP32")
    old = L.dftgpu_get_stream()
    G.set_precision(prec)
    stream = torch.cuda.Stream()
    results = []
    try:
        w, P = G.Wf(shape, 0.8), G.CGrid(shape, 0.8)
        ot = G.OT(9, w, min_ns=2, max_ns=4)
        tw = torch.as_tensor(_Memory(w.grid_ptr, shape, prec), device="cuda")
        tP = torch.as_tensor(_Memory(P.ptr, shape, prec), device="cuda")
        psi = torch.from_numpy(liquid_psi(shape, 0.8, 5)).to(device="cuda", dtype=tw.dtype)
        big = torch.randn(4096, 4096, device="cuda")
        torch.cuda.synchronize()
        G.check(L.dftgpu_set_stream(C.c_void_p(stream.cuda_stream)), "set_stream")
        ot.potential(P, w)                       # buffers and tables
        for wait in (True, False, False):
            sync = torch.cuda.synchronize if wait else (lambda: None)
            out = []
            with torch.cuda.stream(stream):
                tw.zero_()
                tP.zero_()
                for _ in range(8):
                    big = torch.tanh(big @ big)
                tw.copy_(psi)
                sync()
                ot.potential(P, w)
                sync()
                out.append(tP.clone())
                tP.mul_(2.0)
                sync()
                w.propagate(P, 20.0 - 1.0j)
                sync()
                out.append(tw.clone())
                tw.mul_(0.5)
            torch.cuda.synchronize()
            results.append(out)
        for a in results[1:]:
            for x, y in zip(a, results[0]):
                assert torch.equal(torch.view_as_real(x), torch.view_as_real(y))
    finally:
        torch.cuda.synchronize()
        L.dftgpu_set_stream(C.c_void_p(old))
        for o in (ot, P, w):
            o.free()
        G.set_precision(G.FP64)


SHAPES = [(1, 1, 256), (27, 25, 16), (125, 9, 10), (60, 135, 18), (256, 6, 20), (300, 3, 8), (16, 16, 32), (288, 10, 12),
          (320, 30, 6), (1000, 4, 4)]


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_plain_potential_from_the_kernel_spectra(gpu, prec, shape):
    """V = LJ*rho + c2/2 rb^2 + c3/3 rb^3 + w*((c2 rb + c3 rb^2) rho), rb = w*rho: the library's own kernel spectra with
    numpy's transforms.  Four convolutions, whose terms are up to a few times the potential: 16 eps log2 N."""
    G, h = gpu, 0.8
    eps = 2.0 ** -24 if prec else 2.0 ** -53
    G.set_precision(prec)
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
    assert np.linalg.norm(got - ref) <= 16 * eps * max(1.0, np.log2(psi.size)) * np.linalg.norm(ref)
