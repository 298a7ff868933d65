"""The FP64 phase factors (common.cuh: mul_cexp and the series expm1_8th,
cism1_8th for exponents below 1/8) against long double, on the device.  With
u = 2^-53:

* the series: expm1 and sin have their last product, the rounding of its
  factor and a cut-off of 0.21 u: 3 u of the value; cos - 1 one product more:
  4 u;
* psi exp(z) with |Re z|, |Im z| < 1/8: one rounding of each component, three
  more and the series' 4 u on a factor of at most 0.19, in two components: 4 u
  of |psi e^z|; beyond: exp to 2 u, sin and cos to 4 u, a product and the
  complex product's 3 u: 10 u;
* |psi exp(i theta)|^2 - |psi|^2 over 2^18 angles averages to zero within
  u / 20 (independent roundings: u / 512; the constants' own: u / 500).
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.longdouble


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("phase64")
    exe = d / "phase_probe_fp64"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "libdft_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "phase_probe_fp64.cu"), "-o", str(exe)], check=True)

    def run(x, y):
        z = np.stack(np.broadcast_arrays(np.asarray(x, np.float64), np.asarray(y, np.float64)), -1)
        np.ascontiguousarray(z).tofile(d / "in.bin")
        subprocess.run([str(exe), str(d / "in.bin"), str(d / "out.bin")], check=True, timeout=120)
        return np.fromfile(d / "out.bin", dtype=np.float64).reshape(3, -1, 2)
    return run


def mul_error(out, x, y):
    """|psi e^z - exact| / |psi e^z|, psi = 0.6 - 0.8 i"""
    e, c, s = np.exp(LD(1) * x), np.cos(LD(1) * y), np.sin(LD(1) * y)
    a, b = LD(0.6), LD(-0.8)
    ref = np.stack(np.broadcast_arrays(e * (a * c - b * s), e * (a * s + b * c)), -1)
    return np.sqrt(((out - ref) ** 2).sum(-1)) / (e * np.sqrt(a * a + b * b))


def grid(rng, scale, n=1 << 17):
    return scale * rng.uniform(-1, 1, n)


@pytest.mark.parametrize("scale", [0.125, 1e-2, 1e-5, 1e-12])
def test_series(probe, scale):
    rng = np.random.default_rng(int(-np.log10(scale)))
    x, y = grid(rng, scale), grid(rng, scale)
    _, cis, em1 = probe(x, y)
    with np.errstate(invalid="ignore"):
        assert np.max(np.abs(em1[:, 0] / np.expm1(LD(1) * x) - 1)) <= 3 * U
        assert np.max(np.abs(cis[:, 1] / np.sin(LD(1) * y) - 1)) <= 3 * U
        cm1 = -2 * np.sin(LD(0.5) * y) ** 2
        assert np.max(np.abs(cis[:, 0] / cm1 - 1)) <= 4 * U


@pytest.mark.parametrize("kind", ["both", "real", "imaginary"])
@pytest.mark.parametrize("scale", [0.125, 1e-2, 1e-5])
def test_small_exponents(probe, kind, scale):
    """The three forms: both parts, a real exponent (imaginary time), an imaginary one (real time)."""
    rng = np.random.default_rng(7)
    x = grid(rng, scale) if kind != "imaginary" else np.zeros(1 << 17)
    y = grid(rng, scale) if kind != "real" else np.zeros(1 << 17)
    mul = probe(x, y)[0]
    assert mul_error(mul, x, y).max() <= 4 * U
    if kind == "real":   # a real factor: the ratio of the parts stays
        assert np.max(np.abs(mul[:, 1] / mul[:, 0] / (LD(-0.8) / LD(0.6)) - 1)) <= 8 * U


def test_around_the_switch(probe):
    b = 0.125
    edge = np.array([b, np.nextafter(b, 0), np.nextafter(b, 1), 0.0, -0.0, 0.06, 0.2, 0.25, 1e-300, 5e-324])
    edge = np.concatenate([edge, -edge])
    x, y = (v.ravel() for v in np.meshgrid(edge, edge))
    assert mul_error(probe(x, y)[0], x, y).max() <= 10 * U
    rng = np.random.default_rng(9)
    x, y = rng.uniform(-3, 1, 1 << 16), rng.uniform(-20, 20, 1 << 16)
    assert mul_error(probe(x, y)[0], x, y).max() <= 10 * U
    assert np.isnan(probe([np.nan, 0.01, np.nan], [0.01, np.nan, 0.0])[0]).any(-1).all()


def test_pure_phase_has_no_norm_bias(probe):
    theta = np.random.default_rng(4).uniform(-0.12, 0.12, 1 << 18)
    mul = LD(1) * probe(np.zeros(1 << 18), theta)[0]
    assert abs(((mul ** 2).sum(-1) - (LD(0.6) ** 2 + LD(-0.8) ** 2)).mean()) <= U / 20
