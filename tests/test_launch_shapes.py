"""The launch code of the library on the CPU: a stand-in for the CUDA runtime
(tests/cuda/fake_cudart.c) is loaded in front of it in a child process and
records what would have been launched."""
import json
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

PRELUDE = r"""
import ctypes as C, json, sys
fake = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL)     # its symbols are found before the CUDA runtime's
sys.path.insert(0, sys.argv[2])
import libdft_gb300 as G
KEYS = ("gx", "gy", "gz", "bx", "by", "bz", "smem", "device", "granted", "programmatic", "func")
def launches():
    out = (C.c_long * 11)()
    r = []
    for i in range(fake.fake_launches()):
        fake.fake_launch(i, out)
        r.append(dict(zip(KEYS, out)))
    fake.fake_reset()
    return r
def noalloc(shape, prec):
    L = G.lib()
    p = C.c_void_p(1 << 40)
    rc = L.dftgpu_wf_propagate_noalloc(p, p, p, *shape, 0.8, G.HELIUM_MASS, 1.0, 0.0, prec, None)
    assert rc == 0, L.dftgpu_last_error_message()
    return launches()
result = {}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run([os.environ.get("CC", "gcc"), "-O1", "-shared", "-fPIC", "-I", include,
                    os.path.join(ROOT, "tests", "cuda", "fake_cudart.c"), "-o", so], check=True)

    def go(body):
        r = subprocess.run([sys.executable, "-c", PRELUDE + body + "\nprint(json.dumps(result))", so, ROOT],
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1])
    return go


def test_allocation_free_step_on_a_second_device(run):
    """The allocation-free step serves whichever device is current: a kernel that needs more than 48 KB of shared memory
    has been granted it on that device, also when another device was used first."""
    r = run("""
for shape, prec in (((128, 128, 128), 0), ((1, 1, 4096), 0), ((16, 1000, 24), 1)):
    for device in (0, 1):
        fake.fake_set_device(device)
        result["%s %d" % (shape, device)] = noalloc(shape, prec)
""")
    big = 0
    for case, launches in r.items():
        assert len(launches) == 5, (case, len(launches))
        big += sum(l["smem"] > 48 * 1024 for l in launches)
        assert all(l["granted"] for l in launches), (case, [l for l in launches if not l["granted"]])
    assert big >= 4   # the cases do reach it, on both devices


def test_allocation_free_step_without_init(run):
    """The allocation-free step does not need dftgpu_init: its launches are the same before and after it, and small grids
    spread over every SM (four CTAs each where a CTA keeps its least number of lines)."""
    r = run("""
cases = [((64, 64, 64), 0), ((64, 64, 64), 1), ((32, 48, 40), 0)]
result["before"] = [noalloc(*c) for c in cases]
G.check(G.lib().dftgpu_init(0), "init")
fake.fake_reset()
result["after"] = [noalloc(*c) for c in cases]
""")
    assert r["before"] == r["after"]
    assert all(l["gx"] * l["gy"] >= 4 * 152 for l in r["before"][0])


def test_tiles_leave_room_for_three_ctas(run):
    """A tile that can be cut without giving up its runs of 64 bytes (or its FP64 warp of butterflies) lets three CTAs of
    a line or convolution pass, or two of the kinetic pass, share an SM's 228 KB."""
    r = run("""
class Shape(C.Structure):
    _fields_ = [("B", C.c_int), ("logB", C.c_int), ("threads", C.c_int), ("smem", C.c_size_t)]
f = G.lib()._ZN6dftgpu11choose_tileEiiiimibmiPNS_9TileShapeE
f.argtypes = [C.c_int] * 4 + [C.c_size_t, C.c_int, C.c_bool, C.c_size_t, C.c_int, C.POINTER(Shape)]
result["tiles"] = []
for cplx in (8, 16):
    for n in sorted(2 ** a * 3 ** b * 5 ** c for a in range(11) for b in range(7) for c in range(5) if 2 ** a * 3 ** b * 5 ** c <= 1024):
        for bufs in (1, 2, 3, 4):
            for ctas in (2, 3):
                t = Shape()
                assert f(n, 16, 256, 256, cplx, bufs, True, 0, ctas, C.byref(t)) == 0
                result["tiles"].append((cplx, n, ctas, t.B, t.smem))
""")
    for cplx, n, ctas, B, smem in r["tiles"]:
        least = 64 // cplx
        while cplx == 16 and least < 32 and least * n < 32 * 16:
            least *= 2
        assert ctas * (smem + 1024) <= 228 * 1024 or B <= least, (cplx, n, ctas, B, smem)


def test_segments_of_long_rows_are_neighbours(run):
    """Pointwise passes: a row of more than 256 values runs as segments that are neighbours in the grid; a few rows are
    cut into warps."""
    r = run("""
G.check(G.lib().dftgpu_init(0), "init")
for shape in ((64, 64, 384), (64, 64, 512), (40, 48, 1000), (2, 4, 1024), (64, 48, 32)):
    w, P = G.Wf(shape, 0.8), G.CGrid(shape, 0.8)
    G.lib().grid_wf_boundary(w.ptr, None, 1e-4, 0.003, 0, shape[0], 0, shape[1], 8, shape[2] - 8)
    fake.fake_reset()
    G.lib().grid_wf_absorb_potential(w.ptr, P.ptr, 1e-4, 0.003)
    G.check(what="absorb")
    (l,) = launches()
    result[str(shape)] = [l[k] for k in ("gx", "gy", "gz", "bx", "by")]
""")
    assert r == {"(64, 64, 384)": [2, 64, 64, 192, 1], "(64, 64, 512)": [2, 64, 64, 256, 1],
                 "(40, 48, 1000)": [4, 48, 40, 256, 1], "(2, 4, 1024)": [32, 4, 2, 32, 1],
                 "(64, 48, 32)": [1, 12, 64, 32, 4]}


def test_launches_in_many_chunks_are_ordinary(run):
    """A propagation whose kinetic step runs in more than two chunks a branch launches them without programmatic
    serialization; in fewer chunks, and outside the branches, with it."""
    r = run("""
G.check(G.lib().dftgpu_init(0), "init")
G.set_precision(G.FP32)
for shape in ((512, 512, 128), (240, 240, 240), (64, 64, 64)):
    w, V = G.Wf(shape, 0.8), G.CGrid(shape, 0.8)
    fake.fake_reset()
    w.propagate(V, 1.0 + 0j)
    result[str(shape)] = [l["programmatic"] for l in launches()]
""")
    assert r["(512, 512, 128)"] == [1] + 7 * 3 * [0] + [1]
    assert r["(240, 240, 240)"] == [1] + 3 * 3 * [1] + [1]
    assert r["(64, 64, 64)"] == 5 * [1]


def test_large_reductions_are_launched_ordinarily(run):
    """The partial sums of a reduction over 3 * 2^20 terms or more (its last launch but one) start when everything before
    them has ended, on empty SMs; smaller ones programmatically."""
    r = run("""
G.check(G.lib().dftgpu_init(0), "init")
G.set_precision(G.FP32)
for shape in ((160, 160, 160), (128, 128, 128)):
    w = G.Wf(shape, 0.8)
    fake.fake_reset()
    G.lib().grid_wf_kinetic_energy(w.ptr)
    result[str(shape)] = [l["programmatic"] for l in launches()]
""")
    assert r["(160, 160, 160)"] == [1, 1, 1, 0, 1]
    assert r["(128, 128, 128)"] == 5 * [1]
