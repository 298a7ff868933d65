"""FP32 grids large enough that a convolution's planes run in halves on two
branches (spectra above 48 MB) and the kinetic step in chunks (above 40 MB;
beyond four chunks with ordinary launches): bit for bit the results of one
branch (DFTGPU_STREAMS=1), for register-kernel and generic lengths, launched
singly and replayed."""
import hashlib
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CASES = [((192, 192, 192), 9), ((180, 200, 216), 9), ((160, 512, 320), 0)]   # odd numbers of planes; 2, 2 and 6 chunks


def digests(G, shape, model):
    G.set_precision(G.FP32)
    try:
        rng = np.random.default_rng(5)
        rho0 = 0.0218360 * 0.529177210903 ** 3
        psi = np.sqrt(rho0) * (1 + 0.05 * rng.standard_normal(shape)) * np.exp(0.1j * rng.standard_normal(shape))
        w, wp, P = G.Wf(shape, 0.8), G.Wf(shape, 0.8), G.CGrid(shape, 0.8)
        ot = G.OT(model, w, min_ns=2, max_ns=4)
        w.set(psi)
        P.zero()
        ot.potential(P, w)
        out = [hashlib.sha256(P.get().tobytes()).hexdigest()]
        for _ in range(2):   # a potential and a step launched singly, then two of each by the run call
            ot.pc_step(w, wp, P, None, 0.0, 41.3 + 0j)
            out.append(hashlib.sha256(w.get().tobytes()).hexdigest())
        ot.run(w, wp, P, None, 0.0, 41.3 + 0j, 3, False)
        out.append(hashlib.sha256(w.get().tobytes()).hexdigest())
        assert np.isfinite(w.norm())
        for o in (ot, P, wp, w):
            o.free()
    finally:
        G.set_precision(G.FP64)
    return out


CHILD = """
import json, sys
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
import libdft_gb300 as G
from test_parallel_branches import CASES, digests
G.check(G.lib().dftgpu_init(0), "init")
print(json.dumps([digests(G, *c) for c in CASES]))
"""


def test_branches_do_not_change_results(gpu):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=dict(os.environ, DFTGPU_STREAMS="1"), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    for case, one in zip(CASES, json.loads(r.stdout.splitlines()[-1])):
        assert digests(gpu, *case) == one, case
