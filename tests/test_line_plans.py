"""The stages of the generic line transforms, on the CPU (host code of the
library): every length 2^a 3^b 5^c has a plan, every other one is refused, and
the FP32 plans follow one rule at every length."""
import ctypes as C

import numpy as np
import pytest

import libdft_gb300 as G

SMOOTH = sorted(2 ** a * 3 ** b * 5 ** c for a in range(13) for b in range(8) for c in range(6) if 2 ** a * 3 ** b * 5 ** c <= 4096)


def radices(n, prec, small=False):
    f = G.lib()._ZN6dftgpu11fft_radicesEiibPiS0_
    f.argtypes = [C.c_int, C.c_int, C.c_bool, C.POINTER(C.c_int), C.POINTER(C.c_int)]
    r, k = (C.c_int * 16)(), C.c_int()
    rc = f(n, prec, small, r, C.byref(k))
    return list(r[:k.value]) if rc == 0 else None


@pytest.mark.parametrize("prec,small", [(G.FP32, False), (G.FP64, False), (G.FP64, True)])
def test_every_length_has_a_plan(prec, small):
    for n in range(1, 4097):
        r = radices(n, prec, small)
        if n not in SMOOTH:
            assert r is None, n
        else:
            assert np.prod(r, dtype=int) == n and all(2 <= x <= (5 if small else 16) for x in r), (n, r)


def test_fp32_stages():
    """A single 16 stays one stage (as 4 x 4 the error of a line of 16 is 3 % larger), an 8 without a 16 is the first
    stage (its constants offset each other there; second to a 15 it raised the norm tenfold faster), and a 2 beside a 16
    only goes with a 3 or a 5, else the two run as 8 x 4."""
    for n in SMOOTH[1:]:
        r = radices(n, G.FP32)
        two = n & -n
        if two >= 16:
            assert r[0] in (16, 8) and (r[0] == 16 or 4 in r), (n, r)
        if two == 8:
            assert r[0] == 8, (n, r)
        if two == n and 16 <= n:
            assert 2 not in r, (n, r)
        assert not (16 in r and 2 in r), (n, r)
    assert radices(16, G.FP32) == [16]
