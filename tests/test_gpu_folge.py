"""The tiled PCG's 32-bit sequence numbers start again before they wrap: solves and
frames across that point, direct and as a graph, equal those of a fresh handle bit
for bit."""
import ctypes as C

import numpy as np
import pytest

from garmentcraft_b200 import _abi
from garmentcraft_b200._lib import lib
from garmentcraft_b200.implizit import ImplizitCg
from garmentcraft_b200.params import ImplizitParameter
from garmentcraft_b200.szene import Szene
from test_gpu_kachel import laken
from test_gpu_kachel_form import dv0, form, lagen

pytestmark = pytest.mark.gpu


def setze(cg, folge):
    f = lib().k3d_test_folge
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32], C.c_int
    assert f(cg._h, folge) == _abi.K3D_OK


# 400 numbers before the end: four launches of 20 iterations at most (two passes of
# two sums) still fit, the fifth starts again
@pytest.mark.parametrize("szene, mehr", [
    (lambda: laken(41), {}), (lambda: laken(129), {"precision": _abi.K3D_MIXED_STORAGE}),
    (lagen, {"selbstkollision": True, "selbst_zusatzdicke": 4e-3}), (lambda: laken(41), {"graph": True}),
    (lambda: Szene.verbinden([laken(n, seed=n) for n in (3, 40, 17)]), {})])
def test_neuer_anfang(szene, mehr):
    s = szene()

    def neu():
        q = s.copy()
        cg = ImplizitCg(ImplizitParameter(**{**dict(schritte_je_bild=2, cg_max=20, cg_toleranz=1e-14), **mehr}))
        cg.hochladen(q)
        return cg, q
    (a, qa), (b, qb) = neu(), neu()
    assert form(a)[0] > 0
    setze(a, 0xffffffff - 400)
    for _ in range(6):
        assert np.array_equal(a.loese(qa, dv0(s))[0], b.loese(qb, dv0(s))[0])
    setze(a, 0xffffffff - 400)
    for _ in range(6):
        a.bild(qa)
        b.bild(qb)
        assert np.isfinite(qa.x).all() and np.array_equal(qa.x, qb.x) and np.array_equal(qa.v, qb.v)
