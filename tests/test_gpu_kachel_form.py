"""Which PCG launch a scene takes: the tiled one with the tiles that the host planned
(tests/test_kachelplan.py holds the plans to their rules), or the one over ELL rows
where a tile does not fit. The comparisons of tests/test_gpu_kachel.py mean
something only if the tiled launch ran. Also scenes that one handle takes in turn,
and the adjoint on compact tiles."""
import ctypes as C

import numpy as np
import pytest

from garmentcraft_b200 import _abi, synth
from garmentcraft_b200._lib import lib
from garmentcraft_b200.implizit import ImplizitCg, build_scene
from garmentcraft_b200.params import ImplizitParameter
from garmentcraft_b200.szene import Szene
from test_gpu_kachel import gleich, laken

pytestmark = pytest.mark.gpu

F64, F32 = _abi.K3D_FP64, _abi.K3D_MIXED_STORAGE


def form(cg):
    """(rows a thread, 0 on ELL rows; tiles; slabs; streamed slabs)"""
    f = lib().k3d_test_form
    f.argtypes, f.restype = [C.c_void_p, C.POINTER(C.c_int64)], None
    out = (C.c_int64 * 4)()
    f(cg._h, out)
    return tuple(out)


def loeser(s, prec, **mehr):
    cg = ImplizitCg(ImplizitParameter(schritte_je_bild=1, cg_max=20, cg_toleranz=1e-14, precision=prec, **mehr))
    cg.hochladen(s)
    return cg


def dv0(s):
    return np.random.default_rng(1).normal(0.0, 0.01, size=s.x.shape)


def lagen(groesse=0.2, kante_mm=10.0):
    s = build_scene(synth.zwei_lagen(groesse_m=groesse, kante_mm=kante_mm, abstand_m=0.003, versatz_m=(0.0013, 0.0007)))
    synth.pin_teil(s, 0)
    s.param.bild_dt = 1.0 / 600.0
    return s


@pytest.mark.parametrize("n, bloecke, prec, q, strom", [
    (2, 0, F64, 1, False), (33, 0, F32, 1, False), (128, 0, F64, 1, False), (129, 0, F64, 1, False),
    (257, 0, F32, 1, True), (257, 0, F64, 1, True), (300, 0, F64, 2, True), (400, 0, F64, 3, True),
    (400, 0, F32, 3, True), (41, 1, F64, 4, True), (41, 2, F32, 2, True), (41, 7, F64, 1, True)])
def test_form(n, bloecke, prec, q, strom):
    f = form(loeser(laken(n), prec, pcg_bloecke=bloecke))
    assert f[0] == q and 0 < f[1] <= (bloecke or 148) and (f[3] > 0) == strom
    assert form(loeser(laken(n), prec, pcg_bloecke=bloecke, pcg_threads=256)) == (0, 0, 0, 0)


@pytest.mark.parametrize("prec", [F64, F32])
def test_form_andere(prec):
    assert form(loeser(Szene.verbinden([laken(n, seed=n) for n in (3, 9, 40, 95, 17)]), prec))[0] > 0
    assert form(loeser(lagen(), prec, selbstkollision=True))[0] == 1
    assert form(loeser(laken(33), _abi.K3D_MIXED)) == (0, 0, 0, 0)  # FP32 vectors


# more than four rows a thread on one and on three CTAs; FP32 blocks beyond what the shared memory takes
@pytest.mark.parametrize("n, bloecke, prec", [(50, 1, F32), (300, 3, F64), (480, 0, F32)])
def test_zu_gross(n, bloecke, prec):
    s = laken(n)
    a, b = (loeser(s, prec, pcg_bloecke=bloecke, pcg_threads=t) for t in (0, 256))
    assert form(a) == (0, 0, 0, 0)
    gleich(a.loese(s, dv0(s))[0], b.loese(s, dv0(s))[0], "dv")


@pytest.mark.parametrize("selbst", [False, True])
def test_ein_handle_im_wechsel(selbst):
    # tiles, ELL rows, tiles: each scene solved as by a handle of its own
    klein, gross = (lagen(), lagen(0.6, 4.0)) if selbst else (laken(41), laken(300))
    mehr = dict(pcg_bloecke=3, selbstkollision=selbst, selbst_zusatzdicke=4e-3)
    cg = loeser(klein, F64, **mehr)
    for s, q in ((klein, True), (gross, False), (klein, True)):
        cg.hochladen(s)
        assert (form(cg)[0] > 0) == q
        a, b = cg.loese(s, dv0(s))[0], loeser(s, F64, **mehr).loese(s, dv0(s))[0]
        assert np.array_equal(a, b)


def test_adjoint_auf_kompakten_kacheln():
    # 16,900 points: the gradient against the launch over ELL rows. Solves to 1e-14 of
    # the residual at a condition of some 1e5 differ by 1e-9, and few follow one another
    m, body = synth.sheet_over_sphere(n=130, jitter_mm=1.0, seed=5, fall_m=0.002, sdf_n=64, sdf_spacing_m=0.02)
    s = build_scene(m, [body])
    s.param.bild_dt = 1.0 / 1200.0
    s.v[:, 2] -= 1.0
    rng = np.random.default_rng(3)
    gx, gv = rng.normal(size=s.x.shape), 1e-2 * rng.normal(size=s.x.shape)
    aus = []
    for threads in (0, 256):
        cg = ImplizitCg(ImplizitParameter(schritte_je_bild=1, cg_max=100000, cg_toleranz=1e-14, pcg_threads=threads))
        t = s.copy()
        cg.hochladen(t)
        assert (form(cg)[0] > 0) == (threads == 0)
        cg.adjoint_vorwaerts(3, 2)
        aus.append(cg.adjoint_rueckwaerts(gx, gv))
    for k in ("x", "v", "membran", "biegung"):
        a, b = aus[0][k], aus[1][k]
        assert np.linalg.norm(b) > 0.0
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b), k
