"""A device wait of the tiled PCG that runs out: the solve ends with K3D_TIMEOUT
within the limit, later substeps of the frame end at once, and the same handle
then solves as a fresh one does, bit for bit. The wait is for a posted word that
no CTA posts, with a limit of a quarter of a second."""
import ctypes as C
import time

import numpy as np
import pytest

from garmentcraft_b200 import _abi, synth
from garmentcraft_b200._lib import K3dError, lib
from garmentcraft_b200.implizit import ImplizitCg, build_scene
from garmentcraft_b200.params import ImplizitParameter
from test_gpu_kachel import laken

pytestmark = pytest.mark.gpu

FRIST = 0.25


def stumm(cg, sekunden, nach):
    f = lib().k3d_test_wait
    f.argtypes, f.restype = [C.c_void_p, C.c_double, C.c_int64], None
    f(cg._h, sekunden, nach)


def lagen():
    s = build_scene(synth.zwei_lagen(groesse_m=0.2, kante_mm=10.0, abstand_m=0.003, versatz_m=(0.0013, 0.0007)))
    synth.pin_teil(s, 0)
    s.param.bild_dt = 1.0 / 600.0
    return s


# resident slabs alone, and FP64 blocks at two rows a thread, whose next
# product's copies are on their way when the sum fails
@pytest.mark.parametrize("prec, szene, selbst", [
    (_abi.K3D_FP64, lambda: laken(41), False), (_abi.K3D_MIXED_STORAGE, lambda: laken(129), False),
    (_abi.K3D_FP64, lambda: laken(300), False), (_abi.K3D_MIXED_STORAGE, lambda: laken(300), False),
    (_abi.K3D_FP64, lagen, True)])
def test_frist(prec, szene, selbst):
    s = szene()
    dv0 = np.random.default_rng(1).normal(0.0, 0.01, size=s.x.shape)

    def neu():
        q = s.copy()
        cg = ImplizitCg(ImplizitParameter(schritte_je_bild=4, cg_max=20, cg_toleranz=1e-14, precision=prec,
                                          selbstkollision=selbst, selbst_zusatzdicke=4e-3))
        return cg, q, cg.loese(q, dv0)[0]

    cg, q, _ = neu()
    for nach in (0, 3):
        for ruf in (lambda: cg.loese(q, dv0), lambda: cg.bild(q)):
            stumm(cg, FRIST, nach)
            t0 = time.perf_counter()
            with pytest.raises(K3dError) as e:
                ruf()
            assert e.value.status == _abi.K3D_TIMEOUT
            assert time.perf_counter() - t0 < 4 * FRIST
            stumm(cg, 4.0, -1)
            q.x[:], q.v[:] = s.x, s.v
            a, b = cg.loese(q, dv0)[0], neu()[2]
            assert np.isfinite(a).all() and np.array_equal(a, b)
