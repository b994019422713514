"""Self-collision springs far denser than a garment's: the tiled PCG, whose merged
rows are counted before they get their room, against the launch over ELL rows
(pcg_threads=256): the same solve, in no more device memory."""
import numpy as np
import pytest
import torch

from garmentcraft_b200 import _abi, synth
from garmentcraft_b200.implizit import ImplizitCg, build_scene
from garmentcraft_b200.params import ImplizitParameter
from garmentcraft_b200.szene import Szene

pytestmark = pytest.mark.gpu


def stapel(lagen, groesse, abstand):
    """`lagen` square layers of 4 mm meshes, `abstand` apart, as one scene."""
    teile = []
    for k in range(lagen // 2):
        s = build_scene(synth.zwei_lagen(groesse_m=groesse, kante_mm=4.0, abstand_m=abstand, versatz_m=(0.0013, 0.0007)))
        s.x[:, 2] += 2 * abstand * k
        s.x[:, 0] += 0.0003 * k
        teile.append(s)
    s = Szene.verbinden(teile)
    s.instanz_punkte = np.zeros(0, dtype=np.int64)
    s.v[:] = np.random.default_rng(2).normal(0.0, 0.02, size=s.v.shape)
    s.param.bild_dt = 1.0 / 600.0
    return s


# layers, side, distance, extra thickness, least pairs a point: rows of up to some
# 350 neighbours, and of more than the 512 that are counted exactly
@pytest.mark.parametrize("lagen, groesse, abstand, dicke, dicht", [
    (60, 0.04, 5e-4, 2.5e-2, 200), (120, 0.024, 2.5e-4, 2.5e-2, 350)])
@pytest.mark.parametrize("prec", [_abi.K3D_FP64, _abi.K3D_MIXED_STORAGE])
def test_wie_ell(prec, lagen, groesse, abstand, dicke, dicht):
    s = stapel(lagen, groesse, abstand)
    dv0 = np.random.default_rng(1).normal(0.0, 0.01, size=s.x.shape)
    dv, bytes_ = [], []
    for threads in (0, 256):
        q = s.copy()
        cg = ImplizitCg(ImplizitParameter(schritte_je_bild=1, cg_max=20, cg_toleranz=1e-14, precision=prec,
                                          pcg_threads=threads, selbstkollision=True, selbst_zusatzdicke=dicke))
        cg.hochladen(q)
        frei = torch.cuda.mem_get_info()[0]
        dv.append([cg.loese(q, dv0)[0] for _ in range(2)])  # the second run finds its room
        bytes_.append(frei - torch.cuda.mem_get_info()[0])
        paare = len(cg.selbst_paare()["art"])
        del cg
    assert paare > dicht * s.n
    print(f"{s.n} points, {paare} pairs: {bytes_[0] / paare:.0f} bytes a pair, over ELL rows {bytes_[1] / paare:.0f}")
    assert np.array_equal(dv[0][0], dv[0][1])
    assert np.linalg.norm(dv[0][0] - dv[1][0]) <= 1e-9 * np.linalg.norm(dv[1][0])
    assert bytes_[0] <= bytes_[1] + (4 << 20)
