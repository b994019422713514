"""The launch-shape tuner's records outlive the library that wrote them: one that
chose among other launch forms is not replayed (a fake device, no GPU)."""
import json

from garmentcraft_b200 import autotune, synth
from garmentcraft_b200.implizit import build_scene
from garmentcraft_b200.params import ImplizitParameter


class Geraet:
    """The solver's interface as the tuner uses it; 256 CTA threads are slower."""
    gezeitet = 0

    def __init__(self, param, device=0):
        self.param = param

    def loeser_name(self):
        return "B200 (f64)"

    def pcg_bloecke(self):
        return 8

    def hochladen(self, s):
        pass

    def zustand_hochladen(self, s):
        pass

    def bilder_auf_geraet(self, n):
        Geraet.gezeitet += 1

    def letzte_bild_ms(self):
        return 2.0 if self.param.pcg_threads == 256 else 1.0


def test_alte_aufzeichnung(tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "ImplizitCg", Geraet)
    m, k = synth.sheet_over_sphere(n=9, seed=1)
    s, p, pfad = build_scene(m, [k]), ImplizitParameter(), str(tmp_path / "t.json")
    key = autotune.schluessel("B200 (f64)", p, s)
    with open(pfad, "w") as f:  # as the library before the tiled PCG wrote it
        json.dump({key: {"pcg_threads": 256, "pcg_bloecke": 8, "graph": False, "ms_je_bild": 1.0, "bilder": 3,
                         "kandidaten": []}}, f)
    q, _ = autotune.abstimmen(s, p, cache=pfad)
    assert Geraet.gezeitet > 0 and q.pcg_threads == 512
    n = Geraet.gezeitet
    q, rec = autotune.abstimmen(s, p, cache=pfad)
    assert Geraet.gezeitet == n and q.pcg_threads == 512 and rec["formen"] == autotune.FORMEN
