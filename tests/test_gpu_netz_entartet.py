"""Body meshes with triangles whose corners are collinear up to rounding, which
Koerpernetz::neu accepts: nearest queries (in the callers' order and sorted) and
the voxelisation against the oracle, value for value.

Two kinds: a closed mesh whose split edges are filled by collinear triangles
(their neighbours share every point, so an answer taken from the wrong triangle
shows in the index and the region), and collinear triangles that stand alone
(then the distance itself shows it)."""
import numpy as np
import pytest

import oracle_py as O
from garmentcraft_b200 import synth
from garmentcraft_b200.netzkoerper import Koerpernetz

pytestmark = pytest.mark.gpu

WERTE = ("abstand", "punkt", "dreieck", "region")


def gefuellt(anzahl, seed):
    """koerper_netz with `anzahl` edges split on one side only: that triangle
    becomes two, and a triangle of the edge's ends and the new point closes
    the gap."""
    p, d = synth.koerper_netz(48, 17, seed=seed)
    rng = np.random.default_rng(seed)
    p, d = [q for q in p], [tuple(int(i) for i in t) for t in d]
    fill = []
    for t in rng.permutation(len(d))[:anzahl]:
        k = int(rng.integers(3))
        j, i, l = d[t][k], d[t][(k + 1) % 3], d[t][(k + 2) % 3]
        m = len(p)
        p.append(p[i] + rng.uniform(0.2, 0.8) * (p[j] - p[i]))
        d[t] = (j, m, l)
        d.append((m, i, l))
        d.append((j, i, m))
        fill.append(len(d) - 1)
    return np.asarray(p), np.asarray(d, dtype=np.uint32), np.asarray(fill)


def dornen(anzahl, seed):
    """koerper_netz and `anzahl` collinear triangles of their own, 4 cm and more
    off the surface and one another; half with corners on a millimetre grid."""
    p, d = synth.koerper_netz(48, 17, seed=seed)
    rng = np.random.default_rng(seed)
    orte = np.stack(np.meshgrid(np.arange(8), np.arange(8), np.arange(8), indexing="ij"), -1).reshape(-1, 3)[:anzahl]
    neu = []
    for k, o in enumerate(orte):
        a = np.array([0.5, -0.4, 0.2]) + 0.11 * o + rng.uniform(0.0, 0.02, 3)
        e = rng.normal(size=3)
        e *= rng.uniform(0.005, 0.05) / np.linalg.norm(e)
        if k % 2:
            a, e = np.round(a, 3), np.round(e, 3)
            e[0] += 0.003
        neu += [a, a + rng.uniform(0.1, 0.9) * e, a + e]
    n = len(p)
    dn = n + np.arange(3 * anzahl).reshape(-1, 3)
    return np.concatenate([p, neu]), np.concatenate([d, dn]).astype(np.uint32), len(d) + np.arange(anzahl)


def anfragen(p, d, dort, anzahl, rng):
    """Points within 1 cm of the triangles `dort`, and anywhere on the surface."""
    t = d[np.where(rng.random(anzahl) < 0.8, rng.choice(dort, anzahl), rng.integers(0, len(d), anzahl))].astype(int)
    b = rng.dirichlet(np.ones(3), size=anzahl)
    r = rng.normal(size=(anzahl, 3))
    return np.einsum("ik,ikc->ic", b, p[t]) + r / np.linalg.norm(r, axis=1)[:, None] * rng.uniform(0.0, 0.01, (anzahl, 1))


@pytest.mark.parametrize("netz", [gefuellt, dornen])
@pytest.mark.parametrize("n", [4000, 20000])
def test_naechster(netz, n):
    p, d, dort = netz(300, seed=4)
    kg, ko = Koerpernetz(p, d, 0.01), O.Koerpernetz(p, d, 0.01)
    x = anfragen(p, d, dort, n, np.random.default_rng(1))
    a, b = kg.naechster(x, 0.015), ko.naechster(x, 0.015)
    assert (b["dreieck"] >= 0).all()
    for k in WERTE:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("netz", [gefuellt, dornen])
def test_sdf(netz):
    p, d, dort = netz(60, seed=5)
    kg, ko = Koerpernetz(p, d, 0.01), O.Koerpernetz(p, d, 0.01)
    for t in dort[:40:8]:
        o, s = p[d[t].astype(int)].mean(axis=0) - 0.03, 0.004
        a, b, exakt = kg.sdf((16, 15, 17), o, s, band=0.02), ko.sdf((16, 15, 17), o, s, band=0.02), ko.sdf((16, 15, 17), o, s)
        nah = np.abs(exakt) < 0.02  # beyond the band an open surface has no side
        assert nah.sum() > 500
        assert np.array_equal(a[nah], b[nah]) and np.array_equal(np.abs(a), np.abs(b))


# Sizes whose coordinates, squares or roundings leave the range of 32 bits
@pytest.mark.parametrize("masstab", [1e-42, 1e-25, 1e25, 1e40])
def test_masstab(masstab):
    p, d = synth.koerper_netz(48, 17, seed=6)
    x = anfragen(p, d, np.arange(len(d)), 3000, np.random.default_rng(2))
    kg, ko = Koerpernetz(p * masstab, d, 0.01 * masstab), O.Koerpernetz(p * masstab, d, 0.01 * masstab)
    a, b = kg.naechster(x * masstab, 0.008 * masstab), ko.naechster(x * masstab, 0.008 * masstab)
    assert 0.5 < (b["dreieck"] >= 0).mean() < 1.0
    for k in WERTE:
        assert np.array_equal(a[k], b[k]), k
    o, s, band = p[0] * masstab, 0.004 * masstab, 0.02 * masstab
    assert np.array_equal(kg.sdf((9, 8, 7), o, s, band=band), ko.sdf((9, 8, 7), o, s, band=band))


@pytest.mark.parametrize("weit", [1e10, 1e22])
def test_ferne_anfragen(weit):
    p, d = synth.koerper_netz(24, 9, seed=6)
    kg, ko = Koerpernetz(p, d, 0.01), O.Koerpernetz(p, d, 0.01)
    x = np.random.default_rng(3).normal(size=(50, 3))
    x *= weit / np.linalg.norm(x, axis=1)[:, None]
    a, b = kg.naechster(x, 2.0 * weit), ko.naechster(x, 2.0 * weit)
    assert (b["dreieck"] >= 0).all()
    for k in WERTE:
        assert np.array_equal(a[k], b[k]), k
