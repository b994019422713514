"""Nearest queries in bulk: the sorted route (from 16,384 queries on) against
the route in the callers' order, bit for bit, and both against the oracle on a
part; on a body whose poles are slivers, with radii below and above a cell, and
queries outside the grid or not finite."""
import numpy as np
import pytest

import oracle_py as O
from garmentcraft_b200 import synth
from garmentcraft_b200.netzkoerper import Koerpernetz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16383, 16384, 40001])
@pytest.mark.parametrize("radius", [0.004, 0.03])
def test_sortiert_wie_einzeln(n, radius):
    p, d = synth.koerper_netz(96, 31, seed=2)
    kg, ko = Koerpernetz(p, d, 0.01), O.Koerpernetz(p, d, 0.01)
    rng = np.random.default_rng(n)
    t = d[rng.integers(0, d.shape[0], size=n)].astype(np.int64)
    x = np.einsum("ik,ikc->ic", rng.dirichlet(np.ones(3), size=n), p[t]) + rng.normal(0.0, 0.5 * radius, size=(n, 3))
    x[:200] = p[rng.integers(0, p.shape[0], size=200)]        # on points: ties of all their triangles
    x[200:300, 2] += 0.5 * radius                             # off the surface
    x[300:310] = rng.uniform(-5.0, 5.0, size=(10, 3))         # outside the grid
    x[310] = np.nan
    x[311, 0] = np.inf
    a = kg.naechster(x, radius)
    teile = [kg.naechster(x[i:i + 5000], radius) for i in range(0, n, 5000)]
    for k in a:
        assert np.array_equal(a[k], np.concatenate([q[k] for q in teile])), k
    m = 1500
    b = ko.naechster(x[:m], radius)
    assert np.array_equal(a["dreieck"][:m], b["dreieck"])
    hat = b["dreieck"] >= 0
    assert hat.sum() > m // 2
    for k in ("abstand", "punkt", "region"):
        assert np.array_equal(a[k][:m][hat], b[k][hat]), k
