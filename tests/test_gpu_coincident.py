"""Single-precision Barnes-Hut forces on layouts with coincident nodes: a
region of size 0 must not be far from its own nodes because its centre of mass
was rounded off their common position. Bar: the path's own, 1e-4 norm-wise of
the double-precision forces from the same float positions."""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,places", [(2, 1), (12, 3), (300, 20)])
def test_coincident_nodes_match_double(gpu, n, places):
    for seed in range(20):
        rng = np.random.default_rng(seed)
        c = rng.uniform(-500, 500, (places, 2)).astype(np.float32).astype(np.float64)
        pos = c[rng.integers(0, places, n)]
        frm, to = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
        g = Graph(n, frm, to, np.ones(3 * n))
        with Layout(g, pos, precision="double") as L:
            want = L.forces(pos)
        with Layout(g, pos, precision="single") as L:
            assert rel_err(L.forces(pos), want) <= 1e-4, seed
