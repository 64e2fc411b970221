"""Single-precision Barnes-Hut forces with masses of either sign: a region's
centre of mass may lie outside its box, and is taken where it is. Bar: the path's
own, 1e-4 norm-wise of the double-precision forces."""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("n", [40, 700, 3000])
def test_forces_with_signed_masses_match_double(gpu, n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-100, 100, (n, 2)).astype(np.float32).astype(np.float64)
    frm, to = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    g = Graph(n, frm, to, np.ones(3 * n))
    g.mass = np.where(rng.random(n) < 0.3, -1.0, 1.0) * \
        rng.uniform(1, 9, n).astype(np.float32).astype(np.float64)
    with Layout(g, pos, precision="double") as L:
        want = L.forces(pos)
    with Layout(g, pos, precision="single") as L:
        assert rel_err(L.forces(pos), want) <= 1e-4
    with Batch([g], [pos], exact_below=0, threads=256, nodes_per_thread=1) as B:
        B.iterate(1)
        assert rel_err(B.forces(0), want) <= 1e-4
