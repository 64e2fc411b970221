"""The group walk's unused places (odd numbers of far regions) add nothing to
any node, wherever it lies: a node at (-1e18, -1e18) in float, among near
neighbours, in layouts whose forces are finite. Bar: the path's own, 1e-4
norm-wise of the double-precision forces."""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("n", [200, 2000])
def test_node_at_the_old_filler(gpu, n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1e18, 1e18, (n, 2))
    pos[:n // 4] = -1e18 + rng.uniform(-1e17, 1e17, (n // 4, 2))
    pos = pos.astype(np.float32).astype(np.float64)
    pos[n // 8] = float(np.float32(-1e18))
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    # (float places here are 7e10 apart: centres off by 1e-5 of the distances at most)
    settings = dict(gravity=0.0, scaling=2.0)
    with Layout(g, pos, precision="double", **settings) as L:
        want = L.forces(pos)
    assert np.isfinite(want).all()
    with Layout(g, pos, precision="single", **settings) as L:
        for split in (1, 2, 4):
            L.option("walk_split", split)
            assert rel_err(L.forces(pos), want) <= 1e-4, split
    with Batch([g], [pos], exact_below=0, threads=256, nodes_per_thread=1, **settings) as B:
        B.iterate(1)
        B.sync()
        assert rel_err(B.forces(0), want) <= 1e-4
