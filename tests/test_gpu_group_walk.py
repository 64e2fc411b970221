"""The single-precision Barnes-Hut walk of 32 Morton neighbours by a warp
(csrc/group_walk.cuh) at the edges of its groups, blocks and parts.

Bars: the forces of the per-thread walk over the same tree, whose terms it adds
in another order (1e-5: float sums of a few hundred terms); and the path's own,
1e-4 norm-wise (2e-3 with prevent_overlap) of the oracle's restatement, where
the regions' centres are not rounded away (tight clumps far from the origin
lose more than that by the float records alone, in every walk). At theta 0
every pair is summed and no record is used: 1e-4 of the double construction.
"""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


def _positions(kind, n, rng):
    if kind == "uniform":
        pos = rng.uniform(-500, 500, (n, 2))
    elif kind == "clusters":  # coincident nodes in clumps of up to 20
        c = rng.uniform(-500, 500, (max(1, n // 10), 2))
        pos = c[rng.integers(0, len(c), n)]
    else:  # "chain": ever closer to a corner, a tree of long chains
        t = 900.0 * 0.93 ** (np.arange(n) % 200)
        pos = np.stack([t, 0.5 * t], 1) + rng.uniform(0, 1e-3, (n, 2))
    return pos.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("kind", ["uniform", "clusters", "chain"])
@pytest.mark.parametrize("n", [2, 8, 9, 31, 32, 33, 128, 129, 1000, 5003])
def test_group_walk_sizes(gpu, orc, n, kind):
    rng = np.random.default_rng(n)
    pos = _positions(kind, n, rng)
    m = 3 * n
    frm, to = rng.integers(0, n, m), rng.integers(0, n, m)
    if n > 200:
        frm[:300] = 0  # a hub: compensated sums in its warp
    g = Graph(n, frm, to, np.ones(m))
    size = rng.uniform(0.5, 3.0, n).astype(np.float32).astype(np.float64)
    for theta, adjust in ((1.2, False), (0.5, False), (0.0, False), (1.2, True)):
        kw = dict(theta=theta, adjust=adjust, size=size)
        go = orc.prepare_large(n, frm, to, np.ones(m))
        p, keep = orc.full_params(go, scaling=2.0, **kw)
        want = orc.pipe_forces(p, pos, "m" if theta > 0 else "d")
        with Layout(g, pos, precision="single", **kw) as L:
            L.option("walk", 1)
            thread = L.forces(pos)
            L.option("walk", 5)
            for split in (1, 2, 4):
                L.option("walk_split", split)
                got = L.forces(pos)
                if theta > 0:
                    assert rel_err(got, thread) <= 1e-5, (theta, adjust, split)
                if kind != "chain" or theta == 0:
                    assert rel_err(got, want) <= (2e-3 if adjust else 1e-4), \
                        (theta, adjust, split)
            L.iterate(2)
            L.sync()
