"""The tree kernel at the edges of its blocks and windows: keys, order, child,
range and parent equal to the oracle's construction bit for bit, in one launch
and in two, on positions that make balanced trees, long chains and ties."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


def _positions(kind, n, rng):
    if kind == "uniform":
        pos = rng.uniform(-50, 50, (n, 2))
    elif kind == "coincident":
        pos = rng.uniform(-50, 50, (3, 2))[rng.integers(0, 3, n)]
    else:  # "chain": each node twice as close to a corner as the one before
        pos = np.stack([0.5 ** (np.arange(n) % 40)] * 2, 1) + rng.uniform(0, 1e-6, (n, 2))
    return pos.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("kind", ["uniform", "coincident", "chain"])
@pytest.mark.parametrize("n", [2, 3, 64, 127, 128, 129, 192, 193, 256, 257, 1000, 4097])
def test_tree_matches_oracle(gpu, orc, n, kind):
    pos = _positions(kind, n, np.random.default_rng(n))
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    g.mass = np.random.default_rng(1).integers(1, 9, n).astype(np.float64)
    want = orc.pipe_build(n, pos, g.mass, "d")
    for precision in ("double", "single"):
        with Layout(g, pos, precision=precision) as L:
            for climb in (1, 2):
                L.option("climb", climb)
                for again in range(2):  # the splits' slots are left as they were
                    t = L.tree(pos)
                    for k in ("key", "order", "child", "range", "parent"):
                        np.testing.assert_array_equal(t[k], want[k], err_msg=f"{precision} {k}")
                    if precision == "double":
                        np.testing.assert_array_equal(t["ni"], want["ni"])
                    else:
                        np.testing.assert_allclose(t["ni"][:, 2], want["ni"][:, 2], rtol=1e-6)
