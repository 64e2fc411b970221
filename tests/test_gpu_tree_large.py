"""The tree of large layouts, in two launches and with narrow windows (224 leaves
a block): keys, order, child, range and parent equal to the oracle's
construction bit for bit, with coincident nodes and clusters, twice over."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [400_000, 400_001, 403_211])
def test_large_tree_matches_oracle(gpu, orc, n):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1000, 1000, (n, 2))
    third = n // 3
    pos[:third] = rng.uniform(-1000, 1000, (500, 2))[rng.integers(0, 500, third)] + \
        rng.normal(0, 0.3, (third, 2))  # clusters
    ties = rng.integers(0, n, n // 50)
    pos[ties] = pos[rng.integers(0, 40, len(ties))]
    pos = pos.astype(np.float32).astype(np.float64)
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    g.mass = rng.integers(1, 9, n).astype(np.float64)
    want = orc.pipe_build(n, pos, g.mass, "d")
    for precision in ("double", "single"):
        with Layout(g, pos, precision=precision) as L:
            for again in range(2):
                t = L.tree(pos)
                for k in ("key", "order", "child", "range", "parent"):
                    np.testing.assert_array_equal(t[k], want[k], err_msg=f"{precision} {k}")
                if precision == "double":
                    np.testing.assert_array_equal(t["ni"], want["ni"])
                else:
                    np.testing.assert_allclose(t["ni"][:, 2], want["ni"][:, 2], rtol=1e-6)
