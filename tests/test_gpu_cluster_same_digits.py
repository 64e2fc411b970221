"""The cluster sort (k_codes_sort) where its blocks' pairs come from themselves:
digits that all nodes share, or all but one far node, whose passes keep every
pair in its block. Keys, order and tree equal to the tiled sort's bit for bit,
time after time."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["coincident", "outlier", "two places", "line"])
@pytest.mark.parametrize("n", [50, 2001, 8192, 30011])
def test_cluster_sort_of_same_digits(gpu, n, kind):
    rng = np.random.default_rng(n)
    pos = np.full((n, 2), 3.0)
    if kind == "outlier":
        pos = rng.uniform(0, 1, (n, 2))
        pos[n // 2] = 1e4
    elif kind == "two places":
        pos[n // 2:] = 7.0
    elif kind == "line":
        pos[:, 0] = np.arange(n)
    pos = pos.astype(np.float32).astype(np.float64)
    none = np.zeros(0, np.int32)
    with Layout(Graph(n, none, none, np.zeros(0)), pos) as L:
        L.option("sort_cluster", 0)
        L.option("sort_threads", 256)
        want = L.tree(pos)
        assert (want["order"][np.argsort(want["order"])] == np.arange(n)).all()
        for blocks in (1, 2, 4, 16):
            if -(-n // blocks) > 8192:
                continue
            L.option("sort_cluster", blocks)
            for again in range(5):
                got = L.tree(pos)
                for k in ("key", "order", "child", "range", "parent", "ni"):
                    np.testing.assert_array_equal(got[k], want[k], err_msg=f"{blocks} {k}")
