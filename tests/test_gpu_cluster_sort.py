"""Codes and sort of a layout in one thread-block cluster (k_codes_sort) at the
edges of its blocks, rounds and shapes: keys, order and tree equal to the
separate launches' bit for bit (which the other tests hold to the oracle)."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n", [2, 3, 31, 33, 256, 257, 2000, 2001, 8191, 32768, 32769, 65536,
                               65537, 110000])
def test_cluster_sort_equals_tiled(gpu, n, precision):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-100, 100, (n, 2)).astype(np.float32).astype(np.float64)
    pos[n // 3:n // 2] = pos[0]  # equal keys: the order is the index's
    none = np.zeros(0, np.int32)
    with Layout(Graph(n, none, none, np.zeros(0)), pos, precision=precision) as L:
        got = {0: L.tree(pos)}  # the default
        for blocks in (1, 2, 5, 16):
            if -(-n // blocks) <= 8192:
                L.option("sort_cluster", blocks)
                got[blocks] = L.tree(pos)
        L.option("sort_cluster", 0)
        L.option("sort_threads", 256)
        want = L.tree(pos)
        with pytest.raises(RuntimeError):
            L.option("sort_cluster", 17)
    assert len(np.unique(want["order"])) == n
    for blocks, t in got.items():
        for k in ("key", "order", "child", "range", "parent", "ni"):
            np.testing.assert_array_equal(t[k], want[k], err_msg=f"{blocks} {k}")
