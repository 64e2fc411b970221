"""The speed's totals of small FP32 all-pairs layouts (k_small_exact) keep what
the sum over the blocks rounds off.

Places that are powers of two under strong gravity alone make every node's
swinging a power of two exactly. One value of 2^58 meets sums of half its
spacing, 32, at every step of the sum in pairs over the blocks, of which plain
double additions lose all: two spacings with 16 blocks. The totals are within
one spacing of the exact sum (math.fsum)."""
import math

import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout, REPULSION_EXACT

pytestmark = pytest.mark.gpu

N = 1024
SETTINGS = dict(scaling=0.0, strong=True, gravity=1.0, precision="single")


def graph(stride):
    """2^58 at node 0, 32 at the nodes stride 1, 2, 4, 8 and 16."""
    none = np.zeros(0, np.int32)
    pos = np.zeros((N, 2))
    pos[0, 0] = 2.0 ** 58
    for k in (1, 2, 4, 8, 16):
        if k * stride < N:
            pos[k * stride, 0] = 32.0
    return Graph(N, none, none, np.zeros(0)), pos


def check(speed, sw):
    want = math.fsum(sw)
    assert abs(speed["total_swinging"] - want) <= math.ulp(want)
    assert abs(speed["total_traction"] - want / 2) <= math.ulp(want / 2)


@pytest.mark.parametrize("blocks", [2, 4, 8, 16])
def test_cluster_totals_are_compensated(gpu, blocks):
    g, pos = graph(N // blocks)  # a block each
    with Layout(g, pos, repulsion=REPULSION_EXACT, **SETTINGS) as L:
        L.option("exact_cluster", blocks)
        L.iterate(1)
        L.sync()
        sw = L.swing()
        np.testing.assert_array_equal(sw, pos[:, 0])
        check(L.speed(), sw)


@pytest.mark.parametrize("n", [2, 31, 33, 100, 500, 1025, 1500, 2500])
def test_totals_equal_exact_sums(gpu, n):
    """Ordinary values: 1e-12, the bar of the totals elsewhere."""
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    g = Graph(n, a, b, np.ones(3 * n))
    pos = rng.uniform(-50, 50, (n, 2)).astype(np.float32).astype(np.float64)
    with Layout(g, pos, repulsion=REPULSION_EXACT) as L:
        if n <= 1500:
            L.option("exact_cluster", 16)
        L.option("keep_traction", 1)
        L.iterate(3)
        L.sync()
        sw, tr = L.swing(True)
        speed = L.speed()
    for got, vals in ((speed["total_swinging"], sw), (speed["total_traction"], tr)):
        want = math.fsum(vals)
        assert abs(got - want) <= 1e-12 * want


@pytest.mark.parametrize("blocks", [1, 3, 16])
def test_infinite_totals_stop_the_layout(gpu, blocks):
    n = 300
    none = np.zeros(0, np.int32)
    pos = np.random.default_rng(n).uniform(100, 200, (n, 2)).astype(np.float32).astype(np.float64)
    with Layout(Graph(n, none, none, np.zeros(0)), pos, repulsion=REPULSION_EXACT, scaling=0.0,
                strong=True, gravity=3e38) as L:
        L.option("exact_cluster", blocks)
        L.iterate(1)
        with pytest.raises(RuntimeError, match="invalid numbers"):
            L.sync()
        np.testing.assert_array_equal(L.positions(), pos)
