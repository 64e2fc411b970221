"""FP32 graphs whose work outlasts the rest of a batch are laid out by blocks of
1,024 threads: the same layout, bit for bit, as by a block of 256 or 512."""
import numpy as np
import pytest

from forceatlas2_rc_gb300 import graphs as G
from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph

pytestmark = pytest.mark.gpu


def case(n, seed, hub):
    n, a, b = G.erdos_renyi(n, 6.0, seed=seed)
    if hub:  # a node joined to every fourth one
        far = np.arange(1, n, 4)
        a = np.concatenate([a, np.zeros(len(far), a.dtype)])
        b = np.concatenate([b, far.astype(b.dtype)])
    r = 10.0 * np.sqrt(n)
    pos = np.random.default_rng(seed).uniform(-r, r, (n, 2)).astype(np.float32)
    return Graph(n, a, b, np.ones(len(a))), pos.astype(np.float64)


@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("n,hub,settings", [
    (1023, False, {}),  # never wide
    (1024, False, {}),
    (1025, False, dict(linlog=True)),
    (2047, False, dict(strong=True)),
    (2049, True, {}),
    (5003, False, dict(adjust=True)),
    (5003, True, dict(adjust=True)),
])
def test_wide_blocks_give_the_same_layout(gpu, n, hub, settings, threads):
    """Alone a graph is more than its share of the work (a wide block if it has
    1,024 nodes); among 640 equal ones it is less than half of an SM's."""
    args = dict(precision="single", exact_below=64, threads=threads, nodes_per_thread=2,
                scaling=2.0, gravity=1.0, **settings)
    g, pos = case(n, n, hub)

    def run(count, others=()):
        gs = [g] * count + [o[0] for o in others]
        ps = [pos] * count + [o[1] for o in others]
        with Batch(gs, ps, **args) as B:
            B.iterate(3)
            B.iterate(4)
            B.sync()
            return B.positions(0), B.positions(len(gs) - 1), B.speed(0)

    alone = run(1)
    many = run(640)
    np.testing.assert_array_equal(alone[0], many[0])
    np.testing.assert_array_equal(alone[0], many[1])
    assert alone[2] == many[2]
    # wide and other blocks in one launch
    small = [case(k, k, False) for k in (2, 70, 300)]
    mixed = run(3, small)
    np.testing.assert_array_equal(alone[0], mixed[0])
    with Batch([small[-1][0]], [small[-1][1]], **args) as B:
        B.iterate(7)
        B.sync()
        np.testing.assert_array_equal(B.positions(0), mixed[1])
