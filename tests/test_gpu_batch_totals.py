"""The speed's totals of FP32 batches (block_sums) keep what the sum over the
warps rounds off, and infinite ones stop a graph.

Places that are powers of two under strong gravity alone make every node's
swinging a power of two exactly. One value of 2^58 meets sums of half its
spacing, 32, at every step of the sum in pairs over 32 warps: plain double
additions lose 2.5 spacings. The totals are within one spacing of the exact sum
(math.fsum)."""
import math

import numpy as np
import pytest

from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph

pytestmark = pytest.mark.gpu

N = 1024
SETTINGS = dict(scaling=0.0, strong=True, gravity=1.0, precision="single")


def graph():
    """2^58 at node 0, 32 at a node of the warps 1, 2, 4, 8 and 16."""
    none = np.zeros(0, np.int32)
    pos = np.zeros((N, 2))
    pos[0, 0] = 2.0 ** 58
    for k in (1, 2, 4, 8, 16):
        pos[32 * k, 0] = 32.0
    return Graph(N, none, none, np.zeros(0)), pos


def check(speed, sw):
    want = math.fsum(sw)
    assert abs(speed["total_swinging"] - want) <= math.ulp(want)
    assert abs(speed["total_traction"] - want / 2) <= math.ulp(want / 2)


@pytest.mark.parametrize("threads", [256, 512])
def test_batch_totals_are_compensated(gpu, threads):
    g, pos = graph()
    with Batch([g], [pos], exact_below=1 << 20, threads=threads, nodes_per_thread=2,
               **SETTINGS) as B:
        B.iterate(1)
        B.sync()
        sw = np.abs(B.forces(0)[:, 0])
        np.testing.assert_array_equal(sw, pos[:, 0])
        check(B.speed(0), sw)


@pytest.mark.parametrize("n", [1, 20, 33, 300, 1500, 3000])
@pytest.mark.parametrize("exact_below", [1 << 20, 64])
def test_float_batch_stops_at_infinite_totals(gpu, n, exact_below):
    """Forces beyond the float range: infinite totals, no NaN among the nodes'
    values."""
    none = np.zeros(0, np.int32)
    pos = np.random.default_rng(n).uniform(100, 200, (n, 2)).astype(np.float32).astype(np.float64)
    with Batch([Graph(n, none, none, np.zeros(0))], [pos], exact_below=exact_below, threads=256,
               nodes_per_thread=1, scaling=0.0, strong=True, gravity=3e38) as B:
        B.iterate(1)
        with pytest.raises(RuntimeError, match="invalid numbers"):
            B.sync()
        np.testing.assert_array_equal(B.positions(0), pos)
