"""FP64 totals made in parallel (ordered_sum) of values that are not numbers, or
have a sign: a NaN stops a layout, or a batch, before its displacement wherever
it stands among the nodes and whatever its sign, and values of either sign are
added in node order."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph, Layout, REPULSION_BH, REPULSION_EXACT

pytestmark = pytest.mark.gpu


def late_nan(n, value):
    """The last two nodes joined by an edge of strength `value`; the others'
    forces are finite (strong gravity alone)."""
    pos = np.random.default_rng(n).uniform(1, 20, (n, 2))
    g = Graph(n, np.array([n - 2]), np.array([n - 1]), np.ones(1))
    g.inc_coef = np.full(2, value)
    return g, pos


SETTINGS = dict(precision="double", scaling=0.0, strong=True)


@pytest.mark.parametrize("value", [np.nan, -np.nan], ids=["nan", "-nan"])
@pytest.mark.parametrize("n", [4, 40, 300, 2048])
def test_double_layout_stops_at_a_late_nan(gpu, n, value):
    g, pos = late_nan(n, value)
    for repulsion in (REPULSION_EXACT, REPULSION_BH):
        with Layout(g, pos, repulsion=repulsion, **SETTINGS) as L:
            L.iterate(1)
            with pytest.raises(RuntimeError, match="invalid numbers"):
                L.sync()
            np.testing.assert_array_equal(L.positions(), pos)


@pytest.mark.parametrize("value", [np.nan, -np.nan], ids=["nan", "-nan"])
def test_double_batch_stops_at_a_late_nan(gpu, value):
    cases = [late_nan(n, value) for n in (4, 40, 300, 2048)]
    for exact_below in (1 << 20, 0):
        with Batch([c[0] for c in cases], [c[1] for c in cases], exact_below=exact_below,
                   threads=256, nodes_per_thread=1, **SETTINGS) as B:
            B.iterate(1)
            with pytest.raises(RuntimeError, match="invalid numbers"):
                B.sync()
            for k, (_, pos) in enumerate(cases):
                np.testing.assert_array_equal(B.positions(k), pos)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("n", [40, 700, 2048])
def test_double_totals_with_negative_masses(gpu, n, sign):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-20, 20, (n, 2))
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    g.mass = sign * rng.uniform(1, 9, n) * np.where(rng.random(n) < 0.1, -1.0, 1.0)
    with Layout(g, pos, repulsion=REPULSION_EXACT, **SETTINGS) as L:
        L.option("keep_traction", 1)
        L.iterate(1)
        L.sync()
        sw, tr = L.swing(True)
        speed = L.speed()
    assert speed["total_swinging"] == np.cumsum(sw)[-1]
    assert speed["total_traction"] == np.cumsum(tr)[-1]
