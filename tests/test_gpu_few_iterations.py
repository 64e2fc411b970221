"""A call of few iterations launches them kernel by kernel, a longer one through
captured graphs: both take the layout where a session (graphs) takes it, bit for
bit."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Layout, layout_forceatlas2_large, prepare_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("iterations", [1, 63, 64])
@pytest.mark.parametrize("n", [300, 5003, 120000])
def test_few_iterations_equal_session(gpu, n, iterations, precision):
    if precision == "double" and n > 10000:
        n = 20011
    rng = np.random.default_rng(n)
    a = rng.integers(0, n, 2 * n)
    b = (a + 1 + rng.integers(0, n - 1, 2 * n)) % n
    pos = rng.uniform(-100, 100, (n, 2)).astype(np.float32).astype(np.float64)
    edges = np.stack([a, b], 1)
    got = layout_forceatlas2_large(n, edges, iterations=iterations, init=pos, scaling_ratio=2.0,
                                   jitter_tolerance=0.01, precision=precision)
    g = prepare_graph(n, edges)
    with Layout(g, pos, scaling=2.0, jitter_tolerance=0.01, precision=precision) as L:
        L.iterate(iterations)
        L.sync()
        np.testing.assert_array_equal(got, L.positions())
