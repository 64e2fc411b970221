"""The FP64 walk (k_traverse_terms) against the per-thread walk over the same
tree (option "walk" 2): forces equal bit for bit, with pools that stay short,
fill exactly and overflow, opening tests on the boundary, coordinates far from
the origin, and no opening angle."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout

pytestmark = pytest.mark.gpu


def _positions(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(-50, 50, (n, 2))
    if kind == "far":  # the float coordinates hold a few bits of a region's size
        return rng.uniform(-1, 1, (n, 2)) + np.array([3e6, -2e4])
    if kind == "coincident":
        return rng.uniform(-50, 50, (5, 2))[rng.integers(0, 5, n)]
    if kind == "grid":  # many tests on the boundary itself
        return np.stack([np.arange(n) % 64, np.arange(n) // 64], 1) * 1.0
    return rng.uniform(-1, 1, (n, 2)) * 10.0 ** rng.integers(-18, 18, (n, 1))  # "scales"


@pytest.mark.parametrize("adjust", [False, True])
@pytest.mark.parametrize("kind", ["uniform", "far", "coincident", "grid", "scales"])
@pytest.mark.parametrize("n", [2, 9, 31, 32, 33, 64, 65, 500, 5003, 11999, 12001])
def test_terms_walk_equals_thread_walk(gpu, n, kind, adjust):
    rng = np.random.default_rng(n)
    pos = _positions(kind, n, rng)
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    g.mass = rng.integers(1, 9, n).astype(np.float64)
    size = rng.uniform(0.1, 2.0, n) if adjust else None
    for theta in (0.0, 0.5, 1.0, 1.2):
        with Layout(g, pos, precision="double", theta=theta, size=size, adjust=adjust) as L:
            got = L.forces(pos)
            L.option("walk", 2)
            want = L.forces(pos)
        np.testing.assert_array_equal(got, want, err_msg=f"theta {theta}")
