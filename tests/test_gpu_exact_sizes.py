"""The all-pairs repulsion at the edges of its blocks, tiles and rows of
sources. In double every node's terms are added in ascending order of the
source, as the reference adds them: equal bits. In single the path's own bars,
1e-4 norm-wise and 2e-3 with prevent_overlap, of the double forces."""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.layout import REPULSION_EXACT, Graph, Layout

pytestmark = pytest.mark.gpu


def _layout(n, precision, adjust, rng):
    pos = rng.uniform(-300, 300, (n, 2)).astype(np.float32).astype(np.float64)
    pos[n // 2] = pos[0]  # coincident nodes
    size = rng.uniform(0.5, 4.0, n).astype(np.float32).astype(np.float64)
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    g.mass = rng.integers(1, 50, n).astype(np.float64)
    return g, pos, size, Layout(g, pos, size=size, adjust=adjust, gravity=0.0, scaling=2.5,
                                precision=precision, repulsion=REPULSION_EXACT)


@pytest.mark.parametrize("adjust", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 152, 153, 1024, 2432, 2433, 4900])
def test_exact_double_bits(gpu, orc, n, adjust):
    g, pos, size, layout = _layout(n, "double", adjust, np.random.default_rng(n))
    with layout as L:
        got = L.forces(pos)
    want = orc.repulse_exact(n, pos, g.mass, size, adjust, 2.5)
    np.testing.assert_array_equal(got, np.asarray(want).reshape(got.shape))


@pytest.mark.parametrize("adjust", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 31, 33, 255, 257, 512, 513, 1025, 4095, 4096,
                               4097, 6145, 11999, 12000])
def test_exact_single(gpu, n, adjust):
    _, pos, _, double = _layout(n, "double", adjust, np.random.default_rng(n))
    with double as L:
        want = L.forces(pos)
    _, _, _, single = _layout(n, "single", adjust, np.random.default_rng(n))
    with single as L:
        assert rel_err(L.forces(pos), want) <= (2e-3 if adjust else 1e-4)
        L.iterate(2)  # the rows added up in the totals' launch
        L.sync()
        moved = L.positions()
        L.set_positions(pos)
        assert rel_err(L.forces(pos), want) <= (2e-3 if adjust else 1e-4)
    assert np.isfinite(moved).all()


@pytest.mark.parametrize("n", [6999, 7000, 9999, 10000, 15999, 16000])
def test_exact_single_split(gpu, n):
    """Where the nodes a thread and the rows of sources change (without radii:
    among this many nodes some pair is nearer to contact than its float terms
    are good for)."""
    _, pos, _, double = _layout(n, "double", False, np.random.default_rng(n))
    with double as L:
        want = L.forces(pos)
    _, _, _, single = _layout(n, "single", False, np.random.default_rng(n))
    with single as L:
        assert rel_err(L.forces(pos), want) <= 1e-4
