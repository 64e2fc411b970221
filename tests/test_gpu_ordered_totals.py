"""FP64 iterations: the attraction by whole warps (attract_warp) leaves the
forces of the force query bit for bit, hubs and single edges, and the totals
made in parallel (ordered_sum) are the serial sums bit for bit, with values
half-way between two sums' spacings, zeros and wide ranges."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout, REPULSION_BH, REPULSION_EXACT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(), dict(adjust=True), dict(linlog=True, strong=True)])
@pytest.mark.parametrize("repulsion", [REPULSION_BH, REPULSION_EXACT])
@pytest.mark.parametrize("n", [2, 31, 33, 64, 65, 700, 2500])
def test_warp_attraction_equals_force_query(gpu, n, repulsion, opts):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-20, 20, (n, 2))
    pos[n // 2] = pos[0]  # (a pair at distance zero)
    hub = rng.integers(0, min(n, 5), 3 * n)
    a = np.concatenate([hub, rng.integers(0, n, n)])
    b = np.concatenate([rng.integers(0, n, 3 * n), rng.integers(0, n, n)])
    a, b = np.append(a, 0), np.append(b, n // 2)
    g = Graph(n, a, b, rng.uniform(0.1, 2.0, len(a)))
    size = rng.uniform(0.1, 1.0, n) if opts.get("adjust") else None
    with Layout(g, pos, precision="double", size=size, repulsion=repulsion, **opts) as L:
        f = L.forces(pos)
        L.option("keep_traction", 1)
        L.iterate(1)
        L.sync()
        sw, tr = L.swing(True)
    # the previous forces are zero: swinging = mass |f|
    want = g.mass * np.sqrt(f[:, 0] * f[:, 0] + f[:, 1] * f[:, 1])
    np.testing.assert_array_equal(sw, want)
    np.testing.assert_array_equal(tr, 0.5 * want)


@pytest.mark.parametrize("kind", ["uniform", "halves", "zeros", "wide"])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 500, 2047, 2048])
def test_totals_equal_serial_sums(gpu, n, kind):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-20, 20, (n, 2))
    none = np.zeros(0, np.int32)
    g = Graph(n, none, none, np.zeros(0))
    # no repulsion, strong gravity: swinging = mass |mass * position|
    mass = rng.uniform(1, 9, n)
    if kind == "halves":  # a large value, then many of half its spacing, odd and even
        pos = np.zeros((n, 2))
        pos[:, 0] = 2.0 ** -53 * rng.integers(1, 4, n)
        pos[0, 0] = 1.0
        mass = np.ones(n)
    elif kind == "zeros":
        pos[rng.random(n) < 0.9] = 0.0
    elif kind == "wide":
        pos *= 2.0 ** rng.integers(-40, 40, (n, 1))
    g.mass = mass
    fixed = np.zeros(n, np.int32)
    fixed[n // 3] = n > 32
    with Layout(g, pos, precision="double", scaling=0.0, strong=True, fixed=fixed,
                repulsion=REPULSION_EXACT) as L:
        L.option("keep_traction", 1)
        L.iterate(1)
        L.sync()
        sw, tr = L.swing(True)
        speed = L.speed()
    free = fixed == 0
    assert kind == "zeros" or (sw[free] > 0).all()
    assert speed["total_swinging"] == np.cumsum(np.where(free, sw, 0.0))[-1]
    assert speed["total_traction"] == np.cumsum(np.where(free, tr, 0.0))[-1]
