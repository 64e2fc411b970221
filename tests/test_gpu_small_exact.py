"""Whole iterations of a small FP32 all-pairs layout in one cluster launch
(k_small_exact) against the separate launches: the first iteration's forces are
sums of at most n float terms in another order, so the positions agree to
n 2^-24 of the layout's extent (jitter tolerance 1e-3: no step amplifies that
by more than the few iterations made), the totals to the same."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import Graph, Layout, REPULSION_EXACT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjust,linlog", [(False, False), (True, True)])
@pytest.mark.parametrize("n", [2, 3, 31, 33, 150, 511, 512, 513, 1025, 2048])
def test_small_exact_equals_separate_launches(gpu, n, adjust, linlog):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-100, 100, (n, 2)).astype(np.float32).astype(np.float64)
    a = rng.integers(0, n, 2 * n).astype(np.int32)
    b = ((a + 1 + rng.integers(0, n - 1, 2 * n)) % n).astype(np.int32)
    g = Graph(n, a, b, np.ones(2 * n))
    fixed = np.zeros(n, np.int32)
    fixed[n // 2] = 1
    size = rng.uniform(0.01, 0.1, n) if adjust else None
    got = {}
    # (a block owns 512 nodes at most)
    for blocks in [0] + [c for c in (1, 2, 3, 8, 16) if -(-n // c) <= 512]:
        with Layout(g, pos, size=size, fixed=fixed, adjust=adjust, linlog=linlog,
                    repulsion=REPULSION_EXACT, jitter_tolerance=1e-3) as L:
            L.option("keep_traction", 1)
            L.option("exact_cluster", blocks)
            out = []
            for k in (1, 3):
                L.iterate(k)
                out.append(L.positions())
                if k == 1:  # (nothing cancels in the first swinging)
                    out.append(np.array(list(L.speed().values())))
            L.set_positions(pos[::-1])
            L.iterate(1)
            out.append(L.positions())
            L.sync()
            if blocks in (1, 16):
                L.set_positions(pos)
                L.iterate(300)  # two launches
                L.sync()
                assert np.isfinite(L.positions()).all()
            with pytest.raises(RuntimeError):
                L.option("exact_cluster", 17)
        got[blocks] = out
    assert len(got) > 2 or n > 512
    bar = 4 * n * 2.0 ** -24
    for blocks, out in got.items():
        assert np.array_equal(out[0][n // 2], pos[n // 2])
        for x, y in zip(out, got[0]):
            scale = np.abs(y).max() if y.ndim == 2 else np.abs(y)
            assert (np.abs(x - y) <= bar * scale).all(), blocks
