"""The FP32 all-pairs repulsion of a batch's graphs: two nodes a thread, the
sources of small graphs split over the threads.

Bar: 1e-5 norm-wise of the FP64 batch's forces (each of up to 1,500 terms off by
about 2^-22, added in float; 2e-3 with radii, whose distances cancel, as in the
other tests of that option)."""
import numpy as np
import pytest

from conftest import rel_err
from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import Graph

pytestmark = pytest.mark.gpu

# around a warp, the numbers of parts, and one and two nodes a thread
SIZES = [1, 2, 3, 31, 32, 33, 63, 64, 65, 127, 170, 171, 255, 256, 257, 511, 512, 513, 1023, 1024,
         1025, 1500]


def case(n):
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    keep = a != b
    r = 10.0 * np.sqrt(n)
    pos = rng.uniform(-r, r, (n, 2)).astype(np.float32)
    pos[n // 2] = pos[0]  # coincident
    return Graph(n, a[keep], b[keep], np.ones(keep.sum())), pos.astype(np.float64)


@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("adjust", [False, True])
def test_batch_exact_sizes(gpu, threads, adjust):
    many = [case(n) for n in SIZES]
    out = {}
    for precision in ("single", "double"):
        per = [dict(size=np.full(g.n, 0.25)) for g, _ in many] if adjust else None
        with Batch([g for g, _ in many], [p for _, p in many], precision=precision,
                   exact_below=1 << 20, threads=threads, nodes_per_thread=2, adjust=adjust,
                   per_graph=per) as B:
            B.iterate(1)
            B.sync()
            out[precision] = [B.forces(k) for k in range(len(many))]
    for n, got, want in zip(SIZES, out["single"], out["double"]):
        if n == 1:
            np.testing.assert_allclose(got, want, rtol=1e-6)
        else:
            assert rel_err(got, want) <= (2e-3 if adjust else 1e-5), n
