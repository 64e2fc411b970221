"""The layout work that is timed when a kernel changes, through the package's
public entry points.

A case is one call (or one frame of an open session) as a program makes it:

* ``frames``  a device-resident ``Layout``: some iterations, then the positions,
              as a program does that shows the layout while it settles;
* ``call``    a whole ``layout_forceatlas2_gpu`` / ``layout_forceatlas2_large``
              call, from the host's edge list to the host's coordinates;
* ``batch``   a ``Batch`` of many graphs: some iterations of all, then every
              graph's positions.

Positions of single-precision layouts are returned as float32: the values on
the device are floats, and the entry points widen them.

The layouts are refinements with small steps (a small jitter tolerance, start
positions spread as the package spreads them): the work of an iteration does
not depend on the step, and the results of two builds can be compared value by
value. At the default tolerance an iteration moves nodes past many neighbours,
the last bit of a force is multiplied by about ten an iteration, and after five
iterations two correct layouts have nothing but their statistics in common.
"""
import math

import numpy as np
import torch

from forceatlas2_rc_gb300 import graphs
from forceatlas2_rc_gb300.batch import Batch
from forceatlas2_rc_gb300.layout import (REPULSION_BH, REPULSION_EXACT, Graph, Layout,
                                         layout_forceatlas2_gpu, layout_forceatlas2_large,
                                         prepare_graph_device)


def _case(name, kind, graph, n, iterations, *, precision="single", exact=False, linlog=False,
          hubs=False, strong=False, overlap=False, weights=False, fixed=False, entry="large",
          count=1):
    c = dict(kind=kind, graph=graph, n=n, iterations=iterations, precision=precision,
             exact=exact, linlog=linlog, hubs=hubs, strong=strong, overlap=overlap,
             weights=weights, fixed=fixed, entry=entry, count=count)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the package's example graph (5 islands of 30 nodes, exact
        # repulsion): an interactive layout of a small graph, all latency
        _case("frames_islands150", "frames", "islands", 150, 10, exact=True),
        # one call on a graph of ordinary size in double precision, the
        # default (exact) repulsion below 10,000 nodes
        _case("call_pa1500_double", "call", "pa", 1500, 20, precision="double", exact=True,
              entry="gpu"),
        # a graph near the top of the range that uses the exact repulsion by
        # default, sizes that fill no tile
        _case("frames_er6007_exact", "frames", "er", 6007, 10, exact=True),
        # every pair of a large graph (barnes_hut = FALSE)
        _case("frames_ba100k_exact", "frames", "ba", 100003, 4, exact=True),
        # a whole call on a small graph of the all-GPU layout, from its edges
        _case("call_ba3001", "call", "ba", 3001, 20, weights=True),
        # ten thousand nodes, the commonest size of a served layout
        _case("frames_sbm10007", "frames", "sbm", 10007, 10, linlog=True, hubs=True),
        # scale-free graph with lognormal weights, 100,000 nodes
        _case("frames_ba100k", "frames", "ba", 100000, 10, weights=True),
        # radii kept apart and a few pinned nodes (a continuation)
        _case("frames_ba30011_overlap", "frames", "ba", 30011, 10, overlap=True, fixed=True),
        # double precision over the tree, strong gravity
        _case("frames_sbm50021_double", "frames", "sbm", 50021, 4, precision="double",
              strong=True),
        # a whole call on a large community graph, from its edges
        _case("call_sbm300k", "call", "sbm", 300007, 10),
        # the largest ordinary layout: a million nodes, linlog, hubs dissuaded
        _case("frames_sbm1m", "frames", "sbm", 1000000, 10, linlog=True, hubs=True),
        # a collection of small and medium graphs laid out together
        _case("batch_1024", "batch", "mixed", 20000, 10, count=1024),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["exact", "exact_double", "tree", "tree", "tree", "tree_double",
                       "call_small", "call_tree", "call_tree", "batch"])
    graph = rng.choice(["ba", "sbm", "er"])
    opt = dict(linlog=rng.random() < 0.4, hubs=rng.random() < 0.3, strong=rng.random() < 0.2,
               weights=rng.random() < 0.4)
    if what == "exact":
        return _case("", "frames", graph, size(100, 60000), rng.randint(4, 10), exact=True,
                     overlap=rng.random() < 0.2, **opt)
    if what == "exact_double":
        return _case("", "frames", graph, size(100, 5000), rng.randint(4, 10),
                     precision="double", exact=True, **opt)
    if what == "tree":
        return _case("", "frames", graph, size(2000, 900000), rng.randint(4, 10),
                     overlap=rng.random() < 0.2, fixed=rng.random() < 0.2, **opt)
    if what == "tree_double":
        return _case("", "frames", graph, size(2000, 100000), rng.randint(2, 4),
                     precision="double", fixed=rng.random() < 0.2, **opt)
    if what == "call_small":
        return _case("", "call", graph, size(100, 9000), rng.randint(5, 20), exact=True,
                     precision=rng.choice(["single", "double"]), entry="gpu", **opt)
    if what == "call_tree":
        return _case("", "call", graph, size(2000, 300000), rng.randint(5, 10), **opt)
    return _case("", "batch", "mixed", size(2000, 20000), rng.randint(3, 10),
                 count=size(64, 1000), linlog=opt["linlog"], strong=opt["strong"])


# ---- inputs ------------------------------------------------------------------

def _edges(case, seed):
    n, kind = case["n"], case["graph"]
    if kind == "islands":
        return graphs.islands(5, n // 5, 0.3, 2, seed=seed)
    if kind == "pa":
        return graphs.barabasi_albert_fast(n, 2, seed=seed)
    if kind == "ba":
        return graphs.barabasi_albert_fast(n, 3, seed=seed)
    if kind == "sbm":
        return graphs.sbm(n, max(8, n // 1000), seed=seed)
    return graphs.erdos_renyi(n, 8.0, seed=seed)


def _inputs(case, seed):
    """Edges, weights, start positions (values that floats hold), radii and
    pinned nodes."""
    n, frm, to = _edges(case, seed)
    rng = np.random.default_rng(seed + 1)
    r = 10.0 * math.sqrt(n)  # as the package draws start positions
    pos = rng.uniform(-r, r, (n, 2)).astype(np.float32).astype(np.float64)
    w = rng.lognormal(0.0, 0.5, len(frm)) if case["weights"] else np.ones(len(frm))
    radii = rng.uniform(1.0, 5.0, n).astype(np.float32).astype(np.float64) \
        if case["overlap"] else np.ones(n)
    fixed = np.zeros(n, bool)
    if case["fixed"]:
        fixed[rng.integers(0, n, max(1, n // 100))] = True
    return n, frm, to, w, pos, radii, fixed


def _many(case, seed):
    """Erdos-Renyi and island graphs alternately, sizes log-uniform in
    [50, n], mean degree 4-16, start positions in +-10 sqrt(n)."""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["count"]).uniform(math.log(50), math.log(case["n"]),
                                                         case["count"])
    out = []
    for k in range(case["count"]):
        n = int(round(math.exp(sizes[k])))
        deg = float(rng.uniform(4, 16))
        make = graphs.erdos_renyi if k % 2 == 0 else graphs.island_graph
        _, a, b = make(n, deg, seed=int(rng.integers(1 << 30)))
        r = 10.0 * math.sqrt(n)
        out.append((n, a, b, rng.uniform(-r, r, (n, 2)).astype(np.float32).astype(np.float64)))
    return out


# graphs of the batch below this many nodes use the exact repulsion (fixed
# here: the autotuner's choice differs from run to run)
BATCH_EXACT_BELOW = 1200
THETA, SCALING, GRAVITY, JITTER = 1.2, 2.0, 1.0, 1e-7


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "batch":
        many = _many(case, seed)
        s.batch = Batch([Graph(n, a, b, np.ones(len(a))) for n, a, b, _ in many],
                        [p for _, _, _, p in many], precision=case["precision"],
                        linlog=case["linlog"], strong=case["strong"],
                        jitter_tolerance=JITTER, exact_below=BATCH_EXACT_BELOW, threads=512,
                        nodes_per_thread=2)
        s.small = [g for g, (n, _, _, _) in enumerate(many) if n < BATCH_EXACT_BELOW]
        s.large = [g for g, (n, _, _, _) in enumerate(many) if n >= BATCH_EXACT_BELOW]
        return s
    n, frm, to, w, pos, radii, fixed = _inputs(case, seed)
    if case["kind"] == "frames":
        g = prepare_graph_device(n, frm, to, w, dissuade_hubs=case["hubs"])
        s.layout = Layout(g, pos, size=radii, fixed=fixed.astype(np.int32),
                          jitter_tolerance=JITTER, strong=case["strong"],
                          linlog=case["linlog"], adjust=case["overlap"],
                          precision=case["precision"],
                          repulsion=REPULSION_EXACT if case["exact"] else REPULSION_BH)
        return s
    s.args = dict(n=n, edges=np.stack([frm, to], axis=1), iterations=case["iterations"],
                  scaling_ratio=2.0, jitter_tolerance=JITTER,
                  weights=w if case["weights"] else None, init=pos,
                  strong_gravity=case["strong"], linlog=case["linlog"],
                  dissuade_hubs=case["hubs"], precision=case["precision"])
    if case["entry"] == "gpu":
        s.args["barnes_hut"] = not case["exact"]
    return s


def run(state):
    case = state.case
    real = np.float32 if case["precision"] == "single" else np.float64
    if case["kind"] == "batch":
        state.batch.iterate(case["iterations"])
        state.batch.sync()
        return {name: np.concatenate([state.batch.positions(g) for g in which]).astype(real)
                for name, which in (("small", state.small), ("large", state.large)) if which}
    if case["kind"] == "frames":
        state.layout.iterate(case["iterations"])
        state.layout.sync()
        return state.layout.positions().astype(real)
    call = layout_forceatlas2_gpu if case["entry"] == "gpu" else layout_forceatlas2_large
    return call(**state.args).astype(real)


def _sizes(case):
    """Nodes and edges of a case, about."""
    if case["kind"] == "batch":
        mean = (case["n"] - 50) / math.log(case["n"] / 50)
        return case["count"] * mean, case["count"] * mean * 5.0
    degree = {"islands": 9.0, "pa": 4.0, "ba": 6.0, "sbm": 14.0, "er": 8.0}[case["graph"]]
    return case["n"], case["n"] * degree / 2


def work(case):
    """A pass's iterations: every node's position, mass, previous force and
    speed term read and its position and force written, every incidence read;
    the interactions of the force law (every pair, or about 200 regions and
    nodes a node over the tree) at 20 operations each. A session's graph is
    on the device; a call's is read once from the host's arrays."""
    n, m = _sizes(case)
    r = 8 if case["precision"] == "double" else 4
    per_it = n * (2 + 1 + 2 + 2 + 2) * r + 2 * m * (4 + r) + 4 * n
    if case["kind"] == "batch":
        small = math.log(BATCH_EXACT_BELOW / 50) / math.log(case["n"] / 50)
        small = min(1.0, small)
        pairs = case["count"] * small * 2.2e5 + (n - 240 * case["count"] * small) * 200
    else:
        pairs = float(n) * n if case["exact"] else n * 200.0
    k = case["iterations"]
    host = 16 * n if case["kind"] != "call" else 32 * n + 24 * m
    return {"bytes": k * per_it + host, "flops": k * (20.0 * pairs + 16.0 * m + 30.0 * n)}


# ---- the same iterations in 64 bits ------------------------------------------
# Plain torch in double: the all-pairs sum, or the Barnes-Hut sum over the
# radix tree of the Morton codes (16 bits an axis; codes equal to a neighbour's
# are told apart by their place), a region being taken whole when d^2 theta^2
# exceeds 2 (w^2 + h^2), else opened, or summed node by node from 8 nodes down.
# Several graphs are laid out together as segments of the same arrays.


def _segment_reduce(v, seg, nseg, how):
    out = torch.full((nseg,), math.inf if how == "amin" else -math.inf, dtype=v.dtype,
                     device=v.device)
    return out.scatter_reduce_(0, seg, v, how, include_self=True)


def _spread(v):
    for shift, mask in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << shift)) & mask
    return v


def _leading(v):
    """Leading zero bits of 32-bit values (positive int64)."""
    return 32 - torch.frexp(v.double())[1].long()


def _first_below(d, right):
    """For every place p of d: the nearest place right (left) of p whose value
    is below d[p] (len(d), or -1, where there is none)."""
    v = d if right else d.flip(0)
    n = len(v)
    tables, s = [v], 1
    while 2 * s <= n:
        t = tables[-1]
        tables.append(torch.minimum(t[:-s], t[s:]) if len(t) > s else t)
        s *= 2
    at = torch.arange(n, device=v.device) + 1
    for k in range(len(tables) - 1, -1, -1):
        t = tables[k]
        ok = at < len(t)
        hop = torch.zeros_like(ok)
        hop[ok] = t[at[ok]] >= v[ok]
        at = torch.where(hop, at + (1 << k), at)
    return at if right else (n - 1 - at).flip(0)


def _range_extreme(v, lo, hi, least):
    """min (max) of v[lo..hi] for many ranges."""
    out = torch.empty(len(lo), dtype=v.dtype, device=v.device)
    level = torch.frexp((hi - lo + 1).double())[1].long() - 1
    t, s, k = v, 1, 0
    op = torch.minimum if least else torch.maximum
    while True:
        sel = (level == k).nonzero().squeeze(1)
        if len(sel):
            out[sel] = op(t[lo[sel]], t[hi[sel] - s + 1])
        if len(t) <= s:
            return out
        t = op(t[:-s], t[s:])
        s *= 2
        k += 1


def _tree_repulsion(x, y, m, radius, seg, start, adjust):
    dev, total, nseg = x.device, len(x), len(start)
    lox, hix = _segment_reduce(x, seg, nseg, "amin"), _segment_reduce(x, seg, nseg, "amax")
    loy, hiy = _segment_reduce(y, seg, nseg, "amin"), _segment_reduce(y, seg, nseg, "amax")
    extent = torch.maximum(hix - lox, hiy - loy)
    scale = torch.where(extent > 0, 65535.0 / extent, torch.zeros_like(extent))
    cell = lambda v, lo: ((v - lo[seg]) * scale[seg]).clamp(0, 65535).long()  # noqa: E731
    key = (seg << 32) | _spread(cell(x, lox)) | (_spread(cell(y, loy)) << 1)
    key, order = torch.sort(key, stable=True)
    xs, ys, ms, rs, ss = x[order], y[order], m[order], radius[order], seg[order]
    place = torch.arange(total, device=dev)
    local = place - start[ss]
    same = ss[1:] == ss[:-1]
    diff = (key[1:] ^ key[:-1]) & 0xFFFFFFFF
    d = torch.where(diff > 0, _leading(diff.clamp(min=1)),
                    32 + _leading((local[1:] ^ local[:-1]).clamp(min=1)))
    d = torch.where(same, d, torch.full_like(d, -1))
    none = torch.full((1,), -1, dtype=d.dtype, device=dev)
    edge = torch.cat([none, d, none])  # edge[i], edge[i + 1]: before and after node i
    # region p splits after node p: its nodes are lo[p] .. hi[p]
    lo, hi = _first_below(d, False) + 1, _first_below(d, True)
    real = d >= 0
    before, after = edge[lo], edge[hi + 1]
    parent = torch.where(after > before, hi, lo - 1)
    left = place[:-1] + total  # a single node i is total + i
    right = place[1:] + total
    sel = real & (after > before)
    left = left.scatter(0, parent[sel], place[:-1][sel])
    sel = real & (after <= before) & (before >= 0)
    right = right.scatter(0, parent[sel], place[:-1][sel])
    root = torch.full((nseg,), -1, dtype=torch.long, device=dev)
    sel = real & (after < 0) & (before < 0)
    root[ss[:-1][sel]] = place[:-1][sel]
    mid = (lox + hix) / 2, (loy + hiy) / 2
    zero = torch.zeros(1, dtype=x.dtype, device=dev)
    sums = [torch.cat([zero, v.cumsum(0)]) for v in
            (ms, ms * (xs - mid[0][ss]), ms * (ys - mid[1][ss]))]
    hi1 = hi + 1
    mass = sums[0][hi1] - sums[0][lo]
    cx = (sums[1][hi1] - sums[1][lo]) / mass + mid[0][ss[:-1]]
    cy = (sums[2][hi1] - sums[2][lo]) / mass + mid[1][ss[:-1]]
    w = _range_extreme(xs, lo, hi, False) - _range_extreme(xs, lo, hi, True)
    h = _range_extreme(ys, lo, hi, False) - _range_extreme(ys, lo, hi, True)
    size2 = 2.0 * (w * w + h * h)
    fx, fy = torch.zeros_like(x), torch.zeros_like(x)

    def pairs(i, j):
        dx, dy = xs[i] - xs[j], ys[i] - ys[j]
        d2 = dx * dx + dy * dy
        mm = SCALING * ms[i] * ms[j]
        if adjust:
            dist = d2.sqrt() - rs[i] - rs[j]
            g = torch.where(dist > 0, mm / (dist * dist),
                            torch.where(dist < 0, 100.0 * mm, torch.zeros_like(mm)))
        else:
            g = torch.where(d2 > 0, mm / d2, torch.zeros_like(mm))
        g = torch.where(i == j, torch.zeros_like(g), g)
        fx.index_add_(0, i, dx * g)
        fy.index_add_(0, i, dy * g)

    for b in range(0, total, 1 << 18):
        i = place[b:b + (1 << 18)]
        r = root[ss[i]]
        i, r = i[r >= 0], r[r >= 0]
        while len(i):
            one = r >= total
            if bool(one.any()):
                pairs(i[one], r[one] - total)
                i, r = i[~one], r[~one]
            dx, dy = xs[i] - cx[r], ys[i] - cy[r]
            d2 = dx * dx + dy * dy
            far = d2 * (THETA * THETA) > size2[r]
            k, g = i[far], SCALING * ms[i[far]] * mass[r[far]] / d2[far]
            fx.index_add_(0, k, dx[far] * g)
            fy.index_add_(0, k, dy[far] * g)
            i, r = i[~far], r[~far]
            few = hi[r] - lo[r] < 8
            k, q = i[few], r[few]
            for step in range(8):
                j = lo[q] + step
                ok = j <= hi[q]
                pairs(k[ok], j[ok])
            i, r = i[~few], r[~few]
            i, r = torch.cat([i, i]), torch.cat([left[r], right[r]])
    ox, oy = torch.empty_like(fx), torch.empty_like(fy)
    ox[order], oy[order] = fx, fy
    return ox, oy


def _pair_repulsion(x, y, m, radius, start, length, adjust):
    fx, fy = torch.zeros_like(x), torch.zeros_like(x)
    for b, n in zip(start.tolist(), length.tolist()):
        xs, ys, ms, rs = (v[b:b + n] for v in (x, y, m, radius))
        rows = max(1, min(n, (1 << 27) // n))
        for i in range(0, n, rows):
            k = slice(i, i + rows)
            dx, dy = xs[k, None] - xs, ys[k, None] - ys
            d2 = dx * dx + dy * dy
            if adjust:
                dist = d2.sqrt() - rs[k, None] - rs
                g = torch.where(dist > 0, 1.0 / (dist * dist),
                                torch.where(dist < 0, 100.0, 0.0))
            else:
                g = torch.where(d2 > 0, 1.0 / d2, 0.0)
            g *= ms
            fx[b + i:b + min(n, i + rows)] = (dx * g).sum(1) * SCALING * ms[k]
            fy[b + i:b + min(n, i + rows)] = (dy * g).sum(1) * SCALING * ms[k]
    return fx, fy


def _settle(sizes, frm, to, w, pos, radii, fixed, iterations, *, exact, strong, linlog, hubs,
            adjust):
    """The positions after `iterations` iterations of the graphs of `sizes`
    nodes whose arrays are concatenated."""
    dev = torch.device("cuda")
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v)).to(dev)  # noqa: E731
    length = t(np.asarray(sizes, dtype=np.int64))
    nseg = len(length)
    start = length.cumsum(0) - length
    seg = torch.repeat_interleave(torch.arange(nseg, device=dev), length)
    x, y = t(pos[:, 0]).double(), t(pos[:, 1]).double()
    a, b, w = t(frm).long(), t(to).long(), t(w).double()
    radius, move = t(radii).double(), ~t(fixed).bool()
    n = len(x)
    one = torch.ones(len(a), dtype=torch.float64, device=dev)
    m = torch.ones(n, dtype=torch.float64, device=dev).index_add_(0, a, one).index_add_(0, b, one)
    c = w
    if hubs:
        mean = torch.zeros(nseg, dtype=torch.float64, device=dev).index_add_(0, seg, m) / length
        c = mean[seg[a]] * w / m[a]
    keep = a != b
    a, b, c = a[keep], b[keep], c[keep]
    ox, oy = torch.zeros_like(x), torch.zeros_like(x)
    speed = torch.ones(nseg, dtype=torch.float64, device=dev)
    eff = torch.ones_like(speed)
    cnt = length.double()
    for _ in range(iterations):
        if exact:
            fx, fy = _pair_repulsion(x, y, m, radius, start, length, adjust)
        else:
            fx, fy = _tree_repulsion(x, y, m, radius, seg, start, adjust)
        dist = (x * x + y * y).sqrt()
        g = GRAVITY * m if strong else torch.where(dist > 0, GRAVITY * m / dist, 0.0)
        fx -= x * g
        fy -= y * g
        dx, dy = x[a] - x[b], y[a] - y[b]
        g = -c
        if linlog or adjust:
            dist = (dx * dx + dy * dy).sqrt()
            if adjust:
                dist = dist - radius[a] - radius[b]
            if linlog:
                g = g * torch.where(dist > 0, torch.log1p(dist) / dist, 0.0)
            g = torch.where(dist > 0, g, 0.0)
        for f, v in ((fx, dx * g), (fy, dy * g)):
            f.index_add_(0, a, v)
            f.index_add_(0, b, -v)
        swing = m * ((ox - fx) ** 2 + (oy - fy) ** 2).sqrt()
        trac = 0.5 * m * ((ox + fx) ** 2 + (oy + fy) ** 2).sqrt()
        # both totals by the same additions: in the first iteration one is
        # exactly twice the other, which the controller compares
        run_sum = torch.cat([torch.zeros(2, 1, dtype=x.dtype, device=dev),
                             (torch.stack([swing, trac]) * move).cumsum(1)], dim=1)
        ts, tt = run_sum[:, start + length] - run_sum[:, start]
        est = 0.05 * cnt.sqrt()
        jt = JITTER * torch.maximum(est.sqrt(), (est * tt / cnt ** 2).clamp(max=10.0))
        wild = ts > 2.0 * tt
        e = torch.where(wild & (eff > 0.05), 0.5 * eff, eff)
        jt = torch.where(wild, jt.clamp(min=JITTER), jt)
        target = jt * e * tt / ts
        over = ts > jt * tt
        e2 = torch.where(over & (e > 0.05), 0.7 * e, e)
        e2 = torch.where(~over & (speed < 1000), 1.3 * e, e2)
        new = speed + torch.minimum(target - speed, 0.5 * speed)
        speed, eff = torch.where(ts > 0, new, speed), torch.where(ts > 0, e2, eff)
        sp = speed[seg]
        if adjust:
            size = (fx * fx + fy * fy).sqrt()
            k = 0.1 * sp / (1.0 + (sp * swing).sqrt())
            k = torch.where(size > 0, (k * size).clamp(max=10.0) / size, 0.0)
        else:
            k = sp / (1.0 + (sp * swing).sqrt())
        x, y = torch.where(move, x + fx * k, x), torch.where(move, y + fy * k, y)
        ox, oy = fx, fy
    return torch.stack([x, y], dim=1).cpu().numpy()


def exact(case, seed):
    opt = dict(strong=case["strong"], linlog=case["linlog"], hubs=case["hubs"])
    if case["kind"] == "batch":
        many = _many(case, seed)
        out = {}
        for name, which, flag in (("small", [g for g in many if g[0] < BATCH_EXACT_BELOW], True),
                                  ("large", [g for g in many if g[0] >= BATCH_EXACT_BELOW], False)):
            if not which:
                continue
            sizes = [g[0] for g in which]
            off = np.cumsum([0] + sizes[:-1])
            frm = np.concatenate([g[1].astype(np.int64) + o for g, o in zip(which, off)])
            to = np.concatenate([g[2].astype(np.int64) + o for g, o in zip(which, off)])
            pos = np.concatenate([g[3] for g in which])
            out[name] = _settle(sizes, frm, to, np.ones(len(frm)), pos, np.ones(len(pos)),
                                np.zeros(len(pos), bool), case["iterations"], exact=flag,
                                adjust=False, **opt)
        return out
    n, frm, to, w, pos, radii, fixed = _inputs(case, seed)
    return _settle([n], frm, to, w, pos, radii, fixed, case["iterations"],
                   exact=case["exact"], adjust=case["overlap"], **opt)
