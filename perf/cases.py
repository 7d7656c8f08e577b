"""What a user of the layout engine has it do, as cases that can be timed.

A case is one pass through the public entry points of `batchlayoutcode_gb300`
on a seeded synthetic graph (the generator families of the benchmark and the
tests: triangulated grids, random geometric graphs of mean degree 6, Chung-Lu
graphs of exponent 2.5), generated on the GPU from the seed alone.

* minibatch    coordinates in from page-locked host memory, a few iterations
               of algo 2 / 3 / 7 / 8 with the last one's energy, coordinates out
* noalloc      one minibatch iteration on the caller's own device buffers;
               returns the forces too
* barnes_hut   the same round trip as minibatch with algo 4
* greedy       the same with algo 5 (its walk phase and its all-pairs phase)
* batched      a set of small graphs laid out in one launch
* learned_init the learned start of a graph, coordinates out
* train        a few epochs of the initializer's network on a set of graphs

The engine keeps coordinates, minibatch forces and per-graph energies as
float32 values or sums of them and hands them over as doubles; `run` returns
coordinates as the float32 they are.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import batchlayoutcode_gb300 as B
from batchlayoutcode_gb300 import _lib, learned

DEV = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
DECAY = {2: 0.999, 4: 0.999, 7: 0.999, 3: 0.99, 8: 0.99, 5: 0.99}
DEGREE = {"grid": 5.88, "rgg": 6.0, "powerlaw": 10.0}


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # the smallest interactive layout: a mesh of a few thousand vertices, all pairs, in the middle of a run
        dict(name="fr_grid_4k", path="minibatch", algo=2, graph="grid", n=4096, layout="mid", iterations=4, batch=256,
             step=1.0),
        # the all-pairs benchmark graph: one iteration of a social-network-like graph of 100,000 vertices
        dict(name="fr_powerlaw_100k", path="minibatch", algo=2, graph="powerlaw", n=100_000, layout="mid",
             iterations=1, batch=256, step=1.0),
        # a service that owns its device memory and keeps a mid-size layout moving; a batch that divides nothing
        dict(name="linlog_rgg_20k", path="noalloc", algo=3, graph="rgg", n=20_011, layout="mid", iterations=1,
             batch=200, step=0.9),
        # the SD variant with larger batches on a mid-size power-law graph
        dict(name="sd_powerlaw_31k", path="minibatch", algo=7, graph="powerlaw", n=31_337, layout="mid", iterations=2,
             batch=512, step=1.0),
        # the smallest Barnes-Hut layouts: latency and launches
        dict(name="bh_grid_4k", path="barnes_hut", algo=4, graph="grid", n=4096, layout="mid", iterations=4, batch=256,
             theta=1.2, step=1.0),
        # an accurate opening angle on a clustered, skewed layout
        dict(name="bh_powerlaw_100k", path="barnes_hut", algo=4, graph="powerlaw", n=100_003, layout="mid",
             iterations=2, batch=256, theta=0.5, step=1.0),
        # the headline workload: a million vertices, iterations in the middle of a run
        dict(name="bh_rgg_1m", path="barnes_hut", algo=4, graph="rgg", n=1_000_000, layout="mid", iterations=3,
             batch=256, theta=1.2, step=1.0),
        # the largest: an iteration from the random start, odd size, larger batch
        dict(name="bh_rgg_3m", path="barnes_hut", algo=4, graph="rgg", n=3_000_001, layout="disc", iterations=1,
             batch=384, theta=1.2, step=0.7),
        # the greedy approximation in the reference's phase split (9 walk iterations, 1 all-pairs)
        dict(name="greedy_powerlaw_100k", path="greedy", algo=5, graph="powerlaw", n=100_000, layout="mid",
             iterations=10, batch=256, step=1.0),
        # a collection of small graphs in one launch, minibatch below 5,000 vertices and Barnes-Hut from there
        dict(name="batched_192", path="batched", graphs=192, lo=200, hi=20_000, iterations=2, batch=256, theta=1.2),
        # the learned start of a large mesh-like graph
        dict(name="learned_rgg_400k", path="learned_init", graph="rgg", n=400_000),
        # fine-tuning the initializer on a dozen graphs
        dict(name="train_12", path="train", graphs=12, lo=2_000, hi=40_000, epochs=10),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["minibatch"] * 4 + ["noalloc"] * 2 + ["barnes_hut"] * 5 + ["greedy", "batched",
                                                                                  "learned_init", "train"])
    graph = rng.choice(["grid", "rgg", "powerlaw"])
    if path == "minibatch":
        n = _logint(rng, 500, 100_000)
        # (from the dense random start the nearest pairs, 1e-5 apart, make a step of any arithmetic its own)
        return dict(path=path, algo=rng.choice([2, 2, 3, 7, 8]), graph=graph, n=n, layout="mid",
                    iterations=1 if n > 10_000 else rng.choice([1, 2, 4]),
                    batch=rng.choice([64, 128, 256, 256, 384, 1000]), step=round(rng.uniform(0.3, 1.0), 3))
    if path == "noalloc":
        return dict(path=path, algo=rng.choice([2, 3, 8]), graph=graph, n=_logint(rng, 500, 60_000),
                    layout="mid", iterations=1, batch=rng.choice([37, 128, 200, 256]),
                    step=round(rng.uniform(0.3, 1.0), 3))
    if path == "barnes_hut":
        n = _logint(rng, 1_000, 2_500_000)
        layout = rng.choice(["mid", "disc"])  # several iterations from the dense start drift apart by themselves
        return dict(path=path, algo=4, graph=graph, n=n, layout=layout,
                    iterations=1 if n > 300_000 or layout == "disc" else rng.choice([1, 2, 4]),
                    batch=rng.choice([128, 256, 256, 512]),
                    theta=1.2 if n > 300_000 else rng.choice([0.5, 0.8, 1.2]), step=round(rng.uniform(0.3, 1.0), 3))
    if path == "greedy":
        return dict(path=path, algo=5, graph=graph, n=_logint(rng, 1_000, 80_000), layout="mid",
                    iterations=rng.choice([1, 5, 10]), batch=rng.choice([128, 256, 256]),
                    step=round(rng.uniform(0.3, 1.0), 3))
    if path == "batched":
        return dict(path=path, graphs=rng.randint(20, 180), lo=200, hi=_logint(rng, 2_000, 20_000),
                    iterations=rng.choice([1, 2]), batch=rng.choice([128, 256, 256]), theta=rng.choice([0.8, 1.2]))
    if path == "learned_init":
        return dict(path=path, graph=graph, n=_logint(rng, 1_000, 380_000))
    return dict(path=path, graphs=rng.randint(4, 12), lo=1_000, hi=_logint(rng, 4_000, 40_000),
                epochs=rng.choice([4, 8, 10]))


# ---- graphs on the GPU -------------------------------------------------------------

def _rgg_edges(sizes, gen):
    """Random geometric graphs of mean degree 6 (points uniform in the unit
    square), vertices of all graphs numbered through: (points, u, v, the
    vertices in the order of their cells)."""
    dev = DEV
    sz = torch.tensor(sizes, device=dev)
    gid = torch.repeat_interleave(torch.arange(len(sizes), device=dev), sz)
    total = int(sz.sum())
    pts = torch.rand(total, 2, generator=gen, device=dev, dtype=torch.float64)
    r = torch.sqrt(6.0 / (math.pi * sz.double()))
    m = torch.clamp(torch.floor(1.0 / r), min=1).long()
    off = torch.cumsum(m * m, 0) - m * m
    mg, og = m[gid], off[gid]
    cx = torch.minimum((pts[:, 0] * mg).long(), mg - 1)
    cy = torch.minimum((pts[:, 1] * mg).long(), mg - 1)
    order = torch.argsort(og + cy * mg + cx)
    p, g2, cx, cy, mg, og = pts[order], gid[order], cx[order], cy[order], mg[order], og[order]
    count = torch.bincount(og + cy * mg + cx, minlength=int((m * m).sum()))
    start = torch.cumsum(count, 0) - count
    r2 = (r * r)[g2]
    here = torch.arange(total, device=dev)
    us, vs = [], []
    for ox, oy in ((0, 0), (1, 0), (-1, 1), (0, 1), (1, 1)):
        nx, ny = cx + ox, cy + oy
        inside = (nx >= 0) & (nx < mg) & (ny < mg)
        cell = torch.where(inside, og + ny * mg + nx, 0)
        s = start[cell]
        c = torch.where(inside, count[cell], 0)
        for j in range(int(c.max())):
            cand = s + j
            ok = (j < c) & ((cand > here) if (ox, oy) == (0, 0) else True)
            a = here[ok]
            b = cand[ok]
            d = p[a] - p[b]
            near = (d * d).sum(1) <= r2[a]
            us.append(order[a[near]])
            vs.append(order[b[near]])
    return pts, torch.cat(us), torch.cat(vs), order


def _powerlaw_edges(n, degree, gen):
    i0 = max(1.0, n ** (1.0 / 1.5) / 50.0)
    w = (torch.arange(n, device=DEV, dtype=torch.float64) + i0) ** (-1.0 / 1.5)
    cdf = torch.cumsum(w / w.sum(), 0)
    m = int(round(n * degree / 2.0))
    e = torch.searchsorted(cdf, torch.rand(2, m, generator=gen, device=DEV, dtype=torch.float64)).clamp_(max=n - 1)
    return e[0], e[1]


def _grid_edges(rows, cols):
    idx = torch.arange(rows * cols, device=DEV).view(rows, cols)
    u = torch.cat([idx[:, :-1].reshape(-1), idx[:-1].reshape(-1), idx[:-1, :-1].reshape(-1)])
    v = torch.cat([idx[:, 1:].reshape(-1), idx[1:].reshape(-1), idx[1:, 1:].reshape(-1)])
    return u, v


def _links(total, gid, ngraphs, u, v, order):
    """Edges that make every graph connected: the first vertex of each
    component but the graph's largest, joined to the nearest earlier (else
    later) vertex of the largest one in `order`, where graphs follow each
    other and neighbours in a plane are near each other."""
    lab = torch.arange(total, device=DEV)
    uu, vv = torch.cat([u, v]), torch.cat([v, u])
    while True:
        near = lab.scatter_reduce(0, uu, lab[lab][vv], "amin")
        new = lab.scatter_reduce(0, lab, near, "amin")
        new = torch.minimum(torch.minimum(new, near), new[new])
        if torch.equal(new, lab):
            break
        lab = new
    size = torch.bincount(lab, minlength=total)
    best = torch.zeros(ngraphs, dtype=torch.long, device=DEV)
    best = best.scatter_reduce(0, gid, size[lab] * (total + 1) + lab, "amax")
    main = lab == (best % (total + 1))[gid]
    at = torch.arange(total, device=DEV)
    place = torch.empty_like(at)
    place[order] = at
    held = torch.nonzero(main[order])[:, 0]
    stray = torch.nonzero(~main & (lab == at))[:, 0]
    k = torch.searchsorted(held, place[stray])
    before, after = order[held[(k - 1).clamp(min=0)]], order[held[k.clamp(max=held.numel() - 1)]]
    return stray, torch.where((k > 0) & (gid[before] == gid[stray]), before, after)


class Graph:
    """Symmetric CSR on the host (int32, ids ascending per row) and a layout
    with unit spacing to draw mid-run coordinates around."""


def _graphs(kinds, sizes, seed):
    """One connected Graph per (kind, size); a grid has the size of the nearest
    near-square lattice."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    real, shape = [], []
    for k, n in zip(kinds, sizes):
        rows = max(2, int(round(math.sqrt(n))))
        cols = max(2, int(round(n / rows)))
        shape.append((rows, cols))
        real.append(rows * cols if k == "grid" else n)
    offs = np.concatenate([[0], np.cumsum(real)])
    total = int(offs[-1])
    place = torch.zeros(total, 2, dtype=torch.float64, device=DEV)
    order = torch.arange(total, device=DEV)
    us, vs = [], []
    rg = [g for g, k in enumerate(kinds) if k == "rgg"]
    if rg:
        pts, u, v, cells = _rgg_edges([real[g] for g in rg], gen)
        at = torch.cat([torch.arange(offs[g], offs[g + 1], device=DEV) for g in rg])
        scale = torch.cat([torch.full((real[g], 1), math.sqrt(real[g]), dtype=torch.float64, device=DEV) for g in rg])
        place[at] = pts * scale
        order[at] = at[cells]
        us.append(at[u])
        vs.append(at[v])
    for g, k in enumerate(kinds):
        if k == "rgg":
            continue
        if k == "grid":
            u, v = _grid_edges(*shape[g])
            ids = torch.arange(real[g], device=DEV)
            place[offs[g]:offs[g + 1]] = torch.stack([ids % shape[g][1], ids // shape[g][1]], 1).double()
        else:
            u, v = _powerlaw_edges(real[g], DEGREE["powerlaw"], gen)
            z = torch.randn(real[g], 2, generator=gen, dtype=torch.float64, device=DEV)
            place[offs[g]:offs[g + 1]] = z * (0.5 * math.sqrt(real[g]))
        us.append(u + int(offs[g]))
        vs.append(v + int(offs[g]))
    u, v = torch.cat(us), torch.cat(vs)
    gid = torch.repeat_interleave(torch.arange(len(kinds), device=DEV), torch.tensor(real, device=DEV))
    if any(k != "grid" for k in kinds):
        lu, lv = _links(total, gid, len(kinds), u, v, order)
        u, v = torch.cat([u, lu]), torch.cat([v, lv])
    keep = u != v
    n = total
    a, b = torch.minimum(u, v)[keep], torch.maximum(u, v)[keep]
    key = torch.unique(a * n + b)
    a, b = key // n, key % n
    key = torch.sort(torch.cat([a * n + b, b * n + a]))[0]
    rows, cols = key // n, key % n
    rowptr = torch.zeros(n + 1, dtype=torch.long, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    noise = torch.randn(n, 2, generator=gen, dtype=torch.float64, device=DEV)
    ang = torch.rand(n, generator=gen, dtype=torch.float64, device=DEV) * (2 * math.pi)
    rad = 3.0 * torch.sqrt(torch.rand(n, generator=gen, dtype=torch.float64, device=DEV))
    mid = (place + 0.4 * noise).float()
    disc = torch.stack([rad * torch.cos(ang), rad * torch.sin(ang)], 1).float()
    rowptr, cols = rowptr.cpu().numpy(), cols.to(torch.int32).cpu().numpy()
    out = []
    for g in range(len(kinds)):
        v0, v1 = int(offs[g]), int(offs[g + 1])
        e0, e1 = int(rowptr[v0]), int(rowptr[v1])
        G = Graph()
        G.n = v1 - v0
        G.rowptr = np.ascontiguousarray((rowptr[v0:v1 + 1] - e0).astype(np.int32))
        G.colids = np.ascontiguousarray(cols[e0:e1] - np.int32(v0))
        G.mid, G.disc = mid[v0:v1], disc[v0:v1]
        out.append(G)
    return out


def _set_of_graphs(case, seed):
    """Graphs of the three kinds in turn, sizes log-uniform in [lo, hi] (the
    case's own sizes; the seed draws the graphs)."""
    rng = np.random.default_rng(case["graphs"] * 1000003 + case["hi"])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["graphs"])).round().astype(int)
    return _graphs([("grid", "rgg", "powerlaw")[g % 3] for g in range(case["graphs"])], [int(s) for s in sizes], seed)


# ---- state and pass ----------------------------------------------------------------

def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=DEV.type == "cuda")


def prepare(case, seed):
    s = dict(case=case)
    path = case["path"]
    if path == "batched":
        gs = _set_of_graphs(case, seed)
        algo = [2 if g.n < 5000 else 4 for g in gs]
        s["layout"] = B.BatchedLayout([(g.rowptr, g.colids) for g in gs], algo, [g.mid.cpu().numpy() for g in gs])
        s["layout"].set_parts([2, 2, 2])  # a fixed source split: runs repeat bit for bit
        return s
    if path == "train":
        gs = _set_of_graphs(case, seed)
        s["graphs"] = [(g.rowptr, g.colids) for g in gs]
        s["targets"] = [g.mid.double().cpu().numpy() for g in gs]
        s["params"], _ = learned.load_model()
        s["net"] = _lib.Mpnn(s["params"])
        return s
    (g,) = _graphs([case["graph"]], [case["n"]], seed)
    if path == "noalloc":
        mrp, mci = _lib.cursor_neighbours(g.rowptr, g.colids)
        s.update(n=g.n, rowptr=torch.from_numpy(mrp).to(DEV), colids=torch.from_numpy(mci).to(DEV),
                 start=g.mid.clone() if case["layout"] == "mid" else g.disc.clone(),
                 xy=torch.zeros(g.n, 2, device=DEV), force=torch.zeros(g.n, 2, dtype=torch.float64, device=DEV),
                 force32=torch.zeros(g.n, 2, device=DEV), e=torch.zeros(g.n, dtype=torch.float64, device=DEV),
                 energy=_lib.C.c_double())
        return s
    s["engine"] = B.Algorithms(g.rowptr, g.colids)
    s["out"] = _pinned((g.n, 2), torch.float64)
    s["xy"] = torch.zeros(g.n, 2)
    if path == "learned_init":
        s["params"], s["scale"] = learned.load_model()
    else:
        s["start"] = _pinned((g.n, 2), torch.float64)
        s["start"].copy_(g.mid if case["layout"] == "mid" else g.disc)
    return s


def run(s):
    case = s["case"]
    path = case["path"]
    if path == "batched":
        L = s["layout"]
        L.run(case["iterations"], case["batch"], case["theta"])
        xy, energy = L.result()
        return dict(xy=np.concatenate(xy).astype(np.float32), energy=energy.astype(np.float32))
    if path == "train":
        s["net"].set_params(s["params"])
        params, scale, history = s["net"].train(s["graphs"], s["targets"], case["epochs"], lr=3e-4, seed=7)
        return dict(params=params, scale=scale.astype(np.float32), history=history.astype(np.float32))
    if path == "noalloc":
        s["xy"].copy_(s["start"])
        st = torch.cuda.current_stream()
        rc = _lib.load().bl_minibatch_iteration_noalloc(
            s["n"], s["rowptr"].data_ptr(), s["colids"].data_ptr(), s["xy"].data_ptr(), s["force"].data_ptr(),
            s["e"].data_ptr(), case["algo"], case["batch"], 1.0, case["step"], _lib.C.byref(s["energy"]),
            st.cuda_stream)
        if rc:
            raise RuntimeError(f"bl_minibatch_iteration_noalloc: {rc}")
        s["force32"].copy_(s["force"])
        return dict(xy=s["xy"], force=s["force32"], energy=s["energy"].value)
    a = s["engine"]
    if path == "learned_init":
        a.learnedInit(s["params"], s["scale"], 1)
        a.get_coordinates_ptr(s["out"].data_ptr())
        s["xy"].copy_(s["out"])
        return dict(xy=s["xy"])
    a.set_coordinates_ptr(s["start"].data_ptr())
    energy = a.run_resident(case["algo"], case["iterations"], case["batch"], case.get("theta", 1.2), case["step"])
    a.get_coordinates_ptr(s["out"].data_ptr())
    s["xy"].copy_(s["out"])
    return dict(xy=s["xy"], energy=energy)


def work(case):
    """What a pass cannot do without: coordinates and CSR in, coordinates out;
    10 operations per ordered pair of an all-pairs iteration, 20 per record
    of a Barnes-Hut walk (about 4.5 log2(n) / theta^2 records), the products
    of the network."""
    path = case["path"]
    net = 2.0 * (64 * 32 + 2 * 64 * 128 + 2 * 64)

    def bh(n, theta, it):
        return it * n * 20.0 * 4.5 * math.log2(max(n, 2)) / (theta * theta)

    if path in ("batched", "train"):
        lo, hi, count = case["lo"], case["hi"], case["graphs"]
        span = math.log(max(hi, lo + 1) / lo)
        mean = (hi - lo) / span
        if path == "train":
            nv = mean * count
            return dict(bytes=nv * (16 + 4 * 7.3 + 4), flops=3 * net * nv * case["epochs"])
        cut = min(5000, hi)
        pairs = (cut * cut - lo * lo) / (2 * span) * count
        tree = max(hi - cut, 0) / span * count
        return dict(bytes=mean * count * (32 + 4 + 4 * 7.3),
                    flops=10 * pairs * case["iterations"] + bh(tree, case["theta"], case["iterations"]))
    n = case["n"]
    csr = 4.0 * (n + 1) + 4.0 * n * DEGREE[case["graph"]]
    if path == "learned_init":
        return dict(bytes=csr + 16.0 * n, flops=net * n)
    it = case["iterations"]
    if path == "barnes_hut":
        return dict(bytes=csr + 32.0 * n, flops=bh(n, case["theta"], it))
    if path == "greedy":
        walk = min(it, int(0.8 * it) + 1)
        return dict(bytes=csr + 32.0 * n + 8.0 * 22 * n, flops=10.0 * n * n * (it - walk) + 10.0 * 32 * n * walk)
    return dict(bytes=csr + (32.0 if path == "minibatch" else 40.0) * n, flops=10.0 * n * n * it)


# ---- 64-bit values -------------------------------------------------------------------

def _rows(rowptr):
    return torch.repeat_interleave(torch.arange(rowptr.numel() - 1, device=DEV), rowptr[1:] - rowptr[:-1])


def _step(x, f, step):
    mag = f.norm(dim=1, keepdim=True)
    return x + torch.where(mag > 0, f * (step / torch.where(mag > 0, mag, 1.0)), 0.0)


def _exact_minibatch(algo, g, x, batch, iterations, step):
    """sample/algorithms.cpp:739-783 and its variants: attraction instead of
    repulsion for neighbours, repulsion -d/|d|^2 for every other vertex; a
    batch moves together, later batches see it moved."""
    rowptr = g.rowptr.astype(np.int64)
    cols = torch.from_numpy(g.colids.astype(np.int64)).to(DEV)
    rows = _rows(torch.from_numpy(rowptr).to(DEV))
    n = g.n
    x = x.clone()
    force = torch.zeros_like(x)
    for _ in range(iterations):
        for lo in range(0, n, batch):
            hi = min(n, lo + batch)
            dx = x[None, :, 0] - x[lo:hi, 0, None]
            dy = x[None, :, 1] - x[lo:hi, 1, None]
            w = dx * dx + dy * dy
            w = torch.where(w > 0, 1.0 / w, 0.0)
            f = -torch.stack([(dx * w).sum(1), (dy * w).sum(1)], 1)
            del dx, dy, w
            e0, e1 = int(rowptr[lo]), int(rowptr[hi])
            i, j = rows[e0:e1], cols[e0:e1]
            d = x[j] - x[i]
            d2 = (d * d).sum(1)
            far = d2.sqrt()
            pull = far if algo in (2, 7) else torch.log2(1.0 + far) if algo == 3 else torch.ones_like(far)
            pull = pull + torch.where(d2 > 0, 1.0 / d2, 0.0)
            f.index_add_(0, i - lo, d * pull[:, None])
            x[lo:hi] = _step(x[lo:hi], f, step)
            force[lo:hi] = f
        step *= DECAY[algo]
    return x, force, float((force * force).sum())


def _spread(v):
    for s, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F), (2, 0x3333333333333333),
                 (1, 0x5555555555555555)):
        v = (v | (v << s)) & m
    return v


def _tree(x):
    """The quadtree of the points by Morton prefixes: sorted order, frame
    size, and per level the first point of every cell, its first child cell
    on the next level, and its centroid (mean of its children's)."""
    n = x.shape[0]
    low = x.min(0)[0]
    size = float((x.max(0)[0] - low).max())
    q = (4294967295.0 * (x - low) / size).long()
    key = (_spread(q[:, 1]) << 1) | _spread(q[:, 0])
    order = torch.argsort(key ^ (-1 << 63), stable=True)
    k = key[order]
    diff = k[1:] ^ k[:-1]
    top, bot = (diff >> 32) & 0xFFFFFFFF, diff & 0xFFFFFFFF
    bits = torch.where(top > 0, torch.frexp(top.double())[1] + 32, torch.frexp(bot.double())[1])
    same = torch.where(diff == 0, 32, (64 - bits) // 2)  # leading digits in common
    depth = min(32, int(same.max()) + 1)
    first = [torch.cat([torch.zeros(1, dtype=torch.long, device=DEV), 1 + torch.nonzero(same < L)[:, 0]])
             for L in range(depth + 1)]
    levels = [None] * (depth + 1)
    below, cen = torch.arange(n, device=DEV), x[order]
    for L in range(depth, -1, -1):
        f = first[L]
        child = torch.searchsorted(below, f)
        count = torch.diff(child, append=torch.tensor([below.numel()], device=DEV))
        cell = torch.repeat_interleave(torch.arange(f.numel(), device=DEV), count)
        cen = torch.zeros(f.numel(), 2, dtype=torch.float64, device=DEV).index_add_(0, cell, cen) / count[:, None]
        points = torch.diff(f, append=torch.tensor([n], device=DEV))
        levels[L] = (child, count, points, cen)
        below = f
    return order, size, levels


def _exact_repulsion(x, theta):
    """sample/BarnesHut.h:69-86: unit vectors from every accepted cell."""
    order, size, levels = _tree(x)
    n = x.shape[0]
    xs = x[order]
    out = torch.zeros_like(x)
    for c0 in range(0, n, 200_000):
        qi = torch.arange(c0, min(n, c0 + 200_000), device=DEV)
        acc = torch.zeros(qi.numel(), 2, dtype=torch.float64, device=DEV)
        node = torch.zeros_like(qi)
        for L, (child, count, points, cen) in enumerate(levels):
            d = cen[node] - xs[qi]
            dist = (d * d).sum(1).sqrt()
            leaf = points[node] == 1
            near = ~leaf & ~((size / 2.0 ** L) / dist < theta)
            unit = torch.where((~near & (dist > 0))[:, None], d / torch.where(dist > 0, dist, 1.0)[:, None], 0.0)
            acc.index_add_(0, qi - c0, unit)
            qi, node = qi[near], node[near]
            c = count[node]
            first = torch.repeat_interleave(child[node] - (torch.cumsum(c, 0) - c), c)
            qi = torch.repeat_interleave(qi, c)
            node = first + torch.arange(qi.numel(), device=DEV)
        d = xs[node] - xs[qi]  # cells of the last level that were opened: their points
        dist = (d * d).sum(1).sqrt()
        acc.index_add_(0, qi - c0, torch.where((dist > 0)[:, None], d / torch.where(dist > 0, dist, 1.0)[:, None], 0.0))
        out[order[c0:c0 + acc.shape[0]]] = acc
    return out


def _exact_barnes_hut(g, x, batch, iterations, theta, step):
    """sample/algorithms.cpp:1038-1072."""
    rowptr = g.rowptr.astype(np.int64)
    cols = torch.from_numpy(g.colids.astype(np.int64)).to(DEV)
    rows = _rows(torch.from_numpy(rowptr).to(DEV))
    x = x.clone()
    force = torch.zeros_like(x)
    for _ in range(iterations):
        rep = _exact_repulsion(x, theta)
        for lo in range(0, g.n, batch):
            hi = min(g.n, lo + batch)
            e0, e1 = int(rowptr[lo]), int(rowptr[hi])
            i, j = rows[e0:e1], cols[e0:e1]
            d = x[j] - x[i]
            f = (-rep[lo:hi]).index_add_(0, i - lo, d * d.norm(dim=1, keepdim=True))
            x[lo:hi] = _step(x[lo:hi], f, step)
            force[lo:hi] = f
        step *= DECAY[4]
    return x, force, float((force * force).sum())


def exact(case, seed):
    path = case["path"]
    if path in ("learned_init", "train", "greedy"):
        return None  # 16-bit activations; depth-first walks of every vertex
    if path == "batched":
        if case["graphs"] * case["iterations"] > 600:
            return None
        xy, energy = [], []
        for g in _set_of_graphs(case, seed):
            x = g.mid.double()
            if g.n < 5000:
                r = _exact_minibatch(2, g, x, case["batch"], case["iterations"], 1.0)
            else:
                r = _exact_barnes_hut(g, x, case["batch"], case["iterations"], case["theta"], 1.0)
            xy.append(r[0])
            energy.append(r[2])
        return dict(xy=torch.cat(xy), energy=np.array(energy))
    (g,) = _graphs([case["graph"]], [case["n"]], seed)
    x = (g.mid if case["layout"] == "mid" else g.disc).double()
    if path == "barnes_hut":
        r = _exact_barnes_hut(g, x, case["batch"], case["iterations"], case["theta"], case["step"])
        return dict(xy=r[0], energy=np.array(r[2]))
    r = _exact_minibatch(case["algo"], g, x, case["batch"], case["iterations"], case["step"])
    if path == "noalloc":
        return dict(xy=r[0], force=r[1], energy=np.array(r[2]))
    return dict(xy=r[0], energy=np.array(r[2]))
