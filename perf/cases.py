"""Workloads of the library as its users run them, for timing and for comparing outputs.

Every case goes through the package's public functions: the csg reorder on device and on host
arrays, the permutation apply, the fp32 SpMM, one training step of the two-layer GCN, and the
global top-k graph.  Matrices are the five benchmark configurations' families (power-law row
lengths around a band, 9-point mesh, road lattice, R-MAT, symmetrised R-MAT with normalised
values), generated on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import torch

import chunkedgreedy_b200 as sp
from chunkedgreedy_b200 import gcn

# nonzeros per row after duplicates are gone
_MESH_DEG, _ROAD_DEG, _ZIPF_DEG = 9.0, 3.3, 13.8


def listed():
    return [
        # one small matrix, default parameters: what a caller pays when launches and host code count
        dict(name="csg_zipf_4k", op="csg", graph="zipf", rows=4096, k=0, chunk=0, promise=False),
        # benchmark configuration 1: power-law row lengths around a band, rows shuffled
        dict(name="csg_zipf_65k", op="csg", graph="zipf", rows=65536, k=16, chunk=0, promise=False),
        # configuration 2: a finite-element mesh with shuffled labels, symmetry promised
        dict(name="csg_mesh_1m", op="csg", graph="mesh", rows=1 << 20, k=0, chunk=0, promise=True),
        # configuration 4: the power-law graph that the headline figure is quoted on
        dict(name="csg_rmat_22", op="csg", graph="rmat", rows=1 << 22, edges=16, k=0, chunk=0, promise=False),
        # configuration 5's reorder: denser and symmetric, so 30 candidates a row
        dict(name="csg_gcn_20", op="csg", graph="gcn", rows=1 << 20, edges=16, k=0, chunk=0, promise=True),
        # configuration 3 from pinned host arrays to a pinned host permutation: the whole call of a
        # program that keeps its matrices on the host
        dict(name="csg_host_road_2m", op="csg_host", graph="road", rows=2_000_000, k=0, chunk=0, promise=True),
        # P A P^T with values, after the reorder of configuration 4
        dict(name="apply_rmat_22", op="apply", graph="rmat", rows=1 << 22, edges=16, order="csg", symmetric=True,
             values=True),
        # SpMM on the reordered power-law graph at a feature width; the caller waits for C
        dict(name="spmm_rmat_22_w128", op="spmm", graph="rmat", rows=1 << 22, edges=16, order="csg", width=128,
             wait=True),
        # SpMM on a mesh in grid order (what a good ordering looks like), one launch among others
        dict(name="spmm_mesh_1m_w32", op="spmm", graph="mesh", rows=1 << 20, order="grid", width=32, wait=False),
        # a small SpMM with ragged sizes: an odd number of rows, as many columns as a task has classes
        dict(name="spmm_zipf_20k_w41", op="spmm", graph="zipf", rows=20_011, order="given", width=41, wait=False),
        # one full-batch training step of configuration 5: forward, backward and SGD update
        dict(name="gcn_step_20", op="gcn_step", graph="gcn", rows=1 << 20, edges=16, features=128, hidden=128,
             classes=16),
        # the global top-k similarity graph (no chunks), as the analysis scripts build it
        dict(name="topk_graph_rmat_16", op="topk_graph", graph="rmat", rows=1 << 16, edges=16, k=0, promise=False),
    ]


def _log_size(rng, low, high):
    return int(round(2.0 ** rng.uniform(low, high)))


def _draw_graph(rng, largest):
    """A matrix of one of the five families with up to 2**largest rows."""
    graph = rng.choice(("zipf", "mesh", "road", "rmat", "rmat", "gcn"))
    if graph == "zipf":
        return dict(graph=graph, rows=_log_size(rng, 11, min(largest, 17)))
    if graph in ("mesh", "road"):
        return dict(graph=graph, rows=_log_size(rng, 12, min(largest, 20.9)))
    return dict(graph=graph, rows=_log_size(rng, 12, largest if graph == "rmat" else min(largest, 20)),
                edges=rng.randint(4, 16))


def draw(rng):
    """One more case of the ranges above, sizes spread over their logarithm."""
    op = rng.choice(("csg", "csg", "csg", "csg", "csg_host", "apply", "apply", "spmm", "spmm", "spmm", "gcn_step",
                     "topk_graph"))
    if op in ("csg", "csg_host"):
        c = dict(op=op, **_draw_graph(rng, 22))
        c["k"] = rng.choice((0, 0, 16, rng.randint(10, 24 if c["rows"] <= 1 << 20 else 16)))
        c["chunk"] = rng.choice((0, 0, 512, rng.randint(200, 1024)))
        c["promise"] = c["graph"] in ("mesh", "road", "gcn") and rng.random() < 0.7
        return c
    if op == "apply":
        c = dict(op=op, **_draw_graph(rng, 22))
        c["order"] = rng.choice(("csg", "csg", "random"))
        c["symmetric"] = rng.random() < 0.7
        c["values"] = rng.random() < 0.7
        return c
    if op == "spmm":
        c = dict(op=op, **_draw_graph(rng, 22))
        c["order"] = "csg" if c["graph"] in ("rmat", "gcn") else ("grid" if c["graph"] == "mesh" else "given")
        c["width"] = rng.choice((16, 32, 64, 128, 256, rng.randint(5, 200)))
        while c["rows"] * c["width"] > 1 << 29:
            c["width"] = max(1, c["width"] // 2)
        c["wait"] = rng.random() < 0.5
        return c
    if op == "gcn_step":
        return dict(op=op, graph="gcn", rows=_log_size(rng, 12, 20), edges=rng.randint(4, 16),
                    features=rng.choice((64, 100, 128)), hidden=rng.choice((32, 64, 128)),
                    classes=rng.choice((7, 16, rng.randint(3, 47))))
    return dict(op=op, graph=rng.choice(("zipf", "rmat", "gcn")), rows=_log_size(rng, 11, 15.9),
                edges=rng.randint(4, 12), k=rng.choice((0, rng.randint(8, 32))), promise=False)


# ---- matrices ------------------------------------------------------------------------------


def _csr(n, rows, cols):
    """Sorted, duplicate-free CSR pattern from coordinates."""
    return _from_keys(n, torch.unique(rows.long() * n + cols.long()))


def _from_keys(n, key):
    r = torch.div(key, n, rounding_mode="floor")
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
    torch.cumsum(torch.bincount(r, minlength=n), 0, out=ptr[1:])
    return ptr.int(), (key - r * n).int()


def _row_ids(ptr):
    n = ptr.numel() - 1
    return torch.repeat_interleave(torch.arange(n, device=ptr.device), (ptr[1:] - ptr[:-1]).long())


def _thinned(ptr, ind, count, g):
    """`count` of the nonzeros, chosen at random: the same number for every seed."""
    n = ptr.numel() - 1
    pick = torch.randperm(ind.numel(), generator=g, device=g.device)[:count].sort()[0]
    return _from_keys(n, (_row_ids(ptr) * n + ind)[pick])


def _zipf(n, g):
    """Row lengths 3 * Zipf(2) up to 4096, at evenly spaced quantiles; 70 % of the columns within
    512 of a centre of the row's own, the others anywhere; rows in random order."""
    dev = g.device
    k = torch.arange(1, 4096, dtype=torch.float64, device=dev)
    cdf = torch.cumsum(1.0 / (k * k), 0) * (6.0 / math.pi ** 2)
    at = (torch.randperm(n, generator=g, device=dev).double() + 0.5) / n
    length = (3 * (torch.searchsorted(cdf, at) + 1)).clamp(max=min(4096, n))
    rows = torch.repeat_interleave(torch.arange(n, device=dev), length)
    total = rows.numel()
    centre = torch.randint(0, n, (n,), generator=g, device=dev)
    near = (centre[rows] + torch.randint(-512, 513, (total,), generator=g, device=dev)) % n
    far = torch.randint(0, n, (total,), generator=g, device=dev)
    cols = torch.where(torch.rand(total, generator=g, device=dev) < 0.7, near, far)
    return _csr(n, rows, cols)


def _grid(rows):
    a = max(2, math.isqrt(rows))
    return a, max(2, rows // a)


def _mesh(rows, g, shuffled):
    """9-point stencil on a grid, labels shuffled or in grid order."""
    dev = g.device
    height, width = _grid(rows)
    n = height * width
    v = torch.arange(n, device=dev)
    y, x = torch.div(v, width, rounding_mode="floor"), v % width
    rr, cc = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            ok = (y + dy >= 0) & (y + dy < height) & (x + dx >= 0) & (x + dx < width)
            rr.append(v[ok])
            cc.append(v[ok] + dy * width + dx)
    r, c = torch.cat(rr), torch.cat(cc)
    if shuffled:
        q = torch.randperm(n, generator=g, device=dev)
        r, c = q[r], q[c]
    return _csr(n, r, c)


def _road(n, g):
    """Vertices on a jittered lattice, each linked to its 1 to 4 nearest of the eight around it,
    symmetrised, labels shuffled."""
    dev = g.device
    side = math.isqrt(n - 1) + 1
    v = torch.arange(n, device=dev)
    gy, gx = torch.div(v, side, rounding_mode="floor"), v % side
    px = gx + torch.rand(n, generator=g, device=dev) - 0.5
    py = gy + torch.rand(n, generator=g, device=dev) - 0.5
    degree = torch.randint(1, 5, (n,), generator=g, device=dev)
    near, dist = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            if dy == 0 and dx == 0:
                continue
            w = v + dy * side + dx
            ok = (gy + dy >= 0) & (gx + dx >= 0) & (gx + dx < side) & (w >= 0) & (w < n)
            w = torch.where(ok, w, torch.zeros_like(w))
            d = (px - px[w]) ** 2 + (py - py[w]) ** 2
            near.append(w)
            dist.append(torch.where(ok, d, torch.full_like(d, float("inf"))))
    near, dist = torch.stack(near, 1), torch.stack(dist, 1)
    d, at = torch.sort(dist, dim=1, stable=True)
    keep = (torch.arange(8, device=dev)[None, :] < degree[:, None]) & torch.isfinite(d)
    r = v[:, None].expand(-1, 8)[keep]
    c = near.gather(1, at)[keep]
    q = torch.randperm(n, generator=g, device=dev)
    r, c = q[torch.cat([r, c])], q[torch.cat([c, r])]
    return _csr(n, r, c)


def _rmat(n, edges, g, symmetric):
    """R-MAT edges (0.57, 0.19, 0.19, 0.05), vertices of the next power of two scaled onto n;
    `symmetric` adds the transposed edges and the diagonal."""
    dev = g.device
    scale = max(1, (n - 1).bit_length())
    m = n * edges
    r = torch.zeros(m, dtype=torch.int32, device=dev)
    c = torch.zeros(m, dtype=torch.int32, device=dev)
    for _ in range(scale):
        u = torch.rand(m, generator=g, device=dev)
        lower = u >= 0.76
        right = (u >= 0.95) | ((u >= 0.57) & ~lower)
        r = r * 2 + lower
        c = c * 2 + right
    if n != 1 << scale:
        r, c = (r.long() * n) >> scale, (c.long() * n) >> scale
    if symmetric:
        v = torch.arange(n, device=dev)
        r, c = torch.cat([r.long(), c.long(), v]), torch.cat([c.long(), r.long(), v])
    return _csr(n, r, c)


def _pattern(case, g):
    graph, n = case["graph"], case["rows"]
    if graph == "zipf":
        return _zipf(n, g)
    if graph == "mesh":
        return _mesh(n, g, case.get("order") != "grid")
    if graph == "road":
        return _road(n, g)
    return _rmat(n, case["edges"], g, graph == "gcn")


def _values(case, ptr, ind, g):
    """Each family's own: unit weights on roads, the normalised adjacency of the GCN, U(0, 1]
    on R-MAT, U[-1, 1] on the banded one, N(0, 1) on the mesh."""
    graph, m, dev = case["graph"], ind.numel(), ind.device
    if graph == "road":
        return torch.ones(m, device=dev)
    if graph == "gcn":
        return gcn.normalised_values(ptr, ind)
    if graph == "rmat":
        return 1.0 - torch.rand(m, generator=g, device=dev)
    if graph == "zipf":
        return torch.rand(m, generator=g, device=dev) * 2.0 - 1.0
    return torch.randn(m, generator=g, device=dev)


# ---- the cases -----------------------------------------------------------------------------


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    op = case["op"]
    ptr, ind = _pattern(case, g)
    n = ptr.numel() - 1
    if op == "apply":
        ptr, ind = _thinned(ptr, ind, int(_nnz(case)), g)
    s = dict(case=case, op=op, ptr=ptr, ind=ind)
    if op in ("csg", "csg_host"):
        s["options"] = dict(is_symmetric=case["promise"], k=case["k"], chunk_size=case["chunk"])
        if op == "csg_host":
            s["ptr"], s["ind"] = ptr.cpu().pin_memory(), ind.cpu().pin_memory()
            s["out"] = torch.empty(n, dtype=torch.int32).pin_memory()
    elif op == "topk_graph":
        s["options"] = dict(is_symmetric=case["promise"], k=case["k"])
    elif op == "apply":
        s["val"] = _values(case, ptr, ind, g) if case["values"] else None
        s["order"] = (torch.randperm(n, generator=g, device=dev).int() if case["order"] == "random"
                      else sp.chunk_similarity_greedy(ptr, ind))
    elif op == "spmm":
        val = _values(case, ptr, ind, g)
        if case["order"] == "csg":
            ptr, ind, val = sp.reorder(ptr, ind, sp.chunk_similarity_greedy(ptr, ind), val=val, symmetric=True)
        s.update(ptr=ptr, ind=ind, val=val, B=torch.randn((n, case["width"]), generator=g, device=dev))
    else:  # gcn_step
        torch.manual_seed(seed)
        s["model"] = gcn.GCN(case["features"], case["hidden"], case["classes"]).to(dev)
        s["opt"] = torch.optim.SGD(s["model"].parameters(), lr=0.01)
        s["graph"] = gcn.GraphOperator(ptr, ind, _values(case, ptr, ind, g))
        s["x"] = torch.randn((n, case["features"]), generator=g, device=dev)
        s["y"] = torch.randint(0, case["classes"], (n,), generator=g, device=dev)
    return s


def run(s):
    op, case = s["op"], s["case"]
    if op == "csg":
        return sp.chunk_similarity_greedy(s["ptr"], s["ind"], **s["options"])
    if op == "csg_host":
        return sp.chunk_similarity_greedy_host(s["ptr"], s["ind"], out=s["out"], **s["options"])
    if op == "topk_graph":
        return sp.similarity_graph(s["ptr"], s["ind"], **s["options"])
    if op == "apply":
        return sp.reorder(s["ptr"], s["ind"], s["order"], val=s["val"], symmetric=case["symmetric"])
    if op == "spmm":
        return sp.spmm(s["ptr"], s["ind"], s["val"], s["B"], sync=case["wait"])
    model, opt = s["model"], s["opt"]  # the loop body of gcn.train
    opt.zero_grad()
    z = model(s["x"], s["graph"])
    loss = -torch.log_softmax(z, 1).gather(1, s["y"][:, None]).mean()
    loss.backward()
    opt.step()
    return dict(loss=loss.detach(), z=z.detach(), grads=[p.grad for p in model.parameters()],
                weights=[p.detach() for p in model.parameters()])


def _nnz(case):
    """Nonzeros of a case, within some percent (duplicates vary); exact for the apply, whose
    matrices are thinned to this count."""
    n, graph = case["rows"], case["graph"]
    if graph == "mesh":
        m = _MESH_DEG * n * 0.99
    elif graph in ("zipf", "road"):
        m = n * (_ZIPF_DEG if graph == "zipf" else _ROAD_DEG)
    else:  # duplicate edges: more where the hubs meet on small graphs
        lost = 0.0285 * math.exp(0.19 * (22 - math.log2(n))) * (case["edges"] / 16) ** 0.9
        if graph == "rmat":
            m = n * case["edges"] * (1 - lost)
        else:
            m = n * (1 + 2 * case["edges"] * (1 - 1.6 * lost))
    return m * (0.9 if case["op"] == "apply" else 1.0)


def work(case):
    """Each input read once and each output written once; the flops of the products."""
    n, m, op = case["rows"], _nnz(case), case["op"]
    pattern = 4 * (n + 1) + 4 * m
    if op in ("csg", "csg_host"):  # pattern in, permutation out
        return dict(bytes=pattern + 4 * n, flops=0)
    if op == "topk_graph":  # pattern in, k indices and weights a row out
        k = case["k"] or min(32, max(16, 2 * int(m / n)))
        return dict(bytes=pattern + 8 * n * k, flops=0)
    if op == "apply":
        return dict(bytes=2 * (pattern + (4 * m if case["values"] else 0)) + 4 * n, flops=0)
    if op == "spmm":
        return dict(bytes=pattern + 4 * m + 8 * n * case["width"], flops=2 * m * case["width"])
    f, h, c = case["features"], case["hidden"], case["classes"]
    # Both layers' products forward, and backward for the weights and (second layer) the hidden
    # units; the operator twice forward and twice backward at the narrower side of each layer.  Features,
    # hidden units and their gradient once each, logits out, the matrix once per direction.
    flops = 2 * n * (2 * f * h + 3 * h * c) + 2 * m * 2 * (min(f, h) + min(h, c))
    return dict(bytes=2 * (pattern + 4 * m) + 4 * n * (f + 2 * h + 2 * c) + 8 * n, flops=flops)


def tolerance(case):
    if case["op"] == "spmm":  # fp32 sums of up to 1e5 terms in any order
        return {"rel": 1e-5}
    if case["op"] == "gcn_step":  # gradients are fp32 sums over all rows that largely cancel
        return {"rel": 5e-5}
    return "exact"  # permutations, top-k tables and moved values are defined bit for bit
