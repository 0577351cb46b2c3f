"""The workloads this library is timed on: sweeps, preconditioner applications,
plain and batched solves, continuous batching and the admission of a new
matrix, over meshes, random regular and power-law graphs of the sizes the
benchmark, the serving mix and the tests use.

A case is a dict of plain values:
  path    apply | sweep | pcg | batch | lanes | serve | instances | admit
  graph   grid2d (5-point, weights U[1,2), Laplacian), grid3d (7-point, weights
          10^U[-3,3), +1 on the boundary diagonal), regular (random 6-regular,
          weights U[0.5,2), shift 1e-3 of the degree) or rmat (power-law
          Laplacian, largest connected component)
  size    nodes per side (grids), nodes (regular), log2 of the sampled nodes (rmat)
  k       right-hand sides (slots of a batch)
  and, where the path takes them: precision (of the factor: fp64 / fp32 / fp16),
  host (numpy arrays instead of device tensors), lanes, count (instances or
  requests).

The operator and its factor are made here from the seed, on the GPU: an
approximate Cholesky factor by randomized elimination in rounds (each round
eliminates an independent set of low-degree vertices and replaces each
vertex's star by a sampled tree on its neighbours). Weights are whole numbers
times 2^-30, so that sums do not depend on their order and a seed always gives
the same factor.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from apxchol_b200 import native
from apxchol_b200.gen import Matrix
from apxchol_b200.lanes import Lanes
from apxchol_b200.refsetup import Factor

DEV = "cuda" if torch.cuda.is_available() else "cpu"
UNIT = 2.0 ** 30          # weights are whole multiples of 1 / UNIT
DENSE_TAIL = 1024         # the last vertices are eliminated on the host
TOL = 1e-8
DROP = 1e-4               # the factor's default drop threshold
PRECISION = {"fp64": native.PREC_FP64, "fp32": native.PREC_FP32, "fp16": native.PREC_FP16}


def listed():
    return [
        # one preconditioner application from numpy arrays on the small 2D grid: the library's smallest call
        dict(name="apply_grid2d_256", path="apply", graph="grid2d", size=256, precision="fp64", host=True),
        # a whole small solve from numpy arrays
        dict(name="pcg_grid2d_256", path="pcg", graph="grid2d", size=256, precision="fp64", host=True),
        # the headline system's fp64 preconditioner on device vectors, as an outer solver calls it
        dict(name="sweep64_grid3d_128", path="sweep", graph="grid3d", size=128, precision="fp64", k=1),
        # the same from the fp16-stored factor, at the serving mix's 3D size
        dict(name="sweep16_grid3d_96", path="sweep", graph="grid3d", size=96, precision="fp16", k=1),
        # a block of right-hand sides through the fp32 sweeps
        dict(name="sweep32_regular_k16", path="sweep", graph="regular", size=100003, precision="fp32", k=16),
        # the headline system's plain fp64 solve, right-hand side resident
        dict(name="pcg_grid3d_128", path="pcg", graph="grid3d", size=128, precision="fp64", host=False),
        # a block solve at the serving mix's 3D size
        dict(name="batch_grid3d_96_k16", path="batch", graph="grid3d", size=96, precision="fp32", k=16),
        # a power-law system: a deep dependency chain, hub rows, fp32-exact weights
        dict(name="batch_rmat_16_k16", path="batch", graph="rmat", size=16, precision="fp32", k=16),
        # many uneven systems in one batch, 1 to 8 right-hand sides each
        dict(name="instances_12_k8", path="instances", graph="mixed", size=40000, precision="fp32", k=8, count=12),
        # requests through the slots of a running batch, as the solve server drives it
        dict(name="serve_grid2d_1024_k8", path="serve", graph="grid2d", size=1024, precision="fp32", k=8, count=12),
        # a matrix not seen before: factor, operator and batch made, one block solved, all released
        dict(name="admit_grid3d_61_k4", path="admit", graph="grid3d", size=61, precision="fp32", k=4),
        # the headline: the 128^3 system in concurrent 64-slot batches
        dict(name="lanes2_grid3d_128_k64", path="lanes", graph="grid3d", size=128, precision="fp32", k=64, lanes=2),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, nodes):
    """A graph family and the size that gives at most about `nodes` nodes, from the range [~4000, nodes]."""
    graph = rng.choice(["grid2d", "grid3d", "grid3d", "regular", "rmat"])
    n = _log_uniform(rng, 4000, nodes)
    if graph == "grid2d":
        return graph, max(60, int(math.sqrt(n)))
    if graph == "grid3d":
        return graph, max(16, int(round(n ** (1 / 3))))
    if graph == "regular":
        return graph, min(n, 120000)
    return graph, min(16, max(12, int(math.log2(n))))


def draw(rng):
    path = rng.choice(["apply", "sweep", "pcg", "batch", "batch", "instances", "serve", "admit"])
    graph, size = _draw_graph(rng, {"apply": 2e6, "sweep": 2e6, "pcg": 1.2e6}.get(path, 9e5))
    if path == "apply":
        return dict(path=path, graph=graph, size=size, precision=rng.choice(["fp64", "fp64", "fp32", "fp16"]),
                    host=rng.random() < 0.5)
    if path == "sweep":
        precision = rng.choice(["fp64", "fp32", "fp32", "fp16"])
        return dict(path=path, graph=graph, size=size, precision=precision,
                    k=1 if precision == "fp64" else rng.choice([1, 2, 4, 8, 16]))
    if path == "pcg":
        return dict(path=path, graph=graph, size=size, precision="fp64", host=rng.random() < 0.5)
    if path == "batch":
        return dict(path=path, graph=graph, size=size, precision=rng.choice(["fp32", "fp32", "fp32", "fp16"]),
                    k=rng.choice([1, 2, 4, 8, 16, 32, 64, 128] if size < 300 or graph == "regular" else [1, 2, 4, 8, 16]))
    if path == "instances":
        return dict(path=path, graph="mixed", size=_log_uniform(rng, 3000, 50000), precision="fp32",
                    k=rng.choice([4, 8]), count=rng.randint(3, 12))
    if path == "serve":
        k = rng.choice([4, 8, 16])
        return dict(path=path, graph=graph, size=size, precision="fp32", k=k, count=k + rng.randint(1, k))
    return dict(path=path, graph=graph, size=size, precision="fp32", k=rng.choice([1, 2, 4, 8]))


# ---- operators ----

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed & 0x7FFFFFFF)
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, dtype=torch.float64, device=DEV)


def _merge(n, u, v, w):
    """Edges u < v in order, the weights of equal ones summed."""
    key, order = torch.sort(torch.minimum(u, v) * n + torch.maximum(u, v))
    key, inv = torch.unique_consecutive(key, return_inverse=True)
    w = torch.zeros(key.numel(), dtype=torch.int64, device=DEV).index_add_(0, inv, w[order])
    u = torch.div(key, n, rounding_mode="floor")
    return u, key - u * n, w


def _components(n, u, v):
    """Each node's smallest connected node."""
    lab = torch.arange(n, device=DEV)
    while True:
        old = lab
        low = torch.minimum(lab[u], lab[v])
        lab = lab.scatter_reduce(0, u, low, "amin").scatter_reduce(0, v, low, "amin")
        lab = lab[lab]
        if torch.equal(lab, old):
            return lab


def graph_of(graph, size, seed):
    """(nodes, u, v, w, excess): undirected edges with whole weights and the diagonal excess (zero: a Laplacian)."""
    g = _gen(seed)
    if graph in ("grid2d", "grid3d"):
        dim = 2 if graph == "grid2d" else 3
        n = size ** dim
        idx = torch.arange(n, device=DEV).reshape([size] * dim)
        u = torch.cat([idx.narrow(a, 0, size - 1).reshape(-1) for a in range(dim)])
        v = torch.cat([idx.narrow(a, 1, size - 1).reshape(-1) for a in range(dim)])
        r = _rand(g, u.numel())
        w = 1.0 + r if dim == 2 else 10.0 ** (6.0 * r - 3.0)
        excess = torch.zeros([size] * dim, dtype=torch.int64, device=DEV)
        if dim == 3:
            for a in range(3):
                excess.select(a, 0).fill_(int(UNIT))
                excess.select(a, size - 1).fill_(int(UNIT))
        return n, u, v, (w * UNIT).to(torch.int64), excess.reshape(-1)
    if graph == "regular":
        n = size
        perms = [torch.argsort(_rand(g, n)) for _ in range(3)]
        u = torch.cat(perms)
        v = torch.cat([torch.roll(p, -1) for p in perms])
        w = ((0.5 + 1.5 * _rand(g, u.numel())) * UNIT).to(torch.int64)
        u, v, w = _merge(n, u, v, w)
        deg = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
        return n, u, v, w, (1e-3 * UNIT * deg.to(torch.float64)).to(torch.int64)
    # the sampled edges are the same for every seed (the component's size with them); factor and right-hand sides differ
    g = _gen(size)
    n = 1 << size
    m = 16 * n
    u = torch.zeros(m, dtype=torch.int64, device=DEV)
    v = torch.zeros(m, dtype=torch.int64, device=DEV)
    for level in range(size):
        r = _rand(g, m)
        u = 2 * u + (r >= 0.76)
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = u != v
    u, v = u[keep], v[keep]
    u, v, w = _merge(n, u, v, torch.full_like(u, int(UNIT)))
    lab = _components(n, u, v)
    big = torch.bincount(lab, minlength=n).argmax()
    node = lab == big
    new = torch.cumsum(node, 0) - 1
    keep = node[u]
    n = int(node.sum())
    return n, new[u[keep]], new[v[keep]], w[keep], torch.zeros(n, dtype=torch.int64, device=DEV)


def operator_of(n, u, v, w, excess):
    """(colptr, rowidx, vals) of D - W + diag(excess) on the device: full symmetric CSC, rows ascending."""
    diag = excess.clone().index_add_(0, u, w).index_add_(0, v, w)
    node = torch.arange(n, device=DEV)
    key, order = torch.sort(torch.cat([u * n + v, v * n + u, node * (n + 1)]))
    vals = torch.cat([-w, -w, diag])[order].to(torch.float64) / UNIT
    col = torch.div(key, n, rounding_mode="floor")
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
    return ptr, key - col * n, vals


# ---- the factor ----

def _independent(n, alive, deg, u, v, g, passes):
    """An independent set of the alive vertices of about the average degree at most, low degrees first."""
    count = int(alive.sum())
    limit = 1 + max(3, math.ceil(2 * u.numel() / max(1, count)))
    order = deg * (1 << 40) + torch.randint(1 << 40, (n,), generator=g, device=DEV)
    big = torch.iinfo(torch.int64).max
    chosen = torch.zeros_like(alive)
    free = alive & (deg <= limit)
    if not bool(free.any()):
        free = alive
    for _ in range(passes):
        key = torch.where(free, order, big)
        low = torch.full((n,), big, dtype=torch.int64, device=DEV)
        low = low.scatter_reduce(0, u, key[v], "amin").scatter_reduce(0, v, key[u], "amin")
        now = free & (key < low)
        chosen |= now
        beside = torch.zeros(n, dtype=torch.int64, device=DEV)
        beside.index_add_(0, u, now[v].to(torch.int64)).index_add_(0, v, now[u].to(torch.int64))
        free &= ~now & (beside == 0)
        if not bool(free.any()):
            break
    return chosen


def _dense_tail(ids, ground, edges, rng):
    """The last vertices, on the host: rounds of independent vertices, lowest degree first."""
    at = {x: i for i, x in enumerate(ids)}
    s, gi = len(ids), at[ground]
    w = np.zeros((s, s), np.int64)
    for a, b, x in zip(*edges):
        w[at[a], at[b]] += x
        w[at[b], at[a]] += x
    left = np.ones(s, bool)
    left[gi] = False
    src, dst, val, tot, rounds, order = [], [], [], [], [], []
    while left.any():
        deg = (w > 0).sum(1)
        cand = np.flatnonzero(left)
        cand = cand[np.argsort(deg[cand], kind="stable")]
        blocked = np.zeros(s, bool)
        now = []
        limit = max(4, 2 * deg[cand].mean())
        for x in cand:
            if not blocked[x] and (deg[x] <= limit or not now):
                now.append(x)
                blocked |= w[x] > 0
        for x in sorted(now):
            nb = np.flatnonzero(w[x])
            nb = nb[np.argsort(w[x, nb], kind="stable")]
            wx = w[x, nb].copy()
            t = int(wx.sum())
            order.append(ids[x])
            tot.append(t)
            src += [ids[x]] * len(nb)
            dst += [ids[y] for y in nb]
            val += wx.tolist()
            w[x, nb] = 0
            w[nb, x] = 0
            if len(nb) > 1:
                c = np.cumsum(wx)
                suffix = t - c[:-1]
                r = np.floor(rng.random(len(nb) - 1) * suffix).astype(np.int64) + 1
                to = np.minimum(np.searchsorted(c, c[:-1] + r), len(nb) - 1)
                fill = np.maximum(1, np.rint(wx[:-1] * (suffix / t))).astype(np.int64)
                a, b = nb[:-1], nb[to]
                np.add.at(w, (a, b), fill)
                np.add.at(w, (b, a), fill)
            left[x] = False
        rounds.append(len(now))
    return src, dst, val, tot, rounds, order


def factor_of(n, u, v, w, excess, seed):
    """The approximate factor of the operator, as the setup phase hands it over (numpy arrays)."""
    g = _gen(seed + 77)
    sddm = bool((excess > 0).any())
    if sddm:      # the excess is an edge to a ground vertex that is never eliminated
        at = torch.nonzero(excess).reshape(-1)
        u, v, w = torch.cat([u, at]), torch.cat([v, torch.full_like(at, n)]), torch.cat([w, excess[at]])
        total, ground = n + 1, n
    else:
        total = n
        deg = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
        ground = int(deg.argmax())
    alive = torch.ones(total, dtype=torch.bool, device=DEV)
    alive[ground] = False
    u, v, w = _merge(total, u, v, w)
    src, dst, val, tot, order, rounds = [], [], [], [], [], []
    while True:
        left = int(alive.sum())
        if left <= DENSE_TAIL:
            break
        deg = torch.bincount(u, minlength=total) + torch.bincount(v, minlength=total)
        inner = (u != ground) & (v != ground)
        now = _independent(total, alive, deg, u[inner], v[inner], g, 1 if rounds else 8)
        here = now[u] | now[v]
        a, b, x = u[here], v[here], w[here]
        swap = now[b]
        a, b = torch.where(swap, b, a), torch.where(swap, a, b)
        x, i = torch.sort(x, stable=True)            # by weight, then (stable) by eliminated vertex
        a, b = a[i], b[i]
        a, i = torch.sort(a, stable=True)
        b, x = b[i], x[i]
        verts, seg, cnt = torch.unique_consecutive(a, return_inverse=True, return_counts=True)
        c = torch.cumsum(x, 0)
        last = torch.cumsum(cnt, 0) - 1
        end = c[last]
        t = torch.diff(end, prepend=torch.zeros(1, dtype=torch.int64, device=DEV))
        src.append(a); dst.append(b); val.append(x); tot.append(t); order.append(verts)
        rounds.append(int(verts.numel()))
        suffix = end[seg] - c
        more = suffix > 0
        r = (_rand(g, a.numel()) * suffix.to(torch.float64)).to(torch.int64) + 1
        to = torch.minimum(torch.searchsorted(c, c + torch.minimum(r, suffix)), last[seg])
        fill = torch.clamp((x.to(torch.float64) * (suffix.to(torch.float64) / t[seg].to(torch.float64))).round()
                           .to(torch.int64), min=1)
        alive = alive & ~now
        rest = ~here
        p, q = b[more], b[to][more]
        ok = p != q
        u, v, w = _merge(total, torch.cat([u[rest], p[ok]]), torch.cat([v[rest], q[ok]]),
                         torch.cat([w[rest], fill[more][ok]]))
    ids = torch.nonzero(alive).reshape(-1).tolist() + [ground]
    tail = _dense_tail(ids, ground, (u.tolist(), v.tolist(), w.tolist()), np.random.default_rng(seed + 78))
    as_dev = lambda q: torch.tensor(q, dtype=torch.int64, device=DEV)  # noqa: E731
    for q, x in zip((src, dst, val, tot), tail):
        q.append(as_dev(x))
    rounds += tail[4]
    order.append(as_dev(tail[5]))
    src, dst, val, tot, order = (torch.cat(q) for q in (src, dst, val, tot, order))
    pos = torch.full((total,), total - 1, dtype=torch.int64, device=DEV)
    pos[order] = torch.arange(order.numel(), device=DEV)
    # column entries: the diagonal sqrt(t), then -w / sqrt(t) at the rows still left (SDDM: the ground's dropped)
    root = torch.sqrt(tot.to(torch.float64) / UNIT)
    col = pos[src]
    offd = -(val.to(torch.float64) / UNIT) / root[col]
    row = pos[dst]
    if sddm:
        keep = dst != ground
        col, row, offd = col[keep], row[keep], offd[keep]
    else:
        root = torch.cat([root, torch.ones(1, dtype=torch.float64, device=DEV)])
    node = torch.arange(n, device=DEV)
    key, i = torch.sort(torch.cat([node * (n + 1), col * n + row]))
    vals = torch.cat([root, offd])[i].to(torch.float32)
    col = torch.div(key, n, rounding_mode="floor")
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
    if sddm:
        rounds[-1] -= 1      # the last vertex stands outside the rounds
        rounds = [r for r in rounds if r > 0]
    return Factor(n=n, colptr=ptr.cpu().numpy().astype(np.uint32), rowidx=(key - col * n).cpu().numpy().astype(np.uint32),
                  vals=vals.cpu().numpy(), perm=pos[:n].cpu().numpy().astype(np.uint32), sddm=sddm,
                  rounds=np.array(rounds, np.uint64))


def system(graph, size, seed):
    """(matrix, factor, the graph it came from)."""
    made = graph_of(graph, size, seed)
    ptr, idx, vals = operator_of(*made)
    fac = factor_of(*made, seed)
    mat = Matrix(n=made[0], colptr=ptr.cpu().numpy().astype(np.int32), rowidx=idx.cpu().numpy().astype(np.int32),
                 vals=vals.cpu().numpy(), name=graph, sddm=fac.sddm)
    return mat, fac, made


def _rhs(n, count, seed, zero_mean):
    b = torch.randn((count, n), generator=_gen(seed + 991), dtype=torch.float64, device=DEV)
    return b - b.mean(1, keepdim=True) if zero_mean else b


def _instances(case, seed):
    """Uneven systems: 2D grids with a diagonal shift and 6-regular graphs by turns, and their right-hand-side counts."""
    rng = np.random.default_rng(case["count"] + case["size"])   # the sizes and counts do not depend on the seed
    out = []
    for i in range(case["count"]):
        n = int(rng.integers(1000, case["size"] + 1))
        graph, size = ("grid2d", max(32, int(math.sqrt(n)))) if i % 2 == 0 else ("regular", n)
        nodes, u, v, w, excess = graph_of(graph, size, seed + 13 * i)
        if graph == "grid2d":
            deg = torch.bincount(u, minlength=nodes) + torch.bincount(v, minlength=nodes)
            excess = (1e-3 * UNIT * deg.to(torch.float64)).to(torch.int64)
        out.append(((nodes, u, v, w, excess), int(rng.integers(1, case["k"] + 1))))
    return out


# ---- the cases' states and passes ----

class _State:
    """Library objects and vectors of one case, released in order."""

    def __init__(self):
        self.owned = []

    def own(self, o):
        self.owned.append(o)
        return o

    def __del__(self):
        for o in reversed(self.owned):
            o.close()


def prepare(case, seed):
    s = _State()
    s.case, path, k = case, case["path"], case.get("k", 1)
    if path == "instances":
        made = _instances(case, seed)
        s.eng = s.own(native.Engine(0))
        facs, ops, s.nrhs = [], [], np.array([c for _, c in made], np.int32)
        for i, (graph, _) in enumerate(made):
            ptr, idx, vals = operator_of(*graph)
            f = factor_of(*graph, seed + i)
            mat = Matrix(n=graph[0], colptr=ptr.cpu().numpy(), rowidx=idx.cpu().numpy(), vals=vals.cpu().numpy())
            facs.append(s.own(native.DeviceFactor(s.eng, f, precision=PRECISION[case["precision"]])))
            ops.append(s.own(native.DeviceOperator(s.eng, mat, f.perm)))
        s.batch = s.own(native.Batch(s.eng, facs, ops, k))
        s.B = torch.zeros(s.batch.n_total * k, dtype=torch.float64, device=DEV)
        for i, (graph, c) in enumerate(made):
            base, n = k * int(s.batch.offsets[i]), graph[0]
            s.B[base: base + c * n] = _rhs(n, c, seed + i, False).reshape(-1)
        s.X = torch.zeros_like(s.B)
        return s
    mat, fac, _ = system(case["graph"], case["size"], seed)
    m = fac.m
    if path == "lanes":
        s.lanes = s.own(Lanes(mat, fac, k, lanes=case["lanes"]))
        s.B = [_rhs(mat.n, k, seed + j, not fac.sddm).reshape(-1) for j in range(case["lanes"])]
        s.X = [torch.zeros_like(b) for b in s.B]
        s.nrhs = np.array([k], np.int32)
        torch.cuda.synchronize()
        return s
    s.eng = s.own(native.Engine(0))
    count = case.get("count", k)
    if path == "admit":
        s.mat, s.fac = mat, fac
    else:
        s.factor = s.own(native.DeviceFactor(s.eng, fac, precision=PRECISION[case["precision"]]))
        if path not in ("sweep", "apply"):
            s.op = s.own(native.DeviceOperator(s.eng, mat, fac.perm))
    if path == "sweep":
        s.x = torch.randn((m, k), generator=_gen(seed + 990), dtype=torch.float64, device=DEV)
        s.z = torch.empty_like(s.x)
    elif path == "serve":
        s.batch = s.own(native.Batch(s.eng, [s.factor], [s.op], k))
        s.B = _rhs(mat.n, count, seed, not fac.sddm)
        s.X = torch.zeros_like(s.B)
    elif path in ("batch", "admit"):
        if path == "batch":
            s.batch = s.own(native.Batch(s.eng, [s.factor], [s.op], k))
        s.B = _rhs(mat.n, k, seed, not fac.sddm).reshape(-1)
        s.X = torch.zeros_like(s.B)
        s.nrhs = np.array([k], np.int32)
    else:
        s.b = _rhs(mat.n, 1, seed, not fac.sddm)[0]
        if path == "apply" and not case["host"]:
            s.x = s.b[:m].contiguous()
            s.z = torch.empty_like(s.x)
        elif case["host"]:
            s.b = s.b.cpu().numpy()
        else:
            s.x = torch.zeros_like(s.b)
    torch.cuda.synchronize()
    return s


def _serve(s):
    """Requests through the batch's slots in order: a finished slot is retired and given the next request."""
    bt, waiting, holds = s.batch, list(range(len(s.B))), {}
    torch.cuda.current_stream().synchronize()
    while waiting or holds:
        for slot in range(bt.k):
            if slot not in holds and waiting:
                holds[slot] = waiting.pop(0)
                bt.admit(slot, s.B[holds[slot]], tol=TOL, device_ptrs=True)
        done, _, _, _ = bt.slots(bt.step(4))
        for slot in [q for q in holds if done[q]]:
            bt.retire(slot, s.X[holds.pop(slot)], device_ptrs=True)
    s.eng.sync()
    return s.X


def run(s):
    case = s.case
    path = case["path"]
    if path == "apply":
        if case["host"]:
            s.factor.reset_apply_count()
            return s.factor.apply(s.b)[0]
        s.factor.sweep(0, s.x, s.z)
        s.factor.sweep(1, s.z, s.z)
        return s.z
    if path == "sweep":
        if case["precision"] == "fp64" or case["k"] == 1:
            s.factor.sweep_pair(s.x, s.z)
        else:
            s.factor.sweep_pair_multi(case["k"], s.x, s.z)
        return s.z
    if path == "pcg":
        if case["host"]:
            return native.pcg(s.eng, s.factor, s.op, s.b, tol=TOL)[0]
        native.pcg(s.eng, s.factor, s.op, s.b, s.x, tol=TOL, device_ptrs=True)
        return s.x
    if path == "lanes":
        s.lanes.solve_raw(s.B, s.X, s.nrhs, tol=TOL, flags=native.DEVICE_PTRS)
        return s.X
    if path == "serve":
        return _serve(s)
    if path == "admit":
        factor = native.DeviceFactor(s.eng, s.fac, precision=PRECISION[case["precision"]])
        op = native.DeviceOperator(s.eng, s.mat, s.fac.perm)
        batch = native.Batch(s.eng, [factor], [op], case["k"])
        batch.solve_raw(s.B, s.X, s.nrhs, tol=TOL, flags=native.DEVICE_PTRS)
        batch.close()
        op.close()
        factor.close()
        return s.X
    s.batch.solve_raw(s.B, s.X, s.nrhs, tol=TOL, flags=native.DEVICE_PTRS)
    return s.X


# ---- work, tolerances, 64-bit results ----

# per node: operator entries, stored factor entries; and a solve's iterations to 1e-8
SHAPE = {"grid2d": (5, 5.6, 45), "grid3d": (7, 8.0, 42), "regular": (7, 13.0, 24), "rmat": (30, 18.0, 13),
         "mixed": (6, 10.0, 30)}


def _nodes(case):
    if case["path"] == "instances":
        return case["count"] * case["size"] // 2
    graph, size = case["graph"], case["size"]
    if graph == "rmat":
        return int(0.7 * 2 ** size)
    return size ** {"grid2d": 2, "grid3d": 3, "regular": 1}[graph]


def work(case):
    """Bytes: the factor once per sweep, the operator once per product, each vector in and out of each step once."""
    n, (per_a, per_f, its), k = _nodes(case), SHAPE[case["graph"]], case.get("k", 1)
    path = case["path"]
    entry = 6 if case["precision"] == "fp16" else 8
    vec = 8 if case["precision"] == "fp64" else 4
    pair = 2 * n * (per_f * entry + 4) + 4 * n * k * vec
    pair_flops = 4.0 * n * per_f * k
    if path in ("apply", "sweep"):
        return {"bytes": pair, "flops": pair_flops}
    lanes = case.get("lanes", 1)
    cols = k * lanes if path != "serve" else case["count"]
    # one iteration: the product (p in, A p out), x, r and p updates, the two sweeps
    each = pair + n * (per_a * 12 + 4) + n * k * (16 + 88)
    passes = lanes if path != "serve" else case["count"] / k
    return {"bytes": its * each * passes, "flops": its * cols * n * (4.0 * per_f + 2.0 * per_a + 12)}


def tolerance(case):
    """About four times the distance from 64-bit results: sweeps 2e-15 (fp64, up to 1e-14 on large Laplacians) and
    1e-7 (fp32 sums, up to 5e-7); solves to a relative residual of 1e-8 stop within 5e-9 of the solution."""
    path = case["path"]
    if path in ("apply", "sweep"):
        return {"fp64": {"rel": 5e-14}, "fp32": {"rel": 2e-6}, "fp16": {"rel": 2e-6}}[case["precision"]]
    return {"rel": 2e-8}


def _stored(fac):
    """L11 after the drop, on the device: (ptr, row, value, column) without the diagonal, the diagonal, round bounds."""
    m = fac.m
    ptr = torch.from_numpy(fac.colptr.astype(np.int64)).to(DEV)
    row = torch.from_numpy(fac.rowidx.astype(np.int64)).to(DEV)
    val = torch.from_numpy(fac.vals).to(DEV).to(torch.float64)
    col = torch.repeat_interleave(torch.arange(fac.n, device=DEV), ptr[1:] - ptr[:-1])
    diag = val[ptr[:-1]][:m]
    off = (row != col) & (row < m) & (col < m)
    row, val, col = row[off], val[off], col[off]
    zero = torch.zeros(m, dtype=torch.float64, device=DEV)
    scale = zero.scatter_reduce(0, col, val.abs(), "amax")
    keep = (val.abs() >= DROP * scale[col]) & (val != 0)
    gone = zero.index_add(0, col[~keep], val[~keep])
    row, val, col = row[keep], val[keep], col[keep]
    held = zero.index_add(0, col, val.abs())
    per = torch.where(held > 0, gone / torch.where(held > 0, held, 1.0), 0.0)
    val = (val + per[col] * val.abs()).to(torch.float32).to(torch.float64)
    count = torch.bincount(col, minlength=m)
    ptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(count, 0)
    bounds = np.minimum(np.concatenate([[0], np.cumsum(fac.rounds.astype(np.int64))]), m).tolist()
    bounds += range(bounds[-1] + 1, m + 1)
    at = ptr[torch.tensor(bounds, device=DEV)].tolist()
    return row, val, col, diag, list(zip(bounds[:-1], bounds[1:], at[:-1], at[1:]))


def _pair(stored, x):
    """L^T \\ (L \\ x) in 64 bits, level by level; x is (m, k)."""
    row, val, col, diag, levels = stored
    y = x.clone()
    for lo, hi, a, b in levels:
        y[lo:hi] /= diag[lo:hi, None]
        if b > a:
            y.index_add_(0, row[a:b], val[a:b, None] * y[col[a:b]], alpha=-1.0)
    for lo, hi, a, b in reversed(levels):
        if b > a:
            part = torch.zeros((hi - lo, x.shape[1]), dtype=torch.float64, device=DEV)
            part.index_add_(0, col[a:b] - lo, val[a:b, None] * y[row[a:b]])
            y[lo:hi] -= part
        y[lo:hi] /= diag[lo:hi, None]
    return y


def _exact_solve(made, fac, b):
    """A \\ b in 64 bits (zero mean for a Laplacian): conjugate gradients to 1e-12, b is (k, n) in the original order."""
    ptr, idx, vals = operator_of(*made)
    a = torch.sparse_csr_tensor(ptr, idx, vals, size=(made[0], made[0]))
    perm = torch.from_numpy(fac.perm.astype(np.int64)).to(DEV)
    stored, m = _stored(fac), fac.m

    def precondition(r):
        z = torch.zeros_like(r)
        z[perm] = r
        z[:m] = _pair(stored, z[:m])
        z[m:] = 0
        z = z[perm]
        return z if fac.sddm else z - z.mean(0)

    r = b.t().contiguous()
    norm = r.norm(dim=0)
    x = torch.zeros_like(r)
    z = precondition(r)
    p, rz = z, (r * z).sum(0)
    for it in range(150):
        ap = a @ p
        step = rz / (p * ap).sum(0)
        x = x + step * p
        r = r - step * ap
        if it % 4 == 3 and bool((r.norm(dim=0) < 1e-12 * norm).all()):
            break
        z = precondition(r)
        new = (r * z).sum(0)
        p = z + (new / rz) * p
        rz = new
    if not fac.sddm:
        x = x - x.mean(0)
    return x.t().contiguous()


def exact(case, seed):
    path, k = case["path"], case.get("k", 1)
    if path == "instances":
        made = _instances(case, seed)
        out = torch.zeros(k * sum(g[0] for g, _ in made), dtype=torch.float64, device=DEV)
        base = 0
        for i, (graph, c) in enumerate(made):
            n = graph[0]
            x = _exact_solve(graph, factor_of(*graph, seed + i), _rhs(n, c, seed + i, False))
            out[base: base + c * n] = x.reshape(-1)
            base += k * n
        return out
    if _nodes(case) * case.get("count", k) > 40e6:
        return None
    mat, fac, made = system(case["graph"], case["size"], seed)
    if path == "sweep":
        return _pair(_stored(fac), torch.randn((fac.m, k), generator=_gen(seed + 990), dtype=torch.float64, device=DEV))
    if path == "apply":
        b = _rhs(mat.n, 1, seed, not fac.sddm)[0]
        if not case["host"]:
            return _pair(_stored(fac), b[:fac.m, None])[:, 0]
        perm = torch.from_numpy(fac.perm.astype(np.int64)).to(DEV)
        z = torch.zeros_like(b)
        z[perm] = b
        z[:fac.m] = _pair(_stored(fac), z[:fac.m, None])[:, 0]
        z[fac.m:] = 0
        return z[perm]
    x = _exact_solve(made, fac, _rhs(mat.n, case.get("count", k), seed, not fac.sddm))
    if path == "pcg":
        return x[0].cpu().numpy() if case["host"] else x[0]
    return x if path == "serve" else x.reshape(-1)
