"""What a program does with the matcher, as cases that can be timed and compared.

Five kinds of call, each through the package's public entry points:

* ``match``: one pattern against a prepared data graph (``Plan.run``);
* ``batch``: several patterns of uneven size against one data graph (``Batch.run``);
* ``grad``: a recorded match and its four feature gradients
  (``Plan.record`` and ``Plan.backward``);
* ``host``: host arrays in, host mu out (``match_host``), the whole program
  between reading the graph files and writing mu.

Graphs are R-MAT (a = .57, b = c = .19, duplicates and self-loops removed) or
uniform random, features N(0, 1); patterns are planted: connected, on vertices
drawn by degree, their edges added to the data graph, features those of the
planted elements plus N(0, 0.05^2).
"""
import math

import torch

from application_classification_gb300 import matcher
from application_classification_gb300.graph import Graph

NOISE = 0.05


def listed():
    def case(name, kind, precision, graph, n, factor, pn, pe, **more):
        c = dict(name=name, kind=kind, precision=precision, graph=graph, n=n, factor=factor, pn=pn,
                 pe=pe, kv=13, ke=17, cnull=False, patterns=1)
        c.update(more)
        return c

    return [
        # the small uniform graph of the reference's own tests, in both precisions:
        # a call of many short kernels, as a service answers small queries
        case("er1k_fp64", "match", "fp64", "er", 1000, 20, 10, 20),
        case("er1k_mixed", "match", "mixed", "er", 1000, 20, 10, 20),
        # the reference's GPU size
        case("rmat18_fp64", "match", "fp64", "rmat", 1 << 18, 16, 16, 32),
        case("rmat18_mixed", "match", "mixed", "rmat", 1 << 18, 16, 16, 32),
        # a large match at the reference's arithmetic (the package's default precision)
        case("rmat20_fp64", "match", "fp64", "rmat", 1 << 20, 16, 32, 64),
        # the headline workload of the benchmark
        case("rmat22_mixed", "match", "mixed", "rmat", 1 << 22, 16, 32, 64),
        # odd sizes throughout, other feature widths, and the C-null option
        case("er_odd_cnull_fp64", "match", "fp64", "er", 30011, 17, 23, 45, kv=7, ke=31, cnull=True),
        # a pattern wider than 64 edges, most patterns of the many-pattern workload
        case("wide_mixed", "match", "mixed", "rmat", 1 << 18, 16, 40, 120),
        # patterns of 4 to 48 vertices with 2 to 4 edges per vertex, matched as one batch
        case("batch_mixed", "batch", "mixed", "rmat", 1 << 17, 16, 48, 192, patterns=12),
        # training: forward and backward of one match
        case("grad_mixed", "grad", "mixed", "rmat", 1 << 16, 16, 12, 24),
        case("grad_fp64", "grad", "fp64", "rmat", 1 << 14, 16, 12, 24),
        # the whole program from host memory: uploads, preparation, match, mu back
        case("host_mixed", "host", "mixed", "rmat", 1 << 20, 16, 16, 32),
    ]


# edge x pattern-edge x iteration products that bound a drawn case's cost, by precision
CEILING = {"fp64": 2.5e10, "mixed": 6e10}


def draw(rng):
    kind = rng.choice(["match", "match", "match", "match", "batch", "grad", "host"])
    precision = rng.choice(["fp64", "mixed"])
    graph = "rmat" if kind == "grad" else rng.choice(["rmat", "rmat", "er"])
    factor = rng.randint(8 if kind == "grad" else 3, 20)
    low, high = (9, 16) if kind == "grad" else (9, 19) if kind == "batch" else (9, 21)
    n = int(round(2 ** rng.uniform(low, high)))
    if kind == "grad":
        # (patterns sparse or small enough that no edge's cost reaches mu have
        # edge gradients of rounding noise alone)
        pn = rng.randint(10, 24)
        pe = rng.randint(3 * pn // 2, 2 * pn)
    elif kind == "batch":
        pn, pe = 48, 192
    else:
        pn = rng.randint(4, 48)
        pe = rng.randint(pn, min(4 * pn, pn * (pn - 1)))
    patterns = rng.randint(3, 14) if kind == "batch" else 1
    kv, ke = (13, 17) if rng.random() < 0.6 else (rng.randint(2, 32), rng.randint(2, 32))
    cnull = kind in ("match", "batch") and rng.random() < 0.2
    cap = CEILING[precision] / (4 if kind == "grad" else 1)
    # a batch's patterns have about a third of the largest one's columns x iterations
    per_edge = pn * pe * (patterns / 3.0 if kind == "batch" else 1.0)
    while n > 512 and n * factor * per_edge > cap:
        n = int(n / 1.37)
    return dict(kind=kind, precision=precision, graph=graph, n=n, factor=factor, pn=pn, pe=pe, kv=kv,
                ke=ke, cnull=cnull, patterns=patterns)


# ------------------------------------------------------------------ inputs
def _pairs(case, count, g, dev):
    n = case["n"]
    if case["graph"] == "er":
        u = torch.randint(n, (count,), generator=g, device=dev)
        v = torch.randint(n, (count,), generator=g, device=dev)
    else:
        u = torch.zeros(count, dtype=torch.int64, device=dev)
        v = torch.zeros(count, dtype=torch.int64, device=dev)
        for _ in range(max(1, math.ceil(math.log2(n)))):
            r = torch.rand(count, generator=g, device=dev)
            u = 2 * u + (r >= 0.76)
            v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        u, v = u % n, v % n
    return (u * n + v)[u != v]


def _edges(case, g, dev):
    """n * factor distinct directed edges without self-loops, in random order."""
    n, m = case["n"], case["n"] * case["factor"]
    key = torch.unique(_pairs(case, m + m // 8 + 64, g, dev))
    while key.numel() < m:
        key = torch.unique(torch.cat([key, _pairs(case, m // 2 + 64, g, dev)]))
    key = key[torch.randperm(key.numel(), generator=g, device=dev)[:m]]
    return key // n, key % n


def _sizes(case, seed):
    """(vertices, edges) of each pattern."""
    if case["kind"] != "batch":
        return [(case["pn"], case["pe"])]
    g = torch.Generator().manual_seed(seed * 7919 + 5)
    out = []
    for _ in range(case["patterns"]):
        pn = int(torch.randint(4, case["pn"] + 1, (1,), generator=g))
        pe = int(torch.randint(2 * pn, 4 * pn + 1, (1,), generator=g))
        out.append((pn, min(pe, pn * (pn - 1), case["pe"])))
    return out


def _batch_sizes(case):
    """The batch's pattern sizes are the workload's, the same for every seed."""
    return _sizes(case, 3)


def _shape(pn, pe, g):
    """A connected pattern: a random tree, then distinct random pairs."""
    seen, out = set(), []
    for i in range(1, pn):
        j = int(torch.randint(i, (1,), generator=g))
        a, b = (i, j) if int(torch.randint(2, (1,), generator=g)) else (j, i)
        if len(out) < pe:
            seen.add((a, b))
            out.append((a, b))
    while len(out) < pe:
        a, b = (int(x) for x in torch.randint(pn, (2,), generator=g))
        if a != b and (a, b) not in seen:
            seen.add((a, b))
            out.append((a, b))
    return out


def _inputs(case, seed):
    """Device tensors of the data graph and the patterns, and the planted vertices."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    h = torch.Generator().manual_seed(seed)
    srcs, dsts = _edges(case, g, dev)
    ends, plans = torch.stack([srcs, dsts], 1).reshape(-1), []
    for pn, pe in _batch_sizes(case):
        # vertices by degree, as a random walk meets them (distinct)
        at = torch.randint(ends.numel(), (64 * pn,), generator=h).to(dev)
        some = ends[at].cpu().tolist() + torch.randperm(case["n"], generator=h)[:pn].tolist()
        verts = torch.tensor(list(dict.fromkeys(some))[:pn])
        plans.append((verts, torch.tensor(_shape(pn, pe, h))))
    del ends
    m0 = srcs.numel()
    srcs = torch.cat([srcs] + [v[e[:, 0]].to(dev) for v, e in plans])
    dsts = torch.cat([dsts] + [v[e[:, 1]].to(dev) for v, e in plans])
    f64 = dict(generator=g, device=dev, dtype=torch.float64)
    nf = torch.randn(case["n"], case["kv"], **f64)
    ef = torch.randn(srcs.numel(), case["ke"], **f64)
    data, pats, at = (nf, ef, srcs, dsts), [], m0
    for verts, e in plans:
        pnf = nf[verts.to(dev)] + NOISE * torch.randn(len(verts), case["kv"], **f64)
        pef = ef[at:at + len(e)] + NOISE * torch.randn(len(e), case["ke"], **f64)
        at += len(e)
        pats.append((pnf, pef, e[:, 0].to(dev).contiguous(), e[:, 1].to(dev).contiguous()))
    return data, pats, [v.to(dev) for v, _ in plans]


def _weight(case, planted, seed):
    """The gradient of the loss with respect to mu: the sum of mu (a log-probability)
    over the planted pairs, and a term on every pair as a dense loss has."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    w = 0.01 * torch.randn(case["n"], case["pn"], generator=g, device="cuda", dtype=torch.float64)
    w[planted, torch.arange(case["pn"], device="cuda")] += 1.0
    return w


def prepare(case, seed):
    data, pats, planted = _inputs(case, seed)
    kind, prec = case["kind"], case["precision"]
    if kind == "host":
        def host(t):
            a = [x.cpu().pin_memory() for x in t]
            g = Graph(a[0].numpy(), a[1].numpy(), a[2].numpy().view("u8"), a[3].numpy().view("u8"))
            return g, a
        d, keep = host(data)
        p, keep2 = host(pats[0])
        out = torch.empty((case["n"], case["pn"]), dtype=torch.float64).pin_memory()
        return dict(kind=kind, prec=prec, data=d, pattern=p, out=out.numpy(), keep=(keep, keep2, out))
    graph = matcher.DataGraph(matcher.DeviceGraph.from_tensors(*data))
    devs = [matcher.DeviceGraph.from_tensors(*p) for p in pats]
    if kind == "batch":
        b = matcher.Batch(graph, devs, prec, cnull=case["cnull"])
        return dict(kind=kind, batch=b, graph=graph)
    plan = matcher.Plan(graph, devs[0], prec, cnull=case["cnull"])
    state = dict(kind=kind, plan=plan, graph=graph)
    if kind == "grad":
        state["weight"] = _weight(case, planted[0], seed)
    return state


def run(state):
    kind = state["kind"]
    if kind == "match":
        return state["plan"].run()
    if kind == "batch":
        return state["batch"].run()
    if kind == "grad":
        mu = state["plan"].record()
        return [mu, *state["plan"].backward(state["weight"])]
    return matcher.match_host(state["data"], state["pattern"], state["prec"], out=state["out"])


def work(case):
    """The graph's and the patterns' arrays read once, mu (and the gradients)
    written once; the arithmetic of the cost matrices, and of each iteration its
    edge maxima (a difference and a comparison) and its vertex updates."""
    n, m = case["n"], case["n"] * case["factor"]
    kv, ke = case["kv"], case["ke"]
    inputs = 8 * (n * kv + m * ke + 2 * m)
    outputs, flops = 0, 0
    for pn, pe in _batch_sizes(case):
        inputs += 8 * (pn * kv + pe * ke + 2 * pe)
        outputs += 8 * n * pn
        once = 3 * (n * pn * kv + m * pe * ke) + 4 * m * pe
        each = 2 * m * pe + n * (14 * pe + 4 * pn)
        flops += once + pn * each
    if case["kind"] == "grad":
        outputs += 8 * (n * kv + m * ke)
        flops *= 3
    return {"bytes": inputs + outputs, "flops": flops}


# ------------------------------------------------------------------ in 64 bits
class _Segments:
    """Maxima over the edges of each vertex: vertices in classes of similar
    degree, each class one padded index matrix."""

    def __init__(self, nodes, n):
        dev = nodes.device
        order = torch.argsort(nodes, stable=True)
        deg = torch.bincount(nodes, minlength=n)
        off = torch.cumsum(deg, 0) - deg
        self.parts, place, used = [], torch.zeros(n, dtype=torch.int64, device=dev), 0
        order = torch.cat([order, torch.tensor([nodes.numel()], device=dev)])
        lo, hi = 1, 1
        while lo <= int(deg.max()):
            v = torch.nonzero((deg >= lo) & (deg <= hi)).reshape(-1)
            if v.numel():
                k = torch.arange(hi, device=dev)[None, :]
                at = torch.where(k < deg[v][:, None], off[v][:, None] + k, nodes.numel())
                self.parts.append(order[at])
                place[v] = used + torch.arange(v.numel(), device=dev)
                used += v.numel()
            lo, hi = hi + 1, 2 * hi
        place[deg == 0] = used
        self.place = place

    def max(self, x):
        """[n] maxima of the edge values x, -inf where a vertex has none."""
        x = torch.cat([x, x.new_full((1,), -math.inf)])
        out = [x[p].amax(1) for p in self.parts] + [x[-1:]]
        return torch.cat(out)[self.place]


def _match64(data, pat, iters, cnull):
    """mu [n][pn] in 64 bits, differentiable in the features.

    With L a log-softmax over the data axis, RE = VF[src] - L(dE) and
    FE = VR[src] - L(dE), the normalisers over the edges are sums over the
    vertices: logsumexp_e(VF[src_e] - dE_e) = logsumexp_v(VF_v + B_v) with
    B_v = log of the sum of exp(-dE) over v's out-edges."""
    nf, ef, srcs, dsts = data
    pnf, pef, ps, pd = pat
    # edges by destination, so that the maxima over in-edges read them in order
    ids = torch.argsort(dsts, stable=True)
    ef, srcs, dsts = ef[ids], srcs[ids], dsts[ids]
    n, m, pn, pe = nf.shape[0], ef.shape[0], pnf.shape[0], pef.shape[0]
    ps, pd = ps.tolist(), pd.tolist()
    lse = lambda x: torch.logsumexp(x, 0)  # noqa: E731
    out_seg, in_seg = _Segments(srcs, n), _Segments(dsts, n)

    def distance(x, y):
        d = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
        for k in range(x.shape[1]):
            d = d + (x[:, k] - y[k]) ** 2
        return torch.sqrt(d)

    dv = [distance(nf, pnf[p]) for p in range(pn)]
    cv = [d - lse(d) for d in dv]
    mu = [-d - lse(-d) for d in dv]
    de, near, b, r, f, null = [], [], [], [], [], []
    for q in range(pe):
        d = distance(ef, pef[q])
        # the first pn * n elements of the reference's [pe][m] buffers hold the
        # negated costs, the rest zeros
        start = torch.where(ids + q * m < pn * n, -d, torch.zeros_like(d))
        start = start - lse(start)
        r.append(torch.maximum(mu[pd[q]].amax(), out_seg.max(start)))
        f.append(torch.maximum(mu[ps[q]].amax(), in_seg.max(start)))
        total = torch.zeros_like(dv[0]).index_add(0, srcs, torch.exp(-d))
        some = total > 0
        b.append(torch.where(some, torch.log(torch.where(some, total, 1.0)), -math.inf))
        near.append(-out_seg.max(-d))
        de.append(d)
        if cnull:
            null.append(torch.maximum((pef[q] ** 2).sum().sqrt(), (d - lse(d)).amax()))
    null = torch.stack(null) if cnull else torch.zeros(pe, dtype=torch.float64, device=nf.device)
    null = null - lse(null) if cnull else null
    for _ in range(iters):
        raw = [-c for c in cv]
        nf_, nr_ = [], []
        for q in range(pe):
            vf, vr = mu[pd[q]] - f[q], mu[ps[q]] - r[q]
            nr_.append(torch.maximum(vf.amax() - null[q], vf - near[q] - lse(vf + b[q])))
            best = in_seg.max(vr[srcs] - de[q])
            nf_.append(torch.maximum(vr.amax() - null[q], best - lse(vr + b[q])))
        f, r = nf_, nr_
        for q in range(pe):
            raw[pd[q]] = raw[pd[q]] + f[q]
            raw[ps[q]] = raw[ps[q]] + r[q]
        mu = [x - lse(x) for x in raw]
    return torch.stack(mu, 1)


# the edge x column x iteration products that plain passes get through in time
_EXACT = 1.6e11


def exact(case, seed):
    sizes = _batch_sizes(case)
    m = case["n"] * case["factor"]
    if sum(m * pn * pe for pn, pe in sizes) > _EXACT:
        return None
    data, pats, planted = _inputs(case, seed)
    if case["kind"] == "grad":
        feats = [t.clone().requires_grad_() for t in (*data[:2], *pats[0][:2])]
        mu = _match64((feats[0], feats[1], *data[2:]), (feats[2], feats[3], *pats[0][2:]),
                      case["pn"], False)
        loss = (mu * _weight(case, planted[0], seed)).sum()
        grads = torch.autograd.grad(loss, feats)
        return [mu.detach(), *grads]
    with torch.no_grad():
        mus = [_match64(data, p, p[0].shape[0], case["cnull"]) for p in pats]
    if case["kind"] == "host":
        return mus[0].cpu().numpy()
    return mus if case["kind"] == "batch" else mus[0]
