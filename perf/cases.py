"""Cases of the performance measurement: what a user of the engine has it do,
through the package's public entry points.

Four kinds of work:

* ``chain``     a meta-path's matrix chain on resident leaf matrices
                (``Engine.chain``: estimate, order, products), the result
                copied to pinned host buffers as a result sink does it;
* ``estimate``  the RES estimates of a chain and its order, as the query
                server's admission and the estimator-only program ask for them;
* ``product``   one sparse product (``Engine.spgemm``) with path counts as
                values, optionally from host arrays (uploaded on each pass);
* ``batch``     many meta-paths over one graph replayed at once
                (``Batch.run``), whose results are counts and digests.

Graphs follow the configured workloads: the P/A/V citation graph and its
A-P-V-P-A chain, the U/I/C/T retail graph and its four chains, the X/Y/Z
stress graph and its twelve-matrix uint64 chain, the five-type schema of the
batched workload.  ``scale`` multiplies every vertex and edge count.  The
structure of a chain's or product's matrices is one draw for each case, so
that its result has one size; the seed relabels every vertex (any order of
rows and columns is as likely in real use) and draws the values.  Estimates
do not depend on labels: there the seed draws the graph itself.
"""
import math

import numpy as np
import torch

import resmcm_ari_gb300 as rg
from resmcm_ari_gb300 import synth, workloads

# chains as (relation, forward) leaves; relations by their end types
CHAINS = {
    "A-P-V-P-A": ("dblp", [("pa", False), ("pv", True), ("pv", False), ("pa", True)]),
    "I-T-I-C": ("retail", [("it", True), ("it", False), ("ic", True)]),
    "C-I-U-I-C": ("retail", [("ic", False), ("ui", False), ("ui", True), ("ic", True)]),
    "T-I-C-I-T": ("retail", [("it", False), ("ic", True), ("ic", False), ("it", True)]),
    "C-I-T-I-U-I-C": ("retail", [("ic", False), ("it", True), ("it", False), ("ui", False), ("ui", True),
                                 ("ic", True)]),
    "Z-Y-X-Y-X-Y-Z-Y-X-Y-X-Y-Z": ("stress", [("yz", False), ("xy", False), ("xy", True), ("xy", False), ("xy", True),
                                             ("yz", True)] * 2),
}
STRESS = "Z-Y-X-Y-X-Y-Z-Y-X-Y-X-Y-Z"


def listed():
    return [
        # one query on a graph of a few hundred vertices: launches and host round trips
        {"name": "apvpa-tiny", "kind": "chain", "path": "A-P-V-P-A", "scale": 0.01, "bits": 32},
        # the plain single-chain workload at its configured size (109M results)
        {"name": "apvpa-full", "kind": "chain", "path": "A-P-V-P-A", "scale": 1.0, "bits": 32},
        # the retail chains: items by tag and category, an ordinary size
        {"name": "itic-quarter", "kind": "chain", "path": "I-T-I-C", "scale": 0.25, "bits": 32},
        # categories joined through users, at the configured size
        {"name": "ciuic-full", "kind": "chain", "path": "C-I-U-I-C", "scale": 1.0, "bits": 32},
        # tag by tag through categories: every row of the result is full
        {"name": "ticit-quarter", "kind": "chain", "path": "T-I-C-I-T", "scale": 0.25, "bits": 32},
        # the longest retail chain at the configured size: counts outgrow uint32 on the way
        {"name": "citiuic-full", "kind": "chain", "path": "C-I-T-I-U-I-C", "scale": 1.0, "bits": 32},
        # twelve matrices in uint64, at the size the test suite runs
        {"name": "stress-u64", "kind": "chain", "path": STRESS, "scale": 0.01, "bits": 64},
        # admission of a long query on the full retail graph: estimates and order only
        {"name": "estimate-full", "kind": "estimate", "path": "C-I-T-I-U-I-C", "scale": 1.0},
        # one small product
        {"name": "product-small", "kind": "product", "rows": 1000, "inner": 900, "cols": 1100, "deg": 4.0, "skew": 0.0,
         "bits": 32, "host": False},
        # one wide product of odd sizes, short rows, uniform columns
        {"name": "product-odd", "kind": "product", "rows": 100003, "inner": 77777, "cols": 131071, "deg": 6.0,
         "skew": 0.0, "bits": 32, "host": False},
        # popular columns, uint64 counts, operands that arrive from the host with the call
        {"name": "product-skewed-u64", "kind": "product", "rows": 30011, "inner": 30011, "cols": 30011, "deg": 12.0,
         "skew": 1.1, "bits": 64, "host": True},
        # the batched workload: walks over the five-type schema, recorded once and replayed
        {"name": "batch-64", "kind": "batch", "count": 64, "scale": 0.04},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["chain", "chain", "chain", "chain", "estimate", "product", "product", "batch"])
    if kind in ("chain", "estimate"):
        path = rng.choice(sorted(CHAINS))
        # results of T-I-C-I-T are full squares of the tag count
        top = {"T-I-C-I-T": 0.35, "I-T-I-C": 0.5, STRESS: 0.01}.get(path, 1.0)
        low = {STRESS: 0.001, "A-P-V-P-A": 0.005}.get(path, 1.0 / 64)
        case = {"kind": kind, "path": path, "scale": round(_log(rng, low, top), 6)}
        if kind == "chain":
            case["bits"] = 64 if path == STRESS else 32
        return case
    if kind == "product":
        return {"kind": "product", "rows": int(_log(rng, 60, 200_000)), "inner": int(_log(rng, 60, 120_000)),
                "cols": int(_log(rng, 60, 200_000)), "deg": round(_log(rng, 2.0, 12.0), 2),
                "skew": rng.choice([0.0, 0.0, 0.8, 1.1]), "bits": rng.choice([32, 64]),
                "host": rng.random() < 0.3}
    return {"kind": "batch", "count": rng.randrange(8, 49), "scale": round(_log(rng, 0.01, 0.04), 5)}


# ---- inputs -----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _zipf(gen, k, s, n):
    """n 0-based ranks of a Zipf(s) law truncated to k."""
    cdf = torch.from_numpy(synth.zipf_cdf(k, s)).cuda()
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.searchsorted(cdf, u, right=True).clamp_(max=k - 1)


def _pairs(key, n_b):
    return key // n_b, key % n_b


def _chung_lu(gen, n_a, n_b, edges, s_a, s_b):
    """Distinct (a, b) pairs with Zipf degree laws on both sides (the law of
    ``synth.chung_lu``)."""
    ka = synth.zipf_truncation_for_mean(s_a, edges / n_a, max(2, n_b))
    kb = synth.zipf_truncation_for_mean(s_b, edges / n_b, max(2, n_a))
    deg = _zipf(gen, ka, s_a, n_a) + 1
    cdf_b = torch.cumsum(_zipf(gen, kb, s_b, n_b) + 1, 0).double()
    cdf_a = torch.cumsum(deg, 0).double()

    def pick(cdf, n):
        u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
        return torch.searchsorted(cdf, u, right=True).clamp_(max=cdf.numel() - 1)

    a = torch.repeat_interleave(torch.arange(n_a, device="cuda"), deg)
    key = torch.unique(a * n_b + pick(cdf_b, a.numel()))
    for _ in range(4):
        short = edges - key.numel()
        if short <= 0:
            break
        extra = int(short * 1.2) + 16
        key = torch.unique(torch.cat([key, pick(cdf_a, extra) * n_b + pick(cdf_b, extra)]))
    if key.numel() > edges:
        key = key[torch.randperm(key.numel(), generator=gen, device="cuda")[:edges]]
    return _pairs(key, n_b)


def _relations(graph, scale, gen):
    """{relation: (source ids, destination ids, sources, destinations)}"""
    def sc(x):
        return max(2, int(round(x * scale)))

    if graph == "dblp":
        n_a, n_p, n_v = sc(30_000), sc(60_000), max(2, int(round(50 * math.sqrt(scale))))
        cnt = torch.randint(1, 6, (n_p,), generator=gen, device="cuda")
        p = torch.repeat_interleave(torch.arange(n_p, device="cuda"), cnt)
        pa = _pairs(torch.unique(p * n_a + _zipf(gen, n_a, 1.1, p.numel())), n_a)
        return {"pa": pa + (n_p, n_a), "pv": (torch.arange(n_p, device="cuda"), _zipf(gen, n_v, 1.2, n_p), n_p, n_v)}
    if graph == "retail":
        n_u, n_i, n_c, n_t = sc(1_000_000), sc(300_000), sc(2_000), sc(20_000)
        ui = _chung_lu(gen, n_u, n_i, sc(20_000_000), 1.7, 1.3)
        # the other relations do not follow the items' popularity
        pi = torch.randperm(n_i, generator=gen, device="cuda")
        items = torch.arange(n_i, device="cuda")
        cnt = torch.randint(5, 16, (n_i,), generator=gen, device="cuda")
        src = torch.repeat_interleave(items, cnt)
        it = _pairs(torch.unique(src * n_t + torch.randint(0, n_t, (src.numel(),), generator=gen, device="cuda")), n_t)
        return {"ui": (ui[0], pi[ui[1]], n_u, n_i), "ic": (items, _zipf(gen, n_c, 1.1, n_i), n_i, n_c),
                "it": it + (n_i, n_t)}
    n_x, n_y, n_z = sc(5_000_000), sc(5_000_000), sc(100_000)
    x, y = _chung_lu(gen, n_x, n_y, sc(60_000_000), 1.6, 1.6)
    cnt = torch.randint(1, 5, (n_y,), generator=gen, device="cuda")
    src = torch.repeat_interleave(torch.arange(n_y, device="cuda"), cnt)
    yz = _pairs(torch.unique(src * n_z + torch.randint(0, n_z, (src.numel(),), generator=gen, device="cuda")), n_z)
    py = torch.randperm(n_y, generator=gen, device="cuda")   # nor these the degrees of Y
    return {"xy": (x, py[y], n_x, n_y), "yz": yz + (n_y, n_z)}


def _csr(src, dst, rows, cols):
    key = torch.sort(src * cols + dst)[0]
    rowptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(key // cols, minlength=rows), 0)
    return rowptr, (key % cols).int(), cols


def _leaves(case, seed):
    """The chain's leaf matrices, each distinct one once, and their order."""
    graph, path = CHAINS[case["path"]]
    rel = _relations(graph, case["scale"], _gen(seed if case["kind"] == "estimate" else 1))
    gen = _gen(seed)
    labels = {}
    for name, (_, _, ns, nd) in rel.items():
        for t, n in zip(name, (ns, nd)):
            if t not in labels:
                labels[t] = torch.randperm(n, generator=gen, device="cuda")
    out = {}
    for name, fwd in path:
        if (name, fwd) not in out:
            s, d, ns, nd = rel[name]
            s, d = labels[name[0]][s], labels[name[1]][d]
            out[name, fwd] = _csr(s, d, ns, nd) if fwd else _csr(d, s, nd, ns)
    return out, path


def _entries(gen, rows, cols, deg, skew):
    """Distinct entries of a matrix with about ``deg`` a row; ``skew`` > 0
    draws its columns from a Zipf law."""
    cnt = torch.randint(0, int(2 * deg) + 1, (rows,), generator=gen, device="cuda")
    r = torch.repeat_interleave(torch.arange(rows, device="cuda"), cnt)
    if skew > 0:
        c = torch.randperm(cols, generator=gen, device="cuda")[_zipf(gen, cols, skew, r.numel())]
    else:
        c = torch.randint(0, cols, (r.numel(),), generator=gen, device="cuda")
    return _pairs(torch.unique(r * cols + c), cols)


def _operands(case, seed):
    """Both operands of a product: (row pointers, columns, column count, values)."""
    gen, fixed = _gen(seed), _gen(1)
    dims = (case["rows"], case["inner"], case["cols"])
    labels = [torch.randperm(n, generator=gen, device="cuda") for n in dims]
    out = []
    for k in (0, 1):
        r, c = _entries(fixed, dims[k], dims[k + 1], case["deg"], case["skew"])
        rowptr, col, cols = _csr(labels[k][r], labels[k + 1][c], dims[k], dims[k + 1])
        val = torch.randint(1, 100, (col.numel(),), generator=gen, device="cuda", dtype=torch.int64)
        out.append((rowptr, col, cols, val if case["bits"] == 64 else val.int()))
    return out


_engine = None


def _eng():
    """The program's one engine."""
    global _engine
    if _engine is None:
        _engine = rg.Engine(device=0)
    return _engine


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _upload(rowptr, col, cols, val, bits):
    """val None: every count is one."""
    return _eng().upload_ptr(rowptr.data_ptr(), col.data_ptr(), rowptr.numel() - 1, cols,
                             0 if val is None else val.data_ptr(), rg.VAL_U64 if bits == 64 else rg.VAL_U32)


def prepare(case, seed):
    if case["kind"] in ("chain", "estimate"):
        made, path = _leaves(case, seed)
        mats = {}
        for k, (rowptr, col, cols) in made.items():
            mats[k] = _upload(_pinned(rowptr), _pinned(col), cols, None, case.get("bits", 32))
        return {"kind": case["kind"], "chain": [mats[k] for k in path]}
    if case["kind"] == "product":
        ops = []
        for rowptr, col, cols, val in _operands(case, seed):
            host = (_pinned(rowptr), _pinned(col), cols, _pinned(val), case["bits"])
            ops.append(host if case["host"] else _upload(*host))
        return {"kind": "product", "host": case["host"], "ops": ops}
    g = workloads.batch_graph(scale=case["scale"])
    eng = _eng()
    hg = rg.HeteroGraph.from_synthetic(eng, g)
    # walks short enough that no count outgrows 64 bits
    paths = workloads.batch_chains(eng, hg, g, count=case["count"], seed=int(seed), lengths=(2, 6))
    return {"kind": "batch", "graph": hg, "batch": eng.batch(hg, paths, fused=True)}


def _sink(m):
    """The result in pinned host buffers: row pointers, columns, counts."""
    eng = _eng()
    rows, _ = m.shape
    nnz = m.nnz
    rowptr = torch.empty(rows + 1, dtype=torch.int64, pin_memory=True)
    col = torch.empty(max(nnz, 1), dtype=torch.int32, pin_memory=True)
    val = torch.empty(max(nnz, 1), dtype=torch.int64 if m.valtype == rg.VAL_U64 else torch.int32, pin_memory=True)
    eng.download_async(m, rowptr.data_ptr(), col.data_ptr(), val.data_ptr())
    eng.transfers_wait()
    m.free()
    return {"rowptr": rowptr, "col": col[:nnz], "val": val[:nnz]}


def run(state):
    eng = _eng()
    if state["kind"] == "chain":
        m, _, _ = eng.chain(state["chain"])
        return _sink(m)
    if state["kind"] == "estimate":
        c = eng.estimate(state["chain"])
        split, cost, pairs = eng.order(c)
        return {"c": c, "split": split, "cost": cost, "pairs": pairs}
    if state["kind"] == "product":
        a, b = state["ops"]
        if state["host"]:
            a, b = _upload(*a), _upload(*b)
        return _sink(eng.spgemm(a, b))
    nnz, digest, _ = state["batch"].run()
    return {"nnz": nnz, "digest": digest.view(np.int64)}


# ---- what a pass cannot do without --------------------------------------------

def _csr_bytes(rowptr, col, vbytes):
    return 8 * rowptr.numel() + (4 + vbytes) * col.numel()


def work(case):
    """Inputs read once and results written once (row pointers 8 bytes,
    columns 4, counts 4 or 8; leaves hold no counts but ones); two operations
    a multiply-add of the chosen order."""
    if case["kind"] in ("chain", "estimate"):
        made, path = _leaves(case, 0)
        read = sum(_csr_bytes(rp, col, 0) for rp, col, _ in made.values())
        if case["kind"] == "estimate":
            L = len(path)
            # one multiply a leaf entry and target, the subtraction a row and target
            ops = sum(made[k][1].numel() * (L - 1 - i) + made[k][0].numel() * (L - i) for i, k in enumerate(path))
            return {"bytes": read + 8 * L * L, "flops": ops}
        del made
        m, t, _ = _eng().chain(prepare(case, 0)["chain"])
        return {"bytes": read + 8 * (m.shape[0] + 1) + (12 if m.valtype == rg.VAL_U64 else 8) * m.nnz,
                "flops": 2 * t["flops"]}
    if case["kind"] == "product":
        a, b = _operands(case, 0)
        v = case["bits"] // 8
        muls = int((b[0][1:] - b[0][:-1])[a[1].long()].sum())
        st = prepare(case, 0)
        nnz = run(st)["col"].numel()
        return {"bytes": _csr_bytes(a[0], a[1], v) + _csr_bytes(b[0], b[1], v) + 8 * (case["rows"] + 1) + (4 + v) * nnz,
                "flops": 2 * muls}
    # a batch's results stay on the device, only counts and digests leave it:
    # the entries of its results, 8 bytes each, are formed and digested
    st = prepare(case, 0)
    nnz = int(run(st)["nnz"].sum())
    return {"bytes": 8 * nnz + 16 * case["count"], "flops": 2 * nnz}


# ---- 64-bit values of the computed numbers ---------------------------------------

def exact(case, seed):
    """The estimates and the order's cost in float64 (products of the factors
    as sums of logarithms, so that small densities keep their digits); the
    other kinds return whole numbers."""
    if case["kind"] != "estimate":
        return None
    made, path = _leaves(case, seed)
    L = len(path)
    dims = [made[k][2] for k in path]
    c = torch.zeros(L, L, dtype=torch.float64)
    after = {}                                   # target -> densities of the next level's rows
    for i in range(L - 1, -1, -1):
        rowptr, col, cols = made[path[i]]
        lens = rowptr[1:] - rowptr[:-1]
        idx = col.long()
        now = {i: (lens.double() / cols).clamp_(max=1.0)}
        for j, r in after.items():
            t = torch.segment_reduce(torch.log1p(-r)[idx], "sum", lengths=lens, initial=0.0)
            now[j] = -torch.expm1(t)
            c[i, j] = float(now[j].sum()) * dims[j]
        after = now
    c = c.numpy()
    cost = np.zeros((L, L))
    for n in range(1, L):
        for i in range(L - n):
            j = i + n
            cost[i, j] = min(cost[i, k] + cost[k + 1, j] + ((c[i, k] + c[k + 1, j]) + c[i, j]) for k in range(i, j))
    return {"c": c, "split": None, "cost": cost, "pairs": None}
