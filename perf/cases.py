"""Performance cases: the work a program built on this package has it do.

Every case is one pass through public entry points on inputs made from a
seed.  The streams are sliding windows, as a program that follows a graph
runs them: a pass applies one batch of edge insertions (matched), then the
batch that takes the same edges out again, so a pass can be repeated on the
same state and always meets the same index.

Kinds
  engine   Engine: one query.  prepare() does what Stage 1 does: candidate
           vertices per query vertex (label, neighbour-label counts, then
           neighbour candidacy to a fix point), index keys over them, and the
           batch's ins / delta keys.  A pass is apply_batch (index update,
           delta lists, matching) and the index-only batch that retracts it.
           Outputs: the count, the per-edge counts, and (snapshot) the valid
           bits and the whole index.
  multi    MultiQuery: registered queries over one shared index.  A pass is an
           insertion batch (positive matches) and a deletion batch (negative
           matches).  prepare() runs one warm-up window, where the autotuner
           sets the plans, as a serving program does before it opens.
  serve    Server: the same through the serving loop's threads: a burst of
           batches of mixed sizes, then the batches that retract them, all
           submitted at once and collected in order.
  gpma     Gpma: a batch update of the packed-memory-array layout, the
           contents read back per direction, and the reverse update.
  flat     cgb_merge_keys_noalloc: edits merged into a flat sorted key array
           in device memory.

Stage 1 itself (Producer) reads files once, forward only, so it cannot be run
as a repeatable pass; its outputs are made in prepare().
"""
import ctypes
import math

import numpy as np
import torch

from cgbdsm_b200 import Engine, Gpma, MultiQuery, Server, load_library
from cgbdsm_b200.engine import FLAG_VALID_BITS
from cgbdsm_b200.queryset import load as load_queries
from cgbdsm_b200.workloads import GraphData, WorkloadSpec

RMAT = (0.57, 0.19, 0.19)

# Patterns of the package's own configurations (labels, edges), as their
# generator samples them, beside the stored query sets "c2:<i>" and "c3:<i>".
PATTERNS = {
    # R-MAT 1M/10M, 16 labels, 9-vertex dense
    "c2": ([0, 0, 7, 0, 11, 13, 1, 12, 7],
           [(0, 1), (1, 2), (1, 3), (1, 4), (1, 5), (1, 6), (1, 7), (1, 8), (3, 4), (3, 5), (3, 7), (3, 8), (4, 5),
            (4, 7), (5, 7)]),
    # R-MAT 4M/34M, 32 labels, 7-vertex tree and sparse
    "c3_tree": ([0, 23, 25, 6, 14, 2, 1], [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (5, 6)]),
    "c3_sparse": ([7, 6, 2, 0, 19, 10, 6], [(0, 1), (0, 2), (1, 3), (1, 4), (1, 5), (1, 6), (5, 6)]),
    # ER 3k/45k, 3 labels, 6-vertex sparse
    "er_sparse": ([2, 0, 0, 2, 0, 1], [(0, 1), (0, 2), (0, 3), (0, 4), (0, 5), (2, 3)]),
    # ER 3k/30k, 3 labels, 5-vertex tree
    "er_tree": ([1, 1, 1, 0, 2], [(0, 1), (1, 2), (2, 3), (3, 4)]),
    # ER 3k/30k, 12 labels, 6-vertex tree
    "er_path": ([1, 9, 5, 8, 2, 10], [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5)]),
}


def listed():
    return [
        # the smallest single-query call: batches of 1,000 on ER 10k/50k (latency)
        {"name": "er_tree_1k", "kind": "engine", "pattern": "er_tree", "rmat": False, "n": 10_000, "m": 50_000,
         "labels": 3, "zipf": 0.0, "label_seed": 132, "batch": 1_000, "device": False, "snapshot": False},
        # a checked run on a small graph: valid bits kept, masks and index read back
        {"name": "er_sparse_snapshot", "kind": "engine", "pattern": "er_sparse", "rmat": False, "n": 3_001,
         "m": 45_003, "labels": 3, "zipf": 0.0, "label_seed": 122, "batch": 751, "device": False, "snapshot": True},
        # an ordinary call at ragged sizes: a sparse pattern on a middle-sized power-law graph
        {"name": "rmat_sparse_8k", "kind": "engine", "pattern": "c2:30", "rmat": True, "n": 100_003, "m": 1_000_033,
         "labels": 16, "zipf": 1.2, "label_seed": 22, "batch": 8_191, "device": False, "snapshot": False},
        # the dense configuration: R-MAT 1M/10M, 9 vertices, batches of 100,000
        {"name": "rmat_dense_100k", "kind": "engine", "pattern": "c2", "rmat": True, "n": 1_000_000, "m": 10_000_000,
         "labels": 16, "zipf": 1.2, "label_seed": 22, "batch": 100_000, "device": False, "snapshot": False},
        # the largest single-query configuration: R-MAT 4M/34M, batches of 1,000,000, keys resident on the device
        {"name": "rmat_tree_1m", "kind": "engine", "pattern": "c3_tree", "rmat": True, "n": 4_000_000,
         "m": 34_000_000, "labels": 32, "zipf": 1.0, "label_seed": 32, "batch": 1_000_000, "device": True,
         "snapshot": False},
        {"name": "rmat_sparse_1m", "kind": "engine", "pattern": "c3_sparse", "rmat": True, "n": 4_000_000,
         "m": 34_000_000, "labels": 32, "zipf": 1.0, "label_seed": 32, "batch": 1_000_000, "device": True,
         "snapshot": False},
        # the smallest multi-query call: four queries, a few edges per batch (latency)
        {"name": "multi_4_tiny", "kind": "multi", "set": "c2", "first": 32, "queries": 4, "n": 10_007, "m": 90_001,
         "labels": 16, "zipf": 1.2, "label_seed": 22, "batch": 37, "device": False},
        # the full query mix on a middle-sized graph
        {"name": "multi_64", "kind": "multi", "set": "c2", "first": 0, "queries": 64, "n": 200_000, "m": 2_000_000,
         "labels": 16, "zipf": 1.2, "label_seed": 22, "batch": 20_000, "device": False},
        # the serving mix on a large graph, edge pairs resident on the device
        {"name": "multi_16_large", "kind": "multi", "set": "c3", "first": 0, "queries": 16, "n": 2_000_000,
         "m": 17_000_000, "labels": 32, "zipf": 1.0, "label_seed": 32, "batch": 200_000, "device": True},
        # serving: a burst of mixed batches with eight queries live
        {"name": "serve_burst", "kind": "serve", "set": "c3", "first": 8, "queries": 8, "n": 100_000, "m": 850_000,
         "labels": 32, "zipf": 1.0, "label_seed": 32, "batch_lo": 50, "batch_hi": 5_000, "batches": 8},
        # the packed-memory-array layout, mixed update
        {"name": "gpma_100k", "kind": "gpma", "dirs": 12, "n": 150_001, "keys": 2_000_003, "ins": 100_003,
         "del": 99_991},
        # the allocation-free merge into one flat key array
        {"name": "flat_merge_200k", "kind": "flat", "dirs": 28, "n": 203_001, "keys": 8_000_005, "ins": 131_072,
         "del": 65_537},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine", "engine", "engine", "multi", "multi", "serve", "gpma", "flat"])
    if kind == "engine":
        family = rng.choice(["er", "rmat16", "rmat16", "rmat32"])
        if family == "er":
            pattern, labels, label_seed = rng.choice([("er_path", 12, 162), ("er_sparse", 3, 122), ("er_tree", 3, 132)])
            n = _log_uniform(rng, 2_000, 20_000)
            m = int(n * rng.uniform(4, 10))
            return {"kind": "engine", "pattern": pattern, "rmat": False, "n": n, "m": m, "labels": labels,
                    "zipf": 0.0, "label_seed": label_seed, "batch": _log_uniform(rng, 200, m // 10),
                    "device": rng.random() < 0.3, "snapshot": rng.random() < 0.3}
        if family == "rmat16":
            n = _log_uniform(rng, 20_000, 600_000)
            m = int(n * rng.uniform(6, 10))
            return {"kind": "engine", "pattern": "c2:%d" % rng.randrange(64), "rmat": True, "n": n, "m": m,
                    "labels": 16, "zipf": 1.2, "label_seed": 22, "batch": _log_uniform(rng, 300, m // 80),
                    "device": rng.random() < 0.3, "snapshot": False}
        n = _log_uniform(rng, 200_000, 2_000_000)
        m = int(n * rng.uniform(6, 8.5))
        pattern = rng.choice(["c3_tree", "c3_sparse", "c3:%d" % rng.randrange(16)])
        return {"kind": "engine", "pattern": pattern, "rmat": True, "n": n, "m": m, "labels": 32, "zipf": 1.0,
                "label_seed": 32, "batch": _log_uniform(rng, 1_000, m // 80), "device": rng.random() < 0.5,
                "snapshot": False}
    if kind == "multi":
        name, labels, zipf, label_seed = rng.choice([("c2", 16, 1.2, 22), ("c3", 32, 1.0, 32)])
        n = _log_uniform(rng, 10_000, 200_000)
        m = int(n * rng.uniform(6, 10))
        count = _log_uniform(rng, 1, 32 if name == "c2" else 16)
        first = rng.randrange((64 if name == "c2" else 16) - count + 1)
        return {"kind": "multi", "set": name, "first": first, "queries": count, "n": n, "m": m, "labels": labels,
                "zipf": zipf, "label_seed": label_seed, "batch": _log_uniform(rng, 20, m // 100),
                "device": rng.random() < 0.3}
    if kind == "serve":
        n = _log_uniform(rng, 20_000, 100_000)
        count = rng.randrange(1, 9)
        return {"kind": "serve", "set": "c3", "first": rng.randrange(16 - count + 1), "queries": count, "n": n,
                "m": int(n * rng.uniform(6, 8.5)), "labels": 32, "zipf": 1.0, "label_seed": 32, "batch_lo": 20,
                "batch_hi": _log_uniform(rng, 200, 5_000), "batches": rng.randrange(3, 9)}
    n = _log_uniform(rng, 2_000, 200_000)
    dirs = rng.randrange(2, 31)
    most = dirs * n * n // 64  # keys are distinct (direction, vertex, vertex) triples
    if kind == "gpma":
        keys = _log_uniform(rng, 20_000, min(most, 2_000_000))
        return {"kind": "gpma", "dirs": dirs, "n": n, "keys": keys,
                "ins": _log_uniform(rng, 100, keys // 10), "del": _log_uniform(rng, 100, keys // 10)}
    keys = _log_uniform(rng, 20_000, min(most, 8_000_000))
    return {"kind": "flat", "dirs": dirs, "n": n, "keys": keys,
            "ins": _log_uniform(rng, 10, min(keys // 4, 150_000)),
            "del": _log_uniform(rng, 10, min(keys // 4, 100_000))}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _vertex_labels(case):
    """Labels of the vertices 0..n-1, as the package's generator draws them
    (the hubs of an R-MAT graph, its low ids, keep their labels over seeds)."""
    spec = WorkloadSpec("labels", 0, case["n"], 64, case["labels"], case["zipf"], 1, 1, 2, 2, 1, case["label_seed"],
                        3, 4)
    g = GraphData(spec)
    lab = g.labels.copy()
    g.close()
    return lab


def _edges(case, seed):
    """m distinct undirected edges without self-loops (uniform, or R-MAT), in
    random order: int64 tensors x, y on the device."""
    n, m = case["n"], case["m"]
    g = _gen(seed)
    scale = max(1, (n - 1).bit_length())
    a, b, c = RMAT
    have = None
    while have is None or have.numel() < m:
        need = int((m - (0 if have is None else have.numel())) * 1.3) + 4096
        if case.get("rmat", True):
            x = torch.zeros(need, dtype=torch.int64, device="cuda")
            y = torch.zeros(need, dtype=torch.int64, device="cuda")
            for _ in range(scale):
                r = torch.rand(need, device="cuda", generator=g)
                x = (x << 1) | (r >= a + b).long()
                y = (y << 1) | (((r >= a) & (r < a + b)) | (r >= a + b + c)).long()
        else:
            x = torch.randint(0, n, (need,), device="cuda", generator=g)
            y = torch.randint(0, n, (need,), device="cuda", generator=g)
        ok = (x < n) & (y < n) & (x != y)
        x, y = x[ok], y[ok]
        k = (torch.minimum(x, y) << 32) | torch.maximum(x, y)
        have = torch.unique(k if have is None else torch.cat([have, k]))
    order = torch.randperm(have.numel(), device="cuda", generator=g)[:m]
    k = have[order]
    return k >> 32, k & 0xFFFFFFFF


def _pattern(name):
    if name in PATTERNS:
        return PATTERNS[name]
    s, i = name.split(":")
    q = load_queries(s)[int(i)]
    return q["labels"], [tuple(e) for e in q["edges"]]


def _directions(qe):
    """(a, b) of every directed query edge, in index order."""
    nb = {}
    for a, b in qe:
        nb.setdefault(a, []).append(b)
        nb.setdefault(b, []).append(a)
    return [(a, b) for a in sorted(nb) for b in sorted(nb[a])]


def _candidates(lab, src, dst, ql, dirs):
    """Candidate bits [query vertex][data vertex] over the directed edges
    (src, dst): label and neighbour-label counts, then, to a fix point (at
    most four rounds), a candidate neighbour along every query edge."""
    n = lab.numel()
    need = {}
    for a, b in dirs:
        need.setdefault(a, {}).setdefault(ql[b], 0)
        need[a][ql[b]] += 1
    deg = {}
    for lb in set(ql):
        e = lab[dst] == lb
        deg[lb] = torch.bincount(src[e], minlength=n)
    cand = []
    for u, lb in enumerate(ql):
        c = lab == lb
        for l2, k in need[u].items():
            c = c & (deg[l2] >= k)
        cand.append(c)
    sub = []
    for a, b in dirs:
        e = cand[a][src] & cand[b][dst]
        sub.append((src[e], dst[e]))
    for _ in range(4):
        for (a, b), (s, d) in zip(dirs, sub):
            has = torch.zeros(n, dtype=torch.bool, device=lab.device)
            has[s[cand[b][d]]] = True
            cand[a] = cand[a] & has
    return cand


def _stage1(case, seed):
    """Keys of the initial index and of one batch (ins, delta), vertex count."""
    ql, qe = _pattern(case["pattern"])
    dirs = _directions(qe)
    lab = torch.from_numpy(_vertex_labels(case).astype(np.int64)).cuda()
    x, y = _edges(case, seed)
    old = case["m"] - case["batch"]
    src, dst = torch.cat([x, y]), torch.cat([y, x])
    used = torch.zeros(int(lab.max()) + 1, dtype=torch.bool, device="cuda")
    used[torch.tensor(ql, device="cuda")] = True
    is_new = torch.zeros(case["m"], dtype=torch.bool, device="cuda")
    is_new[old:] = True
    is_new = torch.cat([is_new, is_new])
    keep = used[lab[src]] & used[lab[dst]]
    src, dst, is_new = src[keep], dst[keep], is_new[keep]
    before = _candidates(lab, src[~is_new], dst[~is_new], ql, dirs)
    after = _candidates(lab, src, dst, ql, dirs)
    seen = torch.zeros(lab.numel(), dtype=torch.bool, device="cuda")
    for c in after:
        seen |= c
    cid = torch.cumsum(seen.long(), 0) - 1
    init, ins, delta = [], [], []
    for d, (a, b) in enumerate(dirs):
        now = after[a][src] & after[b][dst]
        was = before[a][src] & before[b][dst] & ~is_new
        top = (d << 59) if d < 16 else (d << 59) - (1 << 64)  # two's complement of the unsigned key
        key = (cid[src] << 32 | cid[dst]) + top
        init.append(key[was])
        ins.append(key[now & ~was & ~is_new])
        delta.append(key[now & is_new])
    host = [torch.cat(k).cpu().numpy().view(np.uint64) for k in (init, ins, delta)]
    return ql, qe, int(seen.sum()), host


def _pairs_of(x, y):
    return torch.stack([x, y], 1).cpu().numpy().astype(np.uint32)


def _on_device(a):
    return torch.from_numpy(a.view(np.int64 if a.dtype == np.uint64 else np.int32)).cuda()


def _flat_keys(case, seed):
    """Sorted distinct keys over dirs x n x n (a few long runs, many short
    ones), and disjoint edits: ins (mostly new) and del (mostly present)."""
    g = _gen(seed)
    total = case["keys"] + case["ins"]
    have = None
    while have is None or have.numel() < total:
        need = int(total * 1.3) + 1024
        d = torch.randint(0, case["dirs"], (need,), device="cuda", generator=g)
        u = (torch.rand(need, device="cuda", generator=g, dtype=torch.float64) ** 3 * case["n"]).long()
        v = torch.randint(0, case["n"], (need,), device="cuda", generator=g)
        k = d << 54 | u << 27 | v  # in key order
        have = torch.unique(k if have is None else torch.cat([have, k]))
    sel = torch.randperm(have.numel(), device="cuda", generator=g)[:total]
    ins, old = have[sel[:case["ins"]]], torch.sort(have[sel[case["ins"]:]]).values
    dele = old[torch.randperm(old.numel(), device="cuda", generator=g)[:case["del"]]]
    m27 = (1 << 27) - 1

    def ext(k):
        d = k >> 54
        top = torch.where(d < 16, d << 59, (d - 32) << 59)
        return top + ((k >> 27 & m27) << 32) + (k & m27)

    return [ext(k).cpu().numpy().view(np.uint64) for k in (old, ins, dele)]


# ---------------------------------------------------------------------------
# states and passes
# ---------------------------------------------------------------------------
def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "engine":
        ql, qe, dv, (init, ins, delta) = _stage1(case, seed)
        e = Engine(flags=FLAG_VALID_BITS if case["snapshot"] else 0)
        e.load_query(len(ql), qe, ql)
        e.build_index(init, dv)
        s.update(engine=e, dv=dv, ins=ins, delta=delta, gone=np.concatenate([ins, delta]),
                 none=np.zeros(0, dtype=np.uint64))
        if case["device"]:
            s.update(d_ins=_on_device(ins), d_delta=_on_device(delta), d_gone=_on_device(s["gone"]))
    elif kind in ("multi", "serve"):
        lab = _vertex_labels(case)
        x, y = _edges(case, seed)
        queries = load_queries(case["set"])[case["first"]:case["first"] + case["queries"]]
        if kind == "multi":
            old = case["m"] - case["batch"]
            m = MultiQuery()
            m.load_graph(lab, _pairs_of(x[:old], y[:old]))
            for q in queries:
                m.register(q["qv"], [tuple(e) for e in q["edges"]], q["labels"])
            batch = _pairs_of(x[old:], y[old:])
            m.apply_batch(ins=batch)  # the autotuner runs here
            m.apply_batch(dele=batch)
            s.update(multi=m, batch=batch)
            if case["device"]:
                s["d_batch"] = _on_device(batch)
        else:
            r = np.random.default_rng(seed)
            sizes = np.exp(r.uniform(math.log(case["batch_lo"]), math.log(case["batch_hi"]),
                                     case["batches"])).astype(np.int64)
            old = case["m"] - int(sizes.sum())
            srv = Server(lab, _pairs_of(x[:old], y[:old]))
            for q in queries:
                srv.wait(srv.submit_register(q["qv"], [tuple(e) for e in q["edges"]], q["labels"]))
            stream = _pairs_of(x[old:], y[old:])
            at = np.concatenate([[0], np.cumsum(sizes)])
            s.update(server=srv, batches=[stream[at[i]:at[i + 1]] for i in range(len(sizes))])
            largest = max(s["batches"], key=len)
            srv.wait(srv.submit_batch(ins=largest))  # the autotuner runs here
            srv.wait(srv.submit_batch(dele=largest))
    elif kind == "gpma":
        old, ins, dele = _flat_keys(case, seed)
        g = Gpma(case["dirs"])
        g.bulk_load(old)
        s.update(gpma=g, ins=ins, dele=dele)
    else:
        old, ins, dele = _flat_keys(case, seed)
        s.update(lib=load_library(), old=_on_device(old), ins=_on_device(ins), dele=_on_device(dele))
        s["out"] = torch.empty(len(old) + len(ins), dtype=torch.int64, device="cuda")
        s["out_n"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return s


def _signed(a):
    return a.copy().view(np.int64)


def _padded(a, length):
    out = np.zeros(max(length, len(a)), dtype=a.dtype)
    out[:len(a)] = a
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "engine":
        e, dv, none = state["engine"], state["dv"], state["none"]
        if case["device"]:
            i, d, g = state["d_ins"], state["d_delta"], state["d_gone"]
            count = e.apply_batch_device(dv, i.data_ptr(), i.numel(), 0, 0, d.data_ptr(), d.numel())
        else:
            count = e.apply_batch(dv, state["ins"], none, state["delta"])
        out = {"count": np.array([count], dtype=np.uint64).view(np.int64), "edges": _signed(e.edge_counts())}
        if case["snapshot"]:
            # padded to a length that the case alone decides
            bits, index = e.valid_bits()[0], e.read_index()
            ql, qe = _pattern(case["pattern"])
            out["bits"] = _padded(bits.view(np.int32), len(qe) * len(ql) * ((case["n"] + 31) // 32))
            out["index"] = _padded(index.view(np.int64), len(qe) * case["m"])
        if case["device"]:
            e.apply_batch_device(dv, 0, 0, g.data_ptr(), g.numel(), 0, 0)
        else:
            e.apply_batch(dv, none, state["gone"], none)
        return out
    if kind == "multi":
        m = state["multi"]
        if case["device"]:
            b = state["d_batch"]
            pos, _ = m.apply_batch_device(b.data_ptr(), b.shape[0])
            _, neg = m.apply_batch_device(0, 0, b.data_ptr(), b.shape[0])
        else:
            pos, _ = m.apply_batch(ins=state["batch"])
            _, neg = m.apply_batch(dele=state["batch"])
        return {"pos": pos.view(np.int64), "neg": neg.view(np.int64)}
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit_batch(ins=b) for b in state["batches"]]
        tickets += [srv.submit_batch(dele=b) for b in state["batches"]]
        got = [srv.wait(t) for t in tickets]
        return {"status": np.array([r["status"] for r in got], dtype=np.int64),
                "pos": np.stack([r["pos"] for r in got]).view(np.int64),
                "neg": np.stack([r["neg"] for r in got]).view(np.int64)}
    if kind == "gpma":
        g = state["gpma"]
        g.batch_update(state["ins"], state["dele"])
        out = [g.extract(d).view(np.int64) for d in range(case["dirs"])]
        g.batch_update(state["dele"], state["ins"])
        return {"contents": np.concatenate(out)}
    old, ins, dele, out, out_n = (state[k] for k in ("old", "ins", "dele", "out", "out_n"))
    st = state["lib"].cgb_merge_keys_noalloc(old.data_ptr(), old.numel(), ins.data_ptr(), ins.numel(),
                                             dele.data_ptr(), dele.numel(), case["n"], out.data_ptr(),
                                             out_n.data_ptr(),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st != 0:
        raise RuntimeError("cgb_merge_keys_noalloc: %d" % st)
    return {"keys": out[:int(out_n.item())]}


def work(case):
    kind = case["kind"]
    if kind == "engine":
        # the edges come in and go out again, as 8-byte keys of both
        # directions, each end's list read and written once per batch
        deg = 2.0 * case["m"] / case["n"]
        return {"bytes": case["batch"] * 2 * 2 * (8 + 8 * min(deg, 16.0)), "flops": 0}
    if kind == "multi":
        deg = 2.0 * case["m"] / case["n"]
        return {"bytes": case["batch"] * 2 * (8 + 2 * 8 * deg) + 16 * 256, "flops": 0}
    if kind == "serve":
        deg = 2.0 * case["m"] / case["n"]
        mean = (case["batch_hi"] - case["batch_lo"]) / math.log(case["batch_hi"] / case["batch_lo"])
        return {"bytes": case["batches"] * 2 * (mean * (8 + 2 * 8 * deg) + 16 * 256), "flops": 0}
    if kind == "gpma":
        return {"bytes": 8 * (2 * (case["ins"] + case["del"]) + case["keys"] + case["ins"] - case["del"]), "flops": 0}
    return {"bytes": 8 * (2 * case["keys"] + 2 * case["ins"]), "flops": 0}


def tolerance(case):
    return "exact"  # counts, bit masks and keys: whole numbers throughout


def exact(case, seed):
    """The key sets by plain numpy; an enumeration of the matches by plain
    numpy takes far too long (10^6 to 10^16 per batch)."""
    if case["kind"] not in ("gpma", "flat"):
        return None
    old, ins, dele = _flat_keys(case, seed)
    keys = np.setdiff1d(np.concatenate([old, ins]), dele)
    if case["kind"] == "flat":
        return {"keys": keys.view(np.int64)}
    return {"contents": (keys & np.uint64((1 << 59) - 1)).view(np.int64)}
