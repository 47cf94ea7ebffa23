"""The matcher's and the index update's paths at the sizes where they can go
wrong, against the C restatement (oracle/oracle.c) and plain set arithmetic.

Exact equality throughout: counts, per-edge counts and keys are whole numbers.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from cgbdsm_b200 import Engine, Gpma, MultiQuery
from cgbdsm_b200.engine import FLAG_FORCE_SPLIT, FLAG_MASK_PRUNE, FLAG_NO_STEAL, FLAG_VALID_BITS, CgbError
from oracle import bind


def _key(d, u, v):
    return (np.uint64(d) << np.uint64(59)) | (np.asarray(u, np.uint64) << np.uint64(32)) | np.asarray(v, np.uint64)


def _empty():
    return np.zeros(0, np.uint64)


# ---------------------------------------------------------------------------
# index update: run lengths around the lane / warp / tile limits
# ---------------------------------------------------------------------------
# merged lengths at the edges of the three merges (32; 512) and of a tile
# (2,816 entries), one and several tiles
RUNS = [1, 31, 32, 33, 511, 512, 513, 2815, 2816, 2817, 5632, 5633, 9000]


@pytest.mark.gpu
@pytest.mark.parametrize("edits", [1, 2, 33, 700])
def test_run_lengths_at_the_merge_limits(edits):
    """One run per length in RUNS, updated by adds (new, present and repeated),
    removes (present and absent) and keys both added and removed; the index
    equals (index + ins) - del.  Twice, so that the second update also merges
    runs the first one wrote."""
    rng = np.random.default_rng(edits)
    dv = 20000
    old = {u: rng.choice(dv, n, replace=False) for u, n in enumerate(RUNS)}
    init = np.array([_key(0, u, v) for u, vs in old.items() for v in vs], dtype=np.uint64)
    eng = Engine()
    eng.load_query(2, [(0, 1)], [0, 1])
    eng.build_index(init, dv)
    state = np.unique(init)
    for _ in range(2):
        ins, dele = [], []
        for u, vs in old.items():
            for v in rng.integers(0, dv, edits):
                ins.append(_key(0, u, v))
            for v in rng.choice(vs, min(len(vs), edits // 2 + 1)):
                dele.append(_key(0, u, v))
                ins.append(_key(0, u, v))  # removed although also added
            ins.append(ins[-1])
            dele.append(_key(0, u, int(rng.integers(0, dv))))
        ins, dele = np.array(ins, np.uint64), np.array(dele, np.uint64)
        rng.shuffle(ins)
        rng.shuffle(dele)
        eng.apply_batch(dv, ins, dele, _empty())
        state = np.setdiff1d(np.union1d(state, ins), dele)
        assert np.array_equal(np.sort(eng.read_index()), state)
    eng.close()


@pytest.mark.gpu
def test_delta_merge_back_and_growing_ids():
    """The sorted delta kept for the merge-back is packed again when the vertex
    ids outgrow its bits (20 -> 5,000 vertices between batches)."""
    eng = Engine()
    eng.load_query(2, [(0, 1)], [0, 1])
    eng.build_index(np.array([_key(0, 1, 2), _key(1, 2, 1)], np.uint64), 20)
    delta = np.array([_key(0, 3, 4), _key(1, 4, 3), _key(0, 3, 4), _key(1, 4, 3)], np.uint64)  # repeated entries
    eng.apply_batch(20, _empty(), _empty(), delta)
    ins = np.array([_key(0, 4999, 17), _key(1, 17, 4999)], np.uint64)
    eng.apply_batch(5000, ins, _empty(), _empty())
    want = np.unique(np.concatenate([np.array([_key(0, 1, 2), _key(1, 2, 1)], np.uint64), delta, ins]))
    assert np.array_equal(np.sort(eng.read_index()), want)
    eng.close()


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, FLAG_VALID_BITS, FLAG_MASK_PRUNE])
@pytest.mark.parametrize("bad", [(3, 5, 6), (31, 5, 6), (0, 64, 6), (1, 5, 64), (31, (1 << 27) - 1, (1 << 27) - 1)])
def test_out_of_range_delta_key_is_rejected(flags, bad):
    """A delta key whose direction or vertex is out of range rejects the batch
    (also where valid bits are computed, whose pass over the delta meets the
    key's marker); the engine then matches the next batch as ever."""
    eng = Engine(flags=flags)
    eng.load_query(2, [(0, 1)], [0, 1])
    eng.build_index(np.array([_key(0, 1, 2), _key(1, 2, 1)], np.uint64), 64)
    good = [_key(0, 3, 4), _key(1, 4, 3), _key(0, 63, 62), _key(1, 62, 63)]
    with pytest.raises(CgbError, match="out of range"):
        eng.apply_batch(64, _empty(), _empty(), np.array([*good, _key(*bad)], np.uint64))
    assert eng.apply_batch(64, _empty(), _empty(), np.array(good, np.uint64)) == 2
    eng.apply_batch(64, _empty(), _empty(), _empty())
    assert np.array_equal(np.sort(eng.read_index()), np.unique(np.array([_key(0, 1, 2), _key(1, 2, 1), *good], np.uint64)))
    eng.close()


@pytest.mark.gpu
def test_two_merges_of_a_batch_near_the_end_of_the_pool():
    """A deletion batch merges the pending insertions and then its own edits,
    both rewriting nearly every run.  In a pool that has room for either merge
    but not for both (one of these sizes, after some batches) no batch is lost:
    counts equal those of an engine whose pool is large."""
    rng = np.random.default_rng(11)
    hubs, leaves = 64, 8000
    lab = np.array([0] * hubs + [1] * leaves, np.uint32)
    pick = np.argsort(rng.random((leaves, hubs)), axis=1)[:, :12]  # distinct hubs of every leaf

    def edges(cols):
        return np.array([(pick[x, c], hubs + x) for x in range(leaves) for c in cols], np.uint32)

    engines = []
    for words in (0, *range(520_000, 1_000_000, 60_000)):
        m = MultiQuery(dfs_budget_ms=60000, pool_words=words)
        m.load_graph(lab, edges(range(8)))
        engines.append((m, m.register(3, [(0, 1), (1, 2)], [1, 0, 1])))
    batches = [edges([8 + i]) for i in range(4)]
    for b in batches:
        got = [[int(x) for x in (m.apply_batch(ins=b)[0][q], m.apply_batch(dele=b)[1][q])] for m, q in engines]
        assert got[0][0] == got[0][1] > 0 and all(g == got[0] for g in got)
    for m, _ in engines:
        m.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dv", [1000, 2_100_000, 5_000_000])
def test_reading_the_index_keeps_no_large_buffer(dv):
    """A read-back of an index whose run offsets (4 directions, 8 bytes a
    vertex) are beyond 64 MiB holds none of its memory afterwards."""
    import torch

    eng = Engine()
    eng.load_query(3, [(0, 1), (1, 2)], [0, 1, 2])
    keys = np.unique(np.array([_key(d, u, v) for d, u, v in [(0, 1, 2), (1, 2, 1), (3, dv - 1, 7), (2, 7, dv - 1)]], np.uint64))
    eng.build_index(keys, dv)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        assert np.array_equal(np.sort(eng.read_index()), keys)
    assert free - torch.cuda.mem_get_info()[0] <= 110 << 20  # kept: offsets up to 64 MiB and half as much again
    eng.close()


# ---------------------------------------------------------------------------
# seeds: how the launch's warps claim them
# ---------------------------------------------------------------------------
def test_seeds_are_claimed_by_whatever_part_of_the_grid_runs(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "seed_claim"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(root, "cgbdsm_b200", "csrc"),
                    os.path.join(root, "tests", "native", "seed_claim.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=300).stdout == "ok\n"


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, FLAG_NO_STEAL])
@pytest.mark.parametrize("blocks", [0, 1])
def test_seed_counts_around_the_grid(flags, blocks):
    """As many seeds as blocks and as warps of the grid (148 SMs, 4 or 1 blocks
    each, 8 warps), one fewer and one more; and several rounds of them.  Every
    seed (x, y) of the path 0-1-2 counts y's neighbours of label 2."""
    g = 148 * (blocks or 4)
    n = 20000
    rng = np.random.default_rng(g)
    out = rng.integers(0, 4, 100)  # neighbours of label 2 of the vertices [10000, 10100)
    qe, ql = [(0, 1), (1, 2)], [0, 1, 2]
    orc = bind.Oracle(3, qe)
    d = {(a, b): orc.L.orc_dir(orc.h, a, b) for x, y in qe for a, b in ((x, y), (y, x))}
    init = [k for y, c in enumerate(out) for z in range(c)
            for k in (_key(d[1, 2], 10000 + y, 11000 + z), _key(d[2, 1], 11000 + z, 10000 + y))]
    for seeds in (1, g - 1, g, g + 1, 2 * g + 1, 8 * g - 1, 8 * g, 8 * g + 1, min(3 * 8 * g + 5, 9999)):
        eng = Engine(flags=flags, dfs_blocks_per_sm=blocks)
        eng.load_query(3, qe, ql)
        eng.build_index(np.array(init, np.uint64), n)
        y = rng.integers(0, 100, seeds)
        delta = np.concatenate([_key(d[0, 1], np.arange(seeds), 10000 + y), _key(d[1, 0], 10000 + y, np.arange(seeds))])
        assert eng.apply_batch(n, _empty(), _empty(), delta) == out[y].sum()
        eng.close()


@pytest.mark.gpu
def test_engines_side_by_side_on_one_device():
    """Three engines fed by three threads at once, each with as many matcher
    blocks as an empty device holds: every batch ends, with its count."""
    import threading

    ql, qe = PATTERNS["shared"]
    rng = np.random.default_rng(12)
    n = 400
    lab, pairs = _graph(rng, n, max(ql) + 1, 120)
    rng.shuffle(pairs)
    k = len(pairs) // 10
    orc = bind.Oracle(len(ql), qe)
    init = _keys_of(orc, qe, ql, lab, pairs[6 * k:])
    deltas = [_keys_of(orc, qe, ql, lab, pairs[i * k:(i + 1) * k]) for i in range(6)]
    orc.build(init, n)
    want = [orc.batch(n, _empty(), _empty(), d, None, bind.PER_EDGE) for d in deltas]
    got = [[], [], []]

    def run(out):
        for _ in range(5):
            eng = Engine(dfs_budget_ms=20000)
            eng.load_query(len(ql), qe, ql)
            eng.build_index(init, n)
            out.append([eng.apply_batch(n, _empty(), _empty(), d) for d in deltas])
            eng.close()

    threads = [threading.Thread(target=run, args=(g,)) for g in got]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[want] * 5] * 3


# ---------------------------------------------------------------------------
# per-candidate tails: several lists, shared labels, lists around 32 entries
# ---------------------------------------------------------------------------
PATTERNS = {
    # square with a pendant: the counted vertex has two lists, one off the last core vertex
    "square": ([0, 1, 0, 1, 2], [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4)]),
    # two counted vertices of one label on the same core vertices (inclusion-exclusion)
    "twins": ([0, 1, 2, 2, 1], [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (0, 4)]),
    # three counted vertices of one label
    "triplet": ([0, 0, 1, 1, 1], [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (1, 4)]),
    # diamond with tails whose label is the last core vertex's
    "diamond": ([0, 1, 1, 0, 1], [(0, 1), (0, 2), (1, 2), (1, 3), (2, 3), (3, 4)]),
    # a path whose labels repeat (level sums with prefix vertices subtracted)
    "path": ([0, 1, 0, 1, 0], [(0, 1), (1, 2), (2, 3), (3, 4)]),
    # a hub subtree shared by its prefixes (memo), below a pendant seed edge
    "shared": ([0, 1, 2, 3, 3, 4], [(0, 1), (1, 2), (2, 3), (2, 4), (3, 5)]),
}


def _graph(rng, n, nlabels, hub_degree):
    """Random labelled graph; vertex 0 of every label is a hub of hub_degree."""
    lab = rng.integers(0, nlabels, n)
    lab[:nlabels] = np.arange(nlabels)
    pairs = {(int(min(a, b)), int(max(a, b))) for a, b in rng.integers(0, n, (4 * n, 2)) if a != b}
    for h in range(nlabels):
        for x in rng.choice(np.arange(nlabels, n), min(hub_degree, n - nlabels), replace=False):
            pairs.add((h, int(x)))
    return lab, np.array(sorted(pairs), dtype=np.int64)


def _keys_of(orc, qe, ql, lab, pairs):
    ks = []
    for a, b in qe:
        d0, d1 = orc.L.orc_dir(orc.h, a, b), orc.L.orc_dir(orc.h, b, a)
        for x, y in pairs:
            if lab[x] == ql[a] and lab[y] == ql[b]:
                ks += [_key(d0, x, y), _key(d1, y, x)]
            if lab[y] == ql[a] and lab[x] == ql[b]:
                ks += [_key(d0, y, x), _key(d1, x, y)]
    return np.array(ks, dtype=np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("hub_degree", [0, 31, 33, 120])
@pytest.mark.parametrize("name", sorted(PATTERNS))
def test_tails_per_candidate_match_restatement(name, hub_degree):
    """Counts of two batches equal the restatement's (per query edge), in the
    single-query engine and, in total, in the multi-query engine; then the
    second batch's edges are deleted again (as many negative matches)."""
    ql, qe = PATTERNS[name]
    rng = np.random.default_rng(7 + hub_degree)
    n, nlabels = 160, max(ql) + 1
    lab, pairs = _graph(rng, n, nlabels, hub_degree)
    rng.shuffle(pairs)
    k = len(pairs) // 6
    parts = [pairs[2 * k:], pairs[:k], pairs[k:2 * k]]
    orc = bind.Oracle(len(ql), qe)
    eng = Engine()
    eng.load_query(len(ql), qe, ql)
    init = _keys_of(orc, qe, ql, lab, parts[0])
    orc.build(init, n)
    eng.build_index(init, n)
    m = MultiQuery(dfs_budget_ms=60000)
    m.load_graph(lab.astype(np.uint32), parts[0].astype(np.uint32))
    qid = m.register(len(ql), qe, ql)
    for p in parts[1:]:
        delta = _keys_of(orc, qe, ql, lab, p)
        want = orc.batch(n, _empty(), _empty(), delta, None, bind.PER_EDGE)
        assert eng.apply_batch(n, _empty(), _empty(), delta) == want
        assert np.array_equal(eng.edge_counts(), orc.edge_counts())
        pos, _ = m.apply_batch(ins=p.astype(np.uint32))
        assert int(pos[qid]) == want
    _, neg = m.apply_batch(dele=parts[2].astype(np.uint32))
    assert int(neg[qid]) == want
    eng.close()
    m.close()


# Triangle (1, 3, 4) whose vertex 1 also carries a counted pendant (2) and the
# way to the seed: with no vertex of several lists kept in the tail, the last
# level is one intersection per candidate (pair counting).
PAIRED = ([0, 1, 2, 3, 4, 0], [(0, 1), (1, 2), (1, 3), (1, 4), (3, 4), (0, 5)])

PAIR_CPP = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "query.h"
int main(int argc, char** argv) {  // qv qe labels... edges...: plans with pair counting, per set of list lengths
    uint32_t qv = atoi(argv[1]), qe = atoi(argv[2]);
    std::vector<uint32_t> lab, edges;
    for (uint32_t i = 0; i < qv; ++i) lab.push_back(atoi(argv[3 + i]));
    for (uint32_t i = 0; i < 2 * qe; ++i) edges.push_back(atoi(argv[3 + qv + i]));
    cgb::QueryMeta q;
    if (!cgb::build_query_meta(qv, qe, edges.data(), lab.data(), q, cgb::kMaxQE).empty()) return 1;
    for (int t = 0; t < 50; ++t) {
        float avg[cgb::kMaxDir];
        for (float& x : avg) x = 1.f + rand() % 100;
        std::vector<cgb::EdgePlan> plans(cgb::kMaxQE);
        cgb::plan_edges(q, avg, plans.data(), true, true, true, true, true, false, 0);
        int n = 0;
        for (uint32_t e = 0; e < qe; ++e) n += plans[e].pair_last;
        std::printf("%d\n", n);
    }
}
"""


def _native(tmp_path, name, text, args):
    """Output lines of a C++ program built with the planner."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    csrc = os.path.join(root, "cgbdsm_b200", "csrc")
    src, exe = tmp_path / f"{name}.cpp", tmp_path / name
    src.write_text(text)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, "-I", os.path.join(root, "include"), str(src),
                    os.path.join(csrc, "query.cpp"), "-o", str(exe)], check=True)
    return subprocess.run([str(exe), *[str(x) for x in args]], check=True, capture_output=True,
                          text=True).stdout.splitlines()


def test_paired_pattern_plans_pair_counting(tmp_path):
    """PAIRED reaches pair counting whatever the mean list lengths are, in the
    plans that keep vertices with several lists out of the tail (a variant
    the multi-query engine's autotuner always tries)."""
    ql, qe = PAIRED
    counts = _native(tmp_path, "pairs", PAIR_CPP, [len(ql), len(qe), *ql, *[v for e in qe for v in e]])
    assert len(counts) == 50 and all(int(x) > 0 for x in counts)


@pytest.mark.gpu
@pytest.mark.parametrize("lane_max", [0, 2])
@pytest.mark.parametrize("pendants", [0, 3, 400])
def test_pair_counting_beside_descent_and_empty_tails(lane_max, pendants, monkeypatch):
    """With $CGB_PAIR_LANE_MAX a chunk holds candidates counted at once and
    candidates left to the descent, in lists shorter than a chunk; a prefix
    whose vertex has no pendant neighbour (all but `pendants` of them) has no
    tail, and its chunks are left at once.  Every plan variant's count equals
    the restatement's (the autotuner refuses variants that differ)."""
    monkeypatch.setenv("CGB_PAIR_LANE_MAX", str(lane_max))
    ql, qe = PAIRED
    rng = np.random.default_rng(pendants)
    n = 1500
    lab = np.repeat(np.arange(5), n // 5)
    rng.shuffle(lab)
    by = [np.flatnonzero(lab == k) for k in range(5)]
    pairs = set()
    for x, y, m in [(0, 0, 900), (0, 1, 1500), (1, 3, 4000), (1, 4, 4000), (3, 4, 4000)]:
        pairs |= {(int(a), int(b)) for a, b in zip(rng.choice(by[x], m), rng.choice(by[y], m)) if a != b}
    for a in rng.choice(by[1], min(pendants, len(by[1])), replace=False):
        pairs.add((int(a), int(rng.choice(by[2]))))
    pairs = np.array(sorted({(min(p), max(p)) for p in pairs}), dtype=np.int64)
    rng.shuffle(pairs)
    k = len(pairs) // 5
    parts = [pairs[2 * k:], pairs[:k], pairs[k:2 * k]]
    orc = bind.Oracle(len(ql), qe)
    orc.build(_keys_of(orc, qe, ql, lab, parts[0]), n)
    m = MultiQuery(dfs_budget_ms=60000)
    m.load_graph(lab.astype(np.uint32), parts[0].astype(np.uint32))
    qid = m.register(len(ql), qe, ql)
    total = 0
    for p in parts[1:]:
        want = orc.batch(n, _empty(), _empty(), _keys_of(orc, qe, ql, lab, p), None, bind.PER_EDGE)
        pos, _ = m.apply_batch(ins=p.astype(np.uint32))
        assert int(pos[qid]) == want
        total += want
    assert (total > 0) == (pendants > 0)
    m.close()


@pytest.mark.gpu
@pytest.mark.parametrize("hubs", [1, 3, 40])
def test_level_sum_table_under_contention(hubs):
    """Thousands of prefixes ask the level-sum table for the same few owners at
    once: one of them claims the slot, the others find it busy or published.
    Path 4-0-1-2-3 whose (0, 1) edges all end in `hubs` vertices; counts equal
    the restatement's, in both engines."""
    ql, qe = [0, 1, 2, 3, 4], [(0, 1), (1, 2), (2, 3), (0, 4)]
    rng = np.random.default_rng(hubs)
    n0 = 3000
    v0 = np.arange(n0)
    v1 = n0 + np.arange(hubs)
    v2 = v1[-1] + 1 + np.arange(200)
    v3 = v2[-1] + 1 + np.arange(60)
    v4 = v3[-1] + 1 + np.arange(50)
    n = int(v4[-1]) + 1
    lab = np.zeros(n, np.int64)
    for k, v in enumerate((v0, v1, v2, v3, v4)):
        lab[v] = k
    seeds = np.stack([v0, rng.choice(v1, n0)], 1)
    rest = {(int(a), int(b)) for a, b in zip(rng.choice(v1, 40 * hubs), rng.choice(v2, 40 * hubs))}
    rest |= {(int(a), int(b)) for a, b in zip(rng.choice(v2, 500), rng.choice(v3, 500))}
    rest |= {(int(a), int(b)) for a, b in zip(rng.choice(v0, 4000), rng.choice(v4, 4000))}
    rest = np.array(sorted(rest), dtype=np.int64)
    orc = bind.Oracle(len(ql), qe)
    init = _keys_of(orc, qe, ql, lab, rest)
    delta = _keys_of(orc, qe, ql, lab, seeds)
    orc.build(init, n)
    want = orc.batch(n, _empty(), _empty(), delta, None, bind.PER_EDGE)
    assert want > 0
    eng = Engine()
    eng.load_query(len(ql), qe, ql)
    eng.build_index(init, n)
    assert eng.apply_batch(n, _empty(), _empty(), delta) == want
    eng.close()
    m = MultiQuery(dfs_budget_ms=60000)
    m.load_graph(lab.astype(np.uint32), rest.astype(np.uint32))
    qid = m.register(len(ql), qe, ql)
    pos, _ = m.apply_batch(ins=seeds.astype(np.uint32))
    assert int(pos[qid]) == want
    _, neg = m.apply_batch(dele=seeds.astype(np.uint32))
    assert int(neg[qid]) == want
    m.close()


@pytest.mark.gpu
def test_byte_count_of_long_walks():
    """The statistics' bytes of one warp's 64 steps go beyond 2^34: 2,100
    candidates with 1,600 common neighbours each, counted as a group of three:
    seven walks a candidate, over 2, 4 or 6 lists."""
    K, T = 2100, 1600
    ql, qe = [0, 1, 2, 3, 3, 3], [(0, 1), (0, 2), (1, 3), (1, 4), (1, 5), (2, 3), (2, 4), (2, 5)]
    orc = bind.Oracle(len(ql), qe)
    d = {(a, b): orc.L.orc_dir(orc.h, a, b) for x, y in qe for a, b in ((x, y), (y, x))}
    v0, v1, c, t = 0, 1, 2 + np.arange(K), 2 + K + np.arange(T)
    cc, tt = np.repeat(c, T), np.tile(t, K)
    keys = []
    for a, b, x, y in [(0, 2, np.full(K, v0), c)] + [(1, k, np.full(T, v1), t) for k in (3, 4, 5)] + \
            [(2, k, cc, tt) for k in (3, 4, 5)]:
        keys += [_key(d[a, b], x, y), _key(d[b, a], y, x)]
    eng = Engine(flags=FLAG_NO_STEAL, dfs_budget_ms=60000)
    eng.load_query(len(ql), qe, ql)
    eng.build_index(np.concatenate(keys), 2 + K + T)
    delta = np.array([_key(d[0, 1], v0, v1), _key(d[1, 0], v1, v0)], np.uint64)
    assert eng.apply_batch(2 + K + T, _empty(), _empty(), delta) == K * T * (T - 1) * (T - 2)
    # per common neighbour: its entry in every walk, and searches in the walks' other lists
    want = K * T * (7 * 4 + (3 * 1 + 3 * 3 + 1 * 5) * 32 * (33 - (32 - T.bit_length())))
    assert want * 60 // 64 > 1 << 34
    assert want <= eng.stats()["match_bytes"] < want * 1.01
    eng.close()


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, FLAG_FORCE_SPLIT, FLAG_NO_STEAL])
@pytest.mark.parametrize("hub_degree", [10, 90])
def test_subtree_memos_while_work_is_shared(flags, hub_degree):
    """A plan with a subtree memo (asserted), whose one expansion per vertex is
    handed to other warps part by part (every chunk of it under
    FLAG_FORCE_SPLIT, asserted) while prefixes add their weights: counts per
    query edge equal the restatement's, batch after batch."""
    ql, qe = [0, 1, 2, 3, 4, 5, 1], [(0, 1), (0, 2), (1, 3), (1, 4), (1, 5), (1, 6), (5, 6)]
    rng = np.random.default_rng(hub_degree)
    n = 900
    lab = rng.choice(6, n, p=[0.25, 0.3, 0.2, 0.05, 0.05, 0.15])
    pairs = {(int(min(p)), int(max(p))) for p in rng.integers(0, n, (10 * n, 2)) if p[0] != p[1]}
    for h in np.flatnonzero(lab == 1)[:5]:
        pairs |= {(int(min(h, x)), int(max(h, x))) for x in rng.choice(n, hub_degree, replace=False) if x != h}
    pairs = np.array(sorted(pairs), dtype=np.int64)
    rng.shuffle(pairs)
    k = len(pairs) // 5
    orc = bind.Oracle(len(ql), qe)
    eng = Engine(flags=flags, dfs_budget_ms=60000)
    eng.load_query(len(ql), qe, ql)
    init = _keys_of(orc, qe, ql, lab, pairs[2 * k:])
    orc.build(init, n)
    eng.build_index(init, n)
    assert any(eng.plan_info(e)["memo_from"] for e in range(len(qe)))
    tasks = total = 0
    for p in (pairs[:k], pairs[k:2 * k]):
        delta = _keys_of(orc, qe, ql, lab, p)
        want = orc.batch(n, _empty(), _empty(), delta, None, bind.PER_EDGE)
        assert eng.apply_batch(n, _empty(), _empty(), delta) == want
        assert np.array_equal(eng.edge_counts(), orc.edge_counts())
        tasks += eng.stats()["stolen_tasks"]
        total += want
    assert total > 0
    assert (tasks == 0) if flags == FLAG_NO_STEAL else (tasks > 0 or flags == 0)
    eng.close()


# ---------------------------------------------------------------------------
# packed-memory array: windows of one and of many leaves
# ---------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("n,burst", [(0, 1), (31, 40), (1000, 33), (5000, 2000)])
def test_gpma_windows_and_counts(n, burst):
    """Inserts crowded into one stretch of keys (windows of many leaves) and
    spread ones (single leaves), deletes, and both at once; contents and
    counts per direction equal the set model's after every update."""
    rng = np.random.default_rng(n + burst)
    g = Gpma(3)
    state = np.unique(np.array([_key(int(d), int(u), int(v)) for d, u, v in
                                zip(rng.integers(0, 3, n), rng.integers(0, 500, n), rng.integers(0, 500, n))], np.uint64)) \
        if n else _empty()
    g.bulk_load(state)
    for step in range(4):
        crowd = np.array([_key(1, 250, 1000 + step * burst + i) for i in range(burst)], np.uint64)
        spread = np.array([_key(int(d), int(u), int(v)) for d, u, v in
                           zip(rng.integers(0, 3, burst), rng.integers(0, 500, burst), rng.integers(0, 500, burst))], np.uint64)
        dele = rng.choice(state, len(state) // 4, replace=False) if len(state) else _empty()
        ins = np.concatenate([crowd, spread, dele[:5]])
        g.batch_update(ins, dele)
        state = np.setdiff1d(np.union1d(state, ins), dele)
        for d in range(3):
            mine = state[(state >> np.uint64(59)) == d] & np.uint64((1 << 59) - 1)
            assert np.array_equal(g.extract(d), mine), (step, d)
        assert g.stats()["keys"] == len(state)
    g.close()


def test_buffers_kept_between_calls(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "kept"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(root, "cgbdsm_b200", "csrc"),
                    os.path.join(root, "tests", "native", "kept_buffers.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout == "ok\n"


# ---------------------------------------------------------------------------
# flat merge: tile edges (2,816 entries) and more than 32 tiles back to a prefix
# ---------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("n_old,n_ins,n_del", [(2815, 1, 0), (2815, 1, 1), (2816, 0, 1), (5631, 3, 2), (0, 2817, 0),
                                               (200_000, 5000, 5000)])
def test_flat_merge_tile_edges(n_old, n_ins, n_del):
    import torch

    from cgbdsm_b200 import load_library

    rng = np.random.default_rng(n_old)
    dv = 3000
    pool = np.unique(_key(0, 0, 0) + (rng.integers(0, 4, 2 * (n_old + n_ins) + 64).astype(np.uint64) << np.uint64(59))
                     + (rng.integers(0, dv, 2 * (n_old + n_ins) + 64).astype(np.uint64) << np.uint64(32))
                     + rng.integers(0, dv, 2 * (n_old + n_ins) + 64).astype(np.uint64))
    pick = rng.permutation(len(pool))
    old = np.sort(pool[pick[:n_old]])
    ins = pool[pick[n_old:n_old + n_ins]]
    dele = np.concatenate([rng.choice(old, n_del, replace=False) if n_old else _empty(), ins[:n_ins // 4]])[:max(n_del, 0)]
    want = np.setdiff1d(np.union1d(old, ins), dele)

    def dev(a):
        return torch.from_numpy((a if len(a) else np.zeros(1, np.uint64)).view(np.int64)).cuda()

    t_old, t_ins, t_del = dev(old), dev(ins), dev(dele)
    out = torch.zeros(len(old) + len(ins) + 1, dtype=torch.int64, device="cuda")
    out_n = torch.zeros(1, dtype=torch.int64, device="cuda")
    st = load_library().cgb_merge_keys_noalloc(t_old.data_ptr(), len(old), t_ins.data_ptr(), len(ins), t_del.data_ptr(),
                                               len(dele), dv, out.data_ptr(), out_n.data_ptr(), None)
    torch.cuda.synchronize()
    assert st == 0
    got = out[:int(out_n.item())].cpu().numpy().view(np.uint64)
    assert np.array_equal(got, want)


# ---------------------------------------------------------------------------
# calls into the CUDA runtime that fail or that should not be made
# ---------------------------------------------------------------------------
RETRY_PY = r"""
import sys
import numpy as np
from cgbdsm_b200 import Engine
from cgbdsm_b200.engine import CgbError
z = np.load(sys.argv[1])
ql, qe, n = [int(x) for x in z["ql"]], [tuple(int(v) for v in e) for e in z["qe"]], int(z["n"])
eng = Engine()
eng.load_query(len(ql), qe, ql)
try:
    eng.build_index(z["init"], n)
    print("no failure")
except CgbError as e:
    print("failed" if sys.argv[2] in str(e) else f"other failure: {e}")
eng.build_index(z["init"], n)
none = np.zeros(0, np.uint64)
for k in range(2):
    print(eng.apply_batch(n, none, none, z[f"delta{k}"]))
"""


def _with_shim(tmp_path, script, args, **env):
    """Output lines of a Python script run with the runtime shim preloaded."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    so = tmp_path / "shim.so"
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", os.path.join(root, "tests", "native", "cudart_shim.c"), "-o", str(so),
                    "-ldl"], check=True)
    out = subprocess.run([sys.executable, "-c", script, *[str(x) for x in args]], check=True, capture_output=True, text=True,
                         cwd=root, timeout=300, env={**os.environ, "LD_PRELOAD": str(so), "PYTHONPATH": root, **env}).stdout
    return out.splitlines()


@pytest.mark.gpu
@pytest.mark.parametrize("name,what", [("d_memo_list", 4), ("d_memo", 32), ("d_lsum", 16)])
def test_failed_table_allocation_is_retried(name, what, tmp_path):
    """An allocation that fails while the matcher's tables are made (4,096
    slots at this size) fails the call; the next one makes them, and counts on
    a pattern with a subtree memo equal the restatement's."""
    ql, qe = PATTERNS["shared"]
    rng = np.random.default_rng(3)
    n = 160
    lab, pairs = _graph(rng, n, max(ql) + 1, 33)
    rng.shuffle(pairs)
    k = len(pairs) // 6
    orc = bind.Oracle(len(ql), qe)
    init = _keys_of(orc, qe, ql, lab, pairs[2 * k:])
    deltas = [_keys_of(orc, qe, ql, lab, p) for p in (pairs[:k], pairs[k:2 * k])]
    orc.build(init, n)
    want = [orc.batch(n, _empty(), _empty(), d, None, bind.PER_EDGE) for d in deltas]
    f = tmp_path / "in.npz"
    np.savez(f, ql=ql, qe=qe, n=n, init=init, delta0=deltas[0], delta1=deltas[1])
    got = _with_shim(tmp_path, RETRY_PY, [f, name], CGB_SHIM_FAIL_BYTES=str(4096 * what))
    assert got == ["failed", str(want[0]), str(want[1])]


GROWING_PY = r"""
import sys
import numpy as np
from cgbdsm_b200 import Engine
z = np.load(sys.argv[1])
none = np.zeros(0, np.uint64)
eng = Engine()
eng.load_query(6, [(k, k + 1) for k in range(5)], list(range(6)))
eng.build_index(z["init"], int(z["ids"][0]))
for i, n in enumerate(z["ids"]):
    print(eng.apply_batch(int(n), none, none, z[f"delta{i}"]))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("ids", [(300, 5000), (300, 2000, 9000, 40000)])
def test_dense_level_sums_with_growing_ids(ids, tmp_path):
    """A tree of labels of their own (dense level sums) whose vertex ids outgrow
    the record table between matched batches, with an allocator that hands
    the sums' block out again for their larger arrays: the jobs follow the
    table's width, not the block's address.  Counts equal the restatement's."""
    ql, qe = list(range(6)), [(k, k + 1) for k in range(5)]
    rng = np.random.default_rng(len(ids))

    def some(n, lo, m):
        pairs = {(6 * (int(a) // 6) + x, 6 * (int(b) // 6) + y)
                 for x, y in qe for a, b in zip(rng.integers(lo, n - 6, m), rng.integers(0, n - 6, m))}
        return _keys_of(orc, qe, ql, np.arange(n) % 6, np.array(sorted(pairs), dtype=np.int64))

    orc = bind.Oracle(len(ql), qe)
    init = some(ids[0], 0, 400)
    orc.build(init, ids[0])
    seen, deltas, want = init, {}, []
    for i, n in enumerate(ids):
        keys = np.setdiff1d(some(n, ids[i - 1] if i else 0, 300), seen)
        seen = np.union1d(seen, keys)
        deltas[f"delta{i}"] = keys
        want.append(orc.batch(n, _empty(), _empty(), keys, None, bind.PER_EDGE))
    assert all(w > 0 for w in want)
    f = tmp_path / "in.npz"
    np.savez(f, ids=ids, init=init, **deltas)
    assert _with_shim(tmp_path, GROWING_PY, [f], CGB_SHIM_REUSE="1") == [str(w) for w in want]


CREATE_PY = r"""
import os, sys
from cgbdsm_b200 import Engine, MultiQuery
e, m = Engine(), MultiQuery(dfs_budget_ms=60000)
print(open(os.environ["CGB_SHIM_ATTR_LOG"]).read().split())
m.load_graph([0, 1, 0, 1], [(0, 1)])
q = m.register(2, [(0, 1)], [0, 1])
print(int(m.apply_batch(ins=[(2, 3), (0, 3)])[0][q]))
print(open(os.environ["CGB_SHIM_ATTR_LOG"]).read().split())
"""


@pytest.mark.gpu
def test_creating_an_engine_asks_for_no_clock_rate(tmp_path):
    """The clock rate (attribute 13), slow to read, is asked for by the
    autotuner alone, not by creating a handle."""
    created, count, tuned = _with_shim(tmp_path, CREATE_PY, [], CGB_SHIM_ATTR_LOG=str(tmp_path / "attrs"))
    assert "'13'" not in created and "'16'" in created
    assert count == "2" and tuned.count("'13'") == 1


# ---------------------------------------------------------------------------
# planned subsets (no GPU)
# ---------------------------------------------------------------------------
SUBSETS_CPP = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "query.h"
int main(int argc, char** argv) {  // qv qe fold labels... edges...
    uint32_t qv = atoi(argv[1]), qe = atoi(argv[2]), fold = atoi(argv[3]);
    std::vector<uint32_t> lab, edges;
    for (uint32_t i = 0; i < qv; ++i) lab.push_back(atoi(argv[4 + i]));
    for (uint32_t i = 0; i < 2 * qe; ++i) edges.push_back(atoi(argv[4 + qv + i]));
    cgb::QueryMeta q;
    if (!cgb::build_query_meta(qv, qe, edges.data(), lab.data(), q, cgb::kMaxQE).empty()) return 1;
    float avg[cgb::kMaxDir];
    for (float& x : avg) x = 1.f;
    std::vector<cgb::EdgePlan> plans(cgb::kMaxQE);
    cgb::plan_edges(q, avg, plans.data(), true, true, true, true, true, false, fold);
    for (uint32_t e = 0; e < qe; ++e) {
        const cgb::EdgePlan& p = plans[e];
        std::printf("%u %u %u %u", p.n, p.n_core, p.n_sub, p.sub_base);
        for (uint32_t j = 0; j <= p.n; ++j) std::printf(" %u", p.bn_off[j]);
        for (uint32_t b = 0; b < p.bn_off[p.n]; ++b) std::printf(" %u", p.bn_pos[b]);
        for (uint32_t j = 0; j < p.n; ++j) std::printf(" %u", p.tail_gid[j]);
        for (uint32_t i = 0; i < p.n_sub; ++i) std::printf(" %u %u %u %u", p.sub_lists[i], p.sub_pos[i], p.sub_group[i], p.sub_kind[i]);
        std::printf("\n");
    }
}
"""


def test_planned_subsets_cover_every_tail_group(tmp_path):
    """Every tail label group of k members has its 2^k - 1 member subsets in an
    order whose single members come first, each with the union of its members'
    lists and owners; every tail vertex is in exactly one group."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    csrc = os.path.join(root, "cgbdsm_b200", "csrc")
    src, exe = tmp_path / "subsets.cpp", tmp_path / "subsets"
    src.write_text(SUBSETS_CPP)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, "-I", os.path.join(root, "include"), str(src),
                    os.path.join(csrc, "query.cpp"), "-o", str(exe)], check=True)
    cases = list(PATTERNS.values())
    for s in ("c2", "c3"):
        with open(os.path.join(root, "cgbdsm_b200", "data", f"queries_{s}.json")) as f:
            cases += [(q["labels"], [tuple(e) for e in q["edges"]]) for q in json.load(f)["queries"]]
    folded = 0
    for labels, edges in cases:
        for fold in (0, 3, 12):
            args = [str(x) for x in (len(labels), len(edges), fold, *labels, *[v for e in edges for v in e])]
            out = subprocess.run([str(exe), *args], check=True, capture_output=True, text=True).stdout
            for line in out.splitlines():
                f = [int(x) for x in line.split()]
                n, nc, ns, base = f[:4]
                off, f = f[4:5 + n], f[5 + n:]
                pos, f = f[:off[n]], f[off[n]:]
                gid, f = f[:n], f[n:]
                subs = [f[4 * i:4 * i + 4] for i in range(ns)]
                groups, t = [], nc
                while t < n:
                    e = t
                    while e < n and gid[e] == gid[t]:
                        e += 1
                    groups.append(list(range(t, e)))
                    t = e
                i = 0
                for g in groups:
                    k = len(g)
                    assert 1 <= k <= 3
                    seen = []
                    for lists, owners, group, kind in subs[i:i + 2 ** k - 1]:
                        mask = kind & 7
                        want = 0
                        for mem in range(k):
                            if mask >> mem & 1:
                                for b in range(off[g[mem]], off[g[mem] + 1]):
                                    want |= 1 << (b - base)
                        assert lists == want and owners == sum(1 << x for x in {pos[base + b] for b in range(32) if want >> b & 1})
                        assert owners & ~group == 0 and bool(kind & 0x10) == (k == 3)
                        assert bool(kind & 8) == (len(seen) == 2 ** k - 2)
                        if nc - 1 in [pos[base + b] for b in range(32) if want >> b & 1] and bin(want).count("1") > 1:
                            folded += 1
                        seen.append(mask)
                    assert sorted(seen) == list(range(1, 2 ** k)) and sorted(seen[:k]) == [1 << x for x in range(k)]
                    i += 2 ** k - 1
                assert ns - i <= 1  # then the pair or the level sum
    assert folded > 0
