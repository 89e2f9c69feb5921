"""Performance cases: the work a program has this engine do, through its public entry points.

A case is a dict of plain values.  Its ``path`` says which calls it makes:

* ``program``: one Datalog program (``programs.build_tc`` / ``build_sg``) whose input
  relation is loaded, run to its fixed point and read back -- ``Program.load_rows`` or
  ``load_rows_device``, ``execute``, ``history``, ``counts``, ``dump_full``;
* ``request``: one instance through ``batch.Runner.run_plain`` from host rows, as the server
  runs it alone: upload, packing, fixed point, per-iteration sizes, counts and digests;
* ``wave``: many instances through ``batch.Runner.run_wave``;
* ``described``: one of the reference's generated analyses (``programs.build_described``,
  tests/golden/<name>/), whose tuples hold intern ids and take the wide-tuple path.

Graphs are the generators of ``datagen``: Erdos-Renyi digraphs (``n`` nodes, ``deg`` * n
edges) for transitive closure, breadth-first random trees for same generation.  A case
fixes the graph up to its labels; the seed numbers the nodes (a permutation for the random
digraphs, a rotation for the trees, whose siblings keep neighbouring numbers).
"""
import math
import os

import numpy as np
import torch

import parallel_ra_b200 as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OUTPUT = {"tc": "T", "sg": "SG"}
INPUT = {"tc": "G", "sg": "edge"}


def listed():
    return [
        # a small graph asked for alone: latency, launches and host round trips only
        {"name": "tc-request-300", "path": "request", "program": "tc", "n": 300, "deg": 1.3},
        # the benchmark's first configuration (n = 2,000, m = 3,000), its closure read back
        {"name": "tc-2000-rows", "path": "program", "program": "tc", "n": 2000, "deg": 1.5, "ids": "emission",
         "load": "host"},
        # a dense closure, the largest class of the batched mix (172 million tuples)
        {"name": "tc-16384-dense", "path": "request", "program": "tc", "n": 16384, "deg": 2.0},
        # an ordinary sparse graph of an odd size, its closure read back
        {"name": "tc-131071-rows", "path": "program", "program": "tc", "n": 131071, "deg": 0.95, "ids": "emission",
         "load": "host"},
        # the benchmark's headline configuration: 2^22 nodes, about 80 million tuples
        {"name": "tc-er22", "path": "request", "program": "tc", "n": 1 << 22, "deg": 0.95},
        # the reference's own id numbering: every delta sorted into trie order
        {"name": "tc-100003-refids", "path": "program", "program": "tc", "n": 100003, "deg": 0.95, "ids": "reference",
         "load": "device"},
        # a small same-generation request: two joins through an intermediate relation
        {"name": "sg-request-1000", "path": "request", "program": "sg", "n": 1000, "deg": 0.0},
        # the benchmark's same-generation configuration: 2^15 nodes, about 330 million tuples
        {"name": "sg-tree15", "path": "request", "program": "sg", "n": 1 << 15, "deg": 0.0},
        # a wave of the batched mix: n log-uniform in [64, 16384], degree uniform in [0.8, 2]
        {"name": "wave-tc-64", "path": "wave", "program": "tc", "count": 64, "n_hi": 16384},
        # a wave of same-generation requests
        {"name": "wave-sg-96", "path": "wave", "program": "sg", "count": 96, "n_hi": 4096},
        # generated analyses: many small iterations over wide tuples
        {"name": "cfa-4-4-64", "path": "described", "analysis": "cfa-4-4-64"},
        {"name": "worstcase-110-4", "path": "described", "analysis": "worstcase-110-terms-4-m"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: program kinds, sizes, degrees, id orders, ways to load and to read."""
    path = rng.choice(["program", "program", "program", "program", "request", "request", "wave", "wave", "described"])
    if path == "described":
        return {"path": path, "analysis": rng.choice(["cfa-4-4-64", "cfa-4-4-64", "worstcase-110-terms-4-m"]),
                "labels": rng.randrange(1, 1 << 20)}
    program, graph = rng.choice(["tc", "tc", "sg"]), rng.randrange(1, 1 << 20)
    if path == "wave":
        n_hi = _log_uniform(rng, 512, 16384 if program == "tc" else 4096)
        most = min(512, int(64 * (16384 / n_hi) ** 2))
        return {"path": path, "program": program, "count": _log_uniform(rng, 16, most), "n_hi": n_hi, "graph": graph}
    # programs read their closure back: sizes up to about three million derived tuples
    if program == "sg":
        n, deg = _log_uniform(rng, 64, 2048 if path == "program" else 1 << 15), 0.0
    else:
        n = _log_uniform(rng, 64, 150000 if path == "program" else 1 << 22)
        deg = round(rng.uniform(0.8, 2.0 if n <= 2000 or (path == "request" and n <= 16384) else 0.95), 3)
    case = {"path": path, "program": program, "n": n, "deg": deg, "graph": graph}
    if path == "program":
        case.update(ids=rng.choice(["emission", "emission", "reference"]), load=rng.choice(["host", "device"]))
    return case


def _tuples(program, n, deg):
    """Expected derived tuples (the relations the rules write), for sizing."""
    if program == "sg":   # SG and TMP of a random tree with one to four children per node
        return 0.51 * n * n + n
    if deg > 1.0:
        s = 0.5
        for _ in range(100):
            s = 1.0 - math.exp(-deg * s)
        return (s * n) ** 2 + 2.0 * n
    return n * min(deg / max(1.0 - deg, 1e-9), math.sqrt(n))


def _relabel(pairs, program, n, seed):
    """The same graph with its nodes numbered by the seed."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if program == "sg":
        return (pairs + rng.integers(1, n, dtype=np.uint64)) % np.uint64(n) if n > 1 else pairs
    return rng.permutation(n).astype(np.uint64)[pairs]


def _graph(case, seed):
    program, n, graph = case["program"], case["n"], case.get("graph", 1)
    if program == "sg":
        pairs = P.datagen.random_tree(n, graph)
    else:
        pairs = P.datagen.erdos_renyi(n, min(max(1, round(case["deg"] * n)), n * (n - 1)), graph)
    return P.datagen.with_row_ids(_relabel(pairs, program, n, seed))


def _wave_instances(case, seed):
    sizes = P.datagen.batched_sizes(case["count"], case.get("graph", 1), 64, case["n_hi"])
    return [_graph({"program": case["program"], "n": n, "deg": m / n, "graph": g}, seed + i)
            for i, (n, m, g) in enumerate(sizes)]


class _Relabelled:
    """Builder that renumbers the labels of the input relations: values that carry an
    intern tag are permuted among those of their tag, the others among themselves.
    The analysis is the same one with its program points numbered differently."""

    def __init__(self, prog, rows_by_name, seed):
        self.prog, self.loaded = prog, []
        values = np.unique(np.concatenate([r.ravel() for r in rows_by_name.values()]))
        rng = np.random.Generator(np.random.PCG64(seed))
        renamed = values.copy()
        for tag in np.unique(values >> np.uint64(46)):
            at = np.flatnonzero(values >> np.uint64(46) == tag)
            renamed[at] = values[rng.permutation(at)]
        self.values, self.renamed = values, renamed

    def load_rows(self, rel, rows):
        if rows.shape[0]:
            rows = np.ascontiguousarray(self.renamed[np.searchsorted(self.values, rows)])
            self.loaded.append((rel, rows))
        self.prog.load_rows(rel, rows)

    def __getattr__(self, name):
        return getattr(self.prog, name)


def prepare(case, seed):
    path = case["path"]
    if path == "request":
        # rows in page-locked memory, as a program that uploads many inputs keeps them
        rows = torch.from_numpy(_graph(case, seed).view(np.int64)).pin_memory()
        return {"path": path, "runner": P.batch.Runner(case["program"]), "pinned": rows,
                "rows": rows.numpy().view(np.uint64)}
    if path == "wave":
        return {"path": path, "runner": P.batch.Runner(case["program"]), "instances": _wave_instances(case, seed)}
    if path == "described":
        base = os.path.join(ROOT, "tests", "golden", case["analysis"])
        program, data = os.path.join(base, "program.txt"), os.path.join(base, "data")
        desc = P.programs.read_description(program)
        rows = {r["name"]: P.datagen.read_relation(os.path.join(data, r["file"]))
                for r in desc["relations"] if r["file"]}
        prog = P.Program(0)
        builder = _Relabelled(prog, rows, seed + case.get("labels", 0))
        handles = P.programs.build_described(builder, program, data)
        batch = handles.pop("__batch__")
        # what a user of the analysis reads: its relations, without their index copies and
        # the compiler's intermediate ones
        answers = [r["name"] for r in desc["relations"]
                   if r["canonical"] and not r["name"].startswith(("rel_inter", "rel_inner", "rel_t_"))]
        return {"path": path, "prog": prog, "rels": handles, "batch": batch, "inputs": builder.loaded,
                "answers": answers}
    prog = P.Program(0, id_order=P.engine.IDS_REFERENCE if case["ids"] == "reference" else P.engine.IDS_EMISSION)
    rels = P.programs.PROGRAMS[case["program"]](prog, np.empty((0, 3), dtype=np.uint64))
    rows = _graph(case, seed)
    if case["load"] == "device":
        rows = torch.from_numpy(rows.view(np.int64)).cuda()
    return {"path": path, "prog": prog, "rels": rels, "input": rels[INPUT[case["program"]]],
            "output": rels[OUTPUT[case["program"]]], "rows": rows}


def _history(prog):
    return np.array([pair for _, pairs in prog.history() for pair in pairs], dtype=np.uint64).view(np.int64)


def _instance_arrays(results):
    """What Runner returns for each instance, as arrays: counts, digests and delta sizes."""
    names = sorted(results[0].counts)
    return {"counts": np.array([[r.counts[k] for k in names] for r in results], dtype=np.int64),
            "digests": np.array([[r.digests[k] for k in names] for r in results], dtype=np.uint64).view(np.int64),
            "deltas": np.array([v for r in results for d in r.deltas for v in d], dtype=np.int64),
            "iterations": np.array([[len(d) for d in r.deltas] for r in results], dtype=np.int64)}


def run(state):
    path = state["path"]
    if path == "request":
        return _instance_arrays([state["runner"].run_plain(state["rows"])])
    if path == "wave":
        return _instance_arrays(state["runner"].run_wave(state["instances"]))
    prog, rels = state["prog"], state["rels"]
    if path == "described":
        for rel, rows in state["inputs"]:
            prog.load_rows(rel, rows)
        prog.execute(state["batch"])
        return {"history": _history(prog),
                "counts": np.array([prog.counts(h)[0] for h in rels.values()], dtype=np.int64),
                "rows": {name: prog.dump_full(rels[name]).view(np.int64) for name in state["answers"]}}
    rows = state["rows"]
    if isinstance(rows, torch.Tensor):
        prog.load_rows_device(state["input"], rows.data_ptr(), rows.shape[0])
    else:
        prog.load_rows(state["input"], rows)
    prog.execute()
    got = prog.dump_full(state["output"]).view(np.int64)
    return {"history": _history(prog),
            "counts": np.array([prog.counts(rels[k])[0] for k in sorted(rels)], dtype=np.int64),
            "data": got[:, :-1], "ids": got[:, -1]}


def work(case):
    """Input rows read once (24 bytes each); derived tuples written once (16 bytes as they stay
    in device memory, key and id; rows of 8-byte columns where they are read back)."""
    if case["path"] == "described":
        # facts of the analyses on their own inputs, and their average row width
        facts, width = (6476108, 80) if case["analysis"].startswith("worst") else (40000, 100)
        return {"bytes": float(facts * width), "flops": 0.0}
    if case["path"] == "wave":
        lo, hi, steps = 64.0, float(case["n_hi"]), 64
        n = [lo * (hi / lo) ** ((i + 0.5) / steps) for i in range(steps)]
        deg = [0.8 + 1.2 * (j + 0.5) / 8 for j in range(8)]
        if case["program"] == "sg":
            tuples = sum(_tuples("sg", v, 0.0) for v in n) / steps
            rows = sum(n) / steps
        else:
            tuples = sum(_tuples("tc", v, d) for v in n for d in deg) / (8 * steps)
            rows = 1.4 * sum(n) / steps
        return {"bytes": case["count"] * (24.0 * rows + 16.0 * tuples), "flops": 0.0}
    n, deg, program = case["n"], case["deg"], case["program"]
    rows = n - 1 if program == "sg" else round(deg * n)
    tuples = _tuples(program, n, deg)
    per = 40.0 if case["path"] == "program" else 16.0
    return {"bytes": 24.0 * rows + per * tuples, "flops": 0.0}


# ---------------------------------------------------------------------------
# the same results from plain torch integer arithmetic, semi-naive
# ---------------------------------------------------------------------------

def _join(outer_key, outer_val, inner_key, inner_val):
    """Pairs (outer_val, inner_val) with equal keys; inner_key is sorted."""
    lo = torch.searchsorted(inner_key, outer_key)
    cnt = torch.searchsorted(inner_key, outer_key, right=True) - lo
    o = torch.repeat_interleave(torch.arange(outer_key.numel(), device=outer_key.device), cnt)
    first = torch.cumsum(cnt, 0) - cnt
    i = lo[o] + torch.arange(o.numel(), device=o.device) - first[o]
    return outer_val[o], inner_val[i]


def _minus(cand, known):
    """Distinct values of cand that are not in the sorted array known."""
    cand = torch.unique(cand)
    if not known.numel():
        return cand
    at = torch.searchsorted(known, cand).clamp_(max=known.numel() - 1)
    return cand[known[at] != cand]


def _union(a, b):
    return torch.sort(torch.cat([a, b]))[0] if b.numel() else a


def exact(case, seed):
    """History, counts and rows of a TC or SG program; None for its ids, an order of the engine's own."""
    if case["path"] != "program":
        return None
    rows = _graph(case, seed)
    e = torch.from_numpy(rows[:, :2].astype(np.int64))
    e = e.cuda() if torch.cuda.is_available() else e
    n, m = case["n"], e.shape[0]
    e = e[torch.argsort(e[:, 0] * n + e[:, 1])]
    src, dst = e[:, 0].contiguous(), e[:, 1].contiguous()
    if case["program"] == "tc":
        known = torch.sort(dst * n + src)[0]
        hist, delta = [(m, m)], known
        while True:
            x, z = _join(delta // n, delta % n, src, dst)
            delta = _minus(z * n + x, known)
            hist.append((delta.numel(), m + known.numel()))
            if not delta.numel():
                break
            known = _union(known, delta)
        out, counts = known, [m, known.numel()]                       # G, T
    else:
        x, y = _join(src, dst, src, dst)
        base = torch.unique(x * n + y)
        sg = base[base // n != base % n]
        hist = [(base.numel(), m), (sg.numel(), base.numel())]
        tmp, dsg, dtmp = sg[:0], sg, sg[:0]
        full_sg = full_tmp = 0
        while True:
            full_sg += dsg.numel()
            full_tmp += dtmp.numel()
            y, c = _join(dsg // n, dsg % n, src, dst)
            ntmp = _minus(y * n + c, tmp)
            c, d = _join(dtmp // n, dtmp % n, src, dst)
            nsg = _minus(c * n + d, sg)
            hist.append((nsg.numel() + ntmp.numel(), m + full_sg + full_tmp))
            tmp, sg, dtmp, dsg = _union(tmp, ntmp), _union(sg, nsg), ntmp, nsg
            if not ntmp.numel() and not nsg.numel():
                break
        out, counts = sg, [sg.numel(), base.numel(), tmp.numel(), m]  # SG, SGB, TMP, edge
    return {"history": torch.tensor(hist, dtype=torch.int64), "counts": torch.tensor(counts, dtype=torch.int64),
            "data": torch.stack([out // n, out % n], 1), "ids": None}
