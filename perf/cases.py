"""The work that the framework's speed is measured by: whole Datalog programs through `Executor`
(relations on the device, fixpoint, result fetched) and relational queries through
`KernelProvider` (operators chained on the device, result fetched).

Every pass starts from relations that lie on the device as the host handed them in, evaluates on
fresh copies of them (a program that is run again has new facts: no index, packed copy or result of
an earlier pass is at hand) and fetches the result columns, which is the only way to a result that
the interface has.  One context per kind of work is kept, as a program keeps one.

A case fixes the structure of its graph or tables; the seed renames what is in them (vertices, keys,
groups), draws the values and shuffles the rows.  Another seed is then another input of the same
work, with a result of the same size.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from xlog_b200 import _abi as A
from xlog_b200 import programs, workloads
from xlog_b200.executor import Executor
from xlog_b200.provider import KernelProvider


def listed():
    return [
        # single-source reachability over a power-law graph: a query on a small graph, where launches
        # and waits are everything, and the benchmark configuration at full size (16 M edges)
        {"name": "reach_rmat_s10", "kind": "reach", "scale": 10, "edge_factor": 16},
        {"name": "reach_rmat_s20", "kind": "reach", "scale": 20, "edge_factor": 16},
        # full transitive closure of a small, cyclic, well connected graph (3.9 M tuples)
        {"name": "tc_uniform_2000", "kind": "tc_uniform", "nodes": 2000, "degree": 5},
        # a long chain: an iteration per node with next to nothing in it; ids are 64-bit values
        {"name": "tc_chain_1500_u64", "kind": "tc_chain", "nodes": 1500, "ids": "u64"},
        # complete blocks in a cycle whose ids are spread over millions: too wide for a bitmap
        {"name": "tc_blocks_128_sparse", "kind": "tc_blocks", "block": 128, "stride": 4096},
        # closure of the banded power-law DAG at a reduced scale: most candidates are known already
        {"name": "tc_dag_s14", "kind": "tc_dag", "scale": 14},
        # same generation over a tree with cross edges: a three-atom rule, a large dense result
        {"name": "sg_tree_7001", "kind": "sg", "nodes": 7001},
        # points-to analysis: four rules, two of them with three atoms, over Zipf facts
        {"name": "andersen_0.0005", "kind": "andersen", "scale": 0.0005},
        # semi join, inner join and aggregation: a lookup-sized query, and an analysis-sized one over
        # 64-bit keys
        {"name": "query_3001_u32", "kind": "query", "rows": 3001, "keys": "u32"},
        {"name": "query_4M_u64", "kind": "query", "rows": 4000037, "keys": "u64"},
        # one semi-naive step by operators: candidates sorted and deduplicated, known ones taken off,
        # the rest merged into the relation
        {"name": "step_3M_into_4M", "kind": "step", "rows": 3000017, "full": 4000000, "bits": 12},
        # events ordered by (id, time) with a payload carried along
        {"name": "sort_events_4M", "kind": "sort", "rows": 4000003, "types": "u32,i64,f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reach", "tc_uniform", "tc_chain", "tc_blocks", "tc_dag", "sg", "andersen", "query", "step", "sort"])
    if kind == "reach":
        return {"kind": kind, "scale": rng.randint(10, 20), "edge_factor": rng.randint(4, 16)}
    if kind == "tc_uniform":
        return {"kind": kind, "nodes": _log(rng, 100, 2000), "degree": rng.randint(2, 5)}
    if kind == "tc_chain":
        return {"kind": kind, "nodes": _log(rng, 100, 1500), "ids": rng.choice(["u32", "u64"])}
    if kind == "tc_blocks":
        return {"kind": kind, "block": _log(rng, 16, 128), "stride": rng.choice([1024, 4096])}
    if kind == "tc_dag":
        return {"kind": kind, "scale": rng.randint(10, 14), "edge_factor": rng.randint(4, 8)}
    if kind == "sg":
        return {"kind": kind, "nodes": _log(rng, 300, 7001)}
    if kind == "andersen":
        return {"kind": kind, "scale": round(math.exp(rng.uniform(math.log(0.0001), math.log(0.0005))), 7)}
    if kind == "query":
        return {"kind": kind, "rows": _log(rng, 1000, 4000037), "keys": rng.choice(["u32", "u64"])}
    if kind == "step":
        return {"kind": kind, "rows": _log(rng, 1000, 3000017), "full": _log(rng, 1000, 4000000), "bits": rng.randint(12, 20)}
    return {"kind": kind, "rows": _log(rng, 1000, 4000003), "types": rng.choice(["u32,u32", "u32,u32,u32", "u32,i64,f32"])}


# ---- inputs -----------------------------------------------------------------------------------
_CONTEXTS: dict = {}


def _context(kind):
    """One context (and executor) per kind of work, for the life of the process."""
    if kind not in _CONTEXTS:
        prov = KernelProvider(device=0)
        _CONTEXTS[kind] = (prov, Executor(prov))
    return _CONTEXTS[kind]


STRUCTURE = 20


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _u32(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def _uniform(g, n, below):
    return torch.randint(0, below, (n,), generator=g, device="cuda", dtype=torch.int64)


def _shuffled(cols, seed):
    """The rows in a seeded order: relations do not arrive sorted."""
    perm = np.random.RandomState(seed % (1 << 32)).permutation(len(cols[0]))
    return [np.ascontiguousarray(c[perm]) for c in cols]


def _rmat(scale, edge_factor):
    """R-MAT edges (a=.57 b=.19 c=.19 d=.05, 16-bit thresholds) without loops and duplicates: the
    distribution of `workloads.rmat_graph`, drawn on the device.  Packed (source << 32) | target."""
    g = _generator(STRUCTURE)
    m = edge_factor << scale
    ta, tb, tc = (int(round(x * 65536)) for x in (0.57, 0.57 + 0.19, 0.57 + 0.19 + 0.19))
    s = torch.zeros(m, dtype=torch.int32, device="cuda")
    d = torch.zeros(m, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        x = torch.randint(0, 65536, (m,), generator=g, device="cuda", dtype=torch.int32)
        s = (s << 1) | (x >= tb).int()
        d = (d << 1) | (((x >= ta) & (x < tb)) | (x >= tc)).int()
    return torch.unique(((s.long() << 32) | d.long())[s != d])


def _program_inputs(case, seed):
    """(plan, relation name -> host columns, result name)."""
    kind = case["kind"]
    rng = np.random.RandomState(seed % (1 << 32))
    if kind == "reach":
        # vertices renamed by an exclusive or, which keeps the hubs' neighbourhoods together
        name = int(rng.randint(0, 1 << case["scale"]))
        k = _rmat(case["scale"], case["edge_factor"])
        k = k[torch.randperm(len(k), generator=_generator(seed), device="cuda")] ^ ((name << 32) | name)
        return programs.reach_from_source(name), {"edge": [_u32(k >> 32), _u32(k & 0xFFFFFFFF)]}, "r"
    if kind == "tc_uniform":
        names = rng.permutation(case["nodes"]).astype(np.uint32)
        c = workloads.uniform_digraph(case["nodes"], case["nodes"] * case["degree"], STRUCTURE)
        return programs.transitive_closure(), {"edge": _shuffled([names[x] for x in c], seed)}, "reach"
    if kind == "tc_chain":
        n = case["nodes"]
        plan = programs.transitive_closure()
        if case["ids"] == "u64":
            names = workloads.splitmix64(seed, 0, n)
            for rule in plan.sccs[0].rules:
                rule.head_types = (A.U64, A.U64)
        else:
            names = rng.permutation(n).astype(np.uint32)
        return plan, {"edge": _shuffled([names[:-1], names[1:]], seed)}, "reach"
    if kind == "tc_blocks":
        b, k = case["block"], 4
        names = np.arange(k * b, dtype=np.uint32) * np.uint32(case["stride"])
        names += rng.randint(0, case["stride"], k * b).astype(np.uint32)
        blocks = names.reshape(k, b)
        src = np.concatenate([np.repeat(blocks[i], b) for i in range(k)])
        dst = np.concatenate([np.tile(blocks[(i + 1) % k], b) for i in range(k)])
        return programs.transitive_closure(), {"edge": _shuffled([src, dst], seed)}, "reach"
    if kind == "tc_dag":
        name = np.uint32(rng.randint(0, 1 << case["scale"]))
        c = workloads.rmat_dag(case["scale"], case.get("edge_factor", 8), seed=STRUCTURE)
        return programs.transitive_closure(), {"edge": _shuffled([x ^ name for x in c], seed)}, "reach"
    if kind == "sg":
        name = np.uint32(rng.randint(0, 1 << (case["nodes"] - 1).bit_length()))
        c0, c1, _ = workloads.tree_dag(case["nodes"], 0.05, STRUCTURE)
        return programs.same_generation(), {"edge": _shuffled([c0 ^ name, c1 ^ name], seed)}, "sg"
    rels = workloads.andersen_program(case["scale"], STRUCTURE)
    variables = max(int(2_000_000 * case["scale"]), 16)
    heap = max(int(1_000_000 * case["scale"]), 8)
    names = np.concatenate([rng.permutation(variables), variables + rng.permutation(heap)]).astype(np.uint32)
    return programs.andersen(), {k: _shuffled([names[x] for x in v], seed) for k, v in rels.items()}, "pt"


def prepare(case, seed):
    kind = case["kind"]
    prov, ex = _context(kind)
    state = {"kind": kind, "prov": prov, "ex": ex}
    if kind in ("query", "step", "sort"):
        n = case["rows"]
        fixed, g = _generator(STRUCTURE), _generator(seed)
        if kind == "query":
            # facts (key, group, value), about a third of them active, two dimension rows per key on average
            groups, keys = max(n // 16, 1), max(n // 4, 1)
            if case["keys"] == "u64":
                names = workloads.splitmix64(seed, 0, keys)
            else:
                names = np.random.RandomState(seed % (1 << 32)).permutation(4 * keys)[:keys].astype(np.uint32)
            at = lambda m: names[_uniform(fixed, m, keys).cpu().numpy()]  # noqa: E731
            group = torch.randperm(groups, generator=g, device="cuda")[_uniform(fixed, n, groups)]
            state["fact"] = prov.create_buffer_from_slices([at(n), _u32(group), _u32(_uniform(g, n, 1 << 20))])
            state["active"] = prov.create_buffer_from_slices([at(max(n // 10, 1))])
            state["dim"] = prov.create_buffer_from_slices([at(max(n // 2, 1)), _u32(_uniform(g, max(n // 2, 1), 1 << 16))])
        elif kind == "step":
            d = 1 << case["bits"]
            name = int(_uniform(g, 1, d))
            pairs = lambda m: [_u32(_uniform(fixed, m, d) ^ name), _u32(_uniform(fixed, m, d) ^ name)]  # noqa: E731
            state["bag"] = prov.create_buffer_from_slices(pairs(n))
            state["full"] = prov.dedup_full_row(prov.create_buffer_from_slices(pairs(case["full"])))
        else:
            cols = []
            for i, t in enumerate(case["types"].split(",")):
                if t == "u32":  # ids, then a payload of any value
                    cols.append(_u32(_uniform(g, n, max(n // 8, 2) if i < 2 else 1 << 31)))
                elif t == "i64":  # times around zero, in microseconds
                    cols.append((_uniform(g, n, 1 << 40) - (1 << 39)).cpu().numpy())
                else:
                    cols.append(torch.randn(n, generator=g, device="cuda").cpu().numpy())
            state["rel"] = prov.create_buffer_from_slices(cols)
        return state
    plan, inputs, out = _program_inputs(case, seed)
    for name, rid in plan.rel_ids.items():
        ex.register_relation(rid, name)
    state["plan"] = plan.compile()
    state["inputs"] = {name: prov.create_buffer_from_slices(cols) for name, cols in inputs.items()}
    state["out"] = out
    return state


def run(state):
    prov, ex, kind = state["prov"], state["ex"], state["kind"]
    if kind == "query":
        fact = prov.hash_join_v2(state["fact"], state["active"], [0], [0], A.JOIN_SEMI)
        rows = prov.hash_join_v2(fact, state["dim"], [0], [0])   # key, group, value, key, weight
        return prov.download(prov.groupby_multi_agg(rows, [1], [(2, A.AGG_COUNT), (2, A.AGG_SUM), (4, A.AGG_MIN), (4, A.AGG_MAX)]))
    if kind == "step":
        bag = prov.clone_buffer(state["bag"])
        full = prov.clone_buffer(state["full"])
        new = prov.diff_gpu(prov.dedup_full_row(bag), full)
        return {"new": prov.download(new), "full": prov.download(prov.union_gpu(full, new))}
    if kind == "sort":
        return prov.download(prov.sort(state["rel"], [0, 1]))
    for name, buf in state["inputs"].items():
        ex.put_relation(name, prov.clone_buffer(buf))
    ex.execute_plan(state["plan"])
    result = prov.download(ex.get(state["out"]))
    ex.remove(state["out"])
    return result


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Bytes of the inputs read once and of the result written once (no path here multiplies).  Sizes
    of results that depend on the drawn data are the usual ones of that distribution."""
    kind = case["kind"]
    if kind == "reach":
        edges = 0.96 * case["edge_factor"] * 2 ** case["scale"]
        return {"bytes": 8 * edges + 4 * 0.55 * 2 ** case["scale"], "flops": 0}
    if kind == "tc_uniform":
        n, d = case["nodes"], case["degree"]
        share = {2: 0.63, 3: 0.88, 4: 0.96, 5: 0.98}[d]  # pairs connected in a random digraph of that degree
        return {"bytes": 8 * (n * d + share * n * n), "flops": 0}
    if kind == "tc_chain":
        n, w = case["nodes"], 16 if case["ids"] == "u64" else 8
        return {"bytes": w * (n + n * (n - 1) / 2), "flops": 0}
    if kind == "tc_blocks":
        return {"bytes": 8 * (4 * case["block"] ** 2 + 16 * case["block"] ** 2), "flops": 0}
    if kind == "tc_dag":
        m = case.get("edge_factor", 8) * 2 ** case["scale"]
        return {"bytes": 8 * (0.5 * m + 13.7e6 * 13 ** ((case["scale"] - 14) / 2)), "flops": 0}
    if kind == "sg":
        return {"bytes": 8 * (1.05 * case["nodes"] + 1.45e9 * (case["nodes"] / 60000) ** 2), "flops": 0}
    if kind == "andersen":
        s = case["scale"]
        return {"bytes": 8 * (7e6 * s + 0.44 * 2e6 * s * 1e6 * s), "flops": 0}
    n = case["rows"]
    if kind == "query":
        w = 8 if case["keys"] == "u64" else 4
        return {"bytes": n * (w + 8) + n // 10 * w + n // 2 * (w + 4) + n / 16 * 28, "flops": 0}
    if kind == "step":
        return {"bytes": 8 * (n + case["full"] + 0.75 * n + case["full"] + 0.75 * n), "flops": 0}
    return {"bytes": 2 * n * sum({"u32": 4, "i64": 8, "f32": 4}[t] for t in case["types"].split(",")), "flops": 0}


def tolerance(case):
    """Every result is a sorted set of tuples, a stable order or sums of whole numbers."""
    return "exact"
