"""The calls this project is measured on: what a user's program asks of the PBILS solver, over its real range.

Each case is one call (or one batch of calls) through the public Python API: the one-call solver on a host graph,
the reusable solver on a device graph, the Neighborhood enumerators, the batched engine and the device recount.
Every output is a whole number (objectives, counts, labels, neighbour counts) and the same for the same seed.

A case's fields: `kind` names the entry point; `n`, `p` (edge probability; planted graphs: `p_in`, `p_out`), `k`,
`pop` (population), `iters`, `gww` and `count` (labelings of a recount, instances of a batch) its sizes.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import cuda_graph_clustering_b200 as ccb

MASK64 = (1 << 64) - 1


def listed():
    return [
        # An interactive call: a graph of a few hundred vertices in host memory, solved in one call.  Launch
        # latency, uploads and the per-move chain are all there is.
        {"name": "onecall_n200_k4", "kind": "onecall", "n": 200, "p": 0.4, "k": 4, "pop": 32, "iters": 20, "gww": 0.1},
        # The default benchmark: G(1000, 0.5), five clusters, the full 100 iterations.
        {"name": "solve_n1000_k5", "kind": "solve", "n": 1000, "p": 0.5, "k": 5, "pop": 128, "iters": 100, "gww": 0.1},
        # A row of the published cluster-count sweep: n = 2000, up to 32 clusters, 20 iterations.
        {"name": "solve_n2000_k32", "kind": "solve", "n": 2000, "p": 0.33, "k": 32, "pop": 128, "iters": 20,
         "gww": 0.0},
        # The published population sweep: n = 6000, k = 3, more slots than the device has SMs.
        {"name": "solve_n6000_k3_pop512", "kind": "solve", "n": 6000, "p": 0.33, "k": 3, "pop": 512, "iters": 4,
         "gww": 0.0},
        # The published size sweep, an upper row of it.
        {"name": "solve_n16000_k3", "kind": "solve", "n": 16000, "p": 0.33, "k": 3, "pop": 128, "iters": 3,
         "gww": 0.0},
        # Many clusters on a large graph of ragged size, the heavy end of the batched and serving mixes.
        {"name": "solve_n9001_k24", "kind": "solve", "n": 9001, "p": 0.2, "k": 24, "pop": 64, "iters": 1, "gww": 0.1},
        # The largest graphs of the 16-bit path.
        {"name": "solve_n32000_k8", "kind": "solve", "n": 32000, "p": 0.33, "k": 8, "pop": 128, "iters": 1,
         "gww": 0.1},
        # The wide path (more than 32767 vertices): sparse G(65536, 0.02), two clusters, then three.
        {"name": "wide_n65536_k2", "kind": "solve", "n": 65536, "p": 0.02, "k": 2, "pop": 128, "iters": 2,
         "gww": 0.1},
        {"name": "wide_n65536_k3", "kind": "solve", "n": 65536, "p": 0.02, "k": 3, "pop": 128, "iters": 1,
         "gww": 0.1},
        # The Neighborhood algorithm with a local search from every closed neighbourhood of a planted graph.
        {"name": "neighborhood_ls_n4096", "kind": "neighborhood", "n": 4096, "p_in": 0.6, "p_out": 0.1, "k": 2,
         "pop": 128, "ls": True},
        # A mixed batch of independent instances (sizes, cluster counts and populations of the batched mix).
        {"name": "batch_24", "kind": "batch", "count": 24, "max_n": 5000, "iters": 5},
        # The recount of one solution (the command line's check of its result), with sizes and neighbour counts.
        {"name": "recount_n20000_k16", "kind": "recount", "n": 20000, "p": 0.1, "k": 16, "count": 1, "tensor": False},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["onecall", "few", "few", "many", "many", "wide", "neighborhood", "batch", "recount"])
    if kind == "onecall":
        return {"kind": "onecall", "n": _log_int(rng, 60, 700), "p": round(rng.uniform(0.1, 0.6), 3),
                "k": rng.randint(2, 8), "pop": rng.choice([16, 32, 64]), "iters": rng.randint(5, 20),
                "gww": rng.choice([0.0, 0.1])}
    if kind in ("few", "many"):
        few = kind == "few"
        n = _log_int(rng, 500, 32000) if few else _log_int(rng, 300, 12000)
        k = rng.randint(2, 8) if few else rng.randint(9, 64)
        pop = rng.choice([32, 64, 128, 256] if n < 8000 and few else [32, 64, 128])
        # seconds of an iteration, roughly: the first descent moves most vertices, each move's cost grows with n
        cost = -(-pop // 128) * n * (400.0 + (0.4 if few else 1.8) * n) * 1e-9
        iters = max(1, min(20, int(0.4 / cost)))
        return {"kind": "solve", "n": n, "p": round(rng.uniform(0.1, 0.5), 3), "k": k, "pop": pop, "iters": iters,
                "gww": rng.choice([0.0, 0.1])}
    if kind == "wide":
        n = rng.randint(33000, 65536)
        return {"kind": "solve", "n": n, "p": round(rng.uniform(0.01, 0.03), 4), "k": rng.choice([2, 3]),
                "pop": rng.choice([32, 64, 128]), "iters": 1, "gww": 0.1}
    if kind == "neighborhood":
        ls = rng.random() < 0.5
        return {"kind": "neighborhood", "n": _log_int(rng, 300, 4096 if ls else 10000),
                "p_in": round(rng.uniform(0.4, 0.7), 3), "p_out": round(rng.uniform(0.05, 0.2), 3), "k": 2,
                "pop": rng.choice([64, 100, 128]), "ls": ls}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(8, 28), "max_n": _log_int(rng, 1000, 5000),
                "iters": rng.randint(2, 5)}
    return {"kind": "recount", "n": _log_int(rng, 500, 24000), "p": round(rng.uniform(0.05, 0.5), 3),
            "k": rng.randint(2, 64), "count": _log_int(rng, 1, 64), "tensor": rng.random() < 0.3}


# ---- inputs -------------------------------------------------------------------------------------------------

def _solver_params(case, seed):
    return ccb.PbilsParams(k=case["k"], population=case["pop"], iterations=case["iters"],
                           early_stop=case["iters"] + 1, gww=case["gww"], seed=seed * 7 + 3)


def _packed_graph(n, words, generator, probability, community=None):
    """A random symmetric bitset [n, words] int32 on the GPU and its edge count; `probability` is a number or, with
    `community`, the pair (inside, across)."""
    a = torch.rand(n, n, generator=generator, device="cuda")
    if community is None:
        a = a < probability
    else:
        same = community[:, None] == community[None, :]
        a = torch.where(same, a < probability[0], a < probability[1])
    a = torch.triu(a, 1)
    edges = int(a.sum())
    a = a | a.T
    bits = torch.zeros(n, words, dtype=torch.int32, device="cuda")
    weights = torch.tensor([1 << b for b in range(32)], dtype=torch.int64, device="cuda")
    for r0 in range(0, n, 2048):
        rows = torch.zeros(min(2048, n - r0), words * 32, dtype=torch.bool, device="cuda")
        rows[:, :n] = a[r0:r0 + rows.shape[0]]
        sums = (rows.view(rows.shape[0], words, 32).to(torch.int64) * weights).sum(-1)
        bits[r0:r0 + rows.shape[0]] = torch.where(sums >= 1 << 31, sums - (1 << 32), sums).to(torch.int32)
    return bits, edges


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _planted_inputs(case, seed):
    g = _generator(seed)
    n = case["n"]
    community = torch.randint(0, 2, (n,), generator=g, device="cuda")
    return _packed_graph(n, (n + 31) // 32, g, (case["p_in"], case["p_out"]), community)


def _recount_inputs(case, seed):
    g = _generator(seed)
    n, k, count = case["n"], case["k"], case["count"]
    words = (n + 127) // 128 * 4  # rows of whole 16-byte groups, as the device graph store has them
    bits, edges = _packed_graph(n, words, g, case["p"])
    labels = torch.randint(0, k, (count, n), generator=g, device="cuda", dtype=torch.int32)
    return bits, edges, words, labels


def _batch_instances(case, seed):
    """The batch's instances: the case fixes their sizes, the seed their graphs and trajectories."""
    rng = random.Random(case["count"] * 1009 + case["max_n"])
    seeds = random.Random(seed)
    out = []
    for _ in range(case["count"]):
        n = _log_int(rng, 200, case["max_n"])
        out.append({"n": n, "parts": rng.randint(2, 16), "p_in": rng.uniform(0.3, 0.8),
                    "p_out": rng.uniform(0.01, 0.2), "flip": rng.uniform(0.05, 0.2), "k": rng.randint(2, 64),
                    "pop": rng.choice([32, 64, 128]), "graph_seed": seeds.getrandbits(60), "seed": seeds.getrandbits(60)})
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "onecall":
        graph = ccb.Graph.ErdosRenyi(case["n"], case["p"], seed + 1)
        return {"kind": kind, "graph": graph, "params": _solver_params(case, seed)}
    if kind == "solve":
        graph = ccb.DeviceGraph.erdos_renyi(case["n"], case["p"], seed + 1)
        params = _solver_params(case, seed)
        return {"kind": kind, "graph": graph, "params": params, "solver": ccb.Solver(graph, params)}
    if kind == "neighborhood":
        bits, edges = _planted_inputs(case, seed)
        torch.cuda.synchronize()
        graph = ccb.DeviceGraph(device_ptr=bits.data_ptr(), n=case["n"], words=bits.shape[1], edges=edges)
        params = ccb.PbilsParams(k=2, population=case["pop"])
        return {"kind": kind, "graph": graph, "params": params, "ls": case["ls"], "solver": ccb.Solver(graph, params)}
    if kind == "batch":
        batch, ids = ccb.Batch(), []
        for i in _batch_instances(case, seed):
            graph, _ = ccb.DeviceGraph.planted(i["n"], i["parts"], i["p_in"], i["p_out"], i["flip"], i["graph_seed"])
            ids.append(batch.add(graph, ccb.PbilsParams(k=i["k"], population=i["pop"], iterations=case["iters"],
                                                        early_stop=case["iters"] + 1, seed=i["seed"])))
        return {"kind": kind, "batch": batch, "ids": ids}
    bits, edges, words, labels = _recount_inputs(case, seed)
    n, k, count = case["n"], case["k"], case["count"]
    return {"kind": kind, "tensor": case["tensor"], "n": n, "words": words, "edges": edges, "k": k, "count": count,
            "bits": bits, "labels": labels, "f": torch.empty(count, dtype=torch.int64, device="cuda"),
            "sizes": torch.empty(count, k, dtype=torch.int32, device="cuda"),
            "g": torch.empty(count, k, n, dtype=torch.int32, device="cuda")}


# ---- one pass -----------------------------------------------------------------------------------------------

def _numbers(r):
    return {"objective": r.objective, "labels": r.labels, "iterations": r.iterations_done,
            "clusters": r.clusters_used, "searches": r.local_searches, "moves": r.accepted_moves}


def run(state):
    kind = state["kind"]
    if kind == "onecall":
        return _numbers(ccb.SolveGpu(state["graph"], state["params"]))
    if kind == "solve":
        return _numbers(state["solver"].pbils(state["params"]))
    if kind == "neighborhood":
        return _numbers(state["solver"].neighborhood(state["params"], state["ls"]))
    if kind == "batch":
        state["batch"].run()
        results = [state["batch"].result(i) for i in state["ids"]]
        return {"objective": np.array([r.objective for r in results], np.int64),
                "moves": np.array([r.accepted_moves for r in results], np.int64),
                "labels": np.concatenate([r.labels for r in results])}
    call = ccb.evaluate_labelings_tensor if state["tensor"] else ccb.evaluate_labelings
    call(state["bits"].data_ptr(), state["n"], state["words"], state["edges"], state["k"], state["count"],
         state["labels"].data_ptr(), state["f"].data_ptr(), state["sizes"].data_ptr(), state["g"].data_ptr(),
         torch.cuda.current_stream().cuda_stream)
    return {"f": state["f"], "sizes": state["sizes"], "g": state["g"]}


# ---- what a pass cannot do without --------------------------------------------------------------------------

def _solve_work(n, p, k, pop, iters):
    """One solve: the bitset read once and the labels written once; integer operations: the neighbour counts of every
    labeling built once per iteration (an update for each end of each edge) and, for each move of the descents (about
    n in the first, then about half the vertices), two counters of each neighbour of the moved vertex."""
    degree = p * n
    moves = pop * n * (1.0 + 0.5 * (iters - 1))
    return n * ((n + 31) // 32) * 4 + 4 * n, pop * (iters + 1) * n * degree + 2.0 * moves * degree


def work(case):
    kind = case["kind"]
    if kind in ("onecall", "solve"):
        b, ops = _solve_work(case["n"], case["p"], case["k"], case["pop"], case["iters"])
    elif kind == "neighborhood":
        n = case["n"]
        degree = 0.5 * (case["p_in"] + case["p_out"]) * n
        # every closed neighbourhood's intra-cluster edges; with local searches about n / 4 moves from each
        b, ops = n * ((n + 31) // 32) * 4 + 4 * n, n * n * degree + (2.0 * n * (n / 4) * degree if case["ls"] else 0.0)
    elif kind == "batch":
        b, ops = 0.0, 0.0
        for i in _batch_instances(case, 1):
            p = i["p_in"] / i["parts"] + i["p_out"] * (1 - 1 / i["parts"])
            p = p * (1 - i["flip"]) + (1 - p) * i["flip"]
            bi, oi = _solve_work(i["n"], p, i["k"], i["pop"], case["iters"])
            b, ops = b + bi, ops + oi
    else:
        n, k, count = case["n"], case["k"], case["count"]
        b = n * ((n + 31) // 32) * 4 + 4 * count * n + 8 * count + 4 * count * k + 4 * count * k * n
        ops = count * n * case["p"] * n
    return {"bytes": float(b), "flops": float(ops)}


# ---- the same answers by plain numpy / torch ----------------------------------------------------------------

def _mix(z):
    z = ((z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9))
    z = ((z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB))
    return z ^ (z >> np.uint64(31))


_GAMMA = np.uint64(0x9E3779B97F4A7C15)


def _stream(seed, stream, step):
    """The carried state of the solver's (seed, stream, step) random streams; stream may be an array."""
    s = np.uint64(seed) ^ (np.asarray(stream, np.uint64) * np.uint64(0xD1B54A32D192ED03)) ^ \
        np.uint64((step * 0xA0761D6478BD642F) & MASK64)
    return s + _GAMMA


def _draw(state):
    state = state + _GAMMA
    return state, _mix(state) >> np.uint64(32)


def _below(word, bound):
    return ((word * np.uint64(bound)) >> np.uint64(32)).astype(np.int64)


def _numpy_pbils(adjacency, k, pop, iters, gww, tournament, perturbation, seed):
    """The PBILS of the solver's interface (steepest descents in lock step over the population), in numpy int64."""
    n = adjacency.shape[0]
    a = adjacency.astype(np.int64)
    edges = int(a.sum()) // 2
    index = np.arange(pop * n, dtype=np.uint64).reshape(pop, n)

    def fitness(lab):
        onehot = (lab[:, None, :] == np.arange(k)[None, :, None]).astype(np.int64)
        g = onehot @ a
        size = onehot.sum(2)
        intra = (g * onehot).sum((1, 2))
        return g, size, edges + (size * (size - 1) // 2).sum(1) - intra

    _, word = _draw(_stream(int(_stream(seed, 0xA11CE, 0)), index, 0))
    cur = _below(word, k)
    _, _, f = fitness(cur)
    best, stall, moves = int(f.min()), 0, 0
    labels = cur[int(f.argmin())].copy()
    select, disturb = int(_stream(seed, 0x5E1EC7, 0)), int(_stream(seed, 0xBEEF, 0))
    for it in range(iters):
        state, word = _draw(_stream(select, np.arange(pop), it + 1))
        chosen = _below(word, pop)
        for _ in range(tournament - 1):
            state, word = _draw(state)
            other = _below(word, pop)
            chosen = np.where(f[other] < f[chosen], other, chosen)
        nxt = cur[chosen].copy()
        g, size, fn = fitness(nxt)
        live = np.arange(pop)
        while live.size:
            h = size[live][:, :, None] - 2 * g[live]
            own = np.take_along_axis(h, nxt[live][:, None, :], 1)[:, 0]
            np.put_along_axis(h, nxt[live][:, None, :], 1 << 40, 1)
            target = h.argmin(1)
            gain = np.take_along_axis(h, target[:, None, :], 1)[:, 0] - own + 1
            v = gain.argmin(1)
            at = np.arange(live.size)
            keep = gain[at, v] < 0
            live, v, to, d = live[keep], v[keep], target[at, v][keep], gain[at, v][keep]
            frm = nxt[live, v]
            g[live, frm] -= a[v]
            g[live, to] += a[v]
            size[live, frm] -= 1
            size[live, to] += 1
            nxt[live, v] = to
            fn[live] += d
            moves += live.size
        if int(fn.min()) < best:
            best, stall = int(fn.min()), 0
            labels = nxt[int(fn.argmin())].copy()
        else:
            stall += 1
        source = np.arange(pop)
        copies = int(gww * pop)
        if copies:
            order = np.lexsort((np.arange(pop), fn))
            source[order[::-1][:copies]] = order[:copies]
        nxt = nxt[source]
        state, word = _draw(_stream(disturb, index, it + 0x5000000))
        moved = (word >> np.uint64(8)).astype(np.float32) * np.float32(1 / 16777216) < np.float32(perturbation)
        _, word = _draw(state)
        cur = np.where(moved, (nxt + 1 + _below(word, k - 1)) % k, nxt)
        _, _, f = fitness(cur)
    return {"objective": best, "labels": labels.astype(np.int32), "iterations": iters,
            "clusters": int(np.unique(labels).size), "searches": iters * pop, "moves": moves}


def _numpy_erdos_renyi(n, p, seed):
    pairs = n * (n - 1) // 2
    first = np.uint64(int(_stream(seed, 0xE4D05F, 0)))
    with np.errstate(over="ignore"):
        word = _mix(first + _GAMMA * np.arange(1, pairs + 1, dtype=np.uint64)) >> np.uint64(32)
    joined = (word >> np.uint64(8)).astype(np.float64) / 16777216.0 < p
    a = np.zeros((n, n), bool)
    a[np.tril_indices(n, -1)] = joined
    return a | a.T


def _unpack(bits, n):
    shifts = torch.arange(32, device="cuda", dtype=torch.int32)
    return ((bits[:, :, None] >> shifts) & 1).reshape(bits.shape[0], -1)[:, :n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "onecall" and case["n"] * case["pop"] * case["iters"] * case["k"] <= 1 << 20:
        with np.errstate(over="ignore"):
            a = _numpy_erdos_renyi(case["n"], case["p"], seed + 1)
            return _numpy_pbils(a, case["k"], case["pop"], case["iters"], case["gww"], 5, 0.4, seed * 7 + 3)
    if kind == "neighborhood" and not case["ls"]:
        bits, edges = _planted_inputs(case, seed)
        n = case["n"]
        a = _unpack(bits, n).to(torch.float64)
        degree = a.sum(1)
        triangles = torch.empty(n, dtype=torch.float64, device="cuda")
        for r0 in range(0, n, 2048):
            rows = a[r0:r0 + 2048]
            triangles[r0:r0 + 2048] = ((rows @ a) * rows).sum(1) / 2
        # the closed neighbourhood of v against the rest: its inner edges, the rest's, and the pairs of each side
        inside = degree + triangles
        cut = (a @ degree) + degree - 2 * inside
        size = degree + 1
        f = edges + size * (size - 1) / 2 + (n - size) * (n - size - 1) / 2 - 2 * (edges - cut)
        v = int(torch.argmin(f))
        best = int(f[v])
        v = int(torch.nonzero(f == f[v])[0])
        labels = np.ones(n, np.int32)
        labels[(a[v] > 0).cpu().numpy()] = 0
        labels[v] = 0
        return {"objective": best, "labels": labels, "iterations": 0, "clusters": int(np.unique(labels).size),
                "searches": 0, "moves": 0}
    if kind == "recount":
        bits, edges, words, labels = _recount_inputs(case, seed)
        n, k, count = case["n"], case["k"], case["count"]
        f = torch.empty(count, dtype=torch.int64, device="cuda")
        sizes = torch.empty(count, k, dtype=torch.int32, device="cuda")
        g = torch.empty(count, k, n, dtype=torch.int32, device="cuda")
        onehot = (labels[:, None, :] == torch.arange(k, device="cuda")[None, :, None]).reshape(count * k, n)
        for r0 in range(0, n, 1024):
            rows = _unpack(bits[r0:r0 + 1024], n).to(torch.float64)
            for c0 in range(0, count * k, 256):
                part = onehot[c0:c0 + 256].to(torch.float64) @ rows.T
                g.view(count * k, n)[c0:c0 + 256, r0:r0 + 1024] = part.to(torch.int32)
        sizes.copy_(onehot.view(count, k, n).sum(2).to(torch.int32))
        own = torch.gather(g, 1, labels[:, None, :].long())[:, 0].to(torch.int64).sum(1)
        s = sizes.to(torch.int64)
        f.copy_(edges + (s * (s - 1) // 2).sum(1) - own)
        return {"f": f, "sizes": sizes, "g": g}
    return None
