"""The work that users of graph_analyzer_b200 have it do, as cases that can be timed.

A case names an operation and the graph it runs on. The graphs are the shapes the framework's own benchmark and tests
use: Holme-Kim graphs (a few hundred to 1.7M vertices, heavy-tailed degrees, many triangles per edge), R-MAT graphs
(2^10 to 2^22 vertices, the skewed degrees of web and social graphs) and packed batches of Holme-Kim graphs. The
operations are the public entry points of the package: counts on a resident graph, one-shot counts from host memory,
per-edge and per-vertex supports, participation counts under an alive mask, batch peeling, (k, triangle)-cores,
batches of graphs, a burst of serving requests and the densest-subgraph pipeline of the ga_dsg driver.
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import graph_analyzer_b200 as ga

RMAT_ABC = (0.57, 0.19, 0.19)

# Holme-Kim parameters of the benchmark's two named graphs
HK_SMALL = {"graph": "hk", "n": 8298, "m_lo": 12, "m_hi": 12, "p_hi": 0.0, "triad_p": 0.5}
HK_LARGE = {"graph": "hk", "n": 1_700_000, "m_lo": 6, "m_hi": 7, "p_hi": 0.54, "triad_p": 0.3}
RMAT_22 = {"graph": "rmat", "scale": 22, "edge_factor": 8.52}


def listed():
    return [
        # the smallest call: a count of a graph of some hundred vertices that the program keeps on the device, where
        # only the launch and the read of the result are left
        {"name": "count_hk_901", "op": "count", "graph": "hk", "n": 901, "m_lo": 5, "m_hi": 5, "p_hi": 0.0,
         "triad_p": 0.5},
        # a count of a large graph of short rows (the benchmark's 1.7M-vertex Holme-Kim graph), resident
        {"name": "count_hk_1700k", "op": "count", **HK_LARGE},
        # the headline: a count of a large graph of skewed degrees (R-MAT scale 22), resident
        {"name": "count_rmat_22", "op": "count", **RMAT_22},
        # one call from ordinary host arrays to the count, what a script does once per small graph
        {"name": "oneshot_hk_8298", "op": "oneshot", "pinned": False, **HK_SMALL},
        # the same from page-locked arrays at full size: upload, checks, index, count and release of a new graph
        {"name": "oneshot_rmat_22", "op": "oneshot", "pinned": True, **RMAT_22},
        # triangle support of every edge (k-truss and clustering work), left in the caller's device array
        {"name": "edge_supports_rmat_22", "op": "edge_supports", **RMAT_22},
        # per-vertex counts of an induced subgraph, host mask in and host counts out: one round of a caller's own loop
        {"name": "participation_hk_200k", "op": "participation", "alive": 0.8, "graph": "hk", "n": 200_003, "m_lo": 6,
         "m_hi": 7, "p_hi": 0.54, "triad_p": 0.5},
        # the peeling of the densest-subgraph approximation with its removal rounds, on a resident graph
        {"name": "peel_hk_1700k", "op": "peel", "num": 1, "den": 10, **HK_LARGE},
        # the largest call: the core decomposition of the headline graph, thousands of dependent rounds
        {"name": "cores_rmat_22", "op": "cores", **RMAT_22},
        # many graphs in one call (a dataset of graphs): the count and the peeling of each, with removal rounds
        {"name": "batch_hk_256", "op": "batch", "graphs": 256, "n_lo": 64, "n_hi": 262144, "num": 1, "den": 10},
        # a burst of requests to the server on registered graphs of mixed sizes, two counts to a peeling
        {"name": "serve_hk_48", "op": "serve", "graphs": 24, "requests": 48, "n_lo": 64, "n_hi": 262144, "num": 1,
         "den": 10},
        # the ga_dsg driver's pipeline on its usual graph: cores, greedy bound, prune, Greedy++ and CoreExact
        {"name": "densest_hk_8298", "op": "densest", **HK_SMALL},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_hk(rng, n_lo, n_hi):
    m_lo = rng.randint(2, 12)
    return {"graph": "hk", "n": _log_int(rng, n_lo, n_hi), "m_lo": m_lo, "m_hi": m_lo + rng.randint(0, 3),
            "p_hi": round(rng.uniform(0.0, 0.7), 3), "triad_p": round(rng.uniform(0.1, 0.7), 3)}


def _draw_graph(rng, hk_hi, scale_hi):
    if rng.random() < 0.5:
        return _draw_hk(rng, 300, hk_hi)
    return {"graph": "rmat", "scale": rng.randint(10, scale_hi), "edge_factor": round(rng.uniform(3.0, 8.52), 2)}


def draw(rng):
    op = rng.choice(["count", "count", "oneshot", "oneshot", "edge_supports", "vertex_supports", "participation",
                     "peel", "peel", "cores", "batch", "serve", "densest"])
    num, den = rng.choice([(1, 20), (1, 10), (1, 2)])
    if op == "batch":
        return {"op": op, "graphs": _log_int(rng, 4, 256), "n_lo": 64, "n_hi": _log_int(rng, 1000, 262144),
                "num": num, "den": den}
    if op == "serve":
        k = rng.randint(4, 24)
        return {"op": op, "graphs": k, "requests": k * rng.randint(1, 2), "n_lo": 64,
                "n_hi": _log_int(rng, 2000, 262144), "num": num, "den": den}
    if op == "densest":
        return {"op": op, **_draw_hk(rng, 300, 20_000)}
    if op == "cores":
        return {"op": op, **_draw_graph(rng, 300_000, 21)}
    case = {"op": op, **_draw_graph(rng, 1_700_000, 22)}
    if op == "oneshot":
        case["pinned"] = rng.random() < 0.5
    elif op == "participation":
        case["alive"] = round(rng.uniform(0.3, 1.0), 3)
    elif op == "peel":
        case.update(num=num, den=den)
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------

def _rmat_pairs(scale, edge_factor, seed):
    """Edge samples of an R-MAT graph with permuted ids, drawn on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + scale)
    k, (a, b, c) = int(edge_factor * (1 << scale)), RMAT_ABC
    u = torch.zeros(k, dtype=torch.int64, device="cuda")
    v = torch.zeros_like(u)
    for _ in range(scale):
        r = torch.rand(k, device="cuda", generator=gen)
        u = u * 2 + (r >= a + b)
        v = v * 2 + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    perm = torch.randperm(1 << scale, device="cuda", generator=gen)
    return perm[u], perm[v]


def _oriented(n, u, v):
    """Oriented CSR (rowptr, col) of an undirected pair list: loops and repeats dropped, every edge from its smaller
    to its larger endpoint in (degree, id) order, rows sorted."""
    lo, hi = torch.minimum(u, v), torch.maximum(u, v)
    keep = lo != hi
    key = torch.unique(lo[keep] * n + hi[keep])
    lo, hi = key // n, key % n
    deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
    swap = deg[lo] > deg[hi]
    src, dst = torch.where(swap, hi, lo), torch.where(swap, lo, hi)
    key = torch.sort(src * n + dst).values
    src, dst = key // n, key % n
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return rowptr, src, dst


def _csr(case, seed):
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        u, v = _rmat_pairs(case["scale"], case["edge_factor"], seed)
    else:
        n = case["n"]
        pairs = ga.gen_holme_kim(n, case["m_lo"], case["m_hi"], case["p_hi"], case["triad_p"], seed=seed + 1)
        p = torch.from_numpy(pairs.astype(np.int64)).cuda()
        u, v = p[:, 0], p[:, 1]
    return n, *_oriented(n, u, v)


def _host_graph(case, seed, pinned=False):
    n, rowptr, src, dst = _csr(case, seed)

    def host(t):
        out = torch.empty(t.numel(), dtype=torch.int32, pin_memory=pinned)
        out.copy_(t)
        return out.numpy().view(np.uint32)

    deg = rowptr[1:] - rowptr[:-1]
    return ga.Graph(n, dst.numel(), host(rowptr), host(dst), host(src), int(deg.max()))


def _shape(case, i):
    """Vertices and edges per vertex of graph i of a batch: sizes spread over the logarithm of the range, mean degrees 4
    to 32, in mixed order."""
    k = case["graphs"]
    at = (i * 37 + 11) % k if math.gcd(37, k) == 1 else i
    return int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** ((at + 0.5) / k)), 2 + (i * 5) % 15


def _graphs(case, seed):
    """The graphs of a batch, triad probabilities 0.1 to 0.7, built on several host threads."""
    k = case["graphs"]

    def one(i):
        n, m = _shape(case, i)
        pairs = ga.gen_holme_kim(n, m, m, 0.0, 0.1 + 0.6 * ((i * 7) % 11) / 10, seed=seed * 100003 + i + 1)
        return ga.graph_from_pairs(n, pairs, canonicalize=False)

    with ThreadPoolExecutor(16) as pool:
        return list(pool.map(one, range(k)))


def _edge_room(case):
    """Edges a graph of this case can have at most."""
    if case["graph"] == "rmat":
        return int(case["edge_factor"] * (1 << case["scale"]))
    return case["n"] * case["m_hi"]


def _alive(case, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 5)
    return (torch.rand(n, device="cuda", generator=gen) < case["alive"]).to(torch.uint8).cpu().numpy()


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": case}
    if op == "batch":
        state["batch"] = ga.DeviceBatch(ga.pack_batch(_graphs(case, seed)))
        return state
    if op == "serve":
        server = ga.Server(hbm_budget_bytes=20 << 30)
        ids = [server.add_graph(g) for g in _graphs(case, seed)]
        state.update(server=server, trace=[(ids[(7 * i) % len(ids)], ga.REQ_PEEL if i % 3 == 2 else ga.REQ_TC)
                                           for i in range(case["requests"])])
        return state
    g = _host_graph(case, seed, case.get("pinned", False))
    if op in ("oneshot", "densest"):
        state["graph"] = g
        return state
    state["dev"] = ga.DeviceGraph(g)
    state["dev"].prepare()
    if op == "edge_supports":
        state["sup"] = torch.zeros(_edge_room(case), dtype=torch.int32, device="cuda")   # one buffer for any graph
    elif op == "participation":
        state["alive"] = _alive(case, g.n, seed)
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------

def _densest(g):
    """The stages of the ga_dsg driver: core numbers, lower bound, prune, Greedy++ and CoreExact on what is left."""
    with ga.DeviceGraph(g) as d:
        cores = d.core_decomposition()
        num, den = d.core_level_density(cores.core, cores.kmax)
        greedy = d.greedy_pp(1)
    if greedy.verts and greedy.tri * max(den, 1) > num * greedy.verts:
        num, den = greedy.tri, greedy.verts
    pruned, old, core = ga.prune_to_core(g, cores.core, -(-num // den) if den else 0)
    with ga.DeviceGraph(pruned) as d:
        gpp = d.greedy_pp(10)
        best = d.core_exact(core, seed=gpp)

    def members(ids):   # a returned vertex set as a mask over the input's vertices
        mask = np.zeros(g.n, np.uint8)
        mask[ids] = 1
        return mask

    return {"core": cores.core, "kmax": cores.kmax, "rounds": cores.rounds, "pruned": members(old),
            "greedy": greedy.tri, "greedy_set": members(greedy.set), "gpp": gpp.tri,
            "gpp_set": members(old[gpp.set]), "best": best.tri, "best_set": members(old[best.set])}


def run(state):
    op, case = state["op"], state["case"]
    if op == "count":
        return {"triangles": state["dev"].tc_count()}
    if op == "oneshot":
        return {"triangles": ga.gpu_triangles(state["graph"])}
    if op == "edge_supports":
        return {"triangles": state["dev"].support_edges_device(state["sup"].data_ptr()), "sup": state["sup"]}
    if op == "vertex_supports":
        t, deg = state["dev"].support_vertices()
        return {"triangles": t, "deg": deg}
    if op == "participation":
        t, tri = state["dev"].participation(state["alive"])
        return {"triangles": t, "tri": tri}
    if op == "peel":
        p = state["dev"].batch_peel(case["num"], case["den"])
        return {"best_num": p.best_num, "best_den": p.best_den, "best_round": p.best_round, "rounds": p.rounds,
                "removed_round": p.removed_round}
    if op == "cores":
        c = state["dev"].core_decomposition()
        return {"core": c.core, "kmax": c.kmax, "rounds": c.rounds}
    if op == "batch":
        p = state["batch"].tc_peel(case["num"], case["den"])
        return {"triangles": p.triangles, "best_num": p.best_num, "best_den": p.best_den, "best_round": p.best_round,
                "rounds": p.rounds, "status": p.status, "removed_round": p.removed_round}
    if op == "serve":
        server = state["server"]
        tickets = [server.submit(gid, kind, case["num"], case["den"]) for gid, kind in state["trace"]]
        res = [server.wait(t) for t in tickets]
        return {"status": np.array([r.status for r in res]), "triangles": np.array([r.triangles for r in res]),
                "peel": np.array([[r.peel.best_num, r.peel.best_den, r.peel.best_round, r.peel.rounds]
                                  if kind == ga.REQ_PEEL else [0, 0, 0, 0]
                                  for r, (_, kind) in zip(res, state["trace"])])}
    return _densest(state["graph"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    """Each input read once, each output written once; the kernels do integer set operations, no floating point."""
    op = case["op"]
    if op in ("batch", "serve"):
        k = case["graphs"]
        asked = range(k) if op == "batch" else [(7 * i) % k for i in range(case["requests"])]
        return {"bytes": sum(8 * n + 4 * n * m + 40 for n, m in (_shape(case, i) for i in asked)), "flops": 0}
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        m = 0.97 * case["edge_factor"] * n                                       # repeats and loops dropped
    else:
        n = case["n"]
        m = n * (case["m_lo"] + (case["m_hi"] - case["m_lo"]) * case["p_hi"])
    out = {"count": 8, "oneshot": 8, "edge_supports": 4 * m, "vertex_supports": 8 * n, "participation": 5 * n,
           "peel": 4 * n, "cores": 4 * n, "densest": 8 * n}[op]
    return {"bytes": 4 * (n + 1) + 4 * m + out, "flops": 0}


# ---- the same results in plain torch -----------------------------------------------------------------------------

def _triangles(n, rowptr, src, dst, alive=None):
    """Every triangle as three edge positions (u->a, u->b, the edge between a and b), in pieces: the pairs of each
    row's entries that are joined by an edge."""
    key = src * n + dst
    partners = rowptr[src + 1] - 1 - torch.arange(dst.numel(), device="cuda")   # later entries of the same row
    ends = torch.cumsum(partners, 0)
    at, total = 0, dst.numel()
    while at < total:
        done = int(ends[at - 1]) if at else 0
        to = min(total, max(at + 1, int(torch.searchsorted(ends, done + (1 << 26), right=True))))
        first = torch.repeat_interleave(torch.arange(at, to, device="cuda"), partners[at:to])
        if first.numel():
            start = (ends - partners)[first] - done
            second = first + 1 + torch.arange(first.numel(), device="cuda") - start
            a, b = dst[first], dst[second]
            for x, y in ((a, b), (b, a)):
                want = x * n + y
                pos = torch.searchsorted(key, want).clamp_(max=total - 1)
                hit = key[pos] == want
                if alive is not None:
                    hit &= alive[src[first]] & alive[a] & alive[b]
                yield first[hit], second[hit], pos[hit]
        at = to


def _corners(n, rowptr, src, dst):
    parts = [(src[e], dst[e], dst[f]) for e, f, _ in _triangles(n, rowptr, src, dst)]
    return [torch.cat([p[i] for p in parts] or [src[:0]]) for i in range(3)]


def _counts(n, corners):
    return sum(torch.bincount(c, minlength=n) for c in corners)


def _exact_peel(n, corners, num, den):
    removed = torch.full((n,), 0xFFFFFFFF, dtype=torch.int64, device="cuda")
    alive = torch.ones(n, dtype=torch.bool, device="cuda")
    best, rnd = (0, 0, 0), 0
    while bool(alive.any()):
        t, k = corners[0].numel(), int(alive.sum())
        if best[1] == 0 or t * best[1] > best[0] * k:
            best = (t, k, rnd)
        out = alive & (_counts(n, corners) * (k * den) <= 3 * (den + num) * t)
        removed[out] = rnd
        alive &= ~out
        keep = alive[corners[0]] & alive[corners[1]] & alive[corners[2]]
        corners = [c[keep] for c in corners]
        rnd += 1
    return {"best_num": best[0], "best_den": best[1], "best_round": best[2], "rounds": rnd,
            "removed_round": removed.cpu().numpy().astype(np.uint32)}


def _exact_cores(n, corners):
    core = torch.zeros(n, dtype=torch.int64, device="cuda")
    alive = torch.ones(n, dtype=torch.bool, device="cuda")
    k = rounds = 0
    while bool(alive.any()):
        tri = _counts(n, corners)
        k = max(k, int(tri[alive].min()))
        out = alive & (tri <= k)
        core[out] = k
        alive &= ~out
        keep = alive[corners[0]] & alive[corners[1]] & alive[corners[2]]
        corners = [c[keep] for c in corners]
        rounds += 1
    return {"core": core.cpu().numpy().astype(np.uint32), "kmax": k, "rounds": rounds}


def exact(case, seed):
    op = case["op"]
    if op in ("batch", "serve", "densest"):
        return None
    size = 1 << case["scale"] if case["graph"] == "rmat" else case["n"]
    if op == "cores" and size > 20_000 or op == "peel" and case["graph"] == "rmat" and size > 1 << 19:
        return None   # thousands of rounds, or hundreds of millions of triangles held at once
    n, rowptr, src, dst = _csr(case, seed)
    if op in ("peel", "cores"):
        corners = _corners(n, rowptr, src, dst)
        return _exact_peel(n, corners, case["num"], case["den"]) if op == "peel" else _exact_cores(n, corners)
    alive = torch.from_numpy(_alive(case, n, seed)).cuda().bool() if op == "participation" else None
    total = 0
    sup = torch.zeros(_edge_room(case), dtype=torch.int64, device="cuda")
    per = torch.zeros(n, dtype=torch.int64, device="cuda")
    for e, f, h in _triangles(n, rowptr, src, dst, alive):
        total += e.numel()
        if op == "edge_supports":
            for t in (e, f, h):
                sup += torch.bincount(t, minlength=sup.numel())
        elif op in ("vertex_supports", "participation"):
            per += _counts(n, (src[e], dst[e], dst[f]))
    if op == "edge_supports":
        return {"triangles": total, "sup": sup.to(torch.int32)}
    if op == "vertex_supports":
        return {"triangles": total, "deg": per.cpu().numpy().astype(np.uint64)}
    if op == "participation":
        return {"triangles": total, "tri": per.cpu().numpy().astype(np.uint32)}
    return {"triangles": total}
