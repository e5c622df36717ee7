"""Performance cases: what a user has this library do, through its public entry points.

Kinds of case:

* ``decompose``: a graph goes in (a host CSR for small graphs, a device CSR for
  large ones), the handle decomposes it, the final partition comes out;
* ``batch``: the same for many independent instances in one run;
* ``walk``: walk steps alone, then the potentials (the reference's
  iterateRandomWalk / readRandomWalkValues);
* ``rounds``: rounds driven stage by stage with every download the class offers;
* ``csr``: the CSR of an edge list built on the device;
* ``mtx``: a Matrix Market file read into a device CSR;
* ``hierarchy``: the expander hierarchy of a graph, level by level.

Graph families are those the library is configured, tested and benchmarked
with: planted partitions, 3D grids, R-MAT, near-regular graphs of the pairing
model, and batches of planted partitions.
"""
import math
import tempfile

import numpy as np
import torch

import parex_b200 as P
from parex_b200 import gpu_build, graphs, hierarchy, learn

DEVICE = "cuda:0"
CUT_FIELDS = ("label", "sparsity", "offset")
ORDER_FIELDS = ("nix", "prefix_volume", "prefix_edge_diff", "offset_in_cluster")


def listed():
    return [
        # the smoke-test graph: a request-sized graph, all latency
        {"name": "decompose_sbm2k", "kind": "decompose", "family": "sbm", "n": 2048, "blocks": 8, "d_in": 10.0,
         "d_out": 0.5, "input": "host", "schedule": "plain"},
        # the small configuration: planted partition with 16 blocks
        {"name": "decompose_sbm16k", "kind": "decompose", "family": "sbm", "n": 16384, "blocks": 16, "d_in": 12.0,
         "d_out": 0.5, "input": "host", "schedule": "plain"},
        # the mesh configuration: poor expansion, many split rounds and hundreds of thousands of clusters
        {"name": "decompose_grid128", "kind": "decompose", "family": "grid", "side": 128, "input": "device",
         "schedule": "plain"},
        # skewed degrees, plain form
        {"name": "decompose_rmat22", "kind": "decompose", "family": "rmat", "scale": 22, "edge_factor": 16,
         "input": "device", "schedule": "plain"},
        # the benchmark's graph and form: skewed degrees at full size, learned schedule
        {"name": "decompose_rmat24_learned", "kind": "decompose", "family": "rmat", "scale": 24, "edge_factor": 16,
         "input": "device", "schedule": "learned"},
        # an expander that is never split
        {"name": "decompose_regular22_learned", "kind": "decompose", "family": "regular", "n": 1 << 22, "degree": 8,
         "input": "device", "schedule": "learned"},
        # many uneven instances in one run (an eighth of the 512-instance configuration)
        {"name": "batch_sbm64", "kind": "batch", "count": 64, "n_lo": 1000, "n_hi": 1000000},
        # walk steps alone, the kernel the benchmark's roofline is quoted on
        {"name": "walk_rmat22", "kind": "walk", "family": "rmat", "scale": 22, "edge_factor": 16, "steps": 8},
        # stage by stage with downloads, a ragged size
        {"name": "rounds_grid65", "kind": "rounds", "family": "grid", "side": 65, "rounds": 3},
        # an edge list with duplicates and loops to a device CSR
        {"name": "csr_rmat22", "kind": "csr", "family": "rmat", "scale": 22, "edge_factor": 16, "keep": False},
        # the reference's input format, from a file
        {"name": "mtx_regular", "kind": "mtx", "family": "regular", "n": 200001, "degree": 8},
        # decompose and contract until one vertex is left
        {"name": "hierarchy_sbm16k", "kind": "hierarchy", "family": "sbm", "n": 16384, "blocks": 16, "d_in": 12.0,
         "d_out": 0.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_sbm(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return {"family": "sbm", "n": n, "blocks": rng.randint(2, min(64, n // 32)),
            "d_in": round(rng.uniform(4.0, 32.0), 2), "d_out": round(rng.uniform(0.1, 2.0), 2)}


def _draw_grid(rng, lo, hi):
    return {"family": "grid", "side": _log_int(rng, lo, hi)}


def _draw_rmat(rng, lo, hi):
    return {"family": "rmat", "scale": rng.randint(lo, hi), "edge_factor": rng.randint(6, 16)}


def _draw_regular(rng, lo, hi):
    return {"family": "regular", "n": _log_int(rng, lo, hi), "degree": 2 * rng.randint(2, 6)}


def draw(rng):
    kind = rng.choice(["small", "small", "large", "large", "large", "batch", "walk", "rounds", "csr", "mtx",
                       "hierarchy"])
    if kind == "small":
        g = rng.choice([lambda: _draw_sbm(rng, 1000, 100000), lambda: _draw_grid(rng, 8, 40),
                        lambda: _draw_rmat(rng, 10, 15), lambda: _draw_regular(rng, 500, 60000)])()
        return {"kind": "decompose", **g, "input": "host", "schedule": "plain"}
    if kind == "large":
        g = rng.choice([lambda: _draw_grid(rng, 41, 150), lambda: _draw_rmat(rng, 16, 23),
                        lambda: _draw_regular(rng, 60001, 4000001)])()
        schedule = "plain" if g["family"] == "grid" else rng.choice(["plain", "learned"])
        return {"kind": "decompose", **g, "input": "device", "schedule": schedule}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(8, 96), "n_lo": 1000, "n_hi": _log_int(rng, 20000, 500000)}
    if kind == "walk":
        g = rng.choice([lambda: _draw_rmat(rng, 14, 22), lambda: _draw_grid(rng, 20, 130),
                        lambda: _draw_regular(rng, 10001, 2000001)])()
        return {"kind": "walk", **g, "steps": rng.randint(1, 16)}
    if kind == "rounds":
        g = rng.choice([lambda: _draw_grid(rng, 12, 80), lambda: _draw_sbm(rng, 1000, 50000),
                        lambda: _draw_rmat(rng, 12, 18)])()
        return {"kind": "rounds", **g, "rounds": rng.randint(1, 4)}
    if kind == "csr":
        g = rng.choice([lambda: _draw_rmat(rng, 12, 22), lambda: _draw_regular(rng, 5001, 4000001)])()
        return {"kind": "csr", **g, "keep": rng.random() < 0.5}
    if kind == "mtx":
        return {"kind": "mtx", **_draw_regular(rng, 2001, 300001)}
    g = rng.choice([lambda: _draw_sbm(rng, 1000, 50000), lambda: _draw_grid(rng, 8, 40)])()
    return {"kind": "hierarchy", **g}


# ----------------------------------------------------------------------------
# inputs


def _vertices(case):
    family = case["family"]
    return case["side"] ** 3 if family == "grid" else 1 << case["scale"] if family == "rmat" else case["n"]


def _edge_samples(case):
    """Edges drawn, before duplicates merge (grids and planted partitions: edges expected)."""
    family = case["family"]
    if family == "grid":
        return 3 * case["side"] ** 2 * (case["side"] - 1)
    if family == "rmat":
        return case["edge_factor"] << case["scale"]
    if family == "regular":
        return case["n"] * case["degree"] // 2
    return int(case["n"] * (case["d_in"] + case["d_out"]) / 2)


def _device_edges(case, seed):
    """(u, v) int32 device tensors: loops and duplicates as the family gives them."""
    family = case["family"]
    if family == "rmat":
        return gpu_build.rmat_edges(case["scale"], case["edge_factor"], seed=seed)
    if family == "grid":
        s = case["side"]
        ids = torch.arange(s ** 3, dtype=torch.int32, device=DEVICE).view(s, s, s)
        pairs = [(ids[:, :, :-1], ids[:, :, 1:]), (ids[:, :-1, :], ids[:, 1:, :]), (ids[:-1], ids[1:])]
        return (torch.cat([a.reshape(-1) for a, _ in pairs]), torch.cat([b.reshape(-1) for _, b in pairs]))
    if family == "regular":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)
        stubs = torch.arange(case["n"] * case["degree"], device=DEVICE) // case["degree"]
        stubs = stubs[torch.randperm(stubs.numel(), generator=gen, device=DEVICE)].to(torch.int32)
        return stubs[0::2].contiguous(), stubs[1::2].contiguous()
    u, v = graphs.sbm(case["n"], case["blocks"], case["d_in"], case["d_out"], seed)
    return (torch.from_numpy(u.astype(np.int32)).to(DEVICE), torch.from_numpy(v.astype(np.int32)).to(DEVICE))


def _device_graph(case, seed):
    n = _vertices(case)
    u, v = _device_edges(case, seed)
    offsets, cols, m = gpu_build.build_csr(n, u, v)
    return offsets, cols.clone(), n, m


def _same_graph(case):
    """Cases whose graph is the same for every seed, so that their inputs differ by the walk's seed: a grid is one
    graph, a batch keeps its instances and stage-by-stage runs compare walks on one graph."""
    return case["kind"] in ("batch", "rounds") or case["family"] == "grid"


def _graph_seed(case, seed):
    return 1 if _same_graph(case) else seed


def _walk_seed(case, seed):
    return seed % (1 << 31) if _same_graph(case) else 6582


def _manager(case, seed):
    dm = P.CudaDeviceManager(seed=_walk_seed(case, seed))
    if case.get("schedule") == "learned":
        model = learn.Model.load()
        dm.set_schedule(P._lib.SCHEDULE_LEARNED, model.weights, model.norm, **learn.SHIPPED_SCHEDULE)
    return dm


def _page_locked(n):
    return torch.empty(n, dtype=torch.int32, pin_memory=True).numpy()


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind == "csr":
        state["n"] = _vertices(case)
        state["u"], state["v"] = _device_edges(case, seed)
        # the program's own columns, sized for every edge drawn
        state["cols"] = torch.zeros(2 * state["u"].numel(), dtype=torch.int32, device=DEVICE)
        return state
    if kind == "mtx":
        u, v = _device_edges(case, seed)
        n, lines = case["n"], zip((u + 1).tolist(), (v + 1).tolist())
        state["file"] = tempfile.NamedTemporaryFile(mode="w", suffix=".mtx")
        state["file"].write("%%%%MatrixMarket matrix coordinate pattern symmetric\n%d %d %d\n" % (n, n, u.numel()))
        state["file"].write("\n".join(["%d %d" % p for p in lines]) + "\n")
        state["file"].flush()
        return state
    if kind == "batch":
        offsets, cols, n, m, starts = gpu_build.sbm_batch(case["count"], _graph_seed(case, seed), case["n_lo"],
                                                          case["n_hi"])
        state.update(offsets=offsets, cols=cols.clone(), n=n, m=m, starts=starts, dm=_manager(case, seed),
                     ids=_page_locked(n))
        return state
    offsets, cols, n, m = _device_graph(case, _graph_seed(case, seed))
    if case.get("input") == "host":
        state["graph"] = gpu_build.to_host(offsets, cols)
    else:
        state.update(offsets=offsets, cols=cols, n=n, m=m)
        if kind == "decompose":
            state["ids"] = _page_locked(n)
    if kind == "hierarchy":
        state["seed"] = _walk_seed(case, seed)
    else:
        state["dm"] = _manager(case, seed)
    return state


# ----------------------------------------------------------------------------
# passes


def _load(state):
    dm = state["dm"]
    if "graph" in state:
        dm.initialize(state["graph"])
    else:
        dm.initialize_device(state["n"], state["m"], state["offsets"].data_ptr(), False, state["cols"].data_ptr())
    return dm


def _finish(state):
    """What the reference's application takes from a decomposition (main.cpp): the partition and its cut.  Small
    graphs come back with the certificates and potentials too, large ones into page-locked memory."""
    dm = state["dm"]
    rounds = dm.expanderDecomposition()
    part = dm.getFinalPartition(state.get("ids"))
    out = {"rounds": rounds, "ids": part.clusterIds, "clusters": part.numClusters, "cut": dm.countCutEdges()}
    if "ids" not in state:
        out.update(certificates=dm.downloadCertificates(), potentials=dm.readRandomWalkValues())
    return out


def _padded(a, n):
    out = np.zeros(n, dtype=a.dtype)
    out[:a.shape[0]] = a
    return out


def _ancestors(levels, depth=8):
    """Every vertex's ancestor, the ancestor's volume and its cut at each of the first levels (the top one repeats)."""
    at, out = levels[0].parents, []
    for i in range(depth):
        level = levels[min(i, len(levels) - 1)]
        if 0 < i < len(levels):
            at = level.parents[at]
        out.append([at, level.volumes[at], level.cut_sizes[at]])
    return {"levels": len(levels), "ancestors": out}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "decompose":
        _load(state)
        return _finish(state)
    if kind == "batch":
        state["dm"].initialize_batched_device(state["n"], state["m"], state["offsets"].data_ptr(), False,
                                              state["cols"].data_ptr(), state["starts"])
        return _finish(state)
    if kind == "walk":
        dm = _load(state)
        for _ in range(case["steps"]):
            dm.iterateRandomWalk()
        return {"potentials": dm.readRandomWalkValues()}
    if kind == "rounds":
        dm = _load(state)
        out = []
        for _ in range(case["rounds"]):
            dm.iterateRandomWalk()
            dm.computeSweepCuts()
            order, cuts = dm.downloadPartition(), dm.readSweepCuts()
            dm.cutClusters()
            out.append({"order": [_padded(order[f], dm.n) for f in ORDER_FIELDS],
                        "cuts": [_padded(cuts.cuts[f], dm.n) for f in CUT_FIELDS],
                        "labels": dm.downloadLabels(), "cut": dm.getNumCutEdges()})
        return {"rounds": out, "degrees": dm.downloadDegrees(), "potentials": dm.readRandomWalkValues(),
                "edges": dm.downloadActiveEdgeMap()}
    if kind == "csr":
        build = gpu_build.build_csr_finalize if case["keep"] else gpu_build.build_csr
        offsets, cols, m = build(state["n"], state["u"], state["v"])
        state["cols"][:2 * m] = cols
        return {"offsets": offsets, "cols": state["cols"], "m": m}
    if kind == "mtx":
        offsets, cols, n, m = gpu_build.read_mtx(state["file"].name)
        return {"offsets": offsets, "cols": cols, "n": n, "m": m}
    return _ancestors(hierarchy.build(state["offsets"], state["cols"], seed=state["seed"]))


def work(case):
    """Bytes: inputs once, outputs once.  Operations: one multiply-add per edge
    slot and walk step, with one step for a decomposition (it takes dozens,
    how many depends on the graph)."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        slots = n * 19.05
    else:
        n, slots = _vertices(case), 2 * _edge_samples(case)
    csr = 4 * (n + 1) + 4 * slots
    if kind == "csr":
        return {"bytes": 4 * slots + csr, "flops": 0}
    if kind == "mtx":
        return {"bytes": slots * (1 + math.log10(n)) + csr, "flops": 0}
    if kind == "walk":
        return {"bytes": csr + 4 * n, "flops": 2 * slots * case["steps"]}
    if kind == "rounds":
        return {"bytes": csr + (20 * n + 16) * case["rounds"] + 8 * n + 4 * slots, "flops": 2 * slots * case["rounds"]}
    if kind == "hierarchy":
        return {"bytes": csr + 4 * n, "flops": 2 * slots}
    return {"bytes": csr + (12 if case.get("input") == "host" else 4) * n, "flops": 2 * slots}


# ----------------------------------------------------------------------------
# 64-bit values


def _exact_x0(degrees, walk_seed):
    """x0[v] = N(0, sqrt(deg v)): the hashed seed, one step of the minimal-standard generator, the inverse normal
    distribution, all as the reference defines them (cuda/devRandomWalk.h:22-48)."""
    mask = 0xFFFFFFFF

    def mix(x):
        return (((x >> 16) ^ x) * 0x45D9F3B) & mask

    x = torch.arange(degrees.numel(), dtype=torch.int64, device=degrees.device) ^ walk_seed
    x = mix(mix(x))
    x = ((x >> 16) ^ x) % 2147483647
    x = torch.where(x == 0, torch.ones_like(x), x)
    u = (48271 * x) % 2147483647 - 1
    span = 2147483645
    upper = u > span // 2
    p = (torch.where(upper, span - u, u).double() + 0.5) / span
    z = -torch.special.ndtri(p)
    return torch.where(upper, z, -z) * degrees.double().sqrt()


def exact(case, seed):
    if case["kind"] != "walk":
        return None   # whole numbers, or potentials that follow from dozens of rounds of cuts
    offsets, cols, n, m = _device_graph(case, _graph_seed(case, seed))
    degrees = (offsets[1:] - offsets[:-1]).to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(n, device=DEVICE), degrees)
    x = _exact_x0(degrees, _walk_seed(case, seed))
    for _ in range(case["steps"]):
        spread = torch.where(degrees > 0, x / degrees.clamp(min=1), torch.zeros_like(x))
        total = torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add_(0, rows, spread[cols.long()])
        x = 0.9 * total + 0.1 * x
    return {"potentials": x}
