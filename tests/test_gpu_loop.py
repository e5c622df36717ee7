"""The graph driver's round loop, which graphs too large for the one-kernel
decomposition run through, and its hand-over of the last rounds, against the
CPU oracle: the shapes and options that the small graphs of the other tests no
longer take through it, and the states at its edges."""
import numpy as np
import pytest

import parex_b200 as P
from parex_b200 import graphs as G, learn
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _edges(n, e):
    e = np.asarray(e, dtype=np.int64).reshape(-1, 2)
    return G.csr_from_edges(e[:, 0], e[:, 1], n)


@pytest.mark.parametrize("driver", [P.DRIVER_GRAPH, P.DRIVER_STREAM])
@pytest.mark.parametrize("form", ["plain", "learned"])
def test_graph_without_vertices(driver, form):
    """Every call takes a graph of no vertices: no round runs, every result is empty."""
    dm = P.CudaDeviceManager(driver=driver)
    dm.initialize(G.CSRGraph(np.zeros(1, dtype=np.uint32), np.zeros(0, dtype=np.uint32), "none"))
    if form == "learned":
        model = learn.Model.load()
        dm.set_schedule(P._lib.SCHEDULE_LEARNED, model.weights, model.norm, **learn.SHIPPED_SCHEDULE)
    assert dm.expanderDecomposition() == 0
    dm.iterateRandomWalk()
    dm.computeSweepCuts()
    assert dm.downloadPartition().shape[0] == 0
    dm.cutClusters()
    assert dm.getNumClusters() == 0
    assert dm.getFinalPartition().numClusters == 0
    assert dm.getNumCutEdges() == 0


def _paths(count):
    """A batch of paths of 1 to 7 vertices and its instance starts."""
    sizes = 1 + np.arange(count) % 7
    starts = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    inner = np.ones(int(starts[-1]), dtype=bool)
    inner[starts[1:] - 1] = False
    at = np.nonzero(inner)[0]
    return _edges(int(starts[-1]), np.stack([at, at + 1], axis=1)), starts, sizes


def _batch_oracle(dm, g, sizes):
    count = sizes.shape[0]
    act = np.zeros(g.n, dtype=O.LNODE)
    labels = np.repeat(np.arange(count, dtype=np.int32), sizes)
    act["nix"], act["label"] = np.arange(g.n, dtype=np.uint32), labels
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_state(labels, act, dm.readRandomWalkValues().astype(np.float64),
                  np.diff(g.offsets.astype(np.int64)).astype(np.uint32), g.cols, count, 0)
    return orc


def _run_rounds(orc, rounds=None):
    """The oracle's rounds one by one: how many ran, and the last one's sweep order."""
    done, srt = 0, None
    while orc.n_active and orc.n_clusters and done != rounds:
        orc.walk()
        orc.sweep()
        srt = orc.sorted()
        orc.cut_clusters()
        done += 1
    return done, srt


def _check_sweep_order(dm, srt):
    part = dm.downloadPartition()
    for ours, theirs in (("nix", "nix"), ("prefix_edge_diff", "prefix_edge_diff"),
                         ("prefix_volume", "prefix_volume"), ("offset_in_cluster", "offset")):
        np.testing.assert_array_equal(part[ours], srt[theirs])


@pytest.mark.parametrize("cap", [200000, 2, 4])
def test_sweep_order_after_a_decomposition(cap):
    """Of the last round that ran: after a run handed over or stopped at its cap, then
    after one that ends in its first round and replays the first one's captured loop."""
    g, starts, sizes = _paths(12000)
    dm = P.CudaDeviceManager(max_rounds=cap)
    dm.initialize_batched(g, starts)
    orc = _batch_oracle(dm, g, sizes)
    try:
        rounds = dm.expanderDecomposition()
    except P.PxrError:
        rounds = cap
    done, srt = _run_rounds(orc, cap)
    assert done == rounds
    _check_sweep_order(dm, srt)

    dm.initialize_batched(g, starts)
    dm.set_potentials(np.zeros(g.n))      # no spread anywhere: every cluster is certified at once
    orc = _batch_oracle(dm, g, sizes)
    assert dm.expanderDecomposition() == 1
    done, srt = _run_rounds(orc)
    assert done == 1
    _check_sweep_order(dm, srt)


def _state(g, active, count, n_clusters):
    """Labels that spread the `count` paths of the first `active` vertices over
    [0, n_clusters) at an even step, the rest inactive."""
    sizes = 1 + np.arange(count) % 7
    labels = np.full(g.n, -1, dtype=np.int32)
    labels[:active] = np.repeat(np.arange(count) * (n_clusters // count), sizes)
    return labels


def _loaded_state(g, active, count, n_clusters, full=True, **kw):
    dm = P.CudaDeviceManager(**kw)
    dm.initialize(g)
    x = np.sin(np.arange(g.n) * 0.37)
    dm.set_state(_state(g, active, count, n_clusters), np.arange(active, dtype=np.uint32), x,
                 np.diff(g.offsets.astype(np.int64)).astype(np.uint32), g.cols, n_clusters, -1, full)
    return dm


def test_state_with_more_clusters_than_tables_is_refused():
    """The cluster tables hold a cluster per vertex; a cluster without vertices has no
    root to go on with unless the first round recomputes every component."""
    g, starts, _ = _paths(700)
    active = int(starts[300])
    for n_clusters in (g.n + 1, 0xFFFFFFFF):
        with pytest.raises(P.PxrError):
            _loaded_state(g, active, 300, n_clusters)
    with pytest.raises(P.PxrError):
        _loaded_state(g, active, 300, 301, full=False)
    _loaded_state(g, active, 300, g.n)
    dm = _loaded_state(g, active, 300, 300, full=False)
    assert dm.getNumClusters() == 300


# sampled linking looks a representative up for every cluster
@pytest.mark.parametrize("driver,components", [(P.DRIVER_STREAM, P.COMPONENTS_PLAIN),
                                               (P.DRIVER_STREAM, P.COMPONENTS_SAMPLED),
                                               (P.DRIVER_GRAPH, P.COMPONENTS_PLAIN)])
@pytest.mark.parametrize("count,n_clusters", [(300, 5000), (5000, 17000), (5000, 47000)])
def test_labels_without_vertices(count, n_clusters, driver, components):
    """A state with gaps between its labels and past the last one gives the dense
    one's decomposition, also where the one-kernel form has more clusters than
    vertices to lay its CTAs out for, or more than its largest cluster holds."""
    g, starts, _ = _paths(12000)
    out = []
    for k in (count, n_clusters):
        dm = _loaded_state(g, int(starts[count]), count, k, driver=driver, components=components)
        dm.expanderDecomposition()
        out.append((dm.downloadLabels(), dm.downloadCertificates(), dm.readRandomWalkValues().view(np.uint32)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_memory_of_a_larger_graph_is_given_back():
    """A handle keeps at most 64 MiB more than the graph it holds needs."""
    used, fresh = P.CudaDeviceManager(), P.CudaDeviceManager()
    small = G.grid3d(85)
    used.initialize(G.grid3d(100))
    used.initialize(small)
    fresh.initialize(small)
    assert used.stats()["device_bytes"] <= fresh.stats()["device_bytes"] + (64 << 20)


def test_contraction_runs_without_the_decomposition_s_memory(monkeypatch):
    """A level's contraction has the device to itself but for a small handle kept open for the next level."""
    import torch
    from parex_b200 import hierarchy as H
    open_handles, held = [], []

    class Handle(H.CudaDeviceManager):
        def __init__(self, **kw):
            super().__init__(**kw)
            open_handles.append(self)

        def close(self):
            if self in open_handles:
                open_handles.remove(self)
            super().close()

    contract = H.contract

    def contract_noting(*a, **kw):
        held.append(sum(h.stats()["device_bytes"] for h in open_handles))
        return contract(*a, **kw)

    monkeypatch.setattr(H, "CudaDeviceManager", Handle)
    monkeypatch.setattr(H, "contract", contract_noting)
    g = G.grid3d(80)
    levels = H.build(torch.from_numpy(g.offsets.view(np.int32)), torch.from_numpy(g.cols.view(np.int32)))
    assert len(held) == len(levels) > 1
    assert max(held) <= 64 << 20
    assert not open_handles


HUBS = {30007: 5000, 41000: 1500, 49999: 300}      # long rows among short ones, by vertex
LASTING = (30007, 49999)                           # active when the rounds are handed over


def _with_hubs():
    """8-regular beside a planted partition with hubs."""
    a, b = G.random_regular(30000, 8, seed=1), G.sbm_graph(20000, 40, 9.0, 1.0, 5)
    rng = np.random.default_rng(3)
    src, dst = [], []
    for g, first in ((a, 0), (b, 30000)):
        src.append(np.repeat(np.arange(g.n), np.diff(g.offsets.astype(np.int64))) + first)
        dst.append(g.cols.astype(np.int64) + first)
    for hub, degree in HUBS.items():
        src.append(np.full(degree, hub))
        dst.append(30000 + rng.choice(20000, degree, replace=False))
    src, dst = np.concatenate(src), np.concatenate(dst)
    keep = src != dst
    return G.csr_from_edges(src[keep], dst[keep], 50000)


# beyond the one-kernel decomposition (32,768 vertices); with each a row plan
# under which most rows are long, so that the last rounds are not handed over either
GRAPHS = {
    "sbm40k": (lambda: G.sbm_graph(40000, 40, 9.0, 1.0, 4), (4, 9, 16)),
    "grid35": (lambda: G.grid3d(35), (1, 5, 5)),
    "rmat16": (lambda: G.rmat(16, 8, seed=2), (8, 32, 256)),
}


def _start(g, dm):
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_potentials(dm.readRandomWalkValues().astype(np.float64))
    return orc


def _check_state(dm, orc, srt):
    np.testing.assert_array_equal(dm.downloadLabels(), orc.labels())
    np.testing.assert_array_equal(dm.readRandomWalkValues().view(np.uint32),
                                  np.asarray(orc.potentials(), dtype=np.float32).view(np.uint32))
    np.testing.assert_array_equal(dm.downloadDegrees(), orc.internal_degrees())
    np.testing.assert_array_equal(dm.downloadGraph()[1], orc.cols())
    np.testing.assert_array_equal(dm.downloadCertificates(), orc.certificates())
    _check_sweep_order(dm, srt)
    ids, k = orc.final_partition()
    fp = dm.getFinalPartition()
    assert fp.numClusters == k
    np.testing.assert_array_equal(fp.clusterIds, ids)


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("components,sort_plan",
                         [(P.COMPONENTS_PLAIN, 0), (P.COMPONENTS_PLAIN, 1), (P.COMPONENTS_SAMPLED, 2)])
def test_options_inside_the_captured_loop(name, components, sort_plan):
    """Both component schedules and every sort plan with all rounds in the captured loop."""
    make, plan = GRAPHS[name]
    g = make()
    dm = P.CudaDeviceManager(components=components)
    dm.set_row_plan(*plan)
    dm.set_sort_plan(sort_plan)
    dm.initialize(g)
    assert dm.row_plan()["wide_rows"] + dm.row_plan()["heavy_rows"] > 2048
    orc = _start(g, dm)
    before = dm.stats()["kernel_launches"]
    rounds = dm.expanderDecomposition()
    assert dm.stats()["kernel_launches"] - before > 15 * rounds      # one kernel takes one launch
    done, srt = _run_rounds(orc)
    assert rounds == done
    _check_state(dm, orc, srt)


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("offsets", [np.uint32, np.uint64])
def test_loop_and_hand_over(name, offsets):
    """The tuned plan: the loop, then the one-kernel form where few rows are long."""
    g = GRAPHS[name][0]()
    g = G.CSRGraph(g.offsets.astype(offsets), g.cols, name)
    dm = P.CudaDeviceManager()
    dm.initialize(g)
    orc = _start(g, dm)
    before = dm.stats()["kernel_launches"]
    rounds = dm.expanderDecomposition()
    assert dm.stats()["kernel_launches"] - before > 15 * 2           # at least one body of two rounds
    done, srt = _run_rounds(orc)
    assert rounds == done
    _check_state(dm, orc, srt)


@pytest.mark.parametrize("plan", [None, (8, 64, 1024), (1, 64, 128)])
@pytest.mark.parametrize("offsets", [np.uint32, np.uint64])
def test_long_rows_are_handed_over(plan, offsets):
    g = _with_hubs()
    g = G.CSRGraph(g.offsets.astype(offsets), g.cols, "hubs")
    dm = P.CudaDeviceManager()
    if plan:
        dm.set_row_plan(*plan)
    dm.initialize(g)
    orc = _start(g, dm)
    handed, srt = 0, None
    while orc.n_active > 32768:          # the loop hands over after an even round
        done, srt = _run_rounds(orc, 2)
        handed += done
    assert orc.n_active and all(orc.labels()[hub] >= 0 for hub in LASTING)
    rounds = dm.expanderDecomposition()
    more, srt = _run_rounds(orc)
    assert rounds == handed + more
    _check_state(dm, orc, srt)


def test_round_cap_inside_the_handed_over_rounds():
    """A cap three rounds past the hand-over: the state it leaves, and the rest stage by stage."""
    g = _with_hubs()
    first = P.CudaDeviceManager()
    first.initialize(g)
    orc = _start(g, first)
    handed = 0
    while orc.n_active > 32768:
        handed += _run_rounds(orc, 2)[0]
    dm = P.CudaDeviceManager(max_rounds=handed + 3)
    dm.initialize(g)
    with pytest.raises(P.PxrError):
        dm.expanderDecomposition()
    done, srt = _run_rounds(orc, 4)      # the cap is looked at after every second round
    assert done == 4 and orc.labels()[LASTING[0]] >= 0
    _check_state(dm, orc, srt)
    while dm.getNumClusters():
        dm.iterateRandomWalk()
        dm.computeSweepCuts()
        dm.cutClusters()
    _, srt = _run_rounds(orc)
    _check_state(dm, orc, srt)


def test_slots_up_to_the_end_of_32_bits():
    """2^32 - 2 slots under 32-bit offsets: rows end within a walk's stride of 2^32.
    Cliques of 4,096 vertices in pairs joined by a perfect matching, less one edge."""
    import torch
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("needs 60 GB of device memory")
    n, deg, chunk = 1 << 20, 4096, 1 << 15
    cols = torch.empty(n * deg - 2, dtype=torch.int32, device="cuda")
    at = 0
    for v0 in range(0, n, chunk):
        v = torch.arange(v0, v0 + chunk, dtype=torch.int32, device="cuda")
        rows = torch.sort(v[:, None] ^ torch.arange(1, deg + 1, dtype=torch.int32, device="cuda")[None, :], dim=1)[0]
        rows = rows.reshape(-1)
        if v0 == 0:       # without the edge 0 - 4,096: the last slot of the one row, the first of the other
            rows = torch.cat([rows[: deg - 1], rows[deg: deg * deg], rows[deg * deg + 1:]])
        cols[at: at + rows.shape[0]] = rows
        at += rows.shape[0]
    assert at == cols.shape[0]
    ix = np.arange(n + 1, dtype=np.int64)
    off = (ix * deg - (ix > 0) - (ix > deg)).astype(np.uint32)
    off_d = torch.from_numpy(off.view(np.int32)).cuda()
    dm = P.CudaDeviceManager(tune=P.TUNE_HEURISTIC)
    dm.initialize_device(n, (n * deg - 2) // 2, off_d.data_ptr(), False, cols.data_ptr())

    x = dm.readRandomWalkValues().astype(np.float64)
    dm.iterateRandomWalk()
    degree = np.diff(off.astype(np.int64))
    share = x / degree
    total = share.reshape(-1, deg).sum(axis=1).repeat(deg) - share + share[np.arange(n) ^ deg]
    total[0] -= share[deg]
    total[deg] -= share[0]
    # rounding of 4,096 terms x / degree to 24 bits, of their sum and of the result: 2^-24 max|x| each at most
    np.testing.assert_allclose(dm.readRandomWalkValues(), 0.9 * total + 0.1 * x, rtol=0,
                               atol=2.0**-22 * np.abs(x).max())
    dm.computeSweepCuts()
    dm.cutClusters()
    dm.expanderDecomposition()
    ids = torch.from_numpy(dm.getFinalPartition().clusterIds).cuda()
    pair = torch.arange(n, device="cuda") // (2 * deg)
    one = torch.full((int(ids.max()) + 1,), -1, dtype=torch.int64, device="cuda")
    one[ids.long()] = pair
    assert bool((one[ids.long()] == pair).all())          # no cluster in two components
    cut = 0
    for v0 in range(0, n, chunk):
        b, e = int(off[v0]), int(off[v0 + chunk])
        d = torch.from_numpy(degree[v0: v0 + chunk]).cuda()
        cut += int((ids[v0: v0 + chunk].repeat_interleave(d) != ids[cols[b:e].long()]).sum())
    assert dm.countCutEdges() == cut // 2
    dm.close()
    del cols
    torch.cuda.empty_cache()
