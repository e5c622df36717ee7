"""The one-kernel decomposition of small graphs (graph driver, plain form),
the general path's tile sizes and the sweep order's download against the CPU
oracle: sizes around a warp's, a CTA's and a cluster's share of vertices, rows
in every bin, many clusters from the start, and a run stopped at its round cap
and continued by the general path."""
import numpy as np
import pytest

import parex_b200 as P
from parex_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 255, 257, 1023, 1025, 2047, 2049, 4097, 8191, 32768, 32769]


def _edges(n, e):
    e = np.asarray(e, dtype=np.int64).reshape(-1, 2)
    return G.csr_from_edges(e[:, 0], e[:, 1], n)


# active vertices around the general path's switch of tile sizes (2^19), which the
# run crosses as clusters are certified
LARGE = {"grid81": lambda: G.grid3d(81), "grid80": lambda: G.grid3d(80)}

SHAPES = {
    "path": lambda: _edges(5000, [(i, i + 1) for i in range(4999)]),
    "star": lambda: _edges(20000, [(0, i) for i in range(1, 20000)]),       # one CTA-wide row
    "rmat": lambda: G.rmat(14, 10),                                       # rows in every bin
    "dense": lambda: G.sbm_graph(600, 2, 200.0, 20.0, 3),
    "empty": lambda: _edges(3000, []),
}


def _check(dm, orc, rounds=None):
    done = orc.decompose()
    if rounds is not None:
        assert rounds == done
    np.testing.assert_array_equal(dm.downloadLabels(), orc.labels())
    np.testing.assert_array_equal(dm.readRandomWalkValues().view(np.uint32),
                                  np.asarray(orc.potentials(), dtype=np.float32).view(np.uint32))
    np.testing.assert_array_equal(dm.downloadDegrees(), orc.internal_degrees())
    np.testing.assert_array_equal(dm.downloadGraph()[1], orc.cols())
    ids, k = orc.final_partition()
    fp = dm.getFinalPartition()
    assert fp.numClusters == k
    np.testing.assert_array_equal(fp.clusterIds, ids)


def _loaded(g, **kw):
    dm = P.CudaDeviceManager(**kw)
    dm.initialize(g)
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_potentials(dm.readRandomWalkValues().astype(np.float64))
    return dm, orc


@pytest.mark.parametrize("n", SIZES)
def test_sizes_match_the_oracle(n):
    g = G.sbm_graph(n, max(1, n // 300), 9.0, 1.0, n)
    dm, orc = _loaded(g)
    _check(dm, orc, dm.expanderDecomposition())


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_shapes_match_the_oracle(name):
    dm, orc = _loaded(SHAPES[name]())
    _check(dm, orc, dm.expanderDecomposition())


@pytest.mark.parametrize("name", sorted(LARGE))
def test_tile_sizes_of_the_general_path(name):
    dm, orc = _loaded(LARGE[name]())
    _check(dm, orc, dm.expanderDecomposition())


@pytest.mark.parametrize("cap", [2, 5])
def test_continues_after_the_round_cap(cap):
    """The state left at the cap is one the stage-by-stage calls go on from."""
    dm, orc = _loaded(G.sbm_graph(3000, 10, 9.0, 1.0, 2), max_rounds=cap)
    with pytest.raises(P.PxrError):
        dm.expanderDecomposition()
    while dm.getNumClusters():
        dm.iterateRandomWalk()
        dm.computeSweepCuts()
        dm.cutClusters()
    _check(dm, orc)


def test_many_instances_from_the_start():
    """A batch of 2,500 instances: as many clusters as a CTA's share holds twice."""
    sizes = 1 + np.arange(2500) % 7
    starts = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    e = [(s + i, s + i + 1) for s, k in zip(starts, sizes) for i in range(k - 1)]
    g = _edges(int(starts[-1]), e)
    dm = P.CudaDeviceManager()
    dm.initialize_batched(g, starts)
    act = np.zeros(g.n, dtype=O.LNODE)
    labels = np.repeat(np.arange(2500, dtype=np.int32), sizes)
    act["nix"], act["label"] = np.arange(g.n, dtype=np.uint32), labels
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_state(labels, act, dm.readRandomWalkValues().astype(np.float64),
                  np.diff(g.offsets.astype(np.int64)).astype(np.uint32), g.cols, 2500, 0)
    dm.expanderDecomposition()
    _check(dm, orc)


def test_one_handle_takes_graphs_of_any_size_in_turn():
    """A smaller graph takes over the arena of the last one, a larger one replaces it."""
    dm = P.CudaDeviceManager()
    for n in (3000, 500, 40000, 100, 41000):
        g = G.sbm_graph(n, max(2, n // 300), 9.0, 1.0, n)
        dm.initialize(g)
        orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
        orc.set_potentials(dm.readRandomWalkValues().astype(np.float64))
        _check(dm, orc, dm.expanderDecomposition())


def test_schedule_switched_on_after_plain_graphs():
    """A handle that ran plain graphs starts the learned schedule with every cluster due, as a new one does."""
    from parex_b200 import learn
    model = learn.Model.load()
    used, fresh = P.CudaDeviceManager(), P.CudaDeviceManager()
    for n in (30000, 5000):
        used.initialize(G.sbm_graph(n, 20, 9.0, 1.0, n))
        used.expanderDecomposition()
    g = G.sbm_graph(20000, 20, 9.0, 1.0, 7)
    used.initialize(g)
    out = []
    for dm in (used, fresh):
        if dm is fresh:
            dm.initialize(g)
        dm.set_schedule(P._lib.SCHEDULE_LEARNED, model.weights, model.norm, **learn.SHIPPED_SCHEDULE)
        dm.expanderDecomposition()
        out.append((dm.getFinalPartition().clusterIds, dm.downloadCertificates()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("size", [1023, 1024, 1025, 4095, 4096, 4097])
def test_sort_paths_at_their_largest_clusters(size):
    """Batches whose clusters sit at the bounds of the chunked sort's two shapes and of the global sort."""
    count = 40000 // size + 1
    starts = np.arange(count + 1, dtype=np.int64) * size
    e = []
    for i in range(count):
        p = G.random_regular(size + size % 2, 8, seed=i + 1)   # an even number of stubs; the odd vertex is left out
        src = np.repeat(np.arange(p.n), np.diff(p.offsets.astype(np.int64)))
        keep = (src < p.cols) & (p.cols < size)
        e.append(np.stack([src[keep], p.cols[keep].astype(np.int64)], axis=1) + starts[i])
    g = _edges(int(starts[-1]), np.concatenate(e))
    dm = P.CudaDeviceManager()
    dm.initialize_batched(g, starts)
    act = np.zeros(g.n, dtype=O.LNODE)
    labels = np.repeat(np.arange(count, dtype=np.int32), size)
    act["nix"], act["label"] = np.arange(g.n, dtype=np.uint32), labels
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_state(labels, act, dm.readRandomWalkValues().astype(np.float64),
                  np.diff(g.offsets.astype(np.int64)).astype(np.uint32), g.cols, count, 0)
    dm.expanderDecomposition()
    _check(dm, orc)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 1001, 4097])
def test_sweep_order_download_in_parts(n):
    """The sweep order leaves the device in parts of half the vertices (16 at
    least): a single part, full ones and a short last one."""
    g = _edges(n, [(i, i + 1) for i in range(n - 1)])
    dm = P.CudaDeviceManager(driver=P.DRIVER_STREAM)
    dm.initialize(g)
    orc = O.Oracle(g.offsets, g.cols, O.MODE_PXR)
    orc.set_potentials(dm.readRandomWalkValues().astype(np.float64))
    orc.walk()
    dm.iterateRandomWalk()
    orc.sweep()
    dm.computeSweepCuts()
    part, srt = dm.downloadPartition(), orc.sorted()
    assert part.shape[0] == n
    for ours, theirs in (("nix", "nix"), ("prefix_edge_diff", "prefix_edge_diff"),
                         ("prefix_volume", "prefix_volume"), ("offset_in_cluster", "offset")):
        np.testing.assert_array_equal(part[ours], srt[theirs])
