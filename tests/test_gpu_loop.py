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
