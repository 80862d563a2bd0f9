"""PageRank's edge-parallel step at the sizes where rows cross lanes, windows
and chunks, against the FP64 oracle: 1e-5 relative L1, the bound the other
PageRank tests hold the engine to."""
import numpy as np
import pytest

from kites_b200 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(g, n, R, C, src, iterations, damping=0.85):
    outdeg = np.bincount(src, minlength=n).astype(np.uint32)
    pr, st = g.pagerank(n_real=n, iterations=iterations, damping=damping)
    want = O.pagerank_f64(n, R, C, outdeg, iterations, damping)
    assert st.iterations == iterations
    assert np.abs(pr.astype(np.float64) - want).sum() <= 1e-5 * np.abs(want).sum()


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("deg", [1, 7, 8, 9, 255, 256, 257, 2047, 2048, 2049, 4096, 7000])
def test_long_rows(engine, deg, offsets64):
    """Rows of `deg` in-edges at several places of the edge order, with empty
    rows between them and short rows around."""
    n = 9000
    rng = np.random.default_rng(deg)
    rows = [0, 1, 1000, 4501, n - 1]
    s = np.concatenate([rng.choice(n, deg, replace=False) for _ in rows] +
                       [rng.integers(0, n, 5000)]).astype(np.uint32)
    d = np.concatenate([np.repeat(rows, deg), rng.integers(2, 900, 5000)]).astype(np.uint32)
    R, C, _ = capi.csc_from_edges(n, s, d)
    g = capi.Graph(engine, R, C, None, offsets64=offsets64)
    try:
        for iterations in (1, 2, 3, 20):
            check(g, n, R, C, s, iterations)
    finally:
        g.close()


@pytest.mark.parametrize("n,m", [(1, 0), (2, 1), (40, 8), (129, 255), (300, 2048), (5000, 2049),
                                 (5000, 100003)])
def test_sizes(engine, n, m):
    rng = np.random.default_rng(n + m)
    s = rng.integers(0, n, m, dtype=np.uint32)
    d = rng.integers(0, n, m, dtype=np.uint32)
    R, C, _ = capi.csc_from_edges(n, s, d)
    g = capi.Graph(engine, R, C, None)
    try:
        check(g, n, R, C, s, 20)
        check(g, n, R, C, s, 3, damping=0.5)
    finally:
        g.close()


def test_vertex_groups(engine):
    """Graphs of vertex groups have no row index until PageRank builds one."""
    s, d, w = capi.gen_rmat(12, 30000, seed=3)
    hg = O.build_host_graph(s, d, w, vpg=4, init="source", source=0, inf=(1 << 30) - 1)
    g = capi.Graph(engine, hg.R, hg.C, hg.E, V=hg.V, vpg=4, dir_R=hg.dir_R, dir_C=hg.dir_C)
    try:
        outdeg = np.bincount(hg.C, minlength=hg.n_vertices).astype(np.uint32)
        pr, _ = g.pagerank(n_real=hg.n_vertices, iterations=5)
        want = O.pagerank_f64(hg.n_vertices, hg.R, hg.C, outdeg, 5, 0.85)
        assert np.abs(pr - want).sum() <= 1e-5 * np.abs(want).sum()
    finally:
        g.close()
