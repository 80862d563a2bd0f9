"""The batched pull's row paths: in-rows around the lengths where short, tiled
and line-wise copies take over, whole and split over chunks, against the
single-source distances and the register-load pull."""
import numpy as np
import pytest

from kites_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("k", [16, 64, 128, 256])
@pytest.mark.parametrize("deg", [16, 17, 64, 65, 66, 96, 255, 256, 257, 900])
def test_row_lengths(engine, deg, k, offsets64):
    n = 3000
    rng = np.random.default_rng(deg * 1000 + k)
    rows = rng.choice(n, 40, replace=False).astype(np.uint32)
    ring = np.arange(n, dtype=np.uint32)
    s = np.concatenate([ring] + [rng.choice(n, deg, replace=False) for _ in rows]).astype(np.uint32)
    d = np.concatenate([(ring * 7 + 1) % n, np.repeat(rows, deg)]).astype(np.uint32)
    w = rng.integers(1, 1000, s.shape[0], dtype=np.uint32)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph(engine, R, C, E, offsets64=offsets64)
    try:
        srcs = rng.choice(n, k, replace=False).astype(np.uint32)
        g.set_batch_gather(0)
        loads, _ = g.sssp_batch(srcs)
        g.set_batch_gather(2)
        for strategy in (capi.STRATEGY_PLAIN, capi.STRATEGY_PULL_ALL, capi.STRATEGY_PULL_CHANGED):
            got, _ = g.sssp_batch(srcs, opts=capi.default_opts(strategy=strategy))
            np.testing.assert_array_equal(got, loads)
        for j in (0, k // 2, k - 1):
            np.testing.assert_array_equal(loads[:, j], g.sssp(int(srcs[j]))[0])
    finally:
        g.close()


@pytest.mark.parametrize("k", [64, 128])
@pytest.mark.parametrize("deg", [64, 65, 257, 900])
def test_long_rows_in_large_chunks(engine, deg, k):
    """A graph large enough for 256-item chunks, where line-wise rows occur."""
    import torch

    n = 700001
    rng = np.random.default_rng(deg + k)
    rows = rng.choice(n, 40, replace=False).astype(np.uint32)
    ids = np.arange(n, dtype=np.uint32)   # a tree, three children a vertex
    s = np.concatenate([ids // 3] + [rng.choice(n, deg, replace=False) for _ in rows]).astype(np.uint32)
    d = np.concatenate([ids, np.repeat(rows, deg)]).astype(np.uint32)
    w = rng.integers(1, 1000, s.shape[0], dtype=np.uint32)
    srcs = np.arange(k, dtype=np.uint32)
    g = capi.Graph.from_edges(engine, n, s, d, w)
    try:
        out = [torch.empty((n, k), dtype=torch.int32, device="cuda") for _ in range(2)]
        for mode in (0, 2):
            g.set_batch_gather(mode)
            g.sssp_batch(srcs, out=out[mode // 2])
        assert torch.equal(out[0], out[1])
    finally:
        g.close()
