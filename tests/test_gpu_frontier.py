"""The single-launch frontier loop (default options of kites_sssp, kites_cc,
kites_sssp_multi_seed and kites_process): the oracle's fixed point at the
sizes where its queues and thresholds change shape, and the per-iteration
loop's result from any state kites_process is given."""
import numpy as np
import pytest

from kites_b200 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu

INF = O.INF32
OPS = [(capi.OP_SSSP, O.OP_SSSP_SAT), (capi.OP_BFS, O.OP_BFS_SAT)]


def oracle(R, C, E, n, sources, oop):
    V0 = np.full(n, INF, np.uint32)
    V0[sources] = 0
    return O.sanity_check(R, C, E, V0, op=oop)[0]


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("deg", [1, 31, 33, 255, 256, 257, 512, 513, 4097])
def test_row_lengths(engine, deg, offsets64):
    """Out-rows around the lane, segment and batch sizes: two hubs of `deg`
    out-edges in a ring that reaches every vertex."""
    n = 5000
    rng = np.random.default_rng(deg)
    ring = np.arange(n, dtype=np.uint32)
    hub = np.concatenate([rng.choice(n, deg, replace=False) for _ in range(2)]).astype(np.uint32)
    s = np.concatenate([ring, np.repeat(np.uint32([3, 1700]), deg)]).astype(np.uint32)
    d = np.concatenate([(ring + 1) % n, hub]).astype(np.uint32)
    w = rng.integers(1, 200, s.shape[0], dtype=np.uint32)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph(engine, R, C, E, offsets64=offsets64)
    try:
        for op, oop in OPS:
            for src in (0, 3):
                np.testing.assert_array_equal(g.sssp(src, op=op)[0],
                                              oracle(R, C, E, n, [src], oop))
        seeds = np.array([7, 1700, 4999], np.uint32)
        np.testing.assert_array_equal(g.sssp_multi_seed(seeds)[0],
                                      oracle(R, C, E, n, seeds, O.OP_SSSP_SAT))
        np.testing.assert_array_equal(g.cc()[0], np.zeros(n, np.uint32))
    finally:
        g.close()


@pytest.mark.parametrize("w_hi", [1, 7, 1000, 2**31, 2**32 - 1])
@pytest.mark.parametrize("kind", ["grid", "sparse"])
def test_thresholds(engine, kind, w_hi):
    """Graphs with few edges a vertex order their work by a threshold: unit
    weights, small and large ones, and ones whose sums saturate."""
    rng = np.random.default_rng(w_hi % 1000)
    if kind == "grid":
        n = 70 * 70
        s, d, _ = capi.gen_grid(70, seed=3)
    else:
        n = 20001
        s = rng.integers(0, n, 3 * n, dtype=np.uint32)
        d = rng.integers(0, n, 3 * n, dtype=np.uint32)
    w = rng.integers(1, w_hi, s.shape[0], dtype=np.uint64, endpoint=True).astype(np.uint32)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph(engine, R, C, E)
    try:
        for src in (0, n // 2):
            np.testing.assert_array_equal(g.sssp(src)[0],
                                          oracle(R, C, E, n, [src], O.OP_SSSP_SAT))
    finally:
        g.close()


@pytest.mark.parametrize("scale,factor", [(15, 16), (18, 16), (20, 17)])
def test_wide_iterations(engine, scale, factor):
    """Iterations above the short size, and (from 16 M edges) a threshold on
    an R-MAT graph: the values of the per-iteration loop, whose first
    iteration from them changes nothing."""
    n = 1 << scale
    s, d, w = capi.gen_rmat(scale, factor * n, seed=scale)
    g = capi.Graph.from_edges(engine, n, s, d, w)
    try:
        src = int(s[12345])
        loop = capi.default_opts(device_loop=0)
        for op, _ in OPS:
            dist, _ = g.sssp(src, op=op)
            np.testing.assert_array_equal(dist, g.sssp(src, op=op, opts=loop)[0])
        np.testing.assert_array_equal(g.cc()[0], g.cc(opts=loop)[0])
    finally:
        g.close()


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("deg", [3, 4, 5, 8, 9, 40, 1031, 1032, 1033, 5000])
def test_bottom_up_rows(engine, deg, offsets64):
    """BFS whose second frontier holds most of the edges, so that unreached
    vertices look for a parent: rows of `deg` in-edges whose only parent is
    their last in-neighbour, or that have none."""
    n, mids = 60000, np.arange(57000, 60000, dtype=np.uint32)
    rng = np.random.default_rng(deg)
    far = np.arange(1, 20000, dtype=np.uint32)            # never reached
    s = [np.zeros(mids.shape[0], np.uint32), np.repeat(mids, 100)]
    d = [mids, rng.integers(31000, 57000, 100 * mids.shape[0], dtype=np.uint32)]
    for i, row in enumerate(range(30000, 30010)):
        src = rng.choice(far, deg, replace=False)
        if i % 2:
            src[-1] = mids[7 * i]
        s.append(src)
        d.append(np.full(deg, row, np.uint32))
    s.append(np.arange(30000, 30010, dtype=np.uint32))    # and one level below
    d.append(np.arange(30500, 30510, dtype=np.uint32))
    s, d = np.concatenate(s), np.concatenate(d)
    R, C, _ = capi.csc_from_edges(n, s, d)
    g = capi.Graph(engine, R, C, None, offsets64=offsets64)
    try:
        dist, _ = g.sssp(0, op=capi.OP_BFS)
        np.testing.assert_array_equal(dist, oracle(R, C, None, n, [0], O.OP_BFS_SAT))
        assert dist[30001] == 2 and dist[30000] == INF and dist[30501] == 3
    finally:
        g.close()


@pytest.mark.parametrize("parents", [1, 1500, 3000])
def test_bottom_up_rows_reached_from_several_segments(engine, parents):
    """Rows that several CTAs look through at the same time, each finding a
    parent: one of them queues the row, and the level below it is right."""
    n, mids = 60000, np.arange(57000, 60000, dtype=np.uint32)
    rng = np.random.default_rng(parents)
    rows = np.arange(30000, 30040, dtype=np.uint32)
    s = [np.zeros(mids.shape[0], np.uint32), np.repeat(mids, 100)]
    d = [mids, rng.integers(31000, 57000, 100 * mids.shape[0], dtype=np.uint32)]
    for row in rows:                        # 2,000 in-neighbours never reached come first
        s += [rng.choice(np.arange(1, 20000, dtype=np.uint32), 2000, replace=False),
              rng.choice(mids, parents, replace=False)]
        d.append(np.full(2000 + parents, row, np.uint32))
    s.append(rows)
    d.append(rows + np.uint32(500))
    s, d = np.concatenate(s), np.concatenate(d)
    R, C, _ = capi.csc_from_edges(n, s, d)
    g = capi.Graph(engine, R, C, None)
    try:
        want = oracle(R, C, None, n, [0], O.OP_BFS_SAT)
        for _ in range(5):
            dist, _ = g.sssp(0, op=capi.OP_BFS)
            np.testing.assert_array_equal(dist, want)
        assert (want[rows] == 2).all() and (want[rows + 500] == 3).sum() > 0
    finally:
        g.close()


@pytest.mark.parametrize("op,oop", OPS + [(capi.OP_CC, None)])
@pytest.mark.parametrize("state", ["sources", "missing", "partial", "empty", "settled"])
def test_process_states(engine, op, oop, state):
    """kites_process from a caller's values and frontier gives what the
    per-iteration loop gives, also where an unsatisfied edge leads outside
    the frontier, and leaves an empty frontier."""
    n = 3001
    s, d, w = capi.gen_rmat(12, 20000, seed=5, n_vertices=n)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    rng = np.random.default_rng(11)
    V = np.full(n, INF, np.uint32)
    bits = np.zeros(n, bool)
    srcs = s[[5, 500, 5000]]
    V[srcs] = [0, 40, 7]
    if state == "sources":
        bits[d[np.isin(s, srcs)]] = True
    elif state == "missing":         # one source's out-neighbours are not in the frontier
        bits[d[np.isin(s, srcs[:2])]] = True
    elif state == "partial":
        V = rng.integers(0, 500, n, dtype=np.uint32)
        bits = rng.random(n) < 0.3
    elif state == "settled":
        V[:] = 0
        bits[:] = True
    words = np.packbits(np.pad(bits, (0, -n % 32)), bitorder="little").view(np.uint32)
    got = []
    g = capi.Graph(engine, R, C, E)
    try:
        for loop in (1, 0):
            g.set_values(V)
            g.set_frontier(words, n)
            st = g.process(op, opts=capi.default_opts(device_loop=loop))
            assert st.iterations >= 1
            got.append(g.get_values(n))
            g.process(op, opts=capi.default_opts(device_loop=loop))
            np.testing.assert_array_equal(g.get_values(n), got[-1])
        np.testing.assert_array_equal(got[0], got[1])
    finally:
        g.close()


def test_process_of_an_uneven_state(engine):
    """A start with unsatisfied edges outside the frontier is offered to the
    single-launch loop once, not by every call that goes on from it; values
    set anew are."""
    n = 3001
    s, d, w = capi.gen_rmat(12, 20000, seed=5, n_vertices=n)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph(engine, R, C, E)
    try:
        V = np.full(n, INF, np.uint32)
        V[s[5]] = 0
        none = np.zeros(g.n_padded // 32, np.uint32)
        for _ in range(2):
            g.set_values(V)
            for call in range(3):      # nothing to do in this frontier, much outside it
                g.set_frontier(none, n)
                st = g.process(capi.OP_SSSP)
                assert st.kernel_launches == 3 * st.iterations + (call == 0)
                np.testing.assert_array_equal(g.get_values(n), V)
        want = oracle(R, C, E, n, [int(s[5])], O.OP_SSSP_SAT)
        np.testing.assert_array_equal(g.sssp(int(s[5]))[0], want)
        st = g.process(capi.OP_SSSP)
        assert st.kernel_launches == 1
    finally:
        g.close()


@pytest.mark.parametrize("again", [False, True])
def test_process_of_a_settled_state(engine, again):
    """From settled values, left by a run or set again, a small frontier costs
    its own in-edges and not a walk over the graph."""
    n = 1 << 17
    s, d, w = capi.gen_rmat(17, 16 * n, seed=6)
    R, _, _ = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph.from_edges(engine, n, s, d, w)
    try:
        for op in (capi.OP_SSSP, capi.OP_BFS):
            dist, _ = g.sssp(int(s[77]), op=op)
            if again:
                g.set_values(dist)
            rows = np.array([1, 50, 4000, 65537, n - 1])
            bits = np.zeros(n, np.uint8)
            bits[rows] = 1
            g.set_frontier(np.packbits(bits, bitorder="little").view(np.uint32), n)
            st = g.process(op)
            assert st.edges_traversed == int((R[rows + 1] - R[rows]).sum())
            np.testing.assert_array_equal(g.get_values(n), dist)
    finally:
        g.close()


@pytest.mark.parametrize("m", [1, 7, 20000, 20003])
def test_weights_changed_in_place(engine, m):
    """Runs take the weights that E holds, also those written through the
    device view after the upload, whichever edge they belong to."""
    import torch

    class Words:   # device memory as torch sees it
        def __init__(self, ptr, count):
            self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4",
                                             "data": (ptr, False), "version": 3}

    n = 3001
    rng = np.random.default_rng(m)
    s = rng.integers(0, n, m, dtype=np.uint32)
    d = rng.integers(0, n, m, dtype=np.uint32)
    R, C, E = capi.csc_from_edges(n, s, d, rng.integers(1, 100, m, dtype=np.uint32))
    src = int(C[0])
    g = capi.Graph(engine, R, C, E)
    try:
        dE = torch.as_tensor(Words(g.device_view().E, m), device="cuda")
        bits = np.zeros(g.n_padded // 32, np.uint32)
        for change in ([], [0], [m - 1], [m // 2, m // 3], list(range(m)), []):
            for e in change:
                E[e] = rng.integers(1, 2**32, dtype=np.uint64)
            dE.copy_(torch.from_numpy(E.view(np.int32)))
            torch.cuda.synchronize()
            want = oracle(R, C, E, n, [src], O.OP_SSSP_SAT)
            for strategy in (capi.STRATEGY_PLAIN, capi.STRATEGY_AUTO):
                dist, _ = g.sssp(src, opts=capi.default_opts(strategy=strategy))
                np.testing.assert_array_equal(dist, want)
            np.testing.assert_array_equal(g.sssp_multi_seed(np.array([src], np.uint32))[0], want)
            V = np.full(n, INF, np.uint32)
            V[src] = 0
            hop = C == src
            row = np.repeat(np.arange(n), np.diff(R.astype(np.int64)))
            bits[:] = 0
            np.bitwise_or.at(bits, row[hop] >> 5, (1 << (row[hop] & 31)).astype(np.uint32))
            g.set_values(V)
            g.set_frontier(bits, n)
            g.process(capi.OP_SSSP)
            np.testing.assert_array_equal(g.get_values(n), want)
    finally:
        g.close()


def test_wait_limit():
    """A grid whose CTAs stop waiting for one another ends with an error status,
    and the next call answers as before."""
    n = 1 << 15
    s, d, w = capi.gen_rmat(15, 16 * n, seed=8)
    seeds = np.array([5, 9], np.uint32)
    bits = np.full(n // 32, 0xFFFFFFFF, np.uint32)
    eng = capi.Engine(0)
    try:
        g = capi.Graph.from_edges(eng, n, s, d, w)

        def settle():
            V = np.full(n, INF, np.uint32)
            V[int(s[1])] = 0
            g.set_values(V)
            g.set_frontier(bits, n)
            g.process(capi.OP_SSSP)

        calls = [lambda: g.sssp(int(s[1])), lambda: g.sssp(int(s[1]), op=capi.OP_BFS), g.cc,
                 lambda: g.sssp_multi_seed(seeds), settle]
        want = g.sssp(int(s[1]))[0]
        for call in calls:
            eng.set_wait_limit(1)
            with pytest.raises(capi.KitesError) as e:
                call()
            assert e.value.status == capi.ERR_TIMEOUT
            eng.set_wait_limit(0)
            np.testing.assert_array_equal(g.sssp(int(s[1]))[0], want)
    finally:
        eng.close()


def test_engines_of_several_threads():
    """Engines of different threads answer at the same time, each what it
    answers alone."""
    import threading

    n = 1 << 13
    s, d, w = capi.gen_rmat(13, 16 * n, seed=4)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    want = {src: oracle(R, C, E, n, [src], O.OP_SSSP_SAT) for src in (1, 77)}
    bad = []

    def serve(src):
        eng = capi.Engine(0)
        try:
            g = capi.Graph(eng, R, C, E)
            for _ in range(20):
                if not np.array_equal(g.sssp(src)[0], want[src]):
                    bad.append(src)
        except Exception as e:   # a thread's exception must fail the test
            bad.append(e)
        finally:
            eng.close()

    threads = [threading.Thread(target=serve, args=(src,)) for src in want for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_buffers_give_way():
    """What the single-launch loop keeps on a graph does not take the memory of
    a later call: a batched run whose arrays only fit in its place succeeds."""
    import torch

    n, k = 1 << 23, 16
    ids = np.arange(n, dtype=np.uint32)
    s, d = ids // np.uint32(4), ids          # a tree
    srcs = np.arange(k, dtype=np.uint32)
    got, need, fill = [], 0, None
    for full in (False, True):
        eng = capi.Engine(0)
        try:
            g = capi.Graph.from_edges(eng, n, s, d)
            assert g.sssp(0, op=capi.OP_BFS, out=False)[1].kernel_launches == 1
            got.append(torch.empty((n, k), dtype=torch.int32, device="cuda"))
            if full:                         # 64 MB less than the batched run takes
                free = torch.cuda.mem_get_info()[0]
                fill = torch.empty(free - need + (64 << 20), dtype=torch.uint8, device="cuda")
            before = eng.mem_usage()[2]
            g.sssp_batch(srcs, op=capi.OP_BFS, out=got[-1])
            need = eng.mem_usage()[2] - before
            assert g.sssp(0, op=capi.OP_BFS, out=False)[1].iterations > 1
        finally:
            fill = None
            torch.cuda.empty_cache()
            eng.close()
    assert torch.equal(*got)
