"""Graph construction on the device at the sizes where its kernels change
shape: key widths (n up to 2^16 sorts 32-bit keys), remainders of four edges a
thread, unaligned input, empty rows at both ends -- the arrays of the host
construction, edge list and CSC upload alike, and the out-adjacency."""
import numpy as np
import pytest

from kites_b200 import capi
from test_gpu_ingest import csc_of, dev_array

pytestmark = pytest.mark.gpu


def check(g, n, R, C, E):
    Rd, Cd, Ed = csc_of(g)
    np.testing.assert_array_equal(Rd[: n + 1], R)
    assert np.all(Rd[n:] == C.shape[0])
    np.testing.assert_array_equal(Cd, C)
    if E is not None:
        np.testing.assert_array_equal(Ed, E)
    dv = g.device_view()
    row = np.repeat(np.arange(n), np.diff(R.astype(np.int64)))
    order = np.argsort(C, kind="stable")
    kind = np.uint64 if dv.offsets64 else np.uint32
    dR = dev_array(dv.dir_R, dv.n_vertices + 1, "<i8" if dv.offsets64 else "<i4").view(kind)
    dC = dev_array(dv.dir_C, dv.n_edges, "<i4").view(np.uint32)
    np.testing.assert_array_equal(dC, row[order])
    want = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=int(dv.n_vertices)))])
    np.testing.assert_array_equal(dR, want)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 3), (127, 4), (129, 5), (1000, 1023), (1000, 1024),
                                 (1000, 1025), (65535, 30001), (65536, 30002), (65537, 30003),
                                 (300000, 70007)])
def test_edge_lists(engine, n, m, weighted):
    import torch

    rng = np.random.default_rng(n + m)
    lo, hi = (0, n) if n < 1000 else (n // 5, n - n // 7)   # no edges at either end
    s = rng.integers(lo, hi, m, dtype=np.uint32)
    d = rng.integers(lo, hi, m, dtype=np.uint32)
    w = rng.integers(1, 2**32, m, dtype=np.uint64).astype(np.uint32) if weighted else None
    R, C, E = capi.csc_from_edges(n, s, d, w)
    pad = np.zeros(1, np.uint32)
    lists = [(s, d, w)]
    for off in (0, 1):      # 16-byte aligned device arrays, and not
        lists.append(tuple(None if x is None else
                           torch.from_numpy(np.concatenate([pad] * off + [x]).view(np.int32))
                           .cuda()[off:] for x in (s, d, w)))
    for args in lists:
        g = capi.Graph.from_edges(engine, n, *args)
        try:
            check(g, n, R, C, E)
        finally:
            g.close()


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("n,m", [(3, 1), (128, 7), (129, 8), (5000, 9), (5000, 4001),
                                 (40000, 100003)])
def test_uploads(engine, n, m, offsets64):
    rng = np.random.default_rng(n * 3 + m)
    s = rng.integers(0, n, m, dtype=np.uint32)
    d = (n // 2 + rng.integers(0, max(1, n // 50), m)).astype(np.uint32)   # long empty runs
    w = rng.integers(1, 256, m, dtype=np.uint32)
    R, C, E = capi.csc_from_edges(n, s, d, w)
    g = capi.Graph(engine, R, C, E, offsets64=offsets64)
    try:
        check(g, n, R, C, E)
    finally:
        g.close()


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_edge_lists_at_any_byte(engine, offset):
    """Device arrays that start inside an element are copied, as host arrays
    are."""
    import ctypes

    import torch

    n, m = 3000, 20001
    rng = np.random.default_rng(offset)
    s, d, w = (rng.integers(0, n, m, dtype=np.uint32) for _ in range(3))
    R, C, E = capi.csc_from_edges(n, s, d, w)
    keep = []
    for x in (s, d, w):
        t = torch.zeros(4 * m + 16, dtype=torch.uint8, device="cuda")
        t[offset:offset + 4 * m] = torch.from_numpy(x.view(np.uint8)).cuda()
        keep.append(t)
    torch.cuda.synchronize()
    g = capi.Graph.__new__(capi.Graph)
    g.engine, g._h = engine, ctypes.c_void_p()
    ptrs = [ctypes.c_void_p(t.data_ptr() + offset) for t in keep]
    assert capi.load().kites_graph_from_edges(engine._h, n, m, *ptrs, 1,
                                              ctypes.byref(g._h)) == capi.OK
    try:
        check(g, n, R, C, E)
    finally:
        g.close()


def test_upload_memory():
    """What an upload of more than 2^30 weighted edges holds at the most (the
    pool keeps what it ever held): the sort by source with 32-bit edge numbers
    as its payload needed 40 bytes an edge."""
    import torch

    n, deg = (1 << 20) + 128, 1024
    m = n * deg
    eng = capi.Engine(0)
    try:
        R = torch.arange(n + 1, dtype=torch.int32, device="cuda") * deg
        gen = torch.Generator(device="cuda")
        gen.manual_seed(5)
        C = torch.randint(0, 1024, (n, deg), dtype=torch.int32, device="cuda", generator=gen)
        C += torch.arange(deg, dtype=torch.int32, device="cuda") * 1024      # ascending
        E = torch.randint(1, 1 << 20, (m,), dtype=torch.int32, device="cuda", generator=gen)
        torch.cuda.synchronize()
        g = capi.Graph(eng, R, C, E, on_device=True, n_vertices=n, n_edges=m)
        pool = eng.mem_usage()[2]
        assert pool <= 40 * m + (256 << 20), pool / m
        out = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]
        assert g.sssp(3, out=out[0])[1].kernel_launches == 1         # over the out-edges
        g.sssp(3, out=out[1], opts=capi.default_opts(device_loop=0))   # over the in-edges
        assert torch.equal(*out) and int((out[0] != -1).sum()) == n
    finally:
        eng.close()
        del R, C, E
        torch.cuda.empty_cache()
