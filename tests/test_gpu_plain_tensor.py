"""Large plain batches on the tensor cores (the FP32 arena read as TF32, exact
FP32 re-rank): the answer is the list-major scan's, entry for entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import harmonyclient_b200 as hb  # noqa: E402

NLIST = 48


def _data(d, n, nq, kind, seed=0):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 200, (96, d))
    x = c[rng.integers(0, 96, n)] + 9 * rng.standard_normal((n, d))
    q = c[rng.integers(0, 96, nq)] + 9 * rng.standard_normal((nq, d))
    if kind == "int":
        x, q = np.clip(np.rint(x), 0, 255), np.clip(np.rint(q), 0, 255)
    elif kind == "unit":
        x, q = (v - 100 for v in (x, q))
        x, q = (v / np.linalg.norm(v, axis=1, keepdims=True) for v in (x, q))
    return x.astype(np.float32), q.astype(np.float32)


def _index(x, nprobe=16, metric=hb.METRIC_L2, **kw):
    idx = hb.Index(x.shape[1], NLIST, nprobe, metric, **kw)
    cent = x[:NLIST].copy()
    if metric == hb.METRIC_IP:
        cent /= np.linalg.norm(cent, axis=1, keepdims=True)
    idx.centroid_codes = cent
    idx.add(x)
    return idx


def _same(idx, q, k, nprobes=None, tensor=True):
    run = (lambda: idx.search(q, k)) if nprobes is None else (lambda: idx.search_nprobes(q, k, nprobes))
    idx.set_plain_scan("auto")
    D, I = run()
    st = idx.last_stats()
    idx.set_plain_scan("list")
    Dl, Il = run()
    assert idx.last_stats()["list_major"] == 1
    idx.set_plain_scan("auto")
    assert st["list_major"] == (0 if tensor else 1)
    np.testing.assert_array_equal(I, Il)
    np.testing.assert_array_equal(D, Dl)
    return st


@pytest.mark.parametrize("d", [4, 16, 31, 97, 128, 130, 200, 256, 384])
@pytest.mark.parametrize("kind,metric", [("int", hb.METRIC_L2), ("float", hb.METRIC_L2), ("unit", hb.METRIC_IP),
                                         ("float", hb.METRIC_IP)])
def test_equals_list_major(d, kind, metric):
    x, q = _data(d, 9_001, 1_025, kind, d)
    st = _same(_index(x, metric=metric), q, 23)
    assert st["tile_blocks"] == 0 or st["fallback_queries"] > 0


@pytest.mark.parametrize("k", [1, 32, 33, 100, 256])
@pytest.mark.parametrize("warm", [0, 10])
def test_k_and_warmup(k, warm):
    x, q = _data(64, 12_000, 1_500, "float", 3)
    idx = _index(x)
    idx.preSearch(warmUpSearchList=warm, warmUpSearchListSize=k)
    _same(idx, q, k)


@pytest.mark.parametrize("dim_blocks", [1, 3, 8])
def test_dim_blocks(dim_blocks):
    x, q = _data(100, 8_000, 1_100, "float", 4)
    _same(_index(x, dim_blocks=dim_blocks), q, 10)


def test_ties_and_duplicates():
    x, q = _data(24, 4_000, 1_200, "int", 5)
    x = np.concatenate([x, x, x[:1_000]])
    _same(_index(x), q, 50)


def test_per_query_nprobe_and_learned_bounds():
    x, q = _data(40, 9_000, 2_000, "float", 6)
    _same(_index(x, nprobe=30), q, 12, np.random.default_rng(1).integers(1, 31, len(q)).astype(np.int32))


def test_candidate_overflow():
    x, q = _data(32, 20_000, 1_500, "float", 7)
    idx = _index(x)
    idx.set_batch_params(capq=128)
    assert _same(idx, q, 100)["fallback_queries"] > 0


def test_far_offset_keeps_the_exact_scans():
    x, q = _data(32, 9_000, 1_500, "float", 8)
    _same(_index(x + 30_000), q + 30_000, 10, tensor=False)


@pytest.mark.parametrize("what", ["query", "row"])
def test_nonfinite(what):
    x, q = _data(32, 9_000, 1_500, "float", 9)
    v = q if what == "query" else x
    v[5, 3], v[6, 0], v[700, 31], v[900] = np.inf, -np.inf, np.nan, 3e19
    _same(_index(x), q, 10, tensor=what == "query")


def test_device_calls_and_graph():
    x, q = _data(96, 10_000, 2_048, "float", 10)
    idx = _index(x)
    D, I = idx.search(q, 20)
    dq = torch.from_numpy(q).cuda()
    dD = torch.empty((len(q), 20), device="cuda")
    dI = torch.empty((len(q), 20), dtype=torch.int64, device="cuda")
    for graph in (False, True):
        idx.set_graph(graph)
        for _ in range(3):
            dD.fill_(-1)
            idx.search_device(len(q), dq.data_ptr(), 20, dD.data_ptr(), dI.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(dI.cpu().numpy(), I)
            np.testing.assert_array_equal(dD.cpu().numpy(), D)


def test_first_search_under_capture_keeps_the_list_major_scan():
    """A caller's own capture: the bound terms are not built inside it."""
    x, q = _data(96, 10_000, 2_048, "float", 11)
    idx = _index(x)
    idx.set_plain_scan("list")
    D, I = idx.search(q, 20)  # workspaces exist
    idx.set_plain_scan("auto")
    dq = torch.from_numpy(q).cuda()
    dD = torch.empty((len(q), 20), device="cuda")
    dI = torch.empty((len(q), 20), dtype=torch.int64, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        idx.search_device(len(q), dq.data_ptr(), 20, dD.data_ptr(), dI.data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dI.cpu().numpy(), I)
    np.testing.assert_array_equal(dD.cpu().numpy(), D)


@pytest.mark.parametrize("metric,lists,rows,taken", [
    (hb.METRIC_L2, 0, 20_000, True),  # no warm-up: its size has no say
    (hb.METRIC_IP, 10, 20_000, True),  # none for inner products
    (hb.METRIC_L2, 8, 4_096, True), (hb.METRIC_L2, 8, 4_097, False),  # at and past the limit
    (hb.METRIC_L2, 100, 2_049, False),  # lists count up to nprobe
])
def test_warmup_sizes_as_the_other_scans_take_them(metric, lists, rows, taken):
    x, q = _data(128, 9_001, 1_025, "float", 3)
    idx = _index(x, metric=metric)
    idx.preSearch(warmUpSearchList=lists, warmUpSearchListSize=rows)
    if taken:
        _same(idx, q, 10)
        return
    for mode in ("query", "list", "auto"):
        idx.set_plain_scan(mode)
        with pytest.raises(hb.HyError):
            idx.search(q, 10)
