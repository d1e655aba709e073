"""A caller's own capture of the first search after an add: what the search
builds for later ones (images, bound terms, the certificate, the centroid
image) is built by the graph's replays and not taken for built by other calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("form", ["bf16", "fp8", "triangle"])
def test_search_after_a_capture(form):
    rng = np.random.default_rng(6)
    nlist, d, n, m, k = 64, 40, 20_000, 500, 10
    c = (20 * rng.standard_normal((nlist, d))).astype(np.float32)
    lab = rng.integers(0, nlist, n)
    # Two sets of rows with the same list sizes (one integral, one not).
    x1 = np.rint(c[lab] + rng.standard_normal((n, d))).astype(np.float32)
    x2 = (c[lab] + rng.standard_normal((n, d))).astype(np.float32)
    c2 = (c + 0.01 * rng.standard_normal((nlist, d))).astype(np.float32)
    q = (c[rng.integers(0, nlist, m)] + rng.standard_normal((m, d))).astype(np.float32)

    def make(cent):
        idx = hb.Index(d, nlist, 8, hb.METRIC_L2, hb.OPT_TRIANGLE if form == "triangle" else hb.OPT_NONE)
        idx.centroid_codes = cent
        if form == "triangle":
            idx.set_plain_scan("list")
        else:
            idx.set_form(form)
        return idx

    fresh = make(c2)
    fresh.add(x2)
    D, I = fresh.search(q, k)
    idx = make(c)
    idx.add(x1)
    idx.search(q, k)  # every buffer exists
    idx.centroid_codes = c2
    idx.add(x2)
    dq = torch.from_numpy(q).cuda()
    dD = torch.empty((m, k), device="cuda")
    dI = torch.empty((m, k), dtype=torch.int64, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        idx.search_device(m, dq.data_ptr(), k, dD.data_ptr(), dI.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for a, b in zip((D, I), idx.search(q, k)):  # before any replay
        np.testing.assert_array_equal(a, b)
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dI.cpu().numpy(), I)
    np.testing.assert_array_equal(dD.cpu().numpy(), D)


@pytest.mark.parametrize("opt", [hb.OPT_NONE, hb.OPT_TRIANGLE])
@pytest.mark.parametrize("nlist,n,m,nprobe", [(128, 40_000, 4_000, 32), (128, 40_000, 4_000, 128),
                                              (64, 1_500_000, 15, 16)])
def test_plain_batch_captured_after_an_add(opt, nlist, n, m, nprobe):
    """Large plain batches: the capture runs the list-major or the query-major
    scan, whose buffers the searches before have left large enough."""
    rng = np.random.default_rng(9)
    d, k = 64, 10
    c = (20 * rng.standard_normal((nlist, d))).astype(np.float32)
    lab = rng.integers(0, nlist, n)
    x1, x2 = ((c[lab] + rng.standard_normal((n, d))).astype(np.float32) for _ in range(2))
    q = (c[rng.integers(0, nlist, m)] + rng.standard_normal((m, d))).astype(np.float32)
    idx = hb.Index(d, nlist, nprobe, opt_level=opt)
    idx.centroid_codes = c
    idx.add(x2)
    assert m * nprobe * n / nlist * d * 4 > 1.2e9
    D, I = idx.search(q, k)
    idx = hb.Index(d, nlist, nprobe, opt_level=opt)
    idx.centroid_codes = c
    idx.add(x1)
    dq = torch.from_numpy(q).cuda()
    dD = torch.empty((m, k), device="cuda")
    dI = torch.empty((m, k), dtype=torch.int64, device="cuda")

    def search():
        idx.search_device(m, dq.data_ptr(), k, dD.data_ptr(), dI.data_ptr(), torch.cuda.current_stream().cuda_stream)

    search()
    assert idx.last_stats()["list_major"] == 0
    idx.add(x2)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        search()
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dI.cpu().numpy(), I)
    np.testing.assert_array_equal(dD.cpu().numpy(), D)
