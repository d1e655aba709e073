"""The plain form's choice among its scans where the tensor cores are the slower
one: few queries over long lists, large k, inner products over lists past the
candidate buffer.  Every choice gives the query-major scan's answer, entry for
entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402

QUERY, LIST, TENSOR = "query", "list", "tensor"


@pytest.mark.parametrize("metric,d,n,nlist,nprobe,k,m,scan", [
    (hb.METRIC_L2, 48, 300_000, 250, 100, 20, 12, QUERY),     # few queries
    (hb.METRIC_L2, 48, 300_000, 250, 100, 20, 64, TENSOR),    # no longer few
    (hb.METRIC_L2, 48, 300_000, 60, 60, 20, 12, TENSOR),      # few, but every list shared
    (hb.METRIC_L2, 130, 300_000, 250, 90, 20, 12, TENSOR),    # few, but wide rows
    (hb.METRIC_L2, 48, 300_000, 250, 250, 20, 12, TENSOR),    # many rows each
    (hb.METRIC_L2, 48, 90_000, 500, 2, 176, 4_000, LIST),     # k of the size of what is scanned
    (hb.METRIC_L2, 48, 90_000, 500, 2, 177, 4_000, TENSOR),   # the same, and tight in TF32
    (hb.METRIC_IP, 48, 90_000, 500, 2, 179, 4_000, TENSOR),   # under half of it
    (hb.METRIC_IP, 48, 90_000, 500, 2, 181, 4_000, LIST),     # inner products, over half
    (hb.METRIC_L2, 32, 90_000, 1_500, 150, 250, 200, LIST),   # no two lists hold k rows
    (hb.METRIC_L2, 48, 90_000, 500, 2, 60, 4_000, TENSOR),    # smaller k
    (hb.METRIC_L2, 48, 18_000, 100, 2, 176, 4_000, TENSOR),   # many queries a list
    (hb.METRIC_L2, 32, 30_000, 500, 1, 90, 10_000, LIST),     # many queries, few rows each
    (hb.METRIC_L2, 32, 30_000, 500, 1, 5, 1_000, QUERY),
    (hb.METRIC_IP, 20, 200_000, 16, 3, 10, 300, QUERY),       # lists past the candidate buffer
    (hb.METRIC_IP, 20, 200_000, 64, 12, 10, 300, TENSOR),
    (hb.METRIC_L2, 20, 200_000, 16, 3, 10, 300, TENSOR),
])
def test_scan_and_answer(metric, d, n, nlist, nprobe, k, m, scan):
    rng = np.random.default_rng(n + nlist)
    # far from the origin next to their spread, so that TF32 separates less
    # (k 177: close to it)
    c = ((0.5 if k == 177 else 8) * rng.standard_normal((nlist, d))).astype(np.float32)
    x = (c[rng.integers(0, nlist, n)] + rng.standard_normal((n, d))).astype(np.float32)
    q = (c[rng.integers(0, nlist, m)] + rng.standard_normal((m, d))).astype(np.float32)
    idx = hb.Index(d, nlist, nprobe, metric)
    idx.centroid_codes = c
    idx.add(x)
    idx.set_plain_scan("query")
    want = idx.search(q, k)
    idx.set_plain_scan("auto")
    for a, b in zip(want, idx.search(q, k)):
        np.testing.assert_array_equal(a, b)
    st = idx.last_stats()
    took = LIST if st["list_major"] else QUERY if st["tile_blocks"] else TENSOR
    assert took == scan
