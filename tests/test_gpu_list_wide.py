"""The list-major scan's block widths: one to four groups of 32 dimensions per
block (registers), wider ones (group by group), blocks of unequal width, against
the query-major scan, entry for entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("d,dim_blocks", [(130, 4), (200, 4), (257, 4), (385, 4), (100, 1), (64, 1), (97, 2), (300, 3),
                                          (512, 4), (160, 1), (150, 1), (70, 8)])
@pytest.mark.parametrize("metric,warm", [(hb.METRIC_L2, 0), (hb.METRIC_L2, 10), (hb.METRIC_IP, 0)])
def test_equals_query_major(d, dim_blocks, metric, warm):
    rng = np.random.default_rng(d)
    c = rng.uniform(-1, 1, (40, d))
    x = (c[rng.integers(0, 40, 3_001)] + 0.2 * rng.standard_normal((3_001, d))).astype(np.float32)
    q = (c[rng.integers(0, 40, 203)] + 0.2 * rng.standard_normal((203, d))).astype(np.float32)
    idx = hb.Index(d, 20, 9, metric, dim_blocks=dim_blocks)
    idx.centroid_codes = x[:20]
    idx.add(x)
    idx.preSearch(warmUpSearchList=warm, warmUpSearchListSize=21)
    idx.set_plain_scan("list")
    Dl, Il = idx.search(q, 21)
    st = idx.last_stats()
    assert st["list_major"] == 1 and 0 < st["seg_sums"] <= st["seg_sums_max"]
    if metric == hb.METRIC_IP:
        assert st["seg_sums"] == st["seg_sums_max"]  # nothing is pruned
    idx.set_plain_scan("query")
    D, I = idx.search(q, 21)
    np.testing.assert_array_equal(Il, I)
    np.testing.assert_array_equal(Dl, D)
