"""Values whose squares and products underflow: the tensor-core searches still
give the plain scan's answer, entry for entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("xs,qs", [(1e-14, 1e-14), (1e-18, 1e-18), (1e-20, 1e-20), (1e-25, 1e-5), (1e-25, 1e-18),
                                   (1e-8, 1e-25)])
@pytest.mark.parametrize("form", ["plain", "bf16"])
def test_scaled_rows_and_queries(metric, xs, qs, form):
    rng = np.random.default_rng(7)
    nlist, d, n, m, k = 64, 96, 30_000, 1_200, 10
    c = rng.standard_normal((nlist, d)).astype(np.float32)
    x = c[rng.integers(0, nlist, n)] + np.float32(0.4) * rng.standard_normal((n, d)).astype(np.float32)
    q = c[rng.integers(0, nlist, m)] + np.float32(0.4) * rng.standard_normal((m, d)).astype(np.float32)
    x, q, c = x * np.float32(xs), q * np.float32(qs), c * np.float32(xs)
    # Every probe is taken, so the answer does not depend on the coarse step.
    idx = hb.Index(d, nlist, nlist, metric)
    idx.centroid_codes = c
    idx.add(x)
    assert m * n * d * 4 > 600e6
    idx.set_plain_scan("query")
    want = idx.search(q, k)
    idx.set_plain_scan("auto")
    idx.set_form(form)
    for a, b in zip(want, idx.search(q, k)):
        np.testing.assert_array_equal(a, b)
    # The coarse step: the exact kernel's probes.
    idx.nprobe = 7
    idx.set_coarse("exact")
    probes = idx.probes(q)
    idx.set_coarse("tensor")
    np.testing.assert_array_equal(idx.probes(q), probes)


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
def test_tiny_rows_among_others(metric):
    """Ordinary rows and queries with some tiny and some zero ones among them."""
    rng = np.random.default_rng(8)
    nlist, d, n, m, k = 64, 96, 30_000, 1_200, 10
    c = rng.standard_normal((nlist, d)).astype(np.float32)
    x = c[rng.integers(0, nlist, n)] + np.float32(0.4) * rng.standard_normal((n, d)).astype(np.float32)
    q = c[rng.integers(0, nlist, m)] + np.float32(0.4) * rng.standard_normal((m, d)).astype(np.float32)
    x[::50] *= np.float32(1e-21)
    x[1::500] = 0
    q[::9] *= np.float32(1e-19)
    q[1::9] = 0
    idx = hb.Index(d, nlist, nlist, metric)
    idx.centroid_codes = c
    idx.add(x)
    idx.set_plain_scan("query")
    want = idx.search(q, k)
    idx.set_plain_scan("auto")
    for form in ("plain", "bf16"):
        idx.set_form(form)
        for a, b in zip(want, idx.search(q, k)):
            np.testing.assert_array_equal(a, b)
