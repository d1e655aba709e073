"""Tensor-core assignment of rows to centroids (k-means and add): the lists
equal the ones of the exact kernels, which assign the same rows in batches
below the tensor-core rule, and the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402
from harmonyclient_b200 import _lib  # noqa: E402
from oracle import port  # noqa: E402

EXACT_MAX = (1 << 29) - 1  # rows x centroids x dimensions below the tensor-core rule


def _labels(idx, x):
    """Label of every row, from one add."""
    idx.add(x)
    lab = np.full(len(x), -1, np.int64)
    for l in range(idx.nlist):
        lab[idx.get_list(l)[0]] = l
    return lab


def _exact_labels(idx, x):
    m = EXACT_MAX // (4 * idx.nlist * x.shape[1])
    return np.concatenate([_labels(idx, x[s:s + m]) for s in range(0, len(x), m)])


def _check(x, cent, metric=hb.METRIC_L2):
    # the rule counts rows: the sample is repeated up to it
    reps = EXACT_MAX // (len(x) * len(cent) * x.shape[1]) + 1
    x = np.concatenate([x] * min(reps, 1 + 400_000 // len(x)))
    assert x.shape[0] * len(cent) * x.shape[1] > EXACT_MAX
    idx = hb.Index(x.shape[1], len(cent), 1, metric)
    idx.centroid_codes = cent
    np.testing.assert_array_equal(_labels(idx, x), _exact_labels(idx, x))
    return idx


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("d,nlist,n", [(1, 2_000, 300_001), (16, 128, 280_001), (63, 129, 70_001),
                                       (64, 1_000, 9_001), (65, 257, 33_001), (128, 1_024, 4_097), (130, 200, 21_001),
                                       (200, 64, 43_001), (256, 300, 7_001)])
def test_float_rows(metric, d, nlist, n):
    rng = np.random.default_rng(d * 7 + nlist)
    c = rng.uniform(-3, 3, (nlist, d)).astype(np.float32)
    x = (c[rng.integers(0, nlist, n)] + rng.standard_normal((n, d))).astype(np.float32)
    _check(x, c, metric)


def test_close_centroids():
    """Centroids a few ulp apart, twice and three times the same one: two
    candidates, undecided rows, and ties to the lower centroid."""
    rng = np.random.default_rng(3)
    c = rng.uniform(0, 100, (400, 48)).astype(np.float32)
    c[100:200] = c[:100]
    c[200:250] = c[:50]
    c[250:300] = np.nextafter(c[50:100], np.float32(1e9))
    x = (c[rng.integers(0, 400, 6_000)] + 2 * rng.standard_normal((6_000, 48))).astype(np.float32)
    _check(x, c)
    x = np.concatenate([x] * 5)
    idx = hb.Index(48, 400, 1)
    idx.centroid_codes = c
    idx.add(x)
    lists = port.build_lists(x, c)
    for l in (0, 60, 150, 220, 299, 399):
        np.testing.assert_array_equal(idx.get_list(l)[0], lists.ids[lists.offsets[l]:lists.offsets[l + 1]])


@pytest.mark.parametrize("kind", ["integers", "zeros", "huge", "tiny", "nonfinite", "offset"])
def test_value_ranges(kind):
    rng = np.random.default_rng(11)
    c = rng.integers(0, 256, (300, 33)).astype(np.float32)
    x = np.clip(c[rng.integers(0, 300, 5_000)] + rng.integers(-9, 10, (5_000, 33)), 0, 255).astype(np.float32)
    if kind == "zeros":
        x[::3] = 0
        c[7] = 0
    elif kind == "huge":
        x[::5] *= np.float32(1e17)
        x[1::5] *= np.float32(1e19)
        c[3] *= np.float32(1e18)
    elif kind == "tiny":
        x *= np.float32(1e-24)
        c *= np.float32(1e-24)
        x[::2] *= np.float32(1e-16)
    elif kind == "nonfinite":
        x[5, 2], x[6, 3], x[7, 4] = np.inf, -np.inf, np.nan
        x[8] = np.nan
    elif kind == "offset":
        x += 40_000
        c += 40_000
    _check(x, c)


def test_nonfinite_centroid():
    rng = np.random.default_rng(12)
    c = rng.standard_normal((256, 20)).astype(np.float32)
    c[9, 1], c[10, 1] = np.nan, np.inf
    _check(rng.standard_normal((5_000, 20)).astype(np.float32), c)


def test_list_order_is_the_exact_scores():
    """Rows within a list are ordered by their exact score."""
    rng = np.random.default_rng(13)
    c = rng.uniform(0, 50, (128, 70)).astype(np.float32)
    x = (c[rng.integers(0, 128, 61_000)] + 3 * rng.standard_normal((61_000, 70))).astype(np.float32)
    idx = hb.Index(70, 128, 1)
    idx.centroid_codes = c
    idx.add(x)
    for l in range(0, 128, 17):
        ids = idx.get_list(l)[0]
        t = np.zeros(len(ids), np.float32)
        for j in range(70):  # sequential float32, separately rounded
            dlt = (x[ids, j] - c[l, j]).astype(np.float32)
            t = (t + (dlt * dlt).astype(np.float32)).astype(np.float32)
        assert np.all(np.diff(t) >= 0)


@pytest.mark.parametrize("nlist,d", [(300, 33), (129, 64), (65, 200)])
def test_scores_that_all_overflow(nlist, d):
    """Finite rows whose score against every centroid overflows, beside list
    counts that are no multiple of the tile: the exact kernel's labels."""
    rng = np.random.default_rng(nlist)
    c = rng.integers(1, 256, (nlist, d)).astype(np.float32)
    x = np.clip(c[rng.integers(0, nlist, 5_000)] + rng.integers(-9, 10, (5_000, d)), 0, 255).astype(np.float32)
    x[::7] = -1e37 * rng.uniform(0.9, 1.1, (len(x[::7]), d))
    _check(x, c)
    _check(x, c, hb.METRIC_IP)
    # rows and centroids whose squared norms overflow
    _check(rng.uniform(3e19, 6e19, (5_000, d)).astype(np.float32), c * np.float32(1e19))


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
def test_a_wait_that_gives_up(metric):
    """Device-side waits that run out at their first poll: train and add
    report it and leave the centroids and the lists as they were."""
    L = _lib.load()
    rng = np.random.default_rng(14)
    x = rng.uniform(0, 50, (70_000, 70)).astype(np.float32)
    q = x[:50] + np.float32(0.5)
    idx = hb.Index(70, 130, 8, metric)
    assert len(x) * 130 * 70 > EXACT_MAX and 130 * 256 * 130 * 70 < EXACT_MAX  # add runs there, train does not
    idx.train(x)
    idx.add(x)
    cent = idx.centroid_codes.copy()
    D, I = idx.search(q, 5)
    fresh = hb.Index(70, 1_000, 8, metric)  # its train runs there too
    _lib.check(L.hy_selftest_wait_limit(idx._h, 0))
    _lib.check(L.hy_selftest_wait_limit(fresh._h, 0))
    with pytest.raises(_lib.HyError) as e:
        idx.add(x[::-1].copy())
    assert e.value.code == _lib.HY_ERR_TIMEOUT
    with pytest.raises(_lib.HyError) as e:
        fresh.train(x)
    assert e.value.code == _lib.HY_ERR_TIMEOUT
    np.testing.assert_array_equal(idx.centroid_codes, cent)
    for a, b in zip((D, I), idx.search(q, 5)):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(_lib.HyError) as e:
        fresh.add(x)
    assert e.value.code == _lib.HY_ERR_STATE
    # a trained index keeps its centroids
    _lib.check(L.hy_selftest_wait_limit(fresh._h, 1 << 31))
    fresh.train(x)
    fresh.add(x)
    cent = fresh.centroid_codes.copy()
    D, I = fresh.search(q, 5)
    _lib.check(L.hy_selftest_wait_limit(fresh._h, 0))
    with pytest.raises(_lib.HyError):
        fresh.train(x + np.float32(3))
    np.testing.assert_array_equal(fresh.centroid_codes, cent)
    for a, b in zip((D, I), fresh.search(q, 5)):
        np.testing.assert_array_equal(a, b)
    # and with the limit back, the same calls go through
    _lib.check(L.hy_selftest_wait_limit(idx._h, 1 << 31))
    _lib.check(L.hy_selftest_wait_limit(fresh._h, 1 << 31))
    np.testing.assert_array_equal(_labels(idx, x), _exact_labels(idx, x))
    np.testing.assert_array_equal(_labels(fresh, x), _exact_labels(fresh, x))
