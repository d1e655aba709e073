"""A search's coarse step that leaves its probes unordered (their exact scores
only where the bounds do not decide): the answer equals the exact step's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


def _same(idx, q, k=10):
    idx.set_form("bf16")
    idx.set_coarse("exact")
    D, I = idx.search(q, k)
    idx.set_coarse("tensor")
    Dt, It = idx.search(q, k)
    np.testing.assert_array_equal(It, I)
    np.testing.assert_array_equal(Dt, D)


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("d,nlist,nprobe", [(8, 5, 5), (8, 40, 1), (33, 300, 2), (64, 1024, 3), (128, 1024, 64),
                                            (128, 1000, 256), (200, 64, 63), (420, 2048, 4), (420, 1500, 200)])
def test_answer_equals_exact_step(metric, d, nlist, nprobe):
    rng = np.random.default_rng(d + nlist)
    c = rng.uniform(-1, 1, (nlist, d)).astype(np.float32)
    c[4::9] = c[4]  # equal lists: only the lower ones may be probed
    c[2::11] = 0
    x = (c[rng.integers(0, nlist, 9_000)] + 0.3 * rng.standard_normal((9_000, d))).astype(np.float32)
    q = (c[rng.integers(0, nlist, 500)] + 0.5 * rng.standard_normal((500, d))).astype(np.float32)
    q[3], q[4] = 0, c[4]
    idx = hb.Index(d, nlist, nprobe, metric)
    idx.centroid_codes = c
    idx.add(x)
    _same(idx, q)


@pytest.mark.parametrize("what", ["query", "centroid"])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3e19, -1e30])
@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
def test_nonfinite_values(metric, what, bad):
    rng = np.random.default_rng(5)
    c = rng.standard_normal((200, 40)).astype(np.float32)
    x = (c[rng.integers(0, 200, 5_000)] + 0.3 * rng.standard_normal((5_000, 40))).astype(np.float32)
    q = rng.standard_normal((300, 40)).astype(np.float32)
    idx = hb.Index(40, 200, 30, metric)
    idx.centroid_codes = c
    idx.add(x)
    if what == "query":
        q[3, 5] = bad
    else:
        c[7, 5] = c[150, 0] = bad
        idx.centroid_codes = c
    probes = {}
    for mode in ("exact", "tensor"):
        idx.set_coarse(mode)
        idx.set_form("bf16")
        probes[mode] = np.sort(idx.probes(q), axis=1)
    np.testing.assert_array_equal(probes["tensor"], probes["exact"])
    _same(idx, np.delete(q, 3, 0) if what == "query" and not np.isfinite(bad) else q)


@pytest.mark.parametrize("d,nlist,nprobe", [(24, 40, 40), (128, 1024, 64), (48, 2049, 128), (64, 4096, 200)])
def test_each_query_its_own_nprobe(d, nlist, nprobe):
    """From two launches above 2048 lists; counts of 1, nprobe and past it."""
    rng = np.random.default_rng(nlist)
    c = rng.uniform(-1, 1, (nlist, d)).astype(np.float32)
    c[4::9] = c[4]
    x = (c[rng.integers(0, nlist, 9_000)] + 0.3 * rng.standard_normal((9_000, d))).astype(np.float32)
    q = (c[rng.integers(0, nlist, 700)] + 0.4 * rng.standard_normal((700, d))).astype(np.float32)
    idx = hb.Index(d, nlist, nprobe)
    idx.centroid_codes = c
    idx.add(x)
    idx.set_form("bf16")
    npq = rng.integers(1, nprobe + 1, 700).astype(np.int32)
    npq[:3] = 1, nprobe, nprobe
    out = {}
    for mode in ("exact", "tensor"):
        idx.set_coarse(mode)
        out[mode] = idx.search_nprobes(q, 10, npq)
        if mode == "tensor":
            _same(idx, q)
    for a, b in zip(out["exact"], out["tensor"]):
        np.testing.assert_array_equal(a, b)
