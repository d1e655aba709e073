"""The tensor-core coarse step above 256 dimensions (centroids re-scored in runs
of 128 dimensions): its probes and a search's answer equal the exact step's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


def _probes(idx, q, mode):
    idx.set_coarse(mode)
    return idx.probes(q)


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("d,nlist,nprobe", [(257, 300, 40), (260, 1024, 129), (384, 128, 128), (420, 2048, 64),
                                            (500, 2048, 256), (511, 700, 1), (768, 513, 200)])
def test_probes_equal_exact(metric, d, nlist, nprobe):
    rng = np.random.default_rng(d)
    c = rng.uniform(-1, 1, (nlist, d)).astype(np.float32)
    c[::9] = c[4]  # equal lists
    q = (c[rng.integers(0, nlist, 333)] + 0.3 * rng.standard_normal((333, d))).astype(np.float32)
    q[7] = 0
    idx = hb.Index(d, nlist, nprobe, metric)
    idx.centroid_codes = c
    np.testing.assert_array_equal(_probes(idx, q, "tensor"), _probes(idx, q, "exact"))


@pytest.mark.parametrize("what", ["query", "centroid"])
def test_nonfinite_values(what):
    rng = np.random.default_rng(5)
    c = rng.standard_normal((400, 300)).astype(np.float32)
    q = rng.standard_normal((300, 300)).astype(np.float32)
    v = q if what == "query" else c
    v[3, 5], v[4, 6], v[5] = np.inf, -np.inf, 3e19
    idx = hb.Index(300, 400, 50)
    idx.centroid_codes = c
    np.testing.assert_array_equal(_probes(idx, q, "tensor"), _probes(idx, q, "exact"))


@pytest.mark.parametrize("form", ["plain", "bf16", "fp8"])
def test_search_in_every_form(form):
    rng = np.random.default_rng(6)
    c = rng.uniform(-1, 1, (64, 420))
    x = (c[rng.integers(0, 64, 20_000)] + 0.2 * rng.standard_normal((20_000, 420))).astype(np.float32)
    q = (c[rng.integers(0, 64, 2_000)] + 0.2 * rng.standard_normal((2_000, 420))).astype(np.float32)
    idx = hb.Index(420, 128, 16)
    idx.centroid_codes = x[:128]
    idx.add(x)
    idx.set_form(form)
    idx.set_coarse("exact")
    D, I = idx.search(q, 10)
    idx.set_coarse("tensor")
    Dt, It = idx.search(q, 10)
    np.testing.assert_array_equal(It, I)
    np.testing.assert_array_equal(Dt, D)


@pytest.mark.parametrize("form", ["plain", "fp8", "bf16"])
@pytest.mark.parametrize("nq,tensor", [(1_907, False), (1_908, True)])
def test_small_batches_of_the_other_forms_keep_the_exact_step(form, nq, tensor):
    """2048 lists x 64 dimensions: from 250 million products the plain and e4m3
    forms score on the tensor cores too (the bf16 form always does)."""
    rng = np.random.default_rng(9)
    c = rng.uniform(-1, 1, (2048, 64)).astype(np.float32)
    x = (c[rng.integers(0, 2048, 60_000)] + 0.3 * rng.standard_normal((60_000, 64))).astype(np.float32)
    q = (c[rng.integers(0, 2048, nq)] + 0.3 * rng.standard_normal((nq, 64))).astype(np.float32)
    idx = hb.Index(64, 2048, 128)
    idx.centroid_codes = c
    idx.add(x)
    idx.set_form(form)
    out, launches = {}, {}
    for mode in ("exact", "tensor"):
        idx.set_coarse(mode)
        out[mode] = idx.search(q, 10)
        launches[mode] = idx.last_stats()["launches"]
    for a, b in zip(out["exact"], out["tensor"]):
        np.testing.assert_array_equal(a, b)
    assert (launches["exact"] != launches["tensor"]) == (tensor or form == "bf16")
