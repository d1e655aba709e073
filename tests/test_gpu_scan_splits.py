"""The query-major plain scan's work splits: few queries over many CTAs (tile
splits), probe tables cut into parts, and the fallback whose splits follow
from a device count of overflowed queries.  Oracle: the list-major scan (same
arithmetic, other work distribution), entry for entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import harmonyclient_b200 as hb  # noqa: E402


def _skewed(rng, nlist, d, n):
    """Integer rows in lists of very uneven sizes (1 to about n / 4 rows)."""
    cent = rng.integers(0, 200, (nlist, d)).astype(np.float32)
    w = 1.0 / np.arange(1, nlist + 1)
    lab = rng.choice(nlist, size=n, p=w / w.sum())
    x = np.clip(np.rint(cent[lab] + 12 * rng.standard_normal((n, d))), 0, 255).astype(np.float32)
    return cent, x


@pytest.mark.parametrize("nq,k,nprobe,d", [(1, 1, 1, 97), (1, 256, 64, 32), (3, 33, 60, 97), (37, 17, 64, 40),
                                           (38, 100, 7, 130), (149, 65, 33, 32), (300, 10, 64, 16)])
@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
def test_tile_splits_equal_list_major(nq, k, nprobe, d, metric):
    rng = np.random.default_rng(nq * 1000 + k)
    cent, x = _skewed(rng, 64, d, 12_000)
    idx = hb.Index(d, 64, nprobe, metric)
    idx.centroid_codes = cent
    idx.add(x)
    q = x[rng.choice(len(x), nq)] + rng.integers(-3, 4, (nq, d)).astype(np.float32)
    idx.set_plain_scan("query")
    D, I = idx.search(q, k)
    assert idx.last_stats()["list_major"] == 0
    idx.set_plain_scan("list")
    Dl, Il = idx.search(q, k)
    np.testing.assert_array_equal(I, Il)
    np.testing.assert_array_equal(D, Dl)


def test_probe_table_in_parts():
    """nprobe above the probe table of one part (2048): two parts, each cut
    into tile splits."""
    rng = np.random.default_rng(5)
    x = rng.integers(0, 256, (6_000, 24)).astype(np.float32)
    idx = hb.Index(24, 2_500, 2_300)
    idx.centroid_codes = x[:2_500]
    idx.add(x)
    q = x[::977][:5] + 1
    idx.set_plain_scan("query")
    D, I = idx.search(q, 40)
    idx.set_plain_scan("list")
    Dl, Il = idx.search(q, 40)
    np.testing.assert_array_equal(I, Il)
    np.testing.assert_array_equal(D, Dl)


@pytest.mark.parametrize("noverflow", [1, 5, 160])
def test_fallback_of_a_counted_few(noverflow):
    """noverflow queries sit in lists of more rows than their candidate
    buffers hold, the others in small lists: the counted queries alone go
    through the fallback, whose splits follow from their number."""
    rng = np.random.default_rng(9)
    cent = (rng.integers(0, 2, (32, 48)) * 200 + rng.integers(0, 40, (32, 48))).astype(np.float32)
    lab = np.concatenate([np.full(6_000, 0), rng.integers(1, 32, 3_000)])
    x = np.clip(np.rint(cent[lab] + 3 * rng.standard_normal((len(lab), 48))), 0, 255).astype(np.float32)
    idx = hb.Index(48, 32, 1)
    idx.centroid_codes = cent
    idx.add(x)
    q = np.concatenate([x[:noverflow], x[6_000:6_200]])
    D, I = idx.search(q, 200)
    idx.set_form("bf16")
    idx.set_batch_params(capq=256)  # below list 0's rows, above the other lists'
    Db, Ib = idx.search(q, 200)
    assert idx.last_stats()["fallback_queries"] == noverflow
    np.testing.assert_array_equal(Ib, I)
    np.testing.assert_array_equal(Db, D)


@pytest.mark.parametrize("d,blocks,nlist,nprobes", [(768, 4, 900, range(880, 900, 2)), (192, 6, 2_100, (2_040, 2_048)),
                                                     (384, 4, 3_000, (2_990,))])
def test_probe_tables_that_fill_the_shared_memory(d, blocks, nlist, nprobes):
    """Large k and probe counts about the largest table that fits beside the
    kernel's staging: the answer of the smaller k, few queries and many."""
    rng = np.random.default_rng(d)
    x = rng.standard_normal((6_000, d)).astype(np.float32)
    idx = hb.Index(d, nlist, nprobes[0], dim_blocks=blocks)
    idx.centroid_codes = x[:nlist]
    idx.add(x)
    idx.set_plain_scan("query")
    for nprobe in nprobes:
        idx.nprobe = nprobe
        for n in (8, 300):
            D, I = idx.search(x[:n], 256)
            D1, I1 = idx.search(x[:n], 64)
            np.testing.assert_array_equal(D[:, :64], D1)
            np.testing.assert_array_equal(I[:, :64], I1)
