"""The coarse step's small-batch kernels (scores and selection): the probes are
the large-batch kernels', which score the same queries repeated past the
small-batch rule, ties to the lower list included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("nq,nlist,nprobe,d", [(1, 1, 1, 1), (1, 33, 33, 7), (9, 100, 32, 128), (8, 1024, 64, 129),
                                               (64, 2049, 65, 256), (128, 700, 256, 30), (129, 1024, 128, 257),
                                               (148, 4096, 33, 16), (3, 4097, 256, 20), (2, 600, 300, 12)])
def test_small_batches_equal_large(metric, nq, nlist, nprobe, d):
    rng = np.random.default_rng(nlist + d)
    c = rng.integers(-20, 21, (nlist, d)).astype(np.float32)
    c[nlist // 2:] += rng.standard_normal((nlist - nlist // 2, d)).astype(np.float32)
    c[::7] = c[0]  # equal lists: ties
    q = rng.integers(-20, 21, (nq, d)).astype(np.float32)
    idx = hb.Index(d, nlist, nprobe, metric)
    idx.centroid_codes = c
    idx.set_coarse("exact")
    reps = -(-400 // nq)
    P = idx.probes(q)
    np.testing.assert_array_equal(P, idx.probes(np.concatenate([q] * reps))[:nq])


def test_nonfinite_queries():
    rng = np.random.default_rng(2)
    idx = hb.Index(20, 300, 40)
    idx.centroid_codes = rng.standard_normal((300, 20)).astype(np.float32)
    idx.set_coarse("exact")
    q = rng.standard_normal((6, 20)).astype(np.float32)
    q[0, 1], q[1, 2], q[2] = np.inf, np.nan, -np.inf
    np.testing.assert_array_equal(idx.probes(q), idx.probes(np.concatenate([q] * 70))[:6])
