"""Training on more rows than are sampled: the reference's sample and initial
centroids, at the sizes where the plan's two ways of drawing them meet."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402
from oracle import port  # noqa: E402


@pytest.mark.parametrize("n,nlist", [(65_537, 256), (65_792, 257), (65_793, 257), (150_001, 300)])
def test_centroids_of_a_sample(n, nlist):
    # Whole numbers: the sums are exact in any order, so the steps from the
    # same rows and centroids are the same.
    rng = np.random.default_rng(n)
    x = rng.integers(0, 64, (n, 3)).astype(np.float32)
    x[:, 0] += 4096.0 * (np.arange(n) % 11)
    idx = hb.Index(3, nlist, 1)
    idx.train(x)
    np.testing.assert_allclose(idx.centroid_codes, port.kmeans(x, nlist, fp64=True), rtol=1e-5, atol=1e-4)
