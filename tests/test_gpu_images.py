"""The bf16 and e4m3 images of the lists: block widths that are and are no
multiple of the chunks they are written in, rows that end inside a k-block.
A search over a right image gives the plain form's answer entry for entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("metric", [hb.METRIC_L2, hb.METRIC_IP])
@pytest.mark.parametrize("form", ["bf16", "fp8"])
@pytest.mark.parametrize("d,blocks", [(1, 1), (15, 2), (63, 4), (64, 1), (97, 4), (129, 8), (420, 4), (500, 4), (768, 8)])
def test_forms_equal_plain(form, d, blocks, metric):
    rng = np.random.default_rng(d + blocks)
    x = (rng.standard_normal((2500, d)) * np.exp(rng.uniform(-3, 3, d))).astype(np.float32)
    x[7] = 0.0
    q = x[::25] + 0.1 * rng.standard_normal((100, d)).astype(np.float32)
    idx = hb.Index(d, 9, 4, metric, dim_blocks=blocks)
    idx.centroid_codes = x[:9]
    idx.add(x)
    D, I = idx.search(q, 10)
    idx.set_form(form)
    if form == "fp8":
        idx.set_batch_params(oversample=1000)
    Df, If = idx.search(q, 10)
    np.testing.assert_array_equal(If, I)
    np.testing.assert_array_equal(Df, D)
