"""Query groups of the batched kernel in one buffer or two, at each row width
where the layout changes: the plain and bf16 answers are the list-major
scan's, and every group size's answer is the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402

# 128-byte k-blocks per row; the largest group is 128 queries in two buffers to
# 3, 128 in one to 8, 64 in one above.
KBLOCKS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12]
PER_BLOCK = {"plain": 32, "bf16": 64, "fp8": 128}


@pytest.mark.parametrize("form", ["plain", "bf16", "fp8"])
@pytest.mark.parametrize("nkb", KBLOCKS)
@pytest.mark.parametrize("odd", [0, 7])
def test_answer_of_every_group(form, nkb, odd):
    d = nkb * PER_BLOCK[form] - odd
    rng = np.random.default_rng(d)
    c = rng.uniform(0, 50, (12, d))
    # lists of about 200 to 2,400 rows: a few tiles, and several slices
    w = np.linspace(1, 12, 12)
    x = (c[rng.choice(12, 16_000, p=w / w.sum())] + 4 * rng.standard_normal((16_000, d))).astype(np.float32)
    q = (c[rng.integers(0, 12, 777)] + 4 * rng.standard_normal((777, d))).astype(np.float32)
    # blocks that the fallback scan takes (the plain form pads each to whole k-blocks)
    blocks = (1 if d <= 192 else 2) if form == "plain" else (8 if d > 500 else 4)
    idx = hb.Index(d, 12, 7, dim_blocks=blocks)
    idx.centroid_codes = c.astype(np.float32)
    idx.add(x)
    if form == "fp8":  # re-ranks its best candidates only: the oracle is its own answer in groups of 32
        idx.set_form(form)
        idx.set_batch_params(oversample=1000)
        idx.set_group_size(32)
    else:
        idx.set_plain_scan("list")
    D, I = idx.search(q, 11)
    idx.set_plain_scan("auto")
    idx.set_form(form)
    for group in (32, 64, 128, 0):
        idx.set_group_size(group)
        Dt, It = idx.search(q, 11)
        assert idx.last_stats()["list_major"] == 0
        np.testing.assert_array_equal(It, I)
        np.testing.assert_array_equal(Dt, D)
