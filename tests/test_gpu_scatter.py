"""Rows laid into the lists 32 at a time: every list's rows, ids and norms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4097])
@pytest.mark.parametrize("d,blocks", [(1, 1), (32, 1), (33, 2), (130, 4), (263, 8)])
def test_lists_hold_the_rows(n, d, blocks):
    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    idx = hb.Index(d, 7, 7, dim_blocks=blocks)
    idx.centroid_codes = rng.standard_normal((7, d)).astype(np.float32)
    idx.add(x)
    seen = []
    for l in range(7):
        ids, codes, norms = idx.get_list(l)
        np.testing.assert_array_equal(codes, x[ids])
        s = np.zeros(len(ids), np.float32)
        for j in range(d):  # in dimension order
            s += codes[:, j] * codes[:, j]
        np.testing.assert_array_equal(norms, s)
        seen.append(ids)
    np.testing.assert_array_equal(np.sort(np.concatenate(seen)), np.arange(n))
    q = x[:200]
    D, I = idx.search(q, 3)
    idx.set_form("bf16")  # scores from the stored norms, re-ranked exactly
    Db, Ib = idx.search(q, 3)
    np.testing.assert_array_equal(Ib, I)
    np.testing.assert_array_equal(Db, D)
