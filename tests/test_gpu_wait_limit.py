"""Batched tensor-core scans whose device-side waits give up: the host call
reports it, no matter how far the scan had come, and the next call answers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import harmonyclient_b200 as hb  # noqa: E402
from harmonyclient_b200 import _lib  # noqa: E402

NO_LIMIT = 1 << 31


@pytest.mark.parametrize("form,d,nlist", [("plain", 64, 100), ("bf16", 40, 100), ("bf16", 300, 2_300),
                                          ("fp8", 130, 64)])
def test_search_reports_it_and_recovers(form, d, nlist):
    rng = np.random.default_rng(d)
    c = rng.uniform(-3, 3, (nlist, d)).astype(np.float32)
    x = (c[rng.integers(0, nlist, 60_000)] + rng.standard_normal((60_000, d))).astype(np.float32)
    q = (c[rng.integers(0, nlist, 1_500)] + rng.standard_normal((1_500, d))).astype(np.float32)
    idx = hb.Index(d, nlist, 16)
    idx.centroid_codes = c
    idx.add(x)
    idx.set_form(form)
    want = idx.search(q, 10)
    L = _lib.load()
    # Polls: none at all, then so few that some waits pass and others do not.
    for polls in (0, 1, 4, 64):
        _lib.check(L.hy_selftest_wait_limit(idx._h, polls))
        try:
            got = idx.search(q, 10)
            assert polls > 0
            for a, b in zip(want, got):
                np.testing.assert_array_equal(a, b)
        except _lib.HyError as e:
            assert e.code == _lib.HY_ERR_TIMEOUT
        _lib.check(L.hy_selftest_wait_limit(idx._h, NO_LIMIT))
        for a, b in zip(want, idx.search(q, 10)):
            np.testing.assert_array_equal(a, b)
