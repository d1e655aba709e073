"""A captured search holds the handle's workspaces: a call between two identical
graph searches that makes one of them grow retires the graph."""
import numpy as np
import pytest
import torch

import harmonyclient_b200 as hb
from harmonyclient_b200 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,n", [("plain", 64), ("bf16", 64), ("fp8", 64), ("plain", 3_000)])
@pytest.mark.parametrize("call", ["probes", "search_preassigned", "warmup_tops", "search", "failing"])
def test_a_call_that_grows_a_workspace_retires_the_graph(form, n, call):
    x, q = datasets.gmm_uint8(40_000, 10_000, d=96, ncomp=256, sigma=25.0, seed=5)
    idx = hb.Index(96, 128, 24)
    idx.train(x)
    idx.add(x)
    idx.set_form(form)
    k = 10
    dq = torch.from_numpy(q[:n]).cuda()
    dD = torch.empty((n, k), dtype=torch.float32, device="cuda")
    dI = torch.empty((n, k), dtype=torch.int64, device="cuda")

    def search():
        dD.fill_(0)
        dI.fill_(0)
        torch.cuda.synchronize()
        idx.search_device(n, dq.data_ptr(), k, dD.data_ptr(), dI.data_ptr(), 0)
        torch.cuda.synchronize()
        return idx.last_stats()["graph_replayed"], dD.cpu().numpy(), dI.cpu().numpy()

    idx.set_graph(True)
    _, D, I = search()
    r = search()
    assert r[0] == 1
    np.testing.assert_array_equal(r[2], I)
    pr = np.tile(np.arange(24, dtype=np.int64), (10_000, 1))
    if call == "probes":
        idx.probes(q)
    elif call == "search_preassigned":
        idx.search_preassigned(q, 100, pr)
    elif call == "warmup_tops":
        idx.warmup_tops(q, 10, pr, 10, 100)
    elif call == "search":
        idx.set_graph(False)  # (turning it off drops the graph as well)
        idx.search(q, 100)
        idx.set_graph(True)
    else:
        with pytest.raises(hb.HyError):
            idx.search_preassigned(q, 100, np.full((10_000, 24), 128, np.int64))
    r = search()
    assert r[0] == (1 if call == "failing" else 0)
    np.testing.assert_array_equal(r[1], D)
    np.testing.assert_array_equal(r[2], I)
    r = search()
    assert r[0] == 1
    np.testing.assert_array_equal(r[1], D)
    np.testing.assert_array_equal(r[2], I)
