"""Plain batches on a card with little free memory: a batch whose tensor-core
buffers do not fit runs on the scans that need none of them, with their
answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import harmonyclient_b200 as hb  # noqa: E402


@pytest.fixture()
def full_card():
    """take(left): allocate all but `left` bytes of the card's free memory
    (untouched, and given back after the test)."""
    held = []

    def take(left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        held.append(torch.empty(max(0, free - left), dtype=torch.uint8, device="cuda"))

    yield take
    held.clear()
    torch.cuda.empty_cache()


def test_a_batch_without_memory_for_its_buffers(full_card):
    nlist, d, nprobe, m, k = 4096, 64, 2, 8_000, 10
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    c = 10 * torch.randn((nlist, d), generator=g, device="cuda")
    x = c[torch.randint(0, nlist, (1_000_000,), generator=g, device="cuda")]
    x += torch.randn(x.shape, generator=g, device="cuda")
    q = (c[torch.randint(0, nlist, (m,), generator=g, device="cuda")] +
         torch.randn((m, d), generator=g, device="cuda")).cpu().numpy()
    idx = hb.Index(d, nlist, nprobe)
    idx.centroid_codes = c.cpu().numpy()
    x = x.cpu().numpy()
    idx.add(x)
    assert m * nprobe < 4 * nlist and m * nprobe * (len(x) / nlist) * d * 4 > 600e6  # few shared lists, much work
    idx.set_plain_scan("query")
    want = idx.search(q, k)
    idx.set_plain_scan("auto")
    full_card(420 << 20)  # the batch's candidate buffers take 500 MiB
    for _ in range(2):
        for a, b in zip(want, idx.search(q, k)):
            np.testing.assert_array_equal(a, b)
        assert idx.last_stats()["kernel_launches"] == 1  # one scan, not the tensor cores' two passes
    # a batch whose buffers fit runs there
    idx.nprobe = 6
    idx.set_plain_scan("query")
    want6 = idx.search(q[:2_700], k)
    idx.set_plain_scan("auto")
    for a, b in zip(want6, idx.search(q[:2_700], k)):
        np.testing.assert_array_equal(a, b)
    assert idx.last_stats()["kernel_launches"] == 2


def test_with_memory_for_nothing(full_card):
    """Not even for the rows' bound terms."""
    nlist, d, nprobe, m, k = 256, 32, 4, 250, 10
    rng = np.random.default_rng(5)
    c = (10 * rng.standard_normal((nlist, d))).astype(np.float32)
    x = (c[rng.integers(0, nlist, 2_000_000)] + rng.standard_normal((2_000_000, d))).astype(np.float32)
    q = x[:m] + np.float32(0.1)
    idx = hb.Index(d, nlist, nprobe)
    idx.centroid_codes = c
    idx.add(x)
    assert m * nprobe < 4 * nlist and m * nprobe * (len(x) / nlist) * d * 4 > 600e6
    idx.set_plain_scan("query")
    want = idx.search(q, k)
    idx.set_plain_scan("auto")
    full_card(8 << 20)
    for a, b in zip(want, idx.search(q, k)):
        np.testing.assert_array_equal(a, b)
    assert idx.last_stats()["kernel_launches"] == 1
