"""The work that a user of this engine has it do, as cases that can be timed
and checked: searches from one query to a full batch in every form (plain
FP32, bf16, e4m3, learned probes, per-query nprobe, inner product), through
host and device pointers, and the construction of an index.

Data are seeded synthetic mixtures of the shapes and value ranges that
``harmonyclient_b200.datasets`` describes, drawn on the GPU.  Centroids come
from a few Lloyd steps written here (``_centroids``), so that ``exact`` can
give the same index's answer in 64 bits without the engine.
"""
import ctypes as C
import math

import numpy as np
import torch

import harmonyclient_b200 as hb
from harmonyclient_b200 import _lib
from harmonyclient_b200.index import METRIC_IP, METRIC_L2, OPT_NONE, OPT_TRIANGLE

FLT_MAX = float(np.finfo(np.float32).max)


def _case(**kw):
    """A search case with its defaults filled in."""
    c = dict(job="search", api="device", form="plain", metric="l2", data="u8", base=1_000_000, d=128, nlist=1024,
             nprobe=64, k=10, nq=10_000, graph=False, warm=False, triangle=False, learned=False, mixed=False)
    c.update(kw)
    return c


def listed():
    return [
        # One interactive query on a million vectors: latency.
        _case(name="one_query", api="host", nq=1),
        # The small configuration of the smoke test and the tests: 10,000
        # vectors, 100 queries, the reference's calling sequence.
        _case(name="small_100q", api="host", data="gmm", base=10_000, nlist=100, nprobe=10, nq=100),
        # A ragged batch too small to share lists: odd d, odd list count, odd k.
        _case(name="ragged_33q", data="dense", base=200_003, d=97, nlist=300, nprobe=20, k=17, nq=33),
        # A server's request of 64 queries against the million vectors, in the
        # mode harmony_serve runs (host pointers, graph replay).
        _case(name="serve_64q", api="host", form="bf16", nprobe=16, nq=64, graph=True),
        # The exact FP32 batch search of the main workload, with the
        # reference's default warm-up.
        _case(name="plain_batch", k=100, warm=True),
        # Inner product on unit vectors with the reference's triangle window.
        _case(name="plain_ip_tri", metric="ip", data="unit", base=300_000, d=200, nlist=512, nprobe=32, k=20, nq=2000,
              triangle=True),
        # The main workload on the tensor cores, fixed nprobe, graph replay.
        _case(name="bf16_batch", form="bf16", k=100, warm=True, graph=True),
        # The main workload as a host call with learned probes: the headline
        # configuration end to end.
        _case(name="learned_host", api="host", form="bf16", k=100, warm=True, graph=True, learned=True),
        # Wide dense vectors in the e4m3 form.
        _case(name="fp8_420", form="fp8", data="dense", d=420, nlist=2048),
        # A stream with its own nprobe per query over skewed lists, more lists
        # than one coarse launch takes.
        _case(name="mixed_nprobe", form="bf16", data="zipf", base=2_000_000, nlist=4096, nprobe=128, nq=16_384,
              mixed=True),
        # Sparse wide vectors, many probes: the largest search.
        _case(name="bf16_500", form="bf16", data="sparse", base=500_000, d=500, nlist=2048, nprobe=256, nq=20_000),
        # Building an index (train and add) and asking it a first batch.
        _case(name="build", job="build", nq=1000, k=100),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if rng.random() < 0.15:
        base = log(10_000, 800_000)
        return _case(job="build", base=base, d=log(24, 160), nlist=min(1024, log(32, max(33, base // 64))), nprobe=log(4, 32),
                     nq=log(10, 1000), k=log(1, 100), data=rng.choice(["u8", "gmm", "dense"]))
    form = rng.choice(["plain", "plain", "bf16", "bf16", "fp8"])
    data = rng.choice(["u8", "gmm", "dense", "unit", "sparse", "zipf"])
    metric = "ip" if data == "unit" and rng.random() < 0.7 else "l2"
    d = log(24, 500)
    base = log(10_000, min(1_000_000, 200_000_000 // d))
    nlist = log(32, min(4096, max(64, base // 100)))
    nprobe = log(1, min(128, nlist))
    nq = log(1, 16_000)
    # Under the largest listed case's work: rows scanned x dimensions.
    nq = max(1, min(nq, int(3e11 / (nprobe / nlist * base * d))))
    api = rng.choice(["host", "device", "device"])
    return _case(api=api, form=form, metric=metric, data=data, base=base, d=d, nlist=nlist, nprobe=nprobe,
                 k=log(1, 200), nq=nq, graph=rng.random() < 0.4, warm=rng.random() < 0.5,
                 triangle=metric == "ip" and rng.random() < 0.5, mixed=api == "device" and rng.random() < 0.2)


# ---------------------------------------------------------------------------
# Inputs


def _vectors(g, kind, n, mix):
    """n rows of the mixture `mix` on the GPU, float32."""
    comp = (torch.multinomial(mix["w"], n, replacement=True, generator=g) if mix["w"] is not None else
            torch.randint(0, mix["ncomp"], (n,), generator=g, device="cuda"))
    d = mix["d"]
    out = torch.empty((n, d), device="cuda")
    for s in range(0, n, 1 << 18):
        c = comp[s:s + (1 << 18)]
        m = c.shape[0]
        if kind == "sparse":
            v = torch.empty((m, mix["support"].shape[1]), device="cuda").exponential_(1.0, generator=g)
            rows = torch.zeros((m, d), device="cuda").scatter_(1, mix["support"][c], v)
        else:
            rows = mix["centre"][c] + mix["sigma"] * torch.randn((m, d), generator=g, device="cuda")
        if kind in ("u8", "zipf"):
            rows = rows.round_().clamp_(0, 255)
        elif kind == "gmm":
            rows = rows.clamp_(min=0)
        elif kind in ("unit", "sparse"):
            rows = rows / rows.norm(dim=1, keepdim=True).clamp_min(1e-30)
        out[s:s + m] = rows
    return out


def _inputs(case, seed):
    """Base rows, queries and per-query nprobes (all on the GPU)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + 17)
    kind, n, d = case["data"], case["base"], case["d"]
    ncomp = max(16, min(4096, n // 244)) if kind != "gmm" else 100
    mix = dict(d=d, ncomp=ncomp, w=None)
    if kind == "sparse":
        nnz = max(1, round(0.1 * d))
        mix["support"] = torch.rand((ncomp, d), generator=g, device="cuda").argsort(1)[:, :nnz].contiguous()
    else:
        lo, hi, sigma = {"u8": (0, 255, 20.0), "zipf": (0, 255, 20.0), "gmm": (0, 100, 8.0), "dense": (-1, 1, 0.3),
                         "unit": (-1, 1, 0.3)}[kind]
        mix["centre"] = lo + (hi - lo) * torch.rand((ncomp, d), generator=g, device="cuda")
        mix["sigma"] = sigma
    if kind == "zipf":
        w = 1.0 / torch.arange(1, ncomp + 1, device="cuda", dtype=torch.float64) ** 1.1
        mix["w"] = (w / w.sum()).float()
    x = _vectors(g, kind, n, mix)
    q = _vectors(g, kind, case["nq"], mix)
    npq = torch.randint(min(8, case["nprobe"]), case["nprobe"] + 1, (case["nq"],), generator=g, device="cuda").int()
    return x, q, npq, (g, mix)


def _centroids(case, x):
    """Centroids by a few Lloyd steps on the first rows (which are drawn at
    random): FP32 matrix products, the same on every run."""
    nlist = case["nlist"]
    s = x[:max(nlist, min(x.shape[0], 64 * nlist, 131_072))]
    c = s[:nlist].clone()
    for _ in range(12):
        lab = torch.empty(s.shape[0], dtype=torch.int64, device="cuda")
        for b in range(0, s.shape[0], 1 << 15):
            p = s[b:b + (1 << 15)]
            lab[b:b + (1 << 15)] = ((c * c).sum(1)[None] - 2 * (p @ c.T)).argmin(1)
        sums, cnt = torch.zeros_like(c), torch.zeros(nlist, device="cuda")
        for b in range(0, s.shape[0], 1 << 15):
            one = torch.nn.functional.one_hot(lab[b:b + (1 << 15)], nlist).float()
            sums += one.T @ s[b:b + (1 << 15)]
            cnt += one.sum(0)
        c = torch.where(cnt[:, None] > 0, sums / cnt.clamp_min(1)[:, None], c)
    if case["metric"] == "ip":
        c = c / c.norm(dim=1, keepdim=True).clamp_min(1e-30)
    return c


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    x, q, npq, (g, mix) = _inputs(case, seed)
    idx = hb.Index(case["d"], case["nlist"], case["nprobe"], METRIC_IP if case["metric"] == "ip" else METRIC_L2,
                   OPT_TRIANGLE if case["triangle"] else OPT_NONE)
    st = dict(case=case, idx=idx, q=q, npq=npq)
    if case["api"] == "device":
        st["D"] = torch.empty((case["nq"], case["k"]), device="cuda")
        st["I"] = torch.empty((case["nq"], case["k"]), dtype=torch.int64, device="cuda")
    else:
        st["qh"] = q.cpu().numpy()
    if case["job"] == "build":
        st["x"] = x
        return st
    L = _lib.load()
    idx.centroid_codes = _centroids(case, x).cpu().numpy()
    _lib.check(L.hy_index_add_device(idx._h, x.shape[0], C.c_void_p(x.data_ptr()), C.c_void_p(_stream())))
    if case["warm"]:
        idx.preSearch(warmUpSearchList=10, warmUpSearchListSize=100)
    idx.set_form(case["form"])
    if case["learned"]:
        tq = _vectors(g, case["data"], 4096, mix).cpu().numpy()
        idx.train_probe_model(tq, max_nprobe=case["nprobe"], k_label=10, epochs=5, coverage=0.97)
        idx.set_learned(True)
    if case["graph"]:
        idx.set_graph(True)
    return st


def run(st):
    case, idx = st["case"], st["idx"]
    if case["job"] == "build":
        L, x, s = _lib.load(), st["x"], _stream()
        _lib.check(L.hy_index_train_device(idx._h, x.shape[0], C.c_void_p(x.data_ptr()), 0, C.c_void_p(s)))
        _lib.check(L.hy_index_add_device(idx._h, x.shape[0], C.c_void_p(x.data_ptr()), C.c_void_p(s)))
        idx.search_device(case["nq"], st["q"].data_ptr(), case["k"], st["D"].data_ptr(), st["I"].data_ptr(), s)
        return idx.centroid_codes, st["D"], st["I"]
    if case["api"] == "host":
        return idx.search(st["qh"], case["k"])
    if case["mixed"]:
        idx.search_nprobes_device(case["nq"], st["q"].data_ptr(), case["k"], st["npq"].data_ptr(), case["nprobe"],
                                  st["D"].data_ptr(), st["I"].data_ptr(), _stream())
    else:
        idx.search_device(case["nq"], st["q"].data_ptr(), case["k"], st["D"].data_ptr(), st["I"].data_ptr(), _stream())
    return st["D"], st["I"]


def work(case):
    """Each input read once and each output written once, in the form's own
    element size for the rows a search reads; two operations per (vector,
    vector, dimension) that the search or the assignment compares."""
    n, d, nq, nlist, k = case["base"], case["d"], case["nq"], case["nlist"], case["k"]
    nprobe = case["nprobe"] * (0.53 if case["mixed"] else 0.05 if case["learned"] else 1.0)
    elem = {"plain": 4, "bf16": 2, "fp8": 1}[case["form"]]
    pairs = nq * nprobe / nlist * n  # (query, row) comparisons
    rows = n * (1.0 - (1.0 - min(1.0, nprobe / nlist)) ** nq)  # rows some query reads
    b = rows * d * elem + nlist * d * 4 + nq * d * 4 + nq * k * 12
    f = 2.0 * d * (pairs + nq * nlist)
    if case["job"] == "build":
        b += 2.0 * n * d * 4 + n * 12
        f += 2.0 * d * nlist * (n + 20.0 * min(n, 256 * nlist))
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """The search's answer in 64 bits: distances of the k best rows among the
    probed lists.  Ids are whole numbers and have no value here; a built
    index (k-means steps) and a trained probe model have none either."""
    if case["job"] == "build" or case["learned"]:
        return None
    x, q, npq, _ = _inputs(case, seed)
    c = _centroids(case, x).double()
    ip = case["metric"] == "ip"

    def score(a, b, bn):  # smaller is better
        return -(a @ b.T) if ip else (a * a).sum(1)[:, None] + bn[None] - 2 * (a @ b.T)

    cn = (c * c).sum(1)
    lab = torch.empty(x.shape[0], dtype=torch.int64, device="cuda")
    for s in range(0, x.shape[0], 1 << 15):
        lab[s:s + (1 << 15)] = score(x[s:s + (1 << 15)].double(), c, cn).argmin(1)
    xd = x.double()
    del x
    xn = (xd * xd).sum(1)
    nprobe, k = min(case["nprobe"], case["nlist"]), case["k"]
    out = torch.empty((case["nq"], k), dtype=torch.float64, device="cuda")
    step = max(1, min(512, (1 << 29) // xd.shape[0]))
    for s in range(0, case["nq"], step):
        a = q[s:s + step].double()
        near = score(a, c, cn).topk(nprobe, largest=False).indices
        use = torch.arange(nprobe, device="cuda")[None] < (npq[s:s + step, None] if case["mixed"] else nprobe)
        use = use.expand(near.shape)
        mask = torch.zeros((a.shape[0], case["nlist"]), dtype=torch.bool, device="cuda").scatter_(1, near, use)
        dist = score(a, xd, xn).masked_fill_(~mask[:, lab], math.inf)
        top = dist.topk(min(k, xd.shape[0]), largest=False).values
        out[s:s + step] = math.inf
        out[s:s + step, :top.shape[1]] = top
    out = torch.where(torch.isinf(out), torch.full_like(out, FLT_MAX), out)
    return (-out if ip else out.clamp_min(0)), None
