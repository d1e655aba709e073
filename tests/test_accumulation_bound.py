"""The bound on the tensor cores' accumulation, against a model that cuts every
term and sum off at 24 bits (a worst case for f32 accumulators, whose rounding is
not documented) on the CPU, and against the hardware."""
import ctypes as C
import math

import numpy as np
import pytest

from harmonyclient_b200 import _lib

U = 2.0 ** -24


def _cut(v, top):
    """v with nothing below the 24th bit from `top`'s leading bit."""
    if top == 0.0:
        return 0.0
    ulp = math.ldexp(1.0, math.frexp(top)[1] - 24)
    return math.trunc(v / ulp) * ulp


def _accumulate(p, G):
    """Products p, G an instruction, as terms aligned to the largest and cut."""
    acc = 0.0
    for s in range(0, len(p), G):
        terms = [acc, *p[s:s + G]]
        top = max(abs(t) for t in terms)
        total = sum(_cut(t, top) for t in terms)
        acc = _cut(total, total)
    return acc


def _cases(K, rng):
    """Vectors of K values: one large product and others about the cut, of one
    sign or both, and random ones."""
    for eps in (1.375, 1.40625, 0.99, 1.0):
        for at in (0, K // 2, K - 1):
            for sign in (1, -1):
                a = np.full(K, eps * 2.0 ** -12)
                a[at] = 1.0
                b = a * sign
                b[at] = 1.0
                yield a, b
    for _ in range(20):
        yield rng.standard_normal(K), rng.standard_normal(K)


@pytest.mark.parametrize("G,K", [(8, 64), (8, 384), (16, 64), (16, 768), (32, 128), (32, 1536)])
def test_bound_holds_for_an_accumulator_that_cuts_off(G, K):
    bound = _lib.load().hy_selftest_accum_units(K, G)
    worst = 0.0
    for a, b in _cases(K, np.random.default_rng(K)):
        a, b = a.astype(np.float16).astype(np.float64), b.astype(np.float16).astype(np.float64)  # exact products
        err = abs(_accumulate(list(a * b), G) - math.fsum(a * b))
        worst = max(worst, err / (np.linalg.norm(a) * np.linalg.norm(b)) / U)
    assert worst <= bound
    assert worst > K + 8  # the bound of K rounded additions would not do


@pytest.mark.parametrize("d", [5, 33, 100])
def test_zeros_that_fill_a_block_add_exactly(d):
    """Eight blocks of d dimensions, each filled up to whole instructions."""
    G, w = 8, -(-d // 8) * 8
    bound = _lib.load().hy_selftest_accum_units(8 * d, G)
    for a, b in _cases(8 * d, np.random.default_rng(d)):
        a, b = a.astype(np.float16).astype(np.float64), b.astype(np.float16).astype(np.float64)
        p = np.zeros((8, w))
        p[:, :d] = (a * b).reshape(8, d)
        err = abs(_accumulate(list(p.reshape(-1)), G) - math.fsum(a * b))
        assert err <= bound * U * np.linalg.norm(a) * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("op,K,G", [("", 128, 16), ("_e4m3", 256, 32), ("_tf32", 64, 8)])
def test_bound_holds_on_the_tensor_cores(op, K, G):
    L = _lib.load()
    rng = np.random.default_rng(1)
    scale = 2.0 ** 6 if op == "_e4m3" else 1.0
    rows = []
    for a, b in _cases(K, rng):
        if op == "_e4m3":  # four significant bits, 2^-6 .. 448
            a, b = (np.sign(v) * np.clip(np.abs(v) * scale, 2.0 ** -6, 256) for v in (a, b))
            a, b = (np.ldexp(np.round(np.frexp(v)[0] * 16) / 16, np.frexp(v)[1]) for v in (a, b))
        else:  # eight, as in bf16
            a, b = (np.ldexp(np.round(np.frexp(v)[0] * 256) / 256, np.frexp(v)[1]) for v in (a, b))
        rows.append((a, b))
    A = np.zeros((128, K), np.float32)
    B = np.zeros((128, K), np.float32)
    for i, (a, b) in enumerate(rows):
        A[i], B[i] = a, b
    D = np.zeros((128, 128), np.float32)
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    _lib.check(getattr(L, "hy_selftest_tcgen05" + op)(p(A), p(B), p(D)))
    err = np.abs(D - A.astype(np.float64) @ B.astype(np.float64).T)
    norm = np.linalg.norm(A.astype(np.float64), axis=1)[:, None] * np.linalg.norm(B.astype(np.float64), axis=1)
    n = len(rows)
    assert (err[:n, :n] / norm[:n, :n]).max() / U <= L.hy_selftest_accum_units(K, G)
