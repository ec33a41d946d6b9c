"""Precision of the split tensor-core pass (csrc/kernel_gemm_split.cu): its error is no larger than the FMA kernels' and has no
sign of its own, on data of either sign, and each of its eight sweeps is needed for that.

The CPU tests run the same checks on a model of its arithmetic: pieces of 6, 8 and the remaining bits, addends cut off
toward zero 2 bits below the unit of the accumulator, sums cut off at 24 bits, 32 products of h*h per accumulator."""
import ctypes
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

SWEEPS = [(1, 2), (2, 1), (2, 0), (0, 2), (1, 1), (1, 0), (0, 1)]      # pieces of x and of f; (0, 0) apart


def pieces(v):
    def nearest(a, bits):
        m, e = np.frexp(a)
        return np.ldexp(np.rint(m * 2.0 ** bits), e - bits)
    v = v.astype(np.float64)
    h = nearest(v, 6)
    m = nearest(v - h, 8)
    return h, m, v - h - m


def mma(d, a, b):
    """d + a @ b for one step of 16 products in the tensor cores' accumulator."""
    pr = a[:, :, None] * b[None]
    _, e = np.frexp(np.maximum(np.abs(pr).max(1), np.abs(d)))
    u = np.ldexp(1.0, e - 26)
    s = (np.trunc(d / u) + np.trunc(pr / u[:, None, :]).sum(1)) * u
    m, e = np.frexp(s)
    return np.ldexp(np.trunc(m * 2.0 ** 24), e - 24)


def model(x, f, without=None):
    x = np.pad(x, ((0, 0), (0, -x.shape[1] % 16)))
    f = np.pad(f, ((0, -f.shape[0] % 16), (0, 0)))
    A, B = pieces(x), pieces(f)
    small, total = np.zeros((x.shape[0], f.shape[1])), None
    for k in range(0, x.shape[1], 32):
        d = np.zeros_like(small)
        for i in range(k, min(k + 32, x.shape[1]), 16):
            for p, q in SWEEPS:
                if (p, q) != without:
                    small = mma(small, A[p][:, i:i + 16], B[q][i:i + 16])
            if without != (0, 0):
                d = mma(d, A[0][:, i:i + 16], B[0][i:i + 16])
        total = d.astype(np.float32) if total is None else total + d.astype(np.float32)
    return total + small.astype(np.float32)


def single_products():
    """One nonzero per factor column, and operands whose second and third pieces are as large as they get: 1 + a/32 + m + l
    with m in (0.9, 1) * 2^-6 and l in (0.9, 1) * 2^-15 (24 bits, exact in fp32)."""
    rng = np.random.default_rng(11)

    def draw(n):
        return (1 + rng.integers(0, 6, n) / 32 + rng.integers(231, 255, n) * 2.0 ** -14 + rng.integers(231, 256, n) * 2.0 ** -23).astype(np.float32)
    M, P, Q = 1024, 64, 48
    x = draw(M * P).reshape(M, P) * rng.choice([-1, 1], (M, P)).astype(np.float32)
    f = np.zeros((P, Q), np.float32)
    f[rng.permutation(P)[:Q], np.arange(Q)] = draw(Q)
    return x, f


def single_products_hold(z, x, f):
    """h*h of one product is exact.  The small terms, below 2^-4.4 of it, lose at most 1.25 units in their last place per sweep
    (7 * 1.25 * 2^-28 of the product), l*l is below 2^-29 of it, and the final sum rounds once: 2^-24 * (1 + 0.55 + 0.03) at most."""
    want = x.astype(np.float64) @ f.astype(np.float64)
    return np.all(np.abs(z - want) <= 1.75 * 2.0 ** -24 * np.abs(want))


def test_model_needs_every_sweep():
    x, f = single_products()
    assert single_products_hold(model(x, f), x, f)
    for s in SWEEPS + [(0, 0)]:
        assert not single_products_hold(model(x, f, without=s), x, f), s


@pytest.mark.gpu
def test_every_sweep_is_there():
    import torch
    import fastkron_b200
    from fastkron_b200 import lib as fk
    L = fk.get()
    L.fkbGemmSplitLaunches.restype = ctypes.c_ulonglong
    x, f = single_products()
    n0 = L.fkbGemmSplitLaunches()
    for xd in (torch.from_numpy(x).cuda(), torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()):
        assert single_products_hold(fastkron_b200.gemkm(xd, [torch.from_numpy(f).cuda()]).cpu().numpy(), x, f)
    assert L.fkbGemmSplitLaunches() == n0 + 2


def data(kind, rng, shape):
    if kind == "uniform":
        return rng.uniform(-1, 1, shape)
    if kind == "normal":
        return rng.standard_normal(shape)
    if kind == "positive":
        return rng.uniform(0, 1, shape)
    if kind == "exponential":
        return rng.exponential(size=shape)
    if kind == "lognormal":
        return np.exp(rng.standard_normal(shape))
    d = np.abs(np.arange(shape[0])[:, None] - np.arange(shape[1])[None]).astype(np.float64)
    if kind == "exp-kernel":
        return np.exp(-d / 3)
    if kind == "gauss-kernel":
        return np.exp(-(d / 20) ** 2)
    if kind == "matern-kernel":
        return (1 + 3 ** 0.5 * d / 8) * np.exp(-3 ** 0.5 * d / 8)
    assert kind == "interpolation"
    f, w, c = np.zeros(shape), rng.uniform(0, 1, shape[1]), np.arange(shape[1])
    r = c * (shape[0] - 1) // shape[1]
    f[r, c], f[r + 1, c] = w, 1 - w
    return f


KINDS = ["uniform", "normal", "positive", "exponential", "lognormal", "exp-kernel", "gauss-kernel", "matern-kernel", "interpolation"]


def error_and_mean(z, want):
    d = z - want
    return np.linalg.norm(d) / np.linalg.norm(want), d.mean() / np.sqrt((want ** 2).mean())


def operands(kind, P, n, M):
    rng = np.random.default_rng(P + n)
    matrix = kind.endswith("kernel") or kind == "interpolation"
    x = data("positive" if matrix else kind, rng, (M, P ** n)).astype(np.float32)
    return x, [data(kind, rng, (P, P)).astype(np.float32) for _ in range(n)]


@pytest.mark.parametrize("kind", KINDS)
def test_model_error_is_no_larger_than_the_fma_chain_s(kind):
    x, (f,) = operands(kind, 64, 1, 96)
    want = x.astype(np.float64) @ f.astype(np.float64)
    chain = np.zeros(want.shape, np.float32)
    for p in range(x.shape[1]):
        chain = (chain.astype(np.float64) + x[:, p:p + 1].astype(np.float64) * f[p:p + 1].astype(np.float64)).astype(np.float32)
    err, mean = error_and_mean(model(x, f), want)
    assert err <= error_and_mean(chain, want)[0]
    # one rounding of the result is all that may have a direction
    assert abs(mean) <= 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("P,n,M", [(36, 3, 12), (48, 2, 64), (64, 3, 4), (80, 2, 40), (96, 2, 30), (112, 2, 24), (127, 2, 20), (128, 3, 1)])
def test_error_is_no_larger_than_the_fma_kernels(kind, P, n, M):
    """Relative 2-norm against 64 bits no larger than the FMA kernels' (the same where a factor holds numbers that a split
    does not: the FMA chain runs then), and a mean deviation below one rounding per factor, or theirs."""
    import torch
    import fastkron_b200
    from fastkron_b200 import lib as fk
    L = fk.get()
    L.fkbGemmSplitLaunches.restype = ctypes.c_ulonglong
    x, fs = operands(kind, P, n, M)
    want = x.astype(np.float64)
    for f in reversed(fs):
        want = (want.reshape(-1, P) @ f.astype(np.float64)).reshape(M, -1, P).swapaxes(1, 2).reshape(M, -1)
    xd, fd = torch.from_numpy(x).cuda(), [torch.from_numpy(f).cuda() for f in fs]
    n0 = L.fkbGemmSplitLaunches()
    z = fastkron_b200.gemkm(xd, fd).cpu().numpy().astype(np.float64)
    assert L.fkbGemmSplitLaunches() == n0 + n
    try:
        L.fkbSetSplitOff(1)
        w = fastkron_b200.gemkm(xd, fd).cpu().numpy().astype(np.float64)
    finally:
        L.fkbSetSplitOff(0)
    (err, mean), (err_fma, mean_fma) = error_and_mean(z, want), error_and_mean(w, want)
    assert err <= err_fma
    assert abs(mean) <= max(n * 2.0 ** -25, abs(mean_fma))
