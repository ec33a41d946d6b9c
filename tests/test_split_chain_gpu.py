"""The split tensor-core pass (csrc/kernel_gemm_split.cu) and the chain launches (csrc/kernel_chain.cu) at the
sizes where they can go wrong: partial tiles, remainders of 16 and 32, both orientations, operands that are not
16-byte aligned, beta*Y (also in place of the result), batches, streams, values that a bf16 split cannot hold.

Bound.  One step of P products in precision u errs by at most (P + 2) u of the sum of the products' magnitudes
(one rounding per product for an FMA chain; for the split pass 2.5 u for each 16 products of h*h, a 32nd of that for each of the
seven small terms, one rounding per accumulator and 2^-30 for l*l: test_split_precision.py has the tight checks).  Over the steps the bounds add up, and
alpha and beta*Y add two roundings: |error| <= u * (sum (P_i + 4) + 4) * (|alpha| |X| |F| + |beta| |Y|)."""
import ctypes
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from fastkron_b200 import lib as fk
    L = fk.get()
    L.fkbGemmSplitLaunches.restype = ctypes.c_ulonglong
    L.fkbLaunchCount.restype = ctypes.c_ulonglong
    yield L
    assert L.fkbGemmSplitTimeouts() == 0


@pytest.fixture(autouse=True)
def split_on(lib):
    yield
    lib.fkbSetSplitOff(0)           # process-wide: also after a test that failed while it was set


def product(x, fs):
    t = x
    for f in reversed(fs):
        p, q = f.shape
        t = t.reshape(t.shape[0], -1, p) @ f
        t = t.swapaxes(1, 2).reshape(t.shape[0], -1)
    return t


def check(z, x, fs, alpha, beta, y, u):
    want = alpha * product(x, fs)
    mag = abs(alpha) * product(np.abs(x), [np.abs(f) for f in fs])
    if beta:
        want = want + beta * y
        mag = mag + abs(beta) * np.abs(y)
    bound = u * (sum(f.shape[0] + 4 for f in fs) + 4) * mag
    assert np.all(np.abs(z - want) <= bound), np.max(np.abs(z - want) / np.maximum(bound, 1e-300))


def call(mm, dt, M, ps, qs, tx, tf, beta, shift, seed=0):
    """Runs the front-end on operands `shift` elements off their allocation; returns z and the operands as
    float64 MKM matrices."""
    import torch
    import fastkron_b200
    rng = np.random.default_rng(seed)
    tdt = torch.float32 if dt == "f32" else torch.float64

    def dev(a):
        buf = torch.empty(a.size + shift, dtype=tdt, device="cuda")
        v = buf[shift:].view(*a.shape)
        v.copy_(torch.from_numpy(np.ascontiguousarray(a)))
        return v

    ndt = np.float32 if dt == "f32" else np.float64
    K, L = int(np.prod(ps)), int(np.prod(qs))
    x = rng.uniform(-1, 1, (M, K)).astype(ndt)
    fs = [rng.uniform(-1, 1, (p, q)).astype(ndt) for p, q in zip(ps, qs)]
    y = rng.uniform(-1, 1, (M, L)).astype(ndt)
    xm, fm, ym = (x, fs, y) if mm == "mkm" else (x.T, [f.T for f in fs], y.T)
    xd = dev(xm.T).t() if tx else dev(xm)
    fd = [dev(f.T).t() if tf else dev(f) for f in fm]
    yd = dev(ym) if beta else None
    if mm == "mkm":
        z = fastkron_b200.gemkm(xd, fd, 2.0 if beta else 1.0, beta, yd)
    else:
        z = fastkron_b200.gekmm(fd, xd, 2.0 if beta else 1.0, beta, yd)
    z = z.cpu().numpy().astype(np.float64)
    d = lambda a: a.astype(np.float64)
    return (z if mm == "mkm" else z.T), d(x), [d(f) for f in fs], d(y)


SPLIT = [
    # M, ps, qs
    (128, [33, 17], [32, 61]), (40, [64, 64], [64, 64]), (9, [127, 128], [128, 127]), (33, [128, 40], [96, 128]),
    (17, [65, 80], [113, 49]), (24, [48, 112], [112, 48]), (1, [64, 33, 34], [33, 64, 36]), (300, [128, 128], [128, 128]),
]


@pytest.mark.parametrize("mm,tx,tf,beta,shift", [("mkm", 0, 0, 0.0, 0), ("mkm", 1, 1, 1.0, 0), ("kmm", 0, 0, -0.5, 0),
                                                 ("kmm", 1, 0, 0.0, 0), ("mkm", 0, 1, 1.0, 1), ("kmm", 0, 0, 0.0, 3)])
@pytest.mark.parametrize("M,ps,qs", SPLIT, ids=lambda v: str(v).replace(" ", ""))
def test_split_pass(lib, M, ps, qs, mm, tx, tf, beta, shift):
    n0 = lib.fkbGemmSplitLaunches()
    z, x, fs, y = call(mm, "f32", M, ps, qs, tx, tf, beta, shift)
    assert lib.fkbGemmSplitLaunches() > n0, "the split kernel did not run"
    check(z, x, fs, 2.0 if beta else 1.0, beta, y, 2.0 ** -24)


def test_split_forward_layout(lib):
    """The forward variants' rotating layout: contraction index contiguous in, position index contiguous out."""
    import torch
    import fastkron_b200
    h = fastkron_b200.FastKron()
    M, ps, qs = 37, [33, 64], [40, 127]
    x = torch.rand(M, 33 * 64, device="cuda") - 0.5
    fs = [torch.rand(p, q, device="cuda") - 0.5 for p, q in zip(ps, qs)]
    ye, ie = h.sizes_forward(M, ps, qs)
    z, inter = torch.empty(ye, device="cuda"), [torch.empty(n, device="cuda") for n in ie]
    n0 = lib.fkbGemmSplitLaunches()
    h.raw_forward("mkm", "s", M, ps, qs, x.data_ptr(), 1, [f.data_ptr() for f in fs], 1, z.data_ptr(), [t.data_ptr() for t in inter])
    assert lib.fkbGemmSplitLaunches() == n0 + 2
    xn, fn = x.cpu().numpy().astype(np.float64), [f.cpu().numpy().astype(np.float64) for f in fs]
    check(z.view(M, -1).cpu().numpy(), xn, fn, 1.0, 0.0, None, 2.0 ** -24)
    t = xn.reshape(M, 33, 64) @ fn[1]
    t = t.swapaxes(1, 2).reshape(M, -1)
    err = np.abs(inter[0].view(M, -1).cpu().numpy() - t)
    mag = (np.abs(xn).reshape(M, 33, 64) @ np.abs(fn[1])).swapaxes(1, 2).reshape(M, -1)
    assert np.all(err <= 2.0 ** -24 * 72 * mag)
    h.close()


@pytest.mark.parametrize("where", ["x", "f"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38, -1.8e38, 1e-38, 1e-42, 2e-28, 0.0])
def test_split_pass_on_values_a_bf16_split_cannot_hold(lib, where, value):
    """Same result as the FMA kernels where those give inf or NaN; rows and factor columns of tiny magnitude keep
    their relative precision."""
    import torch
    import fastkron_b200
    torch.manual_seed(1)
    M, P, Q = 2000, 64, 50
    x, f = torch.rand(M, P, device="cuda") - 0.5, torch.rand(P, Q, device="cuda") - 0.5
    if where == "x":
        if 0 < abs(value) < 1:
            x[77] *= value                       # a whole row
            x[1999] = 0
        else:
            x[77, 5] = value
            x[1999, 63] = value
    elif 0 < abs(value) < 1:
        f[:, 7] *= value
    else:
        f[9, 7] = value
    n0 = lib.fkbGemmSplitLaunches()
    z = fastkron_b200.gemkm(x, [f]).cpu().numpy().astype(np.float64)
    assert lib.fkbGemmSplitLaunches() == n0 + 1
    lib.fkbSetSplitOff(1)
    w = fastkron_b200.gemkm(x, [f]).cpu().numpy().astype(np.float64)
    lib.fkbSetSplitOff(0)
    assert np.array_equal(np.isnan(z), np.isnan(w))
    assert np.array_equal(np.isinf(z), np.isinf(w)) and np.array_equal(z[np.isinf(z)], w[np.isinf(w)])
    xn, fn = x.cpu().numpy().astype(np.float64), f.cpu().numpy().astype(np.float64)
    ok = np.isfinite(w)
    with np.errstate(invalid="ignore", over="ignore"):
        want, mag = xn @ fn, np.abs(xn) @ np.abs(fn)
    # 2^-149: the spacing of denormal results, once per product
    assert np.all((np.abs(z - want) <= 2.0 ** -24 * (P + 8) * mag + P * 2.0 ** -149)[ok])


@pytest.mark.parametrize("xs,fs", [(1e38, 1e10), (1e30, 1e9), (1e20, 1e20), (3e37, 1.0), (1e-25, 1e-10), (1e-20, 1e-20), (1e15, 1e-26)])
def test_split_pass_at_the_ends_of_the_range(lib, xs, fs):
    """Products that overflow give the infinities of the FMA chain and no NaN; small ones keep their precision."""
    import torch
    import fastkron_b200
    torch.manual_seed(2)
    M, P, Q = 1500, 64, 48
    x, f = (torch.rand(M, P, device="cuda") + 0.5), (torch.rand(P, Q, device="cuda") + 0.5) * fs
    x[1::7] *= xs
    n0 = lib.fkbGemmSplitLaunches()
    z = fastkron_b200.gemkm(x, [f]).cpu().numpy().astype(np.float64)
    assert lib.fkbGemmSplitLaunches() == n0 + 1
    lib.fkbSetSplitOff(1)
    w = fastkron_b200.gemkm(x, [f]).cpu().numpy().astype(np.float64)
    lib.fkbSetSplitOff(0)
    assert not np.isnan(z).any() and np.array_equal(np.isinf(z), np.isinf(w))
    xn, fn = x.cpu().numpy().astype(np.float64), f.cpu().numpy().astype(np.float64)
    ok = np.isfinite(w)
    err = np.abs(np.where(ok, z, 0) - np.where(ok, xn @ fn, 0))
    assert np.all(err <= 2.0 ** -24 * (P + 8) * (xn @ fn) + P * 2.0 ** -149)


@pytest.mark.parametrize("small_in", ["x", "f"])
def test_split_pass_keeps_small_elements_beside_large_ones(lib, small_in):
    """Every output depends on one element of each operand (one nonzero per factor column), elements of one row or column
    lie up to 2^149 apart, and the large partner brings the product back into the range: no output may lose bits
    because its own element is small beside others of the same row or column.  One product: the bound of check()."""
    import torch
    import fastkron_b200
    rng = np.random.default_rng(7)
    M, P, Q = 1100, 64, 48
    x = (rng.uniform(1, 2, (M, P)) * 10.0 ** rng.uniform(-45, 0, (M, P))).astype(np.float32)
    f = np.zeros((P, Q), np.float32)
    f[rng.permutation(P)[:Q], np.arange(Q)] = (rng.uniform(1, 2, Q) * 2.0 ** rng.integers(60, 110, Q)).astype(np.float32)
    x[:, 0] = 1.0                                       # an ordinary element in every row
    x[::2, 1:] = rng.uniform(-1, 1, (M // 2, P - 1))    # and rows that a split holds, beside the others in a tile
    x[5, 1], f[1, 3] = 1.23456e-38, 1e33
    x[7, 2], f[2, 4] = 2.0 ** -135, 2.0 ** 100
    if small_in == "f":                                 # the mirror case: the same product with the roles exchanged
        x, f = np.ascontiguousarray(np.resize(f.T, (M, P))), np.ascontiguousarray(x[:Q].T)
    n0 = lib.fkbGemmSplitLaunches()
    z = fastkron_b200.gemkm(torch.from_numpy(x).cuda(), [torch.from_numpy(f).cuda()]).cpu().numpy().astype(np.float64)
    assert lib.fkbGemmSplitLaunches() == n0 + 1
    xn, fn = x.astype(np.float64), f.astype(np.float64)
    err, mag = np.abs(z - xn @ fn), np.abs(xn) @ np.abs(fn)
    assert np.all(err <= 2.0 ** -24 * (P + 8) * mag + P * 2.0 ** -149), np.max(err / np.maximum(mag, 1e-300))


@pytest.mark.parametrize("where", ["factor", "every row", "some rows", "one row"])
@pytest.mark.parametrize("mm,tx,tf,beta,M,P,Q", [("mkm", 0, 0, 1.0, 40000, 64, 48), ("kmm", 0, 1, 0.0, 30001, 33, 70), ("kmm", 1, 0, 0.5, 20000, 127, 128),
                                                 ("mkm", 1, 0, 0.0, 25000, 128, 127)])
def test_split_pass_contracts_what_it_cannot_split_like_the_fma_kernels(lib, where, mm, tx, tf, beta, M, P, Q):
    """Rows with elements that a split does not hold, and every row when the factor has one, are the FMA chain's to the
    last bit, in several tiles per CTA, with partial tiles, both layouts, and beta*Y in place of the result (Y is Z)."""
    import torch
    import fastkron_b200
    g = torch.Generator(device="cuda").manual_seed(5)
    x, f = torch.rand(M, P, device="cuda", generator=g) - 0.5, torch.rand(P, Q, device="cuda", generator=g) - 0.5
    rows = {"factor": slice(None), "every row": slice(None), "some rows": slice(3, None, 331), "one row": slice(M - 1, M)}[where]
    if where == "factor":
        f[P - 1, Q - 1] = 1.2345e-39
    else:
        x[rows, P // 2] = 1.2345e-39
        x[rows, P - 1] *= 1e-36
    y = torch.rand(M, Q, device="cuda", generator=g)
    xm, fm, ym = (x, f, y) if mm == "mkm" else (x.t(), f.t(), y.t())
    xd = xm.t().contiguous().t() if tx else xm.contiguous()
    fd = fm.t().contiguous().t() if tf else fm.contiguous()
    h = fastkron_b200.FastKron()
    opx, opf = (2 if tx else 1), (2 if tf else 1)
    t = [torch.empty(M * max(P, Q), device="cuda") for _ in range(2)]

    def run():
        z = ym.contiguous().clone()
        h.raw_gemm(mm, "s", M, [P], [Q], xd.data_ptr(), opx, [fd.data_ptr()], opf, z.data_ptr(), 2.0, beta, z.data_ptr() if beta else 0,
                   t[0].data_ptr(), t[1].data_ptr())
        return z if mm == "mkm" else z.t()
    n0 = lib.fkbGemmSplitLaunches()
    z = run()
    assert lib.fkbGemmSplitLaunches() == n0 + 1
    lib.fkbSetSplitOff(1)
    w = run()
    lib.fkbSetSplitOff(0)
    h.close()
    assert torch.equal(z[rows], w[rows])
    d = lambda v: v.cpu().numpy().astype(np.float64)
    check(d(z), d(x), [d(f)], 2.0, beta, d(y), 2.0 ** -24)


@pytest.mark.parametrize("option", [8, 16], ids=["TF32", "TF32x3"])
@pytest.mark.parametrize("P,split", [(127, True), (36, True), (128, None), (64, False)])
def test_tf32_options_send_what_they_do_not_take_to_the_split_kernel(lib, option, P, split):
    """A handle with a TF32 option runs the passes that its TF32 kernel declines where a handle without it does."""
    import torch
    import fastkron_b200
    split = option == 16 if split is None else split         # 128x128: TF32 takes it, TF32x3 does not
    h = fastkron_b200.FastKron()
    h.set_options(2 | option)
    M = 4096
    x, f = torch.rand(M, P, device="cuda") - 0.5, torch.rand(P, P, device="cuda") - 0.5
    z, t = torch.empty(M, P, device="cuda"), [torch.empty(M * P, device="cuda") for _ in range(2)]
    n0 = lib.fkbGemmSplitLaunches()
    h.raw_gemm("mkm", "s", M, [P], [P], x.data_ptr(), 1, [f.data_ptr()], 1, z.data_ptr(), 1.0, 0.0, 0, t[0].data_ptr(), t[1].data_ptr())
    assert lib.fkbGemmSplitLaunches() - n0 == int(split)
    if split:
        d = lambda v: v.cpu().numpy().astype(np.float64)
        check(d(z), d(x), [d(f)], 1.0, 0.0, None, 2.0 ** -24)
    h.close()


@pytest.mark.parametrize("P,Q,M,runs", [(64, 64, 1023, 0), (64, 64, 1024, 1), (54, 19, 2000, 0), (52, 20, 2000, 1), (16, 64, 2000, 0), (17, 61, 2000, 1),
                                        (31, 33, 2000, 0), (41, 25, 2000, 1), (128, 128, 1100, 1), (129, 40, 1100, 0), (40, 129, 1100, 0)])
def test_split_rule_at_its_edges(lib, P, Q, M, runs):
    """Both sides of every bound of gemmSplitEligible: the kernel that the rule names, the same product."""
    n0 = lib.fkbGemmSplitLaunches()
    z, x, fs, y = call("mkm", "f32", M, [P], [Q], 0, 0, 0.0, 0)
    assert lib.fkbGemmSplitLaunches() - n0 == runs
    check(z, x, fs, 1.0, 0.0, y, 2.0 ** -24)


@pytest.mark.parametrize("P", [64, 128])
def test_split_pass_in_a_strided_batch(lib, P):
    """Batches whose entries run one after the other on the split kernel, with factors and Y of their own."""
    import torch
    import fastkron_b200
    h = fastkron_b200.FastKron()
    batch, M = 3, 1040
    x, f = torch.rand(batch, M, P, device="cuda") - 0.5, torch.rand(batch, P, P, device="cuda") - 0.5
    z = torch.rand(batch, M, P, device="cuda")
    y = z.clone()
    t = [torch.empty(batch * M * P, device="cuda") for _ in range(2)]
    n0 = lib.fkbGemmSplitLaunches()
    h.raw_gemm_strided_batched("mkm", "s", M, [P], [P], x.data_ptr(), 1, M * P, [f.data_ptr()], 1, [P * P], z.data_ptr(), M * P, 2.0, 1.0, batch,
                               z.data_ptr(), M * P, t[0].data_ptr(), t[1].data_ptr())
    assert lib.fkbGemmSplitLaunches() == n0 + batch
    d = lambda v: v.cpu().numpy().astype(np.float64)
    for b in range(batch):
        check(d(z[b]), d(x[b]), [d(f[b])], 2.0, 1.0, d(y[b]), 2.0 ** -24)
    h.close()


def test_split_passes_on_two_streams(lib):
    """Two handles on two streams at once: every CTA takes all of an SM's tensor memory, so the launches take turns on an
    SM, and the results are those of one after the other."""
    import torch
    import fastkron_b200
    M, P = 6000, 96
    handles, args = [], []
    for i in range(2):
        handles.append(fastkron_b200.FastKron(torch.cuda.Stream()))
        x, f = torch.rand(M, P, device="cuda") - 0.5, torch.rand(P, P, device="cuda") - 0.5
        args.append((x, f, torch.empty(M, P, device="cuda"), torch.empty(M * P, device="cuda"), torch.empty(M * P, device="cuda")))

    def go(i):
        x, f, z, t1, t2 = args[i]
        handles[i].raw_gemm("mkm", "s", M, [P], [P], x.data_ptr(), 1, [f.data_ptr()], 1, z.data_ptr(), 1.0, 0.0, 0, t1.data_ptr(), t2.data_ptr())
    torch.cuda.synchronize()
    for i in range(2):
        go(i)
        torch.cuda.synchronize()
    want = [a[2].clone() for a in args]
    for a in args:
        a[2].zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for i in range(2):
            go(i)
    torch.cuda.synchronize()
    for i in range(2):
        assert torch.equal(args[i][2], want[i])
        handles[i].close()


@pytest.mark.parametrize("mm", ["mkm", "kmm"])
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("M,ps,qs", [(40, [12] * 4, [12] * 4), (17, [14, 9], [15, 13]), (5, [10] * 3, [10] * 3)], ids=lambda v: str(v).replace(" ", ""))
def test_chain_epilogue_in_place(lib, M, ps, qs, dt, mm):
    """beta*Y with Y in the place of the result."""
    import torch
    import fastkron_b200
    tdt = torch.float32 if dt == "f32" else torch.float64
    K, L = int(np.prod(ps)), int(np.prod(qs))
    x, fs = torch.rand(M, K, device="cuda", dtype=tdt) - 0.5, [torch.rand(p, q, device="cuda", dtype=tdt) - 0.5 for p, q in zip(ps, qs)]
    y = torch.rand(M, L, device="cuda", dtype=tdt)
    xd, fd, z = (x, fs, y.clone()) if mm == "mkm" else (x.t().contiguous(), [f.t().contiguous() for f in fs], y.t().contiguous())
    h = fastkron_b200.FastKron()
    _, te = h.sizes(M, ps, qs)
    t = [torch.empty(te, device="cuda", dtype=tdt) for _ in range(2)]
    n0 = lib.fkbLaunchCount()
    h.raw_gemm(mm, "s" if dt == "f32" else "d", M, ps, qs, xd.data_ptr(), 1, [f.data_ptr() for f in fd], 1, z.data_ptr(), 2.0, -0.5, z.data_ptr(),
               t[0].data_ptr(), t[1].data_ptr())
    assert lib.fkbLaunchCount() - n0 < len(ps)
    d = lambda v: v.cpu().numpy().astype(np.float64)
    check(d(z if mm == "mkm" else z.t()), d(x), [d(f) for f in fs], 2.0, -0.5, d(y), 2.0 ** -24 if dt == "f32" else 2.0 ** -53)
    h.close()


CHAIN = [
    (1, [10] * 5, [10] * 5), (5, [12] * 4, [12] * 4), (300, [5] * 4, [5] * 4), (3, [14, 19, 34, 21], [15, 13, 23, 34]),
    (1, [2] * 9, [2] * 9), (64, [3, 7], [9, 2]), (7, [32, 9, 5], [11, 31, 6]), (2, [1, 6, 1, 5], [3, 1, 2, 4]),
    (1000, [11, 13], [13, 11]), (4, [3, 5, 16, 16], [3, 5, 16, 16]),
]


@pytest.mark.parametrize("mm,tx,tf,beta,shift", [("mkm", 0, 0, 0.0, 0), ("mkm", 1, 1, 1.0, 0), ("kmm", 0, 0, -0.5, 0),
                                                 ("kmm", 1, 0, 0.0, 0), ("mkm", 0, 1, 1.0, 1)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("M,ps,qs", CHAIN, ids=lambda v: str(v).replace(" ", ""))
def test_chain_launches(lib, M, ps, qs, dt, mm, tx, tf, beta, shift):
    n0 = lib.fkbLaunchCount()
    z, x, fs, y = call(mm, dt, M, ps, qs, tx, tf, beta, shift)
    assert lib.fkbLaunchCount() - n0 < len(ps), "no two factors shared a launch"
    check(z, x, fs, 2.0 if beta else 1.0, beta, y, 2.0 ** -24 if dt == "f32" else 2.0 ** -53)
