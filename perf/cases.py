"""The work this library is measured by: whole calls of its public entry points at listed
sizes, and random further cases of the same ranges.

A case is a dict of plain values:
    call    "gemkm" / "gekmm" (the torch front-end), "batched" (a handle's strided-batched
            GeMKM, every entry with factors of its own) or "forward" (a handle's MKM that
            keeps all intermediates, the call of a training step)
    dt      "f32" or "f64"
    M       rows of X (columns of X for gekmm), per batch entry
    ps, qs  rows and columns of the factors F1 .. FN, comma separated
    tx      X is handed over as the transposed view of a contiguous tensor
    tf      "none", "all" or "first": which factors are transposed views
    alpha, beta     beta != 0 adds beta * Y
    batch   entries of a strided batch (1 otherwise)
    dist    "uniform" on [-1, 1) or "normal": distribution of X and Y
"""
import math

import torch

import fastkron_b200
from fastkron_b200 import lib as fk

DTYPES = {"f32": torch.float32, "f64": torch.float64}


def _case(name, call, dt, M, ps, qs=None, tx=False, tf="none", alpha=1.0, beta=0.0, batch=1, dist="uniform"):
    c = {} if name is None else {"name": name}
    c.update(call=call, dt=dt, M=M, ps=",".join(map(str, ps)), qs=",".join(map(str, qs or ps)), tx=tx, tf=tf,
             alpha=alpha, beta=beta, batch=batch, dist=dist)
    return c


def listed():
    return [
        # a few small factors and a few right-hand sides: one step of an iterative solver on a
        # small grid, where the time of a call is its launches and the host's work
        _case("small", "gemkm", "f32", 10, [8] * 3),
        # one double-precision vector through a chain of factors that are no power of two: the
        # matrix-vector product inside conjugate gradients on a regular grid
        _case("matvec_odd_f64", "gemkm", "f64", 1, [10] * 5),
        # many small independent products with factors of their own (a batch of models)
        _case("batched", "batched", "f32", 16, [16] * 3, batch=64),
        # the benchmark's small-factor configuration
        _case("square16", "gemkm", "f32", 1024, [16] * 4),
        # the benchmark's double-precision configuration: few rows, many columns
        _case("square8_f64", "gemkm", "f64", 16, [8] * 8),
        # the benchmark's left-Kronecker configuration: X stored transposed, alpha and beta*Y
        _case("kmm32_transposed", "gekmm", "f32", 1024, [32] * 3, tx=True, alpha=2.0, beta=1.0, dist="normal"),
        # the benchmark's mixed large-factor configuration, the first factor a transposed view
        _case("mixed128", "gemkm", "f32", 2048, [128, 128, 16], tf="first"),
        # the benchmark's 64x64 configuration with a quarter of its rows: the largest case
        _case("square64", "gemkm", "f32", 64, [64] * 4),
        # large factors of an odd size (grids of 127 points per axis)
        _case("odd127", "gemkm", "f32", 4096, [127] * 2),
        # non-square factors of distinct ragged sizes in double precision (interpolation from
        # one grid to another), with an odd number of columns and beta*Y
        _case("ragged_kmm_f64", "gekmm", "f64", 17, [14, 19, 34, 21], [15, 13, 23, 34], alpha=2.0, beta=1.0),
        # a chain of small factors that are no power of two
        _case("square12", "gemkm", "f32", 1024, [12] * 4),
        # the forward pass of training: the result and every intermediate, which the backward
        # pass reads
        _case("forward32", "forward", "f32", 256, [32] * 3),
    ]


# Bounds of a drawn case: a quarter of the largest listed case's multiply-adds (double precision and
# ragged factors run at lower rates) and of the elements of its widest matrix.
_MAX_MACS = 64 * 64 ** 5
_MAX_ELEMS = 64 * 64 ** 4 // 4


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _widest(ps, qs):
    """Columns of the widest matrix and multiply-adds per row, factors applied last to first."""
    cols = wide = math.prod(ps)
    macs = 0
    for p, q in reversed(list(zip(ps, qs))):
        cols = cols // p * q
        macs += cols * p
        wide = max(wide, cols)
    return wide, macs


def draw(rng):
    """A further case: any of the entry points, equal power-of-two factors, equal factors of any
    size or distinct non-square ones, sizes spread over their logarithm, odd ones among them."""
    while True:
        call = rng.choice(["gemkm", "gemkm", "gemkm", "gekmm", "gekmm", "batched", "forward"])
        dt = rng.choice(["f32", "f32", "f64"])
        kind = rng.choice(["pow2", "pow2", "any", "ragged"])
        if kind == "pow2":
            p = rng.choice([2, 4, 8, 16, 32, 64, 128])
            n = rng.randint(2, 16 if p == 2 else 8 if p <= 8 else 4 if p <= 64 else 3)
            ps = qs = [p] * n
        elif kind == "any":
            p = _log_int(rng, 3, 130)
            n = rng.randint(2, 6 if p <= 10 else 4 if p <= 40 else 2)
            ps = qs = [p] * n
        else:
            n = rng.randint(2, 4)
            hi = 96 if n == 2 else 48 if n == 3 else 34
            ps = [_log_int(rng, 3, hi) for _ in range(n)]
            qs = [_log_int(rng, 3, hi) for _ in range(n)]
        wide, macs = _widest(ps, qs)
        batch = _log_int(rng, 2, 128) if call == "batched" else 1
        # small calls to the bounds of the largest listed one
        top = min(_MAX_ELEMS // wide, _MAX_MACS // macs) // batch
        if dt == "f64":
            top //= 2
        if top < 1:
            continue
        M = _log_int(rng, 1, min(top, 8192))
        plain = call in ("gemkm", "gekmm")
        scaled = plain and rng.random() < 0.4
        return _case(None, call, dt, M, ps, qs, tx=plain and rng.random() < 0.25,
                     tf=rng.choice(["none", "none", "all", "first"]) if plain else "none",
                     alpha=2.0 if scaled else 1.0, beta=1.0 if scaled else 0.0, batch=batch,
                     dist=rng.choice(["uniform", "normal"]))


def _sizes(case):
    ps = [int(v) for v in case["ps"].split(",")]
    qs = [int(v) for v in case["qs"].split(",")]
    return ps, qs, math.prod(ps), math.prod(qs)


def _inputs(case, seed):
    """X, the factors and Y (None without beta) as the call takes them."""
    ps, qs, K, L = _sizes(case)
    dt, M, batch = DTYPES[case["dt"]], case["M"], case["batch"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(*shape):
        return torch.rand(*shape, dtype=dt, device="cuda", generator=gen).mul_(2).sub_(1)

    def data(*shape):
        if case["dist"] == "normal":
            return torch.randn(*shape, dtype=dt, device="cuda", generator=gen)
        return uniform(*shape)

    if case["call"] in ("gemkm", "gekmm"):
        left = case["call"] == "gekmm"
        xshape, zshape = ((K, M), (L, M)) if left else ((M, K), (M, L))
        x = data(*xshape[::-1]).t() if case["tx"] else data(*xshape)
        fs = []
        for i, (p, q) in enumerate(zip(ps, qs)):
            r, c = (q, p) if left else (p, q)
            transposed = case["tf"] == "all" or (case["tf"] == "first" and i == 0)
            fs.append(uniform(c, r).t() if transposed else uniform(r, c))
        return x, fs, data(*zshape) if case["beta"] != 0 else None
    return data(batch, M, K), [uniform(batch, p, q) for p, q in zip(ps, qs)], None


def prepare(case, seed):
    ps, qs, K, L = _sizes(case)
    dt, M, batch = DTYPES[case["dt"]], case["M"], case["batch"]
    s = {"case": case, "ps": ps, "qs": qs}
    s["x"], s["fs"], s["y"] = _inputs(case, seed)
    if case["call"] in ("gemkm", "gekmm"):
        return s
    # what a program that calls a handle keeps: the handle, the result and the work buffers
    h = s["h"] = fastkron_b200.FastKron()
    s["z"] = torch.empty(batch, M, L, dtype=dt, device="cuda")
    if case["call"] == "batched":
        _, te = h.sizes(M, ps, qs)
        s["t"] = [torch.empty(batch * te, dtype=dt, device="cuda") for _ in range(2)]
    else:
        _, sizes = h.sizes_forward(M, ps, qs)
        s["inter"] = [torch.empty(n, dtype=dt, device="cuda") for n in sizes]
    return s


def run(s):
    c = s["case"]
    if c["call"] == "gemkm":
        return fastkron_b200.gemkm(s["x"], s["fs"], c["alpha"], c["beta"], s["y"])
    if c["call"] == "gekmm":
        return fastkron_b200.gekmm(s["fs"], s["x"], c["alpha"], c["beta"], s["y"])
    ps, qs, h, dch = s["ps"], s["qs"], s["h"], "s" if c["dt"] == "f32" else "d"
    fptrs = [f.data_ptr() for f in s["fs"]]
    if c["call"] == "batched":
        M, K, L = c["M"], s["x"].shape[2], s["z"].shape[2]
        h.raw_gemm_strided_batched("mkm", dch, M, ps, qs, s["x"].data_ptr(), fk.OP_N, M * K, fptrs, fk.OP_N,
                                   [p * q for p, q in zip(ps, qs)], s["z"].data_ptr(), M * L, c["alpha"], c["beta"],
                                   c["batch"], 0, 0, s["t"][0].data_ptr(), s["t"][1].data_ptr())
        return s["z"]
    h.raw_forward("mkm", dch, c["M"], ps, qs, s["x"].data_ptr(), fk.OP_N, fptrs, fk.OP_N, s["z"].data_ptr(),
                  [t.data_ptr() for t in s["inter"]])
    return [s["z"]] + s["inter"]


def work(case):
    """X, Y and the factors read once, the result (and the intermediates of a forward call)
    written once; the multiply-adds of the factor-by-factor product."""
    ps, qs, K, L = _sizes(case)
    es = 4 if case["dt"] == "f32" else 8
    _, macs = _widest(ps, qs)
    M = case["M"]
    elems = M * K + M * L * (2 if case["beta"] != 0 else 1) + sum(p * q for p, q in zip(ps, qs))
    if case["call"] == "forward":
        cols = K
        for p, q in reversed(list(zip(ps[1:], qs[1:]))):
            cols = cols // p * q
            elems += M * cols
    return {"bytes": case["batch"] * elems * es, "flops": case["batch"] * 2 * M * macs}


def exact(case, seed):
    """What run returns, in 64-bit arithmetic: the factors from the last to the first, each contracting the
    fastest index and putting its own in front of the others (after all of them the order is the original)."""
    x, fs, y = _inputs(case, seed)
    left = case["call"] == "gekmm"
    if left:
        x, fs = x.t(), [f.t() for f in fs]
    t = x.double()
    if t.dim() == 2:
        t, fs = t[None], [f[None] if f.dim() == 2 else f for f in fs]
    batch, M = t.shape[:2]
    steps = []
    for f in reversed(fs):
        p = f.shape[1]
        t = torch.matmul(t.reshape(batch, -1, p), f.double())                     # [batch][M * S][Q]
        t = t.reshape(batch, M, -1, f.shape[2]).transpose(2, 3).reshape(batch, M, -1)
        if case["call"] == "forward":
            steps.append(t)
    if case["call"] == "forward":
        return [steps[-1]] + [u.reshape(-1) for u in steps[-2::-1]]
    if case["call"] == "batched":
        return t
    z = t[0].t() if left else t[0]
    z = case["alpha"] * z
    return z if y is None else z + case["beta"] * y.double()


def tolerance(case):
    """Four times what the calls were seen to differ from the same product in 64-bit arithmetic with
    the factors applied in the other order: at most 3.5e-7 (largest difference 5.1e-6) in single
    precision and 9.3e-16 (5.1e-15) in double, over the listed and sixty drawn cases."""
    return {"rel": 1.5e-6, "max": 2e-5} if case["dt"] == "f32" else {"rel": 4e-15, "max": 2e-14}
