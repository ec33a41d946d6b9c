"""The launches a plan is regrouped into (csrc/plan.cpp, fuseLaunches), executed pass by pass with numpy from
their printed strides and buffers: the same product as the definition, for every orientation, operand order and
buffer rule, and never a matrix wider than the result in the result used as scratch."""
import ctypes
import re

import numpy as np
import pytest

from fastkron_b200 import lib as fk

LINE = re.compile(r"pass\d+ (\w+) f\[(\d+)\.\.(\d+)\] .* M=(\d+) A=(\d+) B=(\d+) x\((-?\d+),(-?\d+),(-?\d+),(-?\d+)\) "
                  r"z\((-?\d+),(-?\d+),(-?\d+),(-?\d+)\) .* (\w+)->(\w+)( epi)?$")


@pytest.fixture(scope="module")
def L():
    return fk.get()


def launches(L, mm, dt, M, ps, qs, opx="N", t2=1, align=16, name="fkbDescribeLaunches", fusion=1, forward=0):
    buf = ctypes.create_string_buffer(1 << 15)
    n = getattr(L, name)(ctypes.c_int(mm == "kmm"), ctypes.c_int(dt == "f64"), ctypes.c_uint32(M), ctypes.c_uint32(len(ps)),
                         fk.u32arr(ps), fk.u32arr(qs), fk.OP_N if opx == "N" else fk.OP_T, fk.OP_N, forward, t2, fusion,
                         align, buf, ctypes.c_size_t(len(buf)))
    assert n > 0, n
    lines = buf.value.decode().strip().split("\n")
    assert len(lines) == n
    return lines


def execute(lines, x, fs, M, ps, qs):
    """x: flat input as stored.  Returns the flat buffer Z."""
    bufs = {"X": x}
    L_ = int(np.prod(qs))
    for ln in lines:
        m = LINE.match(ln)
        assert m, ln
        f0, f1 = int(m.group(2)), int(m.group(3))
        pM, pA, pB = (int(m.group(i)) for i in (4, 5, 6))
        xsM, xsA, xsG, xsB, zsM, zsA, zsG, zsB = (int(m.group(i)) for i in range(7, 15))
        src, dst = m.group(15), m.group(16)
        assert src != dst and dst != "X"
        G, H = int(np.prod(ps[f0:f1 + 1])), int(np.prod(qs[f0:f1 + 1]))
        pos = lambda sM, sA, sG, sB, n: (np.arange(pM)[:, None, None, None] * sM + np.arange(pA)[:, None, None] * sA +
                                         np.arange(n)[:, None] * sG + np.arange(pB) * sB)
        t = bufs[src][pos(xsM, xsA, xsG, xsB, G)]
        F = np.ones((1, 1))
        for i in range(f0, f1 + 1):
            F = np.kron(F, fs[i])
        out = np.einsum("magb,gh->mahb", t, F)
        idx = pos(zsM, zsA, zsG, zsB, H)
        assert len(np.unique(idx)) == idx.size
        z = np.full(idx.max() + 1, np.nan)
        z[idx] = out
        assert not np.isnan(z).any()
        if dst == "Z":
            assert z.size <= M * L_, "scratch in Z wider than the result"
        bufs = {"X": x, src: bufs[src], dst: z}
    return bufs["Z"]


SHAPES = [
    ([12] * 4, [12] * 4), ([10] * 3, [10] * 3), ([3, 5, 7], [4, 2, 6]), ([2] * 7, [2] * 7), ([6, 1, 5], [1, 9, 3]),
    ([14, 19, 4], [15, 3, 23]), ([3, 5, 8, 8], [3, 5, 8, 8]), ([40, 3, 3], [40, 3, 3]), ([9, 30, 2], [2, 3, 2]),
    ([33, 9], [9, 33]), ([20, 20], [7, 6]), ([5, 6, 4, 4, 3], [5, 6, 4, 4, 3]),
]


@pytest.mark.parametrize("ps,qs", SHAPES, ids=lambda v: "x".join(map(str, v)))
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_launches_compute_the_product(L, dt, ps, qs):
    rng = np.random.default_rng(3)
    K = int(np.prod(ps))
    fs = [rng.uniform(-1, 1, (p, q)) for p, q in zip(ps, qs)]
    big = np.ones((1, 1))
    fewer = 0
    for f in fs:
        big = np.kron(big, f)
    for mm in ("mkm", "kmm"):
        for opx in ("N", "T"):
            for M in (1, 2, 5):
                for t2 in (0, 1):
                    for align in (16, 4):
                        x = rng.uniform(-1, 1, (M, K))
                        want = x @ big
                        row = (mm == "mkm") == (opx == "N")            # X stored [M][K]
                        if mm == "kmm" and M == 1:
                            row = True
                        stored = (x if row else x.T).ravel()
                        lines = launches(L, mm, dt, M, ps, qs, opx, t2, align)
                        fewer += len(lines) < len(launches(L, mm, dt, M, ps, qs, opx, t2, align, "fkbDescribePlan"))
                        z = execute(lines, stored, fs, M, ps, qs)
                        z = z.reshape(M, -1) if mm == "mkm" or M == 1 else z.reshape(-1, M).T
                        assert np.allclose(z, want, rtol=1e-10, atol=1e-10 * np.abs(want).max()), (mm, opx, M, t2, align, lines)
    assert fewer > 0 or max(ps + qs) > 32, "nothing was regrouped"


def test_regrouping_honours_options(L):
    # no fusion and the forward variants: one launch per factor, the plan's own
    for kw in ({"fusion": 0}, {"forward": 1}):
        a = launches(L, "mkm", "f32", 8, [12] * 3, [12] * 3, **kw)
        b = launches(L, "mkm", "f32", 8, [12] * 3, [12] * 3, name="fkbDescribePlan", **kw)
        assert a == b and len(a) == 3


def test_chain_tiles_get_the_ctas_per_sm_they_were_sized_for(tmp_path):
    """Every group that chainShape accepts: the launcher's grid has the CTAs per SM that the tile was sized for (three
    up to kChainSmem3, else two), and they fit."""
    import os
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = tmp_path / "t.cpp"
    src.write_text(r'''
#include "chain_table.h"
#include <stdio.h>
using namespace fkb;
int main() {
  unsigned groups = 0, bad = 0;
  for (int d = 0; d < 2; d++)
    for (uint32_t p0 = 1; p0 <= 32; p0++) for (uint32_t q0 = 1; q0 <= 32; q0 += 3)
      for (uint32_t p1 = 2; p1 <= 32; p1 += 1) for (uint32_t q1 = 2; q1 <= 32; q1 += 5)
        for (uint32_t p2 = 1; p2 <= 16; p2 += 7) {
          const uint32_t P[3] = {p0, p1, p2}, Q[3] = {q0, q1, p2};
          ChainShape s;
          if (!chainShape(d ? DType::F64 : DType::F32, p2 > 1 ? 3 : 2, P, Q, (p0 & 1) != 0, 1 << 20, 148, &s)) continue;
          groups++;
          const unsigned n = chainCtasPerSm(s.smem);
          if (s.smem > kChainSmemMax || n < (s.smem <= kChainSmem3 ? 3u : 2u) || n * (s.smem + 1024) > 228 * 1024) bad++;
        }
  printf("%u %u\n", groups, bad);
}
''')
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(root, "include"), "-I", os.path.join(root, "fastkron_b200", "csrc"), str(src), "-o", exe])
    groups, bad = map(int, subprocess.check_output([exe]).split())
    assert groups > 10000 and bad == 0, (groups, bad)


def test_a_chain_group_has_one_admission_rule():
    """A group of several factors has no kernel to fall back to, so the launcher may decline nothing that the planner forms:
    besides chainShape, which both ask, only calls that never have groups (batches, redistribution over GPUs)."""
    import os
    src = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastkron_b200", "csrc", "kernel_chain.cu")).read()
    guards = re.findall(r"if \(([^;{}]*?)\)\s*return fastKronKernelNotFound;", src, re.S)
    assert len(guards) == 1, guards
    terms = {re.sub(r"\s+", " ", t).strip() for t in guards[0].split("||")} - {"ps.zsG == 1, total, cx.smCount, &s)"}
    assert {t for t in terms if not t.startswith("!chainShape(")} == {"cx.batch > 1", "cx.scatter.parts > 0", "cx.pSplit != 0"}, terms
