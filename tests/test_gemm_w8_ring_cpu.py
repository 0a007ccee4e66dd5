"""The ring of the int8 / int4 products (csrc/gemm_w8.cu), without a GPU: two groups of converters that take
turns must not convert a stage before its load has landed, whatever the order in which loads land."""
import ctypes as C
from functools import lru_cache

import pytest
import torch

from easy_to_hard_b200.ops import _lib, gemm

BUFFER_FIRST, STAGE_FIRST = (0, 1), (1, 0)      # order of a converter's two waits


@lru_cache(None)
def _reads_early(S: int, buffers: int, groups: int, order=BUFFER_FIRST) -> bool:
    """Walks every order in which loads land, groups convert and products finish, for S stages. A wait for
    phase k of a barrier passes when the last phase that completed has k's parity."""
    n = S + buffers + 3
    start = (0, 0, 0, tuple((g, 0) for g in range(groups)))   # landed, products done, converted, (trip, wait)
    seen, todo = {start}, [start]
    passes = lambda completed, k: (completed - 1) % 2 == k % 2
    while todo:
        landed, done, conv, at = todo.pop()
        after = []
        for i in range(min(n, done + S)):                     # a load is issued once its stage is free
            if not landed >> i & 1:
                after.append((landed | 1 << i, done, conv, at))
        if done < n and conv >> done & 1 and landed >> done & 1:
            after.append((landed, done + 1, conv, at))
        for g, (it, wait) in enumerate(at):
            if it >= n:
                continue
            if wait < 2:
                if order[wait] == 0:
                    ok = passes(len(range(it % buffers, done, buffers)), it // buffers - 1)
                else:
                    ok = passes(sum(landed >> i & 1 for i in range(it % S, n, S)), it // S)
                if not ok:
                    continue
                to, c = (it, wait + 1), conv
            elif not landed >> it & 1:
                return True
            else:
                to, c = (it + groups, 0), conv | 1 << it
            after.append((landed, done, c, at[:g] + (to,) + at[g + 1:]))
        for state in after:
            if state not in seen:
                seen.add(state)
                todo.append(state)
    assert any(s[1] == n for s in seen)                       # the walk comes to its end
    return False


def _plan(F, K, T, bits, dual, stages=0, th=None, splitk=None):
    """(tile height, stages, groups, buffers) of a product as ops/gemm.py asks for it."""
    bn = 64 if T <= 64 or dual else 128
    p = _lib.GemmParams()
    bn, split, _, _, _ = gemm.pick_tiles(F, T, K, dual, splitk, bn)
    p.F, p.T, p.K, p.bn, p.splitk, p.dual, p.stages = F, T, K, bn, split, int(dual), stages
    if th is None and split == 1:
        th = gemm.quant_height(F, bits)
    p.th = th or 0
    p.lda, p.ldb, p.lda2 = K * bits // 8, K, K * bits // 8
    p.a = p.a2 = p.b = p.scale = p.qsz = p.qsz2 = 4096
    p.groupsize = 128
    out = (C.c_int * 5)()
    rc = _lib.lib().e2h_gemm_w8_plan(C.byref(p), bits, out)
    assert rc == 0, rc
    return tuple(out)[:4]


# (features, K) of the layers of the configured models and of their shards
LAYERS = sorted({(F // tp, K) for F, K in [
    (4096, 4096), (12288, 4096), (4096, 11008), (11008, 4096), (32016, 4096), (5120, 5120), (15360, 5120),
    (13824, 5120), (5120, 13824), (10240, 8192), (8192, 8192), (22016, 8192), (8192, 22016), (6144, 2048),
    (1376, 1152), (768, 256)] for tp in (1, 2, 4, 8) if F // tp >= 64})


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("dual", [False, True])
def test_planned_rings(bits, dual):
    rings = {_plan(F, K, T, bits, dual)[1:] for F, K in LAYERS for T in (17, 64, 65, 128)}
    rings |= {_plan(F, K, T, bits, dual, stages=s)[1:] for F, K in LAYERS[::5] for T in (17, 128)
              for s in range(1, 9)}
    assert {g for _, g, _ in rings} == {1, 2}
    assert any(g == 2 and s % 2 for s, g, _ in rings)         # odd rings are among them
    for s, g, b in rings:
        assert g == 1 or s % 2 == 0 or s >= b
        assert not _reads_early(s, b, g), (s, g, b)


@pytest.mark.parametrize("S,buffers", [(5, 4), (3, 3)])
def test_stage_before_buffer_reads_early(S, buffers):
    """The order of the waits matters: rings that the products use, with the stage waited for first."""
    assert _reads_early(S, buffers, 2, STAGE_FIRST)
    assert not _reads_early(S, buffers, 2, BUFFER_FIRST)


@pytest.mark.parametrize("S,buffers", [(1, 3), (1, 4), (3, 4)])
def test_rings_of_one_group(S, buffers):
    assert S == 1 or _reads_early(S, buffers, 2)
    assert not _reads_early(S, buffers, 1)
    assert _plan(2048, 4096, 64, 8, buffers == 3, stages=S)[1:] == (S, 1, buffers)


def test_kernel_waits_for_the_buffer_first():
    """The model's order is that of the source."""
    from easy_to_hard_b200.ops.build import CSRC
    src = (CSRC / "gemm_w8.cu").read_text()
    waits = src[src.index("ph_cur = ph;"):src.index("const uint8_t* st = tiles")]
    assert -1 < waits.index("conv_empty[c]") < waits.index("full[s_cur]")


@pytest.mark.parametrize("F,K,T,bits,dual,want", [
    (12288, 4096, 128, 8, False, (88, 5, 2, 4)), (15360, 5120, 128, 8, False, (104, 5, 2, 4)),
    (10240, 8192, 128, 8, False, (72, 5, 2, 4)), (12288, 4096, 128, 4, False, (96, 5, 2, 4)),
    (2752, 4096, 64, 8, True, (128, 3, 2, 3)), (2752, 8192, 64, 8, True, (128, 3, 2, 3))])
def test_odd_rings(F, K, T, bits, dual, want):
    assert _plan(F, K, T, bits, dual) == want
