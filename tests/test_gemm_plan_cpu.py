"""What a GEMM call hands to the tcgen05 kernel for one token tile (csrc/gemm_umma.cu) and what the
kernel's host side makes of it, without a GPU: the launch is recorded instead of made."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from easy_to_hard_b200.ops import _lib, gemm


class OnGpu:
    """A CPU tensor that says it is a CUDA one."""
    is_cuda = True

    def __init__(self, t):
        self._t = t

    def __getattr__(self, name):
        return getattr(self._t, name)


def _plan(p):
    """(k-blocks per stage, stages, loads weights early, staged epilogue) of a launch."""
    out = (C.c_int * 4)()
    rc = _lib.lib().e2h_gemm_umma_plan(C.byref(p), out)
    return rc if rc else tuple(out)


@pytest.fixture
def launches(monkeypatch):
    """The parameter blocks of the e2h_gemm_umma launches of a test."""
    seen = []

    def record(ref, stream):
        p = _lib.GemmParams()
        C.memmove(C.byref(p), ref, C.sizeof(p))
        seen.append(p)
        return 0
    _lib.lib()
    word = torch.zeros(1, dtype=torch.int32)
    fake = SimpleNamespace(e2h_gemm_umma=record)
    monkeypatch.setattr(gemm, "_lib", SimpleNamespace(
        lib=lambda: fake, stream=lambda: 0, check=_lib.check, status_word=lambda device: word))
    monkeypatch.setattr(gemm, "_expand_int8", lambda w, which: OnGpu(w._t.to(torch.bfloat16)))
    monkeypatch.setattr(gemm, "_expand_int4", lambda w, which: OnGpu(w.dequant()))
    return seen


# (whole int8 / int4 tiles of up to 128 tokens stream through a kernel of their own, gated products of
# more tokens through another)
CASES = [(bits, T, K, dual) for bits in (16, 8, 4) for T in (17, 64, 128, 200)
         for K in (688, 1024, 1376) for dual in (False, True)
         if not (bits != 16 and T <= 128 and K % 128 == 0) and not (dual and T > 128)]


@pytest.mark.parametrize("bits,T,K,dual", CASES)
def test_weights_expanded_by_the_call_are_not_loaded_early(launches, bits, T, K, dual):
    """The bf16 image of a quantised matrix is written by the launch before: loads ahead of the wait for
    that launch could read what the buffer held before."""
    F = 256
    x = OnGpu(torch.zeros(T, K, dtype=torch.bfloat16))

    def weight():
        if bits == 16:
            return OnGpu(torch.zeros(F, K, dtype=torch.bfloat16))
        if bits == 8:
            return OnGpu(torch.zeros(F, K, dtype=torch.int8))
        g = 16 if K == 688 else 32
        w = gemm.Int4Weight.from_int(torch.zeros(F, K, dtype=torch.int32), torch.zeros(K // g, F, 2), g)
        w.is_cuda = True
        return w
    out = OnGpu(torch.zeros(T, F, dtype=torch.bfloat16))
    scale = OnGpu(torch.zeros((1 + dual) * F)) if bits == 8 else None
    if dual:
        gemm.linear_swiglu(x, weight(), weight(), out=out, scale=scale)
    else:
        gemm.linear(x, weight(), out=out, scale=scale)
    assert len(launches) == 1
    assert _plan(launches[0])[2] == (bits == 16)


@pytest.mark.parametrize("which", [0, 1])
def test_the_image_of_a_matrix_is_not_overwritten_by_the_next(which):
    """A captured step keeps the address of its image, another stream may still read it."""
    small, large = (torch.randint(-128, 128, (n, 12), dtype=torch.int8) for n in (5, 40))
    images = [(w, gemm._expand_int8(w, which)) for w in (small, large, small + 1, small)]
    codes = torch.randint(0, 16, (6, 8), dtype=torch.int32)
    w4 = gemm.Int4Weight.from_int(codes, torch.rand(2, 6, 2), 4)
    images.append((w4.dequant(), gemm._expand_int4(w4, which)))
    for w, image in images:
        assert torch.equal(image, w.to(torch.bfloat16))
    assert len({image.untyped_storage().data_ptr() for _, image in images}) == len(images)


@pytest.mark.parametrize("tokens,top,half", [(1, 2, False), (2, 2, False), (4, 2, False), (16, 2, True),
                                             (1, 8, True), (32, 8, True)])
def test_ring_of_an_expert_product_follows_the_groups_with_rows(launches, tokens, top, half):
    """8 experts of 2 x 2752 x 2048: half the shared memory per CTA only where the CTAs that find rows
    outnumber the SMs; otherwise stages of several k-blocks."""
    T, E, F, K = tokens * top, 8, 2752, 2048
    x, out = (OnGpu(torch.zeros(T, n, dtype=torch.bfloat16)) for n in (K, F))
    w1, w3 = (OnGpu(torch.zeros(E * F, K, dtype=torch.bfloat16)) for _ in range(2))
    off = torch.zeros(E + 1, dtype=torch.int32)
    gemm.grouped_swiglu(x, w1, w3, out, off, E, tokens)
    kps, stages, early, _ = _plan(launches[0])
    assert not early and stages >= 2 and (kps == 1) == half


@pytest.mark.parametrize("T", [1, 8, 64, 70, 128])
@pytest.mark.parametrize("E,F,K", [(128, 128, 2048), (16, 1000, 4096), (300, 64, 512), (4, 11008, 1024)])
def test_expert_products_keep_two_blocks_in_flight(launches, E, F, K, T):
    """The exchange buffer of split sums counts against half a ring; many groups, few rows."""
    x, out = (OnGpu(torch.zeros(T, n, dtype=torch.bfloat16)) for n in (K, F))
    w1, w3 = (OnGpu(torch.zeros(E * F, K, dtype=torch.bfloat16)) for _ in range(2))
    off = torch.zeros(E + 1, dtype=torch.int32)
    gemm.grouped_swiglu(x, w1, w3, out, off, E, T)
    kps, stages, _, _ = _plan(launches[0])
    assert kps * stages >= 2


@pytest.mark.parametrize("T", [4, 16, 64, 200])
def test_int4_pairs_of_another_layout_go_through_the_general_expansion(launches, monkeypatch, T):
    """The kernels read (scale, zero) pairs as dense bf16: strided, fp32 or odd ones are dequantised."""
    F, K, g = 24, 256, 64
    codes = torch.randint(0, 16, (F, K), dtype=torch.int32)
    sz = torch.rand(K // g, F, 2).bfloat16()
    good = gemm.Int4Weight.from_int(codes, sz, g)
    apart = torch.zeros(K // g, F, 4).bfloat16()
    apart[..., ::2] = sz
    odd = torch.zeros(sz.numel() + 1).bfloat16()[1:].view(sz.shape)
    odd.copy_(sz)
    expanded = []

    def expand(w, which):
        expanded.append(w.dequant().bfloat16())
        return OnGpu(expanded[-1])
    monkeypatch.setattr(gemm, "_expand_int4", expand)
    x, out = (OnGpu(torch.zeros(T, n, dtype=torch.bfloat16)) for n in (K, F))
    assert good.plain()
    for pairs in (apart[..., ::2], sz.permute(1, 0, 2).contiguous().permute(1, 0, 2), odd, sz.float()):
        w = gemm.Int4Weight(good.q, pairs, g, (F, K))
        w.is_cuda = True
        assert not w.plain()
        del expanded[:], launches[:]
        if T > 16:          # (below, a bf16 image takes the kernel for few rows, which is not recorded)
            gemm.linear(x, w, out=out)
            assert len(launches) == 1 and len(expanded) == 1
        assert not gemm.rows_rule(w, None, x, gemm.EPI_STORE_BF16)


@pytest.mark.parametrize("T,tmax", [(0, 0), (0, 1), (0, 8), (4, 0)])
@pytest.mark.parametrize("gated", [False, True])
def test_grouped_products_without_rows_are_refused_by_the_launch(launches, T, tmax, gated):
    K, F, n = 256, 904, 4
    x, out = (OnGpu(torch.zeros(T, width, dtype=torch.bfloat16)) for width in (K, F))
    w = OnGpu(torch.zeros(n * F, K, dtype=torch.bfloat16))
    off = torch.zeros(n + 1, dtype=torch.int32)
    if gated:
        gemm.grouped_swiglu(x, w, w, out, off, n, tmax)
    else:
        gemm.grouped_linear(x, w, out, off, n, tmax)
    assert len(launches) == 1 and _plan(launches[0]) < 0
