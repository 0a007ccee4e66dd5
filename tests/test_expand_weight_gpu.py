"""Expansion of int8 and int4 weights to bf16 (ops/csrc/expand_weight.cu): exact, element by element."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,K,pad", [(1, 8, 0), (130, 72, 8), (333, 4096, 0)])
def test_int8_expansion_is_exact(F, K, pad):
    from easy_to_hard_b200.ops import gemm
    w = torch.randint(-128, 128, (F, K + pad), device="cuda", dtype=torch.int8)[:, :K]
    assert torch.equal(gemm._expand_int8(w, 0), w.to(torch.bfloat16))


@pytest.mark.parametrize("F,K,g", [(1, 8, 8), (130, 96, 32), (333, 4096, 128), (64, 512, 512)])
def test_int4_expansion_is_exact(F, K, g):
    from easy_to_hard_b200.ops import gemm
    codes = torch.randint(0, 16, (F, K), device="cuda", dtype=torch.int32)
    sz = torch.randn(K // g, F, 2, device="cuda").bfloat16()
    w = gemm.Int4Weight.from_int(codes, sz, g)
    assert torch.equal(gemm._expand_int4(w, 1), w.dequant())
