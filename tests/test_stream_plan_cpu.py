"""Tile heights of the skinny GEMM (ops.gemm.stream_plan): what the kernel takes, for every width."""
import pytest

from easy_to_hard_b200.ops import gemm


@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("splitk", [1, 2, 4, 8])
def test_plans_fit_the_kernel_and_the_sms(splitk, dual):
    for F in range(8, 60000, 8):
        plan = gemm.stream_plan(F, splitk, dual)
        if plan is None:
            continue
        th, split = plan
        assert 64 <= th < 128 and th % 8 == 0 and split in (1, 2)
        assert not (dual and split > 1)
        ctas = -(-F // th) * split
        assert ctas <= 2 * gemm.N_SM
        # never fewer CTAs than with 128-row tiles
        assert ctas >= -(-F // 128) * (splitk if splitk == 2 else 1)
        # a stage of two k-blocks always leaves two stages
        assert gemm._smem_bytes(128, th, dual, split, 2, 2) <= 227 * 1024
