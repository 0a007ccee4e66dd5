"""A unit that one rank holds alone hands out views of its own shard instead of copies."""
import pytest
import torch


@pytest.mark.parametrize("param,compute", [(torch.float32, torch.bfloat16), (torch.float32, torch.float32),
                                           (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("shapes", [[(3, 5)], [(4, 8), (7,), (1, 1)]])
def test_views(param, compute, shapes):
    from easy_to_hard_b200.parallel.fsdp import ShardUnit
    want = [torch.randn(s) for s in shapes]
    named = [(f"p{i}", torch.nn.Parameter(w.to(param))) for i, w in enumerate(want)]
    u = ShardUnit(named, None, param, compute, compute)
    buf = torch.full((u.padded,), 7.0, dtype=compute)
    u.gather_into(buf)
    for (_, p), w in zip(named, want):
        assert torch.equal(p.data, w.to(param).to(compute))
        assert p.data.untyped_storage().data_ptr() == u.shard_lp.untyped_storage().data_ptr()
    assert bool((buf == 7.0).all())
    u.shard_lp.mul_(2)                          # an optimizer step is seen without another gather
    for (_, p), w in zip(named, want):
        assert torch.equal(p.data, w.to(param).to(compute) * 2)
    u.release()
    assert all(p.numel() == 0 for _, p in named)
    u.gather_into(buf)
    assert torch.equal(named[0][1].data, want[0].to(param).to(compute) * 2)
