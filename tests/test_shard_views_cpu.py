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


@pytest.mark.parametrize("keep_params", [False, True])
@pytest.mark.parametrize("root", [False, True])
def test_one_rank_holds_no_gather_buffers(keep_params, root):
    """The parameters of a single rank take no memory beside the shards, and loading a state or a new
    low-precision shard is seen by the next use."""
    from mp_workers import tiny_model
    from easy_to_hard_b200.parallel.fsdp import ShardedDataParallel
    model = tiny_model()
    if root:                                    # a trainable tensor outside the blocks
        model.register_parameter("extra", torch.nn.Parameter(torch.ones(24)))
    sdp = ShardedDataParallel(model, process_group=None, keep_params=keep_params)
    assert (sdp.root is not None) == root
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes()
            for owner in (sdp, *sdp._all_units()) for v in vars(owner).values()
            for t in (v if isinstance(v, list) else [v]) if isinstance(t, torch.Tensor)}
    held.pop(sdp._grad_buf.untyped_storage().data_ptr())
    own = {u.shard_lp.untyped_storage().data_ptr() for u in sdp._all_units()}
    own |= {u.shard.untyped_storage().data_ptr() for u in sdp._all_units()}
    assert all(ptr in own for ptr, size in held.items() if size)
    idx = torch.randint(0, 100, (2, 8))
    with torch.no_grad():
        first = sdp(idx)
        sdp.load_full_state_dict({k: v * 1.5 for k, v in sdp.full_state_dict().items() if "w2" in k})
        second = sdp(idx)
        sdp.load_full_state_dict({k: v / 1.5 for k, v in sdp.full_state_dict().items() if "w2" in k})
        third = sdp(idx)
    assert not torch.equal(first, second)
    assert torch.allclose(first, third, rtol=1e-5, atol=1e-5 * float(first.abs().max()))
