"""Decode attention of grouped heads on the tensor cores (ops/csrc/attn_decode.cu) at the edges of its
32-key chunks and 8-key warps, one CTA per pair and several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [4, 8])
@pytest.mark.parametrize("pos,pad", [(0, 0), (7, 0), (8, 3), (31, 0), (32, 0), (33, 33), (63, 40),
                                     (700, 0), (767, 129)])
@pytest.mark.parametrize("n_split", [1, 8])
def test_against_64_bits(G, pos, pad, n_split):
    """Scores and sums carry 24 bits, so that 2^-17 of the largest value is ample for them; the result
    is rounded to bf16 (8 significant bits: at most half a unit in the last place, 2^-8 of it)."""
    from easy_to_hard_b200.ops import _lib, functional as Fn
    B, n_kv, D, smax = 5, 2, 128, 768
    g = torch.Generator(device="cuda").manual_seed(pos + G)
    q = torch.randn(B, n_kv * G * D, device="cuda", generator=g).bfloat16()
    kc, vc = (torch.randn(B, n_kv, smax, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    kc[:, :, pos + 1:], vc[:, :, pos + 1:] = float("nan"), float("nan")      # not live: never read
    kc[:, :, :pad], vc[:, :, :pad] = float("nan"), float("nan")
    left = torch.full((B,), pad, device="cuda", dtype=torch.int32)
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    for _ in range(2):             # the second run finds the first one's rows in shared memory
        out = Fn.attn_decode(q, kc, vc, at, left, n_kv * G, n_split=n_split)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    k, v = (t[:, :, pad:pos + 1].double().repeat_interleave(G, 1) for t in (kc, vc))
    s = (k @ q.double().view(B, n_kv * G, D, 1))[..., 0] * D ** -0.5
    want = (torch.softmax(s, -1)[..., None] * v).sum(2)
    err = (out.double().view(B, n_kv * G, D) - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + 2.0 ** -17 * v.abs().max()).all())


def test_a_captured_step_survives_a_larger_batch():
    """The scratch of a captured launch stays its own when a larger batch asks for more."""
    from easy_to_hard_b200.ops import _lib, functional as Fn
    n_kv, G, D, smax = 8, 8, 128, 512
    at = torch.tensor([500], dtype=torch.int32, device="cuda")

    def case(B):
        g = torch.Generator(device="cuda").manual_seed(B)
        return (torch.randn(B, n_kv * G * D, device="cuda", generator=g).bfloat16(),
                *(torch.randn(B, n_kv, smax, D, device="cuda", generator=g).bfloat16()
                  for _ in range(2)))
    small = case(2)
    want = Fn.attn_decode(*small, at, None, n_kv * G)
    out = torch.empty_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        Fn.attn_decode(*small, at, None, n_kv * G, out=out)
    Fn.attn_decode(*case(96), at, None, n_kv * G)
    torch.cuda.synchronize()
    taken = [torch.full((n,), -1, device="cuda", dtype=torch.int32) for n in (1 << 20, 4096, 4096)]
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert all(bool((t == -1).all()) for t in taken)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("G", [4, 8])
@pytest.mark.parametrize("n_split", [1, 8])
def test_infinite_values_stay_infinite(G, n_split):
    """The probabilities are split into parts, of which some are 0: an infinite value must not meet
    these. Dims without one keep their bound."""
    from easy_to_hard_b200.ops import _lib, functional as Fn
    B, n_kv, D, smax, pos = 3, 2, 128, 128, 100
    g = torch.Generator(device="cuda").manual_seed(G)
    q = torch.randn(B, n_kv * G * D, device="cuda", generator=g).bfloat16()
    q[1] = 0                                        # equal probabilities: exact in the first part
    kc, vc = (torch.randn(B, n_kv, smax, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    vc[:, :, 3, 5], vc[:, 1, 40, 6], vc[:, 0, 100, 127] = float("inf"), float("-inf"), float("inf")
    vc[2, 1, 60, 8], vc[2, 1, 61, 8], vc[0, 0, 9, 9] = float("inf"), float("-inf"), float("nan")
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    out = Fn.attn_decode(q, kc, vc, at, None, n_kv * G, n_split=n_split).view(B, n_kv * G, D)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    k, v = (t[:, :, :pos + 1].double().repeat_interleave(G, 1) for t in (kc, vc))
    s = (k @ q.double().view(B, n_kv * G, D, 1))[..., 0] * D ** -0.5
    want = (torch.softmax(s, -1)[..., None] * v).sum(2)
    live = torch.isfinite(want)
    assert int((~live).sum()) > 0 and torch.equal(torch.isfinite(out), live)
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.equal(out[torch.isinf(want)].double(), want[torch.isinf(want)])
    err = (out.double() - want).abs()
    assert bool((err[live] <= (2.0 ** -8 * want.abs() + 2.0 ** -17 * 8)[live]).all())
