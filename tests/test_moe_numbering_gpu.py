"""Numbering of the choices of many tokens: runs of the 32 warps that end inside, at and before the choices,
experts without tokens, more experts than choices of a token."""
import pytest
import torch

from easy_to_hard_b200.ops import hybrid as hy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E,top", [(300, 4, 2), (512, 1, 1), (513, 3, 3), (1023, 8, 1), (1025, 64, 2),
                                     (4096, 4, 2), (12568, 5, 2)])
def test_numbering(n, E, top):
    g = torch.Generator(device="cuda").manual_seed(n)
    W = 64
    z = torch.randn(n, E, device="cuda", generator=g)
    z[:, 0] -= 20.0 if E > top else 0.0            # an expert that nobody chooses
    h = torch.randn(n, W, device="cuda", generator=g).bfloat16()
    hg = torch.empty(n * top, W, device="cuda").bfloat16()
    off, place = torch.empty(E + 1, device="cuda").int(), torch.empty(n, top, device="cuda").int()
    w, sel = torch.empty(n, top, device="cuda"), torch.empty(n, top, device="cuda").int()
    hy.moe_route(z, E, top, h, hg, off, place, w, sel)
    flat = sel.flatten().long()
    assert torch.equal(flat.view(n, top), z.topk(top, dim=-1).indices)
    order = torch.sort(flat, stable=True).indices
    want = torch.empty_like(order)
    want[order] = torch.arange(n * top, device="cuda")
    assert torch.equal(place.flatten().long(), want)
    count = torch.bincount(flat, minlength=E)
    assert torch.equal(off.long(), torch.cat([count.new_zeros(1), count.cumsum(0)]))
    assert torch.equal(hg[place.long()], h[:, None].expand(-1, top, -1))
