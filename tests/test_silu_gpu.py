"""SiLU of every bf16 number against 64 bits: the fast division has to hold where its divisor leaves the
range that the instruction divides by, and for infinities, NaN and the two zeros."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [0, 1])
def test_silu_all_inputs(sign):
    from easy_to_hard_b200.ops import functional as F
    bits = (torch.arange(32768, dtype=torch.int32) + 32768 * sign).to(torch.int16)
    g = bits.view(torch.bfloat16).cuda()
    got = F.swiglu(g, torch.ones_like(g)).cpu().double()
    x = bits.view(torch.bfloat16).double()
    e = torch.exp(-x)
    want = x / (1 + e)
    nan = torch.isnan(x) | (x == -float("inf"))
    assert torch.isnan(got)[nan].all() and not torch.isnan(got)[~nan].any()
    # exp(-x) is infinite in 32 bits below -88.73: zero there, and within the bound everywhere else
    gone = (x < -88.73) & ~nan
    assert (got[gone] == 0).all()
    rest = ~nan & ~gone
    assert torch.equal(got[rest & torch.isinf(x)], x[rest & torch.isinf(x)])
    rest &= ~torch.isinf(x)
    # one rounding to bf16 (2^-8), the exponential (2 + 1.173 |x| units of 2^-23, as documented), the sum,
    # the division (2 units) and the scale; tiny results also lose what lies below the smallest bf16
    rel = 2.0 ** -8 + (2 + 1.173 * x.abs().clamp(max=128) + 4) * 2.0 ** -23
    err = (got - want).abs()
    assert (err[rest] <= (rel * want.abs() * (1 + 2.0 ** -8) + 2.0 ** -133)[rest]).all()
    assert torch.equal(torch.signbit(got[rest]), torch.signbit(x[rest]))


EXACT = r"""
// bf16 bits of x / (1 + __expf(-x)) with the division that rounds, for x = bf16 number `i`
extern "C" __global__ void silu_exact(unsigned short* out) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const float x = __uint_as_float(i << 16);
  const unsigned b = __float_as_uint(__fdiv_rn(x, 1.f + __expf(-x)));
  const bool nan = (b & 0x7fffffffu) > 0x7f800000u;
  out[i] = nan ? 0x7fff : (unsigned short)((b + 0x7fffu + ((b >> 16) & 1u)) >> 16);   // to nearest even
}
"""


def test_silu_is_the_number_of_the_rounding_division():
    """Bit for bit, for each of the 65536 inputs: the scaled fast division rounds to the same bf16 number."""
    from easy_to_hard_b200.ops import functional as F
    kernel = torch.cuda._compile_kernel(EXACT, "silu_exact")
    want = torch.empty(65536, dtype=torch.int16, device="cuda")
    kernel((256, 1, 1), (256, 1, 1), (want,))
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    got = F.swiglu(g, torch.ones_like(g))
    exact = want.view(torch.bfloat16)
    assert torch.equal(torch.isnan(got), torch.isnan(exact))
    assert torch.equal(got.view(torch.int16)[~torch.isnan(got)], want[~torch.isnan(got)])
