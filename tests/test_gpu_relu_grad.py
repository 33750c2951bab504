"""The ReLU gradient's two forms (four elements per thread for powers of two and aligned tensors, else one): masked
gradients bit for bit, channel sums to the rounding of Float32 sums."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


# lanes of a warp that repeat channels or not, one channel, channels beyond a block's elements, a last step that is
# not full, more steps than one, element counts not divisible by four
@pytest.mark.parametrize("P,C", [(1, 16), (5, 1), (4, 1), (6, 2), (7, 8), (33, 16), (129, 48), (1000, 64), (77, 256),
                                 (9, 1024), (3, 2048), (40000, 32), (20000, 24)])
@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_relu_gradient(shk, cuda, P, C, relu, offset):
    from shakti_b200 import warmstart as ws
    torch, n = cuda, P * C
    gen = torch.Generator("cuda").manual_seed(3)
    dY = torch.randn(n + 8, generator=gen, device="cuda")[offset:offset + n]
    Y = torch.randn(n + 8, generator=gen, device="cuda").relu().bfloat16()[offset:offset + n]
    out = torch.full((n + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    db = torch.ones(C, device="cuda")  # the kernel adds
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = shk._lib.load()
    assert L.shk_nn_relu_grad(ws._fp(dY), ws._p(Y), ws._p(out[offset:]), ws._fp(db), P, C, relu, s) == 0
    want = torch.where(Y.float() > 0, dY, torch.zeros_like(dY)) if relu else dY
    assert torch.equal(out[offset:offset + n], want.bfloat16())
    assert torch.all(out[:offset] == 7) and torch.all(out[offset + n:] == 7)
    sums = want.double().view(P, C)
    # a sum of P terms in any order: P 2^-24 of the magnitudes at worst, plus the rounding of 1 + sum
    bound = (P * 2.0 ** -24 * sums.abs().sum(0) + 2.0 ** -23 * (1 + sums.sum(0).abs())) + 1e-30
    assert torch.all((db.double() - 1.0 - sums.sum(0)).abs() <= bound)
