"""The weight gradient where a block takes several pixel chunks: images of 256 chunks (unaligned tensors: 1024) and
more, with a last block and a last chunk that are not full; and images smaller than half a chunk.

Bound: a block adds at most 64 products of 16 pixels into one Float32 sum, each step off by at most 2^-23 of it, and
the blocks' sums, of magnitude s, are added by atomics, each off by 2^-24 of the running total T.  With sums
of independent signs T is at most the largest gradient and n blocks of s add up to n s = sqrt(n) T, so the error is
below (64 * 2^-23 * sqrt(n) / 2 + n 2^-24) T: 9e-5 T for the 261 blocks of the largest image here."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,offset", [((1, 300, 225, 8, 16), 0), ((3, 211, 173, 24, 48), 0), ((1, 513, 520, 16, 16), 0),
                                          ((1, 513, 520, 8, 16), 1), ((1, 513, 520, 8, 32), 2), ((1, 11, 11, 40, 16), 0),
                                          ((2, 7, 9, 8, 80), 1), ((1, 8, 16, 16, 16), 0), ((1, 3, 43, 16, 16), 3)])
def test_weight_gradient_ranges(shk, cuda, shape, offset):
    from shakti_b200 import warmstart as ws
    torch = cuda
    N, H, W, ci, co = shape
    gen = torch.Generator("cuda").manual_seed(7)

    def tensor(c):
        t = torch.zeros(N * H * W * c + 8, dtype=torch.bfloat16, device="cuda")[offset:offset + N * H * W * c]
        return t.copy_(torch.randn(t.shape, generator=gen, device="cuda")).view(N, H, W, c)

    X, dY = tensor(ci), tensor(co)
    dW = torch.zeros((9, co, ci), device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert shk._lib.load().shk_nn_conv3x3_wgrad(ws._p(X), ws._p(dY), ws._fp(dW), N, H, W, ci, co, s) == 0
    Xp = torch.nn.functional.pad(X.double(), (0, 0, 1, 1, 1, 1))
    ref = torch.stack([torch.einsum("nhwo,nhwi->oi", dY.double(), Xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W])
                       for t in range(9)])
    assert torch.max(torch.abs(dW.double() - ref)) <= 9e-5 * torch.max(torch.abs(ref))
