"""The weight-gradient kernel at the edges of its tiles (32 x 32 channels, 256 pixels) against the CPU
restatement: channel counts that do not fill a tile, chunks that end inside an image row, images smaller
than a chunk, several images per chunk, and tensors that are not 16-byte aligned.

Products of BF16 values are exact in Float32 and at most a few thousand are summed, so each sum is within
a few thousand 2^-24 of the sum of magnitudes at worst and within 1e-6 of it in practice; 1e-5 of the
largest gradient is the bound the kernel has been held to so far."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 16), (1, 2, 3, 24, 16), (3, 5, 7, 24, 48), (2, 16, 16, 16, 32),
                                   (5, 8, 8, 40, 80), (1, 40, 9, 64, 16), (2, 33, 31, 32, 64), (1, 1, 600, 16, 16),
                                   (4, 4, 4, 256, 128)])
@pytest.mark.parametrize("offset", [0, 1])
def test_weight_gradient(shk, cuda, shape, offset):
    import sys
    from pathlib import Path
    sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
    import nn_oracle as no
    from shakti_b200 import warmstart as ws
    torch = cuda
    N, H, W, ci, co = shape
    g = np.random.default_rng(7)

    def tensor(c):  # `offset` elements past an aligned address
        n = N * H * W * c
        t = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")[offset:offset + n]
        t.copy_(torch.from_numpy(g.normal(0, 1, size=n).astype(np.float32)).cuda())
        return t.view(N, H, W, c)

    X, dY = tensor(ci), tensor(co)
    dW = torch.ones((9, co, ci), dtype=torch.float32, device="cuda")  # the kernel adds
    L = shk._lib.load()
    import ctypes
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.shk_nn_conv3x3_wgrad(ws._p(X), ws._p(dY), ws._fp(dW), N, H, W, ci, co, s) == 0
    ref = no.conv3x3_wgrad(X.float().cpu().numpy(), dY.float().cpu().numpy())
    err = np.max(np.abs(dW.cpu().numpy() - 1.0 - ref))
    assert err <= 1e-5 * max(1.0, np.max(np.abs(ref)))
