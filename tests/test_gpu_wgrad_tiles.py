"""The tcgen05 weight gradient (sg_conv3x3_wgrad_tc) against the oracle: every
channel block and output tile, one row and one split, splits that cross image
rows and images, and more splits than chunks.

Tolerance: products of bfloat16 are exact in FP32; a sum of K of them in FP32
with truncation loses at most K 2^-23 of the sum of magnitudes, here at most
768 * 2^-23 * sqrt(768) of a result of size sqrt(768): 9.2e-5 of the largest."""
import ctypes as C

import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,h,w,cin,cout", [(2, 3, 128, 16, 32), (1, 1, 128, 16, 16), (1, 3, 256, 32, 48), (1, 2, 128, 32, 128),
                                            (2, 2, 128, 96, 32), (1, 2, 128, 96, 64), (1, 3, 128, 64, 16), (1, 2, 256, 64, 64),
                                            (1, 2, 128, 192, 128), (1, 1, 384, 160, 32), (2, 1, 128, 48, 80),
                                            (1, 2, 128, 128, 16), (1, 2, 256, 256, 128)])
@pytest.mark.parametrize("splits", [0, 1, 3, 1000])
def test_weight_gradient_tiles_match_oracle(n, h, w, cin, cout, splits):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    rng = np.random.default_rng(cin + cout + h)
    x = torch.from_numpy(rng.standard_normal((n, h, w, cin), dtype=np.float32)).to(torch.bfloat16)
    dz = torch.from_numpy(rng.standard_normal((n, h, w, cout), dtype=np.float32)).to(torch.bfloat16)
    ref = U.conv3x3_wgrad(x.double().numpy(), dz.double().numpy())
    xd, dd = x.cuda(), dz.cuda()
    part = torch.empty(int(L.lib().sg_wgrad_partial_floats(n, h, w, cin, cout)), device="cuda")
    dw = torch.empty((cout, 3, 3, cin), device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    dw.fill_(float("nan"))
    L.call("sg_conv3x3_wgrad_tc", p(xd), p(dd), n, h, w, cin, cout, p(dw), p(part), part.numel(), splits, None)
    torch.cuda.synchronize()
    err = C.c_uint(0)
    L.call("sg_tc_status", C.byref(err), 0)
    assert err.value == 0
    assert np.abs(dw.cpu().numpy() - ref).max() <= 9.2e-5 * np.abs(ref).max()
