"""The persistent tcgen05 convolutions at the edges of their tiles: widths that
are multiples of 128 (rows per tile 1, 2, 4; weights resident and streamed; one
chunk and many; every output tile) and widths that divide 128 (tiles that end past
the last row).  Inputs, weights and bias are small integers, so every sum is exact
in FP32 in any order: z is the exact convolution rounded once to bfloat16, and y
is what the warp-level kernel gives for the same sums."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _check(fn, n, h, w, cin, cout, act):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    rng = np.random.default_rng(cin + cout + h)
    x = torch.from_numpy(rng.integers(-3, 4, (n, h, w, cin)).astype(np.float32)).to(torch.bfloat16)
    wt = torch.from_numpy(rng.integers(-2, 3, (cout, 3, 3, cin)).astype(np.float32)).to(torch.bfloat16)
    b = torch.from_numpy(rng.integers(-4, 5, cout).astype(np.float32))
    exact = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double().permute(0, 3, 1, 2),
                                       b.double() if act else None, padding=1).permute(0, 2, 3, 1)
    assert float(exact.abs().max()) < 2 ** 24
    xd, wd, bd = x.cuda(), wt.cuda(), b.cuda()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    out = {}
    for f in (fn, "sg_conv3x3"):
        z, y = (torch.full((n, h, w, cout), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        L.call(f, p(xd), n, h, w, cin, p(wd), p(bd) if act else None, cout, act, p(z) if act else None, p(y), None)
        out[f] = (z if act else y, y)
    torch.cuda.synchronize()
    err = C.c_uint(0)
    L.call("sg_tc_status", C.byref(err), 0)
    assert err.value == 0
    assert torch.equal(out[fn][0].cpu(), exact.to(torch.bfloat16))
    assert torch.equal(out[fn][1], out["sg_conv3x3"][1])


@pytest.mark.parametrize("n,h,w,cin,cout,act", [(1, 1, 128, 16, 16, 1), (1, 2, 128, 32, 32, 1), (2, 3, 256, 48, 96, 0),
                                                (1, 8, 128, 96, 64, 1), (1, 4, 128, 384, 128, 1), (2, 64, 512, 32, 96, 0),
                                                (4, 128, 256, 64, 64, 1), (2, 160, 256, 16, 32, 1), (1, 6, 128, 256, 160, 0),
                                                (3, 200, 128, 64, 192, 0)])
def test_wide_convolution_is_exact(n, h, w, cin, cout, act):
    _check("sg_conv3x3_tma", n, h, w, cin, cout, act)


@pytest.mark.parametrize("n,h,w,cin,cout,act", [(1, 1, 64, 16, 16, 1), (2, 3, 64, 32, 48, 1), (3, 32, 64, 128, 256, 1),
                                                (1, 5, 32, 64, 64, 0), (2, 9, 16, 96, 32, 1), (1, 17, 8, 256, 128, 0),
                                                (40, 8, 64, 64, 128, 1)])
def test_narrow_convolution_is_exact(n, h, w, cin, cout, act):
    _check("sg_conv3x3_tc", n, h, w, cin, cout, act)


@pytest.mark.parametrize("n,h,w,cin,cout,act", [(1, 1, 1, 16, 16, 1), (2, 3, 9, 32, 48, 0), (1, 13, 9, 256, 64, 1),
                                                (3, 7, 25, 96, 32, 1), (1, 50, 41, 64, 128, 1), (2, 21, 62, 48, 32, 1),
                                                (1, 9, 63, 32, 64, 0), (2, 5, 100, 96, 64, 1), (1, 6, 126, 32, 32, 1),
                                                (1, 6, 127, 128, 32, 0), (2, 4, 129, 16, 32, 1), (1, 11, 130, 64, 16, 1),
                                                (4, 40, 328, 32, 32, 1), (1, 3, 1000, 96, 160, 0),
                                                (1, 2, 2100, 32, 16, 1), (1, 3, 2184, 64, 32, 0)])
def test_any_width_convolution_is_exact(n, h, w, cin, cout, act):
    _check("sg_conv3x3_tc", n, h, w, cin, cout, act)


@pytest.mark.parametrize("fn,w", [("sg_conv3x3_tma", 128), ("sg_conv3x3_tc", 40)])
def test_outputs_that_are_16_byte_aligned_only(fn, w):
    """z and y at 16 bytes from a 32-byte boundary take two stores per sector."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((1, 4, w, 32), generator=g, device="cuda").to(torch.bfloat16)
    wt = torch.randn((48, 3, 3, 32), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(48, generator=g, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    out = []
    for off in (0, 8):
        z, y = (torch.zeros(4 * w * 48 + 16, dtype=torch.bfloat16, device="cuda")[off:off + 4 * w * 48] for _ in range(2))
        L.call(fn, p(x), 1, 4, w, 32, p(wt), p(b), 48, 1, p(z), p(y), None)
        out.append((z, y))
    torch.cuda.synchronize()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
