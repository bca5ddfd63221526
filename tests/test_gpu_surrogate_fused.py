"""The surrogate's one-pass kernels against the calls they stand for, bit for bit,
at sizes that end inside a block, and predict() followed by backward()."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _call(name, *a):
    from fingering_dynamics_gb300 import _lib as L
    L.call(name, *a)


def _rand(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (2 * torch.randn(shape, generator=g, device="cuda")).to(torch.bfloat16)


@pytest.mark.parametrize("n,h,w,c,cy,coff", [(1, 2, 2, 8, 8, 0), (2, 6, 10, 32, 96, 64), (1, 8, 16, 256, 384, 0),
                                             (3, 4, 6, 16, 48, 16)])
@pytest.mark.parametrize("source", [0, 1, 2])
def test_gelu_bias_backward(source, n, h, w, c, cy, coff):
    from fingering_dynamics_gb300 import _lib as L
    z = _rand(1, n, h, w, c)
    P = n * h * w
    part = torch.empty(int(L.lib().sg_bias_partial_floats(c)), device="cuda")
    skip = None
    if source == 0:
        src = dy = _rand(2, n, h, w, c)
    elif source == 1:
        src = _rand(3, n, 2 * h, 2 * w, cy)
        dy = torch.empty_like(z)
        _call("sg_up2_bwd", _p(src), n, h, w, cy, coff, c, _p(dy), None)
    else:
        src, skip = _rand(4, n, h // 2, w // 2, c), _rand(5, n, h, w, cy)
        dy = torch.empty_like(z)
        _call("sg_pool2_bwd", _p(src), n, h, w, c, _p(dy), None)
        _call("sg_add_channels", _p(skip), P, cy, coff, c, _p(dy), None)
    dz, dz1 = torch.empty_like(z), torch.empty_like(z)
    db, db1 = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    _call("sg_gelu_bwd", _p(dy), _p(z), z.numel(), _p(dz), None)
    _call("sg_bias_grad", _p(dz), P, c, _p(db), _p(part), None)
    _call("sg_gelu_bias_bwd", source, _p(src), _p(skip), n, h, w, cy, coff, _p(z), c, _p(dz1), _p(db1), _p(part), None)
    assert torch.equal(dz, dz1) and torch.equal(db, db1)


@pytest.mark.parametrize("n,h,w,c,cs", [(1, 1, 1, 8, 8), (2, 3, 5, 16, 40), (1, 4, 8, 256, 128)])
def test_up_concat(n, h, w, c, cs):
    x, skip = _rand(1, n, h, w, c), _rand(2, n, 2 * h, 2 * w, cs)
    a, b = (torch.zeros((n, 2 * h, 2 * w, c + cs), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _call("sg_up2", _p(x), n, h, w, c, _p(a), c + cs, 0, None)
    _call("sg_copy_channels", _p(skip), n * 4 * h * w, cs, _p(a), c + cs, c, None)
    _call("sg_up2_concat", _p(x), n, h, w, c, _p(skip), cs, _p(b), None)
    assert torch.equal(a, b)


@pytest.mark.parametrize("c,solid", [(16, 0.3), (24, 0.3), (16, 1.0)])
def test_loss_and_prediction(c, solid):
    n, h, w = 2, 9, 13
    x, out, xn = _rand(1, n, h, w, c), _rand(2, n, h, w, c), _rand(3, n, h, w, c)
    x[..., 3] = (torch.rand((n, h, w), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)) < solid)
    P = n * h * w
    from fingering_dynamics_gb300 import _lib as L
    count = max(float((x[..., 3] == 0).sum().item()), 1.0)
    d, d1 = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
    lp, lp1 = (torch.empty(2 * L.lib().sg_loss_blocks(), device="cuda") for _ in range(2))
    cnt, inv = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(2, device="cuda")
    _call("sg_masked_mse", _p(x), _p(out), _p(xn), P, c, _p(d), _p(lp), 1.0 / (3.0 * count), None)
    _call("sg_loss_scale", _p(x), P, c, _p(cnt), _p(inv), None)
    _call("sg_masked_mse_scaled", _p(x), _p(out), _p(xn), P, c, _p(d1), _p(lp1), _p(inv), None)
    assert torch.equal(d, d1) and torch.equal(lp, lp1)
    s = lp.view(-1, 2)[:, 0].sum()
    assert torch.equal(s / (3.0 * count), s * inv[1])
    y = torch.empty_like(x)
    _call("sg_add_prediction", _p(x), _p(out), P, c, _p(y), None)
    ref = x.clone()
    ref[..., :3] = (x[..., :3].float() + out[..., :3].float()).to(torch.bfloat16)
    assert torch.equal(y, ref)


def test_adamw_list_and_predict_then_backward():
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300.surrogate import LAYERS, UNet
    net = UNet((16, 16, 32, 32), seed=3, conv="tma")
    net.w["out"] = torch.from_numpy(np.random.default_rng(1).normal(0, 0.05, net.w["out"].shape).astype(np.float32)).cuda()
    net.w16 = {n: t.to(torch.bfloat16) for n, t in net.w.items()}
    x = _rand(1, 1, 16, 128, 16)
    dout = _rand(2, 1, 16, 128, 16)
    net.forward(x)
    net.backward(dout)
    ref = {n: (net.gw[n].clone(), net.gb[n].clone()) for n in LAYERS}
    net.predict(x)
    net.backward(dout)
    for n in LAYERS:
        assert torch.equal(net.gw[n], ref[n][0]) and torch.equal(net.gb[n], ref[n][1]), n
    want = {}
    for n in LAYERS:
        for k, w, w16, g, m, v, wd in (("w", net.w, net.w16[n].clone(), net.gw, net.mw, net.vw, 1e-2),
                                       ("b", net.b, None, net.gb, net.mb, net.vb, 0.0)):
            t = [a[n].clone() for a in (w, g, m, v)]
            _call("sg_adamw", _p(t[0]), _p(w16), _p(t[1]), _p(t[2]), _p(t[3]), t[0].numel(), 1e-3, 0.9, 0.999, 1e-8, wd, 1, None)
            want[n + k] = (t[0], w16)
    net.adamw(lr=1e-3)
    for n in LAYERS:
        assert torch.equal(net.w[n], want[n + "w"][0]) and torch.equal(net.w16[n], want[n + "w"][1])
        assert torch.equal(net.b[n], want[n + "b"][0])


@pytest.mark.parametrize("n,h,w", [(1, 64, 128), (2, 128, 256)])
def test_a_list_equals_its_operations(n, h, w):
    """Operations of a list overlap (a kernel starts while the previous one
    drains); the buffers are reused by every pass, so a missing wait would show."""
    from fingering_dynamics_gb300.surrogate import UNet
    net = UNet(seed=3, conv="tma")
    net.w16["out"] = _rand(99, *net.w16["out"].shape)  # zero in a new network
    xs = [_rand(k, n, h, w, 16) for k in range(12)]
    listed = [net.predict(x).clone() for x in xs]
    run = net._run_words
    net._run_words = lambda words: [run(words[k:k + 16]) for k in range(0, len(words), 16)]
    for x, y in zip(xs, listed):
        assert torch.equal(net.predict(x), y)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("h,w", [(1, 1), (3, 40), (33, 257)])
def test_frame_equals_the_tensor_operations(dtype, h, w):
    """sg_frame against the tensor operations (which strided fields still take), with infinities and NaN."""
    from fingering_dynamics_gb300.surrogate import frame_from_fields
    g = torch.Generator(device="cuda").manual_seed(h)
    psi, ux, uy = (torch.randn((h, 2 * w), generator=g, device="cuda", dtype=getattr(torch, dtype)) * s
                   for s in (1.0, 3e-2, 1e-9))
    if h > 1:
        ux[0, 0], uy[1, 2], psi[2, 4], ux[1, 0] = float("inf"), float("-inf"), float("nan"), 1e-40
    solid = torch.rand((h, 2 * w), generator=g, device="cuda") < 0.3
    want = frame_from_fields(psi[:, ::2], ux[:, ::2], uy[:, ::2], solid[:, ::2])
    got = frame_from_fields(*(t[:, ::2].contiguous() for t in (psi, ux, uy, solid)))
    assert got.shape == want.shape and torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.nan_to_num(got).view(torch.int16), torch.nan_to_num(want).view(torch.int16))
