"""Steps and predictions recorded in a CUDA graph by the caller and replayed: what a
run outside gives (several of their kernels are launched programmatically)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _lattice(H, W, dtype):
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice
    from fingering_dynamics_gb300.params import walls_reference_params
    prm = walls_reference_params().with_size(H, W)
    prm.u0, prm.inlet_ux = 0.006, np.full(H, 0.006)
    return Lattice(prm, geo.build_geometry(H, W, rects=[((W // 2, 8), (W // 2 + 4, 12))], walls=True), dtype=dtype,
                   rounding="nearest")


@pytest.mark.parametrize("H,W,dtype,rows", [(40, 64, "f64", 0), (40, 64, "f32", 0), (33, 92, "bf16", 0), (64, 128, "f16", 16)])
def test_a_recorded_advance(H, W, dtype, rows):
    a, b = _lattice(H, W, dtype), _lattice(H, W, dtype)
    for lat in (a, b):
        lat.enter_fused()
        lat.advance(2, rows_per_warp=rows)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.advance(4, rows_per_warp=rows)
    for _ in range(3):
        g.replay()
        b.advance(4, rows_per_warp=rows)
    a.exit_fused()
    b.exit_fused()
    assert torch.equal(a.f, b.f) and torch.equal(a.g, b.g) and torch.isfinite(a.f).all()


@pytest.mark.parametrize("rows", [16, 32])  # the staged kernel, the tile kernel
def test_a_recorded_batch_step(rows):
    from fingering_dynamics_gb300.ensemble import Ensemble
    a, b = (Ensemble.from_lattices([_lattice(40, 64, "f32"), _lattice(33, 128, "f32")], rows_per_strip=rows) for _ in range(2))
    for e in (a, b):
        e.step(2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.step(4, use_graph=False)
    for _ in range(3):
        g.replay()
        b.step(4)
    torch.cuda.synchronize()
    for p, q in zip(a.lattices, b.lattices):
        p.exit_fused()
        q.exit_fused()
        assert torch.equal(p.f, q.f) and torch.equal(p.g, q.g)
    a.close()
    b.close()


@pytest.mark.parametrize("h,w", [(64, 128), (40, 72)])
def test_a_recorded_prediction_and_training_step(h, w):
    from fingering_dynamics_gb300.surrogate import UNet
    net = UNet(seed=3)
    net.w16["out"] = torch.randn(net.w16["out"].shape, device="cuda").to(torch.bfloat16) * 0.02
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, xn = (torch.randn((2, h, w, 16), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    x[..., 3] = 0
    want = net.predict(x).clone()
    loss = net.loss_grad(x, xn).clone()
    grads = {n: t.clone() for n, t in net.gw.items()}
    torch.cuda.synchronize()
    gp, gt = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(gp):
        y = net.predict(x)
    with torch.cuda.graph(gt):
        l = net.loss_grad(x, xn)
    for t in net.gw.values():
        t.zero_()
    y.zero_()
    gp.replay()
    gt.replay()
    assert torch.equal(y, want) and torch.equal(l, loss)
    assert all(torch.equal(net.gw[n], grads[n]) for n in grads)
