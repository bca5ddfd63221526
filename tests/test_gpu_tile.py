"""The one-thread-per-cell packed step (csrc/fd_tile.cuh) against the staged
kernel: the same bits at every tile edge, in every storage type, rounding,
scale and variant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _lattice(H, W, variant, dtype, rounding, scales):
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice
    from fingering_dynamics_gb300.params import periodic_reference_params, walls_reference_params
    prm = (walls_reference_params if variant == "walls" else periodic_reference_params)().with_size(H, W)
    prm.M = 4.0
    if variant == "walls":
        prm.u0, prm.inlet_ux = 0.006, np.full(H, 0.006)
    rects = [((W // 2, H // 2 - 1), (W // 2 + 2, H // 2 + 1))] if H >= 16 else []
    g = geo.build_geometry(H, W, rects=rects, walls=variant == "walls")
    lat = Lattice(prm, g, dtype=dtype, rounding=rounding, seed=7)
    lat.storage.f_scale_log2, lat.storage.g_scale_log2 = scales
    lat.enter_fused()
    return lat


@pytest.mark.parametrize("dtype,rounding,scales", [("f32", "nearest", (0, 0)), ("f16", "stochastic", (0, 0)),
                                                   ("f16", "nearest", (4, 2)), ("bf16", "stochastic", (3, 0)),
                                                   ("bf16", "nearest", (0, 0))])
@pytest.mark.parametrize("H,W,variant", [(3, 8, "walls"), (4, 32, "periodic"), (5, 40, "walls"), (16, 24, "periodic"),
                                         (33, 136, "walls"), (64, 128, "periodic"), (130, 264, "walls")])
def test_tile_step_equals_the_staged_step(H, W, variant, dtype, rounding, scales):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a, b = (_lattice(H, W, variant, dtype, rounding, scales) for _ in range(2))
    a.advance(7)
    b.advance(7, rows_per_warp=16)  # a strip height asks for the staged kernel
    for k in ("psi", "ux", "uy", "rho"):
        assert not torch.isnan(getattr(a, k)).any()
    a.exit_fused()
    b.exit_fused()
    assert torch.equal(a.f, b.f) and torch.equal(a.g, b.g) and torch.equal(a.side[a.scur], b.side[b.scur])


@pytest.mark.parametrize("dtype,rounding", [("f32", "nearest"), ("f16", "stochastic"), ("bf16", "nearest")])
def test_small_batch_equals_the_staged_batch(dtype, rounding):
    """A batch small enough for the tile kernel, against the same batch in strips
    of 31 rows (the staged kernel)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300.ensemble import Ensemble
    sizes = [(3, 8, "walls"), (16, 24, "walls"), (33, 136, "walls"), (64, 128, "periodic")]

    def batch():
        lats = [_lattice(H, W, v, dtype, rounding, (0, 0)) for H, W, v in sizes]
        return Ensemble.from_lattices(lats)
    a, b = batch(), batch()
    b.configure(128, 31)
    for n, graph in ((5, True), (1, False), (4, True)):
        a.step(n, use_graph=graph)
        b.step(n, use_graph=graph)
    for p, q in zip(a.lattices, b.lattices):
        p.exit_fused()
        q.exit_fused()
        assert not torch.isnan(p.f).any()
        assert torch.equal(p.f, q.f) and torch.equal(p.g, q.g) and torch.equal(p.side[p.scur], q.side[q.scur])
