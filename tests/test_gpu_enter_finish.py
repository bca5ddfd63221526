"""fd_enter and fd_finish (csrc/fd_finish.cu) against the per-function calls they
stand for: the same bits at every tile edge, type and variant."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
NAMES = ("psi", "npx", "npy", "np2", "rho", "ux", "uy", "p", "mu", "mix_tau")


def _lattice(H, W, variant, dtype):
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice
    from fingering_dynamics_gb300.params import periodic_reference_params, periodic_xy_params, walls_reference_params
    if variant == "periodic_xy":
        prm = periodic_xy_params(H, W, slab=W // 4)
    else:
        prm = (walls_reference_params if variant == "walls" else periodic_reference_params)().with_size(H, W)
    rects = [((W // 2, H // 2 - 1), (W // 2 + 2, H // 2 + 1))] if H >= 16 else []
    g = geo.build_geometry(H, W, rects=rects, walls=variant == "walls")
    rng = np.random.default_rng(H + W)
    lat = Lattice(prm, g, dtype=dtype, rho0=1 + 1e-3 * rng.standard_normal((H, W)), seed=3)
    lat.step_reference(3)
    return lat


@pytest.mark.parametrize("dtype", ["f64", "f32", "f16", "bf16", "f32-exact"])
@pytest.mark.parametrize("H,W,variant", [(3, 8, "walls"), (4, 32, "periodic"), (17, 36, "walls"), (32, 64, "periodic"),
                                         (33, 100, "walls"), (24, 52, "periodic_xy")])
def test_enter_and_finish_equal_the_separate_calls(H, W, variant, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300.lattice import _ptr
    a, b = _lattice(H, W, variant, dtype), _lattice(H, W, variant, dtype)
    a.enter_fused()
    # the separate calls
    b.boundary_fields(b.side[b.scur])
    b.collide()
    src = b.pop[b.cur]
    if b.storage is not None:
        packed = torch.zeros_like(a.ppop[a.pcur])
        a_state = a.current_buffer().clone()
        L.call("fd_pack", C.byref(b.prm), b.fd_dtype, _ptr(src), C.byref(b.storage), _ptr(packed), b._stream())
        P, es = H * W, 4 if dtype == "f32" else 2
        bf, bg = (P * es + 255) // 256 * 256, (P * 4 + 255) // 256 * 256  # planes start on 256-byte boundaries
        spans = [(i * bf, P * es) for i in range(9)] + [(9 * bf, P * 4)] + [(9 * bf + bg + i * bf, P * es) for i in range(8)]
        for o, n in spans:
            assert torch.equal(packed[o:o + n], a_state[o:o + n])
        L.call("fd_unpack", C.byref(b.prm), C.byref(b.storage), _ptr(packed), b.fd_dtype, _ptr(src), b._stream())
    assert torch.equal(a.side[a.scur], b.side[b.scur])
    b._finish_from(src, b.side[b.scur], b.pop[1 - b.cur])
    b.cur = 1 - b.cur
    a.exit_fused()
    assert torch.equal(a.f, b.f) and torch.equal(a.g, b.g)
    assert torch.isfinite(a.f).all() and torch.isfinite(a.psi).all()
    for n in NAMES:
        assert torch.equal(getattr(a, n), getattr(b, n)), n
