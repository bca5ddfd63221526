"""Lattice.peek: the fields of the next iteration in the field tensors, the pending
populations in f and g, and the fused state untouched."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("H,W", [(3, 8), (33, 100), (48, 128)])
def test_peek_shows_the_pending_state(H, W, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import FIELD_NAMES, Lattice, _ptr
    from fingering_dynamics_gb300.params import walls_reference_params
    prm = walls_reference_params().with_size(H, W)
    a, b = (Lattice(prm, geo.build_geometry(H, W, walls=True), dtype=dtype, seed=2) for _ in range(2))
    for lat in (a, b):
        lat.enter_fused()
        lat.advance(3)
    state, side = a.current_buffer().clone(), a.side[a.scur].clone()
    a.peek()
    assert torch.equal(a.current_buffer(), state) and torch.equal(a.side[a.scur], side)
    want = torch.empty_like(a.pop[0])
    L.call("fd_unpack", C.byref(a.prm), C.byref(a.storage), _ptr(state), a.fd_dtype, _ptr(want), a._stream())
    assert torch.equal(a.f, want[:9]) and torch.equal(a.g, want[9:])
    b.exit_fused()
    for n in FIELD_NAMES:
        assert torch.equal(getattr(a, n), getattr(b, n)), n
    a.exit_fused()  # and what follows is what would have followed
    assert torch.equal(a.f, b.f) and torch.equal(a.g, b.g)
