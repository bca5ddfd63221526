"""The densely packed getters (fd_collision_term_fluid, fd_field_fluid) against
the full-grid entry points on the same fields: the same bits on every fluid
cell, every term, direction and type, with the first and last cell of the
lattice fluid or solid."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("H,W,corner_solid", [(4, 8, False), (16, 33, True), (24, 48, False)])
def test_packed_getters_equal_the_full_grid_ones(H, W, corner_solid, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300 import fingering_periodic as fp
    rng = np.random.default_rng(H)
    mask = rng.random((H, W)) < 0.8
    mask[0, 0] = mask[-1, -1] = not corner_solid
    fp.H, fp.W = H, W
    cm = fp.Compute(mask, dtype=getattr(torch, dtype))
    g = torch.Generator().manual_seed(H)
    for t in (cm.f, cm.g, cm.psi, cm.nabla_psix, cm.nabla_psiy, cm.nabla_psi2, *cm._full.values()):
        t.copy_(0.1 + torch.rand(t.shape, generator=g, dtype=torch.float64).to(t.dtype))
    m = torch.from_numpy(mask).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    full = torch.zeros((H, W), dtype=cm._dtype, device="cuda")
    for term, tid in L.TERMS.items():
        for j in range(9):
            L.call("fd_collision_term", C.byref(cm._prm), cm._fd, tid, j, p(cm._word), C.byref(cm._fields()), p(full), None)
            assert torch.equal(cm._term(term, j), full[m]), (term, j)
    for name in ("rho", "mu", "ux", "uy", "p", "mix_tau"):
        L.call("fd_field", C.byref(cm._prm), cm._fd, L.FIELDS[name], p(cm._word), C.byref(cm._fields()), p(full), None)
        assert torch.equal(cm._field(name), full[m]), name
