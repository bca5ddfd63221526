"""Ensemble.use_kernel: a batch of few cells runs the staged kernel on request, in
the default shape too, with the same bits."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_a_small_batch_runs_the_kernel_that_was_asked_for(dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fingering_dynamics_gb300.ensemble import Ensemble, ensemble_specs
    members = [s.build() for s in ensemble_specs(3, 5, sizes_w=(64, 128), sizes_h=(48, 64))]
    a, b = Ensemble(members, dtype=dtype), Ensemble(members, dtype=dtype)
    assert a.kernel == b.kernel == "tile"
    b.use_kernel("staged")
    assert b.kernel == "staged" and b.config == a.config
    for n in (4, 5):
        a.step(n)
        b.step(n)
        b.configure(*b.config)
        assert b.kernel == "staged"
    b.use_kernel("auto")
    a.configure(64, 32)  # a shape that only the staged kernel has
    assert (a.kernel, b.kernel) == ("staged", "tile")
    a.step(3)
    b.step(3)
    for p, q in zip(a.lattices, b.lattices):
        p.exit_fused()
        q.exit_fused()
        assert torch.equal(p.f, q.f) and torch.equal(p.g, q.g)
    with pytest.raises(ValueError):
        a.use_kernel("tile")
    a.close()
    b.close()


def test_arguments_are_checked_on_the_host():
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300 import build
    build.build()
    assert L.lib().fd_batch_kernel(None) == -1
    with pytest.raises(L.FDError) as e:
        L.call("fd_batch_set_kernel", C.c_void_p(), L.FD_BATCH_STAGED)
    assert e.value.code == -1
