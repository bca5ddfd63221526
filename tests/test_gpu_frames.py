"""frame_from_fields and predict on tensors that are more than their values, and on
empty fields: the tensor operations' results."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_a_frame_carries_its_tangent():
    import torch.autograd.forward_ad as fwd
    from fingering_dynamics_gb300.surrogate import VELOCITY_SCALE, frame_from_fields
    psi, ux, uy, dpsi, dux = (torch.randn((4, 24), device="cuda") for _ in range(5))
    solid = torch.rand((4, 24), device="cuda") < 0.3
    with fwd.dual_level():
        v, t = fwd.unpack_dual(frame_from_fields(fwd.make_dual(psi, dpsi), fwd.make_dual(ux, dux), uy, solid))
        v, t = v.clone(), t.clone()
    assert torch.equal(v, frame_from_fields(psi, ux, uy, solid))
    want = torch.zeros_like(t)
    want[..., 0] = dpsi.to(torch.bfloat16)
    want[..., 1] = (torch.where(solid, 0, dux) / VELOCITY_SCALE).to(torch.bfloat16)
    assert torch.equal(t, want)


@pytest.mark.parametrize("h,w", [(0, 8), (8, 0)])
def test_empty_fields_give_an_empty_frame(h, w):
    from fingering_dynamics_gb300.surrogate import frame_from_fields
    a = torch.zeros((h, w), device="cuda")
    assert frame_from_fields(a, a, a, a > 0).shape == (h, w, 16)


def test_a_prediction_stays_attached_to_its_frames():
    from fingering_dynamics_gb300.surrogate import UNet
    net = UNet((16, 16, 32, 32), seed=1)
    x = torch.randn((1, 8, 16, 16), device="cuda").to(torch.bfloat16)
    y = net.predict(x)
    z = net.predict(x.clone().requires_grad_())
    assert z.requires_grad and not y.requires_grad and torch.equal(y, z.detach())
