"""The lists of operations that a network's passes queue, with the launch itself
replaced (no GPU is needed)."""
import pytest

torch = pytest.importorskip("torch")

FLIP, WORDS = 9, 16


@pytest.fixture
def net(monkeypatch):
    from fingering_dynamics_gb300 import build
    from fingering_dynamics_gb300 import surrogate as sg
    build.build()
    net = sg.UNet((16, 16, 32, 32), seed=1, device="cpu")
    net.ran = []
    net._run_words = lambda words: net.ran.append([words[k] for k in range(0, len(words), WORDS)])
    monkeypatch.setattr(torch.cuda, "Event", _no_stopwatch)
    return net


def _no_stopwatch(*a, **k):
    raise AssertionError("a kernel was chosen by its time")


def _frames(n, h, w):
    return torch.zeros((n, h, w, 16), dtype=torch.bfloat16)


@pytest.mark.parametrize("h,w", [(8, 128), (16, 1024), (64, 8), (8, 200)])
def test_auto_chooses_by_shape(net, h, w):
    """conv="auto": the kernel of every convolution follows from its shape alone."""
    x = _frames(1, h, w)
    net.forward(x)
    net.backward(torch.zeros_like(x))
    assert len(net.ran) == 2  # one list a pass
    for key, fn in net.conv_choice.items():
        wide = key[-3] % 128 == 0
        if key[0] == "wgrad":
            assert wide and fn == "sg_conv3x3_wgrad_tc"
        else:
            assert fn == ("sg_conv3x3_tma" if wide else "sg_conv3x3_tc")
    assert len([k for k in net.conv_choice if k[0] != "wgrad"]) >= len(set(net.shapes.values()))


def test_a_choice_that_the_caller_made_stands(net):
    x = _frames(1, 8, 128)
    net.conv_choice[(1, 8, 128, 16, 16)] = "sg_conv3x3"
    net.predict(x)
    assert net.ran[0][:2] == [0, 0]  # enc1a, enc1b


def test_backward_after_one_that_raised_flips_the_weights(net):
    x = _frames(1, 8, 128)
    net.forward(x)
    with pytest.raises(AttributeError):
        net.backward(x.float().numpy())  # no tensor
    net.forward(x)
    net.backward(torch.zeros_like(x))
    assert net.ran[-1].count(FLIP) == len(net.shapes)
    net.backward(torch.zeros_like(x))
    assert FLIP not in net.ran[-1]  # the weights have not changed


@pytest.mark.parametrize("call", ["forward", "predict", "backward"])
def test_a_list_that_was_not_run_leaves_nothing_behind(net, call):
    """The launch of a pass fails once: the retry queues the flips and, if no pass
    has stored the pre-activations, the forward pass."""
    x, dout, run = _frames(1, 8, 128), _frames(1, 8, 128), net._run_words
    net.forward(x)
    forward = net.ran[-1]

    def fails(words):
        net._run_words = run
        raise RuntimeError("launch")
    net._run_words = fails
    with pytest.raises(RuntimeError):
        {"forward": net.forward, "predict": net.predict, "backward": net.backward}[call](x if call != "backward" else dout)
    net.backward(dout)
    kinds = net.ran[-1]
    assert kinds.count(FLIP) == len(net.shapes)
    assert (kinds[:len(forward)] == forward) == (call != "backward")


def test_plain_tensors_only():
    """What is not just its values keeps the tensor operations."""
    import torch.autograd.forward_ad as fwd
    from torch.utils._python_dispatch import TorchDispatchMode
    from fingering_dynamics_gb300.surrogate import _plain
    x = torch.ones(3)
    assert _plain(x, x > 0)
    assert not _plain(x, torch.ones(3, requires_grad=True))
    assert not _plain(torch.nn.Parameter(x, requires_grad=False))
    seen = []
    with fwd.dual_level():
        seen.append(_plain(fwd.make_dual(x, x)))
        assert _plain(x)

    def look(t):
        seen.append(_plain(t))
        return t.sum()
    torch.func.grad(look)(x)
    torch.func.vmap(look)(x[None])
    torch.jit.trace(look, x, check_trace=False)  # its check runs the function eagerly
    with TorchDispatchMode():
        seen.append(_plain(x))
    assert len(seen) >= 5 and not any(seen)
    assert _plain(x)
