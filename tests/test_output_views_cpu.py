"""OutputViews: every call's tensor is one of its own, as if made of the buffer's pointer anew, whatever mode an earlier call ran
in (the buffer a CPU tensor here)."""
import pytest

torch = pytest.importorskip("torch")

from hush_b200 import hush  # noqa: E402


@pytest.fixture
def views(monkeypatch):
    memory = torch.arange(24.0).reshape(2, 3, 4).half()
    monkeypatch.setattr(hush, "device_view", lambda ptr, h, w: torch.from_numpy(memory.numpy()))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    v = hush.OutputViews()
    return lambda: v.get(64, 2, 3)


def test_a_call_under_inference_mode_leaves_later_outputs_alone(views):
    with torch.inference_mode():
        first = views()
        assert first.is_inference()
    out = views()
    assert not out.is_inference()
    x = torch.ones(2, 3, 4, requires_grad=True)
    (x * out).sum().backward()
    assert torch.equal(x.grad, out.float())
    with torch.inference_mode():
        assert views().is_inference()
    assert not views().is_inference()


def test_an_output_has_a_version_counter_of_its_own(views):
    a, b = views(), views()
    x = torch.ones(2, 3, 4, requires_grad=True)
    y = (x * a).sum()
    b.add_(0)
    assert a._version == 0 and b._version == 1 and views()._version == 0
    y.backward()
    assert a.data_ptr() == b.data_ptr() and a is not b and not a._is_view()
