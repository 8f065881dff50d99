"""A timed frame runs the kernels of a replayed one, so that its stage times are of what the replay runs; and the frames after it
are those of an instance that was never timed."""
import pytest

from hush_b200 import Hush, scene

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W, H = 70, 42


class Timer:
    def record(self, timings):
        self.timings = timings


def _kernels(call):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return sorted(e.name for e in p.events() if "hush::" in e.name)


@pytest.mark.parametrize("mlp", ["fp32", "bf16"])
def test_a_timed_frame_runs_the_replayed_kernels(mlp):
    fr = [scene.frame_device(scene.SceneConfig(W, H, 2, seed=3), t) for t in range(2)]
    timed, replayed = Hush(0, {"width": W, "height": H, "mlp": mlp}), Hush(0, {"width": W, "height": H, "mlp": mlp, "graph": True})
    for i in range(4):  # both parities of the instance's images captured
        replayed.denoise(fr[i & 1])
        timed.denoise(fr[i & 1], timer=Timer())
    want = _kernels(lambda: replayed.denoise(fr[0]))
    assert len(want) == 8 and _kernels(lambda: timed.denoise(fr[0], timer=Timer())) == want


def test_frames_after_a_timed_one():
    fr = [scene.frame_device(scene.SceneConfig(W, H, 6, seed=3), t) for t in range(6)]
    a, b = Hush(0, {"width": W, "height": H}), Hush(0, {"width": W, "height": H})
    for t in range(6):
        timer = Timer() if t in (1, 4) else None
        assert torch.equal(a.denoise(fr[t], timer=timer), b.denoise(fr[t]))
        assert timer is None or len(timer.timings) > 0
