"""What a trainer takes of the device's memory, and which form of the window's records it takes when."""
import gc

import numpy as np
import pytest

from hush_b200 import Hush
from hush_b200.train import TrainConfig, Trainer, window, window_scene, xavier_init

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _free():
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_a_trainer_holds_what_its_frame_needs():
    """Per pixel: twelve images of 16 bytes, the TAA adjoint's coefficients and the recombination's values of 48 each, at half
    resolution parameters, levels, their gradients (48 + 2 x 24, 6 x 16, 8 bytes) and the MLP's partial sums: 345 bytes."""
    size = 2048
    den = Hush(0, {"width": size, "height": size, "schedule": "passes"})
    before = _free()
    tr = Trainer(den, xavier_init(TrainConfig().init_seed))
    assert before - _free() <= 348 * size * size
    tr.destroy()


def _taa_launches(call):
    """Launches of the twin's TAA kernel: one per frame forward, so one more per frame whose forward is run again."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return sum("k_taa(" in e.name for e in p.events())


def _gradient(tr, call):
    tr.zero_grad()
    tr.loss_sum()
    call()
    return tr.loss_sum(), tr.grad()


def test_the_form_of_a_window_s_records():
    """A window's forwards are kept whatever windows the trainer has run before, unless that would take more than half of the
    free memory, and with eight lanes while each lane's stay under an eighth of 2 GiB. Both forms give the gradient (1e-5 of the
    largest: FP32 atomics in another order)."""
    size, frames = 512, 4  # 185 MB of records with the forwards, 81 MB without
    cfg = TrainConfig(size=size, frames=frames)
    win = window(cfg, 7)
    den = Hush(0, {"width": size, "height": size, "schedule": "passes"})
    tr = Trainer(den, xavier_init(2))
    short = lambda: tr.window_bptt(win, 0.5)  # noqa: E731
    seeds = list(range(9, 17))
    tr.windows_bptt(window_scene(cfg), seeds, frames, 0.5)  # the lanes and their memory
    tr.destroy()
    tr = Trainer(den, xavier_init(2))
    hold = torch.empty(_free() - (340 << 20), dtype=torch.uint8, device="cuda")
    lean_launches, lean = _taa_launches(short), _gradient(tr, short)
    del hold
    _free()
    assert lean_launches == 2 * frames
    assert _taa_launches(short) == frames
    assert _taa_launches(lambda: tr.window_bptt([win[i % frames] for i in range(50)], 0.5)) == 100  # over 2 GiB
    assert _taa_launches(short) == frames
    loss, grad = _gradient(tr, short)
    assert abs(loss - lean[0]) <= 1e-12 * abs(loss)
    assert np.abs(grad - lean[1]).max() <= 1e-5 * np.abs(grad).max()
    lanes = lambda f, c: _taa_launches(lambda: tr.windows_bptt(window_scene(c), seeds, f, 0.5))  # noqa: E731
    assert lanes(frames, cfg) == 8 * frames
    long = TrainConfig(size=size, frames=8)  # 370 MB a lane
    assert lanes(8, long) == 2 * 8 * 8
    tr.destroy()
