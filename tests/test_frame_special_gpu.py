"""The fused frame on G-buffers with values that are not finite, where only a few pixels hold them: the per-pass schedule's frame (the
general path) within the parity bound on all but SEQ_FRAC of the values."""
import os
import sys

import numpy as np
import pytest

from hush_b200 import Hush, scene
from tests.util import mismatch, to_f32

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SEQ_FRAC = 5e-3
W, H = 161, 91


def frames(name, channel, value, n=4):
    rng = np.random.default_rng(7)
    cfg = scene.SceneConfig(W, H, n, n_moving=2, pan_min=0.5, pan_max=2.0, seed=5)
    for t in range(n):
        f = {k: v.float().cpu().numpy() for k, v in scene.frame_device(cfg, t).items()}
        f[name] = f[name].copy()
        f[name].reshape(-1, 4)[rng.integers(0, W * H, 20), channel] = value
        yield {k: torch.from_numpy(v.astype(np.float16)).cuda() for k, v in f.items()}


@pytest.mark.parametrize("mlp", ["fp32", "bf16"])
@pytest.mark.parametrize("name,channel,value", [
    ("normalDepth", 0, np.nan), ("normalDepth", 1, np.nan), ("normalDepth", 2, np.nan), ("normalDepth", 1, np.inf),
    ("normalDepth", 0, 0.0), ("normalDepth", 3, np.inf), ("material", 3, np.inf)])
def test_frames_match_the_pass_schedule(name, channel, value, mlp):
    a, b = Hush(0, {"width": W, "height": H, "schedule": "passes"}), Hush(0, {"width": W, "height": H, "mlp": mlp})
    for i, f in enumerate(frames(name, channel, value)):
        ref, got = to_f32(a.denoise(f)), to_f32(b.denoise(f))
        assert (np.isfinite(ref) == np.isfinite(got)).all()
        frac, worst, _ = mismatch(np.where(np.isfinite(ref), got, 0.0), np.where(np.isfinite(ref), ref, 0.0))
        assert frac <= SEQ_FRAC, (i, frac, worst)


GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "nan_depth_frames.npz")


def nan_depth_frames(mlp):
    d = Hush(0, {"width": W, "height": H, "mlp": mlp})
    out = [d.denoise(f).cpu().numpy() for f in frames("normalDepth", 3, np.nan)]
    return np.stack([out[0], out[3]])


@pytest.mark.parametrize("mlp", ["fp32", "bf16"])
def test_pixels_of_nan_depth(mlp):
    """A NaN depth is no sky, but no valid neighbour either (there the fused frame has always differed from the passes): the
    frames stored before stage 0 and FINE_FINAL were rewritten (python -m tests.test_frame_special_gpu FILE)."""
    want, got = np.load(GOLDEN)[mlp].astype(np.float32), nan_depth_frames(mlp).astype(np.float32)
    for a, b in zip(want, got):
        frac, worst, _ = mismatch(b, a)
        assert frac <= SEQ_FRAC, (frac, worst)


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{m: nan_depth_frames(m) for m in ("fp32", "bf16")})
