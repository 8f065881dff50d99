"""The fused frame at the edges of its tiles against the per-pass schedule (the general path: one kernel per reference
pass, 16 x 8 tiles, itself held to the oracle pass by pass): single pixels, one texel either side of FINE_FINAL's
32 x 16 and stage 0's 64 x 16 tiles, even and odd widths (16-byte and 8-byte copies), inputs with padded rows, and frames of
more tiles than a grid of two CTAs per SM holds (296 on 148 SMs), which a CTA walks.

Bound: the parity bound of 2e-3 per value (util.mismatch) on all but SEQ_FRAC of the values, as the sequence tests hold; on
images of a few pixels at most one pixel (3 values) may be beyond it. (Against the oracle the per-pass schedule itself is
beyond that on some of these small images, where a few ill-conditioned TAA pixels weigh more.)"""
import numpy as np
import pytest

from hush_b200 import Hush, scene
from hush_b200.scene import NAMES
from tests.util import mismatch, to_f32

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SEQ_FRAC = 5e-3

CASES = [  # width, height, padded columns, mlp
    (1, 1, 0, "fp32"), (3, 2, 1, "fp32"), (31, 15, 0, "fp32"), (32, 16, 0, "bf16"), (33, 17, 0, "fp32"),
    (34, 18, 2, "fp32"), (36, 33, 0, "f16"), (63, 31, 3, "fp32"), (66, 34, 0, "fp32"), (130, 66, 1, "bf16"),
    (997, 301, 0, "fp32"), (1024, 300, 4, "fp32"),
]


def _padded(a, pad):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    if not pad:
        return t
    buf = torch.full((t.shape[0], t.shape[1] + pad, 4), float("nan"), dtype=t.dtype, device="cuda")
    buf[:, :t.shape[1]] = t
    return buf[:, :t.shape[1]]


@pytest.mark.parametrize("w,h,pad,mlp", CASES)
@pytest.mark.parametrize("graph", [False, True])
def test_frame_tile_edges(w, h, pad, mlp, graph):
    cfg = scene.SceneConfig(w, h, 4, n_moving=2, pan_min=0.5, pan_max=2.0, firefly_scale=10.0, seed=w + h)
    o = Hush(0, {"width": w, "height": h, "schedule": "passes"})
    g = Hush(0, {"width": w, "height": h, "mlp": mlp, "graph": graph})
    for i in range(cfg.frames):
        f = scene.frame_host(cfg, i)
        d = {k: _padded(f[k], pad) for k in NAMES}
        ref = to_f32(o.denoise(d))
        got = to_f32(g.denoise(d))
        frac, worst, _ = mismatch(got, ref)
        assert frac * ref.size <= max(3.0, SEQ_FRAC * ref.size), (i, frac, worst)
    assert g.kernel_status() == 0
