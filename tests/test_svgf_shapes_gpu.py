"""SVGF at the edges of its tiles against the oracle: single pixels, one texel either side of the 64-column and
8-lattice-row tiles of the a-trous kernel, images smaller than the widest footprint (64 texels each side at step 16), every
iteration count, a normal exponent other than the default, TAA on and off, and inputs with padded rows.

Bound: the parity bound of 2e-3 per value (util.mismatch) on all but SEQ_FRAC of the values, as the sequence test
holds; on images of a few pixels at most one pixel (3 values) may be beyond it, since a history length that rounds to
the other side of SVGF's threshold of 4 replaces that pixel's variance."""
import numpy as np
import pytest

import oracle
from hush_b200 import SVGF, scene
from tests.util import mismatch, to_f32

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SEQ_FRAC = 5e-3

CASES = [  # width, height, iterations, sigmaN, taa, padded columns
    (1, 1, 5, 128.0, True, 0), (5, 3, 5, 128.0, True, 3), (63, 9, 3, 128.0, True, 0), (64, 8, 1, 128.0, False, 0),
    (65, 17, 4, 128.0, True, 5), (96, 129, 5, 128.0, True, 0), (131, 137, 5, 48.0, True, 1), (33, 260, 2, 0.0, False, 0),
    (257, 31, 5, 128.0, False, 0),
]


def _padded(a, pad):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    if not pad:
        return t
    buf = torch.full((t.shape[0], t.shape[1] + pad, 4), float("nan"), dtype=t.dtype, device="cuda")
    buf[:, :t.shape[1]] = t
    return buf[:, :t.shape[1]]


@pytest.mark.parametrize("w,h,iterations,sigma_n,taa,pad", CASES)
def test_svgf_tile_edges(w, h, iterations, sigma_n, taa, pad):
    cfg = scene.SceneConfig(w, h, 4, n_moving=2, pan_min=0.5, pan_max=2.0, seed=w + h)
    opts = {"iterations": iterations, "sigmaN": sigma_n, "taa": int(taa)}
    o, s, prev = oracle.OracleSVGF(w, h, opts), SVGF(0, w, h, opts), None
    for i in range(cfg.frames):
        f = scene.frame_host(cfg, i)
        g = dict(f, prevNormalDepth=(prev or f)["normalDepth"], prevMotion=(prev or f)["motion"])
        ref = o.encode(g).astype(np.float32)
        got = to_f32(s.encode({k: _padded(v, pad) for k, v in g.items()}))
        frac, worst, _ = mismatch(got, ref)
        assert frac * ref.size <= max(3.0, SEQ_FRAC * ref.size), (i, frac, worst)
        prev = f
