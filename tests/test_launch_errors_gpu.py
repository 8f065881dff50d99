"""A launch that the runtime refuses (an image of more rows of 8 texels than a grid has, 65535) is that call's error alone: the next
calls, of the same class or another, go through.
The tallest image whose rows of 8 texels a grid holds is not refused by any pass."""
import pytest

from hush_b200 import SVGF, Hush, Post, scene
from hush_b200.hush import HushError

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TALL = 600000


def _images(w, h):
    f = {k: torch.ones((h, w, 4), dtype=torch.float16, device="cuda") for k in scene.NAMES}
    return dict(f, prevNormalDepth=f["normalDepth"], prevMotion=f["motion"])


@pytest.mark.parametrize("refused", ["svgf", "post"])
def test_a_refused_launch_is_not_reported_twice(refused):
    f, tall = _images(40, 24), _images(1, TALL)
    calls = {"svgf": SVGF(0, 40, 24).encode, "hush": Hush(0, {"width": 40, "height": 24}).denoise}
    post = Post(0, "rgba8unorm")
    for other in ("svgf", "hush", "post"):
        with pytest.raises(HushError):
            if refused == "svgf":
                SVGF(0, 1, TALL).encode(tall)
            else:
                Post(0, "rgba8unorm").encode(tall["radiance"], tall["radiance"])
        out = post.encode(f["radiance"], f["radiance"]) if other == "post" else calls[other](f)
        torch.cuda.synchronize()
        assert tuple(out.shape) == (24, 40, 4)


def test_the_tallest_image_of_a_grid_is_filtered():
    h = 8 * 65535
    f = _images(1, h)
    f["normalDepth"][..., :2] = 0.0
    svgf = SVGF(0, 1, h, {"iterations": 5})  # (holds the image that encode() returns a view of)
    out = svgf.encode(f)
    assert tuple(out.shape) == (h, 1, 4) and (out[..., :3] == out[0, 0, :3]).all() and abs(out[0, 0, 0].item() - 2.0) < 4e-3
