"""The output tensors of Hush.denoise and SVGF.encode: a tensor of its own per call, over the instance's current output image,
of the current size after a resize (also back to a former one)."""
import pytest

from hush_b200 import SVGF, Hush, scene

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _frames(w, h):
    fr = [scene.frame_device(scene.SceneConfig(w, h, 4, seed=w), t) for t in range(4)]
    return [dict(f, prevNormalDepth=f["normalDepth"], prevMotion=f["motion"]) for f in fr]


@pytest.mark.parametrize("make", [lambda w, h: Hush(0, {"width": w, "height": h}), lambda w, h: SVGF(0, w, h)])
def test_outputs_follow_the_instance(make):
    d = make(40, 24)
    for w, h in ((40, 24), (24, 40), (40, 24), (17, 9), (33, 20)):
        d.resize(w, h)
        outs = []
        for f in _frames(w, h):
            o = d.denoise(f)
            assert tuple(o.shape) == (h, w, 4) and o.dtype == torch.float16 and not o.requires_grad
            assert o.data_ptr() == d.output.data_ptr() and torch.equal(o, d.output)
            o.mark = (w, h)  # an attribute of this call's tensor only
            outs.append(o)
        assert len({id(o) for o in outs}) == len(outs)
        assert not hasattr(d.denoise(_frames(w, h)[0]), "mark")
