"""SVGF's passes, launched as programmatic successors, replayed from a CUDA graph: the frame is the one of the same calls made
directly, bit for bit."""
import pytest

from hush_b200 import SVGF, scene

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h,options", [(70, 41, {}), (33, 20, {"iterations": 3, "taa": 0, "sigmaN": 64.0})])
def test_passes_replay_from_a_graph(w, h, options):
    fr = [scene.frame_device(scene.SceneConfig(w, h, 2, n_moving=1, seed=5), t) for t in range(2)]
    ins = [dict(f, prevNormalDepth=fr[0]["normalDepth"], prevMotion=fr[0]["motion"]) for f in fr]
    a, b = SVGF(0, w, h, options), SVGF(0, w, h, options)
    a.encode(ins[0])
    want = a.encode(ins[1]).clone()
    b.encode(ins[0])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = b.encode(ins[1])
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
