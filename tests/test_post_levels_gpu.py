"""The display post where its passes take the forms for exact 2 : 1 level sizes, and where the levels change from one form to
the other: images of one bloom texel, sizes even on some levels only, all levels, at the edges of a 32 x 8 tile of level
texels; a target with padded rows at an address that is only 4-byte aligned; and the chain of passes replayed from a CUDA
graph. Against the oracle with the bounds of the post's other tests (a 1-ulp flip of the f16 stores; one 8-bit step)."""
import numpy as np
import pytest

import oracle
from hush_b200 import Post
from tests.test_post_gpu import _check, _hdr

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(2, 2), (2, 6), (4, 2), (3, 2), (64, 16), (66, 18), (62, 14), (128, 64), (130, 34), (256, 130), (192, 96)]


@pytest.mark.parametrize("w,h", SIZES)
def test_levels_match_the_oracle(w, h):
    left, right = _hdr(h, w, w), _hdr(h, w, h + 1)
    a, b = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    want = oracle.post(left, right, split=0.45, exposure=1.2)
    post = Post(0, "rgba32float")
    _check(post, want, post.encode(a, b, split=0.45, exposure=1.2).cpu().numpy(), "rgba32float")
    post8 = Post(0, "rgba8unorm")
    buf = torch.zeros((h, w + 3, 4), dtype=torch.uint8, device="cuda")
    got = post8.encode(a, b, split=0.45, exposure=1.2, target=buf[:, 1:w + 1])
    torch.cuda.synchronize()
    _check(post8, want, got.cpu().numpy(), "rgba8unorm")
    assert (buf[:, 0] == 0).all() and (buf[:, w + 1:] == 0).all()


def test_passes_replay_from_a_graph():
    h, w = 90, 160
    a, b = torch.from_numpy(_hdr(h, w, 1)).cuda(), torch.from_numpy(_hdr(h, w, 2)).cuda()
    post = Post(0, "rgba8unorm")
    target = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    want = post.encode(a, b, split=0.3).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        post.encode(a, b, split=0.3, target=target)
    for _ in range(3):
        target.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(target, want)
