"""The display post on images whose passes take more CTAs than one wave holds and whose levels change between the exact 2 : 1 form
and the general one: the target and every level bit for bit as the general forms alone gave them (SHA-256 of their bytes, printed
by python tests/test_post_waves_gpu.py). At these sizes the oracle's sample positions differ by enough of a texel that a few
pixels beside a firefly are beyond the bound of the small images, in either form."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DIGESTS = {
    (1366, 768): "35558a3cac0663fb48173a81ac42ad7565df9dfbd6741071e4e7543a8b273842",
    (1283, 719): "9205350acff3ffe1ba4f0fdfcf9e587741036fadc87f37bd8e7a30776688ba16",
    (1920, 1081): "270f947c8bf9e649ae1bf8a17b9ec0cbd524f31ab65ade97a618c64f17c04874",
    (2050, 1154): "24999271e3ed92d5ff9c3e15924304f89dd51118b68b15c6ff06ff564ee696ca",
}


def digest(w, h):
    from hush_b200 import Post

    rng = np.random.default_rng(w)
    a, b = (torch.from_numpy((rng.random((h, w, 4)) ** 6 * 40).astype(np.float16)).cuda() for _ in range(2))
    sha = hashlib.sha256()
    for fmt in ("rgba32float", "rgba8unorm"):
        post = Post(0, fmt)
        out = post.encode(a, b, split=0.45, exposure=1.2)
        for image in [out] + [post.buffer(i) for i in range(7)]:
            sha.update(image.cpu().numpy().tobytes())
    return sha.hexdigest()


@pytest.mark.parametrize("w,h", sorted(DIGESTS))
def test_large_images_with_odd_levels(w, h):
    assert digest(w, h) == DIGESTS[w, h]


if __name__ == "__main__":
    for size in [(1366, 768), (1283, 719), (1920, 1081), (2050, 1154)]:
        print(f"    {size}: \"{digest(*size)}\",")
