"""The path tracer at the edges of its work distribution, against the oracle: images smaller than a tile, a CTA and the grid,
ragged tiles, one and several samples per pixel, none, no bounce, no light, all light slots with the environment map (the most
shadow rays a vertex can have), one light picked per vertex, and more samples than a path has threads.

Bounds: those of the G-buffer and accumulation tests, 0.5 % of the pixels (at least 2) for the geometry planes and 10 % / 15 %
(at least 2) for the radiance of one / two paths, whose random branches can differ by an ulp."""
import numpy as np
import pytest

from hush_b200 import pt
from tests.test_pt_gpu import _env_image, _gbuf_host, _oracle_scene

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [  # width, height, mode, spp, max_bounces, shadow_tau, lights, environment map
    (1, 1, 0, 1, 3, 0.0, 2, False), (7, 3, 0, 1, 3, 0.0, 2, False), (9, 5, 0, 1, 3, 0.5, 2, True),
    (31, 33, 0, 1, 0, 0.0, 2, False), (33, 17, 0, 1, 3, 0.0, 0, False), (40, 20, 0, 1, 3, 0.0, 8, True),
    (65, 9, 0, 1, 5, 0.5, 8, True), (200, 130, 0, 1, 3, 0.0, 2, False),
    (5, 3, 1, 2, 3, 0.0, 2, False), (33, 18, 1, 2, 3, 0.5, 3, True), (17, 9, 1, 0, 3, 0.0, 2, False),
]


@pytest.mark.parametrize("w,h,mode,spp,bounces,tau,lights,envmap", CASES)
def test_path_tracer_edges(w, h, mode, spp, bounces, tau, lights, envmap):
    sc, env, _ = pt.demo_scene(0, seed=4, n_objects=6)
    have = list(env["lights"])
    e = dict(env, lights=[dict(have[i % len(have)]) for i in range(lights)])
    osc = _oracle_scene(sc)
    if envmap:
        e["map"] = pt.prepare_env_map(_env_image(), sun=True)
        osc.set_env(e["map"].half, e["map"].table)
    p = pt.PathTracer(0, sc, w, h)
    cam = pt.Camera(position=(1.0, 4.0, 13.0), target=(0.0, 0.8, 0.0), fov=50, aspect=w / h)
    p.write_uniforms(camera=cam, frame=2, mode=mode, jitter=pt.JITTER[2], spp=spp, max_bounces=bounces, shadow_tau=tau,
                     env=e)
    p.clear_accum()
    p.encode(0)
    torch.cuda.synchronize()
    want = osc.render(bytes(p._frame), w, h, mode)
    if mode == 0:
        got = [a.astype(np.float32) for a in _gbuf_host(p, 0)]
        want = [a.astype(np.float32) for a in want]
        for k, tol in ((1, 2e-3), (2, 2e-2), (3, 2e-3), (4, 2e-3)):
            d = np.abs(got[k] - want[k]) / np.maximum(1.0, np.abs(want[k]))
            assert (d > tol).any(axis=2).sum() <= max(2, 0.005 * w * h), (pt.GBUF_NAMES[k], d.max())
        got, want, share = got[0], want[0], 0.1
    else:
        got, share = p.accum.cpu().numpy(), 0.15
        assert (got[..., 3] == spp).all()
    assert np.isfinite(got).all()
    r = np.abs(got[..., :3] - want[..., :3]) / np.maximum(0.05, np.abs(want[..., :3]))
    assert (r > 1e-2).any(axis=2).sum() <= max(2, share * w * h)
    p.destroy()
