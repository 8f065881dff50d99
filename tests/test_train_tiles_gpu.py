"""The fused training frame at the edges of its 16 x 8 tiles against the chain of per-pass kernels: the frame keeps the
recombination's forward values for its adjoint, forms loss and TAA adjoint in the TAA kernel and gathers dL/dX
directly, where the per-pass pairs recompute from each pass's inputs. Sizes: one pixel, odd, one pixel either side of a
tile, and images narrower than the recombination's footprint.

Bound: the forward runs the same arithmetic, so loss to 1e-12 (its FP64 sum is split differently) and TAA output to FP32
rounding (1e-6 of max); the adjoints differ in the order of atomic additions and in where a quotient is formed, 1e-5 of the
largest as the existing chain test holds."""
import numpy as np
import pytest

from tests.test_passes_gpu import ORDER, Frame

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (7, 5), (16, 8), (17, 9), (15, 23), (33, 31), (66, 50)])
def test_fused_frame_matches_the_pass_chain_at_tile_edges(w, h):
    fr = Frame(W=w, H=h, seed=w + h)
    tr = fr.tr
    loss_chain = tr.buffer("LOSS").cpu().numpy().copy()
    out_chain = tr.buffer("OUT").cpu().numpy().copy()
    tr.zero_adjoints()
    tr.zero_grad()
    for p in reversed(ORDER):
        tr.bwd(p)
    torch.cuda.synchronize()
    g_chain, (_, d_chain) = tr.grad(), tr.par()
    tr.zero_grad()
    loss = tr.frame(fr.inputs, fr.cleans[2], fr.cleans[1], fr.lam, backward=True)
    g_frame, (_, d_frame) = tr.grad(), tr.par()
    out = tr.buffer("OUT").cpu().numpy()
    assert abs(loss - float(loss_chain[0])) <= 1e-12 * max(1.0, abs(loss))
    assert np.abs(out - out_chain).max() <= 1e-6 * np.abs(out_chain).max()
    assert np.isfinite(g_frame).all() and np.isfinite(d_frame).all()
    assert np.abs(g_chain - g_frame).max() <= 1e-5 * np.abs(g_chain).max()
    assert np.abs(d_chain - d_frame).max() <= 1e-5 * np.abs(d_chain).max()


def test_window_gradient_with_and_without_saved_forwards():
    """A window's records keep the forwards' values while they fit 2 GiB; a trainer that has run a longer window keeps
    the small records and runs the forwards again in the reverse sweep. Both give the window's gradient (the same
    kernels on the same values; FP32 atomics in another order: 1e-5 of the largest, loss to 1e-12), in both MLP forms."""
    from hush_b200 import Hush
    from hush_b200.train import TrainConfig, Trainer, window, xavier_init

    size, long_window = 512, 46  # 46 frames x 48 MB > 2 GiB
    win = window(TrainConfig(size=size, frames=3), 7)
    for mlp in ("fp32", "bf16"):
        got = []
        for lean in (True, False):
            den = Hush(0, {"width": size, "height": size, "schedule": "passes"})
            tr = Trainer(den, xavier_init(2))
            tr.set_mlp(mlp)
            if lean:
                tr.window_bptt([win[i % 3] for i in range(long_window)], 0.5)
            tr.zero_grad()
            tr.loss_sum()
            tr.window_bptt(win, 0.5)
            got.append((tr.loss_sum(), tr.grad()))
            tr.destroy()
            den.destroy()
        (la, ga), (lb, gb) = got
        assert abs(la - lb) <= 1e-12 * abs(lb)
        assert np.abs(ga - gb).max() <= 1e-5 * np.abs(gb).max()
