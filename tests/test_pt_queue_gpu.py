"""The path tracer with an environment map on images whose CTAs hold more pixels than threads (over 148 x 9 x 96 = 128 k), so that a
thread goes on to other pixels after finished paths: ragged edges, G-buffer and two samples accumulated, and one of 195 tiles a
CTA, against the oracle with the bounds of the edge tests."""
import pytest

from tests import test_pt_tiles_gpu as edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,mode,spp,tau,lights", [(523, 331, 0, 1, 0.0, 2), (523, 331, 1, 2, 0.5, 3), (1031, 701, 0, 1, 0.5, 1),
                                                          (3840, 2161, 0, 1, 0.5, 1)])
def test_threads_take_further_pixels(w, h, mode, spp, tau, lights):
    edges.test_path_tracer_edges(w, h, mode, spp, 3, tau, lights, True)
