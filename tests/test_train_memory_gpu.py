"""What a trainer takes of the device's memory, and which form of the window's records it takes when."""
import gc

import pytest

from hush_b200 import Hush
from hush_b200.train import TrainConfig, Trainer, xavier_init

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _free():
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_a_trainer_holds_what_its_frame_needs():
    """Per pixel: twelve images of 16 bytes, the TAA adjoint's coefficients and the recombination's values of 48 each, at half
    resolution parameters, levels, their gradients (48 + 2 x 24, 6 x 16, 8 bytes) and the MLP's partial sums: 345 bytes."""
    size = 2048
    den = Hush(0, {"width": size, "height": size, "schedule": "passes"})
    before = _free()
    tr = Trainer(den, xavier_init(TrainConfig().init_seed))
    assert before - _free() <= 348 * size * size
    tr.destroy()
