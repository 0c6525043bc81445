"""Device memory that a model and a handle keep after their largest calls."""
import gc

import numpy as np
import pytest

from sph_gb300 import LearnedModel, Simulation
from test_gpu_training import still_fluid

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_training_gives_large_batches_back(cuda_lib):
    torch = pytest.importorskip("torch")

    def used():
        gc.collect()
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    rows = 262144
    sc = still_fluid(rows + 2500, seed=9)
    with Simulation.from_scene(sc) as s, LearnedModel(rows, seed=2) as m:
        assert m.collect(s) == rows
        m.train(1, 128, 1e-3)
        before = used()
        m.train(1, rows, 1e-3)  # 294 MB of tile images
        # the images of at most 64 MB, the epoch's order and allocator pages
        assert used() - before <= 64 * MB + 4 * rows + 8 * MB
        m.train(1, 4096, 1e-3)  # and is made again
        assert np.isfinite(m.get_params()).all()
