"""Which particles of a learned step take the network: those of at most 48
neighbours, whatever form of row they are counted from."""
import numpy as np
import pytest

from sph_gb300 import LearnedModel, Simulation, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long_masks", [False, True])
@pytest.mark.parametrize("lattice,side", [(0.25, 60), (0.2, 50), (0.14, 40), (0.1, 36)])
def test_particles_of_few_neighbours_take_the_network(cuda_lib, lattice, side, long_masks):
    """A block, and lines of particles beside it that reach into its edge:
    counts on both sides of 48 from rows of up to 64, 128 and more candidates."""
    rng = np.random.default_rng(side)
    n = side * side
    i = np.arange(n)
    x, y = (3.05 + lattice * (q + rng.uniform(-0.2, 0.2, n)) for q in (i % side, i // side))
    line = np.arange(3.3, 3.0 + lattice * side, 0.3)
    x = np.concatenate([x, line, line + 0.1])
    y = np.concatenate([y, 3.0 + lattice * side + np.repeat([0.55, 0.75], len(line))])
    n = len(x)
    size = int(np.ceil(lattice * side)) + 7
    p = scenes.Params(g=0.0, sigma=0.0, beta=0.0)
    p.node_end_x = float(size)
    sc = scenes.Scene(name="edges", x=x.astype(np.float32), y=y.astype(np.float32), vx=np.zeros(n, np.float32),
                      vy=np.zeros(n, np.float32), box=(0.0, float(size), 0.0, float(size)), params=p,
                      spacing=1.0, size_x=size, size_y=size, max_bucket=200)
    with Simulation.from_scene(sc) as s, LearnedModel(0, seed=2) as m:
        s.set_long_row_masks(long_masks)
        _, count = s.learned_features()
        assert count.max() > LearnedModel.MAX_NEIGHBORS >= np.partition(count, 5)[5] >= 0
        s.set_learned(m, 1e9)  # no error is too large
        s.step(None, 1)
        few = int(((count >= 0) & (count <= LearnedModel.MAX_NEIGHBORS)).sum())
        assert s.learned_counts() == (few, n - few)
