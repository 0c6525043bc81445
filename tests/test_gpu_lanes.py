"""The gathers with several lanes per particle (small handles) against the
one-thread kernels, which a launch shape other than the default selects:
every result bit for bit the same, at the particle counts where the number
of lanes changes and in cells sparse, dense, and fuller than a hit mask, two
hit masks and a bucket hold."""
import numpy as np
import pytest

from conftest import bits_equal
from sph_gb300 import LearnedModel, Simulation, scenes

pytestmark = pytest.mark.gpu

ONE_THREAD = [128, 0, 128, 0, 128, 0]
FIELDS = ("x", "y", "v_x", "v_y", "density", "density_near")


def block(n, lattice, h):
    side = max(1, int(np.sqrt(n)))
    size = float(np.ceil(lattice * side * 1.3) + 4) * h
    p = scenes.Params(smoothing_radius=h, mover_type=scenes.SPHERE_MOVER, mover_width=3.0 * h,
                      mover_center_x=size / 3, mover_center_y=h)
    sc = scenes.dam_break(n, side, size, size, seed=n, name="block", params=p, lattice=lattice * h,
                          jitter=0.05 * h, x0=0.2 * h, y0=0.2 * h)
    if n > 40:  # coincident and nearly coincident pairs
        sc.x[7], sc.y[7] = sc.x[6], sc.y[6]
        sc.x[31], sc.y[31] = sc.x[30], sc.y[30] + np.float32(5e-7)
    return sc


@pytest.mark.parametrize("long_masks", [False, True])
@pytest.mark.parametrize("n,lattice,h", [
    (1, 0.5, 1.0), (2, 0.01, 1.0), (33, 0.5, 1.0), (1500, 0.5, 0.7), (5000, 0.2, 1.0), (5000, 0.14, 1.0),
    (4003, 0.09, 1.0), (5001, 0.2, 1.0), (14000, 0.14, 0.7), (14001, 0.2, 1.0), (30000, 0.5, 1.0),
    (30001, 0.14, 1.0), (40000, 0.45, 1.0), (20000, 0.09, 1.0), (40001, 0.45, 1.0)])
def test_lanes_give_the_one_thread_results(cuda_lib, n, lattice, h, long_masks):
    sc = block(n, lattice, h)
    P = sc.params.as_dict()
    out = []
    for shapes in (None, ONE_THREAD):
        with Simulation.from_scene(sc) as s:
            if shapes:
                s.set_launch_shapes(shapes)
            s.set_long_row_masks(long_masks)
            s.step(P, 3)
            a = s.download()
            s.step(P, 4)
            out.append((a, s.download(), s.counters()))
    assert out[0][2] == out[1][2]
    for k in (0, 1):
        for f in FIELDS:
            assert bits_equal(out[0][k][f], out[1][k][f]), (k, f)


@pytest.mark.parametrize("n", [1, 4000, 16384, 50000, 320000])
@pytest.mark.parametrize("lattice", [0.5, 0.14])
def test_learned_fallback_by_lanes_is_the_plain_step(cuda_lib, n, lattice):
    """Every particle on the learned step's fallback list, from lists of 32
    and 4 lanes a particle to more than the pass has threads: the plain
    step's bits, coincident pairs included."""
    sc = block(n, lattice, 1.0)
    P = sc.params.as_dict()
    with Simulation.from_scene(sc) as plain, Simulation.from_scene(sc) as learned, LearnedModel(0, seed=1) as m:
        plain.set_launch_shapes(ONE_THREAD)
        learned.set_learned(m, threshold=-1.0)
        for s in (plain, learned):
            s.step(P, 5)
        a, b = plain.download(), learned.download()
        assert learned.learned_counts() == (0, 5 * n)
    for f in FIELDS:
        assert bits_equal(a[f], b[f]), f
