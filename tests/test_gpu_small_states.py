"""The forms that a small handle's gathers take by its size and its fullest
cell -- lanes or one thread a particle, rows of up to 32 or 64 candidates
marked -- against the form of large handles: a scene alone and the same scene
in an ensemble of more than 300,000 particles, bit for bit."""
import functools

import numpy as np
import pytest

from conftest import bits_equal
from sph_gb300 import Ensemble, Simulation, scenes
from test_gpu_lanes import ONE_THREAD, block

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "v_x", "v_y", "density", "density_near")
# particles and lattice spacing: the fullest cell below and above the line of
# each gather, rows of 32, 33 to 64 and more candidates, in one warp too
CASES = [(700, 0.95), (5000, 0.5), (5001, 0.3), (11000, 0.34), (14000, 0.25), (14001, 0.25), (20000, 0.3),
         (40000, 0.22), (40000, 0.5), (40001, 0.24), (60001, 0.16)]


def scene(n, lattice):
    sc = block(n, lattice, 1.0)
    # a denser corner: warps of short and long rows, and more coincident pairs
    k = n // 20
    sc.x[:k] *= np.float32(0.6)
    sc.y[:k] *= np.float32(0.6)
    sc.x[50:53], sc.y[50:53] = sc.x[49], sc.y[49]
    return sc


@functools.lru_cache(maxsize=None)
def large_handle(max_bucket):
    scs = [scene(n, a) for n, a in CASES]
    scs.append(block(310000, 0.5, 1.0))
    e = Ensemble(scs, max_bucket, 400)
    e.upload_scenes()
    e.step(None, 5)
    out = e.download()
    return [{f: out[f][e.scene_slice(s)].copy() for f in FIELDS} for s in range(len(CASES))]


@pytest.mark.parametrize("max_bucket", [100, 6])
@pytest.mark.parametrize("long_masks", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_small_handles_equal_large_ones(cuda_lib, case, long_masks, max_bucket):
    n, lattice = CASES[case]
    sc = scene(n, lattice)
    ref = large_handle(max_bucket)[case]
    cfg = dict(sc.config(), max_bucket=max_bucket)
    with Simulation(sc.params.as_dict(), cfg, n) as s:
        s.set_long_row_masks(long_masks)
        s.upload(sc.x, sc.y, sc.vx, sc.vy)
        s.step(None, 5)
        got, fullest = s.download(), s.counters()["max_cell_occupancy"]
    if max_bucket < 100 and fullest <= max_bucket:
        pytest.skip("no overflowing bucket here; in the ensemble there is")
    for f in FIELDS:
        assert bits_equal(got[f], ref[f]), f


@pytest.mark.parametrize("name", ["sigma", "beta", "k", "k_near", "k_spring", "g", "rest_density"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), -1e38])
def test_tunables_without_bounds(cuda_lib, name, value):
    """An infinity or a NaN among the tunables reaches the same particles,
    whether lanes share them or not."""
    sc = block(3000, 0.4, 0.7)
    rng = np.random.default_rng(4)
    v = rng.uniform(-1.0, 1.0, (2, sc.n)).astype(np.float32)
    P = dict(sc.params.as_dict(), **{name: value})
    out = []
    for shapes in (None, ONE_THREAD):
        with Simulation.from_scene(sc) as s:
            if shapes:
                s.set_launch_shapes(shapes)
            s.upload(sc.x, sc.y, *v)
            s.rebuild_neighbors()
            s.step(P, 1)
            out.append(s.download())
    for f in FIELDS:
        assert np.array_equal(out[0][f], out[1][f], equal_nan=True), f
