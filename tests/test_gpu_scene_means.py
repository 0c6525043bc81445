"""Per-scene diagnostics against the downloaded state, with scenes that one
block sums and scenes that are cut into pieces."""
import numpy as np
import pytest

from sph_gb300 import Ensemble, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2048), (2047, 2049, 3), (1, 70000, 4097, 2048), (300,) * 400])
def test_means_of_each_scene(cuda_lib, sizes):
    scs = [scenes.ensemble_scene(40 + k, f"m{k}", (n, n)) for k, n in enumerate(sizes)]
    e = Ensemble(scs, 100, 400)
    e.upload_scenes()
    e.step(None, 3)
    got, st = e.scene_diagnostics(), e.download()
    for s in range(len(sizes)):
        k = e.scene_slice(s)
        v = [st[f][k].astype(np.float64) for f in ("density", "density_near", "v_x", "v_y")]
        want = np.array([v[0].mean(), v[1].mean(), (0.5 * (v[2] ** 2 + v[3] ** 2)).mean()])
        # sums of up to 70,000 terms of one sign in 64 bits
        assert np.all(np.abs(got[s] - want) <= 1e-12 * np.abs(want)), (s, got[s], want)
    e.close()
