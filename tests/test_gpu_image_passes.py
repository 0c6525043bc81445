"""The liquid image at the particle counts where the splat's passes change:
points of few places against the CPU restatement (more than 255 copies of a
point fill every texel it reaches, so that many stand for all), and any points
in two orders, which sample others of them."""
import numpy as np
import pytest

from oracle import liquid_image as li
from sph_gb300 import render_liquid

pytestmark = pytest.mark.gpu

SIZES = [(65536, 160, 120), (300001, 33, 20), (400000, 161, 90), (400001, 320, 40), (1048577, 64, 48)]


@pytest.mark.parametrize("n,W,H", SIZES)
def test_crowded_and_thin_places(cuda_lib, n, W, H):
    rng = np.random.default_rng(n)
    thin = rng.integers(-32767, 32768, (1500, 2))
    crowd = np.concatenate([rng.integers(-20000, 20000, (6, 2)), [[-32767, -32767], [32767, 32767]]])
    pts = np.concatenate([thin, crowd[np.arange(n - len(thin)) % len(crowd)]]).astype(np.int16)
    rgb, a = render_liquid(pts[rng.permutation(n)], W, H)
    ref_rgb, ref_a, _ = li.render(np.concatenate([thin, np.repeat(crowd, 255, 0)]).astype(np.int16), W, H)
    # as in test_gpu_render: the splat is exact, the blur within one level
    d = np.abs(a.astype(int) - ref_a.astype(int))
    assert d.max() <= 1 and (d == 0).mean() > 0.995, (d.max(), (d == 0).mean())
    assert (np.abs(rgb.astype(int) - ref_rgb.astype(int)).max(axis=-1) <= 2).mean() > 0.99


@pytest.mark.parametrize("n,W,H", SIZES + [(200000, 640, 360)])
def test_any_order_gives_the_same_image(cuda_lib, n, W, H):
    rng = np.random.default_rng(n + 1)
    pts = np.concatenate([rng.normal(0.0, 5000.0, (n // 2, 2)).clip(-32767, 32767),
                          rng.integers(-32767, 32768, (n - n // 2, 2))]).astype(np.int16)
    one, two = (render_liquid(p, W, H) for p in (pts, pts[rng.permutation(n)]))
    assert np.array_equal(one[0], two[0]) and np.array_equal(one[1], two[1])
