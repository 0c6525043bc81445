"""Calls of several steps (from the eighth call of four steps or more on, four
steps are one graph) against the same steps one at a time, with
changes of the tunables, the launch shapes, the model and the particles in
between."""
import numpy as np
import pytest

from conftest import bits_equal
from sph_gb300 import LearnedModel, Simulation, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3000, 20000])
def test_many_steps_equal_single_steps(cuda_lib, n):
    sc = scenes.config2(n)
    P = sc.params.as_dict()
    Q = dict(P, k=0.2, sigma=0.9)
    out = []
    with LearnedModel(0, seed=3) as model:
        for single in (False, True):
            with Simulation.from_scene(sc) as s:
                def steps(p, k):
                    if single:
                        for _ in range(k):
                            s.step(p, 1)
                    else:
                        s.step(p, k)
                for p, k in [(P, 4)] * 7 + [(P, 4), (P, 4), (Q, 3), (Q, 9), (P, 8)]:
                    steps(p, k)
                s.set_launch_shapes([128, 0, 128, 0, 128, 0])
                for k in [4] * 8 + [5, 6]:
                    steps(P, k)
                s.set_learned(model, -1.0)
                for k in [4] * 8 + [7]:
                    steps(Q, k)
                s.set_learned(None)
                m = max(1, n // 2)  # fewer particles: the graphs are made again
                s.upload(sc.x[:m], sc.y[:m])
                for k in [4] * 9 + [10]:
                    steps(P, k)
                out.append((s.download(), s.counters()))
    assert out[0][1] == out[1][1]
    for f in ("x", "y", "v_x", "v_y", "density", "density_near"):
        assert bits_equal(out[0][0][f], out[1][0][f]), f
