"""The gathers on stencil rows of given lengths -- around the 32 candidates
that are marked in one piece and the 64 and 128 of the hit masks, the last
row ending the particle array -- against a brute-force FP64 evaluation of
the reference's formulas."""
import numpy as np
import pytest

from sph_gb300 import Simulation, scenes

pytestmark = pytest.mark.gpu


def three_rows(length, h, seed):
    """3 x 3 cells of a wider grid, `length` particles in each row of three."""
    rng = np.random.default_rng(seed)
    x = (1.0 + 3.0 * rng.random(3 * length)) * h
    y = (1.0 + np.repeat(np.arange(3), length) + rng.random(3 * length)) * h
    v = rng.uniform(-2.0, 2.0, (2, 3 * length))
    order = rng.permutation(3 * length)
    f = [np.ascontiguousarray(a[order], np.float32) for a in (x, y, v[0], v[1])]
    p = scenes.Params(smoothing_radius=h, node_end_x=6.0 * h)
    return scenes.Scene(name="rows", x=f[0], y=f[1], vx=f[2], vy=f[3],
                        box=(0.0, float(np.float32(6 * h)), 0.0, float(np.float32(6 * h))), params=p,
                        spacing=h, size_x=6, size_y=6)


def brute(sc):
    P, h = sc.params, float(np.float32(sc.params.smoothing_radius))
    x, y, vx, vy = (a.astype(np.float64) for a in (sc.x, sc.y, sc.vx, sc.vy))
    dx, dy = x[None, :] - x[:, None], y[None, :] - y[:, None]
    r = np.sqrt(dx ** 2 + dy ** 2)
    near = (r <= h) & (r > 0)
    rs = np.where(near, r, 1.0)
    w = np.where(near, 1.0 - r / h, 0.0)
    rho, rhon = (w ** 2).sum(1), (w ** 3).sum(1)
    dt = float(np.float32(P.time_step))
    u = ((vx[:, None] - vx[None, :]) * dx + (vy[:, None] - vy[None, :]) * dy) / rs
    u = np.where(near & (u > 0), u, 0.0)
    imp = dt * w * (P.sigma * u + float(np.float32(P.beta)) * u * u)
    visc = [np.clip(imp * d / rs, -5, 5) for d in (dx, dy)]
    f = lambda v: float(np.float32(v))  # noqa: E731
    pr, pn = f(P.k) * (rho - f(P.rest_density)), f(P.k_near) * rhon
    D = dt * dt * ((pr[:, None] + pr[None, :]) * w + (pn[:, None] + pn[None, :]) * w * w
                   + np.where(near, 0.5 * f(P.k_spring) * (h - r), 0.0))
    mag = dt * dt * ((abs(pr)[:, None] + abs(pr)[None, :] + f(P.k) * f(P.rest_density)) * w
                     + (pn[:, None] + pn[None, :]) * w * w + np.where(near, 0.5 * f(P.k_spring) * h, 0.0))
    return rho, rhon, visc, [-D * d / rs for d in (dx, dy)], [mag * abs(d) / rs for d in (dx, dy)]


@pytest.mark.parametrize("h", [1.0, 0.7])
@pytest.mark.parametrize("length", [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 96, 128, 129, 200])
def test_rows_of_every_length(cuda_lib, length, h):
    sc = three_rows(length, h, seed=length)
    rho, rhon, visc, disp, mag = brute(sc)
    for shapes in (None, [128, 0, 128, 0, 128, 0]):
        with Simulation.from_scene(sc) as s:
            if shapes:
                s.set_launch_shapes(shapes)
            assert s.counters()["max_cell_occupancy"] <= 100
            got = s.probe_density()
            dv, dd = s.probe_viscosity(), s.probe_relaxation()
        for a, b in zip(got, (rho, rhon)):
            assert np.all(np.abs(a - b) <= 1e-5 * b + 1e-12)
        for k in range(2):
            assert np.all(np.abs(dv[k] + 0.5 * visc[k].sum(1)) <= 1e-5 * np.abs(visc[k]).sum(1) + 1e-7)
            # 1e-5 of the summed term magnitudes, each pair term's own parts
            # (before P_i + P_j - 2 k rest cancels) among them
            assert np.all(np.abs(dd[k] - disp[k].sum(1)) <= 1e-5 * mag[k].sum(1) + 1e-9)
