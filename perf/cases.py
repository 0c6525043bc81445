"""Timed cases of the framework's public entry points.

Each case is one pass of something a user's program does over and over:

  frame      the interactive compute rank: one frame of 4 sub-steps, then the
             packed short coordinates for the render rank into page-locked
             memory (the reference's `steps_per_frame` is 4)
  state      an offline run: upload of particle arrays, 2 steps, download of
             the whole state
  ensemble   a frame of many independent scenes in one handle, with the
             per-scene diagnostics a sweep records
  learned    a frame with the learned relaxation attached
  density    the allocation-free density of caller-owned device arrays
  lists      the reference's neighbour half lists of the current state, into
             the caller's buffers
  features   the feature rows of the predicted state (data for one's own
             training)
  forward    the network on host feature rows
  train      a training round: collect one state's samples, one epoch
  image      the liquid image of the current particles

Sizes: 3,000 and 4,194,304 particles are the two dam breaks of the scenes
module, 65,536 the training scenes', 65,536 the allocation-free entry's
largest; the others lie between.
"""
import ctypes
import math

import numpy as np
import torch

from sph_gb300 import Ensemble, LearnedModel, Simulation, _lib, scenes

SUBSTEPS = 4   # sub-steps of a frame
IN, HID, OUT = LearnedModel.IN, LearnedModel.HIDDEN, LearnedModel.OUT
MAX_NB = LearnedModel.MAX_NEIGHBORS
MOVERS = ("none", "sphere", "rectangle")


def listed():
    return [
        # the interactive size: every launch and every host call counts
        dict(name="frame_3k", kind="frame", n=3000, mover="none"),
        # a run whose state goes back to the host, at the training scenes' size
        dict(name="state_64k", kind="state", n=65536, mover="sphere", h=1.0, long_rows=False),
        # the headline workload: the 4,194,304-particle dam break with its mover
        dict(name="frame_4m", kind="frame", n=4194304, mover="sphere"),
        # a parameter sweep: scenes of 1,024 to 65,536 particles together
        dict(name="ensemble_64", kind="ensemble", scenes=64, lo=1024, hi=65536),
        # the learned step at a quarter of the headline size
        dict(name="learned_1m", kind="learned", n=1048576, mover="sphere"),
        # a caller without cudaMalloc, near the entry's largest size, ragged
        dict(name="density_65k", kind="density", n=65521, h=1.0),
        # neighbour lists for an analysis outside the library
        dict(name="lists_256k", kind="lists", n=262144, h=1.0),
        # feature rows of an odd number of particles
        dict(name="features_128k", kind="features", n=131071, h=1.0),
        # the network on a few rows (latency) and on many
        dict(name="forward_1k", kind="forward", n=1000),
        dict(name="forward_512k", kind="forward", n=524288),
        # one state's samples and an epoch on them, at the training scenes' size
        dict(name="train_64k", kind="train", n=65536, batch=4096, h=1.0),
        # the picture of a frame at the usual screen size
        dict(name="image_1080p", kind="image", n=1048576, width=1920, height=1080),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "state", "ensemble", "learned", "density", "lists", "features",
                       "forward", "train", "image"))
    # a grid spacing that is a power of two divides exactly; others do not
    h = rng.choice((1.0, 1.0, 0.5, round(rng.uniform(0.3, 1.3), 3)))
    if kind == "frame":
        return dict(kind=kind, n=_log_int(rng, 500, 4000000), mover=rng.choice(MOVERS))
    if kind == "state":
        return dict(kind=kind, n=_log_int(rng, 500, 500000), mover=rng.choice(MOVERS), h=h,
                    long_rows=rng.random() < 0.3)
    if kind == "ensemble":
        return dict(kind=kind, scenes=_log_int(rng, 2, 200), lo=512, hi=_log_int(rng, 2048, 32768))
    if kind == "learned":
        return dict(kind=kind, n=_log_int(rng, 3000, 2000000), mover=rng.choice(MOVERS))
    if kind == "density":
        return dict(kind=kind, n=_log_int(rng, 100, 65536), h=h)
    if kind == "lists":
        return dict(kind=kind, n=_log_int(rng, 500, 1000000), h=h)
    if kind == "features":
        return dict(kind=kind, n=_log_int(rng, 500, 500000), h=h)
    if kind == "forward":
        return dict(kind=kind, n=_log_int(rng, 1, 1000000))
    if kind == "train":
        return dict(kind=kind, n=_log_int(rng, 4000, 65536),
                    batch=rng.choice((512, 1000, 2048, 4096)), h=h)
    return dict(kind=kind, n=_log_int(rng, 1000, 2000000), width=rng.randint(160, 1920),
                height=rng.randint(120, 1080))


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------

def _mover(kind, h, base, t):
    """Mover fields of the tunables at frame t (as the dam break moves it)."""
    if kind == "none":
        return {}
    cx = base[0] + 20.0 * h * math.sin(2.0 * math.pi * t / 60.0)
    return dict(mover_center_x=float(np.float32(cx)), mover_center_y=float(np.float32(base[1])),
                mover_width=16.0 * h, mover_height=12.0 * h if kind == "rectangle" else 16.0 * h,
                mover_type=scenes.RECTANGLE_MOVER if kind == "rectangle" else scenes.SPHERE_MOVER)


def _dam(n, seed, mover):
    """The dam break of the scenes module at n particles, filled on the GPU:
    a handle and the tunables of 60 frames."""
    s = math.sqrt(n / 4194304)
    w, h_box = float(max(8, math.ceil(3590 * s))), float(max(8, math.ceil(1795 * s)))
    cols = max(8, int(round(2393 * s)))
    p = scenes.Params(node_end_x=w).as_dict()
    # the mover's path lies elsewhere in the fluid for each seed
    base = (598.0 * s * np.random.default_rng(seed).uniform(0.6, 1.4), 438.0 * s)
    frames = [dict(p, **_mover(mover, 1.0, base, t)) for t in range(60)]
    cfg = dict(box=(0.0, w, 0.0, h_box), spacing=1.0, size_x=int(w), size_y=int(h_box),
               max_bucket=100, max_neighbors=400)
    sim = Simulation(frames[0], cfg, n)
    sim.init_lattice([dict(n=n, cols=cols, x0=0.0, y0=0.0, spacing=0.5, jitter=0.05,
                           seed=1002 + seed, counter0=0)])
    return sim, frames


def _fluid(n, seed, h):
    """A stirred block of fluid at its usual density (about 18 neighbours):
    float32 x, y, vx, vy, and the grid of its box."""
    rng = np.random.default_rng(seed)
    cols = max(4, int(math.sqrt(2.0 * n)))
    i = np.arange(n)
    a = 0.42 * h
    x = a * (i % cols + 0.5) + rng.uniform(-0.15, 0.15, n) * h
    y = a * (i // cols + 0.5) + rng.uniform(-0.15, 0.15, n) * h
    sx, sy = int(math.ceil(0.42 * cols * 1.5)) + 2, int(math.ceil(0.42 * (n // cols + 1) * 2)) + 2
    box = (0.0, float(np.float32(sx * h)), 0.0, float(np.float32(sy * h)))
    x, y = np.clip(x, 0.0, None), np.clip(y, 0.0, None)
    v = rng.uniform(-1.0, 1.0, (2, n))
    cfg = dict(box=box, spacing=h, size_x=sx, size_y=sy, max_bucket=100, max_neighbors=400)
    return [np.ascontiguousarray(q, np.float32) for q in (x, y, v[0], v[1])], cfg, (a * cols, a * (n // cols + 1))


def _fluid_params(case, cfg, size):
    h = case["h"]
    base = (0.4 * size[0], 0.4 * size[1])
    p = scenes.Params(smoothing_radius=h, node_end_x=cfg["box"][1]).as_dict()
    return dict(p, **_mover(case.get("mover", "none"), 0.25 * h, base, 3))


def _weights(seed, relax):
    """Network parameters.  relax: the first hidden units carry the
    relaxation's displacement, which is linear in the feature row (2 GELU(z)
    - 2 GELU(-z) = 2 z), the others are random and feed the predicted error
    alone -- what a trained network does; otherwise all random."""
    rng = np.random.default_rng(seed + 77)
    W1 = rng.uniform(-1, 1, (HID, IN)) * math.sqrt(6.0 / (HID + IN))
    W2 = rng.uniform(-1, 1, (HID, HID)) * math.sqrt(6.0 / (2 * HID))
    W3 = rng.uniform(-1, 1, (OUT, HID)) * math.sqrt(6.0 / (OUT + HID))
    b1, b2, b3 = (rng.normal(0.0, 0.02, k) for k in (HID, HID, OUT))
    if relax:
        W1[:4], W2[:4], b1[:4], b2[:4], W3[:3, :] = 0.0, 0.0, 0.0, 0.0, 0.0
        W2[4:, :4] = 0.0
        for c in range(2):
            row = np.zeros(IN)
            row[[17 + c, 19 + c, 21 + c, 23 + c, 25 + c]] = (-4.0, -2.0, -1.0, -4.0, -2.0)
            W1[2 * c], W1[2 * c + 1] = row, -row
            W2[2 * c, [2 * c, 2 * c + 1]] = 0.5, -0.5
            W2[2 * c + 1, [2 * c, 2 * c + 1]] = -0.5, 0.5
            W3[c, [2 * c, 2 * c + 1]] = 0.5, -0.5
        W3[2, 4:] = rng.normal(0.0, 0.01, HID - 4)
        b3[:3] = 0.0, 0.0, 0.3
    return np.concatenate([q.reshape(-1) for q in (W1, b1, W2, b2, W3, b3)]).astype(np.float32)


def _features_rows(n, seed):
    """Feature rows of the usual ranges, the constant feature last."""
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((n, IN), dtype=np.float32) * np.float32(0.5)
    f[:, 27:31] = 0.0
    f[:, 31] = 1.0
    return f


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _sweep_sizes(case):
    """Particles of a sweep's scenes: log-uniform from lo to hi, shuffled."""
    k, lo, hi = case["scenes"], case["lo"], case["hi"]
    sizes = [int(round(lo * (hi / lo) ** ((i + 0.5) / k))) for i in range(k)]
    return [sizes[i] for i in np.random.default_rng(k).permutation(k)]


def _page_locked(n):
    """A coordinate buffer that lives as long as any array on it."""
    return torch.empty((n, 2), dtype=torch.int16, pin_memory=True).numpy()


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind in ("frame", "learned", "image"):
        s["sim"], s["frames"] = _dam(case["n"], seed, case.get("mover", "sphere"))
        s["t"] = 0
        # the fluid is moving before the first pass
        s["sim"].step(s["frames"][0], 40)
        if kind == "learned":
            s["model"] = LearnedModel(0, seed=seed)
            s["model"].set_params(_weights(seed, True))
            s["sim"].set_learned(s["model"], 0.01)
        if kind != "image":
            s["coords"] = _page_locked(case["n"])
        s["sim"].synchronize()
    elif kind == "ensemble":
        scs = [scenes.ensemble_scene(100003 * seed + k, f"sweep_{k}", (m, m))
               for k, m in enumerate(_sweep_sizes(case))]
        s["sim"] = Ensemble(scs, 100, 400)
        s["sim"].upload_scenes()
        s["sim"].step(None, 40)
        s["coords"] = _page_locked(s["sim"].n)
        s["sim"].synchronize()
    elif kind == "forward":
        s["model"] = LearnedModel(0, seed=seed)
        s["model"].set_params(_weights(seed, False))
        s["features"] = _features_rows(case["n"], seed)
    else:
        s["arrays"], cfg, size = _fluid(case["n"], seed, case["h"])
        s["params"] = _fluid_params(case, cfg, size)
        if kind == "density":
            s["x"], s["y"] = (torch.from_numpy(q).cuda() for q in s["arrays"][:2])
            s["rho"], s["rho_near"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
            g = _lib.NeighborGrid()
            g.spacing, g.size_x, g.size_y = cfg["spacing"], cfg["size_x"], cfg["size_y"]
            g.max_bucket_size, g.max_neighbors = cfg["max_bucket"], cfg["max_neighbors"]
            s["grid"], s["tunables"] = g, _lib.tunables(s["params"])
            f = _lib.lib().sph_cuda_density_static
            f.restype = ctypes.c_int
            f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                          ctypes.POINTER(_lib.NeighborGrid), ctypes.POINTER(_lib.TunableParameters),
                          ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        else:
            s["sim"] = Simulation(s["params"], cfg, case["n"])
            if kind == "state":
                s["sim"].set_long_row_masks(case["long_rows"])
            else:
                s["sim"].upload(*s["arrays"])
                s["sim"].rebuild_neighbors()
            if kind == "lists":
                # the caller's buffers: about 9 entries a particle are used
                s["counts"] = np.zeros(case["n"], np.int32)
                s["ids"] = np.zeros(16 * case["n"], np.int32)
            if kind == "train":
                s["model"] = LearnedModel(case["n"], seed=seed)
                s["w0"] = _weights(seed, False)
    return s


def run(s):
    kind = s["kind"]
    if kind in ("frame", "learned"):
        s["sim"].step(s["frames"][s["t"] % len(s["frames"])], nsteps=SUBSTEPS)
        s["t"] += 1
        return s["sim"].pack_coords(s["coords"])
    if kind == "state":
        sim = s["sim"]
        sim.upload(*s["arrays"])
        sim.rebuild_neighbors()
        sim.step(s["params"], nsteps=2)
        return sim.download()
    if kind == "ensemble":
        s["sim"].step(None, nsteps=SUBSTEPS)
        return dict(coords=s["sim"].pack_coords(s["coords"]),
                    diagnostics=s["sim"].scene_diagnostics())
    if kind == "density":
        _lib.check(_lib.lib().sph_cuda_density_static(
            s["x"].data_ptr(), s["y"].data_ptr(), s["case"]["n"], ctypes.byref(s["grid"]),
            ctypes.byref(s["tunables"]), s["rho"].data_ptr(), s["rho_near"].data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return dict(rho=s["rho"], rho_near=s["rho_near"])
    if kind == "lists":
        total = ctypes.c_longlong(0)
        _lib.check(_lib.lib().sph_cuda_neighbor_lists(
            s["sim"].handle, s["counts"].ctypes.data_as(_lib.c_int_p),
            s["ids"].ctypes.data_as(_lib.c_int_p), s["ids"].size, ctypes.byref(total)))
        return dict(total=total.value, counts=s["counts"], ids=s["ids"])
    if kind == "features":
        f, c = s["sim"].learned_features()
        return dict(features=f, counts=c)
    if kind == "forward":
        return s["model"].forward(s["features"])
    if kind == "train":
        m = s["model"]
        m.clear_samples()
        m.collect(s["sim"])
        m.set_params(s["w0"])
        loss = m.train(1, s["case"]["batch"], 1e-3)
        return dict(loss=loss, params=m.get_params())
    return s["sim"].render_liquid(s["case"]["width"], s["case"]["height"])


# multiply-adds of one network row, times two
_ROW_FLOPS = 2 * (IN * HID + HID * HID + HID * OUT)


def work(case):
    kind = case["kind"]
    n = sum(_sweep_sizes(case)) if kind == "ensemble" else case["n"]
    if kind in ("frame", "learned", "ensemble"):
        # position and velocity in and out once a step, the packed coordinates
        # out; about 20 neighbours a particle in three passes of about 30
        # operations each
        flops = n * SUBSTEPS * 20 * 3 * 30
        if kind == "learned":
            flops += n * SUBSTEPS * _ROW_FLOPS
        return dict(bytes=n * (32 * SUBSTEPS + 4), flops=flops)
    if kind == "state":
        return dict(bytes=n * (16 + 2 * 32 + 24), flops=n * 2 * 18 * 3 * 30)
    if kind == "density":
        return dict(bytes=n * 16, flops=n * 18 * 15)
    if kind == "lists":
        return dict(bytes=n * (8 + 4 + 9 * 4), flops=n * 18 * 5)
    if kind == "features":
        return dict(bytes=n * (16 + 4 * IN + 4), flops=n * 18 * 80)
    if kind == "forward":
        return dict(bytes=n * 4 * (IN + OUT), flops=n * _ROW_FLOPS)
    if kind == "train":
        return dict(bytes=n * (16 + 2 * (2 * IN + 16)), flops=n * (3 * _ROW_FLOPS + 18 * 150))
    return dict(bytes=n * 8 + 3 * case["width"] * case["height"],
                flops=n * 60 + case["width"] * case["height"] * 50)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

class _Pairs:
    """All ordered pairs (i, j), i != j, within h of one another."""

    def __init__(self, x, y, h, cfg):
        n, sx, sy = len(x), cfg["size_x"], cfg["size_y"]
        # one ring of empty cells around the grid
        cx = np.clip(np.floor(x / h).astype(np.int64), 0, sx) + 1
        cy = np.clip(np.floor(y / h).astype(np.int64), 0, sy) + 1
        w = sx + 3
        key = cy * w + cx
        order = np.argsort(key, kind="stable")
        start = np.searchsorted(key[order], np.arange(w * (sy + 3) + 1))
        self.order = order
        ii, jj = [], []
        for dy in (-1, 0, 1):
            a, b = start[key + dy * w - 1], start[key + dy * w + 2]
            length = b - a
            i = np.repeat(np.arange(n), length)
            j = np.arange(length.sum()) - np.repeat(np.cumsum(length) - length, length) + np.repeat(a, length)
            j = order[j]
            near = ((x[i] - x[j]) ** 2 + (y[i] - y[j]) ** 2 <= h * h) & (i != j)
            ii.append(i[near])
            jj.append(j[near])
        self.i, self.j, self.n = np.concatenate(ii), np.concatenate(jj), n
        self.ux, self.uy = x[self.j] - x[self.i], y[self.j] - y[self.i]
        self.r = np.sqrt(self.ux ** 2 + self.uy ** 2)
        self.ux, self.uy = self.ux / self.r, self.uy / self.r   # unit offset towards j
        self.w = 1.0 - self.r / h

    def sum(self, v):
        return np.bincount(self.i, v, self.n)


def _boundary(x, y, P, box):
    x, y = x.copy(), y.copy()
    ex, ey = x - P["mover_center_x"], y - P["mover_center_y"]
    if P["mover_type"] == scenes.SPHERE_MOVER:
        rad = 0.5 * P["mover_width"]
        d = np.sqrt(ex ** 2 + ey ** 2)
        m = (d <= rad) & (d > 0)
        x[m] += (rad - d[m]) * ex[m] / d[m]
        y[m] += (rad - d[m]) * ey[m] / d[m]
    else:
        px, py = 0.5 * P["mover_width"] - np.abs(ex), 0.5 * P["mover_height"] - np.abs(ey)
        m = (px > 0) & (py > 0)
        mx, my = m & (px < py), m & ~(px < py)
        x[mx] += np.where(ex[mx] < 0, -px[mx], px[mx])
        y[my] += np.where(ey[my] < 0, -py[my], py[my])
    x = np.where(x < box[0], box[0], np.where(x > box[1], box[1] - 0.001, x))
    y = np.where(y < box[2], box[2], np.where(y > box[3], box[3] - 0.001, y))
    return x, y


def _f64(params):
    return {k: (float(np.float32(v)) if isinstance(v, float) else v) for k, v in params.items()}


def _predict(x, y, vx, vy, P, cfg):
    """Gravity, viscosity impulses, prediction and boundary conditions."""
    q = _Pairs(x, y, P["smoothing_radius"], cfg)
    dt = P["time_step"]
    u = (vx[q.i] - vx[q.j]) * q.ux + (vy[q.i] - vy[q.j]) * q.uy
    u = np.where((u > 0) & (q.r > 0), u, 0.0)
    imp = dt * q.w * (P["sigma"] * u + P["beta"] * u * u)
    vx = vx - 0.5 * q.sum(np.clip(imp * q.ux, -5, 5))
    vy = vy - P["g"] * dt - 0.5 * q.sum(np.clip(imp * q.uy, -5, 5))
    return _boundary(x + vx * dt, y + vy * dt, P, cfg["box"])


def _relax(x, y, P, cfg):
    """Densities and the relaxation's displacements of predicted positions."""
    h = P["smoothing_radius"]
    q = _Pairs(x, y, h, cfg)
    rho, near = q.sum(q.w ** 2), q.sum(q.w ** 3)
    pr, pn = P["k"] * (rho - P["rest_density"]), P["k_near"] * near
    d = P["time_step"] ** 2 * ((pr[q.i] + pr[q.j]) * q.w + (pn[q.i] + pn[q.j]) * q.w ** 2
                               + 0.5 * P["k_spring"] * (h - q.r))
    return q, rho, near, -q.sum(d * q.ux), -q.sum(d * q.uy)


def _exact_state(arrays, params, cfg):
    P = _f64(params)
    x, y, vx, vy = (q.astype(np.float64) for q in arrays)
    for _ in range(2):
        px, py = _predict(x, y, vx, vy, P, cfg)
        _, rho, near, dx, dy = _relax(px, py, P, cfg)
        x1, y1 = _boundary(px + dx, py + dy, P, cfg["box"])
        vx = np.clip((x1 - x) / P["time_step"], -5, 5)
        vy = np.clip((y1 - y) / P["time_step"], -5, 5)
        x, y = x1, y1
    return dict(x=x, y=y, v_x=vx, v_y=vy, density=rho, density_near=near)


def _exact_features(arrays, params, cfg):
    """Feature rows, neighbour counts, and the targets of a training sample."""
    P = _f64(params)
    x, y, vx, vy = (q.astype(np.float64) for q in arrays)
    px, py = _predict(x, y, vx, vy, P, cfg)
    q, rho, near, dx, dy = _relax(px, py, P, cfg)
    h, dt, rest = P["smoothing_radius"], P["time_step"], P["rest_density"]
    ks = np.array([P["k"], P["k_near"], P["k_spring"]])
    ak, an, as_ = ks / ks.sum()
    count = np.bincount(q.i, minlength=q.n)
    sx, sy = (px - x) / h, (py - y) / h
    v1 = q.sum(q.w * q.ux), q.sum(q.w * q.uy)
    v2 = q.sum(q.w ** 2 * q.ux), q.sum(q.w ** 2 * q.uy)
    pr, prn = q.w * (rho[q.j] - rest), q.w ** 2 * near[q.j]
    one = np.ones(q.n)
    f = [rho / 4, near / 2, v1[0] / 4, v1[1] / 4, v2[0] / 2, v2[1] / 2, q.sum(q.w) / 8,
         np.minimum(count, MAX_NB) / MAX_NB, q.sum(q.w * (sx[q.j] - sx[q.i])) * 2.5,
         q.sum(q.w * (sy[q.j] - sy[q.i])) * 2.5, q.sum(q.w * q.ux ** 2) / 4,
         q.sum(q.w * q.ux * q.uy) / 4, q.sum(q.w * q.uy ** 2) / 4, ak * one, an * one, as_ * one,
         rest / 4 * one, ak * (rho - rest) * v1[0] / 4, ak * (rho - rest) * v1[1] / 4,
         an * near * v2[0] / 2, an * near * v2[1] / 2, as_ * v1[0] / 2, as_ * v1[1] / 2,
         ak * q.sum(pr * q.ux) / 4, ak * q.sum(pr * q.uy) / 4, an * q.sum(prn * q.ux) / 2,
         an * q.sum(prn * q.uy) / 2] + [0.0 * one] * 4 + [one]
    s = h * dt * dt * ks.sum()
    return np.stack(f, 1), count, np.stack([dx / s, dy / s], 1), q.order


def _act(z):
    """2 GELU (tanh form)."""
    return z * (1.0 + np.tanh(0.7978845608028654 * (z + 0.044715 * z * z * z)))


def _act_grad(z):
    t = np.tanh(0.7978845608028654 * (z + 0.044715 * z * z * z))
    return 1.0 + t + z * (1.0 - t * t) * 0.7978845608028654 * (1.0 + 0.134145 * z * z)


def _exact_forward(w, x):
    p = {k: v.astype(np.float64) for k, v in LearnedModel.unpack(w).items()}
    h1 = _act(x @ p["W1"].T + p["b1"])
    h2 = _act(h1 @ p["W2"].T + p["b2"])
    y = h2 @ p["W3"].T + p["b3"]
    y[:, 3:] = 0.0
    return y


def _epoch_order(n, seed):
    """The documented shuffle of an epoch: Fisher-Yates over splitmix64."""
    order, mask = list(range(n)), (1 << 64) - 1
    rng = (seed * 0x9E3779B97F4A7C15 + 17) & mask
    for i in range(n - 1, 0, -1):
        rng = (rng + 0x9E3779B97F4A7C15) & mask
        z = rng
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        k = (z ^ (z >> 31)) % (i + 1)
        order[i], order[k] = order[k], order[i]
    return np.array(order)


def _exact_train(w0, X, T, batch, seed):
    """One epoch of Adam on the displacement outputs."""
    p = {k: v.astype(np.float64).copy() for k, v in LearnedModel.unpack(w0).items()}
    # the first bias acts through the constant feature, whose weight alone
    # is trained: b1 stays as it is and the products see the weight
    m = {k: np.zeros_like(v) for k, v in p.items()}
    v = {k: np.zeros_like(q) for k, q in p.items()}
    n = len(X)
    batch = max(128, min(batch, n) // 128 * 128)
    order, loss, steps = _epoch_order(n, seed), 0.0, n // batch
    for t in range(steps):
        rows = order[t * batch:(t + 1) * batch]
        x, tt = X[rows], T[rows]
        z1 = x @ p["W1"].T + p["b1"]
        h1 = _act(z1)
        z2 = h1 @ p["W2"].T + p["b2"]
        h2 = _act(z2)
        d = (h2 @ p["W3"].T + p["b3"])[:, :2] - tt
        loss += float((d * d).sum())
        dy = np.zeros((batch, OUT))
        dy[:, :2] = 2.0 * d / batch
        dz2 = (dy @ p["W3"]) * _act_grad(z2)
        dz1 = (dz2 @ p["W2"]) * _act_grad(z1)
        g = dict(W1=dz1.T @ x, b1=0.0 * p["b1"], W2=dz2.T @ h1, b2=dz2.sum(0), W3=dy.T @ h2, b3=dy.sum(0))
        for k in p:
            m[k] = 0.9 * m[k] + 0.1 * g[k]
            v[k] = 0.999 * v[k] + 0.001 * g[k] ** 2
            p[k] -= 1e-3 * (m[k] / (1 - 0.9 ** (t + 1))) / (np.sqrt(v[k] / (1 - 0.999 ** (t + 1))) + 1e-8)
    return loss / (steps * batch), np.concatenate([p[k].reshape(-1) for k in ("W1", "b1", "W2", "b2", "W3", "b3")])


def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        if case["n"] > 600000:
            return None
        return _exact_forward(_weights(seed, False), _features_rows(case["n"], seed).astype(np.float64))
    if kind not in ("state", "density", "features", "train"):
        return None   # whole numbers, or a state that many steps have led to
    arrays, cfg, size = _fluid(case["n"], seed, case["h"])
    params = _fluid_params(case, cfg, size)
    if kind == "state":
        return _exact_state(arrays, params, cfg) if case["n"] <= 200000 else None
    if kind == "density":
        q = _Pairs(arrays[0].astype(np.float64), arrays[1].astype(np.float64), float(np.float32(case["h"])), cfg)
        return dict(rho=q.sum(q.w ** 2), rho_near=q.sum(q.w ** 3))
    if case["n"] > 200000:
        return None
    f, count, target, order = _exact_features(arrays, params, cfg)
    if kind == "features":
        return dict(features=f, counts=None)
    take = order[count[order] <= MAX_NB]
    loss, w = _exact_train(_weights(seed, False), f[take], target[take], case["batch"], seed)
    return dict(loss=loss, params=w)
