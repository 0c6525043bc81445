"""Host buffers that kernels read and write in the caller's memory against the
copies that other buffers take: the same bytes at the sizes where one gives
way to the other, and for buffers off the alignment of their elements, in
page-locked memory, read-only, or overlapping."""
import ctypes

import numpy as np
import pytest

from conftest import bits_equal
from sph_gb300 import LearnedModel, Simulation, _lib, render_liquid, scenes

pytestmark = pytest.mark.gpu

FP = ctypes.POINTER(ctypes.c_float)


def at_byte(a, offset):
    """A copy of `a` that starts `offset` bytes into its allocation."""
    raw = np.zeros(a.nbytes + 64, np.uint8)
    start = -raw.ctypes.data % 64 + offset
    out = np.frombuffer(raw.data, np.uint8, a.nbytes, start)
    out[:] = a.reshape(-1).view(np.uint8)
    return out


def locked(a):
    import torch
    return torch.from_numpy(a.reshape(-1).view(np.uint8).copy()).pin_memory().numpy()


def ptr(raw):
    return ctypes.cast(raw.ctypes.data, FP)


def random_scene(n, seed=5):
    side = max(4, int(np.sqrt(n / 4)))
    rng = np.random.default_rng(seed)
    f = [rng.random(n, np.float32) * np.float32(side), rng.random(n, np.float32) * np.float32(side),
         rng.standard_normal(n, np.float32), rng.standard_normal(n, np.float32)]
    p = scenes.Params(smoothing_radius=1.0, node_end_x=float(side))
    return scenes.Scene(name="random", x=f[0], y=f[1], vx=f[2], vy=f[3], box=(0.0, float(side), 0.0, float(side)),
                        params=p, spacing=1.0, size_x=side, size_y=side)


@pytest.mark.parametrize("n", [1, 255, 4097, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("place", [lambda a: at_byte(a, 0), lambda a: at_byte(a, 4), lambda a: at_byte(a, 2), locked],
                         ids=["aligned", "element", "off", "locked"])
def test_upload_and_download(cuda_lib, n, place):
    sc = random_scene(n)
    cols = [sc.x, sc.y, sc.vx, sc.vy]
    with Simulation.from_scene(sc) as s:
        raw = [place(c) for c in cols]
        for r in raw[:2]:
            r.setflags(write=False)
        _lib.check(cuda_lib.sph_cuda_upload_soa(s.handle, *[ptr(r) for r in raw], n))
        out = [place(np.full(n, 7.0, np.float32)) for _ in range(6)]
        _lib.check(cuda_lib.sph_cuda_download_soa(s.handle, *[ptr(r) for r in out], n))
        for c, r in zip(cols, out):
            assert bits_equal(r.copy().view(np.float32), c)
        for r in out[4:]:
            assert not r.any()
        # the sort that goes on behind an upload: the step after it is that of
        # a state uploaded as records
        s.rebuild_neighbors()
        s.step(sc.params.as_dict(), 1)
        a = s.download()
        xy = place(np.full(2 * n, 9, np.int16))
        _lib.check(cuda_lib.sph_cuda_pack_coords_short(s.handle, ctypes.cast(xy.ctypes.data, _lib.c_short_p), n))
        packed = s.pack_coords()
        assert np.array_equal(xy.copy().view(np.int16).reshape(n, 2), packed)
        recs = np.zeros(n, _lib.PARTICLE_DTYPE)
        for k, c in (("x", sc.x), ("y", sc.y), ("v_x", sc.vx), ("v_y", sc.vy), ("x_prev", sc.x), ("y_prev", sc.y)):
            recs[k] = c
        _lib.check(cuda_lib.sph_cuda_upload_particles(s.handle, recs.ctypes.data, n))
        s.rebuild_neighbors()
        s.step(sc.params.as_dict(), 1)
        b = s.download()
        for f in ("x", "y", "v_x", "v_y", "density", "density_near"):
            assert bits_equal(a[f], b[f]), f


def test_overlapping_columns_keep_the_later_one(cuda_lib):
    n = 1000
    sc = random_scene(n)
    with Simulation.from_scene(sc) as s:
        buf = np.zeros(n + 100, np.float32)
        x, y = buf[:n], buf[100:]
        null = ctypes.cast(None, FP)
        _lib.check(cuda_lib.sph_cuda_download_soa(s.handle, ptr(x), ptr(y), null, null, null, null, n))
        assert bits_equal(y.copy(), sc.y) and bits_equal(x[:100].copy(), sc.x[:100])


@pytest.mark.parametrize("n", [1, 127, 1025, 8192, 8193])
@pytest.mark.parametrize("place", [lambda a: at_byte(a, 0), lambda a: at_byte(a, 4), locked],
                         ids=["aligned", "element", "locked"])
def test_forward(cuda_lib, n, place):
    x = np.random.default_rng(n).standard_normal((n, LearnedModel.IN)).astype(np.float32)
    x[:, 31] = 1.0
    with LearnedModel(0, seed=2) as m:
        a, y = place(x), place(np.full((n, LearnedModel.OUT), 3.0, np.float32))
        _lib.check(cuda_lib.sph_learned_forward(m._l, ptr(a), n, ptr(y)))
        big = np.concatenate([x, np.zeros((20000, LearnedModel.IN), np.float32)])  # copied
        assert bits_equal(y.copy().view(np.float32).reshape(n, -1), m.forward(big)[:n])


@pytest.mark.parametrize("W,H", [(16, 2), (32, 33), (48, 20), (1024, 9), (1040, 9), (2064, 5), (36, 21), (34, 11), (35, 12)])
@pytest.mark.parametrize("offset", [0, 4, 1])
def test_image(cuda_lib, W, H, offset):
    """Rows of whole 16-byte pieces, of words and of neither, in the caller's
    memory or copied to it: the image of the same coordinates through a
    buffer of the library's own."""
    sc = random_scene(3000)
    with Simulation.from_scene(sc) as s:
        want = render_liquid(s.pack_coords(), W, H)[0]
        raw = at_byte(np.full((H, W, 3), 77, np.uint8), offset)
        up = ctypes.POINTER(ctypes.c_ubyte)
        _lib.check(cuda_lib.sph_cuda_render_liquid(s.handle, W, H, ctypes.cast(raw.ctypes.data, up),
                                                   ctypes.cast(None, up)))
        assert np.array_equal(raw.reshape(H, W, 3), want)
