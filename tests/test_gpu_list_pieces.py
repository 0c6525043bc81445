"""Neighbour lists of more entries than one piece of the library's scratch
(16,777,216) holds: the lists around the piece's border, at both ends and
elsewhere against a brute-force restatement of the reference's order
(hash.c:169-234)."""
import ctypes

import numpy as np
import pytest

from sph_gb300 import Simulation, _lib, scenes

pytestmark = pytest.mark.gpu
PIECE = 16 << 20


def half_list(i, x, y):
    """The half list of particle i in a grid of unit cells."""
    near = np.nonzero((np.abs(x - x[i]) <= 1.5) & (np.abs(y - y[i]) <= 1.5))[0]
    gx, gy = np.floor(x[near]).astype(int), np.floor(y[near]).astype(int)
    cx, cy = int(np.floor(x[i])), int(np.floor(y[i]))
    dx, dy = (x[near] - x[i]).astype(np.float32), (y[near] - y[i]).astype(np.float32)
    hit = (dx * dx + dy * dy).astype(np.float32) <= np.float32(1.0)
    out = []
    for ox, oy in ((0, 0), (0, 1), (1, -1), (1, 0), (1, 1)):
        m = hit & (gx == cx + ox) & (gy == cy + oy)
        if (ox, oy) == (0, 0):
            m &= near > i
        out += sorted(near[m])
    return out


def test_lists_in_several_pieces(cuda_lib):
    n = 1_900_000
    side = int(np.sqrt(n)) + 1
    i = np.arange(n)
    rng = np.random.default_rng(6)
    x = (1.0 + 0.40 * (i % side) + rng.uniform(-0.1, 0.1, n)).astype(np.float32)
    y = (1.0 + 0.40 * (i // side) + rng.uniform(-0.1, 0.1, n)).astype(np.float32)
    size = int(0.40 * side) + 4
    p = scenes.Params(node_end_x=float(size))
    cfg = dict(box=(0.0, float(size), 0.0, float(size)), spacing=1.0, size_x=size, size_y=size,
               max_bucket=100, max_neighbors=400)
    with Simulation(p.as_dict(), cfg, n) as s:
        s.upload(x, y)
        counts, ids = s.neighbor_lists()
        total = ctypes.c_longlong(0)
        small = np.full(1000, -7, np.int32)  # too small: the total, and the buffer as it was
        st = cuda_lib.sph_cuda_neighbor_lists(s.handle, counts.ctypes.data_as(_lib.c_int_p),
                                              small.ctypes.data_as(_lib.c_int_p), 1000, ctypes.byref(total))
        assert st == 4 and total.value == len(ids) and np.all(small == -7)
    assert len(ids) == counts.sum() > PIECE + 1000
    off = np.concatenate([[0], np.cumsum(counts.astype(np.int64))])
    border = int(np.searchsorted(off, PIECE, side="right")) - 1
    for k in [0, 1, n - 1, n - 2, *range(border - 3, border + 4), *rng.integers(0, n, 20)]:
        assert list(ids[off[k]:off[k + 1]]) == half_list(int(k), x, y), k
