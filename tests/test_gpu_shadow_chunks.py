"""Depth draws around the limits of the chunk list (large parts go to warps of their own, 32 rows each): parts
just below and above the direct size, row counts around 32, odd map sizes, spans cut by the map's edges, and
more chunks than the list holds. The storage equals the oracle's bit for bit."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu

pytestmark = pytest.mark.gpu


def _renderer():
    return gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))


def _draws(polys, size, seed):
    """One depth draw per polygon (float x, y lists, clockwise) on one size x size map."""
    rng = np.random.default_rng(seed)
    d = np.zeros(len(polys), abi.DEPTH_DRAW)
    v = []
    for i, p in enumerate(polys):
        d[i]["first_vertex"], d[i]["vertex_count"], d[i]["map_size"] = len(v), len(p), size
        d[i]["depth_eq"] = (rng.uniform(-1e-5, 1e-5), rng.uniform(-1e-5, 1e-5), rng.uniform(0.01, 0.1))
        v += [(int(x * 65536), int(y * 65536)) for x, y in p]
    return d, np.array(v, abi.VERTEX16)


def _check(d, v, size):
    want = np.zeros(size * size, np.float32)
    oracle.shadow_maps(d, v, want)
    r = _renderer()
    try:
        for _ in range(2):  # the list is empty again for the second call
            r.build_shadow_maps(d, v, size * size)
            got = r.read_shadow_maps(size * size)
            assert np.array_equal(want.view(np.uint32), got.view(np.uint32)), int((want != got).sum())
    finally:
        r.close()


@pytest.mark.parametrize("size", [33, 256, 1000, 1024])
def test_parts_around_the_direct_size(gpu_ok, size):
    polys = []
    for rows in (1, 31, 32, 33, 64, 65, size):
        for width in (1, 15, 16, 32, 33, size):
            x, y = size * 0.4 - width * 0.3, size * 0.5 - rows * 0.4  # some of them cut by the map's edges
            polys.append([(x, y), (x + width, y), (x + width, y + rows), (x, y + rows)])
    s = float(size)
    polys += [[(0.0, 0.0), (s, 0.0), (s, s), (0.0, s)], [(s * 0.5, 0.2), (s - 0.3, s * 0.6), (s * 0.1, s - 0.4)],
              [(0.3, 0.3), (1.4, 0.3), (s - 0.2, s - 0.3), (s - 1.5, s - 0.3)]]  # a thin diagonal
    order = np.random.default_rng(size).permutation(len(polys))
    _check(*_draws([polys[i] for i in order], size, size), size)


def test_more_chunks_than_the_list_holds(gpu_ok):
    # 1,100 slivers of 1,024 rows: 35,200 chunks of 32 rows against a list of 32,768
    size = 1024
    polys = []
    for i in range(1100):
        x = (i * 7.31) % (size - 8)
        polys.append([(x, 0.0), (x + 3.0, 0.0), (x + 5.0, 1024.0), (x + 2.0, 1024.0)])
    _check(*_draws(polys, size, 3), size)
