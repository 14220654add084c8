"""Depth draws on both sides of the widths that go to the chunk list, and lists that parts of 3, 5, 30 and 32 chunks fill
past their end, so that a part finds room for some of its chunks only. The storage equals the oracle's bit for
bit, in a second call with other draws too."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu

pytestmark = pytest.mark.gpu

SIZE = 1024


def _bars(spec, seed):
    """Depth draws of (width, rows) each, anywhere on the map, slightly slanted."""
    rng = np.random.default_rng(seed)
    d = np.zeros(len(spec), abi.DEPTH_DRAW)
    v = []
    for i, (w, h) in enumerate(spec):
        x, y = rng.uniform(0, SIZE - w - 2), rng.uniform(0, SIZE - h)
        d[i]["first_vertex"], d[i]["vertex_count"], d[i]["map_size"] = len(v), 4, SIZE
        d[i]["depth_eq"] = (rng.uniform(-1e-5, 1e-5), rng.uniform(-1e-5, 1e-5), rng.uniform(0.01, 0.1))
        v += [(int(a * 65536), int(b * 65536)) for a, b in ((x, y), (x + w, y), (x + w + 2, y + h), (x + 2, y + h))]
    return d, np.array(v, abi.VERTEX16)


def _check(calls):
    want = np.zeros(SIZE * SIZE, np.float32)
    r = gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))
    try:
        for d, v in calls:
            oracle.shadow_maps(d, v, want)
            r.build_shadow_maps(d, v, SIZE * SIZE)
            got = r.read_shadow_maps(SIZE * SIZE)
            assert np.array_equal(want.view(np.uint32), got.view(np.uint32)), int((want != got).sum())
    finally:
        r.close()


def test_widths_around_the_list(gpu_ok):
    spec = [(w, h) for w in (1, 2, 8, 22, 23, 24, 25, 26, 33) for h in (40, 41, 42, 43, 44, 100, 129, 1000)]
    _check([_bars(spec, 1), _bars(spec[::-1], 2)])


@pytest.mark.parametrize("chunks", [(32,), (30,), (5,), (3, 5, 32)])
def test_lists_that_end_inside_a_part(gpu_ok, chunks):
    def call(total, seed):
        # rows just below whole chunks; rounding to pixel centres never adds one
        spec, n = [], 0
        while n < total:
            c = chunks[len(spec) % len(chunks)]
            spec.append((38, c * 32 - 1))
            n += c
        return _bars(spec, seed)
    _check([call(34000, 3), call(33000, 4), call(100, 5)])
