"""The perspective division of the tile pass (2^31 / z from an approximate reciprocal and an integer correction): the
correction is exact for every divisor whichever way the reciprocal is off, and a frame that meets every divisor a
draw can have equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu, synth


def test_correction_is_exact_for_every_divisor():
    for first in range(512, (1 << 24) + 1, 1 << 21):
        z = np.arange(first, min(first + (1 << 21), (1 << 24) + 1), dtype=np.int64)
        exact = np.float32(1.0) / z.astype(np.float32)
        # rcp.approx.ftz.f32 is off by at most one unit in the last place
        for inv in (np.nextafter(exact, np.float32(0)), exact, np.nextafter(exact, np.float32(1))):
            q = (inv * np.float32(2147483648.0) + np.float32(8388608.0)).view(np.uint32).astype(np.int64) & 0x7FFFFF
            r = (1 << 31) - q * z
            assert np.all(r > -z) and np.all(r < 2 * z) and np.all(np.abs(r) < 1 << 31)
            assert np.array_equal(q + (r >= z) - (r < 0), (1 << 31) // z)


@pytest.mark.gpu
@pytest.mark.parametrize("t0,t1", [(32.0, 24.7), (29.3, 31.1), (7.9, 17.3), (1.0, 0.37)])
def test_every_divisor_in_a_frame(gpu_ok, t0, t1):
    """16384 x 128 pixels with inv_z = 256 (1 + x + 16384 y), up to the largest inv_z there is, and textures whose texels are
    their addresses."""
    w, h, side, fmt = 16384, 128, 512, abi.SW_PIXEL_C32
    d = np.zeros(1, abi.DRAW_CMD)
    d["vertex_count"], d["mode"], d["blend"] = 4, abi.SW_RASTER_FULL_PERSPECTIVE, abi.SW_BLEND_NONE
    dx, dy = 2.0 ** -21, 2.0 ** -7
    d["depth_eq"] = (dx, dy, dx - (dx + dy) * 0.5)  # exact in f32
    d["tc_eq"] = (0, 0, 0, 0, t0, t1)
    d["tex_size"] = (side, side)
    v = np.array([(x << 16, y << 16) for x, y in ((0, 0), (w, 0), (w, h), (0, h))], abi.VERTEX16)
    arena = np.arange(side * side, dtype=np.uint32)
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0))
    want, got = np.zeros((h, w), np.uint32), np.zeros((h, w), np.uint32)
    assert oracle.rasterize(d, v, arena, fp, want) == 0
    assert np.unique(want).size > 100
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.frame_begin(fp)
        r.set_surfaces(arena)
        r.submit_draws(d, v)
        r.render(got)
        assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()
