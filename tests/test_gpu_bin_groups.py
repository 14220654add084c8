"""The tile pass's bins on frames with more of them than CTAs fit on the GPU at once (eight bins per CTA there): bin rows
and columns that do and do not fill the groups, over 256 draws, against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import scenes
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu


# bins of 128 x 64: 38 x 32 (a CTA per bin), then groups of 4 x 2: 40 x 31, 41 x 31, 34 x 40
@pytest.mark.parametrize("w,h", [(4864, 2048), (5120, 1984), (5130, 1930), (4250, 2497)])
def test_bins_around_the_line(gpu_ok, w, h):
    fmt = abi.SW_PIXEL_C32
    arena, draws, verts = scenes.make_raster_scene(61, w, h, 40, pixel_format=fmt, texel_density=0.2)
    lite, triangles, tv = scenes.make_triangle_draws(62, w, h, 300, blends=(0, 1, 2, 3, 4))
    draws = scenes.interleave(draws, triangles, 63)
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0))
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_lite_textures(lite)
        r.frame_begin(fp)
        r.set_surfaces(arena)
        r.submit_draws_ex(draws, verts, tv)
        got, want = np.zeros((h, w), np.uint32), np.zeros((h, w), np.uint32)
        r.render(got)
        assert oracle.rasterize(draws, verts, arena, fp, want, tri_vertices=tv, lite=lite) == 0
        assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()
