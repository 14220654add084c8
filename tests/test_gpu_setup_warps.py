"""Raster setup with a CTA per draw and, from 1,024 draws on, with a warp per draw: polygons and triangles in painter's
order at draw counts around the line and around a multiple of eight, against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import scenes
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_quads,num_tris", [(500, 523), (500, 524), (501, 524), (0, 1031), (1100, 0)])
def test_setup_around_the_line(gpu_ok, num_quads, num_tris):
    w, h, fmt = 500, 300, abi.SW_PIXEL_C64
    blends = (0, 1, 2, 3, 4)
    arena, polygons, verts = scenes.make_raster_scene(51, w, h, max(num_quads, 1), modes=(0, 1, 2), blends=blends, pixel_format=fmt)
    lite, triangles, tv = scenes.make_triangle_draws(52, w, h, max(num_tris, 1), blends=blends)
    polygons, triangles = polygons[:num_quads], triangles[:num_tris]
    draws = scenes.interleave(polygons, triangles, 53) if num_quads and num_tris else (polygons if num_quads else triangles)
    assert draws.size == num_quads + num_tris
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0))
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_lite_textures(lite)
        r.frame_begin(fp)
        r.set_surfaces(arena)
        r.submit_draws_ex(draws, verts, tv)
        got, want = np.zeros((h, w), np.uint64), np.zeros((h, w), np.uint64)
        r.render(got)
        assert oracle.rasterize(draws, verts, arena, fp, want, tri_vertices=tv, lite=lite) == 0
        assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()
