"""The untuned tile shape follows the frame's draws (with triangles or without): frames of a pixel less, equal and more
than the tiles, drawn in turn with and without triangles by one context, per call and through the frame graph, at
the untuned shape and the fixed one. Every frame equals the oracle's."""
import numpy as np
import pytest

import oracle
import scenes
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 3])
@pytest.mark.parametrize("w,h", [(63, 31), (64, 32), (65, 33), (128, 16), (129, 63), (200, 15)])
def test_frames_with_and_without_triangles(gpu_ok, w, h, shape):
    fmt = abi.SW_PIXEL_C64
    blends = (0, 1, 2, 3, 4)
    arena, polygons, verts = scenes.make_raster_scene(71, w, h, 12, blends=blends, pixel_format=fmt)
    lite, triangles, tv = scenes.make_triangle_draws(72, w, h, 40, blends=blends)
    mixed = scenes.interleave(polygons, triangles, 73)
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0))
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_tuning(shape, 24)
        r.set_lite_textures(lite)
        want = np.zeros((h, w), np.uint64)
        for draws, t in ((polygons, None), (mixed, tv), (polygons, None), (mixed, tv)):  # the frame buffer carries over
            assert oracle.rasterize(draws, verts, arena, fp, want, tri_vertices=t, lite=lite) == 0
            got = np.zeros((h, w), np.uint64)
            r.frame_begin(fp)
            r.set_surfaces(arena)
            r.submit_draws_ex(draws, verts, t)
            r.render(got)
            assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_tuning(shape, 24)
        r.set_lite_textures(lite)
        want = np.zeros((h, w), np.uint64)
        got = np.zeros((h, w), np.uint64)
        for draws, t in ((triangles, tv), (triangles[:0], None), (triangles, tv)):  # one graph, updated
            assert oracle.rasterize(draws, None, None, fp, want, tri_vertices=t, lite=lite) == 0
            r.draw_frame(r.frame_input(fp, None, None, 0, draws, None, dst=got, tri_vertices=t))
            assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()


@pytest.mark.parametrize("w,h", [(1600, 768), (1600, 769), (1217, 1024)])
def test_frames_around_a_wave_of_tiles(gpu_ok, w, h):
    """600 large tiles (small ones are taken), 625 and 640."""
    fmt = abi.SW_PIXEL_C32
    arena, draws, verts = scenes.make_raster_scene(81, w, h, 30, blends=(0, 1, 2, 3, 4), pixel_format=fmt)
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0))
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.frame_begin(fp)
        r.set_surfaces(arena)
        r.submit_draws(draws, verts)
        got, want = np.zeros((h, w), np.uint32), np.zeros((h, w), np.uint32)
        r.render(got)
        assert oracle.rasterize(draws, verts, arena, fp, want) == 0
        assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    finally:
        r.close()
