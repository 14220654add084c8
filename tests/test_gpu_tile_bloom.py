"""The bloom downscale in the tile pass, for every tile shape (64x32 tiles are drawn in two passes) and every cell size, in
frames that end inside a tile, between its passes and at its edges. Every frame equals the oracle's."""
import numpy as np
import pytest

import oracle
import scenes
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2", [1, 2, 3])
@pytest.mark.parametrize("w,h", [(64, 16), (65, 17), (127, 31), (70, 33), (100, 64), (63, 90)])
def test_every_shape(gpu_ok, w, h, log2):
    fmt = abi.SW_PIXEL_C64
    lite, draws, tv = scenes.make_triangle_draws(w + h, w, h, 40, blends=(0, 1, 2, 3, 4))
    fp = gpu.frame_params(w, h, fmt, (0, 0, 0), clear_background=True)
    hdr = np.zeros((h, w), np.uint64)
    oracle.clear_background(fp, hdr)
    assert oracle.rasterize(draws, None, None, fp, hdr, tri_vertices=tv, lite=lite) == 0
    cfg = abi.PostConfig.default()
    cfg.bloom_buffer_scale_log2 = log2
    want, _, _ = oracle.postprocess(cfg, hdr, 1.0 / 60.0, (1.0, 1.0, 1.0), 1.0)
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_lite_textures(lite)
        for shape in range(abi.SW_RASTER_TILE_VARIANTS):
            r.set_tuning(shape, 24)
            r.set_exposure(1.0)
            got = np.zeros((h, w), np.uint32)
            r.draw_frame(r.frame_input(fp, None, None, 0, draws, None, post_config=cfg, dst=got, tri_vertices=tv))
            assert np.array_equal(want, got), (shape, int((want != got).sum()))
    finally:
        r.close()
