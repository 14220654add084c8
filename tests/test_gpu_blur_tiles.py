"""The bloom blur's tiles: buffers a cell short of, equal to and a cell over 64 columns and 8 and 16 lines, at radii on
both sides of the tile height's line (8) and at the largest (16). Every frame equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.4, 1.0, 2.0, 3.0, 4.0, 8.0])
@pytest.mark.parametrize("bw,bh", [(63, 7), (64, 8), (65, 9), (64, 16), (129, 17), (4, 33), (40, 4)])
def test_tile_edges(gpu_ok, bw, bh, sigma):
    w, h = 2 * bw + 1, 2 * bh
    rng = np.random.default_rng(bw * 100 + bh)
    lanes = rng.integers(0, 65536, (h, w, 4)).astype(np.uint64) >> rng.integers(0, 12, (h, w, 1)).astype(np.uint64)
    hdr = np.ascontiguousarray(lanes[..., 0] | (lanes[..., 1] << np.uint64(16)) | (lanes[..., 2] << np.uint64(32)) | (lanes[..., 3] << np.uint64(48)))
    cfg = abi.PostConfig.default()
    cfg.bloom_buffer_scale_log2, cfg.bloom_sigma = 1, sigma
    want, _, _ = oracle.postprocess(cfg, hdr, 1.0 / 60.0, (1.0, 1.0, 1.0), 1.0)
    r = gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))
    try:
        r.set_framebuffer(hdr, abi.SW_PIXEL_C64)
        r.set_exposure(1.0)
        got = np.zeros((h, w), np.uint32)
        r.postprocess(cfg, 1.0 / 60.0, (1.0, 1.0, 1.0), out=got)
        assert np.array_equal(want, got), int((want != got).sum())
    finally:
        r.close()
