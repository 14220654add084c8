"""The tonemap's bytes where an approximate quotient could go wrong: quotients on and next to integers, black, saturated
and extreme exposures, and the linear bloom's shared columns at every scale, on widths around 4 and cell sizes. Every
frame equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu

pytestmark = pytest.mark.gpu


def _check(hdr, cfg, exposure=1.0, modulate=(1.0, 1.0, 1.0)):
    h, w = hdr.shape
    want, _, _ = oracle.postprocess(cfg, hdr, 1.0 / 60.0, modulate, exposure)
    r = gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))
    try:
        r.set_framebuffer(hdr, abi.SW_PIXEL_C64)
        r.set_exposure(exposure)
        got = np.zeros((h, w), np.uint32)
        r.postprocess(cfg, 1.0 / 60.0, modulate, out=got)
        assert np.array_equal(want, got), int((want != got).sum())
    finally:
        r.close()


def _pack(rgb):
    v = rgb.astype(np.uint64)
    return v[..., 0] | (v[..., 1] << np.uint64(16)) | (v[..., 2] << np.uint64(32)) | np.uint64(255 << 48)


@pytest.mark.parametrize("bloom", [False, True])
@pytest.mark.parametrize("exposure,modulate", [(1.0, (1.0, 1.0, 1.0)), (0.003, (1.0, 0.5, 2.0)), (128.0, (1.0, 1.0, 0.0)), (1.5e-5, (4.0, 1.0, 1e-6))])
def test_every_lane_value(gpu_ok, bloom, exposure, modulate):
    # every 16-bit value in every lane: quotients on both sides of every byte's edge
    v = np.arange(65536, dtype=np.uint64).reshape(256, 256)
    hdr = np.ascontiguousarray(_pack(np.stack([v, v[::-1], (v * 40503) & 65535], -1)))
    cfg = abi.PostConfig.default()
    if not bloom:
        cfg.bloom_scale = 0.0
    _check(hdr, cfg, exposure, modulate)


@pytest.mark.parametrize("scale_log2", [1, 2, 3])
@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("w,h", [(64, 48), (68, 50), (72, 33), (100, 61), (99, 40), (40, 17)])
def test_bloom_columns(gpu_ok, w, h, linear, scale_log2):
    rng = np.random.default_rng(w * h + scale_log2)
    rgb = rng.integers(0, 600, (h, w, 3))
    rgb[rng.random((h, w)) < 0.03] = 20000
    rgb[rng.random((h, w)) < 0.1] = 0
    cfg = abi.PostConfig.default()
    cfg.bloom_buffer_scale_log2, cfg.linear_bloom_filter, cfg.bloom_sigma = scale_log2, linear, 1.5
    _check(np.ascontiguousarray(_pack(rgb)), cfg)
