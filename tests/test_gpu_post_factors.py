"""Tonemap factors around the line from which every lane is divided exactly (divisors below the smallest normal number,
infinite factors), with and without bloom. Every frame equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.0, 1.0])
@pytest.mark.parametrize("exposure", [1e30, 8e37, 1e38, 3e38, 1e-30, 1e-38])
@pytest.mark.parametrize("modulate", [(1.0, 1.0, 1.0), (2.0, 0.25, 1e-3), (0.0, 1.0, 100.0)])
def test_extreme_factors(gpu_ok, exposure, modulate, sigma):
    h, w = 40, 64
    rng = np.random.default_rng(3)
    v = rng.integers(0, 65536, (h, w, 3)).astype(np.uint64) >> rng.integers(0, 16, (h, w, 1)).astype(np.uint64)
    v[rng.random((h, w)) < 0.2] = 0
    hdr = np.ascontiguousarray(v[..., 0] | (v[..., 1] << np.uint64(16)) | (v[..., 2] << np.uint64(32)) | np.uint64(255 << 48))
    cfg = abi.PostConfig.default()
    cfg.bloom_sigma = sigma
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
