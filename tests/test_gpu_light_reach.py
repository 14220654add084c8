"""Surface builds whose lights reach none, some or all of their texels (lights out of reach are skipped where nothing beside
them can be infinite or NaN): both lightmap kinds and pixel formats, roughness 0 and negative, normals and positions too
large for the skip, a camera in the surface's plane. The arena equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [abi.SW_PIXEL_C32, abi.SW_PIXEL_C64])
@pytest.mark.parametrize("directional", [True, False])
@pytest.mark.parametrize("inv_square_radius,scale", [(1e-8, 1.0), (1e-4, 1.0), (1e-2, 1.0), (3e38, 1.0), (1e-4, 1e-12), (1e-4, 1e10), (3e38, 1e19)])
def test_reach(gpu_ok, fmt, directional, inv_square_radius, scale):
    b = synth.BatchedSurfaces(seed=21, count=60, min_side=4, max_side=40, num_lights=6, directional=directional, pixel_format=fmt)
    rng = np.random.default_rng(9)
    b.texels = b.texels.copy()
    odd = rng.random(b.texels.size) < 0.1
    b.texels[odd] &= np.uint64(0x00FFFFFFFFFFFFFF)  # roughness 0
    odd = rng.random(b.texels.size) < 0.1
    b.texels[odd] |= np.uint64(0x8000000000000000)  # negative roughness
    d, lights = b.surfaces, b.lights.copy()
    lights["inv_square_radius"] = np.float32(inv_square_radius) * rng.uniform(0.1, 1.0, lights.size).astype(np.float32)
    for name in ("basis_u", "basis_v", "basis_normal"):
        d[name][::3] *= np.float32(scale)
    lights["position"][0] = d["basis_start"][0]  # at a texel: the smallest distance
    cam = d["basis_start"][1]
    fp = gpu.frame_params(64, 64, fmt, cam, directional=directional)
    with np.errstate(all="ignore"):
        want = oracle.build_surfaces(b.static_data(), d, lights, fp, b.total_texels, num_threads=4)
    r = gpu.GpuRenderer(b.static_data())
    try:
        r.frame_begin(fp, lights)
        r.submit_surfaces(d, b.total_texels)
        assert np.array_equal(want, r.read_surfaces(b.total_texels, fmt))
    finally:
        r.close()
