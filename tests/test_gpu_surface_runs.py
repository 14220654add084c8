"""Surface builds whose 32-texel runs end at row and surface edges: widths around 16, 32 and 64, one- and two-row
surfaces, every lightmap scale, with one and with several runs per search. The arena equals the oracle's."""
import numpy as np
import pytest

import oracle
from sqwheel import abi, gpu, synth

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 40), (4, 9), (15, 5), (16, 4), (17, 7), (31, 3), (32, 2), (33, 3), (47, 1), (63, 2), (64, 5), (65, 4), (128, 1), (200, 3)]


@pytest.mark.parametrize("texels_per_thread", [1, 4])
@pytest.mark.parametrize("directional", [True, False])
def test_runs_at_row_and_surface_edges(gpu_ok, directional, texels_per_thread):
    fmt = abi.SW_PIXEL_C64
    b = synth.BatchedSurfaces(seed=11, count=len(SIZES) * 5, min_side=4, max_side=8, num_lights=2, directional=directional, pixel_format=fmt)
    rng = np.random.default_rng(5)
    d = b.surfaces
    lm_end, off = 1, 0
    for i in range(d.size):
        w, h = SIZES[i % len(SIZES)]
        log2 = i // len(SIZES)  # 0..4
        shift = rng.integers(0, 1 << log2, 2)
        lm = [((s - 1 + int(t)) >> log2) + 2 for s, t in zip((w, h), shift)]
        d[i]["size"], d[i]["lightmap_scale_log2"], d[i]["lightmap_tc_shift"], d[i]["lightmap_size"] = (w, h), log2, shift, lm
        d[i]["lightmap_offset"] = lm_end if i % 7 else abi.SW_NO_LIGHTMAP
        d[i]["out_offset"] = off
        lm_end += lm[0] * lm[1]
        off += w * h
    if directional:
        b.directional_lightmaps = synth.random_directional_lightmap(rng, lm_end)
    else:
        b.lightmaps = rng.uniform(0, 4, (lm_end, 3)).astype(np.float32)
    order = rng.permutation(d.size)
    d = np.ascontiguousarray(d[order])
    fp = gpu.frame_params(64, 64, fmt, b.cam_pos, directional=directional)
    want = oracle.build_surfaces(b.static_data(), d, b.lights, fp, off, num_threads=4)
    r = gpu.GpuRenderer(b.static_data())
    try:
        r.set_tuning(0, 24, texels_per_thread)
        r.frame_begin(fp, b.lights)
        r.submit_surfaces(d, off)
        assert np.array_equal(want, r.read_surfaces(off, fmt))
    finally:
        r.close()
