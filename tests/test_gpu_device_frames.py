"""Raster-only frames in device memory: every call that delivers one (sw_render, sw_draw_frame through the graph and
without it, sw_draw_frame_view) writes the same frame as to host memory, both pixel formats, padded pitches, at the pixel's
own alignment (the tile pass stores it) and at other byte addresses and in page-locked memory (it is copied), and
nothing between the rows or behind them."""
import numpy as np
import pytest

import scenes
from sqwheel import abi, gpu, host, synth

pytestmark = pytest.mark.gpu

W, H = 97, 35
# byte offset of the destination, extra pixels per row
PLACES = [(0, 0), (0, 5), (8, 3), (4, 0), (4, 3), (2, 1), (1, 0), (3, 2)]


def _buffer(fmt, offset, pad, pinned=False):
    import torch
    bpp = 8 if fmt == abi.SW_PIXEL_C64 else 4
    pitch = W + pad
    n = offset + pitch * H * bpp + 64
    t = torch.full((n,), 0xA5, dtype=torch.uint8, pin_memory=True) if pinned else torch.full((n,), 0xA5, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()  # the context's stream does not wait for torch's
    return t, t.data_ptr() + offset, pitch


def _check(t, offset, pad, want):
    raw = t.cpu().numpy()
    bpp = want.itemsize
    rows = raw[offset:offset + (W + pad) * H * bpp].reshape(H, (W + pad) * bpp)
    got = np.ascontiguousarray(rows[:, :W * bpp]).view(want.dtype)
    assert np.array_equal(want, got), f"{(want != got).sum()} pixels differ"
    assert np.all(rows[:, W * bpp:] == 0xA5) and np.all(raw[:offset] == 0xA5) and np.all(raw[offset + rows.size:] == 0xA5)


@pytest.mark.parametrize("fmt", [abi.SW_PIXEL_C32, abi.SW_PIXEL_C64])
def test_submitted_and_graph_frames(gpu_ok, fmt):
    arena, draws, verts = scenes.make_raster_scene(91, W, H, 14, blends=(0, 1, 2, 3, 4), pixel_format=fmt)
    lite, triangles, tv = scenes.make_triangle_draws(92, W, H, 20)
    fp = gpu.frame_params(W, H, fmt, (0, 0, 0))
    dt = np.uint64 if fmt == abi.SW_PIXEL_C64 else np.uint32
    r = gpu.GpuRenderer(synth.BatchedSurfaces(seed=1, count=1, max_side=8).static_data())
    try:
        r.set_lite_textures(lite)
        want = np.zeros((H, W), dt)
        for offset, pad in PLACES:
            for pinned in (False, True):
                # the same draws into host memory from the same frame buffer (it carries over from frame to frame)
                start = r.read_framebuffer(W, H, fmt) if want.any() else want.copy()
                r.frame_begin(fp)
                r.set_surfaces(arena)
                r.submit_draws(draws, verts)
                r.set_framebuffer(start, fmt)
                r.render(want)
                t, ptr, pitch = _buffer(fmt, offset, pad, pinned)
                r.frame_begin(fp)
                r.set_surfaces(arena)
                r.submit_draws(draws, verts)
                r.set_framebuffer(start, fmt)
                r.render(device_ptr=ptr, pitch=pitch)
                r.sync()
                _check(t, offset, pad, want)
        for graph in (True, False):
            r.set_frame_graph(graph)
            for offset, pad in PLACES:  # one graph, whose delivery changes from frame to frame
                r.set_framebuffer(np.zeros((H, W), dt), fmt)
                r.draw_frame(r.frame_input(fp, None, None, 0, triangles, None, dst=want, tri_vertices=tv))
                t, ptr, pitch = _buffer(fmt, offset, pad)
                r.set_framebuffer(np.zeros((H, W), dt), fmt)
                r.draw_frame(r.frame_input(fp, None, None, 0, triangles, None, dst_device_ptr=ptr, pitch=pitch, tri_vertices=tv))
                r.sync()
                _check(t, offset, pad, want)
    finally:
        r.close()


@pytest.mark.parametrize("fmt", [abi.SW_PIXEL_C32, abi.SW_PIXEL_C64])
def test_view_frames(gpu_ok, fmt):
    scene = host.Scene(**host.SMALL_MAP)
    opts = host.frame_options(W, H, fmt, directional=fmt == abi.SW_PIXEL_C64)
    want = np.zeros((H, W), np.uint64 if fmt == abi.SW_PIXEL_C64 else np.uint32)
    rd, rh = host.HostRenderer(scene), host.HostRenderer(scene)
    try:
        for i, (offset, pad) in enumerate(PLACES):
            rh.render_frame(3 * i, opts, out=want)
            t, ptr, pitch = _buffer(fmt, offset, pad)
            rd.render_frame(3 * i, opts, device_ptr=ptr, pitch=pitch)
            rd.sync()
            _check(t, offset, pad, want)
    finally:
        rd.close()
        rh.close()
