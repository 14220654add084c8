"""The host's launch decisions (csrc/launch_rules.h) over their ranges, compiled for the CPU."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "square-wheel_gb300", "csrc")
SHIM = r"""
#include "launch_rules.h"
using namespace swgpu;
extern "C" int store_frame(int device_memory, int managed, int writable, int own_context, int memory_device, uint64_t begin, uint64_t bytes,
	int device, uint64_t dst, uint32_t pitch, uint32_t width, uint32_t height, uint32_t bpp)
{
	const PointerInfo p{device_memory != 0, managed != 0, writable != 0, own_context != 0, memory_device, begin, bytes};
	return can_store_frame(p, device, dst, pitch, width, height, bpp) ? 1 : 0;
}
extern "C" uint32_t runs(uint32_t tuned, uint64_t work, int num_sms) { return surface_runs(tuned, work, num_sms); }
extern "C" int groups(uint32_t bins, uint32_t num_sms) { return bins_in_groups(bins, num_sms) ? 1 : 0; }
extern "C" int warp_draws(uint32_t draws) { return warp_per_draw(draws) ? 1 : 0; }
extern "C" uint32_t num_shapes() { return NUM_TILE_SHAPES; }
extern "C" void shape(uint32_t i, int* s) { s[0] = TILE_SHAPES[i].w, s[1] = TILE_SHAPES[i].h, s[2] = TILE_SHAPES[i].strip, s[3] = TILE_SHAPES[i].passes; }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, lib = d / "rules.cpp", d / "librules.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    so = ctypes.CDLL(str(lib))
    so.store_frame.argtypes = [ctypes.c_int] * 5 + [ctypes.c_uint64] * 2 + [ctypes.c_int, ctypes.c_uint64] + [ctypes.c_uint32] * 4
    so.runs.argtypes = [ctypes.c_uint32, ctypes.c_uint64, ctypes.c_int]
    return so


BASE, SIZE = 1 << 40, 1 << 20


def _store(rules, device_memory=1, managed=0, writable=1, own_context=1, memory_device=0, begin=BASE, size=SIZE, device=0, dst=BASE,
           pitch=64, width=64, height=32, bpp=8):
    return rules.store_frame(device_memory, managed, writable, own_context, memory_device, begin, size, device, dst, pitch, width, height, bpp)


@pytest.mark.parametrize("bpp", [4, 8])
def test_device_destinations_that_kernels_store_to(rules, bpp):
    for off in range(0, 33):
        assert _store(rules, dst=BASE + off, bpp=bpp) == (off % bpp == 0), off
    # other memory than the context's device's is copied to
    assert not _store(rules, device_memory=0, bpp=bpp)
    assert not _store(rules, managed=1, bpp=bpp)
    assert not _store(rules, writable=0, bpp=bpp)
    assert not _store(rules, own_context=0, bpp=bpp)
    assert not _store(rules, memory_device=1, bpp=bpp) and _store(rules, memory_device=1, device=1, bpp=bpp)
    # the frame's last pixel is the allocation's last, or one past it
    for pitch, width, height in ((64, 64, 1), (64, 64, 32), (100, 64, 33), (64, 1, 7), (1 << 31, 3, 1), (16384, 16384, 16384)):
        span = ((height - 1) * pitch + width) * bpp
        for dst in (BASE, BASE + 16 * bpp):
            fits = dict(dst=dst, pitch=pitch, width=width, height=height, bpp=bpp)
            assert _store(rules, size=dst - BASE + span, **fits)
            assert not _store(rules, size=dst - BASE + span - 1, **fits)
        assert not _store(rules, dst=BASE - bpp, size=1 << 45, pitch=pitch, width=width, height=height, bpp=bpp)
    assert not _store(rules, size=0, bpp=bpp)


def test_tile_shapes_are_the_ones_the_tuning_names(rules):
    """SwTuning.raster_tile's shapes; no thread has more than four pixels at a time (longer code is fetched more slowly than
    it saves), and no bloom cell (up to 8 x 8 pixels) straddles two passes."""
    sizes = [(64, 16), (32, 32), (128, 8), (64, 32), (32, 16)]
    assert rules.num_shapes() == len(sizes)
    s = (ctypes.c_int * 4)()
    for i, (w, h) in enumerate(sizes):
        rules.shape(i, s)
        assert tuple(s[:2]) == (w, h) and s[2] <= 4 and 256 * s[2] * s[3] == w * h and h % s[3] == 0 and h // s[3] % 8 == 0


def test_tuned_surface_runs_are_what_they_say(rules):
    for work in (1, 1 << 20, 1 << 26, 1 << 40):
        assert rules.runs(1, work, 152) == 1 and rules.runs(4, work, 152) == 4
    assert [rules.runs(0, w, 152) for w in (0, 1, 622592, 2 * 622592 - 1, 2 * 622592, 8 * 622592, 1 << 50)] == [1, 1, 1, 1, 2, 8, 8]


def test_bins_go_to_groups_where_a_cta_each_does_not_fit(rules):
    for num_sms in (1, 76, 132, 152, 160):
        assert [rules.groups(n, num_sms) for n in (1, 8 * num_sms - 1, 8 * num_sms, 8 * num_sms + 1, 1 << 20)] == [0, 0, 0, 1, 1]


def test_draws_get_a_warp_each_from_a_count_on(rules):
    assert [rules.warp_draws(n) for n in (0, 1, 300, 1023, 1024, 1 << 20)] == [0, 0, 0, 0, 1, 1]
