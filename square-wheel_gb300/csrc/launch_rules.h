// Decisions of the host about where and how a kernel is launched, as functions of sizes and of what the driver reports:
// plain C++, so that they can be checked over their whole range without a GPU.
#pragma once

#include <algorithm>
#include <cstdint>

namespace swgpu
{

// Tile shapes of the tile pass, as SwTuning.raster_tile numbers them: w x h pixels, 256 threads with `strip` pixels each
// at a time, `passes` times one below the other. Every shape gives the same frame.
struct TileShape
{
	int w, h, strip, passes;
};
constexpr uint32_t NUM_TILE_SHAPES = 5;
constexpr TileShape TILE_SHAPES[NUM_TILE_SHAPES] = {{64, 16, 4, 1}, {32, 32, 4, 1}, {128, 8, 4, 1}, {64, 32, 4, 2}, {32, 16, 2, 1}};

// Whether the bins' lists are made by a CTA for eight bins instead of one for each: where a CTA per bin is more than the GPU
// holds at once (eight per SM). There every box is read again for every bin from L2 (5,822 bins of 4,100 draws: 64 us,
// 17 with eight bins per CTA; 1,280 bins of 2,400 draws 13.0 and 9.7). With fewer bins it depends on the draws: 1,020 bins
// of 2,400 small polygons take 10.3 and 9.7 us, of 2,363 draws with triangles among them 9.7 and 12.0, a 1366x768
// frame 3.5 and 4.9.
inline bool bins_in_groups(uint32_t bins, uint32_t num_sms) { return bins > num_sms * 8; }

// Whether the raster setup takes a warp per draw instead of a CTA. With 2,400 small draws a CTA each takes 45 us and a warp
// each 12, with draws of up to 360 rows 49 and 21; at 1,000 of those it is 26 and 20, at 400 16 and 20. At 512 draws
// a lone pass of a frame is 8% slower with a warp each (100 us against 92), although overlapped passes gain 9%; at
// 300 a lone frame loses 11% and overlapped ones gain nothing.
inline bool warp_per_draw(uint32_t draws) { return draws >= 1024; }

// Runs of 32 texels that a warp of the surface build takes per search: the tuned number (SwTuning.surface_texels_per_thread,
// 1 or 4), or with 0 by the work: one while the launch is not several times what the GPU holds at once (a frame's 0.6 M
// texels hide latency by parallelism), up to 8 for large batches.
inline uint32_t surface_runs(uint32_t tuned, uint64_t work, int num_sms)
{
	if (tuned) return tuned;
	const uint64_t resident = uint64_t(num_sms) * 2048 * 2;
	return uint32_t(std::min<uint64_t>(std::max<uint64_t>(work / resident, 1), 8));
}

// What the driver reports about a pointer of the caller's.
struct PointerInfo
{
	bool device_memory; // memory of a device (not the host's)
	bool managed;
	bool writable;       // by kernels of the context's device
	bool own_context;    // allocated in the current context, or in none (memory pools, virtual memory)
	int device;          // whose memory it is
	uint64_t begin, bytes; // the allocation
};

// Whether kernels on `device` may store a frame of width x height pixels of `bpp` bytes, `pitch` pixels per row, at `dst`
// pixel by pixel: whole pixels at their natural alignment in writable memory of that device, all inside one allocation.
// Anything else a device destination may be (another device's memory, managed or page-locked memory, any byte address)
// is left to a copy, which takes it or reports it; a kernel's store would fault.
inline bool can_store_frame(const PointerInfo& p, int device, uint64_t dst, uint32_t pitch, uint32_t width, uint32_t height, uint32_t bpp)
{
	if (dst % bpp != 0 || !p.device_memory || p.managed || !p.writable || !p.own_context || p.device != device) return false;
	const uint64_t span = ((uint64_t(height) - 1) * pitch + width) * bpp;
	return dst >= p.begin && span <= p.bytes && dst - p.begin <= p.bytes - span;
}

} // namespace swgpu
