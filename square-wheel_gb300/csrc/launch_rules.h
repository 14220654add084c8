// Decisions of the host about where and how a kernel is launched, as functions of sizes and of what the driver reports:
// plain C++, so that they can be checked over their whole range without a GPU.
#pragma once

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
