// Learned 2x upscaler (include/swlearn.h): tcgen05 implicit-GEMM 3x3 convolutions (forward, input
// gradient, weight gradient), the pixel-shuffle / bilinear-residual / loss epilogue, Adam, PSNR.
//
// Activation layout in HBM ("row planes"): per image, per row (one halo row above, zero rows below),
// per 8-channel chunk, per pixel (one halo pixel left, zero pixels right) 8 bf16 = 16 bytes:
//   element (img, y, chunk, x, e) at ((img * rows_alloc + y + 1) * chunks + chunk) * wp * 8 + (x + 1) * 8 + e
// A row of 128 pixels of one chunk is therefore 128 contiguous 16-byte rows, which is exactly a stack of
// 16 UMMA core matrices (8 pixels x 16 bytes): an M tile of the implicit GEMM is 128 consecutive pixels of
// one image row, and a tap (dy, dx) of the 3x3 kernel only moves the descriptor's start address. Halo and
// padding pixels are zeroed once at allocation and never written, which gives the zero padding of the
// convolution and of its transpose.
//
// conv_kernel: persistent CTAs with rows of 128 pixels of their own; input rows come in by tiled TMA, their MMAs of
// 128 x 3N x 16 accumulate into a ring of output rows in TMEM, and epilogue warps (warp w = TMEM lanes 32 * (w % 4)..,
// i.e. pixels) apply bias + ReLU (forward), the ReLU mask (input gradient) or the output stage (pixel shuffle +
// bilinear residual, written as Color32 for inference or as the loss gradient for training).
// wgrad_kernel: weight gradient dW[co][dy][dx][ci] = sum_p G[p][co] X[p + (dy, dx)][ci] with both operands
// MN-major: D rows = (input row, chunk, ci % 8) groups at a uniform shared-memory stride, D columns = (gradient row,
// co), one accumulator per dx, K = 16 pixels per MMA; per-CTA partial sums are reduced in a fixed order.
#include "sw_kernels.cuh"
#include "tc05.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "../../include/swlearn.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

using namespace swgpu;
using namespace swgpu::tc05;

namespace
{

constexpr int TILE_X = 128;            // pixels per M tile
constexpr int ROWS = 4;                // output rows per CTA
constexpr uint32_t POLL_LIMIT = 1u << 21;
constexpr int NUM_LAYERS = 4;

// Layer shapes: real channel counts and the padded ones the MMAs use.
struct LayerShape
{
	int cin, cout;     // real
	int c8_in, n_out;  // input chunks (8 channels each), padded output channels
	int param_offset;  // weights, then bias at param_offset + cout*9*cin
};
constexpr LayerShape LAYERS[NUM_LAYERS] = {
	{3, 32, 2, 32, 0},
	{32, 32, 4, 32, 896},
	{32, 32, 4, 32, 896 + 9248},
	{32, 12, 4, 16, 896 + 2 * 9248},
};
static_assert(896 + 2 * 9248 + 3468 == SW_UPSCALER_NUM_PARAMS, "parameter count");
__constant__ LayerShape c_layers[NUM_LAYERS] = {
	{3, 32, 2, 32, 0},
	{32, 32, 4, 32, 896},
	{32, 32, 4, 32, 896 + 9248},
	{32, 12, 4, 16, 896 + 2 * 9248},
};

struct Planes
{
	uint16_t* data; // bf16 bits
	uint32_t images, height, width, chunks, wp, rows_alloc;
};

__host__ __device__ __forceinline__ size_t planes_index(const Planes& p, uint32_t img, int y, uint32_t chunk, int x)
{
	return ((size_t(img) * p.rows_alloc + size_t(y + 1)) * p.chunks + chunk) * p.wp * 8 + size_t(x + 1) * 8;
}

struct CropGpu
{
	const uint32_t* lo;
	const uint32_t* hi;
	uint32_t lo_w, lo_h, lo_pitch, hi_pitch;
	int32_t x, y;
};

enum Epi
{
	EPI_RELU = 0,  // out = bf16(max(acc + bias, 0))
	EPI_MASK = 1,  // out = bf16(acc * (mask > 0))
	EPI_INFER = 2, // Color32 output frame
	EPI_LOSS = 3,  // loss gradient planes + loss partial sums
};

struct ConvArgs
{
	CUtensorMap in_map; // rows of `in`: box = 8 channels x 130 pixels x all chunks x 1 row
	Planes in, out, mask;
	const uint16_t* wpack;
	const float* bias;
	const CropGpu* crops; // EPI_INFER / EPI_LOSS: one per image
	uint32_t* hi_out;     // EPI_INFER
	uint32_t hi_pitch;
	float* loss_partial; // EPI_LOSS: one per CTA
	uint32_t margin;
	int* error;
};

__device__ __forceinline__ uint16_t f2bf(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float bf2f(uint16_t h) { return __uint_as_float(uint32_t(h) << 16); }
__device__ __forceinline__ uint32_t pack2(float a, float b) { return uint32_t(f2bf(a)) | (uint32_t(f2bf(b)) << 16); }

__device__ __forceinline__ uint32_t to_byte(float v)
{
	const float s = rintf(v * 255.0f);
	return uint32_t(fminf(fmaxf(s, 0.0f), 255.0f));
}

// Byte k of w as a float, and the clamped and rounded byte of a value as the low byte of the result, without the
// conversion unit (a quarter of the other pipes' rate): 2^23 + b is exact for a byte, and adding 2^23 to a value
// in [0, 255] rounds it to the nearest even integer. The bounds are integers, so clamping first changes nothing.
template <int k>
__device__ __forceinline__ float byte_float(uint32_t w)
{
	return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | k)) - 8388608.0f;
}
__device__ __forceinline__ uint32_t float_byte(float v)
{
	return __float_as_uint(fminf(fmaxf(v * 255.0f, 0.0f), 255.0f) + 8388608.0f);
}

constexpr int NSTAGE = 6;    // input rows staged in shared memory (ring)
constexpr int CONV_RING = 8; // TMEM output-row accumulators of the convolution

// Staged input row of the convolution: pixels x0 - 1 .. x0 + 134 of every chunk (17 groups of 8 pixels;
// pixel x0 - 1 starts a 128-byte group because of the layout's one-pixel halo offset), so the TMA box's
// innermost extent is a whole 128-byte group of 8 pixels x 8 channels.
constexpr int CXS = 136;
constexpr uint32_t CXS_BYTES = CXS * 16; // 2176: chunk stride of a staged row
// Ring slot of one staged input row: a tiled TMA destination must be 128-byte aligned.
template <int C8>
__host__ __device__ constexpr uint32_t conv_slot_bytes()
{
	return (C8 * CXS_BYTES + 127) / 128 * 128;
}
template <int C8, int N>
__host__ __device__ constexpr uint32_t conv_smem_bytes()
{
	return NSTAGE * conv_slot_bytes<C8>() + 9 * (C8 / 2) * 2 * N * 16 + 512;
}
template <int N>
__host__ __device__ constexpr uint32_t conv_tmem_cols()
{
	return CONV_RING * N <= 128 ? 128 : 256;
}

// Rows [begin, end) of the (strip, y) order a persistent CTA owns; strip = image * tiles_x + x tile.
struct RowRange
{
	uint32_t begin, end;
};
__device__ __forceinline__ RowRange cta_rows(uint32_t total)
{
	return RowRange{uint32_t(uint64_t(blockIdx.x) * total / gridDim.x), uint32_t(uint64_t(blockIdx.x + 1) * total / gridDim.x)};
}

// What the epilogue of one output pixel reads from global memory: the stored activations whose sign gates the gradient
// (EPI_MASK), the source pixels of the bilinear upsample (EPI_INFER, EPI_LOSS) and the four target pixels (EPI_LOSS).
// None of it depends on the accumulators, so it is loaded before the wait for them.
template <int N, int EPI>
struct EpiOperands
{
	uint4 mask[EPI == EPI_MASK ? N / 8 : 1];
	uint32_t src[EPI == EPI_INFER || EPI == EPI_LOSS ? 9 : 1]; // rows y - 1, y, y + 1, columns x - 1, x, x + 1, edges clamped
	uint2 target[EPI == EPI_LOSS ? 2 : 1];
};

template <int N, int EPI>
__device__ __forceinline__ void load_operands(const ConvArgs& a, uint32_t img, int x, int y, EpiOperands<N, EPI>& op)
{
	if (x >= int(a.in.width) || y >= int(a.in.height)) return;
	if (EPI == EPI_MASK)
	{
		const uint16_t* msk = a.mask.data + planes_index(a.mask, img, y, 0, x);
#pragma unroll
		for (int c8 = 0; c8 < N / 8; ++c8) op.mask[c8] = *reinterpret_cast<const uint4*>(msk + c8 * (size_t(a.mask.wp) * 8));
	}
	else if (EPI == EPI_INFER || EPI == EPI_LOSS)
	{
		const CropGpu c = a.crops[img];
		const int lx = c.x + x, ly = c.y + y;
		const int xs[3] = {max(lx - 1, 0), lx, min(lx + 1, int(c.lo_w) - 1)};
		const int ys[3] = {max(ly - 1, 0), ly, min(ly + 1, int(c.lo_h) - 1)};
#pragma unroll
		for (int j = 0; j < 3; ++j)
#pragma unroll
			for (int i = 0; i < 3; ++i) op.src[j * 3 + i] = c.lo[size_t(ys[j]) * c.lo_pitch + xs[i]];
		if (EPI == EPI_LOSS)
#pragma unroll
			for (int sy = 0; sy < 2; ++sy)
				op.target[sy] = *reinterpret_cast<const uint2*>(c.hi + size_t(2 * ly + sy) * c.hi_pitch + 2 * lx);
	}
}

// Epilogue of channels c0 .. c0 + 15 of one output pixel: v = their accumulators, bias = theirs.
template <int N, int EPI>
__device__ __forceinline__ void conv_epilogue(const ConvArgs& a, const EpiOperands<N, EPI>& op, const float (&v)[16],
	const float* bias, int c0, uint32_t img, int x, int y, float& loss)
{
	if (x >= int(a.in.width) || y >= int(a.in.height)) return; // padding pixels stay zero
	if (EPI == EPI_RELU || EPI == EPI_MASK)
	{
		const size_t cstride = size_t(a.out.wp) * 8;
		uint16_t* out = a.out.data + planes_index(a.out, img, y, 0, x) + (c0 / 8) * cstride;
#pragma unroll
		for (int c8 = 0; c8 < 2; ++c8)
		{
			uint32_t o[4];
			if (EPI == EPI_RELU)
			{
#pragma unroll
				for (int q = 0; q < 4; ++q)
					o[q] = pack2(fmaxf(v[c8 * 8 + 2 * q] + bias[c0 + c8 * 8 + 2 * q], 0.0f),
						fmaxf(v[c8 * 8 + 2 * q + 1] + bias[c0 + c8 * 8 + 2 * q + 1], 0.0f));
			}
			else
			{
				const uint4 m = op.mask[EPI == EPI_MASK ? c0 / 8 + c8 : 0];
				const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
				for (int q = 0; q < 4; ++q)
				{
					// ReLU derivative: the stored activation is > 0 (sign clear, magnitude non-zero)
					const float g0 = (mw[q] & 0x7FFFu) && !(mw[q] & 0x8000u) ? v[c8 * 8 + 2 * q] : 0.0f;
					const float g1 = (mw[q] & 0x7FFF0000u) && !(mw[q] & 0x80000000u) ? v[c8 * 8 + 2 * q + 1] : 0.0f;
					o[q] = pack2(g0, g1);
				}
			}
			*reinterpret_cast<uint4*>(out + c8 * cstride) = make_uint4(o[0], o[1], o[2], o[3]);
		}
	}
	else
	{
		// Output stage: channel c*4 + sy*2 + sx is colour c of output pixel (2x + sx, 2y + sy), added to
		// the bilinear 2x upsample of the source (weights 3/4, 1/4; edges clamped).
		float g[16];
#pragma unroll
		for (int j = 0; j < 16; ++j) g[j] = 0.0f;
		const bool in_loss = EPI == EPI_LOSS && x >= int(a.margin) && x < int(a.in.width - a.margin) &&
			y >= int(a.margin) && y < int(a.in.height - a.margin);
		const uint32_t p11 = op.src[4], p10 = op.src[3], p12 = op.src[5];
#pragma unroll
		for (int sy = 0; sy < 2; ++sy)
		{
			const uint32_t p21 = op.src[sy ? 7 : 1], p20 = op.src[sy ? 6 : 0], p22 = op.src[sy ? 8 : 2];
			const uint32_t tp[2] = {op.target[EPI == EPI_LOSS ? sy : 0].x, op.target[EPI == EPI_LOSS ? sy : 0].y};
			uint32_t px[2];
#pragma unroll
			for (int sx = 0; sx < 2; ++sx)
			{
				const int s = sy * 2 + sx;
				const uint32_t a01 = sx ? p12 : p10, a11 = sx ? p22 : p20;
				uint32_t bytes = p11 & 0xFF000000u; // alpha of the source pixel
#pragma unroll
				for (int ch = 0; ch < 3; ++ch)
				{
					const float top = 0.75f * float((p11 >> (8 * ch)) & 255u) + 0.25f * float((a01 >> (8 * ch)) & 255u);
					const float bot = 0.75f * float((p21 >> (8 * ch)) & 255u) + 0.25f * float((a11 >> (8 * ch)) & 255u);
					const float pred = (0.75f * top + 0.25f * bot) * (1.0f / 255.0f) + (v[ch * 4 + s] + bias[ch * 4 + s]);
					if (EPI == EPI_INFER)
						bytes |= to_byte(pred) << (8 * ch);
					else
					{
						const float d = in_loss ? pred - float((tp[sx] >> (8 * ch)) & 255u) * (1.0f / 255.0f) : 0.0f;
						g[ch * 4 + s] = d;
						loss += d * d;
					}
				}
				px[sx] = bytes;
			}
			if (EPI == EPI_INFER)
				*reinterpret_cast<uint2*>(a.hi_out + size_t(2 * (a.crops[img].y + y) + sy) * a.hi_pitch + 2 * (a.crops[img].x + x)) =
					make_uint2(px[0], px[1]);
		}
		if (EPI == EPI_LOSS)
		{
			uint16_t* out = a.out.data + planes_index(a.out, img, y, 0, x);
#pragma unroll
			for (int c8 = 0; c8 < 2; ++c8)
			{
				uint32_t o[4];
#pragma unroll
				for (int q = 0; q < 4; ++q) o[q] = pack2(g[c8 * 8 + 2 * q], g[c8 * 8 + 2 * q + 1]);
				*reinterpret_cast<uint4*>(out + c8 * size_t(a.out.wp) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
			}
		}
	}
}

// Persistent, warp-specialised 3x3 convolution over row planes (CONV_THREADS = 320 threads). The three
// vertical taps are folded into the MMA's N dimension: input row y_in times the weights of all three ky
// gives, for output rows y_in + 1, y_in, y_in - 1, their ky = 0, 1, 2 contributions side by side
// (N = 3 x C_out), accumulated in place into a TMEM ring of R output-row accumulators (C_out columns
// each; the row with counter o sits at block (R - o % R) % R, so rows y_in + 1, y_in, y_in - 1 are
// consecutive blocks; a group that wraps the ring is split in two MMAs). Accumulators start at zero
// (the epilogue zeroes each one after reading it), so every MMA accumulates. One input row is read by
// 3 x (C8 / 2) MMAs of 128 x 3N x 16 and released; an output row is complete after input row y + 1.
//   warp 0 (one lane): bulk-copies the packed weights once, then loads input rows (all chunks, 136
//     pixels; one tiled TMA each) into a ring of NSTAGE shared-memory rows;
//   warp 1 (lane 0 issues; the warp owns the TMEM allocation): per input row waits for it (and, when it
//     starts a new output row, for that row's accumulator to be free), issues the MMAs and commits the
//     row to rowbar[k % NBAR]: that releases the input row's slot and completes output row y_in - 1;
//   warps 2..9: two groups of four (warp w reads TMEM lanes 32*(w%4).., i.e. pixels) taking alternate output
//     rows: what the row's epilogue reads from global memory is loaded first, then TMEM -> registers, the
//     accumulator is zeroed and released, and the epilogue stores the row.
// The issuing thread's own instruction latency bounds the MMA rate, so the common case (three
// contributions, no ring wrap) is straight-line code with compile-time descriptor offsets.
// At a training step's sizes a CTA has three or four rows, so the kernel is bound by the latency of one row's chain
// (load, MMAs, epilogue). With all eight warps on one row and the operands loaded after the accumulators a training
// step of 16 crops (150 us) takes 18 us longer.
// Every wait is bounded: on expiry the role stops, the error flag is set, and the CTA still waits for
// its own MMAs and copies before freeing TMEM.
constexpr int CONV_THREADS = 320;
constexpr int CONV_EPI_WARPS = 8;
constexpr int NBAR = 16; // row-completion barriers (more than the rows the MMA issuer can run ahead)

template <int C8, int N, int EPI>
__global__ void __launch_bounds__(CONV_THREADS, 2) conv_kernel(const __grid_constant__ ConvArgs a)
{
	constexpr int KSTEPS = C8 / 2;      // 16-channel steps per horizontal tap
	constexpr int NB = 3 * N;           // MMA N for a whole input row
	constexpr int R = CONV_RING;        // TMEM output-row accumulators
	constexpr uint32_t ROW_BYTES = C8 * CXS_BYTES;       // bytes of one staged row (the TMA box)
	constexpr uint32_t SLOT_BYTES = conv_slot_bytes<C8>(); // ring stride (128-byte aligned)
	constexpr uint32_t W_BYTES = 3 * KSTEPS * 2 * NB * 16;
	constexpr uint32_t TMEM_COLS = conv_tmem_cols<N>();
	static_assert(C8 % 2 == 0 && N % 16 == 0 && N <= 32, "shape");
	extern __shared__ __align__(1024) unsigned char smem[];
	unsigned char* s_ring = smem;
	unsigned char* s_w = smem + NSTAGE * SLOT_BYTES;
	uint64_t* full = reinterpret_cast<uint64_t*>(s_w + W_BYTES);
	uint64_t* rowbar = full + NSTAGE;
	uint64_t* acce = rowbar + NBAR;
	uint64_t* wbar = acce + R;
	uint64_t* donebar = wbar + 1;
	uint32_t* s_tmem = reinterpret_cast<uint32_t*>(donebar + 1);
	float* s_red = reinterpret_cast<float*>(s_tmem + 4); // [CONV_EPI_WARPS]
	float* s_bias = s_red + CONV_EPI_WARPS;              // [N]

	const int tid = threadIdx.x, lane = tid & 31;
	const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0); // known to be the same in the whole warp
	const uint32_t H = a.in.height;
	const uint32_t tiles_x = (a.in.width + TILE_X - 1) / TILE_X;
	const RowRange rows = cta_rows(a.in.images * tiles_x * H);

	if (tid == 0)
	{
		for (int i = 0; i < NSTAGE; ++i) mbar_init(&full[i], 1);
		for (int i = 0; i < NBAR; ++i) mbar_init(&rowbar[i], 1);
		for (int i = 0; i < R; ++i) mbar_init(&acce[i], CONV_EPI_WARPS / 2);
		mbar_init(wbar, 1);
		mbar_init(donebar, 1);
		fence_mbar_init();
	}
	if (warp == 1)
	{
		tmem_alloc(s_tmem, TMEM_COLS);
		tmem_relinquish();
	}
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);
	if (warp >= 2)
	{
		// every accumulator starts at zero (the MMAs always accumulate)
		const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
		const int half = (warp - 2) >> 2;
		for (int c = half * (R * N / 2); c < (half + 1) * (R * N / 2); c += 8) tmem_zero8(tmem + lane_base + c);
		tmem_st_wait();
	}
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	bool failed = false;
	// everything above touched only the SM: it overlaps the end of the kernel before. The next kernel may be
	// scheduled from here on (this one's TMEM is allocated); it waits for this grid before it reads or writes.
	pdl_trigger();
	pdl_wait();

	if (warp == 0)
	{
		if (lane == 0)
		{
			mbar_expect_tx(wbar, W_BYTES);
			bulk_g2s(s_w, a.wpack, W_BYTES, wbar);
			uint32_t k = 0;
			for (uint32_t r = rows.begin; r < rows.end && !failed;)
			{
				const uint32_t strip = r / H, y_lo = r % H, y_hi = min(H, y_lo + (rows.end - r));
				r += y_hi - y_lo;
				const uint32_t img = strip / tiles_x;
				const int x0 = int(strip % tiles_x) * TILE_X;
				for (int yi = int(y_lo) - 1; yi <= int(y_hi); ++yi, ++k)
				{
					const uint32_t slot = k % NSTAGE;
					if (k >= NSTAGE)
					{
						// the slot's previous row (k - NSTAGE) has been consumed by its MMAs
						const uint32_t kp = k - NSTAGE;
						if (!mbar_wait_bounded(&rowbar[kp % NBAR], (kp / NBAR) & 1, POLL_LIMIT))
						{
							failed = true;
							break;
						}
					}
					mbar_expect_tx(&full[slot], ROW_BYTES);
					// one tiled TMA per input row: pixels x0 - 1 .. x0 + 134 of all chunks
					tma_load_4d(s_ring + slot * SLOT_BYTES, &a.in_map, 0, x0 / 8, 0, int(img * a.in.rows_alloc) + yi + 1, &full[slot]);
				}
			}
			// drain: the last fill of every slot has landed before the CTA can exit
			for (uint32_t kk = k > NSTAGE ? k - NSTAGE : 0; kk < k; ++kk)
				mbar_wait_bounded(&full[kk % NSTAGE], (kk / NSTAGE) & 1, POLL_LIMIT);
		}
	}
	else if (warp == 1)
	{
		{
			const uint32_t issue = lane == 0 ? 1u : 0u; // the whole warp runs the role, lane 0 issues
			// Descriptors are precomputed: the start-address field is the low 14 bits (address >> 4), so a
			// descriptor of base + off is the base descriptor + (off >> 4) (shared addresses stay < 256 KB).
			const uint64_t a_base = make_sdesc(smem_addr(s_ring), CXS_BYTES, 128);
			const uint64_t b_base = make_sdesc(smem_addr(s_w), NB * 16, 128);
			constexpr uint32_t IDESC1 = make_idesc_bf16(128, N, 0, 0);
			constexpr uint32_t IDESC2 = make_idesc_bf16(128, 2 * N, 0, 0);
			constexpr uint32_t IDESC3 = make_idesc_bf16(128, 3 * N, 0, 0);
			failed = !mbar_wait_warp(wbar, 0, POLL_LIMIT);
			uint32_t k = 0, o_base = 0;
			for (uint32_t r = rows.begin; r < rows.end && !failed;)
			{
				const uint32_t y_lo = r % H, y_hi = min(H, y_lo + (rows.end - r));
				r += y_hi - y_lo;
				for (int yi = int(y_lo) - 1; yi <= int(y_hi); ++yi, ++k)
				{
					failed = !mbar_wait_warp(&full[k % NSTAGE], (k / NSTAGE) & 1, POLL_LIMIT);
					// contributions j = 0, 1, 2 go to output rows yi + 1 - j; keep those in [y_lo, y_hi)
					const int j_lo = max(0, yi + 2 - int(y_hi)), j_hi = min(2, yi + 1 - int(y_lo));
					const uint32_t o_first = o_base + uint32_t(yi + 1 - j_lo - int(y_lo)); // counter of row yi + 1 - j_lo
					const uint32_t b0 = (R - o_first % R) % R;
					if (!failed && j_lo == 0 && o_first >= R) // a new row's accumulator must have been drained
						failed = !mbar_wait_warp(&acce[b0], ((o_first / R) - 1) & 1, POLL_LIMIT);
					if (failed) break;
					fence_after_sync();
					const uint64_t a_row = a_base + (((k % NSTAGE) * SLOT_BYTES) >> 4);
					if (j_lo == 0 && j_hi == 2 && b0 + 3 <= uint32_t(R))
					{
						// common case: one MMA per K step over the three blocks
						const uint32_t d = tmem + b0 * N;
#pragma unroll
						for (int dx = 0; dx < 3; ++dx)
#pragma unroll
							for (int ks = 0; ks < KSTEPS; ++ks)
								mma_bf16(d, a_row + ((2 * ks * CXS_BYTES + dx * 16) >> 4),
									b_base + (((dx * KSTEPS + ks) * (2 * NB * 16)) >> 4), IDESC3, 1u, issue);
					}
					else
					{
						// segment edges (fewer contributions) and ring wraps: at most two pieces
						const int nj = j_hi - j_lo + 1;
						const int len0 = min(nj, int(R - b0));
						const uint32_t d0 = tmem + b0 * N, d1 = tmem;
						const uint32_t bo0 = uint32_t(j_lo * N * 16) >> 4, bo1 = uint32_t((j_lo + len0) * N * 16) >> 4;
						const uint32_t id0 = len0 == 1 ? IDESC1 : len0 == 2 ? IDESC2 : IDESC3;
						const uint32_t id1 = nj - len0 == 1 ? IDESC1 : IDESC2;
						const bool two = len0 < nj;
#pragma unroll
						for (int dx = 0; dx < 3; ++dx)
#pragma unroll
							for (int ks = 0; ks < KSTEPS; ++ks)
							{
								const uint64_t ad = a_row + ((2 * ks * CXS_BYTES + dx * 16) >> 4);
								const uint64_t bk = b_base + (((dx * KSTEPS + ks) * (2 * NB * 16)) >> 4);
								mma_bf16(d0, ad, bk + bo0, id0, 1u, issue);
								if (two) mma_bf16(d1, ad, bk + bo1, id1, 1u, issue);
							}
					}
					// one commit: the input row's slot is free and output row yi - 1 (if j_hi == 2) complete
					mma_commit(&rowbar[k % NBAR], issue);
				}
				if (failed) break;
				o_base += y_hi - y_lo;
			}
			mma_commit(donebar, issue);
			if (!mbar_wait_warp(donebar, 0, POLL_LIMIT)) failed = true;
		}
	}
	else
	{
		const int quad = warp & 3;
		const uint32_t group = uint32_t(warp - 2) >> 2;
		const uint32_t lane_base = uint32_t(quad * 32) << 16;
		if (EPI != EPI_MASK)
		{
			// the same values from either group; a warp reads what its own lanes wrote
			if (lane < N) s_bias[lane] = a.bias[lane];
			__syncwarp();
		}
		float loss = 0.0f;
		uint32_t o = 0, k_base = 0;
		EpiOperands<N, EPI> op, next;
		for (uint32_t r = rows.begin; r < rows.end && !failed;)
		{
			const uint32_t strip = r / H, y_lo = r % H, y_hi = min(H, y_lo + (rows.end - r));
			r += y_hi - y_lo;
			const uint32_t img = strip / tiles_x;
			const int x = int(strip % tiles_x) * TILE_X + quad * 32 + lane;
			const uint32_t y_first = y_lo + ((o ^ group) & 1u); // this group's rows: those of its counter's parity
			if (y_first < y_hi) load_operands<N, EPI>(a, img, x, int(y_first), next);
			for (uint32_t y = y_first; y < y_hi; y += 2)
			{
				op = next;
				if (y + 2 < y_hi) load_operands<N, EPI>(a, img, x, int(y + 2), next);
				// output row y is complete once input row y + 1 (ring entry k_base + y - y_lo + 2) is committed
				const uint32_t kc = k_base + (y - y_lo) + 2;
				if (!mbar_wait_warp(&rowbar[kc % NBAR], (kc / NBAR) & 1, POLL_LIMIT))
				{
					failed = true;
					break;
				}
				fence_after_sync();
				const uint32_t b = (R - (o + (y - y_lo)) % R) % R;
				float v[N / 16][16];
#pragma unroll
				for (int c = 0; c < N / 16; ++c) tmem_ld(tmem + lane_base + b * N + c * 16, v[c]);
				tmem_ld_wait();
#pragma unroll
				for (int c8 = 0; c8 < N / 8; ++c8) tmem_zero8(tmem + lane_base + b * N + c8 * 8);
				tmem_st_wait();
				fence_before_sync();
				__syncwarp();
				if (lane == 0) mbar_arrive(&acce[b]);
#pragma unroll
				for (int c = 0; c < N / 16; ++c) conv_epilogue<N, EPI>(a, op, v[c], s_bias, c * 16, img, x, int(y), loss);
			}
			o += y_hi - y_lo;
			k_base += (y_hi - y_lo) + 2;
		}
		if (EPI == EPI_LOSS)
		{
			for (int o2 = 16; o2 > 0; o2 >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o2);
			if (lane == 0) s_red[warp - 2] = loss;
		}
	}
	if (failed) atomicExch(a.error, 1);
	fence_before_sync();
	__syncthreads();
	if (EPI == EPI_LOSS && tid == 0)
	{
		float t = 0.0f;
		for (int w = 0; w < CONV_EPI_WARPS; ++w) t += s_red[w];
		a.loss_partial[blockIdx.x] = t;
	}
	if (warp == 1)
	{
		fence_after_sync();
		tmem_dealloc(tmem, TMEM_COLS);
	}
}

// ---- fused inference: all four layers in one kernel ----
//
// One CTA owns a strip of 128 computed columns [c0, c0 + 128), c0 = 120 t - 4, and a segment of output
// rows [y_lo, y_hi). Every layer computes the strip's 128 columns; a column's value is exact while its
// receptive field lies inside the strip, so after four 3x3 layers the middle 120 columns are exact and
// are the strip's output (8 strips tile 960 columns). Layer l computes rows [y_lo - 3 + l, y_hi + 3 - l),
// reading rows one further up and down; rows or columns outside the frame are zero, exactly as the zero
// padding of the layer-by-layer convolution.
//
// Activations never leave the SM: layer l's input rows live in a shared-memory ring of FNS rows of
// C8_l chunks x 136 pixels (the layout conv_kernel stages from HBM), written by
//   warp 0 (all lanes) for layer 0: Color32 source -> (b, g, r) / 255 in bf16 (the input conversion),
//   the epilogue warps of layer l - 1 for layers 1..3: TMEM -> bias + ReLU -> bf16.
// MMAs are the dy-folded implicit GEMM of conv_kernel, 128 pixels x 3 C_out x 16 each, accumulated in place in
// a TMEM ring of 3 output rows per layer. Input row i adds to output rows i, i - 1 and i - 2 of its layer, which
// are the whole ring, so one MMA per K step always covers it; which of the three vertical taps meets which slot
// rotates from row to row, and the packed weights therefore lie in shared memory as ky = 0, 1, 2, 0, 1, with the
// B descriptor starting at the row's rotation (a ring of 4 slots that split half of the rows' MMAs in two
// pieces cost half as many MMAs again). Each layer has a warp that issues its MMAs, so that the tensor pipe has
// another layer's queued while one waits on its barriers (two issuers with two layers each left it idle a third of
// the time), and an epilogue group of four warps, 4 + 4 l ..: layers 0..2 write the next layer's input row, the
// last one the Color32 output (pixel shuffle + bilinear residual). Output row o is complete after input row
// o + 2. Every wait of layer l's row i is for layer l - 1's row i + 2 or earlier, or for layer l + 1's row
// i - FNS - 3 or earlier, so the roles cannot wait in a circle.
// Bound by shared-memory operand reads (128 bytes a cycle: 57 cycles per MMA of 7 KB, 1,129 for the 21 MMAs of
// one row of every layer) and the epilogues' writes beside them.
constexpr int FNS = 4;          // input-row slots per layer
constexpr int FR = 3;           // TMEM output-row accumulators per layer
constexpr int F_THREADS = 672;  // 21 warps: source, issuers of layers 0..2, 16 epilogue, issuer of layer 3
constexpr int F_VALID = 120;    // output columns per strip
constexpr uint32_t F_TMEM_COLS = 512;

struct FusedArgs
{
	const uint32_t* lo;
	uint32_t lo_w, lo_h, lo_pitch;
	uint32_t* hi;
	uint32_t hi_pitch;
	const uint16_t* w[NUM_LAYERS]; // packed B operands (conv_kernel's forward layout)
	const float* bias[NUM_LAYERS];
	uint32_t strips, segments;     // grid = strips x segments
	int* error;
};

// Per-layer constants.
template <int L>
struct FL
{
	static constexpr int C8 = L == 0 ? 2 : 4;
	static constexpr int N = L == 3 ? 16 : 32;
	static constexpr int KSTEPS = C8 / 2;
	static constexpr int GROUPS = 3 * KSTEPS * 2; // (kx, 16-channel step, half) groups of 8-channel weight rows
	static constexpr int NB = 5 * N;              // rows of a group: ky = 0, 1, 2, 0, 1
	static constexpr uint32_t SLOT = (C8 * CXS_BYTES + 127) / 128 * 128;
	static constexpr uint32_t WBYTES = GROUPS * NB * 16;
	static constexpr uint32_t TCOL = L * FR * 32; // TMEM column base (layers 0..2: 96 columns, 3: 48)
};

struct FusedSmem
{
	static constexpr uint32_t RING0 = 0;
	static constexpr uint32_t RING1 = RING0 + FNS * FL<0>::SLOT;
	static constexpr uint32_t RING2 = RING1 + FNS * FL<1>::SLOT;
	static constexpr uint32_t RING3 = RING2 + FNS * FL<2>::SLOT;
	static constexpr uint32_t W0 = RING3 + FNS * FL<3>::SLOT;
	static constexpr uint32_t W1 = W0 + FL<0>::WBYTES;
	static constexpr uint32_t W2 = W1 + FL<1>::WBYTES;
	static constexpr uint32_t W3 = W2 + FL<2>::WBYTES;
	static constexpr uint32_t BARS = W3 + FL<3>::WBYTES;
	// barriers: full[4][FNS], rowbar[4][NBAR], accfree[4][FR], wbar[4], done[4]
	static constexpr uint32_t NUM_BARS = 4 * FNS + 4 * NBAR + 4 * FR + 8;
	static constexpr uint32_t MISC = BARS + NUM_BARS * 8;
	static constexpr uint32_t TOTAL = MISC + 64;
};
static_assert(FusedSmem::TOTAL <= 227 * 1024, "fused kernel shared memory");

__device__ __forceinline__ uint32_t ring_base(int l)
{
	return l == 0 ? FusedSmem::RING0 : l == 1 ? FusedSmem::RING1 : l == 2 ? FusedSmem::RING2 : FusedSmem::RING3;
}

// Barriers of layer l: full[FNS] (input row written), rowbar[NBAR] (input row's MMAs done), accfree[FR]
// (output-row accumulator drained).
__device__ __forceinline__ uint64_t* f_full(unsigned char* smem, int l)
{
	return reinterpret_cast<uint64_t*>(smem + FusedSmem::BARS) + l * FNS;
}
__device__ __forceinline__ uint64_t* f_rowbar(unsigned char* smem, int l)
{
	return reinterpret_cast<uint64_t*>(smem + FusedSmem::BARS) + 4 * FNS + l * NBAR;
}
// Wait until the MMAs of layer l's input row i are done (its slot is free, output row i - 2 complete).
__device__ __forceinline__ bool f_wait_input_done(unsigned char* smem, int l, int i)
{
	return mbar_wait_warp(&f_rowbar(smem, l)[i % NBAR], (i / NBAR) & 1, POLL_LIMIT);
}
__device__ __forceinline__ uint64_t* f_accfree(unsigned char* smem, int l)
{
	return reinterpret_cast<uint64_t*>(smem + FusedSmem::BARS) + 4 * FNS + 4 * NBAR + l * FR;
}

// Rows of layer l of a segment: outputs [A, B), inputs [A - 1, B] (input index i <-> row A - 1 + i).
// Layer l + 1's input index i is layer l's output index i.
struct LayerRows
{
	int A, B;
	__device__ int inputs() const { return B - A + 2; }
	__device__ int outputs() const { return B - A; }
};
__device__ __forceinline__ LayerRows layer_rows(int l, int y_lo, int y_hi) { return LayerRows{y_lo - 3 + l, y_hi + 3 - l}; }

// Layer 0's source pixels of row y, columns c0 - 1 + j for j = lane + 32 k (the 136 staged pixels); 0
// outside the frame (converts to the zero padding) or when `valid` is false.
constexpr int F0_PX = (CXS + 31) / 32;
constexpr int F0_AHEAD = 3;
__device__ __forceinline__ void f0_load_row(const FusedArgs& a, int y, bool valid, int c0, int lane, uint32_t (&px)[F0_PX])
{
	const bool row_in = valid && y >= 0 && y < int(a.lo_h);
	const uint32_t* row = a.lo + size_t(row_in ? y : 0) * a.lo_pitch;
#pragma unroll
	for (int k = 0; k < F0_PX; ++k)
	{
		const int j = lane + 32 * k, x = c0 - 1 + j;
		px[k] = row_in && j < CXS && x >= 0 && x < int(a.lo_w) ? row[x] : 0u;
	}
}

// Layer `layer`'s MMAs for its input rows in turn (input index i = row A - 1 + i): the dy-folded K steps into the
// TMEM ring, then the row's commit. Called by a whole warp; one instance for layers 1 and 2. Returns false if a
// bounded wait expired.
template <int KSTEPS, int N>
__device__ __forceinline__ bool fused_mmas(unsigned char* smem, uint32_t tmem, int layer, uint32_t slot_bytes, uint32_t weights, int y_lo, int y_hi,
	uint32_t issue)
{
	constexpr int NB = 5 * N;
	constexpr uint32_t ID1 = make_idesc_bf16(128, N, 0, 0), ID3 = make_idesc_bf16(128, 3 * N, 0, 0);
	const LayerRows lr = layer_rows(layer, y_lo, y_hi);
	const int n = lr.inputs(), outputs = lr.outputs();
	const uint64_t a_base = make_sdesc(smem_addr(smem + ring_base(layer)), CXS_BYTES, 128);
	const uint64_t b_base = make_sdesc(smem_addr(smem + weights), NB * 16, 128);
	const uint32_t tcol = tmem + uint32_t(layer) * (FR * 32);
	uint64_t* full = f_full(smem, layer);
	uint64_t* accfree = f_accfree(smem, layer);
	uint64_t* rowbar = f_rowbar(smem, layer);
	for (int i = 0; i < n; ++i)
	{
		if (!mbar_wait_warp(&full[i % FNS], (i / FNS) & 1, POLL_LIMIT)) return false;
		// taps j = 0, 1, 2 go to output indexes i - j; keep those in [0, outputs)
		const int j_lo = max(0, i + 1 - outputs), j_hi = min(2, i);
		const uint32_t b0 = (FR - uint32_t(i) % FR) % FR; // slot of output i; i - 1 and i - 2 follow it around the ring
		if (j_lo == 0 && i >= FR && !mbar_wait_warp(&accfree[b0], ((i / FR) - 1) & 1, POLL_LIMIT)) return false;
		fence_after_sync();
		const uint64_t a_row = a_base + (((i % FNS) * slot_bytes) >> 4);
		if (j_lo == 0 && j_hi == 2)
		{
			// slot k takes tap (k - b0) mod 3: the weight rows from block (3 - b0) % 3 on
			const uint64_t b_row = b_base + ((((FR - b0) % FR) * N * 16) >> 4);
#pragma unroll
			for (int dx = 0; dx < 3; ++dx)
#pragma unroll
				for (int ks = 0; ks < KSTEPS; ++ks)
					mma_bf16(tcol, a_row + ((2 * ks * CXS_BYTES + dx * 16) >> 4), b_row + (((dx * KSTEPS + ks) * (2 * NB * 16)) >> 4), ID3,
						1u, issue);
		}
		else
		{
			// first and last rows of the segment: the taps that have an output row, one slot each
			for (int j = j_lo; j <= j_hi; ++j)
			{
				const uint32_t d = tcol + ((b0 + uint32_t(j)) % FR) * N;
				const uint64_t b_row = b_base + ((uint32_t(j) * N * 16) >> 4);
#pragma unroll
				for (int dx = 0; dx < 3; ++dx)
#pragma unroll
					for (int ks = 0; ks < KSTEPS; ++ks)
						mma_bf16(d, a_row + ((2 * ks * CXS_BYTES + dx * 16) >> 4), b_row + (((dx * KSTEPS + ks) * (2 * NB * 16)) >> 4), ID1,
							1u, issue);
			}
		}
		mma_commit(&rowbar[i % NBAR], issue);
	}
	return true;
}

// bf16 pair (low, high) of (a + bias) after ReLU: packed addition, rounding, then the maximum with 0, which is
// what rounding the maximum gives.
__device__ __forceinline__ uint32_t relu_pack(float a, float b, float2 bias)
{
	uint32_t lo, hi, r;
	asm("{\n\t.reg .b64 v, c;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 c, {%4, %5};\n\tadd.rn.f32x2 v, v, c;\n\tmov.b64 {%0, %1}, v;\n\t}"
		: "=r"(lo), "=r"(hi)
		: "f"(a), "f"(b), "f"(bias.x), "f"(bias.y));
	asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
	asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(0u));
	return r;
}

// Epilogue of layer 0, 1 or 2 for its output rows in turn (output index o = row A + o), by the layer's four warps
// (warp quad = lane quadrant = pixels quad*32..): accumulators -> registers, zero and release the accumulator,
// then the next layer's input row. One instance for the three layers: their code stays in the instruction cache.
__device__ __forceinline__ bool fused_epilogue_mid(const FusedArgs& a, unsigned char* smem, uint32_t tmem, int layer, int y_lo, int y_hi, int c0,
	int quad, int lane)
{
	constexpr int N = 32;
	const LayerRows lr = layer_rows(layer, y_lo, y_hi);
	uint64_t* accfree = f_accfree(smem, layer);
	uint64_t* next_full = f_full(smem, layer + 1);
	const int i = quad * 32 + lane; // pixel of the strip
	const int x = c0 + i;
	const bool x_in = x >= 0 && x < int(a.lo_w);
	const uint32_t tcol = tmem + (uint32_t(quad * 32) << 16) + uint32_t(layer) * (FR * 32);
	unsigned char* ring = smem + ring_base(layer + 1) + (1 + i) * 16;
	float2 bias[N / 2];
#pragma unroll
	for (int c = 0; c < N / 2; ++c) bias[c] = make_float2(a.bias[layer][2 * c], a.bias[layer][2 * c + 1]);
	const int n = lr.outputs();
	for (int o = 0; o < n; ++o)
	{
		if (!f_wait_input_done(smem, layer, o + 2)) return false; // the input row that completes output o
		fence_after_sync();
		const uint32_t b = (FR - uint32_t(o) % FR) % FR;
		float v[N];
		tmem_ld<N>(tcol + b * N, v);
		tmem_ld_wait();
		tmem_zero<N>(tcol + b * N);
		const int y = lr.A + o;
		const bool inside = x_in && y >= 0 && y < int(a.lo_h);
		uint32_t w[N / 2];
#pragma unroll
		for (int c = 0; c < N / 2; ++c) w[c] = relu_pack(v[2 * c], v[2 * c + 1], bias[c]);
		if (!__all_sync(0xFFFFFFFFu, inside)) // the next layer's zero padding
		{
#pragma unroll
			for (int c = 0; c < N / 2; ++c) w[c] = inside ? w[c] : 0u;
		}
		tmem_st_wait();
		fence_before_sync();
		__syncwarp();
		if (lane == 0) mbar_arrive(&accfree[b]);
		// next layer's input index o: wait until its slot's previous row was consumed
		if (o >= FNS && !f_wait_input_done(smem, layer + 1, o - FNS)) return false;
		unsigned char* dst = ring + (o % FNS) * FL<1>::SLOT; // the same slot size for layers 1..3
#pragma unroll
		for (int c8 = 0; c8 < N / 8; ++c8)
			*reinterpret_cast<uint4*>(dst + c8 * CXS_BYTES) = make_uint4(w[c8 * 4], w[c8 * 4 + 1], w[c8 * 4 + 2], w[c8 * 4 + 3]);
		fence_proxy_async();
		__syncwarp();
		if (lane == 0) mbar_arrive(&next_full[o % FNS]);
	}
	return true;
}
static_assert(FL<1>::SLOT == FL<2>::SLOT && FL<2>::SLOT == FL<3>::SLOT, "input rows of layers 1..3");

// Source pixels x - 1, x, x + 1 (clamped) of source row y (clamped), and their horizontal 2x upsample: h[sx][c] is
// colour c of output column 2x + sx.
__device__ __forceinline__ void f3_load(const FusedArgs& a, int x, int y, uint32_t (&p)[3])
{
	const uint32_t* row = a.lo + size_t(min(max(y, 0), int(a.lo_h) - 1)) * a.lo_pitch;
	p[0] = row[max(x - 1, 0)];
	p[1] = row[x];
	p[2] = row[min(x + 1, int(a.lo_w) - 1)];
}
__device__ __forceinline__ void f3_upsample(const uint32_t (&p)[3], float (&h)[2][3])
{
	const float c[3][3] = {{byte_float<0>(p[0]), byte_float<1>(p[0]), byte_float<2>(p[0])},
		{byte_float<0>(p[1]), byte_float<1>(p[1]), byte_float<2>(p[1])}, {byte_float<0>(p[2]), byte_float<1>(p[2]), byte_float<2>(p[2])}};
#pragma unroll
	for (int ch = 0; ch < 3; ++ch)
	{
		h[0][ch] = 0.75f * c[1][ch] + 0.25f * c[0][ch];
		h[1][ch] = 0.75f * c[1][ch] + 0.25f * c[2][ch];
	}
}

// Epilogue of the last layer: the Color32 output rows (pixel shuffle + bilinear residual) of the strip's columns
// c0 + 4 .. c0 + 123 inside the frame. The source rows around the output row are kept upsampled, and the
// next one is loaded a row ahead.
__device__ __forceinline__ bool fused_epilogue_last(const FusedArgs& a, unsigned char* smem, uint32_t tmem, int y_lo, int y_hi, int c0, int quad,
	int lane)
{
	constexpr int N = 16;
	const LayerRows lr = layer_rows(3, y_lo, y_hi);
	uint64_t* accfree = f_accfree(smem, 3);
	const int i = quad * 32 + lane;
	const int x = c0 + i;
	const bool out_px = i >= 4 && i < 4 + F_VALID && x < int(a.lo_w);
	const int xl = min(max(x, 0), int(a.lo_w) - 1); // lanes without an output pixel load some pixel of the row
	const uint32_t tcol = tmem + (uint32_t(quad * 32) << 16) + FL<3>::TCOL;
	float bias[12];
#pragma unroll
	for (int c = 0; c < 12; ++c) bias[c] = a.bias[3][c];
	const int n = lr.outputs();
	float h[3][2][3]; // source rows y - 1, y, y + 1
	uint32_t p[3], alpha, alpha_next;
	f3_load(a, xl, lr.A - 1, p);
	f3_upsample(p, h[0]);
	f3_load(a, xl, lr.A, p);
	f3_upsample(p, h[1]);
	alpha = p[1];
	f3_load(a, xl, lr.A + 1, p);
	f3_upsample(p, h[2]);
	alpha_next = p[1];
	for (int o = 0; o < n; ++o)
	{
		const int y = lr.A + o;
		f3_load(a, xl, y + 2, p);
		if (!f_wait_input_done(smem, 3, o + 2)) return false;
		fence_after_sync();
		const uint32_t b = (FR - uint32_t(o) % FR) % FR;
		float v[N];
		tmem_ld<N>(tcol + b * N, v);
		tmem_ld_wait();
		tmem_zero<N>(tcol + b * N);
		tmem_st_wait();
		fence_before_sync();
		__syncwarp();
		if (lane == 0) mbar_arrive(&accfree[b]);
		if (out_px)
		{
#pragma unroll
			for (int sy = 0; sy < 2; ++sy)
			{
				uint32_t px[2];
#pragma unroll
				for (int sx = 0; sx < 2; ++sx)
				{
					uint32_t q[3];
#pragma unroll
					for (int ch = 0; ch < 3; ++ch)
					{
						const float top = h[1][sx][ch], bot = h[sy ? 2 : 0][sx][ch];
						q[ch] = float_byte((0.75f * top + 0.25f * bot) * (1.0f / 255.0f) + (v[ch * 4 + sy * 2 + sx] + bias[ch * 4 + sy * 2 + sx]));
					}
					// bytes b, g, r of the values and the source pixel's alpha
					px[sx] = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], alpha, 0x0070), 0x5410);
				}
				*reinterpret_cast<uint2*>(a.hi + size_t(2 * y + sy) * a.hi_pitch + 2 * x) = make_uint2(px[0], px[1]);
			}
		}
#pragma unroll
		for (int sx = 0; sx < 2; ++sx)
#pragma unroll
			for (int ch = 0; ch < 3; ++ch)
			{
				h[0][sx][ch] = h[1][sx][ch];
				h[1][sx][ch] = h[2][sx][ch];
			}
		f3_upsample(p, h[2]);
		alpha = alpha_next;
		alpha_next = p[1];
	}
	return true;
}

// The packed weights of layer L (conv_kernel's forward layout, ky = 0, 1, 2 in a group) into shared memory as
// ky = 0, 1, 2, 0, 1; by the layer's issuing warp, one lane per group.
template <int L>
__device__ __forceinline__ void f_load_weights(unsigned char* dst, const uint16_t* w, uint64_t* wbar, int lane)
{
	using F = FL<L>;
	if (lane == 0) mbar_expect_tx(wbar, F::WBYTES);
	__syncwarp();
	if (lane >= F::GROUPS) return;
	const unsigned char* src = reinterpret_cast<const unsigned char*>(w) + lane * (3 * F::N * 16);
	bulk_g2s(dst + lane * (F::NB * 16), src, 3 * F::N * 16, wbar);
	bulk_g2s(dst + lane * (F::NB * 16) + 3 * F::N * 16, src, 2 * F::N * 16, wbar);
}

__global__ void __launch_bounds__(F_THREADS, 1) fused_upscale_kernel(const __grid_constant__ FusedArgs a)
{
	extern __shared__ __align__(1024) unsigned char smem[];
	uint64_t* wbar = reinterpret_cast<uint64_t*>(smem + FusedSmem::BARS) + 4 * FNS + 4 * NBAR + 4 * FR;
	uint64_t* done = wbar + 4; // [4] each: one per MMA issuer
	uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + FusedSmem::MISC);

	const int tid = threadIdx.x, lane = tid & 31;
	const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0); // known to be the same in the whole warp
	const int strip = int(blockIdx.x % a.strips), seg = int(blockIdx.x / a.strips);
	const int H = int(a.lo_h);
	const int y_lo = int((int64_t(seg) * H) / int(a.segments)), y_hi = int((int64_t(seg + 1) * H) / int(a.segments));
	const int c0 = strip * F_VALID - 4;

	// zero what no role writes: layer 0's second chunk, and in layers 1..3 the pixels outside the strip's 128
	constexpr int EDGE = CXS - 128, L0_ZERO = FNS * CXS, ZEROS = L0_ZERO + 3 * FNS * FL<1>::C8 * EDGE;
	for (int z = tid; z < ZEROS; z += F_THREADS)
	{
		uint32_t off;
		if (z < L0_ZERO)
			off = FusedSmem::RING0 + (z / CXS) * FL<0>::SLOT + CXS_BYTES + (z % CXS) * 16;
		else
		{
			const int k = z - L0_ZERO, e = k % EDGE, chunk = k / EDGE % FL<1>::C8, slot = k / (EDGE * FL<1>::C8) % FNS, l = 1 + k / (EDGE * FL<1>::C8 * FNS);
			off = ring_base(l) + slot * FL<1>::SLOT + chunk * CXS_BYTES + (e ? 128 + e : 0) * 16; // pixel 0, pixels 129..135
		}
		*reinterpret_cast<uint4*>(smem + off) = make_uint4(0u, 0u, 0u, 0u);
	}
	if (tid == 0)
	{
		for (int l = 0; l < 4; ++l)
		{
			for (int k = 0; k < FNS; ++k) mbar_init(&f_full(smem, l)[k], l == 0 ? 32 : 4);
			for (int k = 0; k < NBAR; ++k) mbar_init(&f_rowbar(smem, l)[k], 1);
			for (int k = 0; k < FR; ++k) mbar_init(&f_accfree(smem, l)[k], 4);
		}
		for (int l = 0; l < 4; ++l)
		{
			mbar_init(&wbar[l], 1);
			mbar_init(&done[l], 1);
		}
		fence_mbar_init();
	}
	if (warp == 1)
	{
		tmem_alloc(s_tmem, F_TMEM_COLS);
		tmem_relinquish();
	}
	fence_proxy_async();
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);
	if (warp >= 4 && warp < 20)
	{
		// every accumulator starts at zero (the MMAs always accumulate): 96 columns per group
		const uint32_t t = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t((warp - 4) / 4) * (FR * 32);
		for (uint32_t c = 0; c < FR * 32; c += 32) tmem_zero<32>(t + c);
		tmem_st_wait();
	}
	fence_before_sync();
	__syncthreads();
	fence_after_sync();

	const LayerRows lr0 = layer_rows(0, y_lo, y_hi);
	bool failed = false;
	// everything above touched only the SM: it overlaps the end of the kernel before
	pdl_trigger();
	pdl_wait();

	if (warp == 0)
	{
		// layer 0 input rows from the Color32 source. Lane t holds pixels t + 32 k (k < F0_PX) of a row;
		// the loads of a row are issued F0_AHEAD rows before it is stored, so their latency overlaps the
		// waits for ring slots instead of adding to every row.
		uint64_t* full0 = f_full(smem, 0);

		const int n0 = lr0.inputs();
		uint32_t pre[F0_AHEAD + 1][F0_PX];
#pragma unroll
		for (int r = 0; r < F0_AHEAD; ++r) f0_load_row(a, lr0.A - 1 + r, r < n0, c0, lane, pre[r]);
		for (int q = 0; q < n0 && !failed; ++q)
		{
			f0_load_row(a, lr0.A - 1 + q + F0_AHEAD, q + F0_AHEAD < n0, c0, lane, pre[F0_AHEAD]);
			if (q >= FNS && !f_wait_input_done(smem, 0, q - FNS))
			{
				failed = true;
				break;
			}
			unsigned char* dst = smem + FusedSmem::RING0 + (q % FNS) * FL<0>::SLOT;
#pragma unroll
			for (int k = 0; k < F0_PX; ++k)
			{
				const int j = lane + 32 * k;
				if (j < CXS)
				{
					const uint32_t px = pre[0][k];
					uint4 w4;
					w4.x = pack2(byte_float<0>(px) * (1.0f / 255.0f), byte_float<1>(px) * (1.0f / 255.0f));
					w4.y = pack2(byte_float<2>(px) * (1.0f / 255.0f), 0.0f);
					w4.z = 0u;
					w4.w = 0u;
					*reinterpret_cast<uint4*>(dst + j * 16) = w4;
				}
			}
			fence_proxy_async();
			mbar_arrive(&full0[q % FNS]);
#pragma unroll
			for (int r = 0; r < F0_AHEAD; ++r)
#pragma unroll
				for (int k = 0; k < F0_PX; ++k) pre[r][k] = pre[r + 1][k];
		}
	}
	else if (warp <= 3 || warp == 20)
	{
		const int layer = warp == 20 ? 3 : warp - 1;
		const uint32_t issue = lane == 0 ? 1u : 0u; // the whole warp runs the role, lane 0 issues
		if (layer == 0)
			f_load_weights<0>(smem + FusedSmem::W0, a.w[0], &wbar[0], lane);
		else if (layer == 3)
			f_load_weights<3>(smem + FusedSmem::W3, a.w[3], &wbar[3], lane);
		else
			f_load_weights<1>(smem + (layer == 1 ? FusedSmem::W1 : FusedSmem::W2), a.w[layer], &wbar[layer], lane);
		failed = !mbar_wait_warp(&wbar[layer], 0, POLL_LIMIT);
		if (!failed)
		{
			if (layer == 0)
				failed = !fused_mmas<1, 32>(smem, tmem, 0, FL<0>::SLOT, FusedSmem::W0, y_lo, y_hi, issue);
			else if (layer == 3)
				failed = !fused_mmas<2, 16>(smem, tmem, 3, FL<3>::SLOT, FusedSmem::W3, y_lo, y_hi, issue);
			else
				failed = !fused_mmas<2, 32>(smem, tmem, layer, FL<1>::SLOT, layer == 1 ? FusedSmem::W1 : FusedSmem::W2, y_lo, y_hi, issue);
		}
		mma_commit(&done[layer], issue);
		if (!mbar_wait_warp(&done[layer], 0, POLL_LIMIT)) failed = true;
	}
	else
	{
		const int quad = warp & 3;
		const int layer = (warp - 4) >> 2;
		failed = !(layer < 3 ? fused_epilogue_mid(a, smem, tmem, layer, y_lo, y_hi, c0, quad, lane)
							 : fused_epilogue_last(a, smem, tmem, y_lo, y_hi, c0, quad, lane));
	}
	if (failed) atomicExch(a.error, 1);
	fence_before_sync();
	__syncthreads();
	if (warp == 1)
	{
		fence_after_sync();
		tmem_dealloc(tmem, F_TMEM_COLS);
	}
}

// ---- weight gradient ----

struct WgradLayer
{
	Planes x; // layer input
	Planes g; // pre-activation gradient
	float* partial; // per CTA: [3 dx][wgrad_rows(C8X)][NG] then the bias partials [NG]
};
struct WgradArgs
{
	WgradLayer layer[NUM_LAYERS];
	uint32_t blocks; // per layer: images * height / ROWS
	int* error;
};

// The accumulator rows that are taps: (dy, chunk, ci % 8) for dy < 3; the rows above belong to no tap.
__host__ __device__ constexpr uint32_t wgrad_rows(int c8x) { return 3 * c8x * 8; }
__host__ __device__ constexpr uint32_t wgrad_partial_floats(int c8x, int ng) { return 3 * wgrad_rows(c8x) * ng + ng; }

// Crops are one tile wide and their planes CXS pixels, so a row (all its chunks) is one run of memory, and so are
// neighbouring rows.
static_assert(SW_UPSCALER_CROP_W == TILE_X && SW_UPSCALER_CROP_H % ROWS == 0, "a CTA's rows are whole rows of one crop");
constexpr int WG_XROWS = ROWS + 2; // staged input rows
constexpr int WG_STEPS = ROWS / 2; // two gradient rows per MMA
constexpr uint32_t WG_X_BYTES = WG_XROWS * 4 * CXS_BYTES, WG_G_BYTES = ROWS * 4 * CXS_BYTES;
constexpr uint32_t WG_TMEM_COLS = 256;
struct WgradSmem
{
	static constexpr uint32_t X = 0, G = WG_X_BYTES, BARS = G + WG_G_BYTES; // bars: [WG_STEPS] rows loaded, then MMAs done
	static constexpr uint32_t TMEM = BARS + (WG_STEPS + 1) * 8, BIAS = TMEM + 8, TOTAL = BIAS + 128 * 4;
};

// One layer's share of a CTA: ROWS rows of one crop.
template <int C8X, int NG>
__device__ __forceinline__ bool wgrad_rows_block(const WgradLayer& a, uint32_t bid, unsigned char* smem, uint32_t tmem)
{
	constexpr int XM = 16 / C8X; // input rows stacked in M; the first four meet a gradient row
	constexpr int G8 = NG / 8;
	constexpr uint32_t X_ROW = C8X * CXS_BYTES, G_ROW = G8 * CXS_BYTES;
	constexpr uint32_t MR = wgrad_rows(C8X);
	constexpr uint32_t LINE = NG + 4; // floats between the rows of the sums (conflict-free 16-byte accesses)
	// the rows of M that meet no gradient row read whatever lies behind the staged rows
	static_assert(XM >= 4 && (ROWS - 2 + XM) * X_ROW <= WgradSmem::BARS && WG_XROWS * X_ROW <= WG_X_BYTES, "staged rows");
	static_assert(3 * 2 * NG <= int(WG_TMEM_COLS) && 3 * MR * LINE * 4 <= WgradSmem::BARS, "accumulators");
	unsigned char* s_x = smem + WgradSmem::X;
	unsigned char* s_g = smem + WgradSmem::G;
	uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WgradSmem::BARS);
	float* s_bias = reinterpret_cast<float*>(smem + WgradSmem::BIAS);
	const int tid = threadIdx.x, lane = tid & 31;
	const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0); // known to be the same in the whole warp
	const uint32_t row_blocks = a.x.height / ROWS;
	const uint32_t img = bid / row_blocks;
	const int y0 = int(bid % row_blocks) * ROWS;
	bool ok = true;
	if (tid == 0)
		for (int t = 0; t < WG_STEPS; ++t)
		{
			// the input rows y0 + 2t - 1 .. y0 + 2t + 2 that are not staged yet, and gradient rows y0 + 2t, y0 + 2t + 1
			const int first = t ? 2 * t + 2 : 0, n = t ? 2 : 4;
			mbar_expect_tx(&bars[t], n * X_ROW + 2 * G_ROW);
			bulk_g2s(s_x + first * X_ROW, a.x.data + planes_index(a.x, img, y0 - 1 + first, 0, -1), n * X_ROW, &bars[t]);
			bulk_g2s(s_g + 2 * t * G_ROW, a.g.data + planes_index(a.g, img, y0 + 2 * t, 0, -1), 2 * G_ROW, &bars[t]);
		}
	if (warp == 0)
	{
		const uint32_t issue = lane == 0 ? 1u : 0u;
		constexpr uint32_t idesc = make_idesc_bf16(128, 2 * NG, 1, 1);
		// A = X^T: rows (input row, chunk, ci % 8), 8-row groups CXS_BYTES apart; K = 16 pixels, LBO = 8 pixels.
		const uint64_t xb = make_sdesc(smem_addr(s_x), 128, CXS_BYTES);
		// B = G^T: columns (gradient row, co), 8-column groups CXS_BYTES apart; the same 16 pixels.
		const uint64_t gb = make_sdesc(smem_addr(s_g), 128, CXS_BYTES);
		for (int t = 0; t < WG_STEPS; ++t)
		{
			if (!mbar_wait_warp(&bars[t], 0, POLL_LIMIT)) ok = false;
			if (!ok) continue; // every copy has to be waited for before the CTA may leave
			fence_after_sync();
#pragma unroll 2
			for (int kc = 0; kc < TILE_X / 16; ++kc)
#pragma unroll
				for (int d = 0; d < 3; ++d)
					mma_bf16(tmem + d * 2 * NG, xb + ((2 * t * X_ROW + (d + 16 * kc) * 16) >> 4),
						gb + ((2 * t * G_ROW + (1 + 16 * kc) * 16) >> 4), idesc, t || kc ? 1u : 0u, issue);
		}
		mma_commit(&bars[WG_STEPS], issue);
	}
	// Bias gradient partials from the staged gradient rows (pixels 0..127 of the tile).
	{
		constexpr int PARTS = 128 / NG;
		const int co = tid % NG, part = tid / NG;
		const int c8 = co / 8, e = co % 8;
		float s = 0.0f;
		for (int r = 0; r < ROWS; ++r)
		{
			if (!mbar_wait_bounded(&bars[r / 2], 0, POLL_LIMIT)) ok = false;
			if (ok)
				for (int p = part; p < TILE_X; p += PARTS)
					s += bf2f(*reinterpret_cast<const uint16_t*>(s_g + r * G_ROW + c8 * CXS_BYTES + (1 + p) * 16 + e * 2));
		}
		s_bias[tid] = s;
	}
	if (!mbar_wait_bounded(&bars[WG_STEPS], 0, POLL_LIMIT)) ok = false;
	if (__syncthreads_or(!ok)) return false;
	fence_after_sync();
	// Input row i with gradient row j of a step is tap row dy = i - j: row (dy, chunk, ci % 8) of the sum is accumulator row
	// m of the first gradient row and m + C8X * 8 of the second. Added in shared memory (the operands are no longer read),
	// from where whole lines are written.
	float* sums = reinterpret_cast<float*>(smem);
	const uint32_t m = warp * 32 + lane;
	const uint32_t lane_base = uint32_t(warp * 32) << 16;
#pragma unroll
	for (int j = 0; j < 2; ++j)
	{
		const uint32_t row = m - j * C8X * 8; // of the sum; wraps for the rows below
		if (warp * 32 < int(MR) + j * C8X * 8)
#pragma unroll
			for (int d = 0; d < 3; ++d)
#pragma unroll
				for (int c = 0; c < NG; c += 16)
				{
					float v[16];
					tmem_ld(tmem + lane_base + (d * 2 + j) * NG + c, v);
					tmem_ld_wait();
					if (row < MR)
					{
						float4* o = reinterpret_cast<float4*>(sums + (d * MR + row) * LINE + c);
#pragma unroll
						for (int q = 0; q < 4; ++q)
						{
							float4 w = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
							if (j)
							{
								const float4 f = o[q];
								w = make_float4(f.x + w.x, f.y + w.y, f.z + w.z, f.w + w.w);
							}
							o[q] = w;
						}
					}
					__syncwarp(); // the next load of accumulators is the whole warp's
				}
		__syncthreads();
	}
	float* out = a.partial + size_t(bid) * wgrad_partial_floats(C8X, NG);
	for (uint32_t i = tid; i < 3 * MR * (NG / 4); i += 128)
		reinterpret_cast<float4*>(out)[i] = *reinterpret_cast<const float4*>(sums + i / (NG / 4) * LINE + i % (NG / 4) * 4);
	if (tid < NG)
	{
		constexpr int PARTS = 128 / NG;
		float s = 0.0f;
		for (int q = 0; q < PARTS; ++q) s += s_bias[q * NG + tid];
		out[3 * MR * NG + tid] = s;
	}
	return true;
}

// The weight gradients of all four layers, ROWS rows of a crop and one layer per CTA, last layer first. Bound by the
// rate of the MMAs (52 cycles each for 2 * NG <= 64 columns, whatever their number, so two gradient rows share one:
// 48 per CTA instead of 96) and by loading, multiplying and storing one after the other in the two CTAs of an SM.
// 32 us for 16 crops, of a training step of 150; with a launch per layer between the input gradients and a copy per
// row and chunk the step takes 6 us longer, and with one gradient row per MMA another 12.
__global__ void __launch_bounds__(128, 2) wgrad_kernel(const __grid_constant__ WgradArgs a)
{
	extern __shared__ __align__(1024) unsigned char smem[];
	uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WgradSmem::BARS);
	uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + WgradSmem::TMEM);
	const int warp = __shfl_sync(0xFFFFFFFFu, int(threadIdx.x >> 5), 0); // known to be the same in the whole warp
	if (threadIdx.x == 0)
	{
		for (int i = 0; i <= WG_STEPS; ++i) mbar_init(&bars[i], 1);
		fence_mbar_init();
	}
	if (warp == 0)
	{
		tmem_alloc(s_tmem, WG_TMEM_COLS);
		tmem_relinquish();
	}
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);
	pdl_trigger();
	pdl_wait(); // the planes are written
	const uint32_t l = NUM_LAYERS - 1 - blockIdx.x / a.blocks, bid = blockIdx.x % a.blocks;
	static_assert(LAYERS[0].c8_in == 2 && LAYERS[0].n_out == 32 && LAYERS[1].c8_in == 4 && LAYERS[1].n_out == 32 &&
			LAYERS[2].c8_in == 4 && LAYERS[2].n_out == 32 && LAYERS[3].c8_in == 4 && LAYERS[3].n_out == 16, "instances");
	const bool ok = l == 3 ? wgrad_rows_block<4, 16>(a.layer[3], bid, smem, tmem)
		: l == 0           ? wgrad_rows_block<2, 32>(a.layer[0], bid, smem, tmem)
						   : wgrad_rows_block<4, 32>(a.layer[l], bid, smem, tmem);
	if (!ok && threadIdx.x == 0) atomicExch(a.error, 3);
	fence_before_sync();
	__syncthreads();
	if (warp == 0)
	{
		fence_after_sync();
		tmem_dealloc(tmem, WG_TMEM_COLS);
	}
}

// ---- conversion, Adam, reduction ----

__global__ void convert_input_kernel(const CropGpu* crops, Planes p)
{
	const uint32_t img = blockIdx.y;
	const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
	pdl_trigger();
	pdl_wait();
	if (idx >= p.width * p.height) return;
	const int x = int(idx % p.width), y = int(idx / p.width);
	const CropGpu c = crops[img];
	const uint32_t px = c.lo[size_t(c.y + y) * c.lo_pitch + (c.x + x)];
	uint4 o;
	o.x = pack2(float(px & 255u) * (1.0f / 255.0f), float((px >> 8) & 255u) * (1.0f / 255.0f));
	o.y = pack2(float((px >> 16) & 255u) * (1.0f / 255.0f), 0.0f);
	o.z = 0u;
	o.w = 0u;
	*reinterpret_cast<uint4*>(p.data + planes_index(p, img, y, 0, x)) = o;
}

// Adam on the canonical parameters, then repack every weight into the forward and transposed
// (input-gradient) B-operand layouts as bf16 and every bias as f32.
struct AdamArgs
{
	float* params;
	float* m;
	float* v;
	const float* grads;
	float lr, beta1, beta2, eps, bc1, bc2; // bc = 1 - beta^t
	int update;
	uint16_t* wfwd[NUM_LAYERS];
	uint16_t* wbwd[NUM_LAYERS];
	float* bias[NUM_LAYERS];
};

__device__ __forceinline__ void adam_pack(const AdamArgs& a, int idx, float g)
{
	float p = a.params[idx];
	if (a.update)
	{
		const float m = a.beta1 * a.m[idx] + (1.0f - a.beta1) * g;
		const float v = a.beta2 * a.v[idx] + (1.0f - a.beta2) * g * g;
		a.m[idx] = m;
		a.v[idx] = v;
		p -= a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
		a.params[idx] = p;
	}
	int l = NUM_LAYERS - 1;
	while (l > 0 && idx < c_layers[l].param_offset) --l;
	const LayerShape L = c_layers[l];
	const int local = idx - L.param_offset;
	const int nw = L.cout * 9 * L.cin;
	if (local >= nw)
	{
		a.bias[l][local - nw] = p;
		return;
	}
	int r = local;
	const int ci = r % L.cin;
	r /= L.cin;
	const int t = r % 9;
	const int co = r / 9;
	const uint16_t h = f2bf(p);
	const int ky = t / 3, kx = t % 3;
	{
		// B operand of conv_kernel: per (kx, 16-channel step ks, half hh): rows (ky, co) x 8 input channels
		const int ks = ci / 16, hh = (ci / 8) % 2, e = ci % 8;
		const int nb = 3 * L.n_out;
		a.wfwd[l][((kx * (L.c8_in / 2) + ks) * 2 + hh) * nb * 8 + (ky * L.n_out + co) * 8 + e] = h;
	}
	if (a.wbwd[l])
	{
		// input gradient = conv over the gradient (n_out / 8 chunks) producing c8_in * 8 channels with
		// the taps flipped: (ky, kx) -> (2 - ky, 2 - kx), input and output channels swapped
		const int no = L.c8_in * 8;
		const int ks = co / 16, hh = (co / 8) % 2, e = co % 8;
		a.wbwd[l][(((2 - kx) * (L.n_out / 16) + ks) * 2 + hh) * (3 * no) * 8 + ((2 - ky) * no + ci) * 8 + e] = h;
	}
}

// Repacking without an update (new parameters).
__global__ void adam_pack_kernel(AdamArgs a)
{
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx < int(SW_UPSCALER_NUM_PARAMS)) adam_pack(a, idx, 0.0f);
}

// The weight gradients' per-CTA partials of every layer summed (times `scale`) into canonical gradients, and with
// a.update Adam and the repacking right after, one launch for the four layers. A block takes 32 neighbouring
// accumulator columns, so a warp reads whole 128-byte lines of a partial; its eight warps take every eighth
// partial and their sums are added in order, so the result does not depend on the run. Bound by reading the
// partials from L2 (28 MB at 16 crops): 10 us. With one thread per parameter, 256 dependent reads of 4 bytes
// from lines of their own, the four sums took 121 us.
struct ReduceArgs
{
	const float* partial[NUM_LAYERS];
	uint32_t num_ctas;
	float scale;
	float* grads;
	AdamArgs adam;
};
constexpr int REDUCE_WARPS = 8;
__host__ __device__ constexpr int reduce_items(int l) // accumulator columns of layer l: weights, then biases
{
	return 9 * LAYERS[l].cin * LAYERS[l].n_out + LAYERS[l].n_out;
}
__host__ __device__ constexpr int reduce_blocks(int l) { return (reduce_items(l) + 31) / 32; }
__host__ __device__ constexpr int reduce_first(int l) { return l == 0 ? 0 : reduce_first(l - 1) + reduce_blocks(l - 1); }

__global__ void __launch_bounds__(REDUCE_WARPS * 32) wgrad_reduce_kernel(const __grid_constant__ ReduceArgs a)
{
	__shared__ float s_sum[REDUCE_WARPS][32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr int F1 = reduce_first(1), F2 = reduce_first(2), F3 = reduce_first(3);
	const int b = int(blockIdx.x), l = b < F1 ? 0 : b < F2 ? 1 : b < F3 ? 2 : 3;
	const LayerShape L = c_layers[l];
	const int item = (b - (l == 0 ? 0 : l == 1 ? F1 : l == 2 ? F2 : F3)) * 32 + lane, nw = 9 * L.cin * L.n_out;
	const bool valid = item < nw + L.n_out;
	const uint32_t mr = wgrad_rows(L.c8_in), stride = wgrad_partial_floats(L.c8_in, L.n_out);
	const int co = item % L.n_out;
	int idx = -1; // canonical parameter, -1 for the padded output channels
	uint32_t off = 0;
	if (item < nw)
	{
		const int r = item / L.n_out, ci = r % L.cin, t = r / L.cin, ky = t / 3, kx = t % 3;
		off = (uint32_t(kx) * mr + uint32_t((ky * L.c8_in + ci / 8) * 8 + ci % 8)) * L.n_out + co;
		if (co < L.cout) idx = L.param_offset + (co * 9 + t) * L.cin + ci;
	}
	else if (valid)
	{
		off = 3 * mr * L.n_out + co;
		if (co < L.cout) idx = L.param_offset + L.cout * 9 * L.cin + co;
	}
	float s = 0.0f;
	pdl_trigger();
	pdl_wait(); // every layer's partials are written
	if (valid)
	{
		const float* p = a.partial[l] + off;
#pragma unroll 8
		for (uint32_t c = warp; c < a.num_ctas; c += REDUCE_WARPS) s += p[size_t(c) * stride];
	}
	s_sum[warp][lane] = s;
	__syncthreads();
	if (warp || idx < 0) return;
	float t = 0.0f;
#pragma unroll
	for (int w = 0; w < REDUCE_WARPS; ++w) t += s_sum[w][lane];
	t *= a.scale;
	a.grads[idx] = t;
	if (a.adam.update) adam_pack(a.adam, idx, t);
}

__global__ void psnr_kernel(const uint32_t* a, uint32_t ap, const uint32_t* b, uint32_t bp, uint32_t w, uint32_t h,
	unsigned long long* sum)
{
	unsigned long long s = 0;
	for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < w * h; idx += gridDim.x * blockDim.x)
	{
		const uint32_t x = idx % w, y = idx / w;
		const uint32_t pa = a[size_t(y) * ap + x], pb = b[size_t(y) * bp + x];
		for (int ch = 0; ch < 3; ++ch)
		{
			const int d = int((pa >> (8 * ch)) & 255u) - int((pb >> (8 * ch)) & 255u);
			s += unsigned(d * d);
		}
	}
	for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
	if ((threadIdx.x & 31) == 0) atomicAdd(sum, s);
}

// ---- host side ----

struct DevMem
{
	void* ptr = nullptr;
	size_t bytes = 0;
};

uint64_t fnv1a(const void* data, size_t n, uint64_t h = 1469598103934665603ull)
{
	const unsigned char* p = static_cast<const unsigned char*>(data);
	for (size_t i = 0; i < n; ++i)
	{
		h ^= p[i];
		h *= 1099511628211ull;
	}
	return h;
}

uint64_t splitmix(uint64_t& s)
{
	uint64_t z = (s += 0x9E3779B97F4A7C15ull);
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

} // namespace

struct SwUpscaler
{
	int device = 0;
	cudaStream_t stream = nullptr;
	std::string last_error;
	uint64_t steps = 0;
	int num_sms = 1;
	uint32_t loss_ctas = 0; // CTAs of the last loss-epilogue launch
	// canonical parameters and Adam state (device, f32)
	DevMem params, adam_m, adam_v, grads;
	DevMem wfwd[NUM_LAYERS], wbwd[NUM_LAYERS], bias[NUM_LAYERS];
	DevMem error;
	// training workspace (SW_UPSCALER_MAX_CROPS crops)
	DevMem t_x0, t_a[3], t_g4, t_g[3], partial[NUM_LAYERS], loss_partial, crops;
	uint32_t crops_capacity = 0;
	DevMem h_stage; // pinned: crops + loss partials
	// inference workspace
	DevMem i_x0, i_p, i_q, i_crop;
	uint32_t i_w = 0, i_h = 0;
	CropGpu i_crop_host{};
	bool i_crop_valid = false;
	bool fused = true; // inference by fused_upscale_kernel (else the four layer launches)
	DevMem psnr_sum;
	unsigned long long* h_psnr = nullptr;
	cudaEvent_t ev = nullptr;
	// Shared-memory opt-ins made on this upscaler's device (an attribute of the kernel on one device), and the
	// convolutions' CTAs per SM with them (0: not yet). Concurrent first calls make them twice.
	static constexpr int CONV_KEYS = 64;
	std::atomic<int> conv_per_sm[CONV_KEYS] = {};
	std::atomic<bool> wgrad_ready{false}, fused_ready{false};
};

namespace
{

int fail(SwUpscaler* u, int code, const char* fmt, ...)
{
	char buf[512];
	va_list ap;
	va_start(ap, fmt);
	vsnprintf(buf, sizeof(buf), fmt, ap);
	va_end(ap);
	if (u) u->last_error = buf;
	return code;
}

#define UP_CUDA(u, call)                                                                      \
	do                                                                                        \
	{                                                                                         \
		cudaError_t e_ = (call);                                                              \
		if (e_ != cudaSuccess) return fail(u, SW_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
	} while (0)

int dev_alloc(SwUpscaler* u, DevMem& m, size_t bytes, bool zero = true)
{
	if (m.ptr && m.bytes >= bytes) return SW_OK;
	if (m.ptr) cudaFree(m.ptr);
	m.ptr = nullptr;
	m.bytes = 0;
	cudaError_t e = cudaMalloc(&m.ptr, bytes);
	if (e != cudaSuccess)
	{
		cudaGetLastError();
		return fail(u, SW_ERR_OUT_OF_MEMORY, "cudaMalloc(%zu) failed", bytes);
	}
	m.bytes = bytes;
	if (zero)
	{
		// Zeroed on the upscaler's stream and waited for here: a plain cudaMemset runs on the legacy
		// default stream, which the non-blocking streams the buffers are used on do not wait for.
		UP_CUDA(u, cudaMemsetAsync(m.ptr, 0, bytes, u->stream));
		UP_CUDA(u, cudaStreamSynchronize(u->stream));
	}
	return SW_OK;
}

void dev_free(DevMem& m)
{
	if (m.ptr) cudaFree(m.ptr);
	m.ptr = nullptr;
	m.bytes = 0;
}

Planes make_planes(void* data, uint32_t images, uint32_t width, uint32_t height, uint32_t chunks)
{
	Planes p;
	p.data = static_cast<uint16_t*>(data);
	p.images = images;
	p.width = width;
	p.height = height;
	p.chunks = chunks;
	p.wp = ((width + TILE_X - 1) / TILE_X) * TILE_X + 8;
	p.rows_alloc = ((height + ROWS - 1) / ROWS) * ROWS + 10;
	return p;
}

size_t planes_bytes(uint32_t images, uint32_t width, uint32_t height, uint32_t chunks)
{
	const Planes p = make_planes(nullptr, images, width, height, chunks);
	return size_t(images) * p.rows_alloc * chunks * p.wp * 16;
}

// Tensor map of the rows of a row-plane tensor as a 4-D bf16 array [images * rows_alloc][chunks][wp / 8][64]
// (innermost last; 64 elements = 8 pixels x 8 channels = 128 bytes): a box of 64 x 17 x chunks x 1 at
// group x0 / 8 is one input row of the 128-pixel tile starting at x0 with its halo (pixels x0 - 1 ..
// x0 + 134), landing in shared memory as [chunk][136 pixels][8 channels].
int make_row_map(SwUpscaler* u, const Planes& p, CUtensorMap* out)
{
	// the driver's function is the same for every device and thread
	static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
		cudaDriverEntryPointQueryResult q;
		void* fn = nullptr;
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
			q != cudaDriverEntryPointSuccess)
		{
			cudaGetLastError();
			fn = nullptr;
		}
		return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
	}();
	if (!encode) return fail(u, SW_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
	if (p.wp % 8) return fail(u, SW_ERR_KERNEL, "row planes: padded width %u not a multiple of 8", p.wp);
	const cuuint64_t dims[4] = {64, p.wp / 8, p.chunks, cuuint64_t(p.images) * p.rows_alloc};
	const cuuint64_t strides[3] = {128, cuuint64_t(p.wp) * 16, cuuint64_t(p.chunks) * p.wp * 16}; // bytes, dims 1..3
	const cuuint32_t box[4] = {64, CXS / 8, p.chunks, 1};
	const cuuint32_t estr[4] = {1, 1, 1, 1};
	const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, p.data, dims, strides, box, estr,
		CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
		CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) return fail(u, SW_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", int(r));
	return SW_OK;
}

// Persistent grid: as many CTAs as fit on one SM at once (shared memory, and TMEM: 512 columns per SM)
// on every SM, at least 2 output rows each.
template <int C8, int N, int EPI>
int launch_conv(SwUpscaler* u, ConvArgs a, cudaStream_t s)
{
	a.error = static_cast<int*>(u->error.ptr);
	if (a.in.chunks != uint32_t(C8)) return fail(u, SW_ERR_KERNEL, "convolution input has %u chunks, kernel %d", a.in.chunks, C8);
	int r = make_row_map(u, a.in, &a.in_map);
	if (r) return r;
	constexpr uint32_t smem = conv_smem_bytes<C8, N>();
	constexpr int tmem_cols = int(conv_tmem_cols<N>());
	constexpr int KEY = (C8 / 2) * 16 + (N / 16) * 4 + EPI;
	static_assert(KEY < SwUpscaler::CONV_KEYS, "instances");
	int per_sm = u->conv_per_sm[KEY].load(std::memory_order_relaxed);
	if (!per_sm)
	{
		UP_CUDA(u, cudaFuncSetAttribute(conv_kernel<C8, N, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
		UP_CUDA(u, cudaFuncSetAttribute(conv_kernel<C8, N, EPI>, cudaFuncAttributePreferredSharedMemoryCarveout,
							 int(cudaSharedmemCarveoutMaxShared)));
		int smem_sm = 0;
		UP_CUDA(u, cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, u->device));
		const int by_smem = smem_sm / int(smem + 1024); // 1 KB reserved per CTA
		per_sm = std::max(1, std::min(by_smem, 512 / tmem_cols));
		u->conv_per_sm[KEY].store(per_sm, std::memory_order_relaxed);
	}
	const uint32_t rows = a.in.images * ((a.in.width + TILE_X - 1) / TILE_X) * a.in.height;
	const uint32_t blocks = std::max(1u, std::min(uint32_t(u->num_sms * per_sm), (rows + 1) / 2));
	if (EPI == EPI_LOSS)
	{
		if (blocks * 4 > u->loss_partial.bytes) return fail(u, SW_ERR_LIMIT, "loss partial buffer too small");
		u->loss_ctas = blocks;
	}
	UP_CUDA(u, launch_dependent(conv_kernel<C8, N, EPI>, dim3(blocks), dim3(CONV_THREADS), smem, s, a));
	return SW_OK;
}

constexpr uint32_t WGRAD_CTAS_PER_CROP =
	(SW_UPSCALER_CROP_W + TILE_X - 1) / TILE_X * ((SW_UPSCALER_CROP_H + ROWS - 1) / ROWS);

int launch_wgrad(SwUpscaler* u, const Planes (&x)[NUM_LAYERS], const Planes (&g)[NUM_LAYERS], cudaStream_t s)
{
	WgradArgs a;
	a.blocks = x[0].images * WGRAD_CTAS_PER_CROP;
	for (int l = 0; l < NUM_LAYERS; ++l)
	{
		a.layer[l] = WgradLayer{x[l], g[l], static_cast<float*>(u->partial[l].ptr)};
		if (x[l].chunks != uint32_t(LAYERS[l].c8_in) || g[l].chunks != uint32_t(LAYERS[l].n_out / 8) || x[l].wp != CXS || g[l].wp != CXS)
			return fail(u, SW_ERR_KERNEL, "layer %d: planes of another shape", l);
		if (size_t(a.blocks) * wgrad_partial_floats(LAYERS[l].c8_in, LAYERS[l].n_out) * 4 > u->partial[l].bytes)
			return fail(u, SW_ERR_LIMIT, "weight-gradient partial buffer too small");
	}
	a.error = static_cast<int*>(u->error.ptr);
	if (!u->wgrad_ready.load(std::memory_order_relaxed))
	{
		UP_CUDA(u, cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WgradSmem::TOTAL));
		u->wgrad_ready.store(true, std::memory_order_relaxed);
	}
	UP_CUDA(u, launch_dependent(wgrad_kernel, dim3(a.blocks * NUM_LAYERS), dim3(128), WgradSmem::TOTAL, s, a));
	return SW_OK;
}

AdamArgs adam_args(SwUpscaler* u, int update, float lr)
{
	AdamArgs a;
	a.params = static_cast<float*>(u->params.ptr);
	a.m = static_cast<float*>(u->adam_m.ptr);
	a.v = static_cast<float*>(u->adam_v.ptr);
	a.grads = static_cast<const float*>(u->grads.ptr);
	a.lr = lr;
	a.beta1 = 0.9f;
	a.beta2 = 0.999f;
	a.eps = 1e-8f;
	const double t = double(u->steps + (update ? 1 : 0));
	a.bc1 = float(1.0 - std::pow(0.9, t));
	a.bc2 = float(1.0 - std::pow(0.999, t));
	a.update = update;
	for (int l = 0; l < NUM_LAYERS; ++l)
	{
		a.wfwd[l] = static_cast<uint16_t*>(u->wfwd[l].ptr);
		a.wbwd[l] = l > 0 ? static_cast<uint16_t*>(u->wbwd[l].ptr) : nullptr;
		a.bias[l] = static_cast<float*>(u->bias[l].ptr);
	}
	return a;
}

int pack_weights(SwUpscaler* u, cudaStream_t s)
{
	adam_pack_kernel<<<(SW_UPSCALER_NUM_PARAMS + 255) / 256, 256, 0, s>>>(adam_args(u, 0, 0.0f));
	UP_CUDA(u, cudaGetLastError());
	return SW_OK;
}

// The gradients from the step's partials, and with `update` the Adam step.
int reduce_gradients(SwUpscaler* u, uint32_t num_crops, uint32_t count, int update, float lr, cudaStream_t s)
{
	ReduceArgs a;
	for (int l = 0; l < NUM_LAYERS; ++l) a.partial[l] = static_cast<const float*>(u->partial[l].ptr);
	a.num_ctas = num_crops * WGRAD_CTAS_PER_CROP;
	a.scale = 1.0f / float(count);
	a.grads = static_cast<float*>(u->grads.ptr);
	a.adam = adam_args(u, update, lr);
	UP_CUDA(u, launch_dependent(wgrad_reduce_kernel, dim3(reduce_first(NUM_LAYERS)), dim3(REDUCE_WARPS * 32), 0, s, a));
	if (update) ++u->steps;
	return SW_OK;
}

// The failure path every upscaler kernel takes when a bounded mbarrier wait runs out, on a barrier
// that nothing completes: one CTA allocates TMEM as the kernels do, arms an mbarrier with one arrival
// and 16 transaction bytes that no copy will ever deliver (no copy or MMA is issued, so nothing is in
// flight), waits at most max_polls polls, then records code 5 in the error flag, frees the TMEM and
// returns - the recovery the real kernels run.
__global__ void __launch_bounds__(128) wait_probe_kernel(int* error, uint32_t max_polls)
{
	__shared__ __align__(8) uint64_t bar;
	__shared__ uint32_t s_tmem;
	if (threadIdx.x == 0)
	{
		mbar_init(&bar, 1);
		fence_mbar_init();
	}
	if (threadIdx.x < 32)
	{
		tmem_alloc(&s_tmem, 32);
		tmem_relinquish();
	}
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	const uint32_t tmem = s_tmem;
	if (threadIdx.x == 0) mbar_expect_tx(&bar, 16);
	__syncthreads();
	const bool completed = mbar_wait_bounded(&bar, 0, max_polls);
	if (__syncthreads_or(!completed) && threadIdx.x == 0) atomicExch(error, 5);
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	if (threadIdx.x < 32) tmem_dealloc(tmem, 32);
}

int check_error_flag(SwUpscaler* u, cudaStream_t s)
{
	int h = 0;
	UP_CUDA(u, cudaMemcpyAsync(&h, u->error.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
	UP_CUDA(u, cudaStreamSynchronize(s));
	if (h) return fail(u, SW_ERR_KERNEL, "upscaler kernel gave up waiting (code %d)", h);
	return SW_OK;
}

int prepare_training(SwUpscaler* u, uint32_t n)
{
	if (n > u->crops_capacity)
	{
		const uint32_t W = SW_UPSCALER_CROP_W, H = SW_UPSCALER_CROP_H;
		const uint32_t cap = SW_UPSCALER_MAX_CROPS;
		int r;
		if ((r = dev_alloc(u, u->t_x0, planes_bytes(cap, W, H, 2)))) return r;
		for (int i = 0; i < 3; ++i)
		{
			if ((r = dev_alloc(u, u->t_a[i], planes_bytes(cap, W, H, 4)))) return r;
			if ((r = dev_alloc(u, u->t_g[i], planes_bytes(cap, W, H, 4)))) return r;
		}
		if ((r = dev_alloc(u, u->t_g4, planes_bytes(cap, W, H, 2)))) return r;
		const size_t ctas = size_t(cap) * (H / ROWS) * ((W + TILE_X - 1) / TILE_X);
		for (int l = 0; l < NUM_LAYERS; ++l)
			if ((r = dev_alloc(u, u->partial[l], ctas * wgrad_partial_floats(LAYERS[l].c8_in, LAYERS[l].n_out) * 4, false))) return r;
		if ((r = dev_alloc(u, u->loss_partial, std::max<size_t>(ctas, 4096) * 4, false))) return r;
		if ((r = dev_alloc(u, u->crops, cap * sizeof(CropGpu), false))) return r;
		if (!u->h_stage.ptr)
		{
			const size_t hb = cap * sizeof(CropGpu) + std::max<size_t>(ctas, 4096) * 4;
			UP_CUDA(u, cudaMallocHost(&u->h_stage.ptr, hb));
			u->h_stage.bytes = hb;
		}
		u->crops_capacity = cap;
	}
	return SW_OK;
}

// Forward + backward of the crops; gradients (canonical, scaled by 1/n) end in u->grads.
int forward_backward(SwUpscaler* u, const SwUpscalerCrop* crops, uint32_t n, uint32_t* loss_count)
{
	if (!crops || n == 0 || n > SW_UPSCALER_MAX_CROPS) return fail(u, SW_ERR_INVALID_ARGUMENT, "bad crop list");
	const uint32_t W = SW_UPSCALER_CROP_W, H = SW_UPSCALER_CROP_H, M = SW_UPSCALER_CROP_MARGIN;
	for (uint32_t i = 0; i < n; ++i)
	{
		const SwUpscalerCrop& c = crops[i];
		if (!c.lo || !c.hi || c.lo_pitch < c.lo_width || c.hi_pitch < 2 * c.lo_width || (c.hi_pitch & 1) ||
			(reinterpret_cast<uintptr_t>(c.hi) & 7) || c.x < 0 || c.y < 0 ||
			uint64_t(c.x) + W > c.lo_width || uint64_t(c.y) + H > c.lo_height)
			return fail(u, SW_ERR_INVALID_ARGUMENT, "crop %u outside its frame", i);
	}
	int r = prepare_training(u, n);
	if (r) return r;
	cudaStream_t s = u->stream;
	// Crop table through pinned staging (wait for the previous step's use of it first).
	UP_CUDA(u, cudaEventSynchronize(u->ev));
	CropGpu* hc = static_cast<CropGpu*>(u->h_stage.ptr);
	for (uint32_t i = 0; i < n; ++i)
	{
		const SwUpscalerCrop& c = crops[i];
		hc[i] = CropGpu{c.lo, c.hi, c.lo_width, c.lo_height, c.lo_pitch, c.hi_pitch, c.x, c.y};
	}
	UP_CUDA(u, cudaMemcpyAsync(u->crops.ptr, hc, n * sizeof(CropGpu), cudaMemcpyHostToDevice, s));
	UP_CUDA(u, cudaEventRecord(u->ev, s));

	const Planes x0 = make_planes(u->t_x0.ptr, n, W, H, 2);
	Planes A[3], G[3];
	for (int i = 0; i < 3; ++i)
	{
		A[i] = make_planes(u->t_a[i].ptr, n, W, H, 4);
		G[i] = make_planes(u->t_g[i].ptr, n, W, H, 4);
	}
	const Planes g4 = make_planes(u->t_g4.ptr, n, W, H, 2);
	const CropGpu* dcrops = static_cast<const CropGpu*>(u->crops.ptr);

	convert_input_kernel<<<dim3((W * H + 255) / 256, n), 256, 0, s>>>(dcrops, x0);
	UP_CUDA(u, cudaGetLastError());
	ConvArgs a{};
	a.crops = dcrops;
	a.margin = M;
	// forward
	a.in = x0, a.out = A[0], a.wpack = static_cast<uint16_t*>(u->wfwd[0].ptr), a.bias = static_cast<float*>(u->bias[0].ptr);
	if ((r = launch_conv<2, 32, EPI_RELU>(u, a, s))) return r;
	a.in = A[0], a.out = A[1], a.wpack = static_cast<uint16_t*>(u->wfwd[1].ptr), a.bias = static_cast<float*>(u->bias[1].ptr);
	if ((r = launch_conv<4, 32, EPI_RELU>(u, a, s))) return r;
	a.in = A[1], a.out = A[2], a.wpack = static_cast<uint16_t*>(u->wfwd[2].ptr), a.bias = static_cast<float*>(u->bias[2].ptr);
	if ((r = launch_conv<4, 32, EPI_RELU>(u, a, s))) return r;
	a.in = A[2], a.out = g4, a.wpack = static_cast<uint16_t*>(u->wfwd[3].ptr), a.bias = static_cast<float*>(u->bias[3].ptr);
	a.loss_partial = static_cast<float*>(u->loss_partial.ptr);
	if ((r = launch_conv<4, 16, EPI_LOSS>(u, a, s))) return r;

	const uint32_t count = n * (W - 2 * M) * (H - 2 * M) * 4 * 3;
	*loss_count = count;
	// layer 3 (32 -> 12): input gradient into G[2] masked by A[2]
	ConvArgs b{};
	b.in = g4, b.out = G[2], b.mask = A[2], b.wpack = static_cast<uint16_t*>(u->wbwd[3].ptr);
	if ((r = launch_conv<2, 32, EPI_MASK>(u, b, s))) return r;
	// layer 2
	b.in = G[2], b.out = G[1], b.mask = A[1], b.wpack = static_cast<uint16_t*>(u->wbwd[2].ptr);
	if ((r = launch_conv<4, 32, EPI_MASK>(u, b, s))) return r;
	// layer 1
	b.in = G[1], b.out = G[0], b.mask = A[0], b.wpack = static_cast<uint16_t*>(u->wbwd[1].ptr);
	if ((r = launch_conv<4, 32, EPI_MASK>(u, b, s))) return r;
	// the weight gradients of every layer; layer 0 (3 -> 32) has no other
	const Planes wx[NUM_LAYERS] = {x0, A[0], A[1], A[2]}, wg[NUM_LAYERS] = {G[0], G[1], G[2], g4};
	if ((r = launch_wgrad(u, wx, wg, s))) return r;
	return SW_OK;
}

int read_loss(SwUpscaler* u, uint32_t count, float* out_mse)
{
	const uint32_t ctas = u->loss_ctas;
	float* h = reinterpret_cast<float*>(static_cast<unsigned char*>(u->h_stage.ptr) + SW_UPSCALER_MAX_CROPS * sizeof(CropGpu));
	UP_CUDA(u, cudaMemcpyAsync(h, u->loss_partial.ptr, ctas * 4, cudaMemcpyDeviceToHost, u->stream));
	int r = check_error_flag(u, u->stream);
	if (r) return r;
	double s = 0.0;
	for (uint32_t i = 0; i < ctas; ++i) s += h[i];
	*out_mse = float(s / double(count));
	return SW_OK;
}

} // namespace

extern "C" {

int sw_upscaler_create(int device, uint64_t seed, SwUpscaler** out)
{
	if (!out) return SW_ERR_INVALID_ARGUMENT;
	*out = nullptr;
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
	{
		cudaGetLastError();
		return SW_ERR_NO_DEVICE;
	}
	SwUpscaler* u = new (std::nothrow) SwUpscaler();
	if (!u) return SW_ERR_OUT_OF_MEMORY;
	u->device = device;
	int r = SW_OK;
	auto bail = [&](int code) {
		sw_upscaler_destroy(u);
		return code;
	};
	if (cudaSetDevice(device) != cudaSuccess) return bail(SW_ERR_CUDA);
	if (cudaDeviceGetAttribute(&u->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return bail(SW_ERR_CUDA);
	if (cudaStreamCreateWithFlags(&u->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(SW_ERR_CUDA); // before any dev_alloc
	if (cudaEventCreateWithFlags(&u->ev, cudaEventDisableTiming) != cudaSuccess) return bail(SW_ERR_CUDA);
	if (cudaEventRecord(u->ev, u->stream) != cudaSuccess) return bail(SW_ERR_CUDA);
	const size_t pb = SW_UPSCALER_NUM_PARAMS * sizeof(float);
	if ((r = dev_alloc(u, u->params, pb)) || (r = dev_alloc(u, u->adam_m, pb)) || (r = dev_alloc(u, u->adam_v, pb)) ||
		(r = dev_alloc(u, u->grads, pb)) || (r = dev_alloc(u, u->error, 16)) || (r = dev_alloc(u, u->psnr_sum, 16)))
		return bail(r);
	for (int l = 0; l < NUM_LAYERS; ++l)
	{
		const LayerShape& L = LAYERS[l];
		if ((r = dev_alloc(u, u->wfwd[l], size_t(9) * L.c8_in * 8 * L.n_out * 2))) return bail(r);
		if (l > 0 && (r = dev_alloc(u, u->wbwd[l], size_t(9) * L.n_out * L.c8_in * 8 * 2))) return bail(r);
		if ((r = dev_alloc(u, u->bias[l], size_t(L.n_out) * 4))) return bail(r);
	}
	if (cudaMallocHost(reinterpret_cast<void**>(&u->h_psnr), sizeof(unsigned long long)) != cudaSuccess) return bail(SW_ERR_CUDA);
	// Seeded He-normal initialisation (Box-Muller over splitmix64), zero biases, last layer / 10.
	std::vector<float> p(SW_UPSCALER_NUM_PARAMS, 0.0f);
	uint64_t st = seed;
	for (int l = 0; l < NUM_LAYERS; ++l)
	{
		const LayerShape& L = LAYERS[l];
		const float sd = std::sqrt(2.0f / float(9 * L.cin)) * (l == NUM_LAYERS - 1 ? 0.1f : 1.0f);
		const int nw = L.cout * 9 * L.cin;
		for (int i = 0; i < nw; ++i)
		{
			const double u1 = (double(splitmix(st) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
			const double u2 = double(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
			p[L.param_offset + i] = float(std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2)) * sd;
		}
	}
	if ((r = sw_upscaler_set_params(u, p.data(), SW_UPSCALER_NUM_PARAMS))) return bail(r);
	*out = u;
	return SW_OK;
}

int sw_upscaler_destroy(SwUpscaler* u)
{
	if (!u) return SW_ERR_INVALID_ARGUMENT;
	cudaSetDevice(u->device);
	if (u->stream) cudaStreamSynchronize(u->stream);
	DevMem* all[] = {&u->params, &u->adam_m, &u->adam_v, &u->grads, &u->error, &u->t_x0, &u->t_g4,
		&u->loss_partial, &u->crops, &u->i_x0, &u->i_p, &u->i_q, &u->i_crop, &u->psnr_sum};
	for (DevMem* m : all) dev_free(*m);
	for (int i = 0; i < 3; ++i)
	{
		dev_free(u->t_a[i]);
		dev_free(u->t_g[i]);
	}
	for (int l = 0; l < NUM_LAYERS; ++l)
	{
		dev_free(u->partial[l]);
		dev_free(u->wfwd[l]);
		dev_free(u->wbwd[l]);
		dev_free(u->bias[l]);
	}
	if (u->h_stage.ptr) cudaFreeHost(u->h_stage.ptr);
	if (u->h_psnr) cudaFreeHost(u->h_psnr);
	if (u->ev) cudaEventDestroy(u->ev);
	if (u->stream) cudaStreamDestroy(u->stream);
	delete u;
	return SW_OK;
}

const char* sw_upscaler_last_error(const SwUpscaler* u) { return u ? u->last_error.c_str() : "null upscaler"; }

int sw_upscaler_get_params(SwUpscaler* u, float* params, uint32_t count)
{
	if (!u || !params || count != SW_UPSCALER_NUM_PARAMS) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	UP_CUDA(u, cudaMemcpyAsync(params, u->params.ptr, count * 4, cudaMemcpyDeviceToHost, u->stream));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	return SW_OK;
}

int sw_upscaler_set_params(SwUpscaler* u, const float* params, uint32_t count)
{
	if (!u || !params || count != SW_UPSCALER_NUM_PARAMS) return SW_ERR_INVALID_ARGUMENT;
	for (uint32_t i = 0; i < count; ++i)
		if (!std::isfinite(params[i])) return fail(u, SW_ERR_INVALID_ARGUMENT, "parameter %u is not finite", i);
	UP_CUDA(u, cudaSetDevice(u->device));
	UP_CUDA(u, cudaMemcpyAsync(u->params.ptr, params, count * 4, cudaMemcpyHostToDevice, u->stream));
	UP_CUDA(u, cudaMemsetAsync(u->adam_m.ptr, 0, count * 4, u->stream));
	UP_CUDA(u, cudaMemsetAsync(u->adam_v.ptr, 0, count * 4, u->stream));
	u->steps = 0;
	int r = pack_weights(u, u->stream);
	if (r) return r;
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	return SW_OK;
}

int sw_upscaler_gradients(SwUpscaler* u, const SwUpscalerCrop* crops, uint32_t num_crops, float* grads, float* loss)
{
	if (!u || !grads) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	uint32_t count = 0;
	int r = forward_backward(u, crops, num_crops, &count);
	if (r) return r;
	if ((r = reduce_gradients(u, num_crops, count, 0, 0.0f, u->stream))) return r;
	UP_CUDA(u, cudaMemcpyAsync(grads, u->grads.ptr, SW_UPSCALER_NUM_PARAMS * 4, cudaMemcpyDeviceToHost, u->stream));
	float mse = 0.0f;
	if ((r = read_loss(u, count, &mse))) return r;
	if (loss) *loss = 0.5f * mse;
	return SW_OK;
}

int sw_upscaler_train_step(SwUpscaler* u, const SwUpscalerCrop* crops, uint32_t num_crops, float lr, float* mse)
{
	if (!u || !(lr >= 0.0f)) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	uint32_t count = 0;
	int r = forward_backward(u, crops, num_crops, &count);
	if (r) return r;
	if ((r = reduce_gradients(u, num_crops, count, 1, lr, u->stream))) return r;
	if (mse) return read_loss(u, count, mse);
	return SW_OK;
}

int sw_upscaler_steps(SwUpscaler* u, uint64_t* out)
{
	if (!u || !out) return SW_ERR_INVALID_ARGUMENT;
	*out = u->steps;
	return SW_OK;
}

int sw_upscaler_infer(SwUpscaler* u, const uint32_t* lo, uint32_t lo_width, uint32_t lo_height, uint32_t lo_pitch, uint32_t* hi,
	uint32_t hi_pitch, void* stream)
{
	if (!u || !lo || !hi || lo_width == 0 || lo_height == 0 || lo_pitch < lo_width || hi_pitch < 2 * lo_width ||
		(hi_pitch & 1) || (reinterpret_cast<uintptr_t>(hi) & 7))
		return SW_ERR_INVALID_ARGUMENT; // output pixel pairs are stored as 8-byte words
	if (lo_width > 8192 || lo_height > 8192) return fail(u, SW_ERR_LIMIT, "frame too large");
	UP_CUDA(u, cudaSetDevice(u->device));
	cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : u->stream;
	int r;
	if (u->fused)
	{
		if (!u->fused_ready.load(std::memory_order_relaxed))
		{
			UP_CUDA(u, cudaFuncSetAttribute(fused_upscale_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FusedSmem::TOTAL));
			u->fused_ready.store(true, std::memory_order_relaxed);
		}
		FusedArgs f;
		f.lo = lo;
		f.lo_w = lo_width;
		f.lo_h = lo_height;
		f.lo_pitch = lo_pitch;
		f.hi = hi;
		f.hi_pitch = hi_pitch;
		for (int l = 0; l < NUM_LAYERS; ++l)
		{
			f.w[l] = static_cast<const uint16_t*>(u->wfwd[l].ptr);
			f.bias[l] = static_cast<const float*>(u->bias[l].ptr);
		}
		f.strips = (lo_width + F_VALID - 1) / F_VALID;
		f.segments = std::max(1u, std::min(lo_height, uint32_t(u->num_sms) / f.strips));
		f.error = static_cast<int*>(u->error.ptr);
		UP_CUDA(u, launch_dependent(fused_upscale_kernel, dim3(f.strips * f.segments), dim3(F_THREADS), FusedSmem::TOTAL, s, f));
		return SW_OK;
	}
	if (lo_width != u->i_w || lo_height != u->i_h)
	{
		UP_CUDA(u, cudaStreamSynchronize(s));
		UP_CUDA(u, cudaStreamSynchronize(u->stream));
		dev_free(u->i_x0);
		dev_free(u->i_p);
		dev_free(u->i_q);
		if ((r = dev_alloc(u, u->i_x0, planes_bytes(1, lo_width, lo_height, 2)))) return r;
		if ((r = dev_alloc(u, u->i_p, planes_bytes(1, lo_width, lo_height, 4)))) return r;
		if ((r = dev_alloc(u, u->i_q, planes_bytes(1, lo_width, lo_height, 4)))) return r;
		if ((r = dev_alloc(u, u->i_crop, sizeof(CropGpu)))) return r;
		u->i_crop_valid = false;
		u->i_w = lo_width;
		u->i_h = lo_height;
	}
	// The frame record (source pointer, size, pitches) is re-uploaded only when it changes; the copy
	// from pageable memory is staged before cudaMemcpyAsync returns.
	const CropGpu c{lo, nullptr, lo_width, lo_height, lo_pitch, hi_pitch, 0, 0};
	if (!u->i_crop_valid || memcmp(&c, &u->i_crop_host, sizeof(c)) != 0)
	{
		UP_CUDA(u, cudaMemcpyAsync(u->i_crop.ptr, &c, sizeof(c), cudaMemcpyHostToDevice, s));
		u->i_crop_host = c;
		u->i_crop_valid = true;
	}
	const Planes x0 = make_planes(u->i_x0.ptr, 1, lo_width, lo_height, 2);
	const Planes P = make_planes(u->i_p.ptr, 1, lo_width, lo_height, 4);
	const Planes Q = make_planes(u->i_q.ptr, 1, lo_width, lo_height, 4);
	const CropGpu* dc = static_cast<const CropGpu*>(u->i_crop.ptr);
	convert_input_kernel<<<dim3((lo_width * lo_height + 255) / 256, 1), 256, 0, s>>>(dc, x0);
	UP_CUDA(u, cudaGetLastError());
	ConvArgs a{};
	a.crops = dc;
	a.hi_out = hi;
	a.hi_pitch = hi_pitch;
	a.in = x0, a.out = P, a.wpack = static_cast<uint16_t*>(u->wfwd[0].ptr), a.bias = static_cast<float*>(u->bias[0].ptr);
	if ((r = launch_conv<2, 32, EPI_RELU>(u, a, s))) return r;
	a.in = P, a.out = Q, a.wpack = static_cast<uint16_t*>(u->wfwd[1].ptr), a.bias = static_cast<float*>(u->bias[1].ptr);
	if ((r = launch_conv<4, 32, EPI_RELU>(u, a, s))) return r;
	a.in = Q, a.out = P, a.wpack = static_cast<uint16_t*>(u->wfwd[2].ptr), a.bias = static_cast<float*>(u->bias[2].ptr);
	if ((r = launch_conv<4, 32, EPI_RELU>(u, a, s))) return r;
	a.in = P, a.wpack = static_cast<uint16_t*>(u->wfwd[3].ptr), a.bias = static_cast<float*>(u->bias[3].ptr);
	if ((r = launch_conv<4, 16, EPI_INFER>(u, a, s))) return r;
	return SW_OK;
}

int sw_upscaler_set_fused(SwUpscaler* u, int enable)
{
	if (!u) return SW_ERR_INVALID_ARGUMENT;
	u->fused = enable != 0;
	return SW_OK;
}

int sw_upscaler_wait_probe(SwUpscaler* u, uint32_t max_polls, int* out_code)
{
	if (!u || !out_code || max_polls == 0 || max_polls > POLL_LIMIT) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	int prior = 0;
	UP_CUDA(u, cudaMemcpy(&prior, u->error.ptr, sizeof(int), cudaMemcpyDeviceToHost));
	if (prior) return fail(u, SW_ERR_STATE, "an earlier kernel already gave up (code %d)", prior);
	wait_probe_kernel<<<1, 128, 0, u->stream>>>(static_cast<int*>(u->error.ptr), max_polls);
	UP_CUDA(u, cudaGetLastError());
	UP_CUDA(u, cudaMemcpyAsync(out_code, u->error.ptr, sizeof(int), cudaMemcpyDeviceToHost, u->stream));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	// the probe's record is not a failure of the upscaler's work: clear it
	UP_CUDA(u, cudaMemsetAsync(u->error.ptr, 0, sizeof(int), u->stream));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	return SW_OK;
}

int sw_upscaler_check(SwUpscaler* u)
{
	if (!u) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	UP_CUDA(u, cudaDeviceSynchronize());
	return check_error_flag(u, u->stream);
}

int sw_upscaler_psnr(SwUpscaler* u, const uint32_t* a, uint32_t a_pitch, const uint32_t* b, uint32_t b_pitch, uint32_t width,
	uint32_t height, void* stream, double* out_psnr)
{
	if (!u || !a || !b || !out_psnr || width == 0 || height == 0 || a_pitch < width || b_pitch < width)
		return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : u->stream;
	UP_CUDA(u, cudaMemsetAsync(u->psnr_sum.ptr, 0, 8, s));
	psnr_kernel<<<1216, 256, 0, s>>>(a, a_pitch, b, b_pitch, width, height, static_cast<unsigned long long*>(u->psnr_sum.ptr));
	UP_CUDA(u, cudaGetLastError());
	UP_CUDA(u, cudaMemcpyAsync(u->h_psnr, u->psnr_sum.ptr, 8, cudaMemcpyDeviceToHost, s));
	UP_CUDA(u, cudaStreamSynchronize(s));
	const double mse = double(*u->h_psnr) / (3.0 * double(width) * double(height));
	*out_psnr = mse <= 0.0 ? 99.0 : std::min(99.0, 10.0 * std::log10(255.0 * 255.0 / mse));
	return SW_OK;
}

// Checkpoint file: magic "SWUPSCL1", u32 version, u32 num_params, u64 steps, params, m, v (f32 each),
// then the FNV-1a 64 hash of everything before it.
int sw_upscaler_save(SwUpscaler* u, const char* path)
{
	if (!u || !path) return SW_ERR_INVALID_ARGUMENT;
	UP_CUDA(u, cudaSetDevice(u->device));
	const size_t n = SW_UPSCALER_NUM_PARAMS;
	std::vector<unsigned char> buf(8 + 4 + 4 + 8 + 3 * n * 4);
	memcpy(buf.data(), "SWUPSCL1", 8);
	const uint32_t version = 1, np = uint32_t(n);
	memcpy(buf.data() + 8, &version, 4);
	memcpy(buf.data() + 12, &np, 4);
	memcpy(buf.data() + 16, &u->steps, 8);
	unsigned char* p = buf.data() + 24;
	UP_CUDA(u, cudaMemcpyAsync(p, u->params.ptr, n * 4, cudaMemcpyDeviceToHost, u->stream));
	UP_CUDA(u, cudaMemcpyAsync(p + n * 4, u->adam_m.ptr, n * 4, cudaMemcpyDeviceToHost, u->stream));
	UP_CUDA(u, cudaMemcpyAsync(p + 2 * n * 4, u->adam_v.ptr, n * 4, cudaMemcpyDeviceToHost, u->stream));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	const uint64_t h = fnv1a(buf.data(), buf.size());
	FILE* f = fopen(path, "wb");
	if (!f) return fail(u, SW_ERR_INVALID_ARGUMENT, "cannot open %s", path);
	const bool ok = fwrite(buf.data(), 1, buf.size(), f) == buf.size() && fwrite(&h, 1, 8, f) == 8;
	fclose(f);
	return ok ? SW_OK : fail(u, SW_ERR_INVALID_ARGUMENT, "write to %s failed", path);
}

int sw_upscaler_load(SwUpscaler* u, const char* path)
{
	if (!u || !path) return SW_ERR_INVALID_ARGUMENT;
	const size_t n = SW_UPSCALER_NUM_PARAMS;
	std::vector<unsigned char> buf(8 + 4 + 4 + 8 + 3 * n * 4 + 8);
	FILE* f = fopen(path, "rb");
	if (!f) return fail(u, SW_ERR_INVALID_ARGUMENT, "cannot open %s", path);
	const size_t got = fread(buf.data(), 1, buf.size(), f);
	const int extra = fgetc(f);
	fclose(f);
	if (got != buf.size() || extra != EOF) return fail(u, SW_ERR_INVALID_ARGUMENT, "%s: wrong size", path);
	uint32_t version, np;
	memcpy(&version, buf.data() + 8, 4);
	memcpy(&np, buf.data() + 12, 4);
	if (memcmp(buf.data(), "SWUPSCL1", 8) != 0 || version != 1 || np != n)
		return fail(u, SW_ERR_INVALID_ARGUMENT, "%s: not an upscaler checkpoint of this version", path);
	uint64_t h;
	memcpy(&h, buf.data() + buf.size() - 8, 8);
	if (fnv1a(buf.data(), buf.size() - 8) != h) return fail(u, SW_ERR_INVALID_ARGUMENT, "%s: hash mismatch", path);
	uint64_t steps;
	memcpy(&steps, buf.data() + 16, 8);
	const float* p = reinterpret_cast<const float*>(buf.data() + 24);
	int r = sw_upscaler_set_params(u, p, uint32_t(n));
	if (r) return r;
	UP_CUDA(u, cudaMemcpyAsync(u->adam_m.ptr, p + n, n * 4, cudaMemcpyHostToDevice, u->stream));
	UP_CUDA(u, cudaMemcpyAsync(u->adam_v.ptr, p + 2 * n, n * 4, cudaMemcpyHostToDevice, u->stream));
	UP_CUDA(u, cudaStreamSynchronize(u->stream));
	u->steps = steps;
	return SW_OK;
}

int sw_monitor_init(SwMonitor* m, uint32_t check_interval, float threshold_db, uint32_t fallback_frames)
{
	if (!m || check_interval == 0 || fallback_frames == 0 || !std::isfinite(threshold_db)) return SW_ERR_INVALID_ARGUMENT;
	memset(m, 0, sizeof(*m));
	m->check_interval = check_interval;
	m->fallback_frames = fallback_frames;
	m->threshold_db = threshold_db;
	m->recheck = 1; // the first learned frame is checked
	return SW_OK;
}

int sw_monitor_plan(SwMonitor* m, uint32_t* out_plan)
{
	if (!m || !out_plan || m->check_interval == 0) return SW_ERR_INVALID_ARGUMENT;
	if (m->check_pending) return SW_ERR_STATE; // the last checked frame has no report yet
	++m->frames;
	if (m->plain_left > 0)
	{
		--m->plain_left;
		++m->plain_frames;
		*out_plan = SW_PLAN_PLAIN;
		return SW_OK;
	}
	++m->learned_frames;
	if (m->recheck || m->since_check + 1 >= m->check_interval)
	{
		m->recheck = 0;
		m->since_check = 0;
		m->check_pending = 1;
		++m->checks;
		*out_plan = SW_PLAN_LEARNED_CHECKED;
		return SW_OK;
	}
	++m->since_check;
	*out_plan = SW_PLAN_LEARNED;
	return SW_OK;
}

int sw_monitor_report(SwMonitor* m, double psnr_db)
{
	if (!m) return SW_ERR_INVALID_ARGUMENT;
	if (!m->check_pending) return SW_ERR_STATE;
	m->check_pending = 0;
	m->last_psnr_db = float(psnr_db);
	if (!(psnr_db >= double(m->threshold_db))) // NaN fails too
	{
		++m->failed_checks;
		++m->fallbacks;
		m->plain_left = m->fallback_frames;
		m->recheck = 1;
	}
	return SW_OK;
}

} // extern "C"
