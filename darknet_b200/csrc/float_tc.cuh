// Shared by the tensor-core float convolutions: float_conv_tc.cu (few pixels, unprepared filters) and float_conv_tcp.cu (batches).
#pragma once

#include "tc_common.cuh"

namespace xnor
{

constexpr int FT_NF = 128;                                 // filters per tile
constexpr int FT_TILE_BYTES = 128 * 128;                   // 128 rows x 32 tf32
constexpr int FT_MAX_SPLIT = 4;                            // CTAs that share a tile's K blocks

struct FtParams
{
	const float * x;      // [batch][C][HW]
	const float * w;      // RAW: [N][C] (1x1); else [filter tile][K block][hi, lo][128 rows x 32 channels, swizzled]
	const float * bias;   // [N] or nullptr
	float * out;          // [batch][N][HW]
	int C, HW, N;
	int total;            // batch * HW
	int H, W, taps;       // taps 1 or 9
	int cblocks;          // ceil(C / 32): K blocks per tap
	int kblocks;          // taps * cblocks
	int yolo_entries;     // > 0: the [yolo] layer's activation step is applied to the result (xnor_b200_yolo_activate)
	int leaky;
	int tiles_f;
	int split;            // CTAs per tile
	int tile0, tiles;     // first tile of the launch, tiles
	int more;             // float_conv_tcp.cu: another launch with the rest of the tiles follows
	int turn;             // float_conv_tcp.cu: tiles after which the order of the filter tiles moves on by one
	int * status;
	uint32_t spin_limit;
};

// v = hi + lo exactly: hi the nearest value of 11 significant bits (halves away from zero), so that lo, of either sign, fits 12.  An infinity
// or NaN leaves NaN in lo, and so does a value that rounds past the largest: those results are formed again (plain_sum).
__device__ __forceinline__ void split_nearest(float v, float & hi, float & lo)
{
	hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
	lo = __fsub_rn(v, hi);
}

// One result by fp32 multiply-adds from the prepared filters, for those that the split products cannot form: a factor that is infinite,
// NaN or next to the largest value.
__device__ __forceinline__ float plain_sum(const FtParams & p, int img, int pix, int f)
{
	const int py = pix / p.W, px = pix - py * p.W, row = f % FT_NF;
	const float * base = p.x + (size_t)img * p.C * p.HW + pix;
	float acc = 0.0f;
	for (int tap = 0; tap < p.taps; ++tap)
	{
		const int dy = (p.taps == 9) ? tap / 3 - 1 : 0, dx = (p.taps == 9) ? tap % 3 - 1 : 0;
		const bool inside = (py + dy >= 0 && py + dy < p.H && px + dx >= 0 && px + dx < p.W);       // else zeros, as im2col has them
		for (int c = 0; c < p.C; ++c)
		{
			const float * tile = p.w + ((size_t)(f / FT_NF) * p.kblocks + tap * p.cblocks + (c >> 5)) * (2 * FT_TILE_BYTES / 4);
			const int at = row * 32 + ((((c & 31) >> 2) ^ (row & 7)) << 2) + (c & 3);
			acc = fmaf(inside ? __ldg(base + dy * p.W + dx + (size_t)c * p.HW) : 0.0f, __ldg(tile + at) + __ldg(tile + FT_TILE_BYTES / 4 + at), acc);
		}
	}
	return acc;
}

// float_conv_tcp.cu: prepared filters, any number of pixels
int launch_float_tcp(FtParams & p, cudaStream_t stream);
// Kernels that it launches for so many tiles
int float_tcp_launches(long long tiles, int kblocks);

}  // namespace xnor
