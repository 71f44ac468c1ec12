// Sign tensors on the position grid of xnor_conv.cu: [channel block][guard | batch * (h + 1) * pitch positions | fill], one word of
// 32 channels per position.  The padding columns behind every row and the padding row behind every image are shared by their
// neighbours and hold zeros, as does the guard, which is what the first image's upper and left neighbours read.
#pragma once

#include "xnor_common.cuh"

namespace xnor
{

inline int grid_front(int pitch) { return (int)round_up((size_t)pitch + 8, 32); }
inline int grid_block_words(int batch, int h, int pitch) { return (int)round_up((size_t)grid_front(pitch) + (size_t)batch * (h + 1) * pitch, 32); }

// n / d for 0 <= n < 2^31 by multiplication
struct FastDiv
{
	uint32_t d, mul, shift;
};

static FastDiv make_div(uint32_t d)
{
	FastDiv f = {d, 0, 0};
	if (d <= 1) { return f; }
	uint32_t s = 0;
	while ((1ull << s) < d) { ++s; }
	f.mul = (uint32_t)(((1ull << (31 + s)) + d - 1) / d);
	f.shift = s - 1;
	return f;
}

__host__ __device__ __forceinline__ int fdiv(int n, const FastDiv & f)
{
#ifdef __CUDA_ARCH__
	return (f.d <= 1) ? n : (int)(__umulhi((uint32_t)n, f.mul) >> f.shift);
#else
	return (f.d <= 1) ? n : (int)((uint32_t)(((uint64_t)(uint32_t)n * f.mul) >> 32) >> f.shift);
#endif
}

}  // namespace xnor
