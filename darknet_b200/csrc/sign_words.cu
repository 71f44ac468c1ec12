// fp32 tensor -> sign words on the position grid (grid_words.cuh): repack_input + float_to_bit of every image
// (src-lib/gemm.cpp:2202-2220, :1510) for any channel count.  Streams the input once; a thread packs 32 channels of 1, 2 or 4
// neighbouring pixels with 16 loads in flight.  Bound by HBM.
#include "grid_words.cuh"

namespace xnor
{

constexpr int SW_THREADS = 256;

struct SignWordsParams
{
	const float * in;
	uint32_t * words;
	int batch, C, nb, h, w, pitch, hwv;             // hwv: vectors per plane
	int front, block_words;
	FastDiv d_hwv, d_nb, d_w;
	int items;                               // batch * nb * hwv
	int pads;                                // zero words to write as well: padding, guard and fill of every block (0: they are zero already)
	int pads_img;                            // padding positions of an image
	FastDiv d_pads_img;
};

// Loads written as volatile inline PTX: the compiler otherwise folds load, compare and OR into a chain with a handful of loads
// in flight, and this kernel lives on bytes in flight.
template <int VEC> __device__ __forceinline__ void stream_load(const float * p, float (&v)[VEC])
{
	if constexpr (VEC == 4) { asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p)); }
	else if constexpr (VEC == 2) { asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p)); }
	else { asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v[0]) : "l"(p)); }
}

template <int VEC>
__global__ void __launch_bounds__(SW_THREADS)
sign_words_grid_kernel(const __grid_constant__ SignWordsParams p)
{
	pdl_trigger();
	const int idx = blockIdx.x * SW_THREADS + threadIdx.x;
	if (idx < p.items)
	{
		const int blk = fdiv(idx, p.d_hwv);
		const int ev = idx - blk * p.hwv;
		const int img = fdiv(blk, p.d_nb);
		const int cb = blk - img * p.nb;
		const size_t hw = (size_t)p.hwv * VEC;
		const int left = p.C - cb * 32;                           // channels that exist in this block
		const float * src = p.in + ((size_t)img * p.C + cb * 32) * hw + (size_t)ev * VEC;
		uint32_t word[VEC];
		#pragma unroll
		for (int j = 0; j < VEC; ++j) { word[j] = 0; }
		#pragma unroll
		for (int ch0 = 0; ch0 < 32; ch0 += 16)
		{
			float v[16][VEC];
			#pragma unroll
			for (int u = 0; u < 16; ++u)
			{
				#pragma unroll
				for (int j = 0; j < VEC; ++j) { v[u][j] = 0.0f; }
				if (ch0 + u < left) { stream_load<VEC>(src + (size_t)(ch0 + u) * hw, v[u]); }
			}
			#pragma unroll
			for (int u = 0; u < 16; ++u)
			{
				#pragma unroll
				for (int j = 0; j < VEC; ++j) { word[j] |= (v[u][j] > 0.0f ? 1u : 0u) << (ch0 + u); }
			}
		}
		int y = fdiv(ev * VEC, p.d_w);
		int x = ev * VEC - y * p.w;
		uint32_t * dst = p.words + (size_t)cb * p.block_words + p.front + (size_t)img * (p.h + 1) * p.pitch;
		#pragma unroll
		for (int j = 0; j < VEC; ++j)
		{
			dst[y * p.pitch + x] = word[j];
			if (++x == p.w) { x = 0; ++y; }
		}
		return;
	}
	// zeros of block cb: the padding of every image, then what lies in front of and behind the batch
	int q = idx - p.items;
	if (q >= p.pads) { return; }
	const int positions = p.batch * (p.h + 1) * p.pitch;
	const int per_block = p.batch * p.pads_img + p.block_words - positions;
	const int cb = q / per_block;
	q -= cb * per_block;
	uint32_t * dst = p.words + (size_t)cb * p.block_words;
	const int img = fdiv(q, p.d_pads_img);
	if (img < p.batch)
	{
		q -= img * p.pads_img;
		const int cols = p.pitch - p.w;
		const int row = (q < p.h * cols) ? q / cols : p.h;
		const int at = (row < p.h) ? row * p.pitch + p.w + q - row * cols : p.h * p.pitch + q - p.h * cols;
		dst[p.front + (size_t)img * (p.h + 1) * p.pitch + at] = 0;
		return;
	}
	q -= p.batch * p.pads_img;
	dst[(q < p.front) ? q : positions + q] = 0;                     // the fill starts at front + positions
}

int launch_sign_words_grid(const float * input, int batch, int c, int h, int w, int pitch, uint32_t * words, int write_pads, cudaStream_t stream)
{
	SignWordsParams p = {};
	p.in = input; p.words = words;
	p.batch = batch; p.C = c; p.nb = (c + 31) / 32; p.h = h; p.w = w; p.pitch = pitch;
	p.front = grid_front(pitch); p.block_words = grid_block_words(batch, h, pitch);
	p.pads_img = h * (pitch - w) + pitch;
	const long long hw = (long long)h * w;
	const long long blocks = (long long)batch * p.nb;
	// the widest loads that still give every SM two CTAs: bytes in flight per thread are what the kernel lives on
	const long long min_items = 2LL * sm_count() * SW_THREADS;
	int vec = 1;
	if (hw % 4 == 0 && ((uintptr_t)input & 15u) == 0 && blocks * (hw / 4) >= min_items) { vec = 4; }
	else if (hw % 2 == 0 && ((uintptr_t)input & 7u) == 0 && blocks * (hw / 2) >= min_items) { vec = 2; }
	p.hwv = (int)(hw / vec);
	const long long pads = write_pads ? (long long)p.nb * (batch * (long long)p.pads_img + p.block_words - batch * (long long)(h + 1) * pitch) : 0;
	if (blocks * p.hwv + pads + SW_THREADS > 0x7fffffffLL || (long long)p.nb * p.block_words > 0x7fffffffLL) { return XNOR_B200_ERR_TOO_LARGE; }
	p.items = (int)(blocks * p.hwv);
	p.pads = (int)pads;
	p.d_hwv = make_div((uint32_t)p.hwv); p.d_nb = make_div((uint32_t)p.nb); p.d_w = make_div((uint32_t)w);
	p.d_pads_img = make_div((uint32_t)p.pads_img);
	const unsigned grid = (unsigned)((p.items + (long long)p.pads + SW_THREADS - 1) / SW_THREADS);
	if (vec == 4) { sign_words_grid_kernel<4><<<grid, SW_THREADS, 0, stream>>>(p); }
	else if (vec == 2) { sign_words_grid_kernel<2><<<grid, SW_THREADS, 0, stream>>>(p); }
	else { sign_words_grid_kernel<1><<<grid, SW_THREADS, 0, stream>>>(p); }
	return check_launch();
}

}  // namespace xnor

using namespace xnor;

extern "C" int xnor_b200_sign_words(const float * input, int batch, int c, int h, int w, int pitch, uint32_t * words, void * stream)
{
	if (input == nullptr || words == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || c <= 0 || h <= 0 || w <= 0 || pitch <= w) { return XNOR_B200_ERR_INVALID; }
	if (xnor_b200_grid_block_words(batch, h, pitch) == 0) { return XNOR_B200_ERR_TOO_LARGE; }
	return launch_sign_words_grid(input, batch, c, h, w, pitch, words, 1, (cudaStream_t)stream);
}
