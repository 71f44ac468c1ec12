// Direct fp32 convolution for the float layer that sits in FRONT of the xnor path (3 input channels -> 16 or 32
// filters at full image resolution in all three xnor networks), with bias and leaky/linear activation fused.
//
// Stands in for the float branch of forward_convolutional_layer_gpu (src-lib/convolutional_kernels.cu:373-434:
// cuDNN or im2col + cuBLAS sgemm), add_bias_gpu (src-lib/blas_kernels.cu) and activate_array_ongpu
// (src-lib/activation_kernels.cu:34 leaky) for layers with few input channels.  Such a layer is bound by writing
// its output (16 planes of the full-resolution image), not by arithmetic, so one pass that reads the image once
// and writes every output plane once, coalesced, is the whole optimisation; a GEMM formulation would only add an
// im2col buffer.  Accumulation order is (channel, ky, kx) with fused multiply-adds, bias added last.
#include "grid_words.cuh"

namespace xnor
{

constexpr int FC_THREADS = 256;
constexpr int FC_MAX_TAPS = 128;     // c*size*size values a thread keeps in registers
constexpr int FC_FILTERS = 16;       // filters accumulated per pass

struct FloatConvParams
{
	const float * in;
	const float * weights;   // [n][c*size*size]
	const float * biases;    // [n] or nullptr
	float * out;             // [batch][n][oh][ow]
	int batch, C, H, W, N, OH, OW;
	int ks, stride, pad;
	int leaky;
};

// CC, KS > 0: channel count and kernel size known at compile time (the 27 taps of a 3x3 RGB layer then live in
// registers); CC == 0: generic sizes, taps kept in a per-thread array.
template <int CC, int KS>
__global__ void __launch_bounds__(FC_THREADS)
float_conv_small_kernel(const FloatConvParams p)
{
	constexpr int TAPS_MAX = (CC > 0) ? CC * KS * KS : FC_MAX_TAPS;
	const int C = (CC > 0) ? CC : p.C;
	const int ks = (CC > 0) ? KS : p.ks;
	extern __shared__ float s_w[];                       // weights [n][taps] followed by biases [n]
	const int taps = C * ks * ks;
	for (int i = threadIdx.x; i < p.N * taps; i += FC_THREADS) { s_w[i] = p.weights[i]; }
	float * s_b = s_w + p.N * taps;
	for (int i = threadIdx.x; i < p.N; i += FC_THREADS) { s_b[i] = (p.biases != nullptr) ? p.biases[i] : 0.0f; }
	__syncthreads();

	const size_t plane = (size_t)p.OH * p.OW;
	const size_t total = (size_t)p.batch * plane;
	for (size_t idx = (size_t)blockIdx.x * FC_THREADS + threadIdx.x; idx < total; idx += (size_t)gridDim.x * FC_THREADS)
	{
		const int b = (int)(idx / plane);
		const int pix = (int)(idx - (size_t)b * plane);
		const int oy = pix / p.OW;
		const int ox = pix - oy * p.OW;
		const float * img = p.in + (size_t)b * C * p.H * p.W;

		float v[TAPS_MAX];
		int t = 0;
		#pragma unroll
		for (int c = 0; c < C; ++c)
		{
			#pragma unroll
			for (int ky = 0; ky < ks; ++ky)
			{
				const int iy = oy * p.stride - p.pad + ky;
				#pragma unroll
				for (int kx = 0; kx < ks; ++kx, ++t)
				{
					const int ix = ox * p.stride - p.pad + kx;
					const bool ok = (iy >= 0 && iy < p.H && ix >= 0 && ix < p.W);
					if (t < TAPS_MAX) { v[t] = ok ? __ldg(img + ((size_t)c * p.H + iy) * p.W + ix) : 0.0f; }
				}
			}
		}
		float * dst = p.out + (size_t)b * p.N * plane + pix;
		for (int f0 = 0; f0 < p.N; f0 += FC_FILTERS)
		{
			float acc[FC_FILTERS];
			#pragma unroll
			for (int f = 0; f < FC_FILTERS; ++f) { acc[f] = 0.0f; }
			#pragma unroll
			for (int k = 0; k < TAPS_MAX; ++k)
			{
				if (k < taps)
				{
					#pragma unroll
					for (int f = 0; f < FC_FILTERS; ++f)
					{
						if (f0 + f < p.N) { acc[f] = fmaf(v[k], s_w[(f0 + f) * taps + k], acc[f]); }
					}
				}
			}
			#pragma unroll
			for (int f = 0; f < FC_FILTERS; ++f)
			{
				if (f0 + f < p.N)
				{
					float r = acc[f] + s_b[f0 + f];
					if (p.leaky) { r = (r > 0.0f) ? r : r * 0.1f; }
					dst[(size_t)(f0 + f) * plane] = r;
				}
			}
		}
	}
}

// ---- 3 input channels, 3x3, stride 1, pad 1: a thread computes a 4x4 block of outputs, four filters at a time --------------
// The first layer of every xnor network.  Bound by the FMA pipe (27 multiply-adds a value) as long as nothing else is: a CTA
// stages its 32x32 tile with its border in shared memory once; a thread keeps four filters' accumulators for its 16 pixels, so
// that a 16-byte read of weights feeds 64 multiply-adds.  (A 16-byte shared-memory read delivers 512 bytes to a warp and holds the
// SM's one port for four cycles even when every lane reads the same address.  Packed multiply-adds, fma.rn.f32x2, run at the
// same rate -- 61 TFLOP/s measured against 62 -- and need every second pair of columns copied together: 1350 us.)
// 16 filters at 416x416, 256 images, pooled signs: 1489 us with 2x2 pixels and the patch from global memory, 1070 us now; the
// multiply-adds alone take 620 us at the measured rate.
//
// Every map of a multiple of 32 rows and columns is covered without idle threads.  Ways to finish, chosen by the caller:
//   * fp32 output at full resolution (bias, leaky/linear);
//   * the [maxpool] size 2 / stride 2 that follows the layer applied in registers, fp32 output at half resolution
//     (leaky is monotonic, so max(act(v)) == act(max(v)) value for value);
//   * only the SIGN of either, which is what a following xnor layer needs (max > 0 exactly when one of the four values is > 0):
//     as grid words (one 32-channel word per pixel on the padded grid of grid_words.cuh), as channel masks per pixel, or -- pooled
//     only -- as x-packed bit planes uint32 [image][filter][H/2][ceil(W/2/32)].
// Each output value is formed exactly as in float_conv_small_kernel: fmaf over (channel, ky, kx) from zero, then
// + bias, so all variants and that kernel agree bit for bit.
constexpr int FB_THREADS = 64;           // 2 warps; a warp covers 32 columns x 16 rows of the tile, a lane 4 x 4
constexpr int FB_TILE = 32;
constexpr int FB_PITCH = FB_TILE + 4;    // columns -1 .. 32 and two more, so that rows stay 16-byte aligned
constexpr int FB_ROWS = FB_TILE + 2;
constexpr int FB_FILTERS = 4;            // filters at a time
constexpr int FB_MAX_FILTERS = 32;       // most filters per CTA: one sign word
constexpr int FB_SMALL_TILES = 4;        // tiles per SM up to which a CTA takes 8 filters only

struct FloatBlockParams
{
	const float * in;        // [batch][3][H][W]
	const float * weights;   // [n][27]
	const float * biases;    // [n] or nullptr
	float * out;             // fp32 output (full or pooled) or nullptr
	uint32_t * planes;       // pooled sign planes or nullptr
	uint8_t * masks;         // sign masks [image][pixels][ceil(N/8)] (bit f%8 of byte f/8) or nullptr
	uint32_t * words;        // sign words on the grid, or nullptr
	int block_words, front, pitch;
	int H, W, N;
	int OH, OW;              // output map (half the input's when pooled)
	int plane_words;         // ceil(OW / 32)
	int xtiles;
	int fpc;                 // filters per CTA: a multiple of 8, at most FB_MAX_FILTERS (blockIdx.y picks them)
	int pooled;
	int leaky;
};

__global__ void __launch_bounds__(FB_THREADS, 8)
float_conv3_block_kernel(const __grid_constant__ FloatBlockParams p)
{
	__shared__ __align__(16) float s_in[3][FB_ROWS][FB_PITCH];
	__shared__ __align__(16) float s_w[27 * FB_MAX_FILTERS];       // [group of 4 filters][tap][filter]
	__shared__ float s_b[FB_MAX_FILTERS];
	pdl_trigger();
	const int tid = threadIdx.x;
	const int lane = tid & 31, warp = tid >> 5;
	const int f0 = blockIdx.y * p.fpc;
	const int nf = min(p.fpc, p.N - f0);
	const int groups = (nf + FB_FILTERS - 1) / FB_FILTERS;
	for (int i = tid; i < groups * 27 * FB_FILTERS; i += FB_THREADS)
	{
		const int g = i / (27 * FB_FILTERS);
		const int k = (i - g * 27 * FB_FILTERS) / FB_FILTERS;
		const int f = g * FB_FILTERS + i % FB_FILTERS;
		s_w[i] = (f < nf) ? __ldg(p.weights + (size_t)(f0 + f) * 27 + k) : 0.0f;
	}
	for (int f = tid; f < groups * FB_FILTERS; f += FB_THREADS) { s_b[f] = (p.biases != nullptr && f < nf) ? __ldg(p.biases + f0 + f) : 0.0f; }
	const int ty = blockIdx.x / p.xtiles;
	const int tx = blockIdx.x - ty * p.xtiles;
	const int y0 = ty * FB_TILE, x0 = tx * FB_TILE;
	const float * img = p.in + (size_t)blockIdx.z * 3 * p.H * p.W;
	// The tile with its border.  Rows: a warp takes every second one, 17 loads in flight; the columns left and right of the tile are
	// dealt over all threads behind them.  Tiles inside the image need no checks.
	{
		constexpr int ROUNDS = FB_ROWS / 2;
		const bool inside = (y0 > 0 && x0 > 0 && y0 + FB_TILE < p.H && x0 + FB_TILE < p.W);
		const float * at = img + (ptrdiff_t)(y0 - 1 + warp) * p.W + x0 + lane;
		const size_t step = 2 * (size_t)p.W;
		const bool in_x = (x0 + lane < p.W);
		#pragma unroll 1
		for (int c = 0; c < 3; ++c, at += (size_t)p.H * p.W)
		{
			float v[ROUNDS];
			const float * row = at;
			#pragma unroll
			for (int r = 0; r < ROUNDS; ++r, row += step)
			{
				const int iy = y0 - 1 + r * 2 + warp;
				v[r] = (inside || (iy >= 0 && iy < p.H && in_x)) ? __ldg(row) : 0.0f;
			}
			float * dst = &s_in[c][warp][lane + 1];
			#pragma unroll
			for (int r = 0; r < ROUNDS; ++r) { dst[r * 2 * FB_PITCH] = v[r]; }
		}
		for (int i = tid; i < 3 * FB_ROWS * 2; i += FB_THREADS)
		{
			const int right = i & 1, row = i >> 1;
			const int c = row / FB_ROWS, r = row - c * FB_ROWS;
			const int iy = y0 - 1 + r, ix = right ? x0 + FB_TILE : x0 - 1;
			s_in[c][r][right ? FB_TILE + 1 : 0] = (iy >= 0 && iy < p.H && ix >= 0 && ix < p.W) ? __ldg(img + ((size_t)c * p.H + iy) * p.W + ix) : 0.0f;
		}
	}
	__syncthreads();

	const int bx = (lane & 7) * 4;                               // first column and row of this thread's block inside the tile
	const int by = warp * 16 + (lane >> 3) * 4;
	const int gx = x0 + bx, gy = y0 + by;
	const bool live = (gx < p.W && gy < p.H);
	uint32_t bits[16];                                           // sign bits of the filters so far, newest lowest, per pixel (pooled: the first four)
	#pragma unroll
	for (int i = 0; i < 16; ++i) { bits[i] = 0; }
	#pragma unroll 1
	for (int g = 0; g < groups; ++g)
	{
		float acc[FB_FILTERS][4][4];                             // [filter][row][column]
		#pragma unroll
		for (int f = 0; f < FB_FILTERS; ++f)
		{
			#pragma unroll
			for (int i = 0; i < 16; ++i) { acc[f][i / 4][i % 4] = 0.0f; }
		}
		const float4 * wg = reinterpret_cast<const float4 *>(s_w + g * 27 * FB_FILTERS);
		#pragma unroll
		for (int c = 0; c < 3; ++c)
		{
			float v[6][6];
			#pragma unroll
			for (int r = 0; r < 6; ++r)
			{
				const float4 a = *reinterpret_cast<const float4 *>(&s_in[c][by + r][bx]);
				const float2 b = *reinterpret_cast<const float2 *>(&s_in[c][by + r][bx + 4]);
				v[r][0] = a.x; v[r][1] = a.y; v[r][2] = a.z; v[r][3] = a.w; v[r][4] = b.x; v[r][5] = b.y;
			}
			#pragma unroll
			for (int k = 0; k < 9; ++k)
			{
				const int ky = k / 3, kx = k % 3;
				const float4 w4 = wg[c * 9 + k];
				const float w[4] = {w4.x, w4.y, w4.z, w4.w};
				#pragma unroll
				for (int f = 0; f < FB_FILTERS; ++f)
				{
					#pragma unroll
					for (int i = 0; i < 16; ++i) { acc[f][i / 4][i % 4] = fmaf(v[ky + i / 4][kx + i % 4], w[f], acc[f][i / 4][i % 4]); }
				}
			}
		}
		#pragma unroll
		for (int f = 0; f < FB_FILTERS; ++f)
		{
			const int fl = g * FB_FILTERS + f;
			const float b = s_b[fl];
			const float minus_b = __fsub_rn(0.0f, b);            // +0 for a bias of zero: below, +0 - +0 must not come out as -0
			if (p.pooled)
			{
				// adding the bias keeps the order of values, so the largest sum is the largest value plus the bias
				float top[4];
				#pragma unroll
				for (int i = 0; i < 4; ++i)
				{
					const int y = (i >> 1) * 2, x = (i & 1) * 2;
					top[i] = fmaxf(fmaxf(acc[f][y][x], acc[f][y][x + 1]), fmaxf(acc[f][y + 1][x], acc[f][y + 1][x + 1]));
				}
				if (p.out == nullptr && p.planes == nullptr)
				{
					// value > 0 is the sign bit of (0 - bias) - top, whatever the signs of zeros
					#pragma unroll
					for (int i = 0; i < 4; ++i) { bits[i] = __funnelshift_l(__float_as_uint(__fsub_rn(minus_b, top[i])), bits[i], 1); }
					continue;
				}
				#pragma unroll
				for (int y = 0; y < 2; ++y)
				{
					const int oy = (gy >> 1) + y;
					float m[2] = {top[2 * y] + b, top[2 * y + 1] + b};
					if (p.out != nullptr)
					{
						if (!live || oy >= p.OH || fl >= nf) { continue; }
						float * dst = p.out + (((size_t)blockIdx.z * p.N + f0 + fl) * p.OH + oy) * p.OW + (gx >> 1);
						#pragma unroll
						for (int i = 0; i < 2; ++i)
						{
							if (p.leaky) { m[i] = (m[i] > 0.0f) ? m[i] : m[i] * 0.1f; }
							if ((gx >> 1) + i < p.OW) { dst[i] = m[i]; }
						}
					}
					else
					{
						// two bits of the lane's 16-column half word, gathered over the eight lanes of its rows
						uint32_t half = (m[0] > 0.0f ? 1u : 0u) | ((m[1] > 0.0f && (gx >> 1) + 1 < p.OW) ? 2u : 0u);
						half = live ? half << (2 * (lane & 7)) : 0u;
						half |= __shfl_xor_sync(0xffffffffu, half, 1);
						half |= __shfl_xor_sync(0xffffffffu, half, 2);
						half |= __shfl_xor_sync(0xffffffffu, half, 4);
						if ((lane & 7) == 0 && oy < p.OH && fl < nf)
						{
							uint16_t * row = reinterpret_cast<uint16_t *>(p.planes + (((size_t)blockIdx.z * p.N + f0 + fl) * p.OH + oy) * p.plane_words);
							row[tx] = (uint16_t)half;
							if (tx == p.xtiles - 1 && tx % 2 == 0) { row[tx + 1] = 0; }
						}
					}
				}
				continue;
			}
			if (p.out != nullptr)
			{
				if (!live || fl >= nf) { continue; }
				float r[4][4];
				#pragma unroll
				for (int i = 0; i < 16; ++i) { r[i / 4][i % 4] = acc[f][i / 4][i % 4] + b; }
				float * dst = p.out + (((size_t)blockIdx.z * p.N + f0 + fl) * p.H + gy) * p.W + gx;
				#pragma unroll
				for (int y = 0; y < 4; ++y)
				{
					#pragma unroll
					for (int x = 0; x < 4; ++x) { if (p.leaky) { r[y][x] = (r[y][x] > 0.0f) ? r[y][x] : r[y][x] * 0.1f; } }
					if (gy + y >= p.H) { break; }
					if (p.W % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0)
					{
						*reinterpret_cast<float4 *>(dst + (size_t)y * p.W) = make_float4(r[y][0], r[y][1], r[y][2], r[y][3]);
						continue;
					}
					#pragma unroll
					for (int x = 0; x < 4; ++x) { if (gx + x < p.W) { dst[(size_t)y * p.W + x] = r[y][x]; } }
				}
				continue;
			}
			#pragma unroll
			for (int i = 0; i < 16; ++i) { bits[i] = __funnelshift_l(__float_as_uint(__fsub_rn(minus_b, acc[f][i / 4][i % 4])), bits[i], 1); }
		}
	}
	if (p.out != nullptr || p.planes != nullptr || !live) { return; }
	// this CTA's bytes of every pixel's mask or word; filters that do not exist have weights 0 and bias 0: not > 0
	const int bytes = (p.words != nullptr) ? 4 : (p.N + 7) / 8;
	#pragma unroll
	for (int i = 0; i < 16; ++i)
	{
		if (p.pooled && i >= 4) { break; }
		const int oy = p.pooled ? (gy >> 1) + (i >> 1) : gy + (i >> 2);
		const int ox = p.pooled ? (gx >> 1) + (i & 1) : gx + (i & 3);
		if (oy >= p.OH || ox >= p.OW) { continue; }
		const uint32_t word = __brev(bits[i]) >> (32 - groups * FB_FILTERS);         // filter f at bit f
		uint8_t * dst = (p.words != nullptr)
				? reinterpret_cast<uint8_t *>(p.words + (size_t)(f0 >> 5) * p.block_words + p.front + ((size_t)blockIdx.z * (p.OH + 1) + oy) * p.pitch + ox) + ((f0 & 31) >> 3)
				: p.masks + (((size_t)blockIdx.z * p.OH + oy) * p.OW + ox) * bytes + (f0 >> 3);
		// a CTA that has all of a word's filters writes the whole word
		if (p.words != nullptr && (p.fpc == FB_MAX_FILTERS || p.fpc >= p.N)) { *reinterpret_cast<uint32_t *>(dst) = word; }
		else { for (int q = 0; q * 8 < nf; ++q) { dst[q] = (uint8_t)(word >> (8 * q)); } }
	}
}

}  // namespace xnor

using namespace xnor;

extern "C" int xnor_b200_float_conv_small(const xnor_b200_conv_desc * desc, const float * input, const float * weights,
		const float * biases, float * output, void * stream)
{
	if (desc == nullptr || input == nullptr || weights == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	const int taps = desc->c * desc->size * desc->size;
	if (taps > FC_MAX_TAPS || desc->n > 256) { return XNOR_B200_ERR_TOO_LARGE; }
	FloatConvParams p;
	p.in = input; p.weights = weights; p.biases = biases; p.out = output;
	p.batch = desc->batch; p.C = desc->c; p.H = desc->h; p.W = desc->w; p.N = desc->n;
	p.OH = conv_out_dim(desc->h, desc->size, desc->stride, desc->pad);
	p.OW = conv_out_dim(desc->w, desc->size, desc->stride, desc->pad);
	p.ks = desc->size; p.stride = desc->stride; p.pad = desc->pad;
	p.leaky = (desc->activation == XNOR_B200_LEAKY) ? 1 : 0;
	const size_t total = (size_t)p.batch * p.OH * p.OW;
	const size_t smem = ((size_t)p.N * taps + p.N) * sizeof(float);
	const int grid = (int)min((total + FC_THREADS - 1) / FC_THREADS, (size_t)sm_count() * 8);
	if (desc->c == 3 && desc->size == 3)
	{
		rc = ensure_dynamic_smem((const void *)float_conv_small_kernel<3, 3>, smem);
		if (rc != XNOR_B200_OK) { return rc; }
		float_conv_small_kernel<3, 3><<<grid, FC_THREADS, smem, (cudaStream_t)stream>>>(p);
	}
	else
	{
		rc = ensure_dynamic_smem((const void *)float_conv_small_kernel<0, 0>, smem);
		if (rc != XNOR_B200_OK) { return rc; }
		float_conv_small_kernel<0, 0><<<grid, FC_THREADS, smem, (cudaStream_t)stream>>>(p);
	}
	return check_launch();
}

static int launch_conv3(const xnor_b200_conv_desc * desc, int pool, const float * input, const float * weights, const float * biases,
		FloatBlockParams & p, void * stream)
{
	if (desc == nullptr || input == nullptr || weights == nullptr) { return XNOR_B200_ERR_NULL; }
	if ((p.out != nullptr) + (p.planes != nullptr) + (p.masks != nullptr) + (p.words != nullptr) != 1) { return XNOR_B200_ERR_NULL; }
	int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	if (desc->c != 3 || desc->size != 3 || desc->stride != 1 || desc->pad != 1) { return XNOR_B200_ERR_INVALID; }
	if (pool != 0 && pool != 2) { return XNOR_B200_ERR_INVALID; }
	if (pool == 2 && (desc->h % 2 != 0 || desc->w % 2 != 0)) { return XNOR_B200_ERR_INVALID; }
	if (p.planes != nullptr && pool != 2) { return XNOR_B200_ERR_INVALID; }
	p.in = input; p.weights = weights; p.biases = biases;
	p.H = desc->h; p.W = desc->w; p.N = desc->n;
	p.pooled = (pool == 2) ? 1 : 0;
	p.OH = p.pooled ? desc->h / 2 : desc->h;
	p.OW = p.pooled ? desc->w / 2 : desc->w;
	p.plane_words = (p.OW + 31) / 32;
	p.xtiles = (desc->w + FB_TILE - 1) / FB_TILE;
	p.leaky = (desc->activation == XNOR_B200_LEAKY) ? 1 : 0;
	if (p.words != nullptr)
	{
		if (p.pitch == 0) { p.pitch = p.OW + 1; }
		if (p.pitch <= p.OW) { return XNOR_B200_ERR_INVALID; }
		if (xnor_b200_grid_block_words(desc->batch, p.OH, p.pitch) == 0) { return XNOR_B200_ERR_TOO_LARGE; }
		p.front = grid_front(p.pitch);
		p.block_words = grid_block_words(desc->batch, p.OH, p.pitch);
	}
	if (p.words != nullptr)
	{
		// signs only: on the tensor cores, where the shape allows
		rc = launch_float_conv3_signs(*desc, pool, input, weights, biases, p.words, p.pitch, (cudaStream_t)stream);
		if (rc != XNOR_B200_ERR_TOO_LARGE) { return rc; }
	}
	const long long tiles = (long long)p.xtiles * ((desc->h + FB_TILE - 1) / FB_TILE);
	// All of a pixel's filters in one CTA read the tile once and write whole words; with few tiles, eight filters each, so that
	// the GPU fills (one image of 416x416, 16 filters: 169 tiles).
	p.fpc = (tiles * desc->batch <= (long long)FB_SMALL_TILES * sm_count()) ? 8 : FB_MAX_FILTERS;
	const int groups = (desc->n + p.fpc - 1) / p.fpc;
	if (tiles > 0x7fffffffLL || groups > 65535 || desc->batch > 65535) { return XNOR_B200_ERR_TOO_LARGE; }
	float_conv3_block_kernel<<<dim3((unsigned)tiles, (unsigned)groups, (unsigned)desc->batch), FB_THREADS, 0, (cudaStream_t)stream>>>(p);
	return check_launch();
}

extern "C" int xnor_b200_float_conv3_io(const xnor_b200_conv_desc * desc, int pool, const float * input, const float * weights,
		const float * biases, float * output, uint32_t * output_sign_planes, uint8_t * output_sign_masks, void * stream)
{
	FloatBlockParams p = {};
	p.out = output; p.planes = output_sign_planes; p.masks = output_sign_masks;
	return launch_conv3(desc, pool, input, weights, biases, p, stream);
}

extern "C" int xnor_b200_float_conv3_words(const xnor_b200_conv_desc * desc, int pool, const float * input, const float * weights,
		const float * biases, uint32_t * words, int pitch, void * stream)
{
	FloatBlockParams p = {};
	p.words = words;
	p.pitch = pitch;
	return launch_conv3(desc, pool, input, weights, biases, p, stream);
}
