// Signs of the first convolution (3 channels, 3x3, stride 1, pad 1, up to 32 filters) on the tcgen05 tensor cores, exactly.
//
// What the layer behind it wants is one bit per value: fl(sum) + bias > 0, the sum formed by fmaf over (channel, ky, kx) from zero.
// 27 multiply-adds a value on the FMA pipe are 620 us for 16 filters at 416x416 and 256 images (1070 us with everything around
// them).  Here the values are first formed approximately, as fp16 products with fp32 accumulation, together with a bound on how far
// off they can be; wherever the value is farther from zero than that, the sign is known, and the rest -- about a quarter of a percent --
// are formed again in fp32, in the order above.  Every bit is therefore the exact one.
//
//   |approximate - exact| <= ulp(xmax) / 2 + xmax * (d + 5.3e-5) + 1.1e-7
//
// for a filter scaled to sum|w| = 1 and xmax the largest input of the unit: ulp(xmax) / 2 = 2^-12 of the power of two above xmax, what
// rounding an input to fp16 takes at most; d the sum of what rounding took of the weights, the largest of the filters (about 2e-4, 2^-11
// at most); 2^-25 each for subnormal operands; and 5.3e-5 for the rest: 2e-6 for the scaling and the fp32 sum there, and for the sum
// here six instructions of 17 terms that lose up to 2^-23 of the largest each, twice over where the bias is as large as the products
// (2.4e-5).  That loss per term is how fp32 accumulation is taken to be, not something the hardware states.  (Compared in fp16, hence a
// factor of 1.002 and 1.2e-7 more.)  For 8-bit images half of the bound that takes 2^-10 for the two roundings of every product, and half
// as many values to form again.
// Inputs or filters that fp16 cannot hold make the bound infinite or the value NaN, and every value is formed again.
//
// One MMA row is a 2x2 block of pixels, its columns the block's four values of every filter, K the patch of pixels around it: with
// N = 4 * filters and 12 halves of 16 bytes that is 6 instructions per 512 pixels.  The operand is never gathered: an input pixel
// pair (2q, 2q + 1) is 16 bytes [c0 c1 c2 1 | c0 c1 c2 1] in a plane [block row][pair], one plane for even and one for odd pixel
// rows, and a row or a neighbouring pair is another start address (as in xnor_conv.cu; position = (image * (BH + 1) + by) * (BW + 1) +
// bx, the pair behind a row is zero).  The ones carry the bias, as three fp16 parts in the filter operand.
//
// Roles (one CTA per SM): warps 0..11 (unpooled 0..15) epilogue, then converters (global fp32 -> planes), 23 issuer.
// Measured at 416x416, 16 filters, pooled, 64 images: 82 us, 90 with the bound of two roundings a product; 350 with every load followed by its use, 104 with unaligned pairs
// (2q - 1, 2q), a shuffle for each, and bias and bound per filter in the epilogue.  Clock traces: converters and epilogue, bound by
// issue slots and by the latency of the doubtful values, take turns as the bound; HBM would be 22 us.
#include "grid_words.cuh"
#include "tc_common.cuh"

#include <cuda_fp16.h>

namespace xnor
{

constexpr int F3_MMA_WARP = 23;
constexpr int F3_THREADS = (F3_MMA_WARP + 1) * 32;
constexpr int F3_BATCH = 2;                    // window slots a converter thread has in flight
constexpr int F3_STAGES = 3;
constexpr int F3_MAX_PT = 8;                  // tiles of 128 blocks per unit
constexpr int F3_MAX_UNITS_AHEAD = 16;        // entries of the ring of unit maxima: stages + accumulators + 1 are under way
constexpr int F3_QUEUE = 64;                  // values of a warp that wait to be formed exactly
constexpr int F3_HALVES = 12;                 // 16-byte pieces of K: four patch rows x three pairs
constexpr int F3_SMEM_MAX = 190 * 1024;      // dynamic; with the kernel's static part (37 KB for 32 filters) what a block may have

struct F3Params
{
	const float * in;        // [batch][3][H][W]
	const float * weights;   // [n][27]
	const float * biases;    // [n] or nullptr
	uint32_t * words;        // position 0 of the output grid
	int H, W, N;
	int BH, BW, pitch;       // 2x2 blocks; pitch = BW + 1
	int OH, OW, out_pitch;
	FastDiv d_img, d_pitch;  // positions per image, per row
	int total_pos, pt, units;
	int plane_slots;         // window positions of a unit, from one in front of it on: pt * 128 + pitch + 2
	int stage_bytes;
	int vec;                 // 1: rows of whole, aligned pairs
	int * status;
	uint32_t spin_limit;
};

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi)
{
	uint32_t r;
	asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
	return r;
}

// Largest magnitude of the three, NaN if one is
__device__ __forceinline__ float max_abs3(float a, float b, float c)
{
	float r;
	asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}

__device__ __forceinline__ uint32_t larger_half2(uint32_t a, uint32_t b)
{
	uint32_t r;
	asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
	return r;
}

// 0xffff in each half where a > b (not where either is NaN)
__device__ __forceinline__ uint32_t above_half2(uint32_t a, uint32_t b)
{
	return __hgt2_mask(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
}

// Bits 0..3, 8..11 and 16..19, 24..27 -> 0..15
__device__ __forceinline__ uint32_t spread(uint32_t v)
{
	return (v & 0x0f0fu) | ((v >> 12) & 0xf0f0u);
}

__device__ __forceinline__ float half_of(float v)
{
	float r;
	asm("{\n\t.reg .b16 h;\n\tcvt.rn.f16.f32 h, %1;\n\tcvt.f32.f16 %0, h;\n\t}" : "=f"(r) : "f"(v));
	return r;
}

__device__ __forceinline__ uint64_t f3_desc(uint32_t start, uint32_t lbo)
{
	return (uint64_t)(start | (lbo << 16)) | ((uint64_t)(8u | (1u << 14)) << 32);
}

// The exact value, formed as float_conv_small_kernel does.
__device__ __forceinline__ float exact_value(const F3Params & p, int img, int oy, int ox, const float * w, float bias)
{
	const float * base = p.in + (size_t)img * 3 * p.H * p.W;
	float v[27];                                                  // all loads at once: one memory latency
	#pragma unroll
	for (int k = 0; k < 27; ++k)
	{
		const int iy = oy - 1 + (k % 9) / 3, ix = ox - 1 + k % 3;
		v[k] = (iy >= 0 && iy < p.H && ix >= 0 && ix < p.W) ? __ldg(base + ((size_t)(k / 9) * p.H + iy) * p.W + ix) : 0.0f;
	}
	float acc = 0.0f;
	#pragma unroll
	for (int k = 0; k < 27; ++k) { acc = fmaf(v[k], w[k], acc); }
	return acc + bias;
}

// NF filters (16 or 32), POOL: the 2x2 max-pool behind the layer is applied.
template <int NF, bool POOL>
__global__ void __launch_bounds__(F3_THREADS, 1)
float_conv3_signs_kernel(const __grid_constant__ F3Params p)
{
	// the 23 warps beside the issuer: a pooled block leaves one word of 16 bits, an unpooled one four words, for the same input
	constexpr int EPI_WARPS = POOL ? 12 : 16;
	constexpr int CONV_WARPS = F3_MMA_WARP - EPI_WARPS;
	constexpr int NN = 4 * NF;                                  // MMA columns: POOL: filter * 4 + pixel of the block, else pixel * NF + filter
	constexpr int ACC = 512 / NN;
	extern __shared__ __align__(128) uint8_t f3_smem[];         // [stage][odd rows | even rows][slot] of 16 bytes
	__shared__ __align__(128) uint4 s_b[F3_HALVES * NN];                // filter operand [16-byte half of K][column]
	__shared__ float s_w[NF * 27];
	__shared__ float s_bias[NF];                                // as given
	__shared__ float s_dev[NF], s_scale[NF], s_part[NF][3];
	__shared__ float s_xmax[F3_MAX_UNITS_AHEAD][CONV_WARPS];
	__shared__ uint2 s_queue[EPI_WARPS][F3_QUEUE];
	__shared__ uint64_t st_full[F3_STAGES], st_empty[F3_STAGES], acc_full[ACC], acc_empty[ACC], drain_bar, ready_bar;
	static_assert(sizeof(s_b) + sizeof(s_w) + sizeof(s_bias) + sizeof(s_dev) + sizeof(s_scale) + sizeof(s_part) + sizeof(s_xmax) + sizeof(s_queue) + sizeof(st_full) + sizeof(st_empty) + sizeof(acc_full)
			+ sizeof(acc_empty) + 256 + F3_SMEM_MAX <= 227 * 1024, "static and dynamic shared memory of a block");
	__shared__ uint32_t tmem_base_slot;
	__shared__ int s_failed_storage;
	volatile int * s_failed = &s_failed_storage;

	const int tid = threadIdx.x;
	const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
	const int lane = tid & 31;
	const uint32_t limit = p.spin_limit;
	const uint32_t a_base = smem_u32(f3_smem);
	const int my_units = (p.units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

	if (tid == 0)
	{
		for (int s = 0; s < F3_STAGES; ++s)
		{
			mbar_init(&st_full[s], CONV_WARPS);
			mbar_init(&st_empty[s], 1);
		}
		for (int a = 0; a < ACC; ++a)
		{
			mbar_init(&acc_full[a], 1);
			mbar_init(&acc_empty[a], 4);
		}
		mbar_init(&drain_bar, 1);
		mbar_init(&ready_bar, EPI_WARPS);
		s_failed_storage = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == F3_MMA_WARP)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
	pdl_trigger();                                              // this CTA has its tensor memory

	if (warp < EPI_WARPS)
	{
		// ---- epilogue warps, first: the filter operand, while the converters begin.  A warp per filter for its scale and what rounding
		// takes, then an operand entry a thread (a thread per filter, in front of all roles, took a third of the layer at batch 1).
		auto epilogue_warps = [&]() { asm volatile("bar.sync 1, %0;" :: "n"(EPI_WARPS * 32) : "memory"); };
		for (int i = tid; i < NF * 27; i += EPI_WARPS * 32) { s_w[i] = (i < p.N * 27) ? __ldg(p.weights + i) : 0.0f; }
		epilogue_warps();
		for (int f = warp; f < NF; f += EPI_WARPS)
		{
			const float w = (lane < 27) ? s_w[f * 27 + lane] : 0.0f;
			float sum = fabsf(w);
			#pragma unroll
			for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); }
			const float bias = (p.biases != nullptr && f < p.N) ? __ldg(p.biases + f) : 0.0f;
			// a filter of zeros stays as it is; one whose scale fp32 cannot hold, or whose bias fp16 cannot, gets a bias of NaN
			const float scale = (sum > 0.0f) ? 1.0f / sum : 1.0f;
			const bool fits = (sum < 1e30f) && (scale < 1e30f) && (fabsf(bias * scale) < 60000.0f);
			float lost = fabsf(w * scale - half_of(w * scale));
			#pragma unroll
			for (int o = 16; o > 0; o >>= 1) { lost += __shfl_xor_sync(0xffffffffu, lost, o); }
			if (lane == 0)
			{
				s_bias[f] = bias;
				s_dev[f] = fits ? lost : 0.0f;                          // (a bias of NaN leaves no value sure)
				s_scale[f] = fits ? scale : 0.0f;
				const float first = fits ? bias * scale : NAN, second = first - half_of(first);
				s_part[f][0] = first;
				s_part[f][1] = second;
				s_part[f][2] = second - half_of(second);
			}
		}
		epilogue_warps();
		for (int i = tid; i < NF * F3_HALVES * 4; i += EPI_WARPS * 32)
		{
			const int f = i % NF, s = i / NF % 4, h = i / (NF * 4);
			// half h: patch rows 0, 2 (odd pixel rows), 1, 3 (even ones), three pairs each
			const int row = (h / 6) + 2 * ((h / 3) & 1), pair = h % 3;
			const int ky = row - (s >> 1);
			const float scale = s_scale[f];
			float v[8];
			#pragma unroll
			for (int q = 0; q < 8; ++q)
			{
				const int kx = 2 * (pair - 1) + (q >> 2) - (s & 1) + 1, c = q & 3;
				v[q] = (scale > 0.0f && c < 3 && ky >= 0 && ky < 3 && kx >= 0 && kx < 3) ? s_w[f * 27 + (c * 3 + ky) * 3 + kx] * scale : 0.0f;
			}
			if (h < 3) { v[3] = s_part[f][h]; }
			s_b[h * NN + (POOL ? f * 4 + s : s * NF + f)] = make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
		}
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		__syncwarp();
		if (lane == 0) { mbar_arrive(&ready_bar); }

		// ---- epilogue: warp w takes the tiles w / 4, w / 4 + 4, ... of this CTA, lane quarter w % 4 -----------------------------
		const int quarter = warp & 3;
		const int my_tiles = my_units * p.pt;
		int tile = warp >> 2;
		int nu = 0, t = tile;                                    // unit of this CTA, tile of the unit
		while (t >= p.pt) { t -= p.pt; ++nu; }
		int a = tile % ACC;
		uint32_t phase = (uint32_t)((tile / ACC) & 1);
		float dev = (lane < NF) ? s_dev[lane] : 0.0f;            // what rounding took of the weights
		#pragma unroll
		for (int o = 16; o > 0; o >>= 1) { dev = fmaxf(dev, __shfl_xor_sync(0xffffffffu, dev, o)); }
		int have_unit = -1;
		uint32_t limit2 = 0;                                     // the bound of the unit, in both halves
		int q_head = 0, q_count = 0;                             // this warp's ring of values to be formed exactly
		// output word of a position and pixel of its block
		auto word_at = [&](int img, int y, int x) { return p.words + ((size_t)img * (p.OH + 1) + y) * p.out_pitch + x; };
		auto resolve = [&](int n)
		{
			// the n oldest values; POOL: four lanes form one, a pixel of the block each
			constexpr int LANES = POOL ? 4 : 1;
			__syncwarp();
			if (lane < n * LANES)
			{
				const uint2 item = s_queue[warp][(q_head + lane / LANES) % F3_QUEUE];
				const int f = (int)(item.y & 255u), s = POOL ? (lane & 3) : (int)(item.y >> 8);
				const int pos = (int)item.x;
				const int img = fdiv(pos, p.d_img);
				const int r = pos - img * (int)p.d_img.d;
				const int by = fdiv(r, p.d_pitch), bx = r - by * p.pitch;
				const int oy = 2 * by + (s >> 1), ox = 2 * bx + (s & 1);
				if (exact_value(p, img, oy, ox, s_w + f * 27, s_bias[f]) > 0.0f)
				{
					atomicOr(POOL ? word_at(img, by, bx) : word_at(img, oy, ox), 1u << f);
				}
			}
			q_head = (q_head + n) % F3_QUEUE;
			q_count -= n;
		};
		auto enqueue = [&](uint32_t unsure, int pos, int s)
		{
			// one value per lane and round; the words they belong to have been stored
			constexpr int BATCH = POOL ? 8 : 32;
			__syncwarp();
			while (true)
			{
				const unsigned who = __ballot_sync(0xffffffffu, unsure != 0);
				if (who == 0) { break; }
				if (unsure != 0)
				{
					const int f = __ffs(unsure) - 1;
					unsure &= unsure - 1;
					s_queue[warp][(q_head + q_count + __popc(who & ((1u << lane) - 1u))) % F3_QUEUE] = make_uint2((uint32_t)pos, (uint32_t)(f | (s << 8)));
				}
				q_count += __popc(who);
				while (q_count >= BATCH) { resolve(BATCH); }
			}
		};
		while (tile < my_tiles)
		{
			if (!__all_sync(0xffffffffu, mbar_wait<32>(&acc_full[a], phase, s_failed, limit))) { break; }
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			if (nu != have_unit)
			{
				have_unit = nu;
				float xmax = (lane < CONV_WARPS) ? s_xmax[nu % F3_MAX_UNITS_AHEAD][lane] : 0.0f;
				#pragma unroll
				for (int o = 8; o > 0; o >>= 1) { xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, o)); }
				xmax = __shfl_sync(0xffffffffu, xmax, 0);
				// the power of two that xmax does not pass
				const float above = __uint_as_float((__float_as_uint(xmax) + 0x7fffffu) & 0xff800000u);
				// values are compared as fp16, so a little more for their rounding; infinity stays infinity
				const float bound = (above * 2.4439e-4f + xmax * (dev * 1.001f + 5.3e-5f) + 1.1e-7f) * 1.002f + 1.2e-7f;
				limit2 = pack_half2(bound, bound);
			}
			const int pos = (((int)blockIdx.x + nu * (int)gridDim.x) * p.pt + t) * TC_PIX + quarter * 32 + lane;
			const int img = fdiv(pos, p.d_img);
			const int r = pos - img * (int)p.d_img.d;
			const int by = fdiv(r, p.d_pitch), bx = r - by * p.pitch;
			const bool ok = (pos < p.total_pos && by < p.BH && bx < p.BW);
			const uint32_t tacc = tmem_base + (uint32_t)(a * NN) + ((uint32_t)(quarter * 32) << 16);
			if (POOL)
			{
				uint32_t pos_bits[NN / 64], sure_bits[NN / 64];        // of 16 filters: the low half 0..3 | 8..11, the high half 4..7 | 12..15
				#pragma unroll
				for (int g = 0; g < NN / 64; ++g) { pos_bits[g] = 0; sure_bits[g] = 0; }
				#pragma unroll
				for (int h = 0; h < NN / 32; ++h)
				{
					uint32_t d[32];
					tmem_load<32>(tacc + (uint32_t)(h * 32), d);
					tmem_wait<32>(d);
					if (h == NN / 32 - 1)
					{
						asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
						__syncwarp();
						if (lane == 0) { mbar_arrive(&acc_empty[a]); }
					}
					// filters i and i + 4 of these eight side by side
					#pragma unroll
					for (int i = 0; i < 4; ++i)
					{
						uint32_t v = pack_half2(__uint_as_float(d[4 * i]), __uint_as_float(d[4 * i + 16]));
						#pragma unroll
						for (int s = 1; s < 4; ++s) { v = larger_half2(v, pack_half2(__uint_as_float(d[4 * i + s]), __uint_as_float(d[4 * i + 16 + s]))); }
						const uint32_t bit = (1u << i) | (1u << (i + 16));
						pos_bits[h / 2] |= (above_half2(v, limit2) & bit) << (8 * (h & 1));
						sure_bits[h / 2] |= (above_half2(v & 0x7fff7fffu, limit2) & bit) << (8 * (h & 1));
					}
				}
				uint32_t word = 0, unsure = 0;
				#pragma unroll
				for (int g = 0; g < NN / 64; ++g)
				{
					word |= spread(pos_bits[g]) << (16 * g);
					unsure |= spread(sure_bits[g]) << (16 * g);
				}
				unsure = ~unsure & ((NF == 32) ? 0xffffffffu : 0xffffu);
				// filters past the last have weights and bias zero: exact value 0, no sign
				if (ok) { *word_at(img, by, bx) = word; }
				if (!ok) { unsure = 0; }
				if (p.N < 32) { unsure &= (1u << p.N) - 1u; }
				if (__any_sync(0xffffffffu, unsure != 0)) { enqueue(unsure, pos, 0); }
			}
			else
			{
				#pragma unroll 1
				for (int s = 0; s < 4; ++s)
				{
					uint32_t d[NF];
					tmem_load<NF>(tacc + (uint32_t)(s * NF), d);
					tmem_wait<NF>(d);
					if (s == 3)
					{
						asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
						__syncwarp();
						if (lane == 0) { mbar_arrive(&acc_empty[a]); }
					}
					// filters f and f + NF / 2 side by side
					uint32_t word = 0, unsure = 0;
					#pragma unroll
					for (int f = 0; f < NF / 2; ++f)
					{
						const uint32_t v = pack_half2(__uint_as_float(d[f]), __uint_as_float(d[f + NF / 2]));
						const uint32_t bit = (1u << f) | (1u << (f + 16));
						word |= above_half2(v, limit2) & bit;
						unsure |= above_half2(v & 0x7fff7fffu, limit2) & bit;
					}
					if (NF == 16)
					{
						word = (word & 0xffu) | ((word >> 8) & 0xff00u);
						unsure = (unsure & 0xffu) | ((unsure >> 8) & 0xff00u);
					}
					unsure = ~unsure & ((NF == 32) ? 0xffffffffu : 0xffffu);
					const int oy = 2 * by + (s >> 1), ox = 2 * bx + (s & 1);
					const bool in = ok && oy < p.OH && ox < p.OW;
					if (in) { *word_at(img, oy, ox) = word; }
					if (!in) { unsure = 0; }
					if (p.N < 32) { unsure &= (1u << p.N) - 1u; }
					if (__any_sync(0xffffffffu, unsure != 0)) { enqueue(unsure, pos, s); }
				}
			}
			tile += EPI_WARPS / 4;
			a += EPI_WARPS / 4;
			while (a >= ACC) { a -= ACC; phase ^= 1u; }
			t += EPI_WARPS / 4;
			while (t >= p.pt) { t -= p.pt; ++nu; }
		}
		while (q_count > 0) { resolve(min(q_count, POOL ? 8 : 32)); }
	}
	else if (warp < F3_MMA_WARP)
	{
		// ---- converters: a slot is the pair of pixels (2q, 2q + 1) of an odd and of an even row ------------------------------
		const int cw = warp - EPI_WARPS;
		const size_t plane = (size_t)p.H * p.W;
		const int groups = (p.plane_slots + 31) >> 5;
		const int H = p.H, W = p.W, plane_slots = p.plane_slots, total_pos = p.total_pos, pitch = p.pitch;
		const FastDiv d_img = p.d_img, d_pitch = p.d_pitch;
		const bool vec = (p.vec != 0);
		int es = 0;
		uint32_t es_phase = 1;
		bool ok = true;
		for (int nu = 0; nu < my_units && ok; ++nu)
		{
			const int pos0 = ((int)blockIdx.x + nu * (int)gridDim.x) * p.pt * TC_PIX - 1;
			const uint32_t odd = a_base + (uint32_t)(es * p.stage_bytes);
			const uint32_t even = odd + (uint32_t)(plane_slots * 16);
			float top = 0.0f;                                     // largest magnitude
			if (nu >= F3_STAGES)
			{
				ok = __all_sync(0xffffffffu, mbar_wait<32>(&st_empty[es], es_phase, s_failed, limit));
				if (!ok) { break; }
			}
			// F3_BATCH slots at a time, all of their loads first: the kernel lives on bytes in flight
			for (int g0 = cw; g0 < groups; g0 += CONV_WARPS * F3_BATCH)
			{
				float2 v[F3_BATCH][6];                            // [slot][odd, even row x channel]
				#pragma unroll
				for (int i = 0; i < F3_BATCH; ++i)
				{
					const int s = (g0 + i * CONV_WARPS) * 32 + lane;
					const int pos = pos0 + s;
					const int img = fdiv(max(pos, 0), d_img);
					const int r = pos - img * (int)d_img.d;
					const int by = fdiv(max(r, 0), d_pitch), q = r - by * pitch;
					const int ye = 2 * by, x = 2 * q;
					const bool in = (s < plane_slots && pos >= 0 && pos < total_pos && x < W);
					const bool odd_ok = in && ye > 0 && ye - 1 < H, even_ok = in && ye < H;
					const float * at = p.in + (size_t)img * 3 * plane + (ptrdiff_t)ye * W + x;
					#pragma unroll
					for (int c = 0; c < 3; ++c, at += plane)
					{
						v[i][c] = make_float2(0.0f, 0.0f);
						v[i][3 + c] = make_float2(0.0f, 0.0f);
						if (vec)
						{
							if (odd_ok) { v[i][c] = __ldg(reinterpret_cast<const float2 *>(at - W)); }
							if (even_ok) { v[i][3 + c] = __ldg(reinterpret_cast<const float2 *>(at)); }
						}
						else
						{
							if (odd_ok) { v[i][c].x = __ldg(at - W); }
							if (odd_ok && x + 1 < W) { v[i][c].y = __ldg(at - W + 1); }
							if (even_ok) { v[i][3 + c].x = __ldg(at); }
							if (even_ok && x + 1 < W) { v[i][3 + c].y = __ldg(at + 1); }
						}
					}
				}
				#pragma unroll
				for (int i = 0; i < F3_BATCH; ++i)
				{
					const int s = (g0 + i * CONV_WARPS) * 32 + lane;
					#pragma unroll
					for (int k = 0; k < 2; ++k)
					{
						const float2 c0 = v[i][3 * k], c1 = v[i][3 * k + 1], c2 = v[i][3 * k + 2];
						const uint32_t left = pack_half2(c0.x, c1.x), right = pack_half2(c0.y, c1.y), third = pack_half2(c2.x, c2.y);
						top = max_abs3(top, c0.x, c0.y);
						top = max_abs3(top, c1.x, c1.y);
						top = max_abs3(top, c2.x, c2.y);
						if (s < plane_slots)
						{
							constexpr uint32_t ONE = 0x3c00u;
							asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"((k == 0 ? odd : even) + (uint32_t)s * 16u),
									"r"(left), "r"(__byte_perm(third, ONE, 0x5410)), "r"(right), "r"(__byte_perm(third, ONE, 0x5432)));
						}
					}
				}
			}
			float xmax = (top <= 65504.0f) ? top : INFINITY;       // NaN counts as infinity
			#pragma unroll
			for (int o = 16; o > 0; o >>= 1) { xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, o)); }
			if (lane == 0) { s_xmax[nu % F3_MAX_UNITS_AHEAD][cw] = xmax; }
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
			__syncwarp();
			if (lane == 0) { mbar_arrive(&st_full[es]); }
			if (++es == F3_STAGES) { es = 0; es_phase ^= 1u; }
		}
	}
	else
	{
		// ---- issuer -----------------------------------------------------------------------------------------------------
		const bool leader = elect_one();
		// D = f32, A = B = f16, both K-major
		const uint32_t idesc = (1u << 4) | ((uint32_t)(NN >> 3) << 17) | ((uint32_t)(TC_PIX >> 4) << 24);
		const uint32_t b16 = smem_u32(s_b) >> 4;
		int es = 0, a = 0, used = 0;
		uint32_t es_phase = 0, a_phase = 1;
		bool ok = __all_sync(0xffffffffu, mbar_wait<0>(&ready_bar, 0, s_failed, limit));          // the filter operand
		for (int nu = 0; nu < my_units && ok; ++nu)
		{
			ok = __all_sync(0xffffffffu, mbar_wait<0>(&st_full[es], es_phase, s_failed, limit));
			if (!ok) { break; }
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			uint32_t odd = (a_base + (uint32_t)(es * p.stage_bytes)) >> 4;
			for (int t = 0; t < p.pt; ++t, odd += TC_PIX)
			{
				if (used >= ACC)
				{
					ok = __all_sync(0xffffffffu, mbar_wait<32>(&acc_empty[a], a_phase, s_failed, limit));
					if (!ok) { break; }
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				}
				else { ++used; }
				const uint32_t even = odd + (uint32_t)p.plane_slots;
				#pragma unroll
				for (int k = 0; k < F3_HALVES / 2; ++k)
				{
					// per plane: (row 0, pairs 0 and 1), (row 0, pair 2 and row 1, pair 0), (row 1, pairs 1 and 2)
					const uint32_t from = (k < 3) ? odd : even;
					const uint32_t start = from + ((k % 3 == 0) ? 0u : (k % 3 == 1) ? 2u : (uint32_t)p.pitch + 1u);
					const uint32_t lbo = (k % 3 == 1) ? (uint32_t)p.pitch - 2u : 1u;
					if (leader)
					{
						asm volatile(
							"{\n\t.reg .pred p;\n\t"
							"setp.ne.b32 p, %4, 0;\n\t"
							"tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
							:: "r"(tmem_base + (uint32_t)(a * NN)), "l"(f3_desc(start, lbo)), "l"(f3_desc(b16 + (uint32_t)(2 * k * NN), (uint32_t)NN)), "r"(idesc),
							   "r"(k != 0 ? 1u : 0u), "r"(0u) : "memory");
					}
				}
				if (leader)
				{
					asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&acc_full[a])) : "memory");
				}
				if (++a == ACC) { a = 0; a_phase ^= 1u; }
			}
			if (!ok) { break; }
			if (leader)
			{
				asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&st_empty[es])) : "memory");
			}
			if (++es == F3_STAGES) { es = 0; es_phase ^= 1u; }
		}
		if (!ok)
		{
			if (leader)
			{
				asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&drain_bar)) : "memory");
			}
			mbar_wait_plain(&drain_bar, 0, limit);
		}
		__syncwarp();
	}

	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (*s_failed != 0 && tid == 0) { atomicExch(p.status, 1); }
	if (warp == F3_MMA_WARP)
	{
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512u) : "memory");
	}
}

template <int NF, bool POOL>
static int launch_f3(const F3Params & p, size_t smem, cudaStream_t stream)
{
	// (at least 64 KB: with the static part a smaller request would pass the 48 KB that need no asking)
	const int rc = ensure_dynamic_smem((const void *)float_conv3_signs_kernel<NF, POOL>, smem < 65536 ? 65536 : smem);
	if (rc != XNOR_B200_OK) { return rc; }
	const int grid = (p.units < sm_count()) ? p.units : sm_count();
	float_conv3_signs_kernel<NF, POOL><<<grid, F3_THREADS, smem, stream>>>(p);
	return check_launch();
}

// Up to 32 filters and maps whose rows fit the stages; returns ERR_TOO_LARGE for what has to go to the kernel of float_conv.cu.
int launch_float_conv3_signs(const xnor_b200_conv_desc & d, int pool, const float * input, const float * weights, const float * biases,
		uint32_t * words, int pitch, cudaStream_t stream)
{
	F3Params p = {};
	p.in = input; p.weights = weights; p.biases = biases;
	p.H = d.h; p.W = d.w; p.N = d.n;
	p.BH = (d.h + 1) / 2; p.BW = (d.w + 1) / 2; p.pitch = p.BW + 1;
	p.OH = pool ? d.h / 2 : d.h; p.OW = pool ? d.w / 2 : d.w; p.out_pitch = pitch;
	p.words = words + grid_front(pitch);
	const long long total = (long long)d.batch * (p.BH + 1) * p.pitch;
	if (d.n > 32 || p.pitch < 3 || total > 0x7fff0000LL) { return XNOR_B200_ERR_TOO_LARGE; }
	p.total_pos = (int)total;
	p.d_img = make_div((uint32_t)((p.BH + 1) * p.pitch));
	p.d_pitch = make_div((uint32_t)p.pitch);
	p.vec = (d.w % 2 == 0 && ((uintptr_t)input & 7u) == 0) ? 1 : 0;
	// Tiles per unit: a unit costs its blocks and the row below them, and the busiest SM has ceil(units / SMs) of them.
	double best = 1e30;
	for (int pt = 1; pt <= F3_MAX_PT; ++pt)
	{
		const int slots = pt * TC_PIX + p.pitch + 2;
		if ((size_t)F3_STAGES * round_up((size_t)slots * 32, 128) > F3_SMEM_MAX) { break; }
		const int units = (int)((total + pt * TC_PIX - 1) / (pt * TC_PIX));
		const double cost = (double)((units + sm_count() - 1) / sm_count()) * (slots + 60.0);
		if (cost < best) { best = cost; p.pt = pt; p.units = units; p.plane_slots = slots; }
	}
	if (p.pt == 0) { return XNOR_B200_ERR_TOO_LARGE; }
	p.stage_bytes = (int)round_up((size_t)p.plane_slots * 32, 128);
	TcParams common = {};
	const int rc = tc_fill_launch_fields(common);
	if (rc != XNOR_B200_OK) { return rc; }
	p.status = common.status; p.spin_limit = common.spin_limit;
	const size_t smem = (size_t)F3_STAGES * p.stage_bytes;
	if (d.n <= 16) { return pool ? launch_f3<16, true>(p, smem, stream) : launch_f3<16, false>(p, smem, stream); }
	return pool ? launch_f3<32, true>(p, smem, stream) : launch_f3<32, false>(p, smem, stream);
}

}  // namespace xnor
