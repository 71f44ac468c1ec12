// Float 1x1 and 3x3 stride-1 convolutions of whole batches (the layers behind the xnor path) on the tcgen05 tensor cores at fp32 accuracy:
// the GEMM of float_conv_tc.cu (three tf32 products a pair, filters split at load time) as a persistent kernel for more than 1024 pixels.
//
// What bounded that one at batch was shared memory -- 64 KB written and 96 KB read per K block of 32 channels, 1250 cycles against the
// tensor pipe's 880 -- and, for the short sums of a head (8 to 32 K blocks), the start and the end of a CTA for every tile.  Here
//   * the pixel operand goes to tensor memory: the threads that fetch and split it store it there, and an MMA reads it from there, so
//     shared memory holds filters only (32 KB written by one bulk copy and 48 KB read per K block);
//   * a CTA stays on its SM and takes tile after tile: producers fetch the next tile's pixels while the epilogue of the last one runs;
//   * tiles that do not fill a round of the SMs are a launch of their own whose K blocks are dealt to clusters of two to four CTAs.
// The tensor core adds into its accumulator without rounding to nearest, an error that grows with the number of instructions one takes
// (float_conv_tc.cu).  So the sum is taken out after every two K blocks, or after each where a CTA has few (FP_FEW, FP_FEW_3X3), and added in
// fp32 by warps that do nothing else.  2-norm error against fp64, leaky inputs: 3.3e-7 to 4.0e-7 by pairs, up to 144 K blocks, and 0.9e-7 to
// 1.6e-7 one by one.  Accumulators of whole sums left, 1x1, 3.3e-7 (up to 4 K blocks a CTA) to 1.9e-6 (32), and 3x3, where the small products had
// one of their own, 1.8e-7 (3), 2.7e-7 (9), 3.3e-7 (12), 3.8e-7 (14), 4.7e-7 (18) and 1.7e-6 (72).
//
// Roles: warp 0 issues, 1 copies filters, 4..11 produce the pixel operand (a pixel and 16 of the 32 channels each, two K blocks in flight),
// 12..27 collect (a pixel and 32 filters each).  Tensor memory: two buffers of 128 columns for groups of K blocks, four stages of 64
// columns of pixels.  Every wait is bounded.
// Measured, us before and after: 3x3 256 -> 512 on 64 maps of 13x13 170 -> 138, 1x1 256 -> 255 with the yolo step on 64 of 26x26 76 -> 53,
// 512 -> 255 on 64 of 13x13 41 -> 35, 1024 -> 425 on 256 of 13x13 271 -> 232.  Bound by the tensor pipe (about 1100 cycles a K block; 1400
// in all where sums are long) and, in a head of 8 K blocks, by the way out of a tile's values.  With the shared memory's load halved
// twice the producers (148) or half the collectors (137; heads 65 instead of 53) give nothing.
#include "float_tc.cuh"

#include <cooperative_groups.h>

namespace xnor
{

namespace cg = cooperative_groups;

// K blocks of a CTA's sum up to which each is taken out by itself: where pairs would be less accurate than whole sums were (above), in 3x3
// layers, or where it takes no time.  3x3 with 9 K blocks on 64 maps of 13x13, 512 filters: 35.0 us, 30.9 by pairs, 45 by whole sums.
constexpr int FP_FEW = 4, FP_FEW_3X3 = 12;
constexpr int FP_BUFFERS = 2;
constexpr int FP_STAGES = 4;
constexpr int FP_A_COL = FP_BUFFERS * FT_NF;   // tensor-memory column of the first pixel stage: 32 heads, 32 remainders
constexpr int FP_CH = 16;                      // channels of a K block that a producer thread takes
constexpr int FP_PRODUCERS = 8, FP_COLLECTORS = 16;
constexpr int FP_COPY_WARP = 1, FP_FIRST_PRODUCER = 4, FP_FIRST_COLLECTOR = FP_FIRST_PRODUCER + FP_PRODUCERS;
constexpr int FP_THREADS = 32 * (FP_FIRST_COLLECTOR + FP_COLLECTORS);
// Tiles beyond whole rounds are split from so many K blocks on.  A launch for them that starts as SMs become free costs a few us: at 32 K blocks
// (1x1 1024 -> 425 on 256 of 13x13) 240 without, 232 with it; at 16 (512 -> 255 on 64) 33 without.
constexpr int FP_REST_KBLOCKS = 24;
constexpr int FP_COLS = FT_NF / (FP_COLLECTORS / 4);                    // filters of a collector thread
constexpr int FP_STAGE_BYTES = 2 * FT_TILE_BYTES;                       // filters' heads and remainders
constexpr int FP_SUMS_BYTES = FP_COLLECTORS * 32 * FP_COLS * 4;         // a tile's sums on their way out
constexpr int FP_SMEM_BYTES = FP_STAGES * FP_STAGE_BYTES + FP_SUMS_BYTES + 1024;
static_assert((FT_MAX_SPLIT - 1) * FT_NF * TC_PIX * 4 <= FP_STAGES * FP_STAGE_BYTES + FP_SUMS_BYTES, "the partial sums of a cluster's other CTAs");

__device__ __forceinline__ void tmem_store8(uint32_t taddr, const float (&v)[8])
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
		:: "r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

__global__ void __launch_bounds__(FP_THREADS, 1)
float_conv_tcp_kernel(const __grid_constant__ FtParams p)
{
	extern __shared__ uint8_t fp_smem_raw[];
	__shared__ uint64_t full[FP_STAGES], empty[FP_STAGES], acc_full[FP_BUFFERS], acc_empty[FP_BUFFERS], drain_bar;
	__shared__ float s_bias[FP_COLLECTORS][FP_COLS];
	__shared__ uint32_t tmem_base_slot;
	__shared__ int s_failed_storage;
	volatile int * s_failed = &s_failed_storage;

	const int tid = threadIdx.x;
	const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
	const int lane = tid & 31;
	const uint32_t limit = p.spin_limit;
	const uint32_t ring = (smem_u32(fp_smem_raw) + 1023u) & ~1023u;
	float * const room = reinterpret_cast<float *>(fp_smem_raw + (ring - smem_u32(fp_smem_raw)));
	// a cluster of `split` CTAs per tile, or CTAs that take every gridDim.x-th tile
	const int first_tile = p.tile0 + (int)blockIdx.x / p.split;
	const int tile_step = (int)gridDim.x / p.split;
	const int end_tile = p.tile0 + p.tiles;
	const int rank = (int)blockIdx.x % p.split;
	const int per = (p.kblocks + p.split - 1) / p.split;
	const int kb0 = rank * per;
	const int kbn = max(0, min(p.kblocks - kb0, per));                 // this CTA's K blocks of a tile
	const int my_tiles = (end_tile - first_tile + tile_step - 1) / tile_step;
	const int total = my_tiles * kbn;
	const int group_blocks = (per <= ((p.taps == 9) ? FP_FEW_3X3 : FP_FEW)) ? 1 : 2;                  // K blocks whose products meet in tensor memory
	auto filters_of = [&](int tile) { return (tile + tile / p.turn) % p.tiles_f; };                                // filter tile of a tile
	// Filters that its products are formed for: an instruction takes any multiple of 16, in time that goes with it (1x1 256 -> 18 on 64 of 26x26
	// 24.9 -> 22.7 us, 512 -> 75 on 64 of 13x13 18.7 -> 17.8)
	auto width_of = [&](int tile_f) { return min(FT_NF, (p.N - tile_f * FT_NF + 15) & ~15); };

	if (tid == 0)
	{
		for (int s = 0; s < FP_STAGES; ++s)
		{
			mbar_init(&full[s], FP_PRODUCERS + 1);
			mbar_init(&empty[s], 1);
		}
		for (int a = 0; a < FP_BUFFERS; ++a)
		{
			mbar_init(&acc_full[a], 1);
			mbar_init(&acc_empty[a], FP_COLLECTORS);
		}
		mbar_init(&drain_bar, 1);
		s_failed_storage = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (tid < FP_COLLECTORS * FP_COLS) { s_bias[tid / FP_COLS][tid % FP_COLS] = 0.0f; }
	if (warp == 0)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
	// The launch of the tiles that are left over reads nothing of this one's: it starts as SMs become free, and waits for this one's end only so as
	// to end behind it.
	if (p.more) { pdl_trigger(); }
	// producers and collectors: a warp reaches the 32 tensor-memory lanes (pixels) of its number modulo 4
	const int quarter = warp & 3;
	// what every role does at its end: nobody's shared or tensor memory goes while another still works on it
	auto meet = [&]()
	{
		asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
		__syncthreads();
	};
	auto clusters_meet = [&]() { cg::this_cluster().sync(); };

	if (warp == 0)
	{
		// ---- issuer: the warp stays converged, one elected lane issues ---------------------------------------------------------
		const bool leader = elect_one();
		bool ok = true;
		int it = 0, group = 0;
		for (int tile = first_tile; tile < end_tile && ok; tile += tile_step)
		{
			// D = f32, A = B = tf32, both K-major, M = 128
			const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(width_of(filters_of(tile)) >> 3) << 17) | ((uint32_t)(TC_PIX >> 4) << 24);
			for (int kb = 0; kb < kbn; ++kb, ++it)
			{
				const int s = it % FP_STAGES, buffer = group % FP_BUFFERS;
				ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (uint32_t)((it / FP_STAGES) & 1), s_failed, limit));
				if (!ok) { break; }
				if (kb % group_blocks == 0 && group >= FP_BUFFERS)
				{
					ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buffer], (uint32_t)((group / FP_BUFFERS - 1) & 1), s_failed, limit));
					if (!ok) { break; }
				}
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t a_hi = tmem_base + (uint32_t)(FP_A_COL + s * 64), b_hi = ring + (uint32_t)(s * FP_STAGE_BYTES);
				#pragma unroll
				for (int i = 0; i < 12; ++i)
				{
					// 8 channels an instruction; the small products of the block first
					const int term = i / 4, k = i % 4;
					const uint32_t a = a_hi + (uint32_t)((term == 0 ? 32 : 0) + k * 8);
					const uint64_t bdesc = make_smem_desc(b_hi + (uint32_t)((term == 1 ? FT_TILE_BYTES : 0) + k * 32));
					if (leader) asm volatile(
						"{\n\t.reg .pred p;\n\t"
						"setp.ne.b32 p, %4, 0;\n\t"
						"tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
						:: "r"(tmem_base + (uint32_t)(buffer * FT_NF)), "r"(a), "l"(bdesc), "r"(idesc), "r"((kb % group_blocks > 0 || i > 0) ? 1u : 0u), "r"(0u) : "memory");
				}
				if (leader) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&empty[s])) : "memory");
				if (kb % group_blocks == group_blocks - 1 || kb == kbn - 1)
				{
					if (leader) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&acc_full[buffer])) : "memory");
					++group;
				}
			}
		}
		if (!ok)
		{
			// leaving early: what was issued must have finished before the tensor memory is released
			if (leader) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&drain_bar)) : "memory");
			mbar_wait_plain(&drain_bar, 0, limit);
		}
		__syncwarp();
		meet();
		if (p.split > 1)
		{
			clusters_meet();
			clusters_meet();
		}
		if (*s_failed != 0 && lane == 0) { atomicExch(p.status, 1); }
		meet();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512u) : "memory");
	}
	else if (warp < FP_FIRST_PRODUCER)
	{
		// (two warps of these do nothing)
		if (warp == FP_COPY_WARP)
		{
			// ---- filters: one bulk copy per K block ----------------------------------------------------------------------------------
			const bool leader = elect_one();
			bool ok = true;
			int it = 0;
			for (int tile = first_tile; tile < end_tile && ok; tile += tile_step)
			{
				const float * src = p.w + ((size_t)filters_of(tile) * p.kblocks + kb0) * (FP_STAGE_BYTES / 4);
				for (int kb = 0; kb < kbn; ++kb, ++it, src += FP_STAGE_BYTES / 4)
				{
					const int s = it % FP_STAGES;
					if (it >= FP_STAGES)
					{
						ok = __all_sync(0xffffffffu, mbar_wait<32>(&empty[s], (uint32_t)((it / FP_STAGES - 1) & 1), s_failed, limit));
						if (!ok) { break; }
					}
					if (leader)
					{
						mbar_expect_tx(&full[s], (uint32_t)FP_STAGE_BYTES);
						asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
								:: "r"(ring + (uint32_t)(s * FP_STAGE_BYTES)), "l"(src), "r"((uint32_t)FP_STAGE_BYTES), "r"(smem_u32(&full[s])) : "memory");
					}
					__syncwarp();
				}
			}
			// no copy may be in flight when the CTA leaves: the products cover it unless something failed
			if (!ok) { for (int s = 0; s < FP_STAGES && s < it; ++s) { mbar_wait_plain(&full[s], (uint32_t)(((it - 1 - s) / FP_STAGES) & 1), limit); } }
		}
		meet();
		if (p.split > 1)
		{
			clusters_meet();
			clusters_meet();
		}
		meet();
	}
	else if (warp < FP_FIRST_COLLECTOR)
	{
		// ---- producers -----------------------------------------------------------------------------------------------------------
		const int part = (warp - FP_FIRST_PRODUCER) >> 2;
		const int row = quarter * 32 + lane;
		const uint32_t to = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(FP_A_COL + part * FP_CH);
		// what is fetched next
		int tile = first_tile, left = 0, tap = 0, cb = 0, py = 0, px = 0;
		bool row_ok = false;
		const float * base = p.x;
		auto fetch = [&](float (&v)[FP_CH])
		{
			if (left == 0)
			{
				// the next tile's pixel of this thread
				const int g = (tile / p.tiles_f) * TC_PIX + row;
				row_ok = g < p.total;
				const int img = row_ok ? g / p.HW : 0;
				const int pix = row_ok ? g - img * p.HW : 0;
				base = p.x + (size_t)img * p.C * p.HW + pix;
				py = pix / p.W;
				px = pix - py * p.W;
				tap = kb0 / p.cblocks;
				cb = kb0 - tap * p.cblocks;
				left = kbn;
				tile += tile_step;
			}
			const int c0 = cb * 32 + part * FP_CH;
			const float * at = base + (size_t)c0 * p.HW;
			bool ok = row_ok;
			if (p.taps == 9)
			{
				const int dy = tap / 3 - 1, dx = tap - (tap / 3) * 3 - 1;
				ok = ok && py + dy >= 0 && py + dy < p.H && px + dx >= 0 && px + dx < p.W;
				at += dy * p.W + dx;
			}
			if (++cb == p.cblocks) { cb = 0; ++tap; }
			--left;
			#pragma unroll
			for (int k = 0; k < FP_CH; ++k) { v[k] = 0.0f; }
			if (c0 + FP_CH <= p.C)
			{
				#pragma unroll
				for (int k = 0; k < FP_CH; ++k, at += p.HW) { if (ok) { v[k] = __ldg(at); } }
			}
			else
			{
				#pragma unroll
				for (int k = 0; k < FP_CH; ++k, at += p.HW) { if (ok && c0 + k < p.C) { v[k] = __ldg(at); } }
			}
		};
		float buf[2][FP_CH];
		if (total > 0) { fetch(buf[0]); }
		if (total > 1) { fetch(buf[1]); }
		bool ok = true;
		for (int it = 0; it < total && ok; it += 2)
		{
			#pragma unroll
			for (int u = 0; u < 2; ++u)
			{
				if (it + u >= total) { break; }
				const int s = (it + u) % FP_STAGES;
				if (it + u >= FP_STAGES)
				{
					ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], (uint32_t)(((it + u) / FP_STAGES - 1) & 1), s_failed, limit));
					if (!ok) { break; }
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				}
				#pragma unroll
				for (int h = 0; h < FP_CH; h += 8)
				{
					float hi[8], lo[8];
					#pragma unroll
					for (int k = 0; k < 8; ++k) { split_nearest(buf[u][h + k], hi[k], lo[k]); }
					tmem_store8(to + (uint32_t)(s * 64 + h), hi);
					tmem_store8(to + (uint32_t)(s * 64 + 32 + h), lo);
				}
				if (it + u + 2 < total) { fetch(buf[u]); }
				asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) { mbar_arrive(&full[s]); }
			}
		}
		meet();
		if (p.split > 1)
		{
			clusters_meet();
			clusters_meet();
		}
		meet();
	}
	else
	{
		// ---- collectors ----------------------------------------------------------------------------------------------------------
		float sums[FP_COLS];                                               // of this thread's pixel
		// collectors: the tile's values leave, a few filters at a time (the sums lie in shared memory meanwhile: a loop over registers would be
		// unrolled whole, with a logistic for each)
		auto finish = [&](int tile, const float (&sums)[FP_COLS])
		{
			const int cw = warp - FP_FIRST_COLLECTOR;
			const int f0 = filters_of(tile) * FT_NF + (cw >> 2) * FP_COLS;
			const int g = (tile / p.tiles_f) * TC_PIX + quarter * 32 + lane;
			const int n = min(FP_COLS, p.N - f0);
			if (n <= 0) { return; }
			float * mine = room + FP_STAGES * FP_STAGE_BYTES / 4 + (size_t)cw * 32 * FP_COLS + lane;
			__syncwarp();
			if (p.bias != nullptr)
			{
				#pragma unroll
				for (int j = 0; j < FP_COLS; j += 32) { s_bias[cw][j + lane] = (j + lane < n) ? __ldg(p.bias + f0 + j + lane) : 0.0f; }
			}
			uint32_t again = 0;                        // values that the products could not form
			#pragma unroll
			for (int j = 0; j < FP_COLS; ++j)
			{
				mine[j * 32] = sums[j];
				if (!(fabsf(sums[j]) <= 3.0e38f)) { again |= 1u << j; }
			}
			__syncwarp();
			// entries that the [yolo] layer's logistic is not for: width and height of an anchor
			uint32_t plain = 0xffffffffu;
			if (p.yolo_entries > 0) { plain = __ballot_sync(0xffffffffu, (unsigned)((f0 + lane) % p.yolo_entries - 2) < 2u); }
			if (g >= p.total) { return; }
			const int img = g / p.HW, pix = g - img * p.HW;
			float * const out = p.out + ((size_t)img * p.N + f0) * p.HW + pix;
			const float slope = p.leaky ? 0.1f : 1.0f;
			// eight at a time, so that their chains run side by side
			for (int j0 = 0; j0 < n; j0 += 8)
			{
				float v[8];
				#pragma unroll
				for (int q = 0; q < 8; ++q)
				{
					v[q] = __fadd_rn(mine[(j0 + q) * 32], s_bias[cw][j0 + q]);
					v[q] = fmaxf(v[q], __fmul_rn(v[q], slope));
				}
				if (p.yolo_entries > 0)
				{
					float e[8];
					#pragma unroll
					for (int q = 0; q < 8; ++q) { e[q] = 1.0f + expf(-v[q]); }
					#pragma unroll
					for (int q = 0; q < 8; ++q) { e[q] = __frcp_rn(e[q]); }
					#pragma unroll
					for (int q = 0; q < 8; ++q) { v[q] = ((plain >> (j0 + q)) & 1) ? v[q] : e[q]; }
				}
				float * to = out + (size_t)j0 * p.HW;
				if (j0 + 8 <= n)
				{
					#pragma unroll
					for (int q = 0; q < 8; ++q, to += p.HW) { *to = v[q]; }
				}
				else
				{
					#pragma unroll
					for (int q = 0; q < 8; ++q, to += p.HW) { if (j0 + q < n) { *to = v[q]; } }
				}
			}
			for (int j = 0; again != 0 && j < n; ++j)
			{
				if (((again >> j) & 1) == 0) { continue; }
				float v = __fadd_rn(plain_sum(p, img, pix, f0 + j), s_bias[cw][j]);
				v = fmaxf(v, __fmul_rn(v, slope));
				out[(size_t)j * p.HW] = ((plain >> j) & 1) ? v : 1.0f / (1.0f + expf(-v));
			}
		};
		const uint32_t from = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(((warp - FP_FIRST_COLLECTOR) >> 2) * FP_COLS);
		bool ok = true;
		int group = 0;
		for (int tile = first_tile; tile < end_tile && ok; tile += tile_step)
		{
			#pragma unroll
			for (int j = 0; j < FP_COLS; ++j) { sums[j] = 0.0f; }
			for (int kb = 0; kb < kbn; kb += group_blocks, ++group)
			{
				const int buffer = group % FP_BUFFERS;
				ok = __all_sync(0xffffffffu, mbar_wait<64>(&acc_full[buffer], (uint32_t)((group / FP_BUFFERS) & 1), s_failed, limit));
				if (!ok) { break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				#pragma unroll
				for (int h = 0; h < FP_COLS; h += 16)
				{
					uint32_t d[16];
					tmem_load<16>(from + (uint32_t)(buffer * FT_NF + h), d);
					tmem_wait<16>(d);
					#pragma unroll
					for (int j = 0; j < 16; ++j) { sums[h + j] = __fadd_rn(sums[h + j], __uint_as_float(d[j])); }
				}
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) { mbar_arrive(&acc_empty[buffer]); }
			}
			if (ok && p.split == 1) { finish(tile, sums); }
		}
		meet();
		if (p.split > 1)
		{
			// every CTA of the tile is through with its stages; the sums of ranks 1.. go to rank 0's and are added in order
			cg::cluster_group cluster = cg::this_cluster();
			const size_t at = (size_t)((warp - FP_FIRST_COLLECTOR) >> 2) * FP_COLS * TC_PIX + quarter * 32 + lane;
			clusters_meet();
			if (rank > 0)
			{
				float * theirs = cluster.map_shared_rank(room, 0) + (size_t)(rank - 1) * FT_NF * TC_PIX + at;
				#pragma unroll
				for (int j = 0; j < FP_COLS; ++j) { theirs[j * TC_PIX] = sums[j]; }
			}
			clusters_meet();
			if (rank == 0)
			{
				for (int r = 1; r < p.split; ++r)
				{
					const float * others = room + (size_t)(r - 1) * FT_NF * TC_PIX + at;
					#pragma unroll
					for (int j = 0; j < FP_COLS; ++j) { sums[j] = __fadd_rn(sums[j], others[j * TC_PIX]); }
				}
				// (the sums of the last rank may lie where this warp's are about to)
				asm volatile("bar.sync 1, %0;" :: "n"(FP_COLLECTORS * 32) : "memory");
				if (*s_failed == 0) { finish(first_tile, sums); }
			}
		}
		meet();
	}
	pdl_wait();
}

static int launch_tiles(const FtParams & p, cudaStream_t stream, bool behind = false)
{
	const int rc = ensure_dynamic_smem((const void *)float_conv_tcp_kernel, FP_SMEM_BYTES);
	if (rc != XNOR_B200_OK) { return rc; }
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)((p.split > 1) ? p.tiles * p.split : (p.tiles < sm_count()) ? p.tiles : sm_count()), 1, 1);
	cfg.blockDim = dim3(FP_THREADS, 1, 1);
	cfg.dynamicSmemBytes = FP_SMEM_BYTES;
	cfg.stream = stream;
	cudaLaunchAttribute attr[2];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = (unsigned)p.split;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	cfg.attrs = attr;
	attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.numAttrs = behind ? 2 : 1;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, float_conv_tcp_kernel, p);
	return (e == cudaSuccess) ? check_launch() : cuda_fail(e);
}

// Whole rounds of the SMs first; what is left of the tiles (all, if they are fewer than the SMs) with its K blocks dealt to as many CTAs a
// tile as there is room for, four K blocks each at least (about 3 us go into joining the sums).  How many CTAs that is; 1: one launch for all.
static int rest_split(int all, int kblocks)
{
	const int rest = all % sm_count();
	int split = 1;
	for (int s = 2; s <= FT_MAX_SPLIT; ++s) { if (rest * s <= sm_count() && kblocks >= 4 * s) { split = s; } }
	return (rest == 0 || (all > rest && kblocks < FP_REST_KBLOCKS)) ? 1 : split;
}

int float_tcp_launches(long long tiles, int kblocks)
{
	return (tiles >= sm_count() && rest_split((int)tiles, kblocks) > 1) ? 2 : 1;
}

int launch_float_tcp(FtParams & p, cudaStream_t stream)
{
	const long long tiles = (long long)p.tiles_f * ((p.total + (long long)TC_PIX - 1) / TC_PIX);
	if (tiles * FT_MAX_SPLIT > 0x7fffffffLL || tiles / sm_count() * p.kblocks > 0x7ffffff0LL) { return XNOR_B200_ERR_TOO_LARGE; }
	const int all = (int)tiles, rest = all % sm_count(), split = rest_split(all, p.kblocks);
	p.tile0 = 0;
	p.split = 1;
	p.more = 0;
	// Where every CTA would take the same filter tile each time (four of them, 148 SMs), the order moves on by one after every round: the last
	// filter tile may be narrower, and those that had no other would finish early (3x3 512 -> 144 on 128 of 13x13 252 -> 240 us, 1x1 1024 -> 425 on
	// 256 of them 244 -> 240; narrow tiles all at the end instead: 244 and 254, a tile's pixels then come from memory twice).
	p.turn = (sm_count() % p.tiles_f == 0) ? sm_count() : 0x7fffffff;
	if (split == 1)
	{
		p.tiles = all;
		return launch_tiles(p, stream);
	}
	p.tiles = all - rest;
	p.more = 1;
	if (p.tiles > 0)
	{
		const int rc = launch_tiles(p, stream);
		if (rc != XNOR_B200_OK) { return rc; }
	}
	p.tile0 = all - rest;
	p.tiles = rest;
	p.split = split;
	p.more = 0;
	return launch_tiles(p, stream, all > rest);
}

}  // namespace xnor
