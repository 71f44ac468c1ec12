// Float 1x1 and 3x3 stride-1 convolutions (the layers behind the xnor path: yolo and region heads, 255..1024 filters over 256..1024
// channels, and the 3x3 layer in front of a head) on the tcgen05 tensor cores, at
// fp32 accuracy.  A 3x3 layer is the same GEMM with K = (tap, channel): a K block of 32 channels lies in one tap, so its pixel
// rows are the 1x1 layer's, shifted, with zeros where the tap leaves the map.
//
// Replaces, for those layers, the float branch of forward_convolutional_layer_gpu (src-lib/convolutional_kernels.cu:373-434:
// a cuBLAS/cuDNN GEMM per image) + add_bias_gpu + activate_array_ongpu.  out[b][f][p] = bias[f] + sum_c w[f][c] * x[b][c][p].
//
// The tensor core multiplies tf32 (11 significant bits).  Every fp32 operand value v is therefore split into hi, of 11 bits, and lo = v - hi
// (exact in fp32), and three products are accumulated per pair: hi*hi + lo*hi + hi*lo.  The tensor core adds into its fp32 accumulator
// without rounding to nearest: a sum is off by about 2e-8 of itself per accumulating instruction (the small products count for nothing in
// an accumulator of their own).  What decides the accuracy is thus how many instructions one accumulator takes and how the operands are
// split: to the nearest hi, which leaves lo one bit fewer and either sign, or cut off.  Where this kernel stands in for one in plain fp32
// it is no less accurate (2-norm error against fp64, leaky inputs; launch_float_tc has the rule):
//   prepared filters     every K block's sum taken out of tensor memory: 1.2e-7 .. 1.4e-7 (float_conv_map.cu 1.2e-7 .. 3.0e-7); about
//                        650 cycles a block: 3x3 256 -> 512, 4 images of 13x13, 33 us, 27 with 1.3e-6
//   unprepared, 1x1      all products in four accumulators, cut off: 5.6e-7 at 256 channels, 1.9e-6 at 1024 -- far inside what the
//                        reference's own GPU path does (it asks cuDNN for tensor-op math, i.e. single tf32 products, on every
//                        convolution: src-lib/convolutional_layer.cpp:350)
// More than 1024 pixels of a layer with prepared filters: float_conv_tcp.cu.
// Results that the split cannot form (infinite, NaN or nearly infinite factors) are formed again by fp32 multiply-adds, but for the last kind.
//
// One tile of 128 pixels (TMEM lanes; the batch is folded into the pixel index) x 128 filters (TMEM columns) per CTA.  Warp 0 issues
// (converged, one elected lane: a divergent lane takes longer to bring an instruction's operands to the uniform registers than the
// tensor core to execute it): 12 tcgen05.mma.kind::tf32 (M=128, N=128, K=8, 73 cycles each) per K block of 32 channels.  Warps 1..16
// produce the pixel operand -- four threads per row, 8 channels of every K block each, two blocks in flight -- and split it into the
// hi and lo K-major SWIZZLE_128B tiles.  Warp 17 brings the filter operand, which load time has split and laid out in the same form,
// with one 32 KB bulk copy per block.  With few tiles the K blocks are dealt to a cluster of up to four CTAs per tile; the partial
// sums meet in the first one's shared memory and are added in order.  The epilogue adds the bias, applies leaky or the [yolo]
// layer's logistic and stores 32 consecutive pixels of one filter per warp-store.  Every barrier wait is bounded (status word
// shared with the xnor tensor-core kernels).
// Measured: 3x3 256 -> 512 on 4 images of 13x13 33 us (101 without the cluster).  Bound by the tensor pipe and by shared-memory bandwidth
// (64 KB written and 96 KB read per K block: 1280 cycles).
#include "float_tc.cuh"

#include <cooperative_groups.h>

namespace xnor
{

namespace cg = cooperative_groups;

constexpr int FT_ACCS = 4;                                 // accumulators that take the K blocks in turn
constexpr int FT_BUFFERS = 2;                              // K blocks whose sums can be in tensor memory: two accumulators each
constexpr int FT_STAGES = 3;
constexpr int FT_STAGE_BYTES = 4 * FT_TILE_BYTES;          // pixel hi, pixel lo, filter hi, filter lo
constexpr int FT_SMEM_BYTES = FT_STAGES * FT_STAGE_BYTES + 1024;
constexpr int FT_PARTS = 4;                                // producer threads per pixel row: each takes 8 channels of a K block
constexpr int FT_CH = 32 / FT_PARTS;
constexpr int FT_PRODUCER_WARPS = 4 * FT_PARTS;
constexpr int FT_COPY_WARP = FT_PRODUCER_WARPS + 1;
constexpr int FT_THREADS = 32 * (FT_COPY_WARP + 1);

// A thread's part of one operand row of one K block: FT_CH fp32 values -> their 16-byte chunks in the row of the hi tile and
// of the lo tile (chunk c of row r at chunk position c ^ (r % 8); row_swz has the row's swizzle term and the part's first
// chunk folded in).
template <bool NEAREST>
__device__ __forceinline__ void split_row(uint32_t row_swz_hi, uint32_t lo_offset, const float (&v)[FT_CH])
{
	#pragma unroll
	for (int c = 0; c < FT_CH / 4; ++c)
	{
		uint32_t hi[4], lo[4];
		#pragma unroll
		for (int j = 0; j < 4; ++j)
		{
			const uint32_t bits = __float_as_uint(v[4 * c + j]);
			hi[j] = (NEAREST ? bits + 0x1000u : bits) & 0xFFFFE000u;          // split_nearest, or cut off
			lo[j] = __float_as_uint(__fsub_rn(v[4 * c + j], __uint_as_float(hi[j])));
		}
		const uint32_t addr = row_swz_hi ^ (uint32_t)(c << 4);
		asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
		asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(addr + lo_offset), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
	}
}

// The partial sums of the accumulators that were used, added in fp32: 32 columns of this warp's lanes
__device__ __forceinline__ void tile_sums(uint32_t tmem, int used, float (&acc)[32])
{
	#pragma unroll
	for (int j = 0; j < 32; ++j) { acc[j] = 0.0f; }
	#pragma unroll 1
	for (int a = 0; a < used; ++a)
	{
		uint32_t d[32];
		tmem_load<32>(tmem + (uint32_t)(a * FT_NF), d);
		tmem_wait<32>(d);
		#pragma unroll
		for (int j = 0; j < 32; ++j) { acc[j] = (a == 0) ? __uint_as_float(d[j]) : __fadd_rn(acc[j], __uint_as_float(d[j])); }
	}
}

// Adds a group's two accumulators (32 columns of this warp's lanes) to the sums, in fp32.  Eight columns at a time: the loop around it
// keeps the sums and the next K blocks in registers as well.
__device__ __forceinline__ void add_group(uint32_t tmem, float (&sums)[32])
{
	#pragma unroll
	for (int h = 0; h < 32; h += 8)
	{
		uint32_t a[8], b[8];
		asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
			: "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]) : "r"(tmem + (uint32_t)h) : "memory");
		asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
			: "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7]) : "r"(tmem + (uint32_t)(FT_NF + h)) : "memory");
		// nothing uses the registers before the loads have returned
		asm volatile("tcgen05.wait::ld.sync.aligned;"
			: "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
			  "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]) :: "memory");
		#pragma unroll
		for (int j = 0; j < 8; ++j) { sums[h + j] = __fadd_rn(sums[h + j], __fadd_rn(__uint_as_float(a[j]), __uint_as_float(b[j]))); }
	}
}

// RAW: the filters come as Darknet keeps them and are split by the producers as well (callers without a prepared copy, 1x1 only); the K
// blocks then take the accumulators in turn.  Prepared filters: every K block's sum is taken out of tensor memory and added in fp32.
template <bool RAW>
__global__ void __launch_bounds__(FT_THREADS, 1)
float_conv_tc_kernel(const FtParams p)
{
	extern __shared__ uint8_t ft_smem_raw[];
	__shared__ uint64_t bar_full[FT_STAGES];
	__shared__ uint64_t bar_empty[FT_STAGES];
	__shared__ uint64_t bar_done;                              // RAW: the whole tile; else what was issued before a failure
	__shared__ uint64_t acc_full[FT_BUFFERS], acc_empty[FT_BUFFERS];
	__shared__ uint32_t tmem_base_slot;
	__shared__ float s_bias[FT_NF];
	__shared__ int s_failed_storage;
	volatile int * s_failed = &s_failed_storage;

	const int tid = threadIdx.x;
	const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
	const int lane = tid & 31;
	const uint32_t ring = (smem_u32(ft_smem_raw) + 1023u) & ~1023u;
	const int tile = blockIdx.x / p.split;
	const int rank = blockIdx.x - tile * p.split;
	const int tile_p = tile / p.tiles_f;
	const int tile_f = tile - tile_p * p.tiles_f;
	const int f0 = tile_f * FT_NF;
	// this CTA's K blocks
	const int per = (p.kblocks + p.split - 1) / p.split;
	const int kb0 = rank * per;
	const int kbn = max(0, min(p.kblocks - kb0, per));
	const int g0 = tile_p * TC_PIX;                          // first pixel of the tile, batch folded in

	if (tid == 0)
	{
		for (int s = 0; s < FT_STAGES; ++s)
		{
			mbar_init(&bar_full[s], FT_PRODUCER_WARPS + (RAW ? 0 : 1));
			mbar_init(&bar_empty[s], 1);
		}
		mbar_init(&bar_done, 1);
		for (int a = 0; a < (RAW ? 0 : FT_BUFFERS); ++a)
		{
			mbar_init(&acc_full[a], 1);
			mbar_init(&acc_empty[a], FT_PRODUCER_WARPS);
		}
		s_failed_storage = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 0)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
				:: "r"(smem_u32(&tmem_base_slot)), "r"((uint32_t)(FT_ACCS * FT_NF)) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);

	// producers: sums of pixel quarter * 32 + lane, filters of the chunk
	const int quarter = warp & 3, chunk = (warp - 1) >> 2;
	float sums[32];
	if (warp == 0)
	{
		{
			const bool leader = elect_one();
			// instruction descriptor: D = f32, A = B = tf32, both K-major, N = 128, M = 128
			const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(FT_NF >> 3) << 17) | ((uint32_t)(TC_PIX >> 4) << 24);
			bool ok = true;
			for (int kb = 0; kb < kbn && ok; ++kb)
			{
				const int s = kb % FT_STAGES;
				ok = __all_sync(0xffffffffu, mbar_wait(&bar_full[s], (uint32_t)((kb / FT_STAGES) & 1), s_failed, p.spin_limit));
				if (!ok) { break; }
				const int buffer = kb % FT_BUFFERS;
				if (!RAW && kb >= FT_BUFFERS)
				{
					ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buffer], (uint32_t)((kb / FT_BUFFERS - 1) & 1), s_failed, p.spin_limit));
					if (!ok) { break; }
				}
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t a_hi = ring + (uint32_t)s * FT_STAGE_BYTES;
				const uint32_t a_lo = a_hi + FT_TILE_BYTES;
				const uint32_t b_hi = a_hi + 2 * FT_TILE_BYTES;
				const uint32_t b_lo = a_hi + 3 * FT_TILE_BYTES;
				if constexpr (RAW)
				{
					#pragma unroll
					for (int k = 0; k < 4; ++k)                       // 8 tf32 = 32 bytes of every row per instruction
					{
						#pragma unroll
						for (int term = 0; term < 3; ++term)          // the two small terms first, the large one last
						{
							const uint64_t adesc = make_smem_desc((term == 0 ? a_lo : a_hi) + k * 32);
							const uint64_t bdesc = make_smem_desc((term == 1 ? b_lo : b_hi) + k * 32);
							const int turn = kb % FT_ACCS;
							const uint32_t accumulate = (kb >= FT_ACCS || k > 0 || term > 0) ? 1u : 0u;
							if (leader) asm volatile(
								"{\n\t.reg .pred p;\n\t"
								"setp.ne.b32 p, %4, 0;\n\t"
								"tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
								:: "r"(tmem_base + (uint32_t)(turn * FT_NF)), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
						}
					}
				}
				else
				{
					// the small products and the large ones of the first 16 channels in the first accumulator, the other large ones in the second: no
					// sum of large ones takes more than two instructions
					constexpr int FIRST = 2;
					#pragma unroll
					for (int i = 0; i < 12; ++i)
					{
						const int term = i / 4, k = i % 4;
						const bool second = (term == 2 && k >= FIRST);
						const uint64_t adesc = make_smem_desc((term == 0 ? a_lo : a_hi) + k * 32);
						const uint64_t bdesc = make_smem_desc((term == 1 ? b_lo : b_hi) + k * 32);
						const uint32_t accumulate = (i > 0 && !(second && k == FIRST)) ? 1u : 0u;
						if (leader) asm volatile(
							"{\n\t.reg .pred p;\n\t"
							"setp.ne.b32 p, %4, 0;\n\t"
							"tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
							:: "r"(tmem_base + (uint32_t)((2 * buffer + (second ? 1 : 0)) * FT_NF)), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
					}
				}
				if (leader) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
						:: "r"(smem_u32(&bar_empty[s])) : "memory");
				if (!RAW && leader)
				{
					asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&acc_full[buffer])) : "memory");
				}
			}
			if (RAW ? ok : !ok)
			{
				if (leader)
				{
					asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
							:: "r"(smem_u32(&bar_done)) : "memory");
				}
				// leaving early: what was issued must have finished before the tensor memory is released
				if (!RAW) { mbar_wait_plain(&bar_done, 0, p.spin_limit); }
			}
		}
		__syncwarp();
	}
	else if (warp <= FT_PRODUCER_WARPS)
	{
		// ---- producers ------------------------------------------------------------------------------------------------
		const int part = (warp - 1) >> 2;
		const int row = ((warp - 1) & 3) * 32 + lane;
		const uint32_t row_swz0 = (ring + (uint32_t)row * 128u) ^ ((uint32_t)((row & 7) ^ (part * (FT_CH / 4))) << 4);
		const int g = g0 + row, f = f0 + row;
		const bool row_ok = g < p.total;
		const int img = row_ok ? g / p.HW : 0;
		const int pix = row_ok ? g - img * p.HW : 0;
		const float * base = p.x + (size_t)img * p.C * p.HW + pix;
		const int py = pix / p.W, px = pix - py * p.W;
		int tap = kb0 / p.cblocks, cb = kb0 - tap * p.cblocks;    // of the K block that is fetched next
		float buf[2][FT_CH], fil[2][RAW ? FT_CH : 1];
		auto fetch = [&](float (&v)[FT_CH], float (&w)[RAW ? FT_CH : 1])
		{
			const int c0 = cb * 32 + part * FT_CH;
			const float * at = base + (size_t)c0 * p.HW;
			bool ok = row_ok;
			if (p.taps == 9)
			{
				const int dy = tap / 3 - 1, dx = tap - (tap / 3) * 3 - 1;
				ok = ok && py + dy >= 0 && py + dy < p.H && px + dx >= 0 && px + dx < p.W;
				at += dy * p.W + dx;
			}
			if (++cb == p.cblocks) { cb = 0; ++tap; }
			#pragma unroll
			for (int k = 0; k < FT_CH; ++k, at += p.HW)
			{
				v[k] = 0.0f;
				if (ok && c0 + k < p.C) { v[k] = __ldg(at); }
			}
			if constexpr (RAW)
			{
				#pragma unroll
				for (int k = 0; k < FT_CH; ++k) { w[k] = (f < p.N && c0 + k < p.C) ? __ldg(p.w + (size_t)f * p.C + c0 + k) : 0.0f; }
			}
		};
		// the sums of the next group of K blocks, from tensor memory into this thread's
		int n_group = 0;
		#pragma unroll
		for (int j = 0; j < (RAW ? 0 : 32); ++j) { sums[j] = 0.0f; }
		auto collect = [&]()
		{
			const int buffer = n_group % FT_BUFFERS;
			if (!__all_sync(0xffffffffu, mbar_wait<64>(&acc_full[buffer], (uint32_t)((n_group / FT_BUFFERS) & 1), s_failed, p.spin_limit))) { return false; }
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			add_group(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buffer * 2 * FT_NF + chunk * 32), sums);
			++n_group;
			asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
			__syncwarp();
			if (lane == 0) { mbar_arrive(&acc_empty[buffer]); }
			return true;
		};
		if (kbn > 0) { fetch(buf[0], fil[0]); }
		if (kbn > 1) { fetch(buf[1], fil[1]); }
		bool ok = true;
		for (int kb = 0; kb < kbn && ok; kb += 2)
		{
			#pragma unroll
			for (int u = 0; u < 2; ++u)
			{
				if (kb + u >= kbn) { break; }
				const int s = (kb + u) % FT_STAGES;
				if (kb + u >= FT_STAGES)
				{
					ok = mbar_wait(&bar_empty[s], (uint32_t)(((kb + u) / FT_STAGES - 1) & 1), s_failed, p.spin_limit);
					if (!RAW) { ok = __all_sync(0xffffffffu, ok); }
					if (!ok) { break; }
				}
				split_row<!RAW>(row_swz0 + (uint32_t)s * FT_STAGE_BYTES, (uint32_t)FT_TILE_BYTES, buf[u]);
				if constexpr (RAW) { split_row<false>(row_swz0 + (uint32_t)s * FT_STAGE_BYTES + 2u * FT_TILE_BYTES, (uint32_t)FT_TILE_BYTES, fil[u]); }
				if (kb + u + 2 < kbn) { fetch(buf[u], fil[u]); }
				asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
				__syncwarp();
				if (lane == 0) { mbar_arrive(&bar_full[s]); }
				if constexpr (!RAW)
				{
					// a group is taken out while the next is added up: two blocks, which are in flight, behind its last one
					if (kb + u >= n_group + 2) { ok = collect(); }
					if (!ok) { break; }
				}
			}
		}
		if (part == 0) { s_bias[row] = (f < p.N && p.bias != nullptr) ? __ldg(p.bias + f) : 0.0f; }
		if constexpr (!RAW) { while (n_group < kbn && ok) { ok = collect(); } }
	}
	else if (!RAW)
	{
		// ---- filter operand: one bulk copy per K block ------------------------------------------------------------------------
		const bool leader = elect_one();
		const float * src = p.w + ((size_t)tile_f * p.kblocks + kb0) * (2 * FT_TILE_BYTES / 4);
		bool ok = true;
		int issued = 0;
		for (int kb = 0; kb < kbn; ++kb, src += 2 * FT_TILE_BYTES / 4)
		{
			const int s = kb % FT_STAGES;
			if (kb >= FT_STAGES)
			{
				ok = __all_sync(0xffffffffu, mbar_wait<32>(&bar_empty[s], (uint32_t)((kb / FT_STAGES - 1) & 1), s_failed, p.spin_limit));
				if (!ok) { break; }
			}
			if (leader)
			{
				mbar_expect_tx(&bar_full[s], 2u * FT_TILE_BYTES);
				asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
						:: "r"(ring + (uint32_t)s * FT_STAGE_BYTES + 2u * FT_TILE_BYTES), "l"(src), "r"(2u * FT_TILE_BYTES), "r"(smem_u32(&bar_full[s])) : "memory");
			}
			++issued;
			__syncwarp();
		}
		// no copy may be in flight when the CTA leaves: the tile's sums cover it unless something failed
		if (!ok)
		{
			for (int s = 0; s < FT_STAGES && s < issued; ++s) { mbar_wait_plain(&bar_full[s], (uint32_t)(((issued - 1 - s) / FT_STAGES) & 1), p.spin_limit); }
		}
	}

	if (RAW && tid == 0) { mbar_wait<64>(&bar_done, 0, s_failed, p.spin_limit); }
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const bool failed = (*s_failed != 0);
	const int used = min(FT_ACCS, kbn);
	cg::cluster_group cluster = cg::this_cluster();
	if (p.split > 1)
	{
		// every CTA of the tile is through with its stages; the sums of ranks 1.. go to rank 0's
		cluster.sync();
		if (rank > 0 && warp >= 1 && warp <= FT_PRODUCER_WARPS)
		{
			float * theirs = cluster.map_shared_rank(reinterpret_cast<float *>(ft_smem_raw + (ring - smem_u32(ft_smem_raw))), 0) + (size_t)(rank - 1) * FT_NF * TC_PIX;
			if constexpr (RAW) { tile_sums(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(chunk * 32), used, sums); }
			#pragma unroll
			for (int j = 0; j < 32; ++j) { theirs[(chunk * 32 + j) * TC_PIX + quarter * 32 + lane] = sums[j]; }
		}
		cluster.sync();
	}

	if (!failed && rank == 0 && warp >= 1 && warp <= FT_PRODUCER_WARPS)
	{
		// warp w reads the TMEM lanes of quarter w % 4 and one of the four 32-filter chunks
		const int g = g0 + quarter * 32 + lane;
		const bool col_ok = g < p.total;
		const int img = col_ok ? g / p.HW : 0;
		const int pix = col_ok ? g - img * p.HW : 0;
		float * out_pix = p.out + ((size_t)img * p.N + f0 + chunk * 32) * p.HW + pix;
		const float slope = p.leaky ? 0.1f : 1.0f;
		if constexpr (RAW) { tile_sums(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(chunk * 32), used, sums); }
		const float * others = reinterpret_cast<const float *>(ft_smem_raw + (ring - smem_u32(ft_smem_raw))) + (size_t)chunk * 32 * TC_PIX + quarter * 32 + lane;
		for (int r = 1; r < p.split; ++r, others += FT_NF * TC_PIX)
		{
			#pragma unroll
			for (int j = 0; j < 32; ++j) { sums[j] = __fadd_rn(sums[j], others[j * TC_PIX]); }
		}
		const int e0 = (p.yolo_entries > 0) ? (f0 + chunk * 32) % p.yolo_entries : 0;
		int e = e0;
		uint32_t again = 0;
		#pragma unroll
		for (int j = 0; j < 32; ++j)
		{
			if (!RAW && !(fabsf(sums[j]) <= 3.0e38f)) { again |= 1u << j; }
			float v = __fadd_rn(sums[j], s_bias[chunk * 32 + j]);
			v = fmaxf(v, __fmul_rn(v, slope));
			if (p.yolo_entries > 0)
			{
				// logistic on every entry of an anchor but its width and height (head_activate.cu)
				if (e != 2 && e != 3) { v = 1.0f / (1.0f + expf(-v)); }
				if (++e == p.yolo_entries) { e = 0; }
			}
			if (col_ok && f0 + chunk * 32 + j < p.N) { out_pix[(size_t)j * p.HW] = v; }
		}
		if constexpr (!RAW)
		{
			for (int j = 0; j < 32; ++j)
			{
				if (((again >> j) & 1u) == 0 || !col_ok || f0 + chunk * 32 + j >= p.N) { continue; }
				float v = __fadd_rn(plain_sum(p, img, pix, f0 + chunk * 32 + j), s_bias[chunk * 32 + j]);
				v = fmaxf(v, __fmul_rn(v, slope));
				const int entry = (p.yolo_entries > 0) ? (e0 + j) % p.yolo_entries : 2;
				if (entry != 2 && entry != 3) { v = 1.0f / (1.0f + expf(-v)); }
				out_pix[(size_t)j * p.HW] = v;
			}
		}
	}
	else if (failed && tid == 0)
	{
		atomicExch(p.status, 1);
	}

	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == 0)
	{
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"((uint32_t)(FT_ACCS * FT_NF)) : "memory");
	}
}

// Darknet's [n][c][taps] -> the swizzled hi and lo tiles of every K block (tap, 32 channels)
__global__ void float_conv_tc_weights_kernel(const float * __restrict__ w, float * __restrict__ out, int n, int C, int taps, int cblocks)
{
	const int kb = blockIdx.x, tile_f = blockIdx.y;
	const int tap = kb / cblocks, c0 = (kb - tap * cblocks) * 32;
	float * dst = out + ((size_t)tile_f * gridDim.x + kb) * (2 * FT_TILE_BYTES / 4);
	for (int i = threadIdx.x; i < 128 * 32; i += blockDim.x)
	{
		const int row = i >> 5, k = i & 31;
		const int f = tile_f * FT_NF + row, c = c0 + k;
		const float v = (f < n && c < C) ? w[((size_t)f * C + c) * taps + tap] : 0.0f;
		float hi, lo;
		split_nearest(v, hi, lo);
		if (!(fabsf(v) <= 3.0e38f))
		{
			// parts that still add up to v: an infinity or NaN stays in the first
			const bool finite = fabsf(v) <= 3.4028235e38f;
			hi = finite ? __uint_as_float(__float_as_uint(v) & 0xFFFFE000u) : v;
			lo = finite ? __fsub_rn(v, hi) : 0.0f;
		}
		const int at = row * 32 + (((k >> 2) ^ (row & 7)) << 2) + (k & 3);
		dst[at] = hi;
		dst[FT_TILE_BYTES / 4 + at] = lo;
	}
}

// 1x1 / pad 0, or 3x3 / pad 1 over whole K blocks; stride 1
static bool ft_shape_ok(const xnor_b200_conv_desc * d)
{
	return d->stride == 1 && ((d->size == 1 && d->pad == 0) || (d->size == 3 && d->pad == 1 && d->c % 32 == 0));
}

// What of the parameters follows from the shape; tiles of 128 pixels and 128 filters
static int ft_shape(const xnor_b200_conv_desc & d, FtParams & p, long long & total, long long & tiles)
{
	total = (long long)d.batch * d.h * d.w;
	if (total > 0x7fffffffLL - TC_PIX) { return XNOR_B200_ERR_TOO_LARGE; }
	p.C = d.c; p.H = d.h; p.W = d.w; p.HW = d.h * d.w; p.N = d.n;
	p.total = (int)total;
	p.taps = d.size * d.size;
	p.cblocks = (d.c + 31) / 32;
	p.kblocks = p.taps * p.cblocks;
	p.leaky = (d.activation == XNOR_B200_LEAKY) ? 1 : 0;
	p.tiles_f = (d.n + FT_NF - 1) / FT_NF;
	tiles = (long long)p.tiles_f * ((total + TC_PIX - 1) / TC_PIX);
	return (tiles * FT_MAX_SPLIT > 0x7fffffffLL) ? XNOR_B200_ERR_TOO_LARGE : XNOR_B200_OK;
}

template <bool RAW>
static int launch_float_tc(const xnor_b200_conv_desc * desc, const float * input, const float * weights, const float * biases, float * output,
		int yolo_entries, cudaStream_t stream)
{
	if (desc == nullptr || input == nullptr || weights == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	if (!ft_shape_ok(desc)) { return XNOR_B200_ERR_INVALID; }
	if (yolo_entries < 0 || (yolo_entries > 0 && (yolo_entries < 5 || desc->n % yolo_entries != 0))) { return XNOR_B200_ERR_INVALID; }
	if (!RAW && ((uintptr_t)weights & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
	FtParams p;
	long long total = 0, tiles = 0;
	rc = ft_shape(*desc, p, total, tiles);
	if (rc != XNOR_B200_OK) { return rc; }
	p.x = input; p.w = weights; p.bias = biases; p.out = output;
	p.yolo_entries = yolo_entries;
	TcParams tp = TcParams();
	rc = tc_fill_launch_fields(tp);
	if (rc != XNOR_B200_OK) { return rc; }
	p.status = tp.status;
	p.spin_limit = tp.spin_limit;
	// as many CTAs per tile as leave the grid one wave and each of them a few K blocks (about 3 us go into joining the sums)
	p.split = 1;
	for (int s = 2; s <= FT_MAX_SPLIT; ++s) { if (tiles * s <= sm_count() && p.kblocks >= 4 * s) { p.split = s; } }
	if (!RAW && total > 1024) { return launch_float_tcp(p, stream); }
	const auto kernel = float_conv_tc_kernel<RAW>;
	rc = ensure_dynamic_smem((const void *)kernel, FT_SMEM_BYTES);
	if (rc != XNOR_B200_OK) { return rc; }
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)(tiles * p.split), 1, 1);
	cfg.blockDim = dim3(FT_THREADS, 1, 1);
	cfg.dynamicSmemBytes = FT_SMEM_BYTES;
	cfg.stream = stream;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = (unsigned)p.split;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
	return (e == cudaSuccess) ? check_launch() : cuda_fail(e);
}

}  // namespace xnor

using namespace xnor;

extern "C" size_t xnor_b200_float_conv_tc_weights_bytes(const xnor_b200_conv_desc * desc)
{
	if (desc == nullptr || validate_desc(desc) != XNOR_B200_OK || !ft_shape_ok(desc)) { return 0; }
	const size_t tiles_f = (size_t)(desc->n + FT_NF - 1) / FT_NF;
	return tiles_f * (size_t)((desc->c + 31) / 32 * desc->size * desc->size) * 2 * FT_TILE_BYTES;
}

extern "C" int xnor_b200_float_conv_tc_prepare(const xnor_b200_conv_desc * desc, const float * weights, float * tc_weights, void * stream)
{
	if (desc == nullptr || weights == nullptr || tc_weights == nullptr) { return XNOR_B200_ERR_NULL; }
	const int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	if (!ft_shape_ok(desc)) { return XNOR_B200_ERR_INVALID; }
	if (((uintptr_t)tc_weights & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
	const int taps = desc->size * desc->size, cblocks = (desc->c + 31) / 32, tiles_f = (desc->n + FT_NF - 1) / FT_NF;
	if (tiles_f > 65535) { return XNOR_B200_ERR_TOO_LARGE; }
	float_conv_tc_weights_kernel<<<dim3((unsigned)(taps * cblocks), (unsigned)tiles_f, 1), 256, 0, (cudaStream_t)stream>>>(
			weights, tc_weights, desc->n, desc->c, taps, cblocks);
	return check_launch();
}

extern "C" int xnor_b200_float_conv_tc(const xnor_b200_conv_desc * desc, const float * input, const float * tc_weights,
		const float * biases, float * output, int yolo_entries, void * stream)
{
	return launch_float_tc<false>(desc, input, tc_weights, biases, output, yolo_entries, (cudaStream_t)stream);
}

extern "C" int xnor_b200_float_conv_tc_launches(const xnor_b200_conv_desc * desc)
{
	FtParams p;
	long long total = 0, tiles = 0;
	if (desc == nullptr || validate_desc(desc) != XNOR_B200_OK || !ft_shape_ok(desc) || ft_shape(*desc, p, total, tiles) != XNOR_B200_OK) { return 0; }
	return (total > 1024) ? float_tcp_launches(tiles, p.kblocks) : 1;
}

extern "C" int xnor_b200_float_conv_1x1_tc(const xnor_b200_conv_desc * desc, const float * input, const float * weights,
		const float * biases, float * output, void * stream)
{
	if (desc != nullptr && desc->size != 1) { return XNOR_B200_ERR_INVALID; }
	return launch_float_tc<true>(desc, input, weights, biases, output, 0, (cudaStream_t)stream);
}
