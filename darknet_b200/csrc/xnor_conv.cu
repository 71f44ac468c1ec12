// XNOR convolution straight from sign words, without an im2col operand: persistent tcgen05 kernel, kind::mxf4.
//
// A binary dot product is an ordinary one over +1 / -1, which the tensor core takes as 4-bit floats (e2m1 +1.0 = 0x2, -1.0 = 0xA,
// block scale factors 2^0, exact fp32 accumulators).  The packed im2col rows of the GEMM kernels repeat every input bit nine
// times in memory and widen it nine times in shared memory; those kernels sit at the shared-memory bandwidth while the tensor
// pipe idles at a third.  Here a pixel's 32-channel sign word is widened ONCE per tile, to 16 bytes, into a plane
// [channel block][position] of shared memory.  The MMA's operand layout without a swizzle -- 8-row x 16-byte core matrices, free
// strides between them -- reads such a plane from any 16-byte boundary, so a filter tap is nothing but another start address:
//
//   position = (image * (H + 1) + y) * pitch + x        one padding row per image and pitch - W >= 1 padding columns, shared by
//   tap (ky, kx) of position p = position p + (ky - 1) * pitch + (kx - 1)                                           neighbours
//
// and the 128 rows of an MMA are 128 consecutive positions (those on the padding are computed and dropped).  pitch = W + 1
// computes the fewest; a multiple of 8 over rows of a multiple of 8 pixels keeps a warp's fp32 rows on whole 32-byte sectors:
// a read-and-write pass of this shape runs at 5.8 TB/s then, at 3.5 over partly written sectors (both with evict-first stores).
// Sign tensors are kept on this grid ("grid words": [channel block][position], zeros on the padding, which is "not > 0"), so the
// window of a tile is one contiguous run per channel block, fetched by one bulk copy, and a tile's sign words are stored where
// its positions are.  A stride-2 layer widens into four planes, one per parity of (y, x), on the output's grid.  Filters are
// widened the same way into [K word][filter] and stay in shared memory for the life of the CTA where they fit (128 filters x
// 2304 bits); channels that do not exist are +0.0 in the filters and contribute nothing.  K order: channel block outer, tap inner.
//
// The input may be read through what lies between two layers: a 2x2 max-pool (OR of four words), a nearest x2 upsample, a
// channel concatenation of two tensors.  Output: sign words, fp32, or the fp32 sum with a fused [shortcut] and its sign words.
//
// Roles (one CTA per SM): warps 0..15 epilogue, 16..21 expanders, 22 bulk copies, 23 issuer.  A stage is G channel blocks of the
// unit's window (and, when the filters do not fit, the filters' words of the same K range); a unit is PT tiles of 128 positions
// that share a stage; accumulators form a ring in tensor memory, so the epilogue of one tile runs under the MMAs of the next.
// Every wait is bounded as in the GEMM kernels.
//
// What was learned on the way (1024 filters, K = 9216, 43264 pixels): words gathered with loads by the expanders 1400 us, with
// asynchronous 4-byte copies 1000 us -- about 80 instructions a word either way, the expanders bound everything -- hence the grid
// and the bulk copies.  A single lane in a divergent branch issues an MMA every 80 to 350 cycles because every operand has to
// be moved to the uniform registers; a converged warp with one elected lane issues at the pipe's rate (47 / 56 / 73 cycles for
// 32 / 64 / 128 filters x 64 bits).
//
// Measured (B200, 64 images, before and after the shortcut operand's loads lost their conditions and values went in pairs): 128 -> 256
// 3x3 56x56 with a shortcut 153 -> 88 us (63 at the copy rate), 256 -> 512 28x28 88 -> 59; 128 -> 256 104x104 to fp32 188 -> 172
// (108 at the copy rate).  Bound by the SM's issue slots, 53 % busy for the last of these, and the shared-memory pipe (68 %); with a
// shortcut and both tensors written, by memory latency (issue slots 26 %, DRAM 41 %).  Twice the expanders (188 us), half the epilogue warps (225), scales kept in registers (172): no gain.
#include "grid_words.cuh"
#include "tc_common.cuh"

namespace xnor
{

constexpr int XC_EPI_WARPS = 16;
constexpr int XC_EXP_WARPS = 6;
constexpr int XC_COPY_WARP = XC_EPI_WARPS + XC_EXP_WARPS;
constexpr int XC_MMA_WARP = XC_COPY_WARP + 1;
constexpr int XC_THREADS = (XC_MMA_WARP + 1) * 32;     // 24 warps: six per scheduler, 80 registers a thread
constexpr int XC_EXP_THREADS = XC_EXP_WARPS * 32;
constexpr int XC_ITEMS = 8;                   // words of a stage per expander thread
constexpr int XC_MAX_STAGES = 4;
constexpr int XC_RAW_STAGES = 3;              // stages whose bits are on their way
constexpr int XC_TABLES = XC_RAW_STAGES + 1;  // window tables: one per unit that can be under way
constexpr int XC_MAX_ACC = 14;
constexpr long long XC_STREAM_BYTES = 32 << 20;   // fp32 tensors above this size do not expect their reader to find them in the L2
constexpr int XC_TMEM_COLS = 512;
constexpr int XC_SF_COL = 448;                // accumulators below, scale factors (pixels here, filters at + 8) above
constexpr int XC_MAX_KW = 18;                 // K words of a stage
constexpr int XC_SMEM_MAX = 222 * 1024;       // dynamic shared memory; the rest is static

// How the positions of a window are found in a source
enum { XC_LINEAR = 0,       // same grid: a contiguous run
       XC_SINGLE = 1,       // one word each, through the window table (upsampled, or a 1x1 layer of stride 2)
       XC_OR4 = 2,          // through the table, 2x2 max-pool: OR of four words
       XC_PLANES4 = 3 };    // 3x3 layer of stride 2: four words, one for each parity plane

struct XcSource
{
	const uint32_t * words;  // position 0 of block 0 minus the guard: [blocks][block_words]
	int blocks, h, w, pitch;
	int front, block_words;  // guard words in front of position 0, words of a block
	int mode;
	int scale;               // source row / column of output row / column: 2 (times two), 1, 0 (half)
};

struct XcParams
{
	XcSource src[2];
	int n_src, tabled;          // tabled: the sources need the window table
	const uint32_t * weights;   // [filters / 128][K word][128]
	const float * mean_arr;
	const float * bias;
	float * out;
	uint32_t * signs;
	const float * sc_in;
	float * sc_out;
	uint32_t * sc_signs;
	int M, K;                // filters; channels * taps: the largest magnitude an accumulator can have
	int leaky;
	float minus_zero;        // -0.0f
	int stream_values;       // the fp32 tensors are too large for the L2: what is read goes first
	int stream_out;          // ... and what is written, unless a layer behind this one reads its end first
	int backwards;           // the last unit of the batch first
	int batch, OH, OW, n_pix;   // images, output map
	int out_front, out_block_words;   // of sign words on the output's grid
	int stride, taps;
	int nb, G, stages_k;     // channel blocks, blocks per stage, stages per unit
	int kwords;              // nb * taps
	uint32_t last_mask;      // channels that exist in the last block
	FastDiv d_img, d_pitch;  // positions per image, positions per row
	FastDiv d_kw;            // K words of a full stage (kw_full)
	int pitch, rows;         // of the position grid
	int total_pos, halo;     // positions of the batch; positions in front of a tile that its window needs
	int planes, slots_plane; // parity planes, window positions of one
	int slots;               // planes * slots_plane
	int pt, units;           // tiles per unit, units
	int fgroups;             // filter groups of NF
	int ring;                // operand stages
	int kw_full;             // K words of a full stage, rounded up to even
	int a_stage_bytes, b_stage_bytes;
	int raw_words;           // words of one channel block's run in a raw stage (a multiple of 4)
	int raw_stage_bytes;
	int * status;
	uint32_t spin_limit;
	int withhold;
};

// The accesses of the expanders carry no memory clobber: volatile keeps them in order among themselves and with the barrier
// operations, and the compiler may keep the kernel's parameters in registers across them.
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint4 v)
{
	asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
}

// Shared-memory matrix descriptor, K-major without swizzle: 8-row core matrices of 128 contiguous bytes, the two 16-byte K halves
// of an instruction `start_lbo >> 16` 16-byte units apart, consecutive 8-row groups 128 bytes apart; low half: start in 16-byte units.
__device__ __forceinline__ uint64_t plane_desc(uint32_t start_lbo)
{
	return (uint64_t)start_lbo | ((uint64_t)(8u | (1u << 14)) << 32);
}

// Filter word -> 16 bytes of e2m1; channels outside `mask` become +0.0.
__device__ __forceinline__ uint4 expand_filter(uint32_t bits, uint32_t mask)
{
	uint4 v = expand_fp4(bits);
	if (mask != 0xffffffffu)
	{
		v.x &= (mask & 0x11111111u) * 15u;
		v.y &= ((mask >> 1) & 0x11111111u) * 15u;
		v.z &= ((mask >> 2) & 0x11111111u) * 15u;
		v.w &= ((mask >> 3) & 0x11111111u) * 15u;
	}
	return v;
}

// Channel block (within its stage) of K word j: stages hold at most two blocks of nine taps, or up to eight of one.
__device__ __forceinline__ int block_of(int j, int taps) { return (taps == 1) ? j : (j >= 9 ? 1 : 0) + (j >= 18 ? 1 : 0); }

// K word j of a stage: which tap it is.  The two words of an instruction must lie in order of address, and with parity planes the
// taps' addresses are not in tap order, so there they are walked plane by plane.
__device__ __forceinline__ int tap_of(int j, int stride, int taps)
{
	if (stride == 1 || taps == 1) { return j; }
	// planes (even y, even x): tap 4; (even, odd): 3, 5; (odd, even): 1, 7; (odd, odd): 0, 2, 6, 8
	constexpr uint64_t order = 0x862071534ull;
	return (int)((order >> (4 * j)) & 15u);
}

// Where tap t of a stage's first channel block starts, in 16-byte units from the start of that block's planes.
__device__ __forceinline__ int tap_offset(const XcParams & p, int t, int stride, int taps)
{
	if (taps == 1) { return 0; }
	const int ky = t / 3, kx = t - ky * 3;
	if (stride == 1) { return ky * p.pitch + kx; }
	const int plane = ((ky == 1) ? 0 : 2) + ((kx == 1) ? 0 : 1);
	return plane * p.slots_plane + p.halo + ((ky == 0) ? -p.pitch : 0) + ((kx == 0) ? -1 : 0);
}

// K word j of stage st, widened into its place in the filter operand; what does not exist is +0.0.
template <int NF>
__device__ __forceinline__ void put_filter(const XcParams & p, int taps, uint32_t dst, int st, int j, int f, uint32_t bits)
{
	const int k = st * p.G * taps + j;
	uint4 v = make_uint4(0, 0, 0, 0);
	if (k < p.kwords && j < p.G * taps) { v = expand_filter(bits, (k >= p.kwords - taps) ? p.last_mask : 0xffffffffu); }
	st_shared_v4(dst + (uint32_t)(j * NF + f) * 16u, v);
}

__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr)
{
	uint32_t v;
	asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
	return v;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const uint32_t * src, uint32_t bytes, uint64_t * bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
			:: "r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// fp32 values that pass through the L2 once: evicted first
__device__ __forceinline__ uint64_t stream_policy(bool stream)
{
	uint64_t first, normal;
	asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
	asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
	return stream ? first : normal;
}

__device__ __forceinline__ float ld_policy(const float * at, uint64_t policy)
{
	float v;
	asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(at), "l"(policy));
	return v;
}

__device__ __forceinline__ void st_policy(float * at, float v, uint64_t policy)
{
	asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" :: "l"(at), "f"(v), "l"(policy));
}

// Two fp32 operations in one instruction, each rounded as the plain one is.
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
	uint64_t v;
	asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
	return v;
}

__device__ __forceinline__ void unpack2(uint64_t v, float & lo, float & hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
	uint64_t v;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
	return v;
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
	uint64_t v;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
	return v;
}

// The run of a source's words (from its block start, 16-byte aligned) that holds the window of unit u, and where in it the
// window's first position lies (linear sources).
struct XcRun
{
	int start, words, shift;
};

// KNOWN: 0 linear, 1 not, -1 either.
template <int KNOWN>
__host__ __device__ __forceinline__ XcRun run_of(const XcParams & p, const XcSource & src, int u)
{
	XcRun r;
	const int pos0 = u * p.pt * TC_PIX - p.halo;
	int lo, hi;
	if (KNOWN == 0 || (KNOWN < 0 && src.mode == XC_LINEAR))
	{
		lo = src.front + pos0;
		hi = lo + p.slots_plane;
	}
	else
	{
		// whole source rows, from that of the first position inside the batch to that of the last
		auto row_of = [&](int pos)
		{
			const int img = fdiv(pos, p.d_img);
			const int y = fdiv(pos - img * (int)p.d_img.d, p.d_pitch);
			return img * (src.h + 1) + ((src.scale == 2) ? 2 * y : (src.scale == 1) ? y : y >> 1);
		};
		// (a unit that begins in the padding behind the last image needs no row; it copies the last one)
		const int a = min(row_of(max(pos0, 0)), p.batch * (src.h + 1) - 1);
		const int b = row_of(min(pos0 + p.slots_plane - 1, p.total_pos - 1)) + ((src.scale != 0) ? 1 : 0);
		lo = src.front + a * src.pitch;
		hi = src.front + (b + 1) * src.pitch;
	}
	r.start = lo & ~3;
	r.shift = lo - r.start;
	r.words = min((hi + 3) & ~3, src.block_words) - r.start;
	return r;
}

// MODE 0: sign words only.  1: fp32 output (and its sign words).  2: fp32 sum with a shortcut operand (its sign words, and the
// layer's own output if asked for).  STREAM: the filters come through the stages instead of staying in shared memory.  SPLIT: the epilogue
// warps that would take different tiles share one, a part of its filters each.  KIND: where the window comes from and how many taps it has.
// PLAIN: whole words of filters, and (mode 2) the layer's own output is not asked for.
// (A kernel holds only the code it runs: layers wait for their instructions as well.  With the table's code in every kernel darknet53 took
// 349 us at batch 1, 337 without, 326 with 1x1 layers apart and 317 without what partial words of filters and a sum's own tensor need;
// tiny-yolo at batch 256 1342 and 1279.  Nine taps stay a parameter: known to the compiler they cost 16 -> 32 on 208x208 217 us, 199 so.)
enum { XC_ROWS = 0, XC_POINTS = 1, XC_TABLE = 2 };          // 3x3 and 1x1 of stride 1 from a run of words; any layer through the table

template <int NF, int MODE, bool STREAM, bool SPLIT, int KIND, bool PLAIN>
__global__ void __launch_bounds__(XC_THREADS, 1)
xnor_conv_kernel(const __grid_constant__ XcParams p)
{
	constexpr int ACC = (XC_SF_COL / NF < XC_MAX_ACC) ? XC_SF_COL / NF : XC_MAX_ACC;
	constexpr bool TABLED = (KIND == XC_TABLE);
	constexpr int RUN = TABLED ? 1 : STREAM ? -1 : 0;            // (streamed filters: no difference but in the compiler's order, 211 / 201 us)
	const int taps = (KIND == XC_POINTS) ? 1 : p.taps;
	const int stride = TABLED ? p.stride : 1;
	constexpr int MAX_STEPS = (KIND == XC_POINTS) ? 4 : XC_MAX_KW / 2;          // instructions of a stage: 64 K bits each
	constexpr int CHUNKS = NF / 32;
	constexpr int SHARES = 4 / CHUNKS;                         // epilogue warps of a lane quarter that are at a chunk of 32 filters
	constexpr int COLS = SPLIT ? 32 / SHARES : 32;             // filters of a warp
	constexpr int TILE_STEP = SPLIT ? 1 : SHARES;
	extern __shared__ __align__(128) uint8_t xc_smem[];
	__shared__ uint64_t raw_full[XC_RAW_STAGES];
	__shared__ uint64_t raw_empty[XC_RAW_STAGES];
	__shared__ uint64_t op_full[XC_MAX_STAGES];
	__shared__ uint64_t op_empty[XC_MAX_STAGES];
	__shared__ uint64_t acc_full[ACC];
	__shared__ uint64_t acc_empty[ACC];
	__shared__ uint64_t drain_bar;
	__shared__ uint64_t ready_bar;                              // filters and scale factors are in place
	__shared__ uint32_t tmem_base_slot;
	__shared__ __align__(16) float s_thr[NF];                  // MODE 0: smallest accumulator whose output is > 0
	__shared__ __align__(16) float s_mean[NF];
	__shared__ __align__(16) float s_bias[NF];
	__shared__ int s_failed_storage;
	volatile int * s_failed = &s_failed_storage;

	const int tid = threadIdx.x;
	const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // uniform to the compiler as well
	const int lane = tid & 31;
	const uint32_t limit = p.spin_limit;
	const uint32_t a_base = smem_u32(xc_smem);
	// ring of pixel stages, then the filters (all of them, or a ring beside the pixel stages), the raw ring, the window tables
	const uint32_t b_base = a_base + (uint32_t)(p.ring * p.a_stage_bytes);
	const uint32_t raw_base = b_base + (uint32_t)((STREAM ? p.ring : p.stages_k) * p.b_stage_bytes);
	int * s_table = reinterpret_cast<int *>(xc_smem + (raw_base - a_base) + (size_t)XC_RAW_STAGES * p.raw_stage_bytes);
	const int fg = blockIdx.x % p.fgroups;
	const int f0 = fg * NF;
	const int unit0 = blockIdx.x / p.fgroups;
	const int unit_step = gridDim.x / p.fgroups;
	const int my_units = (p.units - unit0 + unit_step - 1) / unit_step;
	auto place = [&](int u) { return p.backwards ? p.units - 1 - u : u; };         // where in the batch this CTA's unit u lies
	// this filter group's words: [K word][128]
	const uint32_t * my_filters = p.weights + (size_t)(f0 >> 7) * p.kwords * 128 + (f0 & 127);

	// What runs in front of pdl_wait reads filters, means and biases only, which were written long before the previous kernel; behind a
	// kernel of the same forward it runs while that one finishes.  The roles part as soon as barriers and tensor memory exist: the first
	// bits are on their way while the epilogue warps, which have nothing to do yet, widen the filters (all in one prologue in front of the
	// copies a layer at batch 1 took about 2 us longer wherever its CTAs had to wait for SMs).
	if (warp == XC_COPY_WARP)
	{
		if (lane < XC_RAW_STAGES)
		{
			mbar_init(&raw_full[lane], 2);                        // the copies (with their bytes), and the window table
			mbar_init(&raw_empty[lane], XC_EXP_WARPS);
		}
		if (lane < XC_MAX_STAGES)
		{
			mbar_init(&op_full[lane], XC_EXP_WARPS);
			mbar_init(&op_empty[lane], 1);
		}
		if (lane < ACC)
		{
			mbar_init(&acc_full[lane], 1);
			mbar_init(&acc_empty[lane], 4 * CHUNKS * (SPLIT ? SHARES : 1));
		}
		if (lane == 31)
		{
			mbar_init(&drain_bar, 1);
			mbar_init(&ready_bar, XC_EPI_WARPS);
			s_failed_storage = 0;
		}
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == XC_MMA_WARP)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
				:: "r"(smem_u32(&tmem_base_slot)), "r"((uint32_t)XC_TMEM_COLS) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
	if (warp < XC_EPI_WARPS)
	{
		// ---- epilogue warps, first: what the tiles need besides the bits ---------------------------------------------------
		float mean = 0.0f, bias = -0.0f;                           // v + -0.0 is v
		if (tid < NF && f0 + tid < p.M)
		{
			mean = __ldg(p.mean_arr + f0 + tid);
			if (p.bias != nullptr) { bias = __ldg(p.bias + f0 + tid); }
		}
		if (warp < 4)
		{
			// the block scale factors, all 2^0
			const uint32_t taddr = tmem_base + (uint32_t)XC_SF_COL + ((uint32_t)(warp * 32) << 16);
			asm volatile(
				"tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
				:: "r"(taddr), "r"(0x7F7F7F7Fu) : "memory");
			asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
			asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
		}
		if (!STREAM)
		{
			// a warp takes 32 filters of every STEP-th K word, four loads in flight per thread (eight are more
			// code, which every launch fetches anew: darknet53 at batch 1 333 us, 329 with four)
			constexpr int STEP = XC_EPI_WARPS * 32 / NF;
			const int f = tid % NF;
			const int total = p.stages_k * p.kw_full;
			const int g_words = p.G * taps;
			for (int k0 = tid / NF; k0 < total; k0 += 4 * STEP)
			{
				uint32_t bits[4];
				int at[4];                                            // stage and word of the stage
				#pragma unroll
				for (int q = 0; q < 4; ++q)
				{
					bits[q] = 0;
					const int kk = k0 + q * STEP;
					const int st = fdiv(kk, p.d_kw);
					at[q] = kk - st * p.kw_full | (st << 8);
					const int k = st * g_words + (at[q] & 255);
					if (kk < total && (at[q] & 255) < g_words && k < p.kwords) { bits[q] = __ldg(my_filters + (size_t)k * 128 + f); }
				}
				#pragma unroll
				for (int q = 0; q < 4; ++q)
				{
					if (k0 + q * STEP < total) { put_filter<NF>(p, taps, b_base + (uint32_t)((at[q] >> 8) * p.b_stage_bytes), at[q] >> 8, at[q] & 255, f, bits[q]); }
				}
			}
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		}
		__syncwarp();
		if (lane == 0) { mbar_arrive(&ready_bar); }
		if (tid < NF)
		{
			s_mean[tid] = mean;
			s_bias[tid] = bias;
			if (MODE == 0)
			{
				// fl(fl(d * mean) + bias) grows with d, so its sign is one comparison with the smallest d that makes it positive
				auto positive = [&](int d) { return __fadd_rn(__fmul_rn((float)d, mean), bias) > 0.0f; };
				int lo = -p.K - 1, hi = p.K + 1;                     // positive(hi) assumed, positive(lo) assumed not
				while (hi - lo > 1)
				{
					const int mid = lo + ((hi - lo) >> 1);
					if (positive(mid)) { hi = mid; } else { lo = mid; }
				}
				s_thr[tid] = (f0 + tid < p.M) ? (float)hi : 3.0e38f;
			}
		}
		asm volatile("bar.sync 1, %0;" :: "n"(XC_EPI_WARPS * 32) : "memory");

		// ---- epilogue: a warp takes every fourth (tile, 32-filter chunk) of its lane quarter -----------------------------
		// Parameters in registers, whole groups of filters without per-filter checks: about 11 instructions a value with a shortcut.
		const int quarter = warp & 3;
		const int share = warp >> 2;
		// items of this warp: CHUNKS of 1, 2 or 4 divide the four shares, so the chunk is always the same
		const int chunk = share % CHUNKS;
		const int part = SPLIT ? share / CHUNKS : 0;
		const int fb = chunk * 32 + part * COLS;
		const FastDiv d_img = p.d_img, d_pitch = p.d_pitch;
		const int pitch = p.pitch, OH = p.OH, OW = p.OW, total_pos = p.total_pos, pt = p.pt, batch = p.batch;
		const size_t n_pix = (size_t)p.n_pix;
		const int left = p.M - f0 - fb;                          // filters of this chunk that exist
		const size_t img_elems = (size_t)p.M * n_pix;
		struct Item { bool ok; size_t elem; int pos; };          // this lane's position; element of its pixel in the chunk's first filter
		auto locate = [&](int pos)
		{
			Item it;
			const int img = fdiv(pos, d_img);
			const int r = pos - img * (int)d_img.d;
			const int y = fdiv(r, d_pitch);
			const int x = r - y * pitch;
			it.ok = (pos < total_pos && y < OH && x < OW && left > 0);
			it.pos = pos;
			// off the map: the address of a pixel beside it, so that loads need no condition
			it.elem = (MODE == 0) ? 0 : (size_t)min(img, batch - 1) * img_elems + (size_t)(f0 + fb) * n_pix + (size_t)(min(y, OH - 1) * OW + min(x, OW - 1));
			return it;
		};
		const float slope = p.leaky ? 0.1f : 1.0f;               // leaky(v) = max(v, 0.1 v), linear(v) = max(v, v)
		const uint64_t slope2 = pack2(slope, slope);
		// a * b is a * b + -0 with a zero that the compiler does not know: it joins a packed product and the sum behind it into one rounding
		const uint64_t minus_zero2 = pack2(p.minus_zero, p.minus_zero);
		const uint32_t step = (uint32_t)p.n_pix * 4u;            // bytes from one filter's plane to the next
		uint32_t * words = (MODE == 2) ? p.sc_signs : p.signs;
		if (words != nullptr) { words += (size_t)((f0 + fb) >> 5) * p.out_block_words + p.out_front; }
		float * const out = p.out;
		float * const sc_out = p.sc_out;
		const float * const sc_in = p.sc_in;
		const uint64_t policy = stream_policy(p.stream_values != 0), out_policy = stream_policy(p.stream_out != 0);
		const int my_tiles = my_units * pt;
		int tile = SPLIT ? 0 : share / CHUNKS;                   // tiles of this CTA, counted over its units
		int u = unit0, t = tile;                                 // ... as unit and tile of the unit
		while (t >= pt) { t -= pt; u += unit_step; }
		int a = tile % ACC;                                      // accumulator, and the parity of its phase
		uint32_t phase = 0;
		auto pos_of = [&]() { return (place(u) * pt + t) * TC_PIX + quarter * 32 + lane; };
		// The shortcut operand: a ring of four groups of eight filters, each asked for again, for the next item, as soon as it has
		// been used, so that a thread always has 24 to 32 loads in flight.
		float sc[MODE == 2 ? COLS : 1];
		auto load8 = [&](const Item & it, int h)
		{
			if constexpr (MODE == 2)
			{
				// No condition per value: a load behind one was waited for on the spot, four times the latency per 32 values.  Filters
				// that do not exist read the last one that does.
				const char * at = reinterpret_cast<const char *>(sc_in + it.elem);
				if (PLAIN || left >= COLS)
				{
					at += (size_t)step * (uint32_t)h;
					#pragma unroll
					for (int i = 0; i < 8; ++i) { sc[h + i] = ld_policy(reinterpret_cast<const float *>(at + (size_t)step * (uint32_t)i), policy); }
				}
				else
				{
					#pragma unroll
					for (int i = 0; i < 8; ++i) { sc[h + i] = ld_policy(reinterpret_cast<const float *>(at + (size_t)step * (uint32_t)min(h + i, left - 1)), policy); }
				}
			}
		};
		Item it = Item{false, 0, 0};
		if (tile < my_tiles) { it = locate(pos_of()); }
		// everything the previous kernel wrote, and everything it read and this one overwrites, from here on
		pdl_wait();
		if (tile < my_tiles)
		{
			if (left > 0)
			{
				#pragma unroll
				for (int h = 0; h < COLS; h += 8) { load8(it, h); }
			}
		}
		while (tile < my_tiles)
		{
			const uint32_t tacc = tmem_base + (uint32_t)(a * NF + fb) + ((uint32_t)(quarter * 32) << 16);
			const int a_now = a;
			if (!__all_sync(0xffffffffu, mbar_wait<32>(&acc_full[a], phase, s_failed, limit))) { break; }
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			tile += TILE_STEP;
			a += TILE_STEP;
			if (a >= ACC) { a -= ACC; phase ^= 1u; }
			t += TILE_STEP;
			while (t >= pt) { t -= pt; u += unit_step; }
			uint32_t word = 0;
			Item next = Item{false, 0, 0};
			if (MODE == 0)
			{
				uint32_t d[32];
				tmem_load<32>(tacc, d);
				if (tile < my_tiles) { next = locate(pos_of()); }
				tmem_wait<32>(d);
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) { mbar_arrive(&acc_empty[a_now]); }
				// bit j = (d >= threshold), gathered as sign bits of d - threshold from the last filter down
				#pragma unroll
				for (int j = 28; j >= 0; j -= 4)
				{
					const float4 th = *reinterpret_cast<const float4 *>(s_thr + fb + j);
					word = __funnelshift_l(__float_as_uint(__fsub_rn(__uint_as_float(d[j + 3]), th.w)), word, 1);
					word = __funnelshift_l(__float_as_uint(__fsub_rn(__uint_as_float(d[j + 2]), th.z)), word, 1);
					word = __funnelshift_l(__float_as_uint(__fsub_rn(__uint_as_float(d[j + 1]), th.y)), word, 1);
					word = __funnelshift_l(__float_as_uint(__fsub_rn(__uint_as_float(d[j + 0]), th.x)), word, 1);
				}
				word = ~word;
			}
			else
			{
				const bool more = (tile < my_tiles && left > 0);
				if (more) { next = locate(pos_of()); }
				char * const dst = reinterpret_cast<char *>(((MODE == 2) ? sc_out : out) + it.elem);
				char * const own = reinterpret_cast<char *>((MODE == 2 && out != nullptr) ? out + it.elem : nullptr);
				const bool store = it.ok && (MODE == 1 || sc_out != nullptr);       // else only the sum's signs are wanted
				constexpr int W = (COLS < 16) ? COLS : 16;
				#pragma unroll
				for (int h = 0; h < COLS; h += W)
				{
					uint32_t d[W];
					tmem_load<W>(tacc + (uint32_t)h, d);
					tmem_wait<W>(d);
					if (h + W == COLS)
					{
						asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
						__syncwarp();
						if (lane == 0) { mbar_arrive(&acc_empty[a_now]); }
					}
					#pragma unroll
					for (int u0 = 0; u0 < W; u0 += 8)
					{
						const int j0 = h + u0;
						uint64_t w[4];                           // eight values, in pairs
						#pragma unroll
						for (int i = 0; i < 4; i += 2)
						{
							const ulonglong2 m = *reinterpret_cast<const ulonglong2 *>(s_mean + fb + j0 + 2 * i);
							const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(s_bias + fb + j0 + 2 * i);
							const int at = u0 + 2 * i;
							w[i] = add2(fma2(pack2(__uint_as_float(d[at]), __uint_as_float(d[at + 1])), m.x, minus_zero2), b.x);
							w[i + 1] = add2(fma2(pack2(__uint_as_float(d[at + 2]), __uint_as_float(d[at + 3])), m.y, minus_zero2), b.y);
						}
						float v[8];
						#pragma unroll
						for (int i = 0; i < 4; ++i)
						{
							float lo, hi;
							unpack2(fma2(w[i], slope2, minus_zero2), lo, hi);
							unpack2(w[i], v[2 * i], v[2 * i + 1]);
							v[2 * i] = fmaxf(v[2 * i], lo);
							v[2 * i + 1] = fmaxf(v[2 * i + 1], hi);
						}
						if (MODE == 2)
						{
							if (!PLAIN && own != nullptr && it.ok)
							{
								#pragma unroll
								for (int i = 0; i < 8; ++i) { if (j0 + i < left) { st_policy(reinterpret_cast<float *>(own + (size_t)step * (uint32_t)(j0 + i)), v[i], out_policy); } }
							}
							#pragma unroll
							for (int i = 0; i < 8; ++i) { v[i] = __fadd_rn(sc[MODE == 2 ? j0 + i : 0], v[i]); }
							if (more) { load8(next, j0); }
						}
						if (store && (PLAIN || left >= COLS))
						{
							#pragma unroll
							for (int i = 0; i < 8; ++i) { st_policy(reinterpret_cast<float *>(dst + (size_t)step * (uint32_t)(j0 + i)), v[i], out_policy); }
						}
						else if (!PLAIN && store)
						{
							#pragma unroll
							for (int i = 0; i < 8; ++i) { if (j0 + i < left) { st_policy(reinterpret_cast<float *>(dst + (size_t)step * (uint32_t)(j0 + i)), v[i], out_policy); } }
						}
						if (words != nullptr)
						{
							// v > 0 is the sign bit of 0 - v (zeros of either sign give +0), shifted in from below and turned round at the end
							#pragma unroll
							for (int i = 0; i < 8; ++i) { word = __funnelshift_l(__float_as_uint(__fsub_rn(0.0f, v[i])), word, 1); }
						}
					}
				}
				word = __brev(word) >> (32 - COLS);
			}
			if (words != nullptr && it.ok)
			{
				if constexpr (COLS == 32) { words[it.pos] = word; }
				else if constexpr (COLS == 16) { reinterpret_cast<uint16_t *>(words + it.pos)[part] = (uint16_t)word; }
				else { reinterpret_cast<uint8_t *>(words + it.pos)[part] = (uint8_t)word; }
			}
			it = next;
		}
	}
	else if (warp < XC_COPY_WARP)
	{
		// ---- expanders: raw words -> 16 bytes of e2m1 each ------------------------------------------------------------------
		// Everything the loops need lives in registers: a parameter read again per word (they are re-read behind every asm with a
		// memory clobber, and the source's through a dynamic index) cost 800 cycles per word and warp.
		const int ew = warp - XC_EPI_WARPS;
		const int et = ew * 32 + lane;
		const int slots_plane = p.slots_plane, G = p.G, nb = p.nb, stages_k = p.stages_k, ring = p.ring, units = p.units;
		const int table_len = p.n_src * slots_plane;
		const int blocks0 = p.src[0].blocks;
		const int mode = p.src[0].mode;                          // OR4 and SINGLE may meet in one layer (a route); both work as OR4
		constexpr bool tabled = TABLED;
		const uint32_t down0 = (p.src[0].mode == XC_SINGLE) ? 0u : (uint32_t)p.src[0].pitch * 4u;
		const uint32_t down1 = (p.src[1].mode == XC_SINGLE) ? 0u : (uint32_t)p.src[1].pitch * 4u;
		const uint32_t raw_bytes = (uint32_t)p.raw_words * 4u, raw_stage = (uint32_t)p.raw_stage_bytes;
		const uint32_t a_stage = (uint32_t)p.a_stage_bytes, b_stage = (uint32_t)p.b_stage_bytes;
		const uint32_t block_bytes = (uint32_t)p.slots * 16u, plane_bytes = (uint32_t)slots_plane * 16u;
		const bool withhold = (p.withhold != 0 && ew == 0);
		const int g_words = G * taps, kw_full = p.kw_full;
		const uint32_t last_mask = p.last_mask;
		// The words this thread widens lie at the same places in every stage (a last stage with fewer channel blocks is widened whole:
		// no filter reads what lies behind its blocks).  The loops over them are straight-line code: with the dealing done by
		// branches a word took 280 cycles.
		const int n_items = (G * slots_plane + XC_EXP_THREADS - 1) / XC_EXP_THREADS;
		const int full_items = (G * slots_plane) / XC_EXP_THREADS;                  // rounds in which every thread has a word
		const bool has_last = (et < G * slots_plane - full_items * XC_EXP_THREADS);
		uint32_t from[XC_ITEMS], to[XC_ITEMS];                   // byte offsets in the raw and in the operand stage; tabled: see below
		{
			int g = et / slots_plane, pos = et - g * slots_plane;
			#pragma unroll
			for (int j = 0; j < XC_ITEMS; ++j)
			{
				// tabled: window position and the block's first raw word
				from[j] = tabled ? (uint32_t)pos | ((uint32_t)(g * p.raw_words) << 16) : (uint32_t)g * raw_bytes + (uint32_t)pos * 4u;
				to[j] = (uint32_t)g * block_bytes + (uint32_t)pos * 16u;
				pos += XC_EXP_THREADS;
				while (pos >= slots_plane && g < G) { pos -= slots_plane; ++g; }
			}
		}
		uint32_t k = 0;                                          // stages passed
		int es = 0, rs = 0;
		uint32_t es_phase = 1, rs_phase = 0;                     // es_phase: parity of the wait for an emptied stage
		bool ok = true;
		int n_unit = 0;
		for (int u = unit0; u < units && ok; u += unit_step, ++n_unit)
		{
			const uint32_t table_addr = smem_u32(s_table + (n_unit % XC_TABLES) * table_len);
			const uint32_t shift0 = TABLED ? 0u : (uint32_t)run_of<RUN>(p, p.src[0], place(u)).shift * 4u;
			const uint32_t shift1 = (TABLED || p.n_src == 1) ? 0u : (uint32_t)run_of<RUN>(p, p.src[1], place(u)).shift * 4u;
			for (int st = 0; st < stages_k; ++st, ++k)
			{
				const int cb0 = st * G;
				ok = __all_sync(0xffffffffu, mbar_wait<0>(&raw_full[rs], rs_phase, s_failed, limit));
				if (!ok) { break; }
				if (k >= (uint32_t)ring)
				{
					// the MMAs that read this stage's previous contents have completed
					ok = __all_sync(0xffffffffu, mbar_wait<32>(&op_empty[es], es_phase, s_failed, limit));
					if (!ok) { break; }
				}
				const uint32_t a_dst = a_base + (uint32_t)es * a_stage;
				const uint32_t raw = raw_base + (uint32_t)rs * raw_stage;
				const bool second = (cb0 >= blocks0);            // the blocks of a stage come from one source
				// item j of this thread exists: always but for the last round
				auto has = [&](int j) { return j < full_items || (j == full_items && has_last); };
				if constexpr (!TABLED)
				{
					const uint32_t src = raw + (second ? shift1 : shift0);
					#pragma unroll
					for (int j0 = 0; j0 < XC_ITEMS; j0 += 4)
					{
						if (j0 >= n_items) { break; }
						uint32_t w[4];
						#pragma unroll
						for (int q = 0; q < 4; ++q) { if (has(j0 + q)) { w[q] = ld_shared_u32(src + from[j0 + q]); } }
						#pragma unroll
						for (int q = 0; q < 4; ++q) { if (has(j0 + q)) { st_shared_v4(a_dst + to[j0 + q], expand_fp4(w[q])); } }
					}
				}
				else
				{
					const uint32_t tab = table_addr + (second ? (uint32_t)slots_plane * 4u : 0u);
					const uint32_t down = second ? down1 : down0;
					const uint32_t right = (down != 0u) ? 4u : 0u;
					#pragma unroll
					for (int j0 = 0; j0 < XC_ITEMS; j0 += 2)
					{
						if (j0 >= n_items) { break; }
						uint32_t w0[2], w1[2], w2[2], w3[2], keep[2];
						int e[2];
						#pragma unroll
						for (int q = 0; q < 2; ++q) { if (has(j0 + q)) { e[q] = (int)ld_shared_u32(tab + (from[j0 + q] & 0xffffu) * 4u); } }
						#pragma unroll
						for (int q = 0; q < 2; ++q)
						{
							if (!has(j0 + q)) { continue; }
							// padding (-1) reads the run's first words and drops them
							const uint32_t at = raw + ((uint32_t)max(e[q], 0) + (from[j0 + q] >> 16)) * 4u;
							keep[q] = ~(uint32_t)(e[q] >> 31);
							w0[q] = ld_shared_u32(at);
							w1[q] = ld_shared_u32(at + right);
							w2[q] = ld_shared_u32(at + down);
							w3[q] = ld_shared_u32(at + down + right);
						}
						#pragma unroll
						for (int q = 0; q < 2; ++q)
						{
							if (!has(j0 + q)) { continue; }
							const uint32_t dst = a_dst + to[j0 + q];
							if (mode == XC_PLANES4)
							{
								st_shared_v4(dst, expand_fp4(w0[q] & keep[q]));
								st_shared_v4(dst + plane_bytes, expand_fp4(w1[q] & keep[q]));
								st_shared_v4(dst + 2u * plane_bytes, expand_fp4(w2[q] & keep[q]));
								st_shared_v4(dst + 3u * plane_bytes, expand_fp4(w3[q] & keep[q]));
							}
							else { st_shared_v4(dst, expand_fp4((w0[q] | w1[q] | w2[q] | w3[q]) & keep[q])); }
						}
					}
				}
				if constexpr (STREAM)
				{
					const uint32_t b_dst = a_base + (uint32_t)ring * a_stage + (uint32_t)es * b_stage + (uint32_t)et * 16u;
					const uint32_t fil = raw + (uint32_t)G * raw_bytes + (uint32_t)et * 4u;
					const int n = kw_full * NF;
					const bool plain = (cb0 + G < nb || (last_mask == 0xffffffffu && cb0 + G == nb)) && (g_words == kw_full);
					constexpr int FIL_ITEMS = XC_MAX_KW * NF / XC_EXP_THREADS;
					static_assert(FIL_ITEMS * XC_EXP_THREADS == XC_MAX_KW * NF && FIL_ITEMS % 6 == 0, "whole rounds of filter words");
					#pragma unroll
					for (int i0 = 0; i0 < FIL_ITEMS; i0 += 6)
					{
						uint32_t w[6];
						#pragma unroll
						for (int q = 0; q < 6; ++q)
						{
							if (et + (i0 + q) * XC_EXP_THREADS < n) { w[q] = ld_shared_u32(fil + (uint32_t)((i0 + q) * XC_EXP_THREADS * 4)); }
						}
						if (plain)
						{
							#pragma unroll
							for (int q = 0; q < 6; ++q)
							{
								if (et + (i0 + q) * XC_EXP_THREADS < n) { st_shared_v4(b_dst + (uint32_t)((i0 + q) * XC_EXP_THREADS * 16), expand_fp4(w[q])); }
							}
						}
						else
						{
							#pragma unroll
							for (int q = 0; q < 6; ++q)
							{
								const int i = et + (i0 + q) * XC_EXP_THREADS;
								if (i < n) { put_filter<NF>(p, taps, b_dst - (uint32_t)et * 16u, st, i / NF, i % NF, w[q]); }
							}
						}
					}
				}
				asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
				__syncwarp();
				if (lane == 0)
				{
					// every raw word has been stored widened by now, so its read has returned
					mbar_arrive(&raw_empty[rs]);
					if (!(withhold && k == 0)) { mbar_arrive(&op_full[es]); }
				}
				if (++rs == XC_RAW_STAGES) { rs = 0; rs_phase ^= 1u; }
				if (++es == ring) { es = 0; es_phase ^= 1u; }
			}
		}
	}
	else if (warp == XC_COPY_WARP)
	{
		// ---- bulk copies ------------------------------------------------------------------------------------------------------
		const bool leader = elect_one();
		int rs = 0;
		uint32_t rs_phase = 1, k = 0;
		bool ok = true;
		int n_unit = 0;
		// which word of the run each position of unit u's window is (-1: padding)
		auto fill_table = [&](int u, const XcRun & run0, const XcRun & run1)
		{
			int * tab = s_table + (n_unit % XC_TABLES) * (p.n_src * p.slots_plane);
			const int slots_plane = p.slots_plane, pitch = p.pitch, OH = p.OH, OW = p.OW, total_pos = p.total_pos;
			const FastDiv d_img = p.d_img, d_pitch = p.d_pitch;
			const int pos0 = place(u) * p.pt * TC_PIX - p.halo;
			for (int si = 0; si < p.n_src; ++si, tab += slots_plane)
			{
				const int down = 2 - p.src[si].scale, src_pitch = p.src[si].pitch, src_rows = p.src[si].h + 1;
				const int base = p.src[si].front - (si ? run1.start : run0.start);
				// a division per entry: two independent ones at a time beat four, and one chain of steps of 32 positions (104x104 83 / 115 us)
				#pragma unroll 2
				for (int s = lane; s < slots_plane; s += 32)
				{
					const int pos = pos0 + s;
					const int img = fdiv(pos, d_img);
					const int r = pos - img * (int)d_img.d;
					const int y = fdiv(r, d_pitch);
					const int x = r - y * pitch;
					const int sy = (2 * y) >> down, sx = (2 * x) >> down;
					tab[s] = (pos >= 0 && pos < total_pos && y < OH && x < OW) ? base + (img * src_rows + sy) * src_pitch + sx : -1;
				}
			}
		};
		for (int u = unit0; u < p.units && ok; u += unit_step, ++n_unit)
		{
			const XcRun run0 = run_of<RUN>(p, p.src[0], place(u));
			const XcRun run1 = (p.n_src > 1) ? run_of<RUN>(p, p.src[1], place(u)) : run0;
			if (n_unit == 0)
			{
				// the first table while the previous kernel finishes; then its stores -> this one's bulk copies
				if (TABLED) { fill_table(u, run0, run1); }
				pdl_wait();
				asm volatile("fence.proxy.async.global;" ::: "memory");
			}
			for (int st = 0; st < p.stages_k; ++st, ++k)
			{
				if (k >= XC_RAW_STAGES)
				{
					ok = __all_sync(0xffffffffu, mbar_wait<64>(&raw_empty[rs], rs_phase, s_failed, limit));
					if (!ok) { break; }
				}
				const int cb0 = st * p.G;
				const int blocks = min(p.G, p.nb - cb0);
				if (leader)
				{
					const uint32_t dst = raw_base + (uint32_t)(rs * p.raw_stage_bytes);
					const bool second = (cb0 >= p.src[0].blocks);          // the blocks of a stage come from one source
					const XcSource & src = p.src[second ? 1 : 0];
					const XcRun run = second ? run1 : run0;
					const uint32_t * words = src.words + (size_t)(second ? cb0 - p.src[0].blocks : cb0) * src.block_words + run.start;
					const int fil_words = STREAM ? min(p.G * taps, p.kwords - cb0 * taps) * NF : 0;
					mbar_expect_tx(&raw_full[rs], (uint32_t)(blocks * run.words + fil_words) * 4u);
					for (int g = 0; g < blocks; ++g)
					{
						bulk_load(dst + (uint32_t)(g * p.raw_words * 4), words + (size_t)g * src.block_words, (uint32_t)run.words * 4u, &raw_full[rs]);
					}
					if (STREAM)
					{
						bulk_load(dst + (uint32_t)(p.G * p.raw_words * 4), my_filters + (size_t)cb0 * taps * 128, (uint32_t)fil_words * 4u, &raw_full[rs]);
					}
					if (k == 0) { pdl_trigger(); }
				}
				// the copies are on their way meanwhile
				if (TABLED && st == 0 && n_unit > 0) { fill_table(u, run0, run1); }
				__syncwarp();
				if (lane == 0) { mbar_arrive(&raw_full[rs]); }
				if (++rs == XC_RAW_STAGES) { rs = 0; rs_phase ^= 1u; }
			}
		}
		// no copy of this CTA may still be in flight when it exits: the newest of every raw stage
		for (uint32_t s = 0; s < (uint32_t)XC_RAW_STAGES && s < k; ++s)
		{
			const uint32_t last = ((k - 1 - s) / XC_RAW_STAGES) * XC_RAW_STAGES + s;
			mbar_wait_plain(&raw_full[s], (last / XC_RAW_STAGES) & 1u, limit);
		}
		__syncwarp();
	}
	else
	{
		// ---- issuer: the warp stays converged, one elected lane issues ----------------------------------------------------------
		const bool leader = elect_one();
		const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(NF >> 3) << 17) | (1u << 23) | ((uint32_t)(TC_PIX >> 4) << 24);
		const uint32_t sfa = tmem_base + (uint32_t)XC_SF_COL;
		const uint32_t sfb = sfa + 8u;
		// the pixel operand's offsets, the same in every stage: lane k makes those of instruction k, start | LBO << 16
		uint32_t koff = 0;
		if (lane < p.kw_full / 2)
		{
			const int j0 = 2 * lane, j1 = 2 * lane + 1;
			const int g0 = block_of(j0, taps), g1 = block_of(j1, taps);
			const int o0 = g0 * p.slots + tap_offset(p, tap_of(j0 - g0 * taps, stride, taps), stride, taps);
			// the word past an odd number meets zero filters: any finite operand will do
			const int o1 = (g1 < p.G) ? g1 * p.slots + tap_offset(p, tap_of(j1 - g1 * taps, stride, taps), stride, taps) : o0;
			koff = (uint32_t)o0 | ((uint32_t)(o1 - o0) << 16);
		}
		uint32_t ko[MAX_STEPS];
		#pragma unroll
		for (int k = 0; k < MAX_STEPS; ++k) { ko[k] = __shfl_sync(0xffffffffu, koff, k); }
		int es = 0;
		uint32_t es_phase = 0;
		int a_unit = 0, used = 0;                                // accumulator of the unit's first tile; tiles started so far, up to ACC
		uint32_t a_phase = 1;                                    // parity of the wait for an emptied accumulator, for a_unit
		// filters and scale factors
		bool ok = __all_sync(0xffffffffu, mbar_wait<0>(&ready_bar, 0, s_failed, limit));
		for (int u = unit0; u < p.units && ok; u += unit_step)
		{
			for (int st = 0; st < p.stages_k && ok; ++st)
			{
				ok = __all_sync(0xffffffffu, mbar_wait<0>(&op_full[es], es_phase, s_failed, limit));
				if (!ok) { break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const int blocks = min(p.G, p.nb - st * p.G);
				const int steps = (blocks * taps + 1) / 2;
				uint32_t at = (a_base + (uint32_t)(es * p.a_stage_bytes)) >> 4;
				const uint32_t b16 = ((b_base + (uint32_t)((STREAM ? es : st) * p.b_stage_bytes)) >> 4) | ((uint32_t)NF << 16);
				int a = a_unit;
				uint32_t ap = a_phase;
				for (int t = 0; t < p.pt; ++t, at += TC_PIX)
				{
					if (st == 0)
					{
						if (used >= ACC)
						{
							ok = __all_sync(0xffffffffu, mbar_wait<32>(&acc_empty[a], ap, s_failed, limit));
							if (!ok) { break; }
							asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
						}
						else { ++used; }
					}
					const uint32_t acc = tmem_base + (uint32_t)(a * NF);
					#pragma unroll
					for (int k = 0; k < MAX_STEPS; ++k)
					{
						if (k >= steps) { break; }
						if (leader)
						{
							asm volatile(
								"{\n\t.reg .pred p;\n\t"
								"setp.ne.b32 p, %4, 0;\n\t"
								"tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
								:: "r"(acc), "l"(plane_desc(at + ko[k])), "l"(plane_desc(b16 + (uint32_t)(2 * k * NF))), "r"(idesc),
								   "r"((st | k) != 0 ? 1u : 0u), "r"(sfa), "r"(sfb) : "memory");
						}
					}
					if (st == p.stages_k - 1 && leader)
					{
						asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
								:: "r"(smem_u32(&acc_full[a])) : "memory");
					}
					if (++a == ACC) { a = 0; ap ^= 1u; }
				}
				if (!ok) { break; }
				if (leader)
				{
					asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
							:: "r"(smem_u32(&op_empty[es])) : "memory");
				}
				if (st == p.stages_k - 1) { a_unit = a; a_phase = ap; }
				if (++es == p.ring) { es = 0; es_phase ^= 1u; }
			}
		}
		if (!ok)
		{
			// leaving early: what was issued must have finished before the tensor memory is released
			if (leader)
			{
				asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
						:: "r"(smem_u32(&drain_bar)) : "memory");
			}
			mbar_wait_plain(&drain_bar, 0, limit);
		}
		__syncwarp();
	}

	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (*s_failed != 0 && tid == 0) { atomicExch(p.status, 1); }
	if (warp == XC_MMA_WARP)
	{
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"((uint32_t)XC_TMEM_COLS) : "memory");
	}
}

// ---- host side ----------------------------------------------------------------------------------------------------------

// Shapes the kernel's indices take: 3x3 / pad 1 or 1x1 / pad 0, stride 1 or 2.  Whether a window fits is the plan's to say.
static bool shape_taken(const xnor_b200_conv_desc & d)
{
	if (!((d.size == 3 && d.pad == 1) || (d.size == 1 && d.pad == 0)) || (d.stride != 1 && d.stride != 2)) { return false; }
	const long long blocks = (d.c + 31) / 32;
	if (blocks * d.size * d.size > 65535) { return false; }                      // grid rows of conv_words_weights_kernel
	if (blocks * (d.batch * (d.h + 1LL) * (d.w + 1) + d.w + 64) > 0x7fff0000LL) { return false; }      // words that sign_words counts
	// the source's grid is the larger one; a fused 2x2 max-pool doubles it again
	return (long long)d.batch * (2LL * d.h + 2) * (4LL * d.w + 16) < 0x7ffff000LL;
}

struct XcPlan
{
	int nf, pt, stream, g, ring, a_stage, b_stage, kw_full, stages_k, slots_plane, raw_words, raw_stage, grid;
	size_t smem;
	double cost;
};

// Words of the longest run a window of `slots` positions needs from a source.
static int raw_words_of(const XcParams & p, const XcSource & s, int slots)
{
	if (s.mode == XC_LINEAR) { return (int)round_up((size_t)slots, 4) + 8; }
	const long long rw = (slots - 1) / p.pitch + 2;              // rows of this grid that the window touches
	long long rows = rw;
	if (s.scale == 2) { rows = 2 * rw; }
	if (s.scale == 1) { rows = rw + 1 + (rw / p.rows + 1) * ((s.h > p.OH) ? s.h - p.OH : 0); }
	const long long words = rows * s.pitch + 12;
	return (words > (1 << 20)) ? (1 << 20) : (int)round_up((size_t)words, 4);
}

// Fills the sizes that follow from a choice of filters per group, tiles per unit and filter placement; false: does not fit.
static bool plan_sizes(const XcParams & p, int nf, int pt, int stream, XcPlan * out)
{
	XcPlan q = {};
	q.nf = nf; q.pt = pt; q.stream = stream;
	q.slots_plane = pt * TC_PIX + ((p.taps == 1) ? 0 : (p.stride == 1) ? 2 * p.halo : p.halo);
	const int slots = p.planes * q.slots_plane;
	const int most = XC_ITEMS * XC_EXP_THREADS / q.slots_plane;                  // channel blocks the expanders' registers hold
	if (most < 1) { return false; }
	q.g = (p.taps == 1) ? 8 : 2;
	q.g = (q.g > most) ? most : q.g;
	q.g = (q.g > p.nb) ? p.nb : q.g;
	while (p.n_src > 1 && p.src[0].blocks % q.g != 0) { --q.g; }                 // a stage's blocks come from one source
	q.stages_k = (p.nb + q.g - 1) / q.g;
	q.kw_full = (q.g * p.taps + 1) / 2 * 2;
	q.a_stage = q.g * slots * 16;
	q.b_stage = q.kw_full * nf * 16;
	if (q.g * slots >= 16384 || q.slots_plane > 0xffff) { return false; }                                  // operand offsets inside a stage: 14 bits
	for (int i = 0; i < p.n_src; ++i)
	{
		const int w = raw_words_of(p, p.src[i], q.slots_plane);
		if (w > q.raw_words) { q.raw_words = w; }
	}
	if (p.tabled && (long long)q.g * q.raw_words > 0xffff) { return false; }
	q.raw_stage = (q.g * q.raw_words + (stream ? q.kw_full * nf : 0)) * 4;
	const size_t table = p.tabled ? XC_TABLES * (size_t)p.n_src * q.slots_plane * sizeof(int) : 0;
	const size_t fixed = (size_t)XC_RAW_STAGES * q.raw_stage + table;
	for (q.ring = XC_MAX_STAGES; q.ring >= 2; --q.ring)
	{
		q.smem = (size_t)q.ring * q.a_stage + (size_t)(stream ? q.ring : q.stages_k) * q.b_stage + fixed;
		if (q.smem <= XC_SMEM_MAX) { break; }
	}
	if (q.ring < 2) { return false; }
	*out = q;
	return true;
}

// Estimated cycles of the busiest SM, fitted to clock traces of the roles.  Per tile: MMAs (73 / 56 / 47 cycles per 64 bits for 128 /
// 64 / 32 filters), epilogue (about 130 issue slots per sign word; 450 with fp32 values, some more than it takes since values go in pairs, which
// ranks the plans as well and is kept); per stage the
// expanders: 350 cycles of hand-overs and 110 per round of words (170 through the table with a pool, 350 for four parity planes).
// The slowest role sets the pace, the others take issue slots and shared-memory bandwidth from it.
static double plan_cost(const XcParams & p, const XcPlan & q, int mode, int sms)
{
	const int fgroups = (p.M + q.nf - 1) / q.nf;
	const int units = (int)((p.total_pos + (long long)q.pt * TC_PIX - 1) / (q.pt * TC_PIX));
	const int lanes = sms / fgroups;                                             // CTAs per filter group
	if (lanes < 1) { return 1e30; }
	const double waves = (double)((units + lanes - 1) / lanes);
	const double steps = 0.5 * q.kw_full * q.stages_k;
	const double mma = q.pt * steps * ((q.nf >= 128) ? 73.0 : (q.nf == 64) ? 56.0 : 47.0);
	const double epi = q.pt * (q.nf / 32) * (mode == 0 ? 130.0 : 450.0);
	const double round = (p.src[0].mode == XC_LINEAR) ? 110.0 : (p.src[0].mode == XC_PLANES4) ? 350.0 : 170.0;
	const double rounds = (double)((q.g * q.slots_plane + XC_EXP_THREADS - 1) / XC_EXP_THREADS);
	const double exp = q.stages_k * (350.0 + rounds * round + (q.stream ? 110.0 * (q.kw_full * q.nf / XC_EXP_THREADS) : 0.0));
	const double busiest = (mma > epi) ? ((mma > exp) ? mma : exp) : ((epi > exp) ? epi : exp);
	const double fill = q.stream ? 0.0 : (double)q.kw_full * q.nf * q.stages_k * (14.0 / 32.0) / 4.0;
	return 4000.0 + fill + (exp + mma) / q.stages_k + epi + waves * (0.75 * busiest + 0.25 * (mma + epi + exp) + 150.0);
}

static void fill_params(const xnor_b200_conv_desc & d, XcParams & p, int pitch)
{
	p.OH = conv_out_dim(d.h, d.size, d.stride, d.pad);
	p.OW = conv_out_dim(d.w, d.size, d.stride, d.pad);
	p.minus_zero = -0.0f;
	p.batch = d.batch;
	p.n_pix = p.OH * p.OW;
	p.M = d.n; p.K = d.c * d.size * d.size;
	p.stride = d.stride; p.taps = d.size * d.size;
	p.leaky = (d.activation == XNOR_B200_LEAKY) ? 1 : 0;
	p.nb = (d.c + 31) / 32;
	p.kwords = p.nb * p.taps;
	p.last_mask = (d.c % 32 == 0) ? 0xffffffffu : (1u << (d.c % 32)) - 1u;
	p.planes = (d.size == 3 && d.stride == 2) ? 4 : 1;
	p.pitch = (pitch > 0) ? pitch : p.OW + 1; p.rows = p.OH + 1;
	p.total_pos = d.batch * p.rows * p.pitch;
	p.halo = (d.size == 3) ? p.pitch + 1 : 0;
	p.d_img = make_div((uint32_t)(p.rows * p.pitch));
	p.d_pitch = make_div((uint32_t)p.pitch);
	p.out_front = grid_front(p.pitch);
	p.out_block_words = grid_block_words(d.batch, p.OH, p.pitch);
}

template <int NF, int MODE, bool STREAM, bool SPLIT>
static int launch_conv(XcParams & p, const XcPlan & q, cudaStream_t stream)
{
	auto kernel = p.tabled ? xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_TABLE, true>
			: (p.taps == 1) ? xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_POINTS, true> : xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_ROWS, true>;
	if constexpr (MODE != 0)
	{
		if (p.M % 32 != 0 || (MODE == 2 && p.out != nullptr))
		{
			kernel = p.tabled ? xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_TABLE, false>
					: (p.taps == 1) ? xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_POINTS, false> : xnor_conv_kernel<NF, MODE, STREAM, SPLIT, XC_ROWS, false>;
		}
	}
	int rc = ensure_dynamic_smem((const void *)kernel, q.smem);
	if (rc != XNOR_B200_OK) { return rc; }
	return launch_behind(kernel, (unsigned)q.grid, XC_THREADS, q.smem, stream, p);
}

static XcPlan best_plan(const XcParams & p, int mode)
{
	XcPlan best = {};
	best.cost = 1e30;
	const int sms = sm_count();
	for (int nf = 32; nf <= 128; nf *= 2)
	{
		for (int pt = 1; pt <= 4; pt *= 2)
		{
			for (int st = 0; st <= 1; ++st)
			{
				// filters are streamed in groups of 128 for one or two tiles; three accumulators of 128 filters fit, seven of 64
				if (st ? (nf != 128 || pt > 2) : (nf == 128 && pt > 1)) { continue; }
				XcPlan q;
				if (!plan_sizes(p, nf, pt, st, &q)) { continue; }
				q.cost = plan_cost(p, q, mode, sms);
				if (q.cost < best.cost) { best = q; }
			}
		}
	}
	return best;
}

static int apply_plan(XcParams & p, int mode, XcPlan & best)
{
	best = best_plan(p, mode);
	if (best.cost >= 1e30) { return XNOR_B200_ERR_TOO_LARGE; }
	p.pt = best.pt;
	p.G = best.g; p.stages_k = best.stages_k; p.ring = best.ring; p.kw_full = best.kw_full;
	p.d_kw = make_div((uint32_t)best.kw_full);
	p.a_stage_bytes = best.a_stage; p.b_stage_bytes = best.b_stage;
	p.raw_words = best.raw_words; p.raw_stage_bytes = best.raw_stage;
	p.slots_plane = best.slots_plane;
	p.slots = p.planes * p.slots_plane;
	p.units = (int)((p.total_pos + (long long)p.pt * TC_PIX - 1) / (p.pt * TC_PIX));
	p.fgroups = (p.M + best.nf - 1) / best.nf;
	const int lanes = sm_count() / p.fgroups;
	best.grid = p.fgroups * ((p.units < lanes) ? p.units : lanes);
	return XNOR_B200_OK;
}

template <int MODE>
static int launch_mode(XcParams & p, cudaStream_t stream)
{
	XcPlan best;
	int rc = apply_plan(p, MODE, best);
	if (rc != XNOR_B200_OK) { return rc; }
	TcParams common = {};
	rc = tc_fill_launch_fields(common);
	if (rc != XNOR_B200_OK) { return rc; }
	p.status = common.status; p.spin_limit = common.spin_limit; p.withhold = common.withhold;
	if (best.stream) { return launch_conv<128, MODE, true, false>(p, best, stream); }
	if (best.nf == 128) { return launch_conv<128, MODE, false, false>(p, best, stream); }
	if constexpr (MODE != 0)
	{
		// Fewer tiles a CTA than epilogue warps of a lane quarter that would take one each: at batch 1 a quarter or half of the warps did
		// all of a sum with its shortcut, 2 us of a layer's 7 (darknet53 at batch 1: 382 us, 360 with the filters shared).
		const int tiles = (p.units * p.fgroups + best.grid - 1) / best.grid * p.pt;
		if (tiles < 128 / best.nf) { return (best.nf == 64) ? launch_conv<64, MODE, false, true>(p, best, stream) : launch_conv<32, MODE, false, true>(p, best, stream); }
	}
	if (best.nf == 64) { return launch_conv<64, MODE, false, false>(p, best, stream); }
	return launch_conv<32, MODE, false, false>(p, best, stream);
}

// [filter][K in the layout of xnor_b200_binary_align_weights] -> [filters / 128][channel block * taps + tap, in the order the stages
// walk them][128 filters]
__global__ void conv_words_weights_kernel(const uint32_t * __restrict__ in, uint32_t * __restrict__ out, int n, int C, int taps, int stride, int lda_words)
{
	const int f = blockIdx.x * 128 + threadIdx.x;
	const int kw = blockIdx.y;
	const int cb = kw / taps;
	const int t = tap_of(kw - cb * taps, stride, taps);
	uint32_t v = 0;
	if (f < n)
	{
		const uint32_t * row = in + (size_t)f * lda_words;
		if (C % 32 == 0) { v = row[cb * taps + t]; }
		else
		{
			for (int b = 0; b < 32 && cb * 32 + b < C; ++b)
			{
				const int k = (cb * 32 + b) * taps + t;
				v |= ((row[k >> 5] >> (k & 31)) & 1u) << b;
			}
		}
	}
	out[((size_t)blockIdx.x * gridDim.y + kw) * 128 + threadIdx.x] = v;
}

}  // namespace xnor

using namespace xnor;

extern "C" size_t xnor_b200_grid_block_words(int batch, int h, int pitch)
{
	if (batch <= 0 || h <= 0 || pitch <= 1 || (long long)batch * (h + 1) * pitch > 0x7ffff000LL) { return 0; }
	return (size_t)grid_block_words(batch, h, pitch);
}

extern "C" int xnor_b200_grid_front(int pitch) { return (pitch > 1) ? grid_front(pitch) : 0; }

extern "C" size_t xnor_b200_conv_words_weights_bytes(const xnor_b200_conv_desc * desc)
{
	if (desc == nullptr || validate_desc(desc) != XNOR_B200_OK || !shape_taken(*desc)) { return 0; }
	alignas(16) static const uint32_t any[4] = {};
	xnor_b200_words_io io = {};
	io.n_sources = 1;
	io.sources[0].words = any;
	io.sources[0].blocks = (desc->c + 31) / 32;
	io.sources[0].h = desc->h; io.sources[0].w = desc->w;
	io.output = (float *)any;
	if (xnor_b200_conv_words_plan(desc, &io, nullptr) != XNOR_B200_OK) { return 0; }
	XcParams p = {};
	fill_params(*desc, p, 0);
	return (size_t)p.kwords * round_up((size_t)p.M, 128) * 4;
}

extern "C" int xnor_b200_conv_words_weights(const xnor_b200_conv_desc * desc, const uint8_t * align_bit_weights, uint32_t * conv_weights, void * stream)
{
	if (desc == nullptr || align_bit_weights == nullptr || conv_weights == nullptr) { return XNOR_B200_ERR_NULL; }
	const int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	if (!shape_taken(*desc)) { return XNOR_B200_ERR_INVALID; }
	if (((uintptr_t)align_bit_weights & 3u) != 0 || ((uintptr_t)conv_weights & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
	const int taps = desc->size * desc->size;
	const int kwords = (desc->c + 31) / 32 * taps;
	conv_words_weights_kernel<<<dim3((unsigned)((desc->n + 127) / 128), (unsigned)kwords, 1), 128, 0, (cudaStream_t)stream>>>(
			(const uint32_t *)align_bit_weights, conv_weights, desc->n, desc->c, taps, desc->stride, aligned_lda(taps * desc->c) / 32);
	return check_launch();
}

// Checks the call and fills everything that does not depend on the plan; *mode: what the epilogue writes.
static int conv_words_params(const xnor_b200_conv_desc * desc, const xnor_b200_words_io * io, XcParams & p, int * mode)
{
	if (desc == nullptr || io == nullptr) { return XNOR_B200_ERR_NULL; }
	int rc = validate_desc(desc);
	if (rc != XNOR_B200_OK) { return rc; }
	if (!shape_taken(*desc) || io->n_sources < 1 || io->n_sources > 2) { return XNOR_B200_ERR_INVALID; }
	// rows of the position grid are at most about twice as long as they have to be
	if (io->pitch < 0 || (io->pitch > 0 && (io->pitch <= conv_out_dim(desc->w, desc->size, desc->stride, desc->pad) || io->pitch > 2 * desc->w + 8))) { return XNOR_B200_ERR_INVALID; }
	fill_params(*desc, p, io->pitch);
	int blocks = 0;
	p.n_src = io->n_sources;
	for (int i = 0; i < io->n_sources; ++i)
	{
		const xnor_b200_words_source & s = io->sources[i];
		if (s.words == nullptr) { return XNOR_B200_ERR_NULL; }
		if (((uintptr_t)s.words & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
		if (s.blocks <= 0 || s.h <= 0 || s.w <= 0) { return XNOR_B200_ERR_INVALID; }
		if ((s.upsample != 0 && s.upsample != 1 && s.upsample != 2) || s.pool_stride < 0 || s.pool_stride > 2 || s.pool_pad < 0 || s.pool_pad > 1) { return XNOR_B200_ERR_INVALID; }
		const bool pooled = (s.pool_stride != 0), up = (s.upsample == 2);
		// a pool or an upsample is read through by stride-1 layers only
		if ((pooled && up) || ((pooled || up) && desc->stride != 1)) { return XNOR_B200_ERR_INVALID; }
		int h = s.h, w = s.w;
		if (pooled)
		{
			h = (h + s.pool_pad - 2) / s.pool_stride + 1;
			w = (w + s.pool_pad - 2) / s.pool_stride + 1;
		}
		if (up) { h *= 2; w *= 2; }
		if (h != desc->h || w != desc->w) { return XNOR_B200_ERR_INVALID; }
		XcSource & t = p.src[i];
		t.words = s.words; t.blocks = s.blocks; t.h = s.h; t.w = s.w;
		t.pitch = (s.pitch > 0) ? s.pitch : s.w + 1;
		if (t.pitch <= s.w || t.pitch > 2 * s.w + 8) { return XNOR_B200_ERR_INVALID; }
		t.front = grid_front(t.pitch);
		t.block_words = grid_block_words(desc->batch, s.h, t.pitch);
		t.mode = pooled ? XC_OR4 : (up || (desc->stride == 2 && p.taps == 1)) ? XC_SINGLE : (desc->stride == 2) ? XC_PLANES4
				: (t.pitch == p.pitch) ? XC_LINEAR : XC_SINGLE;
		t.scale = up ? 0 : pooled ? s.pool_stride : desc->stride;
		p.tabled |= (t.mode != XC_LINEAR) ? 1 : 0;
		blocks += s.blocks;
	}
	// one source through the table: both
	for (int i = 0; i < p.n_src; ++i) { if (p.tabled && p.src[i].mode == XC_LINEAR) { p.src[i].mode = XC_SINGLE; } }
	if (blocks != p.nb || (io->n_sources == 2 && desc->c % 32 != 0)) { return XNOR_B200_ERR_INVALID; }
	if (io->n_sources == 1) { p.src[1] = p.src[0]; }
	const bool sum = (io->shortcut_out != nullptr || io->shortcut_signs != nullptr);
	if (sum != (io->shortcut_in != nullptr)) { return XNOR_B200_ERR_NULL; }
	if (io->output == nullptr && io->output_signs == nullptr && !sum) { return XNOR_B200_ERR_NULL; }
	if (sum && io->output_signs != nullptr) { return XNOR_B200_ERR_INVALID; }
	if ((io->output_signs != nullptr || io->shortcut_signs != nullptr) && desc->n % 32 != 0) { return XNOR_B200_ERR_INVALID; }
	p.out = io->output; p.signs = io->output_signs;
	p.sc_in = io->shortcut_in; p.sc_out = io->shortcut_out; p.sc_signs = io->shortcut_signs;
	p.stream_values = ((long long)desc->batch * p.M * p.n_pix * 4 > XC_STREAM_BYTES) ? 1 : 0;
	// Layers of a network that write fp32 walk the batch in turn from either end: the next one then begins with what this one wrote last,
	// which the L2 still has (darknet53 at batch 64, sums of 50 to 820 MB: 3467 -> 3256 us; kept in the L2 alone 3375, in turn alone 3431).
	p.stream_out = (p.stream_values && g_walk == WALK_ALONE) ? 1 : 0;
	p.backwards = (p.stream_values && g_walk == WALK_BACKWARDS) ? 1 : 0;
	*mode = sum ? 2 : (io->output != nullptr) ? 1 : 0;
	return XNOR_B200_OK;
}

extern "C" int xnor_b200_conv_words(const xnor_b200_conv_desc * desc, const xnor_b200_words_io * io, const uint32_t * conv_weights,
		const float * mean_arr, const float * biases, void * stream)
{
	XcParams p = {};
	int mode = 0;
	const int rc = conv_words_params(desc, io, p, &mode);
	if (rc != XNOR_B200_OK) { return rc; }
	if (conv_weights == nullptr || mean_arr == nullptr) { return XNOR_B200_ERR_NULL; }
	if (((uintptr_t)conv_weights & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
	p.weights = conv_weights; p.mean_arr = mean_arr; p.bias = biases;
	cudaStream_t s = (cudaStream_t)stream;
	if (mode == 2) { return launch_mode<2>(p, s); }
	return (mode == 1) ? launch_mode<1>(p, s) : launch_mode<0>(p, s);
}

extern "C" int xnor_b200_conv_words_plan(const xnor_b200_conv_desc * desc, const xnor_b200_words_io * io, xnor_b200_words_plan * plan)
{
	XcParams p = {};
	int mode = 0;
	int rc = conv_words_params(desc, io, p, &mode);
	if (rc != XNOR_B200_OK) { return rc; }
	XcPlan best;
	rc = apply_plan(p, mode, best);
	if (rc != XNOR_B200_OK || plan == nullptr) { return rc; }
	*plan = {best.nf, best.pt, p.units, best.grid, best.ring, best.stream, best.smem, 0x7fffffff, 0, best.raw_words, best.cost};
	for (int u = 0; u < p.units; ++u)
	{
		for (int i = 0; i < p.n_src; ++i)
		{
			const int words = run_of<-1>(p, p.src[i], u).words;
			plan->run_words_min = min(plan->run_words_min, words);
			plan->run_words_max = max(plan->run_words_max, words);
		}
	}
	return XNOR_B200_OK;
}
