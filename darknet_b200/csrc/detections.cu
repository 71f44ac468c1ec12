// Detection heads on the device: what Darknet does on the host after every forward of a [yolo] network.
//
//   xnor_b200_yolo_detections   get_yolo_detections + get_yolo_box + correct_yolo_boxes
//                               (src-lib/yolo_layer.cpp:1306-1348, :22-42, :1161-1222): every (cell, anchor) whose objectness
//                               exceeds the threshold becomes a detection -- box, objectness, objectness * class
//                               probability per class (0 where not above the threshold) -- stored in the reference's scan
//                               order (cells outer, anchors inner), the heads of a network one after the other;
//   xnor_b200_nms_sort          do_nms_sort (src-lib/box.cpp:951-1003) with box_iou (:310-344): per class, detections sorted by
//                               that class's probability, a kept detection zeroes the probability of every later one
//                               whose IoU with it exceeds the threshold;
//   xnor_b200_detection_rows    the surviving (detection, class) pairs as rows {x, y, w, h, objectness, class, probability}:
//                               the compact result a host copies back instead of the whole head tensors (Darknet pulls
//                               batch * outputs floats per head and walks them on the CPU).
//
//   xnor_b200_detect            the three in one launch.
//
// All run on the caller's stream, allocate nothing and synchronise nothing; counts live in device memory, so a head can
// be appended behind another without the host knowing how many detections the first one found.
#include "xnor_common.cuh"

#include <cooperative_groups.h>
#include <cuda.h>       // pointer attributes and contexts; the calls themselves are fetched by name
#include <cudaTypedefs.h>

#include <mutex>
#include <type_traits>

namespace xnor
{

namespace cg = cooperative_groups;

constexpr int DET_CLUSTER = 8;            // CTAs per image
constexpr int DET_THREADS = 512;
constexpr int DET_WARPS = DET_THREADS / 32;
constexpr int DET_ALL_WARPS = DET_CLUSTER * DET_WARPS;
constexpr int DET_STEP = 8;               // candidates a thread looks at between two scans
constexpr int DET_MAX_ANCHORS = 16;
constexpr int DET_MAX_HEADS = XNOR_B200_DETECT_HEADS;
constexpr int DET_LIST_BYTES = 8;         // per candidate of one class: score, storage index, rank order
constexpr int DET_SMEM_BUDGET = 192 * 1024;
constexpr int DET_SMEM_HALF = 104 * 1024; // two CTAs on an SM, as many as their registers allow,
constexpr int DET_SMEM_SHARED = 72 * 1024; // and the matrix of one of them: what it takes more is missing as cache
constexpr int DET_MATRIX_MAX = 768;       // detections whose overlaps are kept as a bit matrix (72 KB of shared memory)
constexpr int DET_MATRIX_WORDS = DET_MATRIX_MAX / 32;    // of a row, also of fewer (a length that is a parameter costs 3 to 5 % of a crowded list)
// Up to so many detections the matrix costs less than asking whether it is worth it; beyond, only where a class has more than DET_FEW candidates
constexpr int DET_MATRIX_SURE = 256;
constexpr int DET_FEW = 96;
constexpr int DET_RANK_MAX = 128;         // candidates of one class that a warp ranks by itself; more go to the whole CTA
constexpr int DET_WARP_MAX = 64;          // without the matrix: candidates of one class that a warp suppresses by itself
constexpr int DET_BLOCK = 128;            // ranks the CTA settles at a time

struct YoloHeadParams
{
	const float * head;          // [batch][n][4 + 1 + classes][lh * lw], activated (xnor_b200_yolo_activate)
	unsigned first;              // candidates of the heads before this one
	int lw, lh, n, new_coords;
	float anchor_w[DET_MAX_ANCHORS], anchor_h[DET_MAX_ANCHORS];      // biases[2 * mask[a]], biases[2 * mask[a] + 1]
};

struct DetectParams
{
	// decode (n_heads > 0)
	YoloHeadParams heads[DET_MAX_HEADS];
	int n_heads, append;
	int netw, neth, img_w, img_h, relative, letter;
	float thresh;
	// the lists
	float * boxes;               // [batch][max_dets][4]
	float * objectness;          // [batch][max_dets]
	float * probs;               // [batch][max_dets][classes]
	int * count;                 // [batch]: detections found so far (may exceed max_dets: the surplus is not stored)
	int max_dets, classes;
	// suppression
	int nms;
	float nms_thresh;
	int matrix_max;              // detections up to which the overlap matrix is used: at most min(max_dets, DET_MATRIX_MAX)
	int lists, matrix_lists;     // per-class candidate lists that fit a CTA's shared memory (at most one per warp), without and with the matrix
	// compaction (rows != nullptr)
	float * rows;                // [batch][max_rows][7]
	int * row_count;             // [batch]: pairs found (may exceed max_rows: the surplus is not stored)
	int max_rows;
};

// box_iou of src-lib/box.cpp:68-113, :310-344, operation for operation (no contraction into FMAs)
__device__ __forceinline__ float overlap_1d(float x1, float w1, float x2, float w2)
{
	// (half of a value is the same by a division and by a product)
	const float h1 = __fmul_rn(w1, 0.5f), h2 = __fmul_rn(w2, 0.5f);
	const float l1 = __fsub_rn(x1, h1), l2 = __fsub_rn(x2, h2);
	const float r1 = __fadd_rn(x1, h1), r2 = __fadd_rn(x2, h2);
	return __fsub_rn(fminf(r1, r2), fmaxf(l1, l2));
}

__device__ __forceinline__ float box_iou_dev(const float4 a, const float4 b)
{
	const float w = overlap_1d(a.x, a.z, b.x, b.z);
	if (w <= 0.0f) { return 0.0f; }
	const float h = overlap_1d(a.y, a.w, b.y, b.w);
	if (h <= 0.0f) { return 0.0f; }
	const float inter = __fmul_rn(w, h);
	if (inter == 0.0f) { return 0.0f; }
	const float uni = __fsub_rn(__fadd_rn(__fmul_rn(a.z, a.w), __fmul_rn(b.z, b.w)), inter);
	return __fdiv_rn(inter, uni);
}

// Whether box_iou_dev(a, b) > thresh: by a product where the two are farther apart than rounding can take them, else by that division.
__device__ __forceinline__ bool overlap_exceeds(const float4 a, const float4 b, float thresh)
{
	const float w = overlap_1d(a.x, a.z, b.x, b.z), h = overlap_1d(a.y, a.w, b.y, b.w);
	const float inter = __fmul_rn(w, h);
	if (w <= 0.0f || h <= 0.0f || inter == 0.0f) { return 0.0f > thresh; }
	const float uni = __fsub_rn(__fadd_rn(__fmul_rn(a.z, a.w), __fmul_rn(b.z, b.w)), inter);
	const float line = thresh * uni;
	// (a quotient near a threshold that is nearly subnormal rounds by more than the margin; thresholds and unions below zero meet as a line above it)
	if (thresh > 1e-30f && line > 1e-30f)
	{
		if (inter > line * 1.000001f) { return true; }
		if (inter < line * 0.999999f) { return false; }
	}
	return __fdiv_rn(inter, uni) > thresh;
}

// Rank of candidate c by score, highest first; equal scores keep their storage order.
__device__ __forceinline__ int score_rank(const float * s_score, int m, int c)
{
	const float s = s_score[c];
	int rank = 0;
	#pragma unroll 4
	for (int o = 0; o < m; ++o)
	{
		const float t = s_score[o];
		rank += (t > s || (t == s && o < c)) ? 1 : 0;
	}
	return rank;
}

// Lists that the matrix has no room for: greedy suppression of one class's m <= DET_WARP_MAX candidates by one warp.  The boxes go to
// shared memory in rank order, lane l decides about ranks l, l + 32, ...; its verdicts stay in a register, so a step is one shuffle, one
// broadcast read and the overlaps (reading order, score and box per step from memory took 600 cycles a candidate, this takes about 150).
__device__ __forceinline__ void suppress_warp(const DetectParams & p, int m, const float * s_score, const uint16_t * s_idx, uint16_t * s_order,
		float4 * s_box, const float4 * boxes, float * probs, int k)
{
	const int lane = threadIdx.x & 31;
	for (int c = lane; c < m; c += 32)
	{
		const int rank = score_rank(s_score, m, c);
		s_order[rank] = s_idx[c];
		s_box[rank] = __ldcg(boxes + s_idx[c]);
	}
	__syncwarp();
	unsigned dead = 0;                                            // bit j: rank lane + 32 j is suppressed
	for (int r = 0; r < m - 1; ++r)
	{
		const unsigned owner = __shfl_sync(0xffffffffu, dead, r & 31);
		if ((owner >> (r >> 5)) & 1u) { continue; }
		const float4 a = s_box[r];
		for (int j = r >> 5; j * 32 < m; ++j)
		{
			const int r2 = j * 32 + lane;
			if (r2 > r && r2 < m && box_iou_dev(a, s_box[r2]) > p.nms_thresh) { dead |= 1u << j; }
		}
	}
	for (int j = 0; j * 32 < m; ++j)
	{
		if ((dead >> j) & 1u) { probs[(size_t)s_order[j * 32 + lane] * p.classes + k] = 0.0f; }
	}
}

// The same for a crowded class of such a list, by the whole CTA, DET_BLOCK ranks at a time: every overlap inside the block at once as a
// bit matrix, one warp walks the matrix in rank order (a step costs a shuffle), then the block's survivors are held against all later
// ranks at once.  Step by step over the list, as a warp does it, 170 candidates took 45 us.
__device__ __forceinline__ void suppress_cta(const DetectParams & p, int m, float * s_score, const uint16_t * s_idx, uint16_t * s_order,
		const float4 * boxes, float * probs, int k)
{
	constexpr int WORDS = DET_BLOCK / 32;
	static_assert(DET_BLOCK * WORDS == DET_THREADS, "one thread per word of the block's matrix");
	__shared__ float4 s_box[DET_BLOCK];
	__shared__ uint32_t s_hits[DET_BLOCK][WORDS + 1];
	__shared__ uint32_t s_dead[WORDS];
	const int tid = threadIdx.x;
	for (int c = tid; c < m; c += DET_THREADS) { s_order[score_rank(s_score, m, c)] = (uint16_t)c; }
	__syncthreads();
	for (int r0 = 0; r0 < m; r0 += DET_BLOCK)
	{
		const int nb = min(DET_BLOCK, m - r0);
		if (tid < nb) { s_box[tid] = boxes[s_idx[s_order[r0 + tid]]]; }
		if (tid < WORDS) { s_dead[tid] = 0; }
		__syncthreads();
		const int r = tid / WORDS, w = tid % WORDS;
		uint32_t hits = 0;
		if (r < nb)
		{
			const float4 a = s_box[r];
			for (int j = max(w * 32, r + 1); j < min(nb, w * 32 + 32); ++j)
			{
				if (box_iou_dev(a, s_box[j]) > p.nms_thresh) { hits |= 1u << (j & 31); }
			}
			if (s_score[s_order[r0 + r]] <= 0.0f && w == 0) { atomicOr(&s_dead[r >> 5], 1u << (r & 31)); }     // an earlier block's verdict
		}
		s_hits[r][w] = hits;
		__syncthreads();
		if (tid < 32)
		{
			uint32_t dead = (tid < WORDS) ? s_dead[tid] : 0;
			for (int i = 0; i < nb; ++i)
			{
				const uint32_t word = __shfl_sync(0xffffffffu, dead, i >> 5);
				if (((word >> (i & 31)) & 1u) == 0 && tid < WORDS) { dead |= s_hits[i][tid]; }
			}
			if (tid < WORDS) { s_dead[tid] = dead; }
		}
		__syncthreads();
		if (tid < nb && ((s_dead[tid >> 5] >> (tid & 31)) & 1u)) { probs[(size_t)s_idx[s_order[r0 + tid]] * p.classes + k] = 0.0f; }
		for (int q = r0 + DET_BLOCK + tid; q < m; q += DET_THREADS)
		{
			const int c = s_order[q];
			if (s_score[c] <= 0.0f) { continue; }
			const float4 z = boxes[s_idx[c]];
			for (int i = 0; i < nb; ++i)
			{
				if (((s_dead[i >> 5] >> (i & 31)) & 1u) == 0 && box_iou_dev(s_box[i], z) > p.nms_thresh)
				{
					s_score[c] = -1.0f;
					break;
				}
			}
		}
		__syncthreads();
	}
}

// The detections of class k that a warp has to deal with: their scores and numbers, in storage order.  Returns how many.
__device__ __forceinline__ int gather_class(const DetectParams & p, int n, const float * probs, int k, float * s_score, uint16_t * s_idx)
{
	const int lane = threadIdx.x & 31;
	int m = 0;
	for (int d0 = 0; d0 < n; d0 += 8 * 32)
	{
		float s[8];
		#pragma unroll
		for (int j = 0; j < 8; ++j)
		{
			const int d = d0 + j * 32 + lane;
			s[j] = (d < n) ? __ldcg(probs + (size_t)d * p.classes + k) : 0.0f;
		}
		#pragma unroll
		for (int j = 0; j < 8; ++j)
		{
			const unsigned mask = __ballot_sync(0xffffffffu, s[j] > 0.0f);
			if (s[j] > 0.0f)
			{
				const int at = m + __popc(mask & ((1u << lane) - 1u));
				s_score[at] = s[j];
				s_idx[at] = (uint16_t)(d0 + j * 32 + lane);
			}
			m += __popc(mask);
		}
	}
	__syncwarp();
	return m;
}

// Greedy suppression of one class by one warp: its m detections in rank order, each looked up in the bits of those that a kept one has
// overlapped, and its own row of the overlap matrix added where it is kept.  Lane l holds the bits of detections 32 l ...; returns them.
// Overlaps are symmetric and a kept detection overlaps no kept one before it, so a row marks nothing that was kept.  The rows of four
// ranks are read ahead: a step is a shuffle and a few logical operations, about 40 cycles.
__device__ __forceinline__ uint32_t walk_class(int m, int words, const uint16_t * s_order, const uint32_t * s_over)
{
	const int lane = threadIdx.x & 31;
	uint32_t dead = 0;
	for (int r0 = 0; r0 < m; r0 += 4)
	{
		int d[4];
		uint32_t row[4];
		#pragma unroll
		for (int j = 0; j < 4; ++j)
		{
			d[j] = s_order[min(r0 + j, m - 1)];
			row[j] = (lane < words) ? s_over[d[j] * DET_MATRIX_WORDS + lane] : 0u;
		}
		#pragma unroll
		for (int j = 0; j < 4; ++j)
		{
			const uint32_t word = __shfl_sync(0xffffffffu, dead, d[j] >> 5);
			if (r0 + j < m && ((word >> (d[j] & 31)) & 1u) == 0) { dead |= row[j]; }
		}
	}
	return dead;
}

// The same for a class of at most DET_FEW candidates without the matrix: lane l holds the boxes of ranks l, l + 32, l + 64 and returns, as bits,
// which of them go; s_order has the detections in rank order.
constexpr int DET_FEW_LANE = DET_FEW / 32;

__device__ __forceinline__ uint32_t suppress_few(int m, const float * s_score, const uint16_t * s_idx, uint16_t * s_order, const float4 * s_box,
		float thresh)
{
	const int lane = threadIdx.x & 31;
	for (int c = lane; c < m; c += 32) { s_order[score_rank(s_score, m, c)] = s_idx[c]; }
	__syncwarp();
	float4 box[DET_FEW_LANE];
	#pragma unroll
	for (int j = 0; j < DET_FEW_LANE; ++j) { box[j] = s_box[s_order[min(j * 32 + lane, m - 1)]]; }
	uint32_t gone = 0;
	for (int r = 0; r < m - 1; ++r)
	{
		const uint32_t owner = __shfl_sync(0xffffffffu, gone, r & 31);
		if ((owner >> (r >> 5)) & 1u) { continue; }
		const float4 a = s_box[s_order[r]];
		#pragma unroll
		for (int j = 0; j < DET_FEW_LANE; ++j)
		{
			if (j * 32 >= m) { break; }
			const int r2 = j * 32 + lane;
			if (r2 > r && r2 < m && overlap_exceeds(a, box[j], thresh)) { gone |= 1u << j; }
		}
	}
	return gone;
}

// One cluster of DET_CLUSTER CTAs per image runs decode, suppression and compaction back to back: a frame has some tens of
// detections, so each step is a few microseconds of latency and the launches between them would cost as much again.  Work is
// dealt to warps (a warp per detection, per class, per detection again), the scans that fix the order are short enough for every
// CTA to do them all.  Values that another CTA of the cluster wrote are read past the L1 (__ldcg).
// Measured at 416x416, 80 classes, one image, in a CUDA graph, with the overlap matrix and without it (the candidates of each class held
// against one another on the way): 174 detections and 883 rows 20.5 and 26.7 us, 13 detections and 61 rows 12.4 and 16.5, none 8.3; 300 /
// 500 / 768 detections of five classes each 24.7 / 36.9 / 51.3 and 34.9 / 53.4 / 80.5, 174 of all 80 classes each 57 and 682.
__global__ void __cluster_dims__(DET_CLUSTER, 1, 1) __launch_bounds__(DET_THREADS)
detect_kernel(const __grid_constant__ DetectParams p)
{
	extern __shared__ __align__(16) uint8_t det_smem[];
	__shared__ __align__(16) int s_cnt[DET_STEP * DET_WARPS];
	__shared__ int s_m[DET_WARPS];
	__shared__ int s_most[2][DET_CLUSTER];                       // candidates of the largest class of each CTA's, in rounds of classes in turn
	cg::cluster_group cluster = cg::this_cluster();
	pdl_trigger();                                               // (rows_host_kernel; it reads nothing before this one has finished)
	const int rank = (int)cluster.block_rank();
	const int b = blockIdx.x / DET_CLUSTER;
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	const int all_warp = rank * DET_WARPS + warp;
	float * probs = p.probs + (size_t)b * p.max_dets * p.classes;
	const float4 * boxes = reinterpret_cast<const float4 *>(p.boxes) + (size_t)b * p.max_dets;
	int found = (p.n_heads == 0 || p.append) ? p.count[b] : 0;

	if (p.n_heads > 0)
	{
		unsigned * s_hit = reinterpret_cast<unsigned *>(det_smem);       // candidate number of each new detection, counted over the heads
		const int first = found;
		const int entries = 4 + 1 + p.classes;
		const YoloHeadParams & last = p.heads[p.n_heads - 1];
		const unsigned candidates = last.first + (unsigned)(last.lw * last.lh) * (unsigned)last.n;     // of all heads: below 2^32
		auto head_of = [&](unsigned c)
		{
			int hd = 0;
			while (hd + 1 < p.n_heads && c >= p.heads[hd + 1].first) { ++hd; }
			return hd;
		};
		for (unsigned long long q0 = 0; q0 < candidates; q0 += DET_STEP * DET_THREADS)
		{
			// reference order: heads, cells, anchors from outer to inner
			float obj[DET_STEP];
			#pragma unroll
			for (int j = 0; j < DET_STEP; ++j)
			{
				const unsigned long long c = q0 + j * DET_THREADS + threadIdx.x;
				obj[j] = -INFINITY;
				if (c < candidates)
				{
					const YoloHeadParams & h = p.heads[head_of((unsigned)c)];
					const unsigned q = (unsigned)c - h.first;
					const unsigned i = q / (unsigned)h.n, a = q - i * (unsigned)h.n;
					const size_t cells = (size_t)(h.lw * h.lh);
					obj[j] = __ldg(h.head + (((size_t)b * h.n + a) * entries + 4) * cells + i);
				}
			}
			unsigned hits[DET_STEP];
			#pragma unroll
			for (int j = 0; j < DET_STEP; ++j)
			{
				const bool in = q0 + j * DET_THREADS + threadIdx.x < candidates;
				hits[j] = __ballot_sync(0xffffffffu, in && obj[j] > p.thresh);
				if (lane == 0) { s_cnt[j * DET_WARPS + warp] = __popc(hits[j]); }
			}
			__syncthreads();
			// prefix sums over (j, warp): four counts a lane
			static_assert(DET_STEP * DET_WARPS == 128, "four counts per lane");
			const int4 c4 = *reinterpret_cast<const int4 *>(s_cnt + 4 * lane);
			int incl = c4.x + c4.y + c4.z + c4.w;
			const int own = incl;
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const int u = __shfl_up_sync(0xffffffffu, incl, o);
				if (lane >= o) { incl += u; }
			}
			const int part = warp & 3;                            // of a lane's four counts, those before this warp's
			const int before = incl - own + ((part > 0) ? c4.x : 0) + ((part > 1) ? c4.y : 0) + ((part > 2) ? c4.z : 0);
			#pragma unroll
			for (int j = 0; j < DET_STEP; ++j)
			{
				const int slot = found + __shfl_sync(0xffffffffu, before, j * (DET_WARPS / 4) + warp / 4) + __popc(hits[j] & ((1u << lane) - 1u));
				if (((hits[j] >> lane) & 1u) && slot < p.max_dets) { s_hit[slot - first] = (unsigned)(q0 + j * DET_THREADS + threadIdx.x); }
			}
			found += __shfl_sync(0xffffffffu, incl, 31);
			__syncthreads();
		}
		// correct_yolo_boxes: the network-to-image mapping, in double as the reference computes it
		int new_w = p.netw, new_h = p.neth;
		if (p.letter)
		{
			if (((float)p.netw / p.img_w) < ((float)p.neth / p.img_h)) { new_w = p.netw; new_h = (p.img_h * p.netw) / p.img_w; }
			else { new_h = p.neth; new_w = (p.img_w * p.neth) / p.img_h; }
		}
		const float deltaw = (float)(p.netw - new_w), deltah = (float)(p.neth - new_h);
		const float ratiow = (float)new_w / p.netw, ratioh = (float)new_h / p.neth;
		const bool whole = (new_w == p.netw && new_h == p.neth);  // the mapping takes 0 off and divides by 1
		const int stored = min(found, p.max_dets);
		// a warp per detection; its first three entries a lane are asked for while the one before is worked on
		constexpr int AHEAD = 3;
		struct Found { const float * e; int hd, i, a; float v[AHEAD]; };          // a detection's first entry, head, cell, anchor
		auto fetch = [&](int slot)
		{
			Found f = {};
			if (slot >= stored) { return f; }
			const unsigned hit = s_hit[slot - first];
			f.hd = head_of(hit);
			const YoloHeadParams & h = p.heads[f.hd];
			const unsigned q = hit - h.first, i = q / (unsigned)h.n, a = q - i * (unsigned)h.n;
			const size_t cells = (size_t)(h.lw * h.lh);
			f.i = (int)i;
			f.a = (int)a;
			f.e = h.head + ((size_t)b * h.n + a) * entries * cells + i;
			#pragma unroll
			for (int j = 0; j < AHEAD; ++j) { f.v[j] = (lane + 32 * j < entries) ? __ldg(f.e + (lane + 32 * j) * cells) : 0.0f; }
			return f;
		};
		Found next = fetch(first + all_warp);
		for (int slot = first + all_warp; slot < stored; slot += DET_ALL_WARPS)
		{
			const Found now = next;
			next = fetch(slot + DET_ALL_WARPS);
			const YoloHeadParams & h = p.heads[now.hd];
			const int i = now.i, a = now.a;
			const float tx = __shfl_sync(0xffffffffu, now.v[0], 0), ty = __shfl_sync(0xffffffffu, now.v[0], 1);
			const float tw = __shfl_sync(0xffffffffu, now.v[0], 2), th = __shfl_sync(0xffffffffu, now.v[0], 3);
			const float obj = __shfl_sync(0xffffffffu, now.v[0], 4);
			float * pr = probs + (size_t)slot * p.classes;
			#pragma unroll
			for (int j = 0; j < AHEAD; ++j)
			{
				const int at = lane + 32 * j;
				const float prob = __fmul_rn(obj, now.v[j]);
				if (at >= 5 && at < entries) { pr[at - 5] = (prob > p.thresh) ? prob : 0.0f; }
			}
			for (int j = lane + 32 * AHEAD; j < entries; j += 32)
			{
				const float prob = __fmul_rn(obj, __ldg(now.e + (size_t)j * (h.lw * h.lh)));
				pr[j - 5] = (prob > p.thresh) ? prob : 0.0f;
			}
			const int row = i / h.lw, col = i - row * h.lw;
			float bx = ((float)col + tx) / (float)h.lw;
			float by = ((float)row + ty) / (float)h.lh;
			float bw, bh;
			if (h.new_coords)
			{
				bw = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(tw, tw), 4.0f), h.anchor_w[a]), (float)p.netw);
				bh = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(th, th), 4.0f), h.anchor_h[a]), (float)p.neth);
			}
			else
			{
				bw = __fdiv_rn(__fmul_rn(expf(tw), h.anchor_w[a]), (float)p.netw);
				bh = __fdiv_rn(__fmul_rn(expf(th), h.anchor_h[a]), (float)p.neth);
			}
			if (!whole)
			{
				bx = (float)(((double)bx - (double)deltaw / 2. / p.netw) / (double)ratiow);
				by = (float)(((double)by - (double)deltah / 2. / p.neth) / (double)ratioh);
				bw = __fmul_rn(bw, __fdiv_rn(1.0f, ratiow));
				bh = __fmul_rn(bh, __fdiv_rn(1.0f, ratioh));
			}
			if (!p.relative)
			{
				bx = __fmul_rn(bx, (float)p.img_w); bw = __fmul_rn(bw, (float)p.img_w);
				by = __fmul_rn(by, (float)p.img_h); bh = __fmul_rn(bh, (float)p.img_h);
			}
			if (lane == 0)
			{
				const size_t d = (size_t)b * p.max_dets + slot;
				*reinterpret_cast<float4 *>(p.boxes + d * 4) = make_float4(bx, by, bw, bh);
				p.objectness[d] = obj;
			}
		}
		cluster.sync();                                          // the lists are complete; every CTA has read the old count
		if (rank == 0 && threadIdx.x == 0) { p.count[b] = found; }
	}
	else { cluster.sync(); }                                     // every CTA runs: its shared memory may be written to
	const int n = min(found, p.max_dets);

	// With the matrix the counts and first rows of the detections need no pass of their own: the suppression counts what it leaves.
	const bool matrix = (p.nms && n <= p.matrix_max);
	int * const s_rows = reinterpret_cast<int *>(det_smem);      // rows of a detection
	if (matrix)
	{
		float4 * s_box = reinterpret_cast<float4 *>(s_rows + ((p.matrix_max + 3) & ~3));
		uint32_t * s_over = reinterpret_cast<uint32_t *>(s_box + p.matrix_max);
		float * s_lists = reinterpret_cast<float *>(s_over + p.matrix_max * DET_MATRIX_WORDS);
		static_assert(DET_MATRIX_MAX <= 2 * DET_THREADS, "two boxes a thread");
		float4 box[2];                                           // (stored behind the first gathering, whose loads wait beside these)
		#pragma unroll
		for (int q = 0; q < 2; ++q)
		{
			const int d = threadIdx.x + q * DET_THREADS;
			if (d < n) { box[q] = __ldcg(boxes + d); }
		}
		float * s_score = s_lists + (size_t)warp * p.matrix_max * (DET_LIST_BYTES / 4);
		uint16_t * s_idx = reinterpret_cast<uint16_t *>(s_score + p.matrix_max);
		uint16_t * s_order = s_idx + p.matrix_max;
		const int words = (n + 31) / 32;
		bool formed = false;                                     // the matrix
		int round = 0;
		for (int k0 = 0; k0 < p.classes; k0 += DET_CLUSTER * p.matrix_lists, ++round)
		{
			// warps 0 .. lists-1 of every CTA: one class each
			const int k = k0 + warp * DET_CLUSTER + rank;
			const int m = (warp < p.matrix_lists && k < p.classes) ? gather_class(p, n, probs, k, s_score, s_idx) : 0;
			if (lane == 0) { s_m[warp] = m; }
			if (k0 == 0)
			{
				#pragma unroll
				for (int q = 0; q < 2; ++q)
				{
					const int d = threadIdx.x + q * DET_THREADS;
					if (d < n)
					{
						s_rows[d] = 0;
						s_box[d] = box[q];
					}
				}
			}
			__syncthreads();
			// All pairs cost what the list's square does, the pairs of a class its own (500 detections of one class each out of 80: 43 us, 23 without)
			bool crowded = formed || n <= DET_MATRIX_SURE;
			if (!crowded)
			{
				int most = 0;
				#pragma unroll
				for (int w = 0; w < DET_WARPS; ++w) { most = max(most, s_m[w]); }
				if (threadIdx.x < DET_CLUSTER) { *cluster.map_shared_rank(&s_most[round & 1][rank], threadIdx.x) = most; }
				cluster.sync();                                  // (and everybody's counts are zero)
				#pragma unroll
				for (int q = 0; q < DET_CLUSTER; ++q) { crowded |= s_most[round & 1][q] > DET_FEW; }
			}
			if (!crowded)
			{
				if (m > 0)
				{
					const uint32_t gone = suppress_few(m, s_score, s_idx, s_order, s_box, p.nms_thresh);
					for (int j = 0; j * 32 + lane < m; ++j)
					{
						const int d = s_order[j * 32 + lane];
						if ((gone >> j) & 1u) { probs[(size_t)d * p.classes + k] = 0.0f; }
						else
						{
							#pragma unroll
							for (int r = 0; r < DET_CLUSTER; ++r) { atomicAdd(cluster.map_shared_rank(s_rows + d, r), 1); }
						}
					}
				}
				__syncthreads();
				continue;
			}
			if (!formed)
			{
				#pragma unroll 2
				for (int i = all_warp; i < n * words; i += DET_ALL_WARPS)
				{
					const int r = i / words, w = i - r * words, c = w * 32 + lane;
					const bool over = (c < n && c != r) && overlap_exceeds(s_box[r], s_box[c], p.nms_thresh);
					const uint32_t bits = __ballot_sync(0xffffffffu, over);
					if (lane < DET_CLUSTER) { *cluster.map_shared_rank(s_over + r * DET_MATRIX_WORDS + w, lane) = bits; }
				}
			}
			if (m <= DET_RANK_MAX)
			{
				for (int c = lane; c < m; c += 32) { s_order[score_rank(s_score, m, c)] = s_idx[c]; }
			}
			for (int w = 0; w < p.matrix_lists; ++w)             // crowded classes: ranked by the whole CTA
			{
				const int mw = s_m[w];
				if (mw <= DET_RANK_MAX) { continue; }
				const float * score = s_lists + (size_t)w * p.matrix_max * (DET_LIST_BYTES / 4);
				const uint16_t * idx = reinterpret_cast<const uint16_t *>(score + p.matrix_max);
				uint16_t * order = const_cast<uint16_t *>(idx) + p.matrix_max;
				for (int c = threadIdx.x; c < mw; c += DET_THREADS) { order[score_rank(score, mw, c)] = idx[c]; }
			}
			if (!formed) { cluster.sync(); }                      // the matrix is complete, everybody's counts are zero
			else { __syncthreads(); }
			formed = true;
			if (m > 0)
			{
				const uint32_t dead = walk_class(m, words, s_order, s_over);
				for (int c0 = 0; c0 < m; c0 += 32)
				{
					const int d = s_idx[min(c0 + lane, m - 1)];
					const uint32_t word = __shfl_sync(0xffffffffu, dead, d >> 5);
					if (c0 + lane >= m) { continue; }
					if ((word >> (d & 31)) & 1u) { probs[(size_t)d * p.classes + k] = 0.0f; }
					else
					{
						#pragma unroll
						for (int r = 0; r < DET_CLUSTER; ++r) { atomicAdd(cluster.map_shared_rank(s_rows + d, r), 1); }
					}
				}
			}
			__syncthreads();
		}
		cluster.sync();
	}
	else if (p.nms)
	{
		const int warp_max = min(DET_WARP_MAX, p.max_dets);
		float4 * s_boxes = reinterpret_cast<float4 *>(det_smem + (((size_t)p.lists * p.max_dets * DET_LIST_BYTES + 15) & ~(size_t)15));
		for (int k0 = 0; k0 < p.classes; k0 += DET_CLUSTER * p.lists)
		{
			// warps 0 .. lists-1 of every CTA: one class each
			const int k = k0 + warp * DET_CLUSTER + rank;
			float * s_score = reinterpret_cast<float *>(det_smem + (size_t)warp * p.max_dets * DET_LIST_BYTES);
			uint16_t * s_idx = reinterpret_cast<uint16_t *>(s_score + p.max_dets);
			uint16_t * s_order = s_idx + p.max_dets;
			int m = 0;
			if (warp < p.lists && k < p.classes)
			{
				m = gather_class(p, n, probs, k, s_score, s_idx);
				if (m > 1 && m <= DET_WARP_MAX) { suppress_warp(p, m, s_score, s_idx, s_order, s_boxes + warp * warp_max, boxes, probs, k); }
			}
			if (lane == 0) { s_m[warp] = m; }
			__syncthreads();
			for (int w = 0; w < p.lists; ++w)                    // crowded classes: the whole CTA, one after the other
			{
				const int mw = s_m[w];
				if (mw <= DET_WARP_MAX) { continue; }
				float * score = reinterpret_cast<float *>(det_smem + (size_t)w * p.max_dets * DET_LIST_BYTES);
				uint16_t * idx = reinterpret_cast<uint16_t *>(score + p.max_dets);
				suppress_cta(p, mw, score, idx, idx + p.max_dets, boxes, probs, k0 + w * DET_CLUSTER + rank);
			}
			__syncthreads();
		}
		cluster.sync();
	}

	if (p.rows != nullptr)
	{
		// rows per detection, then the prefix sums every CTA needs for its own detections
		int * s_start = s_rows + (matrix ? p.matrix_max : p.max_dets);
		if (!matrix)
		{
			for (int d = all_warp; d < n; d += DET_ALL_WARPS)
			{
				int c = 0;
				for (int k = lane; k < p.classes; k += 32) { c += (__ldcg(probs + (size_t)d * p.classes + k) > 0.0f) ? 1 : 0; }
				c = __reduce_add_sync(0xffffffffu, c);
				if (lane < DET_CLUSTER) { cluster.map_shared_rank(s_rows, lane)[d] = c; }
			}
			cluster.sync();
		}
		int base = 0;
		for (int d0 = 0; d0 < n; d0 += DET_THREADS)
		{
			const int d = d0 + threadIdx.x;
			int c = 0;
			if (d < n) { c = s_rows[d]; }
			int incl = c;
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const int u = __shfl_up_sync(0xffffffffu, incl, o);
				if (lane >= o) { incl += u; }
			}
			if (lane == 31) { s_cnt[warp] = incl; }
			__syncthreads();
			int before = 0, all = 0;
			#pragma unroll
			for (int w = 0; w < DET_WARPS; ++w)
			{
				if (w < warp) { before += s_cnt[w]; }
				all += s_cnt[w];
			}
			if (d < n) { s_start[d] = base + before + incl - c; }
			base += all;
			__syncthreads();
		}
		for (int d = all_warp; d < n; d += DET_ALL_WARPS)
		{
			int slot = s_start[d];
			const size_t dd = (size_t)b * p.max_dets + d;
			const float4 box = __ldcg(boxes + d);
			const float obj = __ldcg(p.objectness + dd);
			for (int k0 = 0; k0 < p.classes; k0 += 4 * 32)
			{
				float s[4];
				#pragma unroll
				for (int j = 0; j < 4; ++j)
				{
					const int k = k0 + j * 32 + lane;
					s[j] = (k < p.classes) ? __ldcg(probs + (size_t)d * p.classes + k) : 0.0f;
				}
				#pragma unroll
				for (int j = 0; j < 4; ++j)
				{
					const unsigned mask = __ballot_sync(0xffffffffu, s[j] > 0.0f);
					const int at = slot + __popc(mask & ((1u << lane) - 1u));
					if (s[j] > 0.0f && at < p.max_rows)
					{
						float * r = p.rows + ((size_t)b * p.max_rows + at) * 7;
						r[0] = box.x; r[1] = box.y; r[2] = box.z; r[3] = box.w; r[4] = obj; r[5] = (float)(k0 + j * 32 + lane); r[6] = s[j];
					}
					slot += __popc(mask);
				}
			}
		}
		if (rank == 0 && threadIdx.x == 0) { p.row_count[b] = base; }
	}
}

// The counts and first rows of every image, stored straight into page-locked host memory; a CTA column per image.
// Its stores hold the SMs while they cross, and cross no faster than the copy engine's: us issued / alone / a 512 MB pass on another stream
// beside it, by the kernel and by two copies: 14 KB 6.2 / 13.9 / - and 6.9 / 15.3 / -, 112 KB 6.2 / 17.7 / 161 and 8.9 / 17.4 / 159, 224 KB
// 8.2 / 19.1 / 161 and 10.8 / 18.9 / 159, 448 KB 13.2 / 23.9 / 163 and 14.6 / 23.1 / 159, 3.5 MB 74 / 84 / 212 and 71 / 79 / 161.
constexpr size_t ROWS_KERNEL_BYTES = 256 << 10;

__global__ void __launch_bounds__(256)
rows_host_kernel(const float * __restrict__ rows, int max_rows, const int * __restrict__ row_count, int take, float * __restrict__ host_rows,
		int * __restrict__ host_count)
{
	pdl_wait();                                                  // launched while the kernel in front of it, detect_kernel as a rule, finishes
	const size_t b = blockIdx.y;
	const size_t floats = (size_t)take * 7;
	const float * from = rows + b * max_rows * 7;
	float * to = host_rows + b * floats;
	for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < floats; i += (size_t)gridDim.x * 256) { to[i] = __ldcg(from + i); }
	if (blockIdx.x == 0 && threadIdx.x == 0) { host_count[b] = __ldcg(row_count + b); }
}

struct DriverCalls
{
	PFN_cuPointerGetAttributes_v7000 attributes;
	PFN_cuStreamGetCtx_v9020 stream_context;
	PFN_cuCtxGetCurrent_v4000 context;
};

// nullptr: not to be had
static const DriverCalls * driver()
{
	static std::once_flag once;
	static DriverCalls calls = {};
	static bool all = false;
	std::call_once(once, []()
	{
		// each in the version of its type: the newest cuStreamGetCtx has another parameter
		auto find = [](const char * name, unsigned version, auto & fn)
		{
			void * sym = nullptr;
			cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
			if (cudaGetDriverEntryPointByVersion(name, &sym, version, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) { return false; }
			fn = (std::remove_reference_t<decltype(fn)>)sym;
			return true;
		};
		all = find("cuPointerGetAttributes", 7000, calls.attributes) && find("cuStreamGetCtx", 9020, calls.stream_context)
				&& find("cuCtxGetCurrent", 4000, calls.context);
	});
	return all ? &calls : nullptr;
}

// The address at which a kernel may write the given bytes of host memory; nullptr unless they lie in one page-locked allocation or
// registration, which the device may write to.  (Where first and last byte are says nothing: two registrations keep the distance of their
// host addresses, with memory between them that the device does not have.)
static void * device_view(void * host, size_t bytes)
{
	const DriverCalls * const calls = driver();
	CUpointer_attribute which[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
			CU_POINTER_ATTRIBUTE_RANGE_SIZE, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
	unsigned type = 0, access = 0;
	CUdeviceptr at = 0, start = 0;
	size_t size = 0;
	void * out[5] = {&type, &at, &start, &size, &access};
	if (calls == nullptr || calls->attributes(5, which, out, (CUdeviceptr)host) != CUDA_SUCCESS) { return nullptr; }        // (pageable memory: all zero)
	const CUdeviceptr first = (CUdeviceptr)host;
	const bool whole = type == CU_MEMORYTYPE_HOST && at != 0 && start <= first && first - start <= size && bytes <= size - (first - start);
	return (whole && access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE) ? (void *)at : nullptr;
}

// Whether the stream and what a kernel on it would read belong to the current device (copies take any)
static bool of_this_device(const float * rows, const int * row_count, cudaStream_t stream)
{
	// (the stream's context: asking for its device would end a capture)
	const DriverCalls * const calls = driver();
	int device = -1;
	CUcontext current = nullptr, streams = nullptr;
	if (calls == nullptr || cudaGetDevice(&device) != cudaSuccess || calls->context(&current) != CUDA_SUCCESS
			|| calls->stream_context((CUstream)stream, &streams) != CUDA_SUCCESS || streams != current) { return false; }
	for (const void * at : {(const void *)rows, (const void *)row_count})
	{
		CUpointer_attribute which[2] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL};
		unsigned type = 0;
		int owner = -1;
		void * out[2] = {&type, &owner};
		if (calls->attributes(2, which, out, (CUdeviceptr)at) != CUDA_SUCCESS || type != CU_MEMORYTYPE_DEVICE || owner != device) { return false; }
	}
	return true;
}

static int check_dets(const xnor_b200_detections * d, int batch)
{
	if (d == nullptr || d->boxes == nullptr || d->objectness == nullptr || d->probs == nullptr || d->count == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || d->classes <= 0 || d->max_dets <= 0) { return XNOR_B200_ERR_INVALID; }
	if (d->max_dets > XNOR_B200_MAX_DETECTIONS) { return XNOR_B200_ERR_TOO_LARGE; }
	if ((((uintptr_t)d->boxes) & 15u) != 0) { return XNOR_B200_ERR_ALIGNMENT; }
	return XNOR_B200_OK;
}

static int add_head(const xnor_b200_yolo_head & head, int classes, DetectParams & p)
{
	if (head.output == nullptr) { return XNOR_B200_ERR_NULL; }
	if (head.w <= 0 || head.h <= 0 || head.n <= 0 || head.n > DET_MAX_ANCHORS || head.classes != classes) { return XNOR_B200_ERR_INVALID; }
	const long long candidates = (long long)head.w * head.h * head.n;
	long long first = 0;
	for (int i = 0; i < p.n_heads; ++i) { first += (long long)p.heads[i].lw * p.heads[i].lh * p.heads[i].n; }
	if (candidates > 0x7fffffffLL || first + candidates > 0xffffffffLL) { return XNOR_B200_ERR_TOO_LARGE; }
	YoloHeadParams & h = p.heads[p.n_heads++];
	h.first = (unsigned)first;
	h.head = head.output;
	h.lw = head.w; h.lh = head.h; h.n = head.n; h.new_coords = head.new_coords;
	for (int a = 0; a < DET_MAX_ANCHORS; ++a)
	{
		h.anchor_w[a] = (a < head.n) ? head.anchors[2 * a] : 0.0f;
		h.anchor_h[a] = (a < head.n) ? head.anchors[2 * a + 1] : 0.0f;
	}
	return XNOR_B200_OK;
}

static int set_decode(DetectParams & p, int netw, int neth, int img_w, int img_h, float thresh, int relative, int letter, int append)
{
	if (netw <= 0 || neth <= 0 || img_w <= 0 || img_h <= 0) { return XNOR_B200_ERR_INVALID; }
	p.netw = netw; p.neth = neth; p.img_w = img_w; p.img_h = img_h;
	p.thresh = thresh; p.relative = relative; p.letter = letter; p.append = append;
	return XNOR_B200_OK;
}

static int set_rows(DetectParams & p, float * rows, int max_rows, int * row_count)
{
	if (rows == nullptr || row_count == nullptr) { return XNOR_B200_ERR_NULL; }
	if (max_rows <= 0) { return XNOR_B200_ERR_INVALID; }
	p.rows = rows; p.row_count = row_count; p.max_rows = max_rows;
	return XNOR_B200_OK;
}

static int launch_detect(DetectParams & p, const xnor_b200_detections * d, int batch, void * stream)
{
	if (batch > (p.nms ? 65535 : 0x7fffffff / DET_CLUSTER)) { return XNOR_B200_ERR_TOO_LARGE; }
	p.boxes = d->boxes; p.objectness = d->objectness; p.probs = d->probs; p.count = d->count;
	p.max_dets = d->max_dets; p.classes = d->classes;
	// shared memory: the hit list; then, with the overlap matrix, counts, boxes, the matrix and candidate lists (as many as the classes of a
	// CTA ask for), or without it candidate lists of max_dets (as many as the budget allows) and the boxes of a warp; then two ints per detection
	const int want = min(DET_WARPS, (p.classes + DET_CLUSTER - 1) / DET_CLUSTER);
	const int list_bytes = p.max_dets * DET_LIST_BYTES;
	const int box_bytes = min(DET_WARP_MAX, p.max_dets) * (int)sizeof(float4);
	p.lists = max(1, min(want, DET_SMEM_BUDGET / (list_bytes + box_bytes)));
	p.matrix_lists = want;
	size_t smem = (size_t)list_bytes;
	if (p.nms)
	{
		smem = round_up((size_t)p.lists * list_bytes, 16) + (size_t)p.lists * box_bytes;
		// The matrix takes what there is, but not the place of an SM's second CTA where the images are more than the SMs take at once and the
		// lists leave it (64 images, lists of 768, 13 / 100 / 174 found: 49 / 62 / 78 us with a matrix for all of them, 31 / 41 / 54 with what
		// half an SM has, 30 / 37 / 47 so; 33 / 39 / 49 before there was a matrix).
		// Lists beyond it pay where nearly every detection is of nearly every class: 500 of all 80 each 3.4 ms, 0.9 with a matrix for all
		const bool shared = (long long)batch * DET_CLUSTER > sm_count() && smem <= DET_SMEM_HALF;
		const size_t room = shared ? max(smem, (size_t)DET_SMEM_SHARED) : DET_SMEM_BUDGET;
		auto matrix_bytes = [&](int max)
		{
			return round_up((size_t)max, 4) * 4 + (size_t)max * (sizeof(float4) + DET_MATRIX_WORDS * 4 + (size_t)want * DET_LIST_BYTES);
		};
		p.matrix_max = min(p.max_dets, DET_MATRIX_MAX);
		while (matrix_bytes(p.matrix_max) > room) { p.matrix_max = (p.matrix_max - 1) & ~31; }
		if (p.matrix_max >= p.max_dets) { smem = (size_t)list_bytes; }             // no list goes without it
		smem = max(smem, matrix_bytes(p.matrix_max));
	}
	const int rc = ensure_dynamic_smem((const void *)detect_kernel, smem);
	if (rc != XNOR_B200_OK) { return rc; }
	detect_kernel<<<(unsigned)batch * DET_CLUSTER, DET_THREADS, smem, (cudaStream_t)stream>>>(p);
	return check_launch();
}

}  // namespace xnor

using namespace xnor;

extern "C" int xnor_b200_yolo_detections(const xnor_b200_yolo_head * head, int batch, int netw, int neth, int img_w, int img_h,
		float thresh, int relative, int letter, int append, const xnor_b200_detections * dets, void * stream)
{
	if (head == nullptr || head->output == nullptr) { return XNOR_B200_ERR_NULL; }
	int rc = check_dets(dets, batch);
	if (rc != XNOR_B200_OK) { return rc; }
	DetectParams p = {};
	rc = add_head(*head, dets->classes, p);
	if (rc != XNOR_B200_OK) { return rc; }
	rc = set_decode(p, netw, neth, img_w, img_h, thresh, relative, letter, append);
	return (rc != XNOR_B200_OK) ? rc : launch_detect(p, dets, batch, stream);
}

extern "C" int xnor_b200_nms_sort(const xnor_b200_detections * dets, int batch, float nms_thresh, void * stream)
{
	const int rc = check_dets(dets, batch);
	if (rc != XNOR_B200_OK) { return rc; }
	DetectParams p = {};
	p.nms = 1;
	p.nms_thresh = nms_thresh;
	return launch_detect(p, dets, batch, stream);
}

extern "C" int xnor_b200_detection_rows(const xnor_b200_detections * dets, int batch, float * rows, int max_rows, int * row_count, void * stream)
{
	int rc = check_dets(dets, batch);
	if (rc != XNOR_B200_OK) { return rc; }
	DetectParams p = {};
	rc = set_rows(p, rows, max_rows, row_count);
	return (rc != XNOR_B200_OK) ? rc : launch_detect(p, dets, batch, stream);
}

extern "C" int xnor_b200_detect(const xnor_b200_yolo_head * heads, int n_heads, int batch, int netw, int neth, int img_w, int img_h,
		float thresh, int relative, int letter, float nms_thresh, const xnor_b200_detections * dets,
		float * rows, int max_rows, int * row_count, void * stream)
{
	if (heads == nullptr) { return XNOR_B200_ERR_NULL; }
	int rc = check_dets(dets, batch);
	if (rc != XNOR_B200_OK) { return rc; }
	if (n_heads <= 0) { return XNOR_B200_ERR_INVALID; }
	if (n_heads > DET_MAX_HEADS) { return XNOR_B200_ERR_TOO_LARGE; }
	DetectParams p = {};
	for (int i = 0; i < n_heads; ++i)
	{
		rc = add_head(heads[i], dets->classes, p);
		if (rc != XNOR_B200_OK) { return rc; }
	}
	rc = set_decode(p, netw, neth, img_w, img_h, thresh, relative, letter, 0);
	if (rc != XNOR_B200_OK) { return rc; }
	rc = set_rows(p, rows, max_rows, row_count);
	if (rc != XNOR_B200_OK) { return rc; }
	p.nms = (nms_thresh > 0.0f) ? 1 : 0;
	p.nms_thresh = nms_thresh;
	return launch_detect(p, dets, batch, stream);
}

extern "C" int xnor_b200_rows_to_host(const float * rows, int max_rows, const int * row_count, int batch, int take, float * host_rows,
		int * host_count, void * stream)
{
	if (rows == nullptr || row_count == nullptr || host_rows == nullptr || host_count == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || take <= 0 || take > max_rows) { return XNOR_B200_ERR_INVALID; }
	const size_t bytes = (size_t)batch * take * 7 * sizeof(float);
	float * rows_at = nullptr;
	int * count_at = nullptr;
	if (bytes <= ROWS_KERNEL_BYTES && batch <= 65535 && of_this_device(rows, row_count, (cudaStream_t)stream))
	{
		rows_at = (float *)device_view(host_rows, bytes);
		count_at = (int *)device_view(host_count, (size_t)batch * sizeof(int));
	}
	if (rows_at != nullptr && count_at != nullptr && (((uintptr_t)rows_at | (uintptr_t)count_at) & 3u) == 0)
	{
		// one launch for two copies of 3 to 8 us each and the gap between them
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3((unsigned)((take * 7LL + 1023) / 1024), (unsigned)batch, 1);
		cfg.blockDim = dim3(256, 1, 1);
		cfg.stream = (cudaStream_t)stream;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[0].val.programmaticStreamSerializationAllowed = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
		const cudaError_t e = cudaLaunchKernelEx(&cfg, rows_host_kernel, rows, max_rows, row_count, take, rows_at, count_at);
		return (e == cudaSuccess) ? check_launch() : cuda_fail(e);
	}
	cudaError_t e = cudaMemcpyAsync(host_count, row_count, (size_t)batch * sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
	if (e != cudaSuccess) { return cuda_fail(e); }
	const size_t row = 7 * sizeof(float);
	e = cudaMemcpy2DAsync(host_rows, take * row, rows, max_rows * row, take * row, (size_t)batch, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
	return (e == cudaSuccess) ? XNOR_B200_OK : cuda_fail(e);
}
