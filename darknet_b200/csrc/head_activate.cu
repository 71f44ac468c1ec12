// Activation steps of the [yolo] and [region] heads that close the xnor networks, one kernel each.
//
// forward_yolo_layer_gpu (src-lib/yolo_layer.cpp:1439-1489) applies the logistic function to the x, y entries and
// to the objectness + class entries of every anchor (two activate_array_ongpu launches per anchor and image) and
// leaves w, h raw.  The tensor is [batch][anchors][4 + 1 + classes][h*w]; one pass reads and writes it once.
// logistic(x) = 1 / (1 + expf(-x)), the form of src-lib/activation_kernels.cu (logistic_activate_kernel).
#include "xnor_common.cuh"

namespace xnor
{

__global__ void __launch_bounds__(256)
yolo_activate_kernel(const float * __restrict__ in, float * __restrict__ out, size_t total, int entries, int hw)
{
	for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (size_t)gridDim.x * 256)
	{
		const int e = (int)((i / hw) % entries);
		float v = in[i];
		if (e != 2 && e != 3) { v = 1.0f / (1.0f + expf(-v)); }
		out[i] = v;
	}
}

// [region] head (src-lib/region_layer.cpp:494-537): per image, anchor and cell the logistic function on x, y and the
// objectness entry, w and h raw, and -- with softmax=1 -- a softmax over the class entries (max subtracted, temperature
// 1: softmax_cpu in src-lib/blas.cpp).  The tensor is [batch][anchors][coords + 1 + classes][h*w].
//
// region_group_kernel: one anchor of one image per block, its entries side by side in shared memory.  Bound by memory: planes of
// 13x13 cells start on no boundary, so reading them plane by plane takes a third more sectors and leaves partly written ones; the
// whole group is one run that is read and written once, in order.  The classes of a cell are dealt to as many threads as there are (three of
// 512 for 13x13): a thread per cell walked 80 classes three times, and the SM waited for it (256 images of 5 anchors: 66 us, 55 now, 23 by
// memory).
constexpr int RG_THREADS = 512;
constexpr size_t RG_MAX_BYTES = 100 * 1024;              // two blocks on an SM

__global__ void __launch_bounds__(RG_THREADS)
region_group_kernel(const float * __restrict__ in, float * __restrict__ out, int coords, int classes, int hw)
{
	extern __shared__ float s_group[];
	__shared__ float s_part[RG_THREADS];
	const int total = (coords + 1 + classes) * hw;
	const size_t base = (size_t)blockIdx.x * total;
	#pragma unroll 8
	for (int i = threadIdx.x; i < total; i += RG_THREADS) { s_group[i] = in[base + i]; }
	__syncthreads();
	for (int i = threadIdx.x; i < 3 * hw; i += RG_THREADS)
	{
		const int e = i / hw;
		float * at = s_group + (e == 2 ? coords : e) * hw + (i - e * hw);
		*at = 1.0f / (1.0f + expf(-*at));
	}
	float * cls = s_group + (coords + 1) * hw;
	const int parts = max(1, min(min(RG_THREADS / hw, 8), classes)), per = (classes + parts - 1) / parts;
	for (int i0 = 0; i0 < hw * parts; i0 += RG_THREADS)           // (once, but for maps of more cells than threads, whose cells have one part)
	{
		const int i = i0 + threadIdx.x;
		const bool on = i < hw * parts;
		const int part = on ? i / hw : 0, cell = on ? i - part * hw : 0;
		const int first = part * per, end = on ? min(classes, first + per) : 0;
		float top = -INFINITY, sum = 0.0f;
		#pragma unroll 8
		for (int c = first; c < end; ++c) { top = fmaxf(top, cls[c * hw + cell]); }
		if (parts > 1)
		{
			s_part[threadIdx.x] = top;
			__syncthreads();
			for (int q = 0; q < parts; ++q) { top = fmaxf(top, s_part[q * hw + cell]); }
			__syncthreads();
		}
		#pragma unroll 4
		for (int c = first; c < end; ++c)
		{
			const float v = expf(cls[c * hw + cell] - top);
			cls[c * hw + cell] = v;
			sum += v;
		}
		if (parts > 1)
		{
			s_part[threadIdx.x] = sum;
			__syncthreads();
			sum = 0.0f;
			for (int q = 0; q < parts; ++q) { sum += s_part[q * hw + cell]; }
			__syncthreads();
		}
		#pragma unroll 4
		for (int c = first; c < end; ++c) { cls[c * hw + cell] = cls[c * hw + cell] / sum; }
	}
	__syncthreads();
	#pragma unroll 8
	for (int i = threadIdx.x; i < total; i += RG_THREADS) { out[base + i] = s_group[i]; }
}

// Without a softmax, and groups that do not fit: a thread owns one (image, anchor, cell), so every access of a warp is 32
// consecutive cells of one entry plane; the class scores are read three times, from the L1 / L2.
__global__ void __launch_bounds__(256)
region_activate_kernel(const float * __restrict__ in, float * __restrict__ out, size_t cells, int coords, int classes, int softmax, int hw)
{
	const int entries = coords + 1 + classes;
	for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < cells; i += (size_t)gridDim.x * 256)
	{
		const size_t group = i / hw;                          // image * anchors + anchor
		const size_t base = group * entries * hw + (i - group * hw);
		for (int e = 0; e <= coords; ++e)
		{
			float v = in[base + (size_t)e * hw];
			if (e < 2 || e == coords) { v = 1.0f / (1.0f + expf(-v)); }
			out[base + (size_t)e * hw] = v;
		}
		const float * cls = in + base + (size_t)(coords + 1) * hw;
		float * dst = out + base + (size_t)(coords + 1) * hw;
		if (!softmax)
		{
			for (int c = 0; c < classes; ++c) { dst[(size_t)c * hw] = cls[(size_t)c * hw]; }
			continue;
		}
		float largest = -INFINITY;
		for (int c = 0; c < classes; ++c) { largest = fmaxf(largest, cls[(size_t)c * hw]); }
		float sum = 0.0f;
		for (int c = 0; c < classes; ++c) { sum += expf(cls[(size_t)c * hw] - largest); }
		for (int c = 0; c < classes; ++c) { dst[(size_t)c * hw] = expf(cls[(size_t)c * hw] - largest) / sum; }
	}
}

}  // namespace xnor

using namespace xnor;

extern "C" int xnor_b200_region_activate(const float * input, float * output, int batch, int anchors, int coords, int classes,
		int softmax, int hw, void * stream)
{
	if (input == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || anchors <= 0 || coords < 2 || classes < 0 || hw <= 0 || input == output) { return XNOR_B200_ERR_INVALID; }
	const size_t cells = (size_t)batch * anchors * hw;
	const size_t group_bytes = (size_t)(coords + 1 + classes) * hw * sizeof(float);
	if (softmax && group_bytes <= RG_MAX_BYTES && (long long)batch * anchors <= 0x7fffffffLL)
	{
		const int rc = ensure_dynamic_smem((const void *)region_group_kernel, group_bytes);
		if (rc != XNOR_B200_OK) { return rc; }
		region_group_kernel<<<(unsigned)(batch * anchors), RG_THREADS, group_bytes, (cudaStream_t)stream>>>(input, output, coords, classes, hw);
		return check_launch();
	}
	const int grid = (int)min((cells + 255) / 256, (size_t)sm_count() * 8);
	region_activate_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(input, output, cells, coords, classes, softmax, hw);
	return check_launch();
}

extern "C" int xnor_b200_yolo_activate(const float * input, float * output, int batch, int anchors, int classes, int hw, void * stream)
{
	if (input == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || anchors <= 0 || classes < 0 || hw <= 0) { return XNOR_B200_ERR_INVALID; }
	const int entries = 4 + 1 + classes;
	const size_t total = (size_t)batch * anchors * entries * hw;
	const int grid = (int)min((total + 255) / 256, (size_t)sm_count() * 8);
	yolo_activate_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(input, output, total, entries, hw);
	return check_launch();
}
