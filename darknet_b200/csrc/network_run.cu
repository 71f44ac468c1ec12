// A network's forward as one call: the layers' launches, resolved once into an array of operations (xnor_b200_op), are issued back
// to back from native code.  The layer loop of forward_network_gpu (src-lib/network_kernels.cu:30-65) without its per-layer host work:
// walked from Python a layer costs about 20 us, more than its kernel at batch 1.
#include "xnor_common.cuh"

namespace xnor
{

thread_local bool g_behind_kernel = false;
thread_local int g_walk = WALK_ALONE;

// A pointer of an operation: an address, or (small values) the network's input or one of its heads.
static const void * resolve(const void * at, const void * input, void * const * heads, int n_heads)
{
	const uintptr_t v = (uintptr_t)at;
	if (v == XNOR_B200_OP_INPUT) { return input; }
	if (v >= XNOR_B200_OP_HEAD && v < XNOR_B200_OP_HEAD + (uintptr_t)n_heads) { return heads[v - XNOR_B200_OP_HEAD]; }
	return at;
}

// mean over each (image, channel) plane: avgpool_layer (src-lib/avgpool_layer.cpp:42-60); a warp per plane
__global__ void __launch_bounds__(256)
avgpool_kernel(const float * __restrict__ in, float * __restrict__ out, int planes, int hw)
{
	const int plane = blockIdx.x * 8 + (threadIdx.x >> 5);
	const int lane = threadIdx.x & 31;
	if (plane >= planes) { return; }
	const float * at = in + (size_t)plane * hw;
	float sum = 0.0f;
	for (int i = lane; i < hw; i += 32) { sum += __ldg(at + i); }
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); }
	if (lane == 0) { out[plane] = sum / (float)hw; }
}

// softmax over all values of each image (softmax_cpu, src-lib/blas.cpp, temperature 1); a CTA per image
__global__ void __launch_bounds__(256)
softmax_kernel(const float * __restrict__ in, float * __restrict__ out, int n)
{
	__shared__ float s_part[8];
	const float * at = in + (size_t)blockIdx.x * n;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	float top = -INFINITY;
	for (int i = threadIdx.x; i < n; i += 256) { top = fmaxf(top, __ldg(at + i)); }
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) { top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o)); }
	if (lane == 0) { s_part[warp] = top; }
	__syncthreads();
	#pragma unroll
	for (int w = 0; w < 8; ++w) { top = fmaxf(top, s_part[w]); }
	__syncthreads();
	float sum = 0.0f;
	for (int i = threadIdx.x; i < n; i += 256) { sum += expf(__ldg(at + i) - top); }
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); }
	if (lane == 0) { s_part[warp] = sum; }
	__syncthreads();
	sum = 0.0f;
	#pragma unroll
	for (int w = 0; w < 8; ++w) { sum += s_part[w]; }
	for (int i = threadIdx.x; i < n; i += 256) { out[(size_t)blockIdx.x * n + i] = expf(__ldg(at + i) - top) / sum; }
}

}  // namespace xnor

using namespace xnor;

extern "C" int xnor_b200_avgpool(const float * input, float * output, int planes, int hw, void * stream)
{
	if (input == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	if (planes <= 0 || hw <= 0) { return XNOR_B200_ERR_INVALID; }
	avgpool_kernel<<<(unsigned)((planes + 7) / 8), 256, 0, (cudaStream_t)stream>>>(input, output, planes, hw);
	return check_launch();
}

extern "C" int xnor_b200_softmax(const float * input, float * output, int batch, int n, void * stream)
{
	if (input == nullptr || output == nullptr) { return XNOR_B200_ERR_NULL; }
	if (batch <= 0 || n <= 0) { return XNOR_B200_ERR_INVALID; }
	softmax_kernel<<<(unsigned)batch, 256, 0, (cudaStream_t)stream>>>(input, output, n);
	return check_launch();
}

extern "C" int xnor_b200_run_ops(const xnor_b200_op * ops, int n_ops, const float * input, void * const * heads, int n_heads, void * stream,
		void * side_stream, void * fork_event, void * join_event)
{
	if (ops == nullptr || input == nullptr || (n_heads > 0 && heads == nullptr)) { return XNOR_B200_ERR_NULL; }
	void * at = stream;
	struct Reset { ~Reset() { g_behind_kernel = false; g_walk = WALK_ALONE; } } reset;
	int layers = 0;                                            // xnor convolutions that write fp32
	auto writes_fp32 = [](const xnor_b200_op & op) { return op.kind == XNOR_B200_OP_CONV_WORDS && (op.io.output != nullptr || op.io.shortcut_in != nullptr); };
	for (int i = 0; i < n_ops; ++i) { layers += writes_fp32(ops[i]) ? 1 : 0; }
	int walk = WALK_FORWARDS;
	// Behind a fork the caller's stream waits for the side stream before this call returns, whether or not all was issued: what the caller
	// queues next may read, or overwrite, what the side stream works on.
	bool forked = false;
	bool behind = false;                                       // the stream's last entry is a kernel of this call
	auto join = [&](int rc)
	{
		if (!forked) { return rc; }
		cudaError_t e = cudaEventRecord((cudaEvent_t)join_event, (cudaStream_t)side_stream);
		if (e == cudaSuccess) { e = cudaStreamWaitEvent((cudaStream_t)stream, (cudaEvent_t)join_event, 0); }
		return (rc == XNOR_B200_OK && e != cudaSuccess) ? cuda_fail(e) : rc;
	};
	for (int i = 0; i < n_ops; ++i)
	{
		const xnor_b200_op & op = ops[i];
		const float * in = (const float *)resolve(op.input, input, heads, n_heads);
		float * out = (float *)resolve(op.output, input, heads, n_heads);
		const xnor_b200_conv_desc & d = op.desc;
		int rc = XNOR_B200_OK;
		g_behind_kernel = behind;
		const bool was_behind = behind;
		behind = true;
		switch (op.kind)
		{
			case XNOR_B200_OP_CONV3: rc = xnor_b200_float_conv3_words(&d, op.arg, in, (const float *)op.weights, op.biases, (uint32_t *)out, op.pitch, at); break;
			case XNOR_B200_OP_SIGN_WORDS: rc = xnor_b200_sign_words(in, d.batch, d.c, d.h, d.w, op.pitch, (uint32_t *)out, at); break;
			case XNOR_B200_OP_CONV_WORDS:
				if (layers > 1 && writes_fp32(op))
				{
					g_walk = walk;
					walk = (walk == WALK_FORWARDS) ? WALK_BACKWARDS : WALK_FORWARDS;
				}
				rc = xnor_b200_conv_words(&d, &op.io, (const uint32_t *)op.weights, op.mean_arr, op.biases, at);
				g_walk = WALK_ALONE;
				break;
			case XNOR_B200_OP_FLOAT_MAP: rc = xnor_b200_float_conv_map_yolo(&d, in, (const float *)op.weights, op.biases, out, op.arg, at); break;
			case XNOR_B200_OP_FLOAT_TC: rc = xnor_b200_float_conv_tc(&d, in, (const float *)op.weights, op.biases, out, op.arg, at); break;
			case XNOR_B200_OP_YOLO: rc = xnor_b200_yolo_activate(in, out, d.batch, d.n, op.arg, d.h * d.w, at); break;
			case XNOR_B200_OP_REGION: rc = xnor_b200_region_activate(in, out, d.batch, d.n, op.pitch, op.arg, d.activation, d.h * d.w, at); break;
			case XNOR_B200_OP_AVGPOOL: rc = xnor_b200_avgpool(in, out, d.batch * d.c, d.h * d.w, at); break;
			case XNOR_B200_OP_SOFTMAX: rc = xnor_b200_softmax(in, out, d.batch, d.c * d.h * d.w, at); break;
			case XNOR_B200_OP_CONV:
				rc = xnor_b200_conv_forward(&d, in, (const uint8_t *)op.weights, op.mean_arr, op.biases, out, op.io.shortcut_in, op.io.shortcut_out,
						op.scratch, op.scratch_bytes, at);
				break;
			case XNOR_B200_OP_FILTERS:
			{
				behind = false;                                  // seldom made again, and the kernel that reads them does so before it waits
				cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
				if (op.arg == 0)
				{
					const cudaError_t e = cudaStreamIsCapturing((cudaStream_t)at, &capture);
					if (e != cudaSuccess) { return join(cuda_fail(e)); }
				}
				if (op.arg != 0 || capture != cudaStreamCaptureStatusNone) { rc = xnor_b200_conv_words_weights(&d, (const uint8_t *)op.weights, (uint32_t *)out, at); }
				break;
			}
			case XNOR_B200_OP_FORK:
			{
				// what follows runs on the side stream, behind everything issued so far
				if (side_stream == nullptr || fork_event == nullptr || join_event == nullptr) { return join(XNOR_B200_ERR_NULL); }
				cudaError_t e = cudaEventRecord((cudaEvent_t)fork_event, (cudaStream_t)stream);
				if (e == cudaSuccess) { e = cudaStreamWaitEvent((cudaStream_t)side_stream, (cudaEvent_t)fork_event, 0); }
				if (e != cudaSuccess) { return join(cuda_fail(e)); }
				at = side_stream;
				forked = true;
				behind = false;
				break;
			}
			case XNOR_B200_OP_BACK: at = stream; behind = false; break;
			case XNOR_B200_OP_MARK:
			{
				behind = was_behind && out == nullptr;
				if (out != nullptr)
				{
					const cudaError_t e = cudaEventRecord((cudaEvent_t)(void *)out, (cudaStream_t)at);
					if (e != cudaSuccess) { return join(cuda_fail(e)); }
				}
				break;
			}
			default: return join(XNOR_B200_ERR_INVALID);
		}
		if (rc != XNOR_B200_OK) { return join(rc); }
	}
	return join(XNOR_B200_OK);
}
