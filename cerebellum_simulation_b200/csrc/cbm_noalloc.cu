// PF->PC input sums with no device allocation.
//
// Some host programs cannot let a library allocate device memory when they
// call it: frameworks that own every device allocation through their own
// pool (a foreign cudaMalloc escapes their budget and fragments their
// arena), and real-time control loops that cannot absorb the latency of an
// allocation.
// For them this file computes the per-PC parallel-fibre input sums (the
// reference's updatePFPCOutGPU followed by sumInputsNew, in the same float
// order) from buffers the caller already holds, in one launch that keeps its
// partial sums in shared memory.
//
// Limits and behaviour:
//   - numPC x bs <= kMaxPartials, where bs is the reduction width the
//     reference picks for a row of numGR/numPC fibres (512 for rows of 2048
//     or more); larger networks are rejected with CBM_ERR_ARG.
//   - The first call on a device loads the kernel; make it before any stream
//     capture.
//   - A CUDA error already pending in the calling thread (from the
//     caller's own earlier launches) is reported as such and left pending;
//     nothing is launched then.
#include <algorithm>
#include <cstdint>
#include <string>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/cbm_b200.h"

namespace {

constexpr uint32_t kMaxPartials = CBM_NOALLOC_MAX_PARTIALS;
constexpr uint32_t kCols = 64;      // reduction columns a CTA takes
constexpr uint32_t kThreads = 512;  // at most

// callSumKernel's block size for a row (CBM_CORE_LIB_MGPU_DEV/src/cuda/kernels.cu:445-469)
uint32_t rowBlockSize(uint32_t rowLength)
{
	if (rowLength >= 2048) return 512;
	if (rowLength >= 512) return 128;
	if (rowLength >= 128) return 32;
	if (rowLength >= 32) return 8;
	return 2;
}

// V consecutive 32-bit words.
template <int V> struct Words { uint32_t x[V]; };
template <int V> __device__ __forceinline__ Words<V> loadWords(const uint32_t *p)
{
	Words<V> r;
	if constexpr (V == 4) {
		const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
		r.x[0] = q.x; r.x[1] = q.y; r.x[2] = q.z; r.x[3] = q.w;
	} else {
		r.x[0] = __ldg(p);
	}
	return r;
}

// The input sums of one PC a cluster.  Column j's partial is the running sum, from
// 0, of the pairs x[i] + x[i+bs] for i = j, j+2bs, ... of the PC's row,
// x = w * (apBuf & mask != 0); the sum is sumInputsNew's halving tree over the bs
// partials (strides bs/2 ... 1, kernels.cu:326-362).
// Memory bound (12 bytes a fibre), and only with enough loads in flight: a thread
// makes V neighbouring columns' terms of one pair row, so a CTA of 64 columns has
// 32 rows' loads (16 bytes each when the buffers are aligned) in flight at once,
// and one thread a column then adds the terms in order from shared memory.  A
// thread a column walking its rows, and the tree as a launch of its own behind
// scratch in global memory, took 14.3 us on 32 PCs of 32,768 fibres; this takes
// 8.4, launch included.
template <int V>
__global__ void __launch_bounds__(kThreads) pfpcSumsKernel(const uint32_t *apBuf, const uint32_t *mask, const float *w,
		uint32_t P, uint32_t bs, uint32_t cols, float *sums)
{
	namespace cg = cooperative_groups;
	__shared__ __align__(16) float sTerm[kThreads * V];
	__shared__ float sPart[512];  // the PC's partials (in the cluster's first CTA)
	cg::cluster_group cluster = cg::this_cluster();
	// a CTA's shared memory may be written from another one once it has started:
	// every CTA says so here, and the others wait for that behind their loads
	cluster.barrier_arrive();
	const uint32_t part = cluster.block_rank(), pc = blockIdx.x / cluster.num_blocks();
	const uint32_t tid = threadIdx.x, lanes = cols / V, rows = blockDim.x / lanes;
	const uint32_t j = part * cols + tid % lanes * V, r = tid / lanes, K = P / (2 * bs);
	const size_t at = (size_t)pc * P + j;
	float s = 0;
	for (uint32_t k0 = 0; k0 < K; k0 += rows) {
		const uint32_t n = min(rows, K - k0);
		if (r < n) {
			const size_t a = at + (size_t)(k0 + r) * 2 * bs, b = a + bs;
			const Words<V> apA = loadWords<V>(apBuf + a), mA = loadWords<V>(mask + a);
			const Words<V> wA = loadWords<V>(reinterpret_cast<const uint32_t *>(w) + a);
			const Words<V> apB = loadWords<V>(apBuf + b), mB = loadWords<V>(mask + b);
			const Words<V> wB = loadWords<V>(reinterpret_cast<const uint32_t *>(w) + b);
#pragma unroll
			for (int v = 0; v < V; v++) {
				const unsigned int pa = (apA.x[v] & mA.x[v]) > 0, pb = (apB.x[v] & mB.x[v]) > 0;
				sTerm[tid * V + v] = __uint_as_float(wA.x[v]) * pa + __uint_as_float(wB.x[v]) * pb;
			}
		}
		__syncthreads();
		if (tid < cols)
#pragma unroll 8
			for (uint32_t q = 0; q < n; q++) s += sTerm[q * cols + tid];
		__syncthreads();
	}
	// the partials to the cluster's first CTA
	cluster.barrier_wait();
	if (tid < cols) cluster.map_shared_rank(sPart, 0)[part * cols + tid] = s;
	cluster.sync();
	if (part || tid >= 32) return;
	// lane l holds partials l, l + 32, ...: strides of 32 and more combine
	// registers of a lane
	float v[16];
	const uint32_t m = bs / 32;
#pragma unroll
	for (uint32_t q = 0; q < 16; q++) v[q] = tid + 32 * q < bs ? sPart[tid + 32 * q] : 0.0f;
#pragma unroll
	for (uint32_t h = 8; h >= 1; h /= 2)
		if (h < m)
#pragma unroll
			for (uint32_t q = 0; q < h; q++) v[q] = v[q] + v[q + h];
	for (uint32_t h = min(bs, 32u) / 2; h >= 1; h /= 2) v[0] = v[0] + __shfl_down_sync(0xffffffffu, v[0], h);
	if (tid == 0) sums[pc] = v[0];
}

}  // namespace

// the C ABI's per-thread error message (cbm_capi.cu), read by cbm_last_error
extern thread_local std::string g_cbmLastError;

static int fail(int code, const std::string &msg)
{
	g_cbmLastError = msg;
	return code;
}

extern "C" int cbm_pfpc_sums_noalloc(const uint32_t *apBuf, const uint32_t *pfDelayMask, const float *weights,
		uint32_t numGR, uint32_t numPC, float *sums, void *stream)
{
	if (!apBuf || !pfDelayMask || !weights || !sums) return fail(CBM_ERR_ARG, "null buffer");
	if (numPC == 0 || numGR % numPC) return fail(CBM_ERR_ARG, "numGR must be a multiple of numPC");
	const uint32_t P = numGR / numPC;
	if (P < 4 || (P & (P - 1))) return fail(CBM_ERR_ARG, "fibres per PC must be a power of two >= 4");
	const uint32_t bs = rowBlockSize(P);
	if ((uint64_t)numPC * bs > kMaxPartials)
		return fail(CBM_ERR_ARG, "numPC x reduction width exceeds CBM_NOALLOC_MAX_PARTIALS (" +
				std::to_string(kMaxPartials) + ")");
	cudaError_t e = cudaPeekAtLastError();
	if (e != cudaSuccess)
		return fail(CBM_ERR_CUDA, std::string("a CUDA error is already pending in this thread: ") + cudaGetErrorString(e));
	// 16-byte loads where every row of every buffer is aligned for them
	const uintptr_t bits = (uintptr_t)apBuf | (uintptr_t)pfDelayMask | (uintptr_t)weights;
	const bool wide = bs >= 4 && (bits & 15) == 0;
	const uint32_t cols = std::min(bs, kCols), lanes = wide ? cols / 4 : cols, K = P / (2 * bs);
	// a thread for each of the rows' terms, whole warps
	const uint32_t threads = std::max(32u, std::min(kThreads, lanes * std::max(K, wide ? 4u : 1u)));
	cudaLaunchConfig_t c = {};
	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeClusterDimension;
	at.val.clusterDim.x = bs / cols;
	at.val.clusterDim.y = at.val.clusterDim.z = 1;
	c.gridDim = dim3(numPC * (bs / cols));
	c.blockDim = dim3(threads);
	c.stream = (cudaStream_t)stream;
	c.attrs = &at;
	c.numAttrs = 1;
	e = cudaLaunchKernelEx(&c, wide ? pfpcSumsKernel<4> : pfpcSumsKernel<1>, apBuf, pfDelayMask, weights, P, bs, cols, sums);
	if (e != cudaSuccess) {
		cudaGetLastError();
		return fail(CBM_ERR_CUDA, std::string("PF->PC sums launch: ") + cudaGetErrorString(e));
	}
	return CBM_OK;
}
