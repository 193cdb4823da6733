// The sweep surrogate: a small MLP (nIn -> h1 -> h2 -> nOut, ReLU) trained and
// run on the GPU with this file's own kernels.  Every matrix product is one
// kernel, gemmKernel, on the 5th-generation tensor cores: BF16 operands staged
// in shared memory in the canonical K-major layout, tcgen05.mma issued by one
// thread, the FP32 accumulator in tensor memory read back with tcgen05.ld for
// the epilogue (bias, ReLU, ReLU derivative or loss gradient, FP32 and/or BF16
// store).  Weights are kept in FP32 (Adam) and rounded to BF16 for the products.
// A minibatch is a chain of eight small launches, each waiting for the last on
// the device (programmatic dependent launch).
//
// No counterpart in the reference (its parameter sweeps simulate every
// candidate).
#include <cstdint>
#include <cstdio>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/cbm_surrogate.h"
#include "cbm_device.cuh"
#include "cbm_kernels.cuh"
#include "cbm_tma.cuh"

extern thread_local std::string g_cbmLastError;

namespace cbm {
namespace mlp {

constexpr uint64_t kMmaWaitLimitNs = 2000000000ull;
constexpr int kTileM = 128, kTileN = 32;  // one CTA's output
constexpr int kThreads = 256;
constexpr int kKChunk = 256;              // K elements staged per round
// A staged operand: row r, 16-byte K piece c at (r / 8) kSBO + c kLBO + (r % 8) 16.
// The 16 bytes beyond a core matrix, and beyond a row group, keep neighbouring
// pieces and neighbouring row groups on different banks.
constexpr uint32_t kLBO = 128 + 16, kSBO = (kKChunk / 8) * kLBO + 16;
constexpr uint32_t kGemmSmem = 128 + (kTileM + kTileN) / 8 * kSBO;

__device__ __forceinline__ uint32_t smemU32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a K-major, unswizzled operand: core
// matrices of 8 rows x 16 bytes, 8-row groups sbo bytes apart, the two
// 8-element K halves of an MMA lbo bytes apart.
__device__ __forceinline__ uint64_t smemDesc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
	uint64_t d = 0;
	d |= (uint64_t)((addr >> 4) & 0x3FFFu);
	d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
	d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
	d |= 1ull << 46;  // descriptor version of this architecture
	// base offset 0, absolute LBO mode 0, layout type 0 (no swizzle)
	return d;
}

// Instruction descriptor of kind::f16: BF16 A and B, FP32 D, both K-major,
// M = 128, N = n.
__host__ __device__ constexpr uint32_t instrDesc(uint32_t n)
{
	return (1u << 4)            // D format F32
		| (1u << 7)             // A format BF16
		| (1u << 10)            // B format BF16
		| ((n >> 3) << 17)      // N / 8
		| ((128u >> 4) << 24);  // M / 16
}

// Rows a forward pass takes at a time (a larger maxBatch takes that many): the
// 4096 rows of a 64-256-256-50 network went in 16 chunks of 256, each with a
// pageable copy in, one out and a wait, in 928 us; so they take 205.
constexpr uint32_t kRows = 4096;

// One product, out[m][n] = f(sum_k A(m,k) B(n,k)) for m < M, n < N, or the
// column sums of a matrix (colSum != null).
// A(m,k) is A[m lda + k], or A[k lda + m] with tA (a product over the batch, or
// with a transposed weight matrix, reads its operand as it lies); B alike.  N, lda
// and ldb are multiples of 64, and K, but for an operand pair that is transposed.
struct GemmJob {
	const __nv_bfloat16 *A = nullptr, *B = nullptr;
	int M = 0, N = 0, K = 0, lda = 0, ldb = 0;
	bool tA = false, tB = false, relu = false;
	const float *bias = nullptr;          // [N], added
	const __nv_bfloat16 *mask = nullptr;  // [M][N]: 0 where it is not positive (the ReLU derivative)
	// mean squared error against target [M][nOut]: the outputs are 2 (v - target) / (M nOut),
	// 0 for n >= nOut, and the squares are added to *loss
	const float *target = nullptr;
	float *loss = nullptr;
	float *outF = nullptr;                // FP32 [M][ldo], columns < nOut
	__nv_bfloat16 *outH = nullptr;        // BF16 [M][N]
	int ldo = 0, nOut = 0;
	const float *colSum = nullptr;        // [M][N]: outF[n] = sum over m
};
struct GemmJobs {
	GemmJob j[4];
};

// Rows [r0, r0 + ROWS) of an operand (R valid), K elements [k0, k0 + kPad) of
// K, into its staged layout; zeros outside.
template <int ROWS>
__device__ __forceinline__ void stageOperand(uint8_t *s, const __nv_bfloat16 *X, int ld, bool trans, int r0, int R,
		int k0, int K, int kPad)
{
	const int tid = threadIdx.x;
	if (!trans) {
		// 16-byte pieces along K, all in flight (no registers)
		const int pieces = kPad / 8;
		for (int q = tid; q < ROWS * pieces; q += kThreads) {
			const int r = q / pieces, c = q % pieces;
			uint8_t *d = s + (r / 8) * kSBO + c * kLBO + (r % 8) * 16;
			if (r0 + r < R)
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smemU32(d)),
						"l"(X + (size_t)(r0 + r) * ld + k0 + c * 8) : "memory");
			else
				*reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
		}
		return;
	}
	// two consecutive K rows of eight elements at a time, transposed in registers
	constexpr int G = ROWS / 8, U = ROWS >= 128 ? 8 : 2;
	const int pairs = kPad / 2 * G;
	for (int q0 = tid; q0 < pairs; q0 += U * kThreads) {
		uint4 v[U][2];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const int q = q0 + u * kThreads, g = q % G, k = k0 + 2 * (q / G);
			v[u][0] = v[u][1] = make_uint4(0, 0, 0, 0);
			if (q < pairs && r0 + 8 * g < R) {
				if (k < K) v[u][0] = *reinterpret_cast<const uint4 *>(X + (size_t)k * ld + r0 + 8 * g);
				if (k + 1 < K) v[u][1] = *reinterpret_cast<const uint4 *>(X + (size_t)(k + 1) * ld + r0 + 8 * g);
			}
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			const int q = q0 + u * kThreads, g = q % G, k = 2 * (q / G);
			if (q >= pairs) break;
			uint8_t *d = s + g * kSBO + (k / 8) * kLBO + (k % 8) * 2;
			const uint32_t a[4] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w};
			const uint32_t b[4] = {v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
#pragma unroll
			for (int i = 0; i < 4; i++) {
				*reinterpret_cast<uint32_t *>(d + 32 * i) = __byte_perm(a[i], b[i], 0x5410);
				*reinterpret_cast<uint32_t *>(d + 32 * i + 16) = __byte_perm(a[i], b[i], 0x7632);
			}
		}
	}
}

// Column sums of columns [32 blockIdx.y, + 32), row after row: a sum's sign can
// decide an Adam step, so the order stays that of one thread walking its column.
// The rows come to shared memory 256 at a time, all their loads in flight (a
// thread a column loading as it adds took 16 us over 256 rows).
__device__ void colSums(const GemmJob &J, float *s)
{
	const int tid = threadIdx.x, c4 = tid % 8, r0 = tid / 8, n0 = 32 * blockIdx.y;
	float x = 0.0f;
	for (int m0 = 0; m0 < J.M; m0 += 256) {
		const int rows = min(256, J.M - m0);
		float4 v[8];
#pragma unroll
		for (int u = 0; u < 8; u++)
			if (r0 + 32 * u < rows)
				v[u] = *reinterpret_cast<const float4 *>(J.colSum + (size_t)(m0 + r0 + 32 * u) * J.N + n0 + 4 * c4);
#pragma unroll
		for (int u = 0; u < 8; u++)
			if (r0 + 32 * u < rows) *reinterpret_cast<float4 *>(s + 32 * (r0 + 32 * u) + 4 * c4) = v[u];
		__syncthreads();
		if (tid < 32)
#pragma unroll 16
			for (int r = 0; r < rows; r++) x += s[32 * r + tid];
		__syncthreads();
	}
	if (tid < 32) J.outF[n0 + tid] = x;
}

// The products of these layers (at most 256 wide) are tiny: what bounds them is
// latency, one round trip for the operands, the MMAs, one store.  So a CTA takes
// 128 x 32 outputs and stages its operands' whole depth (up to 256) with every
// load in flight before one wait; two independent products of the backward pass
// share a launch (blockIdx.z).  A 128 x 256 tile in rounds of 64 K elements, each
// waiting for its loads and its MMAs, on one or two CTAs took 30-62 us a product;
// transposed copies of the operands, the ReLU derivative and the loss were
// launches of their own.  A 64-256-256-50 network's gradients over 200 rows took
// 523 us and take 143, a training minibatch of 256 took 484 and takes 68, a
// forward pass over 4096 rows 3670 and 215 (copies to and from the host included).
__global__ void __launch_bounds__(kThreads) gemmKernel(const __grid_constant__ GemmJobs jobs, uint32_t *err)
{
	pdlLaunchDependents();
	extern __shared__ uint8_t gemmSmemRaw[];
	const GemmJob &J = jobs.j[blockIdx.z];
	const int m0 = blockIdx.x * kTileM, n0 = blockIdx.y * kTileN;
	uint8_t *sA = gemmSmemRaw + ((128u - (smemU32(gemmSmemRaw) & 127u)) & 127u);
	if (n0 >= J.N || (J.colSum ? blockIdx.x > 0 : m0 >= J.M)) return;
	if (J.colSum) {
		pdlWait();
		colSums(J, reinterpret_cast<float *>(sA));
		return;
	}
	uint8_t *sB = sA + kTileM / 8 * kSBO;
	__shared__ __align__(8) uint64_t bar;
	__shared__ uint32_t tmemBase;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemU32(&tmemBase)),
				"r"((uint32_t)kTileN) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	if (tid == 0) {
		tma::mbarInit(&bar, 1);
		tma::fenceBarrierInit();
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem = tmemBase;
	pdlWait();

	constexpr uint32_t idesc = instrDesc(kTileN);
	bool ok = true;
	for (int k0 = 0, round = 0; k0 < J.K; k0 += kKChunk, round++) {
		const int kPad = (min(kKChunk, J.K - k0) + 15) & ~15;
		stageOperand<kTileM>(sA, J.A, J.lda, J.tA, m0, J.M, k0, J.K, kPad);
		stageOperand<kTileN>(sB, J.B, J.ldb, J.tB, n0, J.N, k0, J.K, kPad);
		asm volatile("cp.async.wait_all;" ::: "memory");
		// make the generic-proxy stores visible to the tensor cores
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		__syncthreads();
		if (tid == 0) {
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			for (int ks = 0; ks < kPad; ks += 16) {
				const uint64_t da = smemDesc(smemU32(sA) + (ks / 8) * kLBO, kLBO, kSBO);
				const uint64_t db = smemDesc(smemU32(sB) + (ks / 8) * kLBO, kLBO, kSBO);
				const uint32_t accumulate = (k0 > 0 || ks > 0) ? 1u : 0u;
				asm volatile(
					"{\n\t.reg .pred p;\n\t"
					"setp.ne.b32 p, %4, 0;\n\t"
					"tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
					::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
					: "memory");
			}
			asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
					::"r"(smemU32(&bar)) : "memory");
		}
		// the chunk's MMAs have read shared memory once the barrier flips
		const bool done = tma::waitBounded(&bar, (uint32_t)(round & 1), kMmaWaitLimitNs);
		if (!__syncthreads_and(done)) {
			ok = false;
			break;
		}
		asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	}
	float e2 = 0.0f;
	if (!ok) {
		if (tid == 0) atomicOr(err, 1u);
	} else {
		// epilogue: warp w owns TMEM lanes (rows) 32 (w mod 4).. and columns 16 (w / 4)..
		const int m = m0 + (warp % 4) * 32 + lane, c0 = warp / 4 * 16, n1 = n0 + c0;
		uint32_t r[16];
		const uint32_t taddr = tmem + ((uint32_t)(warp % 4 * 32) << 16) + (uint32_t)c0;
		asm volatile(
			"tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
			: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
			  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
			: "r"(taddr));
		asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
		if (m < J.M) {
			float v[16];
#pragma unroll
			for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
			if (J.bias)
#pragma unroll
				for (int j = 0; j < 16; j++) v[j] += __ldg(J.bias + n1 + j);
			if (J.relu)
#pragma unroll
				for (int j = 0; j < 16; j++) v[j] = v[j] > 0.0f ? v[j] : 0.0f;
			if (J.mask) {
				__align__(16) __nv_bfloat16 h[16];
				*reinterpret_cast<uint4 *>(h) = *reinterpret_cast<const uint4 *>(J.mask + (size_t)m * J.N + n1);
				*reinterpret_cast<uint4 *>(h + 8) = *reinterpret_cast<const uint4 *>(J.mask + (size_t)m * J.N + n1 + 8);
#pragma unroll
				for (int j = 0; j < 16; j++) v[j] = __bfloat162float(h[j]) > 0.0f ? v[j] : 0.0f;
			}
			if (J.target)
#pragma unroll
				for (int j = 0; j < 16; j++) {
					float g = 0.0f;
					if (n1 + j < J.nOut) {
						const float d = v[j] - J.target[(size_t)m * J.nOut + n1 + j];
						e2 += d * d;
						g = 2.0f * d / ((float)J.M * (float)J.nOut);
					}
					v[j] = g;
				}
			if (J.outF) {
				float *o = J.outF + (size_t)m * J.ldo + n1;
				if (J.ldo == J.N)
#pragma unroll
					for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4 *>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
				else
#pragma unroll
					for (int j = 0; j < 16; j++)
						if (n1 + j < J.nOut) o[j] = v[j];
			}
			if (J.outH) {
				__align__(16) __nv_bfloat16 h[16];
#pragma unroll
				for (int j = 0; j < 16; j++) h[j] = __float2bfloat16_rn(v[j]);
				uint4 *o = reinterpret_cast<uint4 *>(J.outH + (size_t)m * J.N + n1);
				o[0] = *reinterpret_cast<const uint4 *>(h);
				o[1] = *reinterpret_cast<const uint4 *>(h + 8);
			}
		}
		if (J.target) {
			for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
			if (lane == 0 && e2 != 0.0f) atomicAdd(J.loss, e2);
		}
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTileN) : "memory");
}

// ------------------------------------------------------------ elementwise
// The rows x nIn input as BF16 rows of I (zeros beyond nIn), the parameters as
// BF16 (nP of them, or 0 to leave the copy), and the loss to 0.
__global__ void prepareKernel(const float *x, uint32_t rows, uint32_t nIn, uint32_t I, __nv_bfloat16 *X, const float *P,
		size_t nP, __nv_bfloat16 *Wh, float *loss)
{
	pdlLaunchDependents();
	pdlWait();
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, n = (size_t)rows * I;
	if (i == 0) *loss = 0.0f;
	if (i < n) {
		const uint32_t r = (uint32_t)(i / I), c = (uint32_t)(i % I);
		X[i] = __float2bfloat16_rn(c < nIn ? x[(size_t)r * nIn + c] : 0.0f);
	} else if (i - n < nP) {
		Wh[i - n] = __float2bfloat16_rn(P[i - n]);
	}
}

// Adam (Kingma and Ba, 2015) on n parameters, bias-corrected step t, and the
// parameters' BF16 copy.  Not on the gradients of a product that failed, which the
// host hears of at the end of the epoch.
__global__ void adamKernel(float *p, const float *g, float *m, float *v, size_t n, float lr, float b1, float b2,
		float eps, float c1, float c2, __nv_bfloat16 *h, const uint32_t *err)
{
	pdlLaunchDependents();
	pdlWait();
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n || *err) return;
	const float gi = g[i];
	const float mi = b1 * m[i] + (1 - b1) * gi, vi = b2 * v[i] + (1 - b2) * gi * gi;
	m[i] = mi;
	v[i] = vi;
	const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	p[i] = pi;
	h[i] = __float2bfloat16_rn(pi);
}

}  // namespace mlp
}  // namespace cbm

using namespace cbm::mlp;

// ---------------------------------------------------------------- host side
struct cbm_mlp {
	int device = 0;
	uint32_t nIn = 0, h1 = 0, h2 = 0, nOut = 0;   // logical sizes
	uint32_t I = 0, H1 = 0, H2 = 0, O = 0;        // padded to multiples of 64
	uint32_t maxBatch = 0;                        // rows of a minibatch
	uint32_t rows = 0;                            // rows a forward pass takes at a time, and a training upload brings
	cudaStream_t s = nullptr;
	// FP32 master parameters (flat: W1 [H1][I], b1, W2 [H2][H1], b2, W3 [O][H2], b3), grads, Adam moments
	float *P = nullptr, *G = nullptr, *Mo = nullptr, *Ve = nullptr;
	size_t nP = 0;
	size_t oW1 = 0, ob1 = 0, oW2 = 0, ob2 = 0, oW3 = 0, ob3 = 0;
	// BF16 copies and activations
	__nv_bfloat16 *Wh = nullptr;
	__nv_bfloat16 *X = nullptr, *H1h = nullptr, *H2h = nullptr, *dYh = nullptr, *dH2h = nullptr, *dH1h = nullptr;
	// inputs, outputs and targets as the caller has them; FP32 gradients of the layers' outputs
	float *Xf = nullptr, *Yf = nullptr, *Tf = nullptr, *dYf = nullptr, *dH2f = nullptr, *dH1f = nullptr;
	float *loss = nullptr;                        // a minibatch's, of an upload
	// pinned halves of the training upload (rows in their order, losses), each
	// reused once the event behind it has passed
	float *hX[2] = {}, *hT[2] = {}, *hLoss[2] = {};
	cudaEvent_t done[2] = {};
	uint32_t *err = nullptr;
	uint64_t adamStep = 0;
	void *arena = nullptr;                        // every device array above
};

static int mfail(int code, const std::string &m)
{
	g_cbmLastError = m;
	return code;
}

#define MCK(call, what) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) return mfail(CBM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e_)); } while (0)

static uint32_t pad(uint32_t x, uint32_t m) { return (x + m - 1) / m * m; }

// One launch that may start while the one before it ends (each kernel waits for
// it on the device, pdlWait).
template <typename... P, typename... A>
static int launch(cbm_mlp *n, void (*k)(P...), dim3 grid, size_t smem, const char *what, A... args)
{
	cudaLaunchConfig_t c = {};
	c.gridDim = grid;
	c.blockDim = dim3(kThreads);
	c.dynamicSmemBytes = smem;
	c.stream = n->s;
	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	c.attrs = &at;
	c.numAttrs = 1;
	MCK(cudaLaunchKernelEx(&c, k, args...), what);
	return CBM_OK;
}

// Independent products (and column sums), one launch.
static int gemm(cbm_mlp *n, const std::vector<GemmJob> &jobs)
{
	GemmJobs J;
	dim3 grid(1, 1, (unsigned)jobs.size());
	for (size_t i = 0; i < jobs.size(); i++) {
		J.j[i] = jobs[i];
		if (!jobs[i].colSum) grid.x = std::max(grid.x, (unsigned)((jobs[i].M + kTileM - 1) / kTileM));
		grid.y = std::max(grid.y, (unsigned)(jobs[i].N / kTileN));
	}
	return launch(n, gemmKernel, grid, kGemmSmem, "launching a tensor-core product", J, n->err);
}

static GemmJob product(const __nv_bfloat16 *A, int lda, bool tA, const __nv_bfloat16 *B, int ldb, bool tB, int M, int N,
		int K)
{
	GemmJob j;
	j.A = A; j.lda = lda; j.tA = tA;
	j.B = B; j.ldb = ldb; j.tB = tB;
	j.M = M; j.N = N; j.K = K;
	j.ldo = j.nOut = N;
	return j;
}

static GemmJob columnSums(const float *g, int M, int N, float *out)
{
	GemmJob j;
	j.colSum = g;
	j.M = M; j.N = N;
	j.outF = out;
	return j;
}

static int checkErr(cbm_mlp *n)
{
	uint32_t e = 0;
	MCK(cudaMemcpyAsync(&e, n->err, 4, cudaMemcpyDeviceToHost, n->s), "reading the error word");
	MCK(cudaStreamSynchronize(n->s), "surrogate");
	if (e) return mfail(CBM_ERR_CUDA, "tensor-core product: a completion wait timed out on the device");
	return CBM_OK;
}

#define MTRY(x) do { int r_ = (x); if (r_ != CBM_OK) return r_; } while (0)

// The BF16 input from b uploaded rows (x on the device, b x nIn), and the
// weights' copy when it may be old.
static int prepare(cbm_mlp *n, const float *x, uint32_t b, bool weights, float *loss)
{
	const size_t count = (size_t)b * n->I + (weights ? n->nP : 0);
	return launch(n, prepareKernel, dim3((unsigned)((count + kThreads - 1) / kThreads)), 0, "cast", x, b, n->nIn, n->I,
			n->X, (const float *)n->P, weights ? n->nP : (size_t)0, n->Wh, loss);
}

// Forward over b rows: the outputs to Yf (b x nOut), or, with a target (b x nOut,
// on the device), the mean squared error's gradient to dYf and dYh and its sum to
// *loss.
static int forward(cbm_mlp *n, uint32_t b, const float *target, float *loss)
{
	const __nv_bfloat16 *W1 = n->Wh + n->oW1, *W2 = n->Wh + n->oW2, *W3 = n->Wh + n->oW3;
	const int B = (int)b;
	GemmJob l1 = product(n->X, n->I, false, W1, n->I, false, B, n->H1, n->I);
	l1.bias = n->P + n->ob1; l1.relu = true; l1.outH = n->H1h;
	GemmJob l2 = product(n->H1h, n->H1, false, W2, n->H1, false, B, n->H2, n->H1);
	l2.bias = n->P + n->ob2; l2.relu = true; l2.outH = n->H2h;
	GemmJob l3 = product(n->H2h, n->H2, false, W3, n->H2, false, B, n->O, n->H2);
	l3.bias = n->P + n->ob3; l3.nOut = n->nOut;
	if (target) {
		l3.target = target; l3.loss = loss;
		l3.outF = n->dYf; l3.outH = n->dYh;
	} else {
		l3.outF = n->Yf; l3.ldo = n->nOut;
	}
	MTRY(gemm(n, {l1}));
	MTRY(gemm(n, {l2}));
	return gemm(n, {l3});
}

// Gradients of the mean squared error over the b rows of the last forward into G.
static int backward(cbm_mlp *n, uint32_t b)
{
	const __nv_bfloat16 *W2 = n->Wh + n->oW2, *W3 = n->Wh + n->oW3;
	const int B = (int)b;
	// weight gradients: dY^T H, products over the batch
	auto weights = [&](const __nv_bfloat16 *d, uint32_t out, const __nv_bfloat16 *h, uint32_t in, float *g) {
		GemmJob j = product(d, out, true, h, in, true, out, in, B);
		j.outF = g;
		return j;
	};
	// a layer's upstream gradient through the ReLU: dY W
	auto upstream = [&](const __nv_bfloat16 *d, uint32_t out, const __nv_bfloat16 *W, uint32_t in,
			const __nv_bfloat16 *h, float *f, __nv_bfloat16 *o) {
		GemmJob j = product(d, out, false, W, in, true, B, in, out);
		j.mask = h; j.outF = f; j.outH = o;
		return j;
	};
	MTRY(gemm(n, {weights(n->dYh, n->O, n->H2h, n->H2, n->G + n->oW3),
			upstream(n->dYh, n->O, W3, n->H2, n->H2h, n->dH2f, n->dH2h)}));
	MTRY(gemm(n, {weights(n->dH2h, n->H2, n->H1h, n->H1, n->G + n->oW2),
			upstream(n->dH2h, n->H2, W2, n->H1, n->H1h, n->dH1f, n->dH1h)}));
	return gemm(n, {weights(n->dH1h, n->H1, n->X, n->I, n->G + n->oW1), columnSums(n->dYf, B, n->O, n->G + n->ob3),
			columnSums(n->dH2f, B, n->H2, n->G + n->ob2), columnSums(n->dH1f, B, n->H1, n->G + n->ob1)});
}

extern "C" {

int cbm_mlp_create(unsigned nIn, unsigned h1, unsigned h2, unsigned nOut, unsigned maxBatch, uint64_t seed, int device,
		cbm_mlp **out)
{
	if (!out) return mfail(CBM_ERR_ARG, "null argument: out");
	if (!nIn || !h1 || !h2 || !nOut || !maxBatch) return mfail(CBM_ERR_ARG, "sizes must be positive");
	if (pad(nIn, 64) > 256 || pad(h1, 64) > 256 || pad(h2, 64) > 256 || pad(nOut, 64) > 256)
		return mfail(CBM_ERR_ARG, "layers are at most 256 wide");
	cbm_mlp *n = new cbm_mlp();
	n->device = device;
	n->nIn = nIn; n->h1 = h1; n->h2 = h2; n->nOut = nOut;
	n->I = pad(nIn, 64); n->H1 = pad(h1, 64); n->H2 = pad(h2, 64); n->O = pad(nOut, 64);
	n->maxBatch = maxBatch;
	n->rows = std::max(maxBatch, kRows);
	if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&n->s, cudaStreamNonBlocking) != cudaSuccess) {
		delete n;
		return mfail(CBM_ERR_CUDA, "stream");
	}
	if (cudaFuncSetAttribute(gemmKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem) != cudaSuccess) {
		cudaStreamDestroy(n->s);
		delete n;
		return mfail(CBM_ERR_CUDA, "tensor-core product shared memory");
	}
	n->oW1 = 0; n->ob1 = n->oW1 + (size_t)n->H1 * n->I;
	n->oW2 = n->ob1 + n->H1; n->ob2 = n->oW2 + (size_t)n->H2 * n->H1;
	n->oW3 = n->ob2 + n->H2; n->ob3 = n->oW3 + (size_t)n->O * n->H2;
	n->nP = n->ob3 + n->O;
	const size_t B = maxBatch, R = n->rows;
	// one allocation, zeroed: measured first, then handed out
	auto layout = [&](uint8_t *base) {
		size_t o = 0;
		auto take = [&](auto *&p, size_t count) {
			p = base ? (std::remove_reference_t<decltype(p)>)(base + o) : nullptr;
			o += (count * sizeof(*p) + 255) & ~(size_t)255;
		};
		take(n->P, n->nP);
		take(n->G, n->nP);
		take(n->Mo, n->nP);
		take(n->Ve, n->nP);
		take(n->Wh, n->nP);
		take(n->X, R * n->I);
		take(n->H1h, R * n->H1);
		take(n->H2h, R * n->H2);
		take(n->Xf, R * n->nIn);
		take(n->Yf, R * n->nOut);
		take(n->Tf, R * n->nOut);
		take(n->dYf, B * n->O);
		take(n->dYh, B * n->O);
		take(n->dH2f, B * n->H2);
		take(n->dH2h, B * n->H2);
		take(n->dH1f, B * n->H1);
		take(n->dH1h, B * n->H1);
		take(n->loss, R);
		take(n->err, 1);
		return o;
	};
	const size_t bytes = layout(nullptr);
	// on the handle's stream, like everything after it (the default stream would not
	// be waited for)
	if (cudaMalloc(&n->arena, bytes) != cudaSuccess || cudaMemsetAsync(n->arena, 0, bytes, n->s) != cudaSuccess) {
		cbm_mlp_destroy(n);
		return mfail(CBM_ERR_CUDA, "device allocation failed");
	}
	layout((uint8_t *)n->arena);
	// He-uniform initial weights (logical part only), zero biases
	std::vector<float> p(n->nP, 0.0f);
	std::mt19937_64 rng(seed);
	auto init = [&](size_t off, uint32_t rows, uint32_t cols, uint32_t ld, uint32_t fanIn) {
		std::uniform_real_distribution<float> u(-1.0f, 1.0f);
		const float a = std::sqrt(6.0f / (float)fanIn);
		for (uint32_t r = 0; r < rows; r++)
			for (uint32_t c = 0; c < cols; c++) p[off + (size_t)r * ld + c] = a * u(rng);
	};
	init(n->oW1, h1, nIn, n->I, nIn);
	init(n->oW2, h2, h1, n->H1, h1);
	init(n->oW3, nOut, h2, n->H2, h2);
	if (cudaMemcpyAsync(n->P, p.data(), p.size() * 4, cudaMemcpyHostToDevice, n->s) != cudaSuccess ||
			cudaStreamSynchronize(n->s) != cudaSuccess) {
		cbm_mlp_destroy(n);
		return mfail(CBM_ERR_CUDA, "uploading parameters");
	}
	*out = n;
	return CBM_OK;
}

void cbm_mlp_destroy(cbm_mlp *n)
{
	if (!n) return;
	if (n->arena) cudaFree(n->arena);
	for (int h = 0; h < 2; h++) {
		for (float *p : {n->hX[h], n->hT[h], n->hLoss[h]}) if (p) cudaFreeHost(p);
		if (n->done[h]) cudaEventDestroy(n->done[h]);
	}
	if (n->s) cudaStreamDestroy(n->s);
	delete n;
}

uint64_t cbm_mlp_num_params(cbm_mlp *n) { return n ? n->nP : 0; }

int cbm_mlp_layout(cbm_mlp *n, unsigned *I, unsigned *H1, unsigned *H2, unsigned *O)
{
	if (!n || !I || !H1 || !H2 || !O) return mfail(CBM_ERR_ARG, "null argument");
	*I = n->I; *H1 = n->H1; *H2 = n->H2; *O = n->O;
	return CBM_OK;
}

int cbm_mlp_get_params(cbm_mlp *n, float *dst, uint64_t count)
{
	if (!n || !dst) return mfail(CBM_ERR_ARG, "null argument");
	if (count != n->nP) return mfail(CBM_ERR_ARG, "parameter count mismatch");
	cudaSetDevice(n->device);
	MCK(cudaMemcpyAsync(dst, n->P, count * 4, cudaMemcpyDeviceToHost, n->s), "reading parameters");
	MCK(cudaStreamSynchronize(n->s), "reading parameters");
	return CBM_OK;
}

int cbm_mlp_set_params(cbm_mlp *n, const float *src, uint64_t count)
{
	if (!n || !src) return mfail(CBM_ERR_ARG, "null argument");
	if (count != n->nP) return mfail(CBM_ERR_ARG, "parameter count mismatch");
	cudaSetDevice(n->device);
	MCK(cudaMemcpyAsync(n->P, src, count * 4, cudaMemcpyHostToDevice, n->s), "writing parameters");
	MCK(cudaMemsetAsync(n->Mo, 0, count * 4, n->s), "resetting Adam");
	MCK(cudaMemsetAsync(n->Ve, 0, count * 4, n->s), "resetting Adam");
	MCK(cudaStreamSynchronize(n->s), "writing parameters");  // src is the caller's again
	n->adamStep = 0;
	return CBM_OK;
}

int cbm_mlp_forward(cbm_mlp *n, const float *x, unsigned batch, float *y)
{
	if (!n || !x || !y) return mfail(CBM_ERR_ARG, "null argument");
	cudaSetDevice(n->device);
	for (unsigned b0 = 0; b0 < batch; b0 += n->rows) {
		const unsigned b = std::min(n->rows, batch - b0);
		MCK(cudaMemcpyAsync(n->Xf, x + (size_t)b0 * n->nIn, 4ull * b * n->nIn, cudaMemcpyHostToDevice, n->s), "input");
		MTRY(prepare(n, n->Xf, b, b0 == 0, n->loss));
		MTRY(forward(n, b, nullptr, nullptr));
		MCK(cudaMemcpyAsync(y + (size_t)b0 * n->nOut, n->Yf, 4ull * b * n->nOut, cudaMemcpyDeviceToHost, n->s), "output");
		MTRY(checkErr(n));
	}
	return CBM_OK;
}

int cbm_mlp_gradients(cbm_mlp *n, const float *x, const float *target, unsigned batch, float *grads, float *loss)
{
	if (!n || !x || !target || !grads) return mfail(CBM_ERR_ARG, "null argument");
	if (batch == 0 || batch > n->maxBatch) return mfail(CBM_ERR_ARG, "batch must be 1..maxBatch");
	cudaSetDevice(n->device);
	MCK(cudaMemcpyAsync(n->Xf, x, 4ull * batch * n->nIn, cudaMemcpyHostToDevice, n->s), "input");
	MCK(cudaMemcpyAsync(n->Tf, target, 4ull * batch * n->nOut, cudaMemcpyHostToDevice, n->s), "target");
	MTRY(prepare(n, n->Xf, batch, true, n->loss));
	MTRY(forward(n, batch, n->Tf, n->loss));
	MTRY(backward(n, batch));
	MCK(cudaMemcpyAsync(grads, n->G, n->nP * 4, cudaMemcpyDeviceToHost, n->s), "gradients");
	float l = 0;
	MCK(cudaMemcpyAsync(&l, n->loss, 4, cudaMemcpyDeviceToHost, n->s), "loss");
	MTRY(checkErr(n));
	if (loss) *loss = l / ((float)batch * (float)n->nOut);
	return CBM_OK;
}

int cbm_mlp_train(cbm_mlp *n, const float *x, const float *target, unsigned count, unsigned batch, unsigned epochs,
		float lr, uint64_t seed, float *lastLoss)
{
	if (!n || !x || !target) return mfail(CBM_ERR_ARG, "null argument");
	if (batch == 0 || batch > n->maxBatch || count < batch) return mfail(CBM_ERR_ARG, "batch must be 1..maxBatch and <= count");
	cudaSetDevice(n->device);
	std::vector<uint32_t> order(count);
	for (uint32_t i = 0; i < count; i++) order[i] = i;
	std::mt19937_64 rng(seed);
	// Minibatches go up some at a time, through two pinned halves, and the host
	// waits for a half's work only when it needs the half again: it gathers the
	// next rows while the GPU works.  (With a pageable copy, and a wait for the
	// loss, for each minibatch, 16 of 256 rows took 1.46 ms; so 1.07.)
	const uint32_t perUpload = std::max(1u, kRows / 8 / batch);
	const size_t halfRows = std::max<size_t>(n->maxBatch, kRows / 8);
	MCK(cudaStreamSynchronize(n->s), "training");  // a call that failed may have left copies from them
	for (int h = 0; h < 2; h++) {
		// (each by itself: a call that failed between them left the others)
		if (!n->hX[h]) MCK(cudaMallocHost((void **)&n->hX[h], 4 * halfRows * n->nIn), "pinned rows");
		if (!n->hT[h]) MCK(cudaMallocHost((void **)&n->hT[h], 4 * halfRows * n->nOut), "pinned targets");
		if (!n->hLoss[h]) MCK(cudaMallocHost((void **)&n->hLoss[h], 4 * halfRows), "pinned losses");
		if (!n->done[h]) MCK(cudaEventCreateWithFlags(&n->done[h], cudaEventDisableTiming), "event");
	}
	double epochLoss = 0;
	for (unsigned e = 0; e < epochs; e++) {
		std::shuffle(order.begin(), order.end(), rng);
		epochLoss = 0;
		const uint32_t nb = count / batch;
		uint32_t inFlight[2] = {0, 0};  // minibatches whose losses the half brings back
		auto finish = [&](int h) -> int {
			if (!inFlight[h]) return CBM_OK;
			MCK(cudaEventSynchronize(n->done[h]), "training");
			for (uint32_t i = 0; i < inFlight[h]; i++) epochLoss += n->hLoss[h][i] / ((double)batch * n->nOut);
			inFlight[h] = 0;
			return CBM_OK;
		};
		int h = 0;
		for (uint32_t m0 = 0; m0 < nb; m0 += perUpload, h ^= 1) {
			const uint32_t k = std::min(perUpload, nb - m0), rows = k * batch;
			MTRY(finish(h));
			for (uint32_t r = 0; r < rows; r++) {
				const size_t src = order[(size_t)m0 * batch + r];
				memcpy(n->hX[h] + (size_t)r * n->nIn, x + src * n->nIn, 4ull * n->nIn);
				memcpy(n->hT[h] + (size_t)r * n->nOut, target + src * n->nOut, 4ull * n->nOut);
			}
			MCK(cudaMemcpyAsync(n->Xf, n->hX[h], 4ull * rows * n->nIn, cudaMemcpyHostToDevice, n->s), "input");
			MCK(cudaMemcpyAsync(n->Tf, n->hT[h], 4ull * rows * n->nOut, cudaMemcpyHostToDevice, n->s), "target");
			for (uint32_t i = 0; i < k; i++) {
				// Adam keeps the weights' copy from the first minibatch on
				MTRY(prepare(n, n->Xf + (size_t)i * batch * n->nIn, batch, e == 0 && m0 + i == 0, n->loss + i));
				MTRY(forward(n, batch, n->Tf + (size_t)i * batch * n->nOut, n->loss + i));
				MTRY(backward(n, batch));
				n->adamStep++;
				const float b1 = 0.9f, b2 = 0.999f;
				const float c1 = 1.0f - (float)std::pow(b1, (double)n->adamStep), c2 = 1.0f - (float)std::pow(b2, (double)n->adamStep);
				MTRY(launch(n, adamKernel, dim3((unsigned)((n->nP + kThreads - 1) / kThreads)), 0, "Adam", n->P,
						(const float *)n->G, n->Mo, n->Ve, n->nP, lr, b1, b2, 1e-8f, c1, c2, n->Wh,
						(const uint32_t *)n->err));
			}
			MCK(cudaMemcpyAsync(n->hLoss[h], n->loss, 4ull * k, cudaMemcpyDeviceToHost, n->s), "loss");
			MCK(cudaEventRecord(n->done[h], n->s), "training");
			inFlight[h] = k;
		}
		// the older half first: the losses add up in the minibatches' order
		MTRY(finish(h));
		MTRY(finish(h ^ 1));
		MTRY(checkErr(n));
		epochLoss /= std::max(1u, nb);
	}
	if (lastLoss) *lastLoss = (float)epochLoss;
	return CBM_OK;
}

}  // extern "C"
