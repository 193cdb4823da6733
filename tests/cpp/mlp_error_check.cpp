// Training after a product that failed on the device reports the error and leaves
// the parameters as they were.  The failure is an error word set from the host:
// cudaMemcpyAsync below stands in for the runtime's and notes where the library
// reads that word from.  Pinned memory that runs out between the two training halves
// fails one call, is had by the next, and all of it is given back.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>
#include <dlfcn.h>

#include "cbm_surrogate.h"

static const void *lastWord = nullptr;  // source of the last 4-byte read

extern "C" cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t s)
{
	static const auto real = (cudaError_t(*)(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t))dlsym(RTLD_NEXT,
			"cudaMemcpyAsync");
	if (n == 4 && kind == cudaMemcpyDeviceToHost) lastWord = src;
	return real(dst, src, n, kind, s);
}

static int pinned = 0, pinnedLeft = -1;

extern "C" cudaError_t cudaMallocHost(void **p, size_t n)
{
	static const auto real = (cudaError_t(*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMallocHost");
	if (pinnedLeft == 0) return cudaErrorMemoryAllocation;
	if (pinnedLeft > 0) pinnedLeft--;
	pinned++;
	return real(p, n);
}

extern "C" cudaError_t cudaFreeHost(void *p)
{
	static const auto real = (cudaError_t(*)(void *))dlsym(RTLD_NEXT, "cudaFreeHost");
	pinned--;
	return real(p);
}

#define CHECK(c) do { if (!(c)) { fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)

int main()
{
	const unsigned I = 12, O = 5, rows = 96, batch = 32;
	cbm_mlp *n = nullptr;
	CHECK(cbm_mlp_create(I, 40, 24, O, batch, 7, 0, &n) == 0);
	std::vector<float> x(rows * I), t(rows * O), y(rows * O);
	for (size_t k = 0; k < x.size(); k++) x[k] = (float)(k % 17) / 17 - 0.5f;
	for (size_t k = 0; k < t.size(); k++) t[k] = (float)(k % 5) / 5;
	CHECK(cbm_mlp_forward(n, x.data(), rows, y.data()) == 0);
	CHECK(lastWord != nullptr);
	std::vector<float> p(cbm_mlp_num_params(n)), q(p.size());
	float loss = 0;
	CHECK(cbm_mlp_get_params(n, p.data(), p.size()) == 0);
	for (int k : {2, 1, 0}) {
		pinnedLeft = k;
		CHECK(cbm_mlp_train(n, x.data(), t.data(), rows, batch, 1, 1e-2f, 3, &loss) != 0);
		pinnedLeft = -1;
	}
	CHECK(cbm_mlp_get_params(n, q.data(), q.size()) == 0);
	CHECK(memcmp(p.data(), q.data(), 4 * p.size()) == 0);
	CHECK(cbm_mlp_train(n, x.data(), t.data(), rows, batch, 1, 1e-2f, 3, &loss) == 0);
	CHECK(cbm_mlp_get_params(n, q.data(), q.size()) == 0);
	CHECK(memcmp(p.data(), q.data(), 4 * p.size()) != 0);  // it trains
	const uint32_t failed = 1;
	CHECK(cudaMemcpy(const_cast<void *>(lastWord), &failed, 4, cudaMemcpyHostToDevice) == cudaSuccess);
	CHECK(cudaDeviceSynchronize() == cudaSuccess);
	CHECK(cbm_mlp_train(n, x.data(), t.data(), rows, batch, 1, 1e-2f, 3, &loss) != 0);
	CHECK(cbm_mlp_get_params(n, p.data(), p.size()) == 0);
	CHECK(memcmp(p.data(), q.data(), 4 * p.size()) == 0);  // none of it was applied
	cbm_mlp_destroy(n);
	CHECK(pinned == 0);
	return 0;
}
