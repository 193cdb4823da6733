// Kernel entry points of the step (definitions in cbm_kernels.cu).
#pragma once
#include <cstdint>
#include "cbm_device.cuh"

namespace cbm {

constexpr int kPassThreads = 256;
// 24 warps: at 80 registers a thread the small-cell update keeps every value
// in registers (at 1024 threads, 64 registers, it spilled, and the spill
// reloads went to L2 between its phases)
constexpr int kTailThreads = 768;

// Programmatic dependent launch between the two kernels of consecutive
// steps.  With the per-tile pass, steps run as small-cell(t) -> pass(t) ->
// small-cell(t+1) -> ..., each launched as the programmatic dependent of the
// kernel before it (one at a time, and in the graphs of chunked runs), so that
// the next kernel is resident before its predecessor ends.  In graphs whose
// steps joined both kernels before the next one, a step took 0.6-1.3 us longer
// (14.2 against 13.6 us on 1M GR, 14.3 against 13.0 on 256K).  Two rules keep
// that equal to full stream order:
//  - the small-cell kernel waits for its predecessor (the previous step's
//    GR pass) before it reads anything, and only then lets its own
//    dependent (this step's GR pass) launch;
//  - the last CTA of such a GR pass to finish waits for its predecessor
//    (this step's small-cell kernel) before it exits, so that a finished
//    GR pass means a finished step (passExitWait).
// A pass lets the next small-cell kernel launch from its start.  Launched
// without the attribute (the other passes), each wait returns at once.
__device__ __forceinline__ void pdlWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdlLaunchDependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// At the end of a GR-pass CTA, after a barrier of the whole CTA: with a
// counter (chained steps), the launch's last CTA to get here resets
// it and waits for the step's small-cell kernel; the others exit, so that
// the slots of early CTAs go to later waves.
__device__ __forceinline__ void passExitWait(uint32_t *exitCount)
{
	if (exitCount && threadIdx.x == 0 && atomicAdd(exitCount, 1u) == gridDim.x - 1u) {
		*exitCount = 0;
		pdlWait();
	}
}

__global__ void grPassKernel(const DevNet *const *nets, const uint32_t *blockOffset, int numNets,
		uint32_t stepOffset);
// Each CTA of a batch's per-tile pass: the network, and its tile or (events)
// the block of cells whose events it takes.
struct PassBlock {
	const DevNet *net;
	uint32_t tile, events;
};
// Per-tile GR pass (cbm_pass_event.cu) with W consumer warps and S stages;
// launched with 32 * (W + 1) threads and (blocks, event CTAs, stepOffset,
// descriptor of a single network or null, MF words, exit counter); oneZone:
// every network has one zone and at most 15 inputs of a kind a cell.  Returns null for a geometry that is not
// compiled in.
const void *passTmaKernelFor(int W, int S, bool oneZone);
// The compiled per-tile geometries, in table order.
int passTmaConfigCount();
void passTmaConfig(int i, int *W, int *S, int *B);
// GR arrays between the reference's order and the per-tile pass's.
__global__ void evOrderKernel(const DevNet *N, const void *src, void *dst, uint32_t size, uint32_t rows, bool toTile);
// Building a network's event tables (numMF + numGO sources): cells per
// (block, source), their prefix sums per block, per-block bases, the lists, and
// the cell-major GR->GO table; and the ring's arrivals after step T.
__global__ void evCountKernel(const DevNet *N, uint32_t *cnt);
__global__ void evScanKernel(uint32_t *cnt, uint32_t nSrc);
__global__ void evBaseKernel(uint32_t *start, uint32_t *next, const uint32_t *base, uint32_t nSrc);
__global__ void evFillKernel(const DevNet *N, uint32_t *next, uint16_t *entry);
__global__ void evUnusedKernel(uint32_t *p, size_t n, uint32_t x);
__global__ void evOutKernel(const DevNet *N, uint4 *outCell, uint4 *outMore, uint32_t *more);
__global__ void goRingFillKernel(const DevNet *N, uint64_t T);
__global__ void conductancesKernel(const DevNet *N, uint64_t T, float *outE, float *outI);
// Persistent single-network TMA GR pass: W consumer warps (2W rows per
// unit), S stages, B resident CTAs per SM, slot bound M; grid of any size,
// 32 * (W + 1) threads, the grPassKernel arguments with one network.
const void *passPersistentKernelFor(int W, int S, int B, int M);
// Vector GR pass (cbm_pass_vec.cu): single network of the compiled shape,
// kVecWarps warps per CTA, arguments (descriptor, stepOffset, units per
// claim), passVecSmemBytes of dynamic shared memory.  The first
// passVecReduceCTAs CTAs take the previous step's PF->PC reduction; the
// others are persistent and claim units of 128 cells from DevNet::passClaim.
constexpr int kVecWarps = 8;
constexpr int kVecMinBlocks = 3;
constexpr uint32_t kVecClaim = 2;
constexpr uint32_t kVecBatchClaim = 8;
constexpr int kVecBatchMinBlocks = 2;
// The batched form (several networks of the shape; arguments nets,
// unitOffset, pcOffset, numNets, stepOffset, claim counters [3]).
const void *passVecBatchKernel();
bool passVecCapable(const DevNet &h);
size_t passVecSmemBytes(const DevNet &h);
uint32_t passVecReduceCTAs(const DevNet &h);
const void *passVecKernel();
// pairReduceKernel(N, t): step t's PF->PC running sums from its pair sums
// (numPC * bs threads), for a switch away from the vector pass.
const void *pairReduceKernelFn();
// pcTreeKernel(N, t): step t's PF->PC input sums (pcSum) from its partial
// sums, one block of 256 threads per PC, for a switch to the vector pass.
const void *pcTreeKernelFn();
// Small-cell update; stageBytes[n] is network n's staging block size (0:
// its microzone CTA works on global memory).  With one network, net0 and
// stage0 give its descriptor and staging size directly (else null, 0).
// ncMailbox (one network, or null): mapped host memory that receives the
// step's NC spikes and then the step number (publishNC).  mfp.n > 0 (one
// network): the step's MF spike words, which the Golgi CTA also writes into
// the MF ring for the kernels after the step.
__global__ void tailKernel(const DevNet *const *nets, const uint32_t *stageBytes, uint32_t stepOffset,
		const DevNet *net0, uint32_t stage0, uint8_t *ncMailbox, const __grid_constant__ MFParam mfp);
__global__ void outCon16Kernel(const uint32_t *in, uint16_t *out, size_t n);
__global__ void protocolPrimeKernel(const DevNet *N);
// The records of step t = stepsDone(N) + 1 + stepOffset, after both kernels of
// that step: ECTrialsData on the first trialBlocks blocks, a cell a thread, then
// the GR peri-stimulus histogram, 8 GR a thread.  May be launched as the
// programmatic dependent of the step's GR pass.
__global__ void recordKernel(const DevNet *N, uint32_t stepOffset, uint32_t trialBlocks);
// All networks of a batch: cellOffset[n] is the first grid thread of network
// n's small cells (cellOffset[numNets] the total).
__global__ void trialDataBatchKernel(const DevNet *const *nets, const uint32_t *cellOffset, int numNets,
		uint32_t stepOffset);
__global__ void advanceStepKernel(uint64_t *const *tBases, int numNets, uint32_t steps);
__global__ void extractSpikesKernel(const uint32_t *apBuf, uint8_t *out, uint32_t n);
__global__ void flushReadKernel(const uint4 *buf, size_t n, uint32_t *sink);
__global__ void expfProbeKernel(const float *in, float *out, uint32_t n);
__global__ void expProbeKernel(const double *in, double *out, uint32_t n);
// The state-variable input's MF rates for row `row` of its values.
__global__ void stateVarRatesKernel(const DevNet *N, uint64_t row, float *out);

}  // namespace cbm
