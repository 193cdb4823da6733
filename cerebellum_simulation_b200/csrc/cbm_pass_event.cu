// The per-tile GR pass: event-driven synapses beside a streamed cell update.
//
// A granule cell's membrane state changes every step and has to be streamed
// (54 bytes a cell: six 4-byte state arrays in and out, the PF->PC weight, the
// PF delay, the arrived spikes), but its synapses matter only when a spike
// arrives: about 1 % of the MF, 1-12 % of the GO and 0.1-3 % of the GR spike
// in a step.  So the synapse tables are not streamed.  They are kept by source:
//   MF->GR and GO->GR: per block of evCells cells, each source's list of
//     target cells (evStart, evEntry).  An event CTA walks the lists of the
//     step's spiking sources and counts into half a byte per cell and kind (a
//     byte with more than 15 inputs of a kind) in shared memory; the counts are the integers the per-cell gather of
//     kernels.cu:169-199 gives.
//   GR->GO: a cell's spike adds its synapses to the counts of the step they
//     arrive in, t + delay, in a ring of kGoRing steps (outCell).  The
//     reference tests every delay bit of every cell in the step of arrival
//     (kernels.cu:112-167); the integer counts are the same.
// Neither is waited for: the counts enter the conductances that the next step
// reads, so the next pass applies them when it loads the conductances, and a
// spike recorded by one pass is delivered by the next, before any of its
// synapses is due.
//
// While this pass runs, the GR arrays are in tile order (evCell): a tile's
// cells are consecutive, so a CTA streams a few long pieces by bulk copies.
//
// What bounds it: on up to 1M GR, latency (a CTA's prologue, its 2-4 rounds and
// its sums, 11-13 us beside the small-cell kernel's 11); beyond, the streaming
// (53 us of the dense 4M network's 67 us step, 38 of them the bytes at the measured
// copy bandwidth) and there the Golgi CTA beside it.
// Streaming the tables instead (14 B of indices and 8-16 B of GR->GO slots a
// cell, with seven gathers and four delay tests), a step took 93 us on the
// dense 4M-GR network (here 67), 92 us on 64 networks of 16K GR, whose 128-cell
// tiles were prologue only (33), 83 us on six of 256K-2M (62), 15.6 us on 1M GR
// (13.1).  Other homes for the lists that were measured: each CTA's
// own 2048 cells (a GO's list has 1.5 cells there on the 4M network: as long
// again as the streaming), and counts in global memory (random reductions there
// slow the streaming stores: 29 us a step on the 1M network).
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "cbm_device.cuh"
#include "cbm_kernels.cuh"
#include "cbm_tma.cuh"

namespace cbm {

constexpr uint64_t kPassWaitLimitNs = 2000000000ull;

__device__ __forceinline__ void raisePassError(const DevNet *N)
{
	// mapped host memory, one error kind: a plain store (see errFlag)
	*reinterpret_cast<volatile uint32_t *>(N->errFlag) = kErrPassWait;
	__threadfence_system();
}

// (x >> d) & 1, and 0 for d >= 32 (kNoDelay): PTX shifts clamp.
__device__ __forceinline__ uint32_t delayedBit(uint32_t x, uint32_t d)
{
	uint32_t r;
	asm("shr.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(d));
	return r & 1u;
}

// The reference's number of the cell at index p in tile order, and back.
__device__ __forceinline__ uint32_t evCell(const DevNet *N, uint32_t p)
{
	const uint32_t TC = N->evRows << N->evWdShift, tile = p / TC, local = p % TC;
	return ((tile / N->evTilesX) * N->evRows + (local >> N->evWdShift)) * N->bs +
		((tile % N->evTilesX) << N->evWdShift) + (local & ((1u << N->evWdShift) - 1u));
}
__device__ __forceinline__ uint32_t evIndex(const DevNet *N, uint32_t g)
{
	const uint32_t row = g / N->bs, col = g % N->bs, wd = 1u << N->evWdShift;
	return (((row / N->evRows) * N->evTilesX + (col >> N->evWdShift)) * N->evRows + row % N->evRows) * wd + (col & (wd - 1u));
}

// Count one arriving spike for each of eight cells (unused entries lead to a
// dummy behind the cells) in one byte a cell; inc: 1 for an MF spike, 16 for a
// GO one.
__device__ __forceinline__ void countCells(uint8_t *sCnt, const uint4 &e, uint32_t inc)
{
	const uint32_t p[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
	for (int k = 0; k < 4; k++) {
		atomicAdd(reinterpret_cast<uint32_t *>(sCnt + (p[k] & 0xFFFCu)), inc << ((p[k] << 3) & 24u));
		atomicAdd(reinterpret_cast<uint32_t *>(sCnt + ((p[k] >> 16) & 0xFFFCu)), inc << ((p[k] >> 13) & 24u));
	}
}

// Event CTA `block` of network N in step t: the spikes that arrive at cells
// [block evCells, + evCells) in this step.  Bound by latency (spike words and
// lists are dependent round trips of 1-1.5 us beside the streaming CTAs) and by
// the instructions of a few warps (about six a counted cell): so the lists of a
// usual step are taken in one round, as many lanes an item as a usual list has
// eights of cells (up to eight; a longer list is several items), eight items a group
// of lanes in flight (ten: 75 KB of code instead of 71, a 1M-GR step 0.2-0.4 us
// slower).  Its time grows with the sources that spike, where streaming the tables
// did not: with all Golgi cells spiking a step takes 10.3 us on 16K GR, 16.4 on 256K,
// 23.5 on 1M and 103 on dense 4M (streaming: 12, 12, 13 and 81), with 20 % of them
// 10.8, 11.4, 13.7 and 62.6 (12, 12, 15 and 83).
// WIDE: the network may have two planes of counts.
template <bool WIDE>
__device__ __forceinline__ void eventRole(const DevNet *__restrict__ N, uint64_t t, uint32_t block, uint8_t *smem, const MFParam &mfp)
{
	constexpr uint32_t U = 8;
	const uint32_t tid = threadIdx.x, nThr = blockDim.x, lane = tid & 31u;
	uint32_t *ctr = reinterpret_cast<uint32_t *>(smem);          // items
	const uint32_t evCells = N->evCells;
	const uint32_t planes = WIDE ? N->evPlanes : 1u, plane = evCells + 16u;
	uint8_t *sCnt = smem + 16;                                   // [planes][evCells, a dummy behind]
	uint32_t *sItem = reinterpret_cast<uint32_t *>(sCnt + planes * plane);  // [kEvListCap] source | item << 20
	// where a GO spike counts, and as what
	uint8_t *const sCntGO = planes == 2u ? sCnt + plane : sCnt;
	const uint32_t incGO = planes == 2u ? 1u : 16u;
	const uint32_t numMF = N->numMF, numGO = N->numGO, numGR = N->numGR;
	const uint32_t mfWords = N->mfWords, nWords = mfWords + N->goWords;
	const uint32_t *mfSrc = N->mfBits + (size_t)stepMod(t - 1, N->mfRing) * mfWords;
	const uint32_t *goSrc = N->goBits + (size_t)((t - 1) & 1) * N->goWords;
	const uint32_t *const start = N->evStart + (size_t)block * eventStartWords(numMF + numGO);
	const uint4 *const entry = N->evEntry;
	const uint32_t laneShift = N->evLaneShift, lanes = 1u << laneShift, l = tid & (lanes - 1u);
	const uint32_t cells = min(evCells, numGR - block * evCells), perMF = N->evPerMF, perGO = N->evPerGO;
	// the block's list starts on their way to shared memory beside the spike words
	// (one dependent round trip less), where they are few enough
	uint32_t *const sStart = sItem + kEvListCap;
	const uint32_t nStart = eventStartWords(numMF + numGO);
	const bool staged = nStart <= kEvStartCap;
	if (staged)
#pragma unroll 1
		for (uint32_t i = 4u * tid; i < nStart; i += 4u * nThr)
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tma::smemAddr(sStart + i)), "l"(start + i) : "memory");
	for (uint32_t w0 = 0; w0 < nWords; w0 += nThr) {
		// a thread a word; MF words come from the launch when it carries them
		const uint32_t w = w0 + tid;
		const bool go = w >= mfWords;
		const uint32_t x0 = 32u * (go ? w - mfWords : w), xs = go ? numGO : numMF, per = go ? perGO : perMF;
		uint32_t word = w >= nWords ? 0u : go ? __ldg(goSrc + (w - mfWords)) : mfp.n ? mfp.w[w] : __ldg(mfSrc + w);
		// bits past the last source are no spikes
		if (w < nWords && xs - x0 < 32u) word &= (1u << (xs - x0)) - 1u;
		if (tid == 0) *ctr = 0;
		if (w0 == 0)
			for (uint32_t i = tid; i < planes * (plane / 16u); i += nThr) reinterpret_cast<uint4 *>(sCnt)[i] = make_uint4(0, 0, 0, 0);
		__syncthreads();
		for (;;) {
			const uint32_t mine = per * (uint32_t)__popc(word);
			uint32_t at = mine;  // prefix sum over the warp
#pragma unroll
			for (uint32_t o = 1; o < 32u; o *= 2) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, at, o);
				if (lane >= o) at += y;
			}
			uint32_t base = 0;
			if (lane == 31u && at) base = atomicAdd(ctr, at);
			at += __shfl_sync(0xffffffffu, base, 31) - mine;
			const uint32_t src0 = go ? numMF + x0 : x0;
			const bool fits = at + mine <= kEvListCap;
			// a lane lists its word's spikes; where some word has many, the warp takes
			// the words in turn, a lane a bit (a lane alone stores 32 times, all lanes to
			// one bank: 10,000 cycles a round with every source spiking)
			if (__any_sync(0xffffffffu, fits && __popc(word) > 4)) {
				for (uint32_t pend = __ballot_sync(0xffffffffu, fits && word); pend; pend &= pend - 1u) {
					const uint32_t k = (uint32_t)__ffs((int)pend) - 1u;
					const uint32_t wk = __shfl_sync(0xffffffffu, word, k), sk = __shfl_sync(0xffffffffu, src0, k);
					const uint32_t pk = __shfl_sync(0xffffffffu, per, k), ak = __shfl_sync(0xffffffffu, at, k);
					if ((wk >> lane) & 1u) {
						uint32_t *const o = sItem + ak + pk * (uint32_t)__popc(wk & ((1u << lane) - 1u));
#pragma unroll 1
						for (uint32_t q = 0; q < pk; q++) o[q] = (sk + lane) | (q << 20);
					}
				}
				if (fits) word = 0;
			} else if (fits) {
#pragma unroll 1
				for (; word; word &= word - 1u)
#pragma unroll 1
					for (uint32_t q = 0; q < per; q++) sItem[at++] = (src0 + (uint32_t)__ffs((int)word) - 1u) | (q << 20);
			}
			if (!fits) {
				// a word whose items do not fit waits for another round (kEvListCap
				// holds those of one word)
				for (; at < kEvListCap; at++) sItem[at] = kEvNone;
			}
			if (staged) asm volatile("cp.async.wait_all;" ::: "memory");
			const bool again = __syncthreads_or(word != 0);
			const uint32_t n = min(*ctr, kEvListCap);
			const uint32_t groups = nThr >> laneShift, grp = tid >> laneShift;
			for (uint32_t i0 = grp; i0 < n; i0 += U * groups) {
				uint32_t a[U], b[U], gos = 0, lasts = 0;
				uint4 e[U];
#pragma unroll
				for (uint32_t u = 0; u < U; u++) {
					const uint32_t i = i0 + u * groups;
					a[u] = b[u] = 0;
					const uint32_t x = i < n ? sItem[i] : kEvNone;
					if (x != kEvNone) {
						const uint32_t src = x & 0xFFFFFu, q = x >> 20;
						if (src >= numMF) gos |= 1u << u;
						if (q + 1u == (src >= numMF ? perGO : perMF)) lasts |= 1u << u;
						a[u] = (staged ? sStart[src] : __ldg(start + src)) + (q << laneShift) + l;
						b[u] = staged ? sStart[src + 1u] : __ldg(start + src + 1u);
					}
				}
#pragma unroll
				for (uint32_t u = 0; u < U; u++)
					if (a[u] < b[u]) e[u] = __ldg(entry + a[u]);
#pragma unroll
				for (uint32_t u = 0; u < U; u++) {
					if (a[u] >= b[u]) continue;
					const bool isGO = (gos >> u) & 1u;
					const uint32_t inc = isGO ? incGO : 1u;
					uint8_t *const cnt = WIDE && isGO ? sCntGO : sCnt;
					countCells(cnt, e[u], inc);
					// a list's last item takes what is left of it
					if ((lasts >> u) & 1u)
						for (a[u] += lanes; a[u] < b[u]; a[u] += lanes) countCells(cnt, __ldg(entry + a[u]), inc);
				}
			}
			__syncthreads();
			if (!again) break;
			if (tid == 0) *ctr = 0;
			__syncthreads();
		}
	}
	// the counts, for the next pass
	for (uint32_t q = 0; q < planes; q++) {
		uint4 *const out = reinterpret_cast<uint4 *>(N->evCnt + (size_t)((t & 1) * planes + q) * numGR + (size_t)block * evCells);
		for (uint32_t i = tid; i < cells / 16u; i += nThr) out[i] = reinterpret_cast<const uint4 *>(sCnt + q * plane)[i];
	}
}

// One warp of a streaming CTA: the GR->GO synapses of its tile's cells that
// spiked in the last step, into the steps they arrive in (none is due before
// this step).  pump() is called between the dependent round trips.
template <typename Pump>
__device__ __forceinline__ void deliverSpikes(const DevNet *__restrict__ N, uint64_t t, uint32_t cell0, uint32_t TC,
		uint16_t *sCell, Pump pump)
{
	const uint32_t lane = threadIdx.x & 31u, numGO = N->numGO;
	const uint32_t *const spk = N->spkBits + (size_t)((t - 1) & 1) * (N->numGR / 32u) + cell0 / 32u;
	for (uint32_t w0 = 0; w0 < TC / 32u; w0 += 64u) {
		uint32_t c[2], n = 0;
#pragma unroll
		for (uint32_t u = 0; u < 2u; u++) {
			c[u] = w0 + lane + 32u * u < TC / 32u ? __ldg(spk + w0 + lane + 32u * u) : 0u;
			n += (uint32_t)__popc(c[u]);
		}
		uint32_t at = n;  // prefix sum over the warp
#pragma unroll
		for (uint32_t o = 1; o < 32u; o *= 2) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, at, o);
			if (lane >= o) at += y;
		}
		const uint32_t total = __shfl_sync(0xffffffffu, at, 31);
		at -= n;
		for (uint32_t from = 0; from < total; from += kEvCellCap) {
#pragma unroll
			for (uint32_t u = 0; u < 2u; u++) {
				const uint32_t w = w0 + 32u * u + lane;
				// bit b of word w: cell 4 b + w mod 4 of the run of 128 cells w / 4
				for (; c[u] && at < from + kEvCellCap; c[u] &= c[u] - 1u, at++)
					sCell[at - from] = (uint16_t)(128u * (w >> 2) + 4u * ((uint32_t)__ffs((int)c[u]) - 1u) + (w & 3u));
			}
			__syncwarp();
			const uint32_t m = min(total - from, kEvCellCap);
			for (uint32_t i0 = lane; i0 - lane < m; i0 += 96u) {
				uint4 o[3];
#pragma unroll
				for (uint32_t u = 0; u < 3u; u++) {
					o[u] = make_uint4(kNoDelay, kNoDelay, kNoDelay, kNoDelay);
					if (i0 + 32u * u < m) o[u] = __ldg(N->outCell + cell0 + sCell[i0 + 32u * u]);
				}
				pump();
#pragma unroll
				for (uint32_t u = 0; u < 3u; u++) {
					for (;;) {
						const uint32_t q[4] = {o[u].x, o[u].y, o[u].z, o[u].w};
#pragma unroll
						for (int k = 0; k < 4; k++) {
							const uint32_t dl = q[k] & 0xFFu;
							if (dl < 32u) atomicAdd(&N->goCount[(size_t)((t - 1 + dl) & (kGoRing - 1u)) * numGO + (q[k] >> 8)], 1u);
						}
						if ((q[3] & 0xFFu) != kOutMore) break;
						o[u] = __ldg(N->outMore + (q[3] >> 8));
					}
				}
			}
			__syncwarp();
		}
	}
}

// The float of byte c of x (a small count): exact, without the conversion unit.
template <int c> __device__ __forceinline__ float byteFloat(uint32_t x)
{
	return __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7540u | c)) - 8388608.0f;
}

// Streaming CTAs: one per tile, the whole reduction columns (2K rows) of
// 1 << evWdShift thread indices j of one or several PCs, in stages of 128 W
// cells.  W consumer warps update 128 cells of a stage each, four consecutive
// cells a lane, so that every state array is one 16-byte access; the last warp
// copies the stages in bulk into an S-deep ring and delivers the tile's spikes of
// the last step.  The launch's first CTAs take the event role: evBlocks of them
// with one network, those marked in `blocks` in a batch.
// Waits are bounded (kPassWaitLimitNs); a time-out sets kErrPassWait.
// ZS: the number of zones, with one plane of counts, or 0 to read both at run time.
template <int W, int S, int MINB, int ZS>
__global__ void __launch_bounds__(32 * (W + 1), MINB) grPassTmaKernel(const PassBlock *blocks, uint32_t evBlocks,
		uint32_t stepOffset, const DevNet *net0, const __grid_constant__ MFParam mfp, uint32_t *exitCount)
{
	// the next step's small-cell kernel may launch (it waits for this pass)
	pdlLaunchDependents();
	constexpr uint32_t SC = 128u * W;
	constexpr uint32_t ZMAX = ZS ? ZS : kMaxZones;
	constexpr uint32_t nThr = 32u * W;
	const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	// one network: its descriptor comes as a parameter (a round trip fewer)
	uint32_t tile = blockIdx.x - evBlocks;
	bool events = blockIdx.x < evBlocks;
	const DevNet *__restrict__ N = net0;
	if (!N) {
		const PassBlock pb = blocks[blockIdx.x];
		N = pb.net;
		tile = pb.tile;
		events = pb.events != 0;
	} else if (events) {
		tile = blockIdx.x;
	}
	// the whole descriptor into L1 in one round trip: its fields are read all
	// over the kernel, each first touch of a line a round trip of its own
	if (tid < (uint32_t)(offsetof(DevNet, zones) + ZMAX * sizeof(DevZone) + 127) / 128u) {
		uint32_t x;
		asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(x) : "l"(reinterpret_cast<const char *>(N) + 128u * tid));
	}
	extern __shared__ uint8_t passSmemRaw[];
	uint8_t *const smem = passSmemRaw + ((128u - (tma::smemAddr(passSmemRaw) & 127u)) & 127u);
	if (events) {
		eventRole<ZS == 0>(N, stepsDone(N) + 1 + stepOffset, tile, smem, mfp);
		if (exitCount) __syncthreads();
		passExitWait(exitCount);
		return;
	}
	uint64_t *full = reinterpret_cast<uint64_t *>(smem);  // stage landed
	uint64_t *empty = full + S;                           // stage updated (W consumers)
	static_assert(16 * S <= (int)kEvBarBytes, "barriers");
	if (tid == 0) {
		for (int s = 0; s < S; s++) {
			tma::mbarInit(&full[s], 1);
			tma::mbarInit(&empty[s], W);
		}
		tma::fenceBarrierInit();
	}
	__syncthreads();

	const uint64_t t = stepsDone(N) + 1 + stepOffset;
	const uint32_t Z = ZS ? ZS : N->numZones, rowsPC = 2u * N->K, wdShift = N->evWdShift, Wd = 1u << wdShift;
	const uint32_t TC = N->evRows << wdShift, nStages = TC / SC;
	const uint32_t planes = ZS ? 1u : N->evPlanes;
	const EventLayout L = eventLayout(SC, Z, planes);
	const EventSmem M = eventSmem(min((uint32_t)S, nStages), L.bytes, TC, Z, N->evPCs, N->evBC + N->evSC);
	float *sStep = reinterpret_cast<float *>(smem + M.step);      // [evPCs][Z] plasticity steps
	uint32_t *sBC = reinterpret_cast<uint32_t *>(smem + M.bc);
	uint32_t *sSC = sBC + N->evBC;
	uint32_t *sSpk = reinterpret_cast<uint32_t *>(smem + M.spk);  // [TC / 128][4]: cell 4 lane + c of a run spiked
	float *sX = reinterpret_cast<float *>(smem + M.x);            // [Z][TC] PF->PC outputs x
	uint8_t *const stages = smem + M.stages;
	const bool plastStep = stepMod(t, N->tsPerHistBinGR) == 0;
	// rows per PC and tiles side by side are powers of two
	const uint32_t pcShift = (uint32_t)__ffs((int)rowsPC) - 1u, txShift = (uint32_t)__ffs((int)N->evTilesX) - 1u;
	const uint32_t row0 = (tile >> txShift) * N->evRows, x0 = (tile & (N->evTilesX - 1u)) << wdShift;
	const uint32_t pc0 = row0 >> pcShift, bs = N->bs;
	const uint32_t cell0 = tile * TC;  // the tile's first cell
	const uint32_t bcShift = N->bcShift, scShift = N->scShift;
	const uint32_t bcBase = (row0 * bs) >> bcShift, scBase = (row0 * bs) >> scShift;

	if (warp == W) {
		bool ok = true;
		uint32_t issued = 0;
		const uint8_t *const evCnt = N->evCnt + (size_t)((t - 1) & 1) * planes * N->numGR;
		auto issue = [&]() {  // the next stage
			if (lane == 0) {
				uint8_t *b = stages + (size_t)(issued % S) * L.bytes;
				uint64_t *bar = &full[issued % S];
				const uint32_t c = cell0 + issued * SC;
				tma::arriveExpectTx(bar, L.tx);
				tma::loadBulk(b, N->vGR + c, 4u * SC, bar);
				tma::loadBulk(b + 4u * SC, N->gKCaGR + c, 4u * SC, bar);
				tma::loadBulk(b + 8u * SC, N->threshGR + c, 4u * SC, bar);
				tma::loadBulk(b + 12u * SC, N->gESum + c, 4u * SC, bar);
				tma::loadBulk(b + 16u * SC, N->gISum + c, 4u * SC, bar);
				tma::loadBulk(b + 20u * SC, N->apBufGR + c, 4u * SC, bar);
				for (uint32_t z = 0; z < Z; z++) tma::loadBulk(b + L.w + z * 4u * SC, N->zones[z].w + c, 4u * SC, bar);
				tma::loadBulk(b + L.pfDelay, N->evPfDelay + c, SC, bar);
				tma::loadBulk(b + L.cnt, evCnt + c, SC, bar);
				if (planes == 2u) tma::loadBulk(b + L.cnt + SC, evCnt + N->numGR + c, SC, bar);
			}
			issued++;
		};
		while (issued < nStages && issued < (uint32_t)S) issue();
		for (uint32_t i = lane; i < N->evBC + N->evSC; i += 32u) sBC[i] = 0;
		if (plastStep)
			for (uint32_t i = lane; i < N->evPCs * Z; i += 32u) {
				const uint32_t z = i % Z, pc = pc0 + i / Z;
				sStep[i] = plasticityStep(N, t, z, N->zones[z].plastSel[(t & 1) * N->numIO + N->zones[z].ioOfPC[pc]]);
			}
		// the consumers' first stage needs the counters and steps set
		asm volatile("bar.arrive 1, %0;" ::"r"(nThr + 32u) : "memory");
		// refill the ring as its slots come free (they are only read, so no
		// proxy fence is needed)
		auto pump = [&]() {
			while (issued < nStages) {
				const uint32_t prev = issued - S;
				if (!__all_sync(0xffffffffu, tma::tryWait(&empty[prev % S], (prev / S) & 1u))) break;
				issue();
			}
		};
		if (!N->outNow) deliverSpikes(N, t, cell0, TC, reinterpret_cast<uint16_t *>(smem + M.cells), pump);
		while (issued < nStages) {
			const uint32_t prev = issued - S;
			ok = __all_sync(0xffffffffu, tma::waitBounded(&empty[prev % S], (prev / S) & 1u, kPassWaitLimitNs));
			if (!ok) break;
			issue();
		}
		if (!ok && lane == 0) {
			raisePassError(N);
			// let the copies in flight land before the CTA's shared memory is released
			for (uint32_t st = issued > (uint32_t)S ? issued - S : 0; st < issued; st++)
				tma::waitBounded(&full[st % S], (st / S) & 1u, kPassWaitLimitNs);
		}
	} else {
		// ---- consumers
		const float gLeak = N->gLeakGR, eLeak = N->eLeakGR, eGOIn = N->eGOGR;
		const float threshBase = N->threshRestGR, threshMax = N->threshMaxGR, threshDecay = N->threshDecGR;
		const float gDecMF = N->gDecMFtoGR, gIncMF = N->gIncMFtoGR, gDecGO = N->gDecGOtoGR, gIncGO = N->gIncGOtoGR;
		const float threshMax0 = 0.0f * threshMax;
		float *const vGR = N->vGR, *const gKCaGR = N->gKCaGR, *const threshGR = N->threshGR;
		float *const gESum = N->gESum, *const gISum = N->gISum;
		uint32_t *const apBufGR = N->apBufGR;
		uint64_t *const historyGR = N->historyGR;
		// the first pass of a run finds conductances with nothing to add
		const bool pending = t != N->evFirst;
		const uint32_t e = tid * 4u;  // first of the lane's four cells within a stage
		asm volatile("bar.sync 1, %0;" ::"r"(nThr + 32u) : "memory");
		bool ready = true;
		for (uint32_t st = 0; st < nStages; st++) {
			const uint8_t *const b = stages + (size_t)(st % S) * L.bytes;
			const uint32_t local = st * SC + e, g = cell0 + local;  // within the tile, and in the GR arrays
			uint64_t h[4] = {0, 0, 0, 0};
			if (plastStep) {
				const ulonglong2 ha = *reinterpret_cast<const ulonglong2 *>(historyGR + g);
				const ulonglong2 hb = *reinterpret_cast<const ulonglong2 *>(historyGR + g + 2);
				h[0] = ha.x; h[1] = ha.y; h[2] = hb.x; h[3] = hb.y;
			}
			ready = __all_sync(0xffffffffu, tma::waitBounded(&full[st % S], (st / S) & 1u, kPassWaitLimitNs));
			if (!ready) break;
			const float4 v4 = *reinterpret_cast<const float4 *>(b + 4u * e);
			const float4 gk4 = *reinterpret_cast<const float4 *>(b + 4u * SC + 4u * e);
			const float4 th4 = *reinterpret_cast<const float4 *>(b + 8u * SC + 4u * e);
			const float4 gE4 = *reinterpret_cast<const float4 *>(b + 12u * SC + 4u * e);
			const float4 gI4 = *reinterpret_cast<const float4 *>(b + 16u * SC + 4u * e);
			const uint4 ab4 = *reinterpret_cast<const uint4 *>(b + 20u * SC + 4u * e);
			const uint32_t c4 = *reinterpret_cast<const uint32_t *>(b + L.cnt + e);
			const uint32_t d4 = *reinterpret_cast<const uint32_t *>(b + L.pfDelay + e);
			const float vI[4] = {v4.x, v4.y, v4.z, v4.w}, gkI[4] = {gk4.x, gk4.y, gk4.z, gk4.w};
			const float thI[4] = {th4.x, th4.y, th4.z, th4.w};
			float gE[4] = {gE4.x, gE4.y, gE4.z, gE4.w}, gI[4] = {gI4.x, gI4.y, gI4.z, gI4.w};
			const uint32_t abI[4] = {ab4.x, ab4.y, ab4.z, ab4.w};
			// updateGRInOPGPU of the last step: its MF spikes, and the GO
			// spikes of the one before (kernels.cu:169-199)
			if (pending) {
				uint32_t mf = c4 & 0x0F0F0F0Fu, go = (c4 >> 4) & 0x0F0F0F0Fu;
				if (planes == 2u) {
					mf = c4;
					go = *reinterpret_cast<const uint32_t *>(b + L.cnt + SC + e);
				}
				gE[0] = gE[0] * gDecMF + gIncMF * byteFloat<0>(mf); gI[0] = gI[0] * gDecGO + gIncGO * byteFloat<0>(go);
				gE[1] = gE[1] * gDecMF + gIncMF * byteFloat<1>(mf); gI[1] = gI[1] * gDecGO + gIncGO * byteFloat<1>(go);
				gE[2] = gE[2] * gDecMF + gIncMF * byteFloat<2>(mf); gI[2] = gI[2] * gDecGO + gIncGO * byteFloat<2>(go);
				gE[3] = gE[3] * gDecMF + gIncMF * byteFloat<3>(mf); gI[3] = gI[3] * gDecGO + gIncGO * byteFloat<3>(go);
				*reinterpret_cast<float4 *>(gESum + g) = make_float4(gE[0], gE[1], gE[2], gE[3]);
				*reinterpret_cast<float4 *>(gISum + g) = make_float4(gI[0], gI[1], gI[2], gI[3]);
			}
			float vO[4], gkO[4], thO[4];
			uint32_t abO[4], pf[4];
			bool ap[4];
#pragma unroll
			for (int c = 0; c < 4; c++) {
				const float v = vI[c], gk = gkI[c], th = thI[c];
				// calcActivityGRGPU (kernels.cu:79-110)
				const float tempV = v + (gLeak + gk * gk * gk * gk) * (eLeak - v) - (gE[c]) * v + (gI[c]) * (eGOIn - v);
				const float tempThresh = th + (threshBase - th) * threshDecay;
				ap[c] = tempV > tempThresh;
				// The reference's ap * a + (!ap) * b on a 0/1 ap, value for value
				// (infinities and NaN make NaN through 0 * x), but selecting
				// where it multiplies: ap ? a + 0 b : 0 a + b.
				thO[c] = ap[c] ? threshMax + 0.0f * tempThresh : threshMax0 + tempThresh;
				// here 0 b and 0 a are +0 or NaN (b = -0: 0 a + b = +0)
				const float gkd = gk * 0.9999f;
				gkO[c] = (ap[c] ? gkd + 0.003f : gkd) + fabsf(0.0f * gkd);
				vO[c] = tempV;
				abO[c] = abI[c] + abI[c] + (ap[c] ? 1u : 0u);
				pf[c] = delayedBit(abO[c], (d4 >> (8 * c)) & 0xFFu);
			}
			*reinterpret_cast<float4 *>(vGR + g) = make_float4(vO[0], vO[1], vO[2], vO[3]);
			*reinterpret_cast<float4 *>(gKCaGR + g) = make_float4(gkO[0], gkO[1], gkO[2], gkO[3]);
			*reinterpret_cast<float4 *>(threshGR + g) = make_float4(thO[0], thO[1], thO[2], thO[3]);
			*reinterpret_cast<uint4 *>(apBufGR + g) = make_uint4(abO[0], abO[1], abO[2], abO[3]);
			// plasticity (phase 1, kernels.cu:282-291) before this step's PF->PC
			// output (phase 2)
#pragma unroll
			for (uint32_t z = 0; z < ZMAX; z++) {
				if (z >= Z) break;
				const float4 w4 = *reinterpret_cast<const float4 *>(b + L.w + 4u * (z * SC + e));
				float w[4] = {w4.x, w4.y, w4.z, w4.w};
				if (plastStep) {
					const float stepW = sStep[(local >> (wdShift + pcShift)) * Z + z];
#pragma unroll
					for (int c = 0; c < 4; c++) {
						w[c] = w[c] + ((h[c] & 0x0000008000000000ull) > 0) * stepW;
						w[c] = (w[c] > 0) * w[c];
						w[c] = (w[c] > 1) + (w[c] <= 1) * w[c];
					}
					*reinterpret_cast<float4 *>(N->zones[z].w + g) = make_float4(w[0], w[1], w[2], w[3]);
				}
				// w * pf of a 0/1 pf
#pragma unroll
				for (int c = 0; c < 4; c++) w[c] = pf[c] ? w[c] : w[c] * 0.0f;
				*reinterpret_cast<float4 *>(sX + z * TC + local) = make_float4(w[0], w[1], w[2], w[3]);
			}
			if (plastStep) {
				// updateGRHistory (kernels.cu:241-246)
#pragma unroll
				for (int c = 0; c < 4; c++) h[c] = (h[c] << 1) | ((abO[c] & 0x0000001Fu) > 0);
				*reinterpret_cast<ulonglong2 *>(historyGR + g) = make_ulonglong2(h[0], h[1]);
				*reinterpret_cast<ulonglong2 *>(historyGR + g + 2) = make_ulonglong2(h[2], h[3]);
			}
			// the run's spikes, one word per cell of a lane; the ballots also
			// order the lanes' accesses to the stage before its release
			const uint32_t k0 = __ballot_sync(0xffffffffu, ap[0]), k1 = __ballot_sync(0xffffffffu, ap[1]);
			const uint32_t k2 = __ballot_sync(0xffffffffu, ap[2]), k3 = __ballot_sync(0xffffffffu, ap[3]);
			__syncwarp();
			if (lane == 0) {
				tma::arrive(&empty[st % S]);
				*reinterpret_cast<uint4 *>(sSpk + local / 32u) = make_uint4(k0, k1, k2, k3);
			}
			// PF->BC and PF->SC counts (kernels.cu:247-260): a lane's four cells
			// share a block when blocks hold four or more
			const uint32_t pfSum = pf[0] + pf[1] + pf[2] + pf[3];
			if (pfSum) {
				// the reference's number of the lane's first cell
				const uint32_t r = (row0 + (local >> wdShift)) * bs + x0 + (local & (Wd - 1u));
				if (bcShift >= 2) atomicAdd(&sBC[(r >> bcShift) - bcBase], pfSum);
				if (scShift >= 2) atomicAdd(&sSC[(r >> scShift) - scBase], pfSum);
				if (bcShift < 2 || scShift < 2)
#pragma unroll
					for (uint32_t c = 0; c < 4; c++) {
						if (bcShift < 2 && pf[c]) atomicAdd(&sBC[((r + c) >> bcShift) - bcBase], 1u);
						if (scShift < 2 && pf[c]) atomicAdd(&sSC[((r + c) >> scShift) - scBase], 1u);
					}
			}
		}
		if (!ready && lane == 0) raisePassError(N);
	}
	__syncthreads();

	// the running sums of the PF->PC reduction (sumInputsNew's per-thread
	// tempSum += x[i] + x[i+bs], kernels.cu:326-362), a thread per j of a PC
	const uint32_t buf = (uint32_t)(t % 3);
	for (uint32_t i = tid; i < (TC >> pcShift) * Z; i += nThr + 32u) {
		const uint32_t z = ZS == 1 ? 0u : i / (TC >> pcShift), c = ZS == 1 ? i : i % (TC >> pcShift);
		const uint32_t pc = c >> wdShift, j = c & (Wd - 1u);
		const float *x = sX + z * TC + ((pc << pcShift) << wdShift) + j;
		float sum = 0;
#pragma unroll 8
		for (uint32_t k = 0; k < rowsPC; k += 2) sum += x[k << wdShift] + x[(k + 1u) << wdShift];
		N->zones[z].pcPartial[((size_t)buf * N->numPC + pc0 + pc) * bs + x0 + j] = sum;
	}
	// the BC and SC counts of the tile
	uint32_t *bcOut = N->bcCount + (size_t)buf * N->numBC;
	uint32_t *scOut = N->scCount + (size_t)buf * N->numSC;
	for (uint32_t i = tid; i < N->evBC + N->evSC; i += blockDim.x) {
		const uint32_t c = sBC[i];
		if (!c) continue;
		if (i < N->evBC) atomicAdd(&bcOut[bcBase + i], c);
		else atomicAdd(&scOut[scBase + i - N->evBC], c);
	}
	// its spiking cells, for the next step's pass; delivered at once in
	// networks with synapses that have no delay
	for (uint32_t i = tid; i < TC / 32u; i += blockDim.x) {
		uint32_t v = sSpk[i];
		N->spkBits[(size_t)(t & 1) * (N->numGR / 32u) + cell0 / 32u + i] = v;
		if (!N->outNow) continue;
		for (; v; v &= v - 1u) {
			const uint32_t cell = cell0 + 128u * (i >> 2) + 4u * ((uint32_t)__ffs((int)v) - 1u) + (i & 3u);
			const uint32_t g = evCell(N, cell);
			for (uint32_t s = 0; s < N->nOutSlots; s++) {
				const uint32_t o = N->outCon[(size_t)s * N->numGR + g], dl = o & 0xFFu;
				if (dl < 32u) atomicAdd(&N->goCount[(size_t)((t + dl) & (kGoRing - 1u)) * N->numGO + (o >> 8)], 1u);
			}
		}
	}
	if (exitCount) __syncthreads();
	passExitWait(exitCount);
}

// ----------------------------------------------------------- tile order
// rows arrays of numGR elements of `size` bytes (1, 2, 4 or 8) from tile order
// to the reference's order (toTile: back).  A tile's rows are at least 32
// consecutive cells in both.
__global__ void evOrderKernel(const DevNet *N, const void *src, void *dst, uint32_t size, uint32_t rows, bool toTile)
{
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t numGR = N->numGR;
	if (i >= (uint64_t)numGR * rows) return;
	const uint64_t base = i / numGR * numGR;
	const uint64_t p = base + (uint32_t)(i % numGR), g = base + evCell(N, (uint32_t)(i % numGR));
	const uint64_t from = toTile ? g : p, to = toTile ? p : g;
	if (size == 4) ((uint32_t *)dst)[to] = ((const uint32_t *)src)[from];
	else if (size == 8) ((uint64_t *)dst)[to] = ((const uint64_t *)src)[from];
	else if (size == 2) ((uint16_t *)dst)[to] = ((const uint16_t *)src)[from];
	else ((uint8_t *)dst)[to] = ((const uint8_t *)src)[from];
}

// The conductances after step T, which the per-tile pass leaves for its next
// step to make: outE, outI (may be the state arrays themselves), in tile order.
__global__ void conductancesKernel(const DevNet *N, uint64_t T, float *outE, float *outI)
{
	const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= N->numGR) return;
	const uint8_t *cnt = N->evCnt + (size_t)(T & 1) * N->evPlanes * N->numGR + p;
	const uint32_t c = *cnt;
	const int mf = (int)(N->evPlanes == 2u ? c : c & 15u), go = (int)(N->evPlanes == 2u ? cnt[N->numGR] : c >> 4);
	if (outE) outE[p] = N->gESum[p] * N->gDecMFtoGR + N->gIncMFtoGR * (mf);
	if (outI) outI[p] = N->gISum[p] * N->gDecGOtoGR + N->gIncGOtoGR * (go);
}

// Geometries the host can pick: (consumer warps, stages, minimum resident CTAs
// per SM).  The first that fits is the default.  Four stages serve tiles of four
// stages and more whose state streams from HBM, eight warps the largest tiles, two
// and one warp tiles below 512 cells, which four cannot take.
#define CBM_PASS_TMA_CONFIGS(X) X(4, 2, 4) X(4, 4, 4) X(8, 3, 2) X(2, 4, 4) X(1, 4, 4)

int passTmaConfigCount()
{
	int n = 0;
#define CBM_PASS_TMA_COUNT(w, d, b) n++;
	CBM_PASS_TMA_CONFIGS(CBM_PASS_TMA_COUNT)
#undef CBM_PASS_TMA_COUNT
	return n;
}

void passTmaConfig(int i, int *W, int *S, int *B)
{
	int k = 0;
#define CBM_PASS_TMA_NTH(w, d, b) if (k++ == i) { *W = w; *S = d; *B = b; return; }
	CBM_PASS_TMA_CONFIGS(CBM_PASS_TMA_NTH)
#undef CBM_PASS_TMA_NTH
}

const void *passTmaKernelFor(int W, int S, bool oneZone)
{
#define CBM_PASS_TMA_PICK(w, d, b) \
	if (W == w && S == d) \
		return oneZone ? (const void *)&grPassTmaKernel<w, d, b, 1> : (const void *)&grPassTmaKernel<w, d, b, 0>;
	CBM_PASS_TMA_CONFIGS(CBM_PASS_TMA_PICK)
#undef CBM_PASS_TMA_PICK
	return nullptr;
}

// ------------------------------------------------------- event tables
// cnt[block][source] += 1 for every MF->GR and GO->GR synapse.
__global__ void evCountKernel(const DevNet *N, uint32_t *cnt)
{
	const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= N->numGR) return;
	uint32_t *c = cnt + (size_t)(evIndex(N, g) / N->evCells) * eventStartWords(N->numMF + N->numGO);
	for (uint32_t s = 0; s < N->nMFSlots; s++) {
		const uint32_t i = N->mfIdx[(size_t)s * N->numGR + g];
		if (i < N->numMF) atomicAdd(&c[i], 1u);
	}
	for (uint32_t s = 0; s < N->nGOSlots; s++) {
		const uint32_t i = N->goIdx[(size_t)s * N->numGR + g];
		if (i < N->numGO) atomicAdd(&c[N->numMF + i], 1u);
	}
}

// One CTA of 256 threads per block of cells: counts -> list starts within the
// block, in groups of eight entries (the exclusive prefix sums of
// ceil(count / 8)); the block's total at the end of its row.
__global__ void evScanKernel(uint32_t *cnt, uint32_t nSrc)
{
	__shared__ uint32_t part[256];
	uint32_t *c = cnt + (size_t)blockIdx.x * eventStartWords(nSrc);
	const uint32_t per = (nSrc + 255u) / 256u, from = threadIdx.x * per, to = min(nSrc, from + per);
	uint32_t sum = 0;
	for (uint32_t i = from; i < to; i++) sum += (c[i] + 7u) / 8u;
	part[threadIdx.x] = sum;
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t run = 0;
		for (uint32_t k = 0; k < 256u; k++) { const uint32_t x = part[k]; part[k] = run; run += x; }
		c[nSrc] = run;
	}
	__syncthreads();
	uint32_t run = part[threadIdx.x];
	for (uint32_t i = from; i < to; i++) { const uint32_t n = (c[i] + 7u) / 8u; c[i] = run; run += n; }
}

// start[block][*] += base[block], and next = the list's first entry.
__global__ void evBaseKernel(uint32_t *start, uint32_t *next, const uint32_t *base, uint32_t nSrc)
{
	uint32_t *c = start + (size_t)blockIdx.x * eventStartWords(nSrc), *k = next + (size_t)blockIdx.x * eventStartWords(nSrc);
	for (uint32_t i = threadIdx.x; i <= nSrc; i += blockDim.x) {
		c[i] += base[blockIdx.x];
		k[i] = 8u * c[i];
	}
}

// n words set to x.
__global__ void evUnusedKernel(uint32_t *p, size_t n, uint32_t x)
{
	for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = x;
}

// Every synapse's target cell (within its block) into its source's list (the
// order within a list does not matter: the pass counts).
__global__ void evFillKernel(const DevNet *N, uint32_t *next, uint16_t *entry)
{
	const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= N->numGR) return;
	const uint32_t p = evIndex(N, g);
	uint32_t *c = next + (size_t)(p / N->evCells) * eventStartWords(N->numMF + N->numGO);
	for (uint32_t s = 0; s < N->nMFSlots; s++) {
		const uint32_t i = N->mfIdx[(size_t)s * N->numGR + g];
		if (i < N->numMF) entry[atomicAdd(&c[i], 1u)] = (uint16_t)(p % N->evCells);
	}
	for (uint32_t s = 0; s < N->nGOSlots; s++) {
		const uint32_t i = N->goIdx[(size_t)s * N->numGR + g];
		if (i < N->numGO) entry[atomicAdd(&c[N->numMF + i], 1u)] = (uint16_t)(p % N->evCells);
	}
}

// Rows of four that the synapses of a cell beyond its own row take: a row holds
// three and the index of the next, the last one up to four.
__device__ __forceinline__ uint32_t outRows(uint32_t n) { return n <= 4u ? 0u : n <= 7u ? 1u : 1u + (n - 7u + 2u) / 3u; }

// outCell and outMore from the slot-major table: every GR->GO synapse that has
// a delay.  With outCell null, the rows of outMore that takes, in *more; else
// *more counts them up from 0.
__global__ void evOutKernel(const DevNet *N, uint4 *outCell, uint4 *outMore, uint32_t *more)
{
	const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= N->numGR) return;
	const uint32_t g = evCell(N, p), slots = N->nOutSlots;
	uint32_t n = 0;
	for (uint32_t s = 0; s < slots; s++) n += (N->outCon[(size_t)s * N->numGR + g] & 0xFFu) < 32u;
	uint32_t rows = outRows(n), next = rows ? atomicAdd(more, rows) : 0u;
	if (!outCell) return;
	uint4 *row = outCell + p;
	uint32_t q[4] = {kNoDelay, kNoDelay, kNoDelay, kNoDelay}, k = 0;
	for (uint32_t s = 0; s < slots; s++) {
		const uint32_t c = N->outCon[(size_t)s * N->numGR + g];
		if ((c & 0xFFu) >= 32u) continue;
		if (k == 3u && rows) {
			// more than one is left: the row's last entry leads on
			*row = make_uint4(q[0], q[1], q[2], (next << 8) | kOutMore);
			row = outMore + next++;
			rows--;
			q[0] = q[1] = q[2] = q[3] = kNoDelay;
			k = 0;
		}
		q[k++] = c;
	}
	*row = make_uint4(q[0], q[1], q[2], q[3]);
}

// The GR->GO arrivals of the steps after step T that earlier spikes cause
// (bits of the spike buffers younger than their synapse's delay): what the
// event-driven pass would have put into the ring by now.
__global__ void goRingFillKernel(const DevNet *N, uint64_t T)
{
	const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= N->numGR) return;
	const uint32_t ab = N->apBufGR[g];
	if (!ab) return;
	for (uint32_t s = 0; s < N->nOutSlots; s++) {
		const uint32_t c = N->outCon[(size_t)s * N->numGR + g], dl = c & 0xFFu;
		if (dl >= 32u) continue;
		// bit b: a spike of step T - b, which arrives at step T - b + dl
		for (uint32_t m = dl ? ab & (0xFFFFFFFFu >> (32u - dl)) : 0u; m; m &= m - 1u) {
			const uint32_t b = (uint32_t)__ffs((int)m) - 1u;
			atomicAdd(&N->goCount[(size_t)((T + dl - b) & (kGoRing - 1u)) * N->numGO + (c >> 8)], 1u);
		}
	}
}

}  // namespace cbm
