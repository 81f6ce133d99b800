// Persistent (cooperative) kernel support: a grid barrier whose every wait is
// bounded, and a deterministic block reduction.
#pragma once
#include "common.cuh"

namespace alpb {

// Barrier state in device memory; zero-initialise before the launch.  The
// arrival counter only grows: barrier k of the launch completes when it
// reaches k * gridDim.x, so no block resets it and no second word is flipped.
// The counter and the error flag sit on separate 128-byte lines.
struct alignas(128) GridSync {
	unsigned long long count;
	unsigned int pad0[30];
	unsigned int gen;   // not used by grid_sync (kept for the layout)
	int err;    // 1: a barrier or tile wait gave up (the kernel exits; host reports PANIC)
	unsigned int pad1[30];
};

// A few seconds of polls (each an L2 round trip of about 0.2 us; grid_reduce
// waits an eighth of that): far beyond any legitimate wait of a co-resident
// grid, short enough to keep the context usable on a fault.
constexpr long long kSpinLimit = 1ll << 24;

// All blocks of a cooperative launch call this the same number of times.
// Thread 0 arrives with one acquire-release add (its block's writes before
// the barrier are released; the last arrival acquires everyone's) and the
// others poll the counter with acquire loads until their barrier's target,
// so the last block to arrive goes on after one atomic round trip and the
// others one poll later.  Returns false once any block has timed out; callers
// then leave their loop.
__device__ __forceinline__ bool grid_sync(GridSync *gs) {
	__syncthreads();
	int bad = 0;
	if (threadIdx.x == 0) {
		const unsigned long long G = gridDim.x;
		unsigned long long old;
		asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;"
					 : "=l"(old) : "l"(&gs->count) : "memory");
		const unsigned long long target = (old / G + 1) * G;
		volatile int *verr = &gs->err;
		for (long long spins = 0;; ++spins) {
			// the error flag's load is in flight with the counter's: read after
			// the barrier it cost every thread one more L2 round trip
			const int e = *verr;
			unsigned long long c;
			asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
						 : "=l"(c) : "l"(&gs->count) : "memory");
			bad = e;
			if (c >= target || bad) break;
			if (spins > kSpinLimit) {
				atomicExch(&gs->err, 1);
				bad = 1;
				break;
			}
		}
	}
	return !__syncthreads_or(bad);
}

// Sum over the block in a fixed order (warp trees, then warp 0 over the warp
// sums); the result is returned to every thread.
__device__ __forceinline__ double block_sum(double v, double *smem /* >= 33 */) {
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
	__syncthreads();
	if (lane == 0) smem[wid] = v;
	__syncthreads();
	if (wid == 0) {
		const int nw = (blockDim.x + 31) >> 5;
		double w = lane < nw ? smem[lane] : 0.0;
		for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
		if (lane == 0) smem[32] = w;
	}
	__syncthreads();
	return smem[32];
}

// Every block sums the same array in the same order (same value everywhere).
__device__ __forceinline__ double block_sum_array(const double *a, int64_t n, double *smem) {
	double v = 0.0;
	for (int64_t k = threadIdx.x; k < n; k += blockDim.x) v += ((const volatile double *) a)[k];
	return block_sum(v, smem);
}

// Grid barrier and sum in one: every block leaves its partial beside the
// counter and the blocks read all partials once the counter is complete.
// What bounds it is latency across the chip: about 700 cycles for the atomic
// (300-700 by the die that holds the line), 300-400 each for a poll and for
// the partials.  Measured with 148 blocks of 512 threads, fences included:
// 2.0 us; value-carrying slots polled by every block took 3.8 us (the polls
// contend with the stores), pushed to every block's own lines 2.9 us, and
// gathered and broadcast by one block 3.1 us.
constexpr int GRID_REDUCE_BLOCKS = 256;
constexpr int GRID_REDUCE_VALUES = 2;
struct alignas(128) GridReduce {
	unsigned long long count;
	unsigned int pad[30];
	// [epoch parity][value][block]
	double part[2][GRID_REDUCE_VALUES][GRID_REDUCE_BLOCKS];
};

// All threads call, with epoch = 1, 2, ... ; v: this thread's terms of NV sums;
// sum: the grid's totals in a fixed order (lanes, warps, blocks), the same bits
// in every thread.  Needs gridDim.x <= min(blockDim.x, GRID_REDUCE_BLOCKS), *g
// zeroed before the launch.  Global writes of any block before the call are
// visible to plain loads of all after it.  false: a wait gave up (*err is set).
template <int NV>
__device__ __forceinline__ bool grid_reduce(GridReduce *g, unsigned epoch, const double (&v)[NV],
	double (&sum)[NV], double *smem /* >= 64 NV */, int *err) {
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int nwarps = blockDim.x >> 5, G = gridDim.x;
	double(*part)[GRID_REDUCE_BLOCKS] = g->part[epoch & 1];
#pragma unroll
	for (int q = 0; q < NV; ++q) {
		double t = v[q];
		for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
		if (lane == 0) smem[64 * q + w] = t;
	}
	__syncthreads();
	int bad = 0;
	if (w == 0) {
#pragma unroll
		for (int q = 0; q < NV; ++q) {
			double t = lane < nwarps ? smem[64 * q + lane] : 0.0;
			for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
			if (lane == 0) part[q][blockIdx.x] = t;
		}
		if (lane == 0) {
			unsigned long long c;
			asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;"
						 : "=l"(c) : "l"(&g->count) : "memory");
			const unsigned long long target = (unsigned long long) epoch * G;
			for (long long spins = 0;; ++spins) {
				asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
							 : "=l"(c) : "l"(&g->count) : "memory");
				if (c >= target) break;
				if ((spins & 255) == 255 && *reinterpret_cast<volatile int *>(err)) bad = 1;
				if (spins > kSpinLimit / 8) {
					atomicExch(err, 1);
					bad = 1;
				}
				if (bad) break;
			}
		}
	}
	if (__syncthreads_or(bad)) return false;
	const int gw = (G + 31) >> 5;
	if (w < gw) {
		double t[NV];
#pragma unroll
		for (int q = 0; q < NV; ++q) t[q] = int(threadIdx.x) < G ? __ldcg(part[q] + threadIdx.x) : 0.0;
#pragma unroll
		for (int q = 0; q < NV; ++q) {
			for (int o = 16; o > 0; o >>= 1) t[q] += __shfl_xor_sync(0xffffffffu, t[q], o);
			if (lane == 0) smem[64 * q + 32 + w] = t[q];
		}
	}
	__syncthreads();
#pragma unroll
	for (int q = 0; q < NV; ++q) {
		double r = 0.0;
		for (int k = 0; k < gw; ++k) r += smem[64 * q + 32 + k];
		sum[q] = r;
	}
	return true;
}

// One sum.
__device__ __forceinline__ bool grid_reduce(GridReduce *g, unsigned epoch, double v, double *sum,
	double *smem, int *err) {
	const double in[1] = {v};
	double out[1];
	const bool ok = grid_reduce<1>(g, epoch, in, out, smem, err);
	*sum = out[0];
	return ok;
}

// Largest grid of `kernel` whose blocks are all co-resident.
template <class K>
int cooperative_grid(K kernel, int block, size_t smem, int64_t want) {
	int per_sm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess)
		return 0;
	int64_t g = int64_t(per_sm) * sm_count();
	if (want > 0 && want < g) g = want;
	return int(g);
}

// Grid of a persistent solver kernel over `ntiles` warp tiles: about four
// tiles per warp, at least two blocks per SM (latency hiding), at most the
// co-resident maximum.  Every grid barrier and every scalar reduction costs
// time in proportion to the block count, so small systems get small grids.
template <class K>
int solver_grid(K kernel, int block, int64_t ntiles, int warps_per_block, size_t smem = 0) {
	const int max_grid = cooperative_grid(kernel, block, smem, 0);
	int64_t g = ntiles / (4 * int64_t(warps_per_block));
	if (g < 2 * int64_t(sm_count())) g = 2 * int64_t(sm_count());
	if (g > max_grid) g = max_grid;
	return int(g);
}

} // namespace alpb
