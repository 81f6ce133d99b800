// Fused PageRank: algorithms::simple_pagerank
// (include/graphblas/algorithms/simple_pagerank.hpp:146-533) as ONE
// persistent cooperative launch with one bounded grid barrier per iteration.
//
// Per iteration the reference pre-scales pr by alpha / outdegree (keeping
// the dangling mass apart), runs vxm over L (a gather over L's CCS), adds the
// teleport + dangling term and measures the L1 change.  Here the CCS gather
// runs on merge-path tiles and its row epilogue does all of the rest for the
// column it just finished: new pr_j, |new - old|, and already the pre-scaled
// input of the NEXT iteration (pr_next, double-buffered) with its dangling
// mass, so the next gather can start right after the barrier.
#include "common.cuh"
#include "merge.cuh"
#include "wmerge.cuh"
#include "persist.cuh"
#include "spmv.cuh"

#include <cmath>
#include <cstddef>

namespace alpb {

using RF = RingPlusTimesF64;

struct PrState {
	GridReduce gr;
	int err;           // a barrier or tile wait gave up
	int64_t iterations;
	double residual;
	int zero_values;   // a stored value of the CRS is zero
};

struct PrArgs {
	MergeTables mt;                // over the CCS
	const int64_t *ccs_ptr;
	const uint32_t *ccs_row;
	const double *ccs_val;
	const int64_t *crs_ptr;
	const double *crs_val;
	double *pr, *rs, *next0, *next1;
	int64_t n, max_iter;
	double alpha, conv;
	int init_given;
	PrState *st;
};

// One block of 16 warps per SM: the iteration of a small graph is its barrier,
// whose cost grows with the blocks (grid_reduce), and a tile or two per warp.
constexpr int PR_WARPS = 16;

struct PrWarpSmem {
	WarpSmem<RF> tile;
	double old_pr[WM_TILE];
	double rs[WM_TILE];
};

struct PrEpi {
	const PrArgs *a;
	PrWarpSmem *sm;
	double *next_out;
	double d;
	int64_t base = 0;
	double acc_res = 0.0, acc_dang = 0.0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) {
			sm->old_pr[k] = __ldcg(a->pr + i0 + k);
			sm->rs[k] = __ldg(a->rs + i0 + k);
		}
	}
	__device__ __forceinline__ void row(int64_t j, double v, bool has) {
		const double nn = has ? 0.0 + v : 0.0;       // pr_nextnext = 0; += pr_next L
		const double old = sm->old_pr[j - base];
		const double nw = nn + d;                    // pr = pr_nextnext + dangling
		a->pr[j] = nw;
		acc_res += old > nw ? old - nw : nw - old;
		const double rsj = sm->rs[j - base];
		if (rsj == 0.0) {                            // input of the next iteration
			next_out[j] = 0.0;
			acc_dang += nw;
		} else {
			next_out[j] = nw * rsj;
		}
	}
};

// *zero = 1 where a stored value is zero: without one, a row's out-degree is
// its length, and the set-up need not walk the rows (a hub row of 1e5 entries
// on one warp took most of its 320 us on a graph of a million rows; this
// streaming pass takes about 20)
__global__ void __launch_bounds__(256) k_pr_zero_values(const double *__restrict__ val,
	const int64_t *__restrict__ ptr, int64_t n, int *zero) {
	const int64_t nnz = ptr[n];
	bool z = false;
	for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nnz;
		 k += int64_t(gridDim.x) * blockDim.x)
		z |= __ldcs(val + k) == 0.0;
	if (__any_sync(0xffffffffu, z) && (threadIdx.x & 31) == 0) *zero = 1;
}

// Row i of the set-up (:224-289 and the initial guess): its scale alpha /
// count, pr, the pre-scaled first input; returns its dangling mass.
template <class Args>
__device__ __forceinline__ double pr_setup_row(const Args &a, int64_t i, double cnt) {
	const double rsi = cnt > 0.0 ? a.alpha / cnt : 0.0;
	a.rs[i] = rsi;
	const double p = a.init_given ? a.pr[i] : 1.0 / double(a.n);
	a.pr[i] = p;
	a.next0[i] = rsi == 0.0 ? 0.0 : p * rsi;
	return rsi == 0.0 ? p : 0.0;
}

// The set-up's rows of this block; the thread's share of the dangling mass.
// zero: some stored value is zero, so the out-degrees are counted (one warp
// per row); otherwise they are the row lengths (one thread per row).
template <class Args>
__device__ __forceinline__ double pr_setup_rows(const Args &a, bool zero) {
	double dang = 0.0;
	const int64_t tid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
	const int64_t nt = int64_t(gridDim.x) * blockDim.x;
	if (!zero) {
		for (int64_t i = tid; i < a.n; i += nt)
			dang += pr_setup_row(a, i, double(a.crs_ptr[i + 1] - a.crs_ptr[i]));
		return dang;
	}
	const int lane = threadIdx.x & 31;
	for (int64_t i = tid >> 5; i < a.n; i += nt >> 5) {
		const int64_t b = a.crs_ptr[i], e = a.crs_ptr[i + 1];
		double cnt = 0.0;
		for (int64_t k = b + lane; k < e; k += 32) cnt += a.crs_val[k] != 0.0 ? 1.0 : 0.0;
		for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
		if (lane == 0) dang += pr_setup_row(a, i, cnt);
	}
	return dang;
}

struct GatherL2 {
	const double *x;
	__device__ __forceinline__ double operator()(uint32_t j) const { return __ldcg(x + j); }
};

// One barrier per iteration, which carries the iteration's two sums (the L1
// change and the dangling mass).
__global__ void __launch_bounds__(32 * PR_WARPS, 1) k_pagerank(PrArgs a) {
	extern __shared__ __align__(16) unsigned char pr_smem[];
	PrWarpSmem *sm = reinterpret_cast<PrWarpSmem *>(pr_smem);   // one per warp
	__shared__ double red[64 * 2];
	PrState *st = a.st;
	int *err = &st->err;
	const int64_t G = gridDim.x, n = a.n, nt = a.mt.ntiles;
	const int w = threadIdx.x >> 5;
	// tiles go round the blocks first, so a small graph uses every SM
	const int64_t gw = int64_t(w) * G + blockIdx.x, nw = G * PR_WARPS;
	unsigned epoch = 0;
	// setup: out-degree counts of nonzero-valued entries (the pattern ring of
	// :224-237), alpha / count (:281-289), initial guess, pre-scaled input
	for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < nt;
		 t += G * blockDim.x)
		a.mt.ready[t] = 0;
	double dang;
	if (!grid_reduce(&st->gr, ++epoch, pr_setup_rows(a, st->zero_values != 0), &dang, red, err))
		return;

	int64_t iter = 0;
	double residual = 0.0;
	double *cur = a.next0, *nxt = a.next1;
	for (;;) {
		const double d = (a.alpha * dang + 1 - a.alpha) / double(n);  // (:390)
		PrEpi epi{&a, &sm[w], nxt, d};
		GatherL2 xl{cur};
		int64_t t = gw;
		WmMeta g = wm_meta(a.mt, t);
		while (t < nt) {
			const WmMeta next = wm_meta(a.mt, t + nw);
			if (!warp_tile_ordered<RF>(t, g, a.mt, a.ccs_ptr, a.ccs_row, a.ccs_val, xl, epi, 1,
					sm[w].tile, int32_t(iter + 1), err))
				break;
			t += nw;
			g = next;
		}
		const double v[2] = {epi.acc_res, epi.acc_dang};
		double sum[2];
		if (!grid_reduce<2>(&st->gr, ++epoch, v, sum, red, err)) return;
		residual = sum[0];
		dang = sum[1];
		++iter;
		if (a.conv != 0.0 && residual <= a.conv) break;   // (:490)
		if (iter >= a.max_iter) break;
		double *tmp = cur;
		cur = nxt;
		nxt = tmp;
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) {
		st->iterations = iter;
		st->residual = residual;
	}
}

// ------------------------------------------------ large graphs: per-step --
// For large graphs one cooperative kernel is the wrong shape: its columns
// that cross warp tiles wait on each other in tile order, and its grid is
// capped at what stays co-resident.  There every iteration is instead
// two ordinary launches -- the product over the CCS with the same row epilogue
// (k_pr_step; a column that crosses tiles leaves per-tile partials), and the
// crossing columns' epilogue (k_pr_fix), whose last block sums the block
// partials in a fixed order and decides whether to stop.
// Iterations are queued in chunks; once the stop is decided every queued
// kernel returns at once, and the host reads the state once per chunk.
constexpr int PRS_WARPS = 4;
constexpr int PRS_CHUNK = 8;

struct PrStepState {
	int64_t iterations;
	double residual, d;
	int done;
	int zero_values;          // a stored value of the CRS is zero
	unsigned int arrived;     // blocks of k_pr_fix that left their partials
};

struct PrStepArgs {
	MergeTables mt;                // over the CCS
	const int64_t *ccs_ptr;
	const uint32_t *ccs_row;
	const double *ccs_val;
	const int64_t *crs_ptr;
	const double *crs_val;
	double *pr, *rs, *next0, *next1;
	double *blk;                   // [2][grid]: residual, dangling of k_pr_step
	double *fix;                   // [2][fix_grid]: the same of k_pr_fix
	int grid, fix_grid;
	int64_t n, max_iter;
	double alpha, conv;
	int init_given;
	PrStepState *st;
};

// Shared memory of a warp of k_pr_step: the compact tile, whose y entries hold
// the rows' old pr, and the scales of the tile's first PRS_RS rows (the others
// are read where they are needed).  3.2 KB instead of 7.2: what is left of the
// SM's memory holds the L1 lines of the gathers in flight.
constexpr int PRS_RS = 64;
struct PrsWarpSmem {
	WarpSmemCompact<RF> tile;
	double rs[PRS_RS];
};

// the row epilogue (old pr and the row scale fetched with the tile)
struct PrStepEpi {
	const PrStepArgs *a;
	PrsWarpSmem *sm;
	double *next_out;
	double d;
	int64_t base = 0;
	double acc_res = 0.0, acc_dang = 0.0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) {
			sm->tile.y(k) = a->pr[i0 + k];
			if (k < PRS_RS) sm->rs[k] = __ldg(a->rs + i0 + k);
		}
	}
	__device__ __forceinline__ void row(int64_t j, double v, bool has) {
		const double nn = has ? 0.0 + v : 0.0;       // pr_nextnext = 0; += pr_next L
		const int q = int(j - base);
		const double old = sm->tile.y(q);
		const double nw = nn + d;                    // pr = pr_nextnext + dangling
		a->pr[j] = nw;
		acc_res += old > nw ? old - nw : nw - old;
		const double rsj = q < PRS_RS ? sm->rs[q] : __ldg(a->rs + j);
		if (rsj == 0.0) {                            // input of the next iteration
			next_out[j] = 0.0;
			acc_dang += nw;
		} else {
			next_out[j] = nw * rsj;
		}
	}
};

struct GatherRO {
	const double *__restrict__ x;
	__device__ __forceinline__ double operator()(uint32_t j) const { return __ldg(x + j); }
};

// set-up of the per-step solve: the rows, and the blocks' dangling mass
__global__ void __launch_bounds__(256) k_pr_setup(PrStepArgs a) {
	__shared__ double red[33];
	const double dang = block_sum(pr_setup_rows(a, a.st->zero_values != 0), red);
	if (threadIdx.x == 0) {
		a.blk[blockIdx.x] = 0.0;
		a.blk[a.grid + blockIdx.x] = dang;
	}
}

// Six blocks of four warps per SM: with 5 / 7 / 8 of them 118 / 121 / 139 us per
// iteration instead of 113 (R-MAT, 1,000,003 vertices; 124 with 7.2 KB a warp).
__global__ void __launch_bounds__(32 * PRS_WARPS, 6) k_pr_step(PrStepArgs a, int parity) {
	if (a.st->done) return;
	__shared__ PrsWarpSmem sm[PRS_WARPS];
	__shared__ double red[33];
	const int w = threadIdx.x >> 5;
	PrStepEpi epi{&a, &sm[w], parity ? a.next0 : a.next1, a.st->d};
	GatherRO xl{parity ? a.next1 : a.next0};
	const int64_t nw = int64_t(gridDim.x) * PRS_WARPS;
	int64_t t = int64_t(blockIdx.x) * PRS_WARPS + w;
	WmMeta g = wm_meta(a.mt, t);
	while (t < a.mt.ntiles) {
		const WmMeta next = wm_meta(a.mt, t + nw);
		warp_tile<RF, GatherRO, PrStepEpi, WarpSmemCompact<RF>, WM_LOADS_FIRST>(t, g, a.mt, a.ccs_ptr, a.ccs_row, a.ccs_val, xl, epi, 0, sm[w].tile);
		t += nw;
		g = next;
	}
	const double s1 = block_sum(epi.acc_res, red);
	const double s2 = block_sum(epi.acc_dang, red);
	if (threadIdx.x == 0) {
		a.blk[blockIdx.x] = s1;
		a.blk[a.grid + blockIdx.x] = s2;
	}
}

// The four sums that close an iteration in one pass: a thread's loads of all
// four arrays are in flight together, and each sum keeps block_sum_array's
// order (the thread's elements in stride order, then block_sum's tree), so the
// values are those of four block_sum_array calls bit for bit.
// setup != 0: the first teleport term only (no iteration has run).
__device__ __forceinline__ void pr_finish_sums(const PrStepArgs &a, int setup,
	double (*smem)[33], double out[4]) {
	double v[4] = {0.0, 0.0, 0.0, 0.0};
	for (int64_t k = threadIdx.x; k < a.grid; k += blockDim.x) {
		v[0] += __ldcg(a.blk + k);
		v[1] += __ldcg(a.blk + a.grid + k);
	}
	if (!setup)
		for (int64_t k = threadIdx.x; k < a.fix_grid; k += blockDim.x) {
			v[2] += __ldcg(a.fix + k);
			v[3] += __ldcg(a.fix + a.fix_grid + k);
		}
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
	for (int q = 0; q < 4; ++q)
		for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
	if (lane == 0)
		for (int q = 0; q < 4; ++q) smem[q][wid] = v[q];
	__syncthreads();
	if (wid == 0) {
		const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			double w = lane < nw ? smem[q][lane] : 0.0;
			for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
			if (lane == 0) smem[q][32] = w;
		}
	}
	__syncthreads();
	for (int q = 0; q < 4; ++q) out[q] = smem[q][32];
}

// One block: the sums, the next teleport term, and whether to stop: after an
// iteration whose residual is <= conv (:490), or at max_iter.
__device__ __forceinline__ void pr_finish(const PrStepArgs &a, int setup) {
	__shared__ double red[4][33];
	PrStepState *st = a.st;
	double sums[4];
	pr_finish_sums(a, setup, red, sums);
	if (threadIdx.x == 0) {
		const double dang = setup ? sums[1] : sums[1] + sums[3];
		st->d = (a.alpha * dang + 1 - a.alpha) / double(a.n);     // (:390)
		if (!setup) {
			st->residual = sums[0] + sums[2];
			st->iterations += 1;
			if ((a.conv != 0.0 && st->residual <= a.conv) || st->iterations >= a.max_iter)
				st->done = 1;
		}
	}
}

__global__ void __launch_bounds__(256) k_pr_first(PrStepArgs a) { pr_finish(a, 1); }

// columns that cross tiles: their partials summed in tile order (tail slots
// of the first..last-1 tiles, head slot of the last), then the epilogue.  A
// lane's column, its old value and scale and its slots are loaded side by
// side: the chain of dependent loads is what bounds this kernel.  The last
// block to leave its partials closes the iteration (no launch of its own).
__global__ void __launch_bounds__(256) k_pr_fix(PrStepArgs a, int parity) {
	if (a.st->done) return;
	__shared__ double red[33];
	__shared__ bool last;
	const MergeTables &mt = a.mt;
	double *next_out = parity ? a.next0 : a.next1;
	const double d = a.st->d;
	double acc_res = 0.0, acc_dang = 0.0;
	// the row epilogue of k_pr_step on column j with old value and scale loaded
	const auto finish = [&](int64_t j, double v, double old, double rsj) {
		const double nw = (0.0 + v) + d;
		a.pr[j] = nw;
		acc_res += old > nw ? old - nw : nw - old;
		next_out[j] = rsj == 0.0 ? 0.0 : nw * rsj;
		if (rsj == 0.0) acc_dang += nw;
	};
	const int lane = threadIdx.x & 31;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	for (int64_t base = warp * 32; base < mt.ntiles; base += nwarps * 32) {
		const int64_t t = base + lane;
		const int32_t n = t < mt.ntiles ? mt.span_len[t] : 0;
		const int64_t j = t < mt.ntiles ? mt.tile_row[t + 1] : 0;
		if (n > 0 && n <= 32) {
			const double old = a.pr[j], rsj = a.rs[j];
			const double head = load_bits<double>(mt.head_val + t + n - 1);
			double v = wm_sum_slots<RF>(0.0, mt.tail_val, t, t + n - 1);
			v += head;
			finish(j, v, old, rsj);
		}
		unsigned long_rows = __ballot_sync(0xffffffffu, n > 32);
		while (long_rows) {
			const int src = __ffs(long_rows) - 1;
			long_rows &= long_rows - 1;
			const int64_t f = base + src;
			const int32_t nn = __shfl_sync(0xffffffffu, n, src);
			const int64_t jj = __shfl_sync(0xffffffffu, j, src);
			double v = wm_sum_slots32<RF>(0.0, mt.tail_val, f + lane, f + nn - 1);
			for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
			if (lane == 0) {
				v += load_bits<double>(mt.head_val + f + nn - 1);
				finish(jj, v, a.pr[jj], a.rs[jj]);
			}
		}
	}
	const double s1 = block_sum(acc_res, red);
	const double s2 = block_sum(acc_dang, red);
	if (threadIdx.x == 0) {
		a.fix[blockIdx.x] = s1;
		a.fix[a.fix_grid + blockIdx.x] = s2;
		__threadfence();
		last = atomicAdd(&a.st->arrived, 1u) == gridDim.x - 1;
		if (last) {
			a.st->arrived = 0;
			__threadfence();
		}
	}
	__syncthreads();
	if (last) pr_finish(a, 0);
}

static int pagerank_steps(const PrStepArgs &tmpl, alpb_spmv_plan plan, int64_t *iterations,
	double *residual, cudaStream_t s) {
	PrStepArgs a = tmpl;
	static int per_sm = 0;
	if (!per_sm) {
		ALPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pr_step,
			32 * PRS_WARPS, 0));
		if (per_sm < 1) per_sm = 1;
	}
	int64_t g = (plan->ntiles + PRS_WARPS - 1) / PRS_WARPS;
	if (g > int64_t(per_sm) * sm_count()) g = int64_t(per_sm) * sm_count();
	a.grid = int(g < 1 ? 1 : g);
	a.fix_grid = int(grid_for((plan->ntiles + 31) / 32 * 32, 256));
	double *part = nullptr;
	PrStepState *st = nullptr;
	ALPB_CUDA(cudaMallocAsync(&part, size_t(2 * a.grid + 2 * a.fix_grid) * 8, s));
	ALPB_CUDA(cudaMallocAsync(&st, sizeof(PrStepState), s));
	ALPB_CUDA(cudaMemsetAsync(st, 0, sizeof(PrStepState), s));
	a.blk = part;
	a.fix = part + 2 * a.grid;
	a.st = st;
	if (a.crs_val) {
		k_pr_zero_values<<<grid_for(plan->nnz, 256), 256, 0, s>>>(a.crs_val, a.crs_ptr, a.n,
			&st->zero_values);
		ALPB_LAUNCHED();
	}
	k_pr_setup<<<a.grid, 256, 0, s>>>(a);
	ALPB_LAUNCHED();
	k_pr_first<<<1, 256, 0, s>>>(a);
	ALPB_LAUNCHED();
	PrStepState h{};
	int64_t queued = 0;
	while (queued < a.max_iter) {
		const int64_t chunk = a.max_iter - queued < PRS_CHUNK ? a.max_iter - queued : PRS_CHUNK;
		for (int64_t k = 0; k < chunk; ++k) {
			const int parity = int((queued + k) & 1);
			k_pr_step<<<a.grid, 32 * PRS_WARPS, 0, s>>>(a, parity);
			ALPB_LAUNCHED();
			k_pr_fix<<<a.fix_grid, 256, 0, s>>>(a, parity);
			ALPB_LAUNCHED();
		}
		queued += chunk;
		ALPB_CUDA(cudaMemcpyAsync(&h, st, sizeof(PrStepState), cudaMemcpyDeviceToHost, s));
		ALPB_CUDA(cudaStreamSynchronize(s));
		if (h.done) break;
	}
	ALPB_CUDA(cudaFreeAsync(part, s));
	ALPB_CUDA(cudaFreeAsync(st, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	*iterations = h.iterations;
	*residual = h.residual;
	if (!(h.residual <= a.conv)) {
		set_error("alpb_pagerank: not converged after %lld iterations (residual %g)",
			(long long) h.iterations, h.residual);
		return ALPB_FAILED;
	}
	return ALPB_SUCCESS;
}

// Graphs from this many nonzeroes on take the per-step launches.  Measured us
// per solve, one kernel against steps, R-MAT: 0.86 M nonzeroes 440 / 557, 1.2 M
// 501 / 496, 2.1 M 750 / 715, 2.9 M 986 / 840, 4.3 M 1358 / 1005.
// On stencils (the CCS plan's tiles hold whole columns) nothing crosses tiles and
// the one kernel has no wait but its barrier: 27-point 1.6 M 608 / 932, 4.6 M
// 1217 / 1426, 8.2 M 1921 / 2001, 13.5 M 3107 / 2992 (40 iterations), 5-point 4 M
// 1400 / 1609, 7.2 M 2270 / 2348, 9.8 M 3003 / 2997.
constexpr int64_t kPrStepNnz = int64_t(1) << 20;
constexpr int64_t kPrStepNnzWhole = int64_t(1) << 23;

// The solve proper.  plan: a WM_TILE plan of the CCS offsets, or null (one is
// made and destroyed here); work: 3n doubles of scratch, or null.
static int pagerank_run(int64_t n, const int64_t *crs_row_ptr, const double *crs_values,
	const int64_t *ccs_col_ptr, const uint32_t *ccs_row_idx, const double *ccs_values, double *pr,
	int init_given, double alpha, double conv, int64_t max_iter, int64_t *iterations,
	double *residual, double *work, alpb_spmv_plan plan, cudaStream_t s) {
	alpb_spmv_plan own_plan = nullptr;
	if (!plan) {
		int64_t nnz = 0;
		ALPB_CUDA(cudaMemcpyAsync(&nnz, ccs_col_ptr + n, 8, cudaMemcpyDeviceToHost, s));
		ALPB_CUDA(cudaStreamSynchronize(s));
		int rc = plan_create_tiles(&own_plan, n, nnz, ccs_col_ptr, ALPB_SCHED_MERGE_PATH, 0,
			WM_TILE, s);
		if (rc != ALPB_SUCCESS) return rc;
		plan = own_plan;
	}
	if (plan->nnz >= (plan->tile_d ? kPrStepNnzWhole : kPrStepNnz)) {
		double *vecs = work, *own_vecs = nullptr;
		if (!vecs) {
			ALPB_CUDA(cudaMallocAsync(&own_vecs, size_t(3 * n) * 8, s));
			vecs = own_vecs;
		}
		PrStepArgs a{};
		a.mt = merge_tables(*plan);
		a.ccs_ptr = ccs_col_ptr;
		a.ccs_row = ccs_row_idx;
		a.ccs_val = ccs_values;
		a.crs_ptr = crs_row_ptr;
		a.crs_val = crs_values;
		a.pr = pr;
		a.rs = vecs;
		a.next0 = vecs + n;
		a.next1 = vecs + 2 * n;
		a.n = n;
		a.max_iter = max_iter;
		a.alpha = alpha;
		a.conv = conv;
		a.init_given = init_given;
		const int rc = pagerank_steps(a, plan, iterations, residual, s);
		if (own_vecs) {
			cudaFreeAsync(own_vecs, s);
			cudaStreamSynchronize(s);
		}
		alpb_spmv_plan_destroy(own_plan);
		return rc;
	}
	const size_t smem = sizeof(PrWarpSmem) * PR_WARPS;
	static std::atomic<unsigned long long> allowed_in;
	const cudaError_t allowed = allow_smem(k_pagerank, smem, allowed_in);
	if (allowed != cudaSuccess) {
		alpb_spmv_plan_destroy(own_plan);
		set_error("alpb_pagerank: %s", cudaGetErrorString(allowed));
		return ALPB_PANIC;
	}
	const int sms = sm_count() < GRID_REDUCE_BLOCKS ? sm_count() : GRID_REDUCE_BLOCKS;
	const int grid = cooperative_grid(k_pagerank, 32 * PR_WARPS, smem, sms);
	if (grid <= 0) {
		alpb_spmv_plan_destroy(own_plan);
		set_error("alpb_pagerank: no cooperative occupancy");
		return ALPB_PANIC;
	}
	double *vecs = work, *own_vecs = nullptr;
	PrState *st = nullptr;
	if (!vecs) {
		ALPB_CUDA(cudaMallocAsync(&own_vecs, size_t(3 * n) * 8, s));
		vecs = own_vecs;
	}
	ALPB_CUDA(cudaMallocAsync(&st, sizeof(PrState), s));
	ALPB_CUDA(cudaMemsetAsync(st, 0, sizeof(PrState), s));
	PrArgs a;
	a.mt = merge_tables(*plan);
	a.ccs_ptr = ccs_col_ptr;
	a.ccs_row = ccs_row_idx;
	a.ccs_val = ccs_values;
	a.crs_ptr = crs_row_ptr;
	a.crs_val = crs_values;
	a.pr = pr;
	a.rs = vecs;
	a.next0 = vecs + n;
	a.next1 = vecs + 2 * n;
	a.n = n;
	a.max_iter = max_iter;
	a.alpha = alpha;
	a.conv = conv;
	a.init_given = init_given;
	a.st = st;
	if (crs_values) {
		k_pr_zero_values<<<grid_for(plan->nnz, 256), 256, 0, s>>>(crs_values, crs_row_ptr, n,
			&st->zero_values);
		ALPB_LAUNCHED();
	}
	void *args[] = {&a};
	ALPB_CUDA(cudaLaunchCooperativeKernel((void *) k_pagerank, dim3(grid), dim3(32 * PR_WARPS), args,
		smem, s));
	ALPB_LAUNCHED();
	PrState h;
	ALPB_CUDA(cudaMemcpyAsync(&h.err, &st->err, sizeof(PrState) - offsetof(PrState, err),
		cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(st, s));
	if (own_vecs) ALPB_CUDA(cudaFreeAsync(own_vecs, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	alpb_spmv_plan_destroy(own_plan);
	ALPB_CHECK(h.err == 0, ALPB_PANIC, "alpb_pagerank: a grid barrier or tile wait timed out");
	*iterations = h.iterations;
	*residual = h.residual;
	if (!(h.residual <= conv)) {
		set_error("alpb_pagerank: not converged after %lld iterations (residual %g)",
			(long long) h.iterations, h.residual);
		return ALPB_FAILED;
	}
	return ALPB_SUCCESS;
}

static int pagerank_checks(int64_t n, double alpha, int64_t max_iter, const int64_t *iterations,
	const double *residual) {
	ALPB_CHECK(alpha > 0 && alpha < 1, ALPB_ILLEGAL, "alpb_pagerank: alpha must be in (0, 1)");
	ALPB_CHECK(max_iter > 0, ALPB_ILLEGAL, "alpb_pagerank: max must be positive");
	ALPB_CHECK(iterations && residual, ALPB_ILLEGAL, "alpb_pagerank: null output");
	ALPB_CHECK(n > 0, ALPB_ILLEGAL, "alpb_pagerank: empty graph");
	return ALPB_SUCCESS;
}

} // namespace alpb

using namespace alpb;

extern "C" int alpb_pagerank(int64_t n, const int64_t *crs_row_ptr, const uint32_t *crs_col_idx,
	const double *crs_values, const int64_t *ccs_col_ptr, const uint32_t *ccs_row_idx,
	const double *ccs_values, double *pr, int init_given, double alpha, double conv,
	int64_t max_iter, int64_t *iterations, double *residual, void *stream) {
	(void) crs_col_idx;
	const int rc = pagerank_checks(n, alpha, max_iter, iterations, residual);
	if (rc != ALPB_SUCCESS) return rc;
	return pagerank_run(n, crs_row_ptr, crs_values, ccs_col_ptr, ccs_row_idx, ccs_values, pr,
		init_given, alpha, conv, max_iter, iterations, residual, nullptr, nullptr,
		as_stream(stream));
}

extern "C" int alpb_pagerank_planned(int64_t n, const int64_t *crs_row_ptr,
	const uint32_t *crs_col_idx, const double *crs_values, const int64_t *ccs_col_ptr,
	const uint32_t *ccs_row_idx, const double *ccs_values, double *pr, int init_given,
	double alpha, double conv, int64_t max_iter, int64_t *iterations, double *residual,
	double *work, alpb_spmv_plan ccs_plan, void *stream) {
	(void) crs_col_idx;
	const int rc = pagerank_checks(n, alpha, max_iter, iterations, residual);
	if (rc != ALPB_SUCCESS) return rc;
	ALPB_CHECK(!ccs_plan || (ccs_plan->m == n && ccs_plan->offsets == ccs_col_ptr &&
			ccs_plan->tile == WM_TILE), ALPB_MISMATCH,
		"alpb_pagerank_planned: plan was made for another storage");
	return pagerank_run(n, crs_row_ptr, crs_values, ccs_col_ptr, ccs_row_idx, ccs_values, pr,
		init_given, alpha, conv, max_iter, iterations, residual, work, ccs_plan,
		as_stream(stream));
}
