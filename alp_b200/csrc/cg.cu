// Fused conjugate gradient: algorithms::preconditioned_conjugate_gradient,
// unpreconditioned branch (include/graphblas/algorithms/conjugate_gradient.hpp:
// 191-483), as ONE persistent cooperative launch.
//
// The reference makes, per iteration, one mxv and nine passes over n-vectors
// with three host-visible dot products.  Here an iteration is two phases
// separated by a bounded grid barrier, with every scalar kept on the device:
//
//   A: temp = A u_new, gathering u_new_j = r_j + gamma u_old_j on the fly
//      (warp merge-path tiles, wmerge.cuh); the row epilogue writes temp_i
//      and u_new_i and forms the terms of beta = temp . u_new.
//   B: alpha = sigma / beta; x += alpha u_new; r -= alpha temp; r . r.
//
// The u update of the reference (u = r + (r.r / sigma) u, :455-468) is thus
// folded into the next SpMV's gather.  r and u are stored side by side, one
// 16-byte pair per row, so that the gather of a nonzero is ONE load (one L1
// wavefront) that brings both; phase A writes u_new to its own array, which
// phase B folds back into the pairs, so no block overwrites a pair that
// another block still gathers.  Convergence is tested exactly as the
// reference does (sqrt(r.r) < tol * ||b||, :437), and the returned residual
// is r.r.  Work space: pairs (2n doubles), u_new (n), temp (n); on return
// its first n doubles hold the final residual vector r.
#include "common.cuh"
#include "merge.cuh"
#include "wmerge.cuh"
#include "persist.cuh"
#include "spmv.cuh"

#include <cmath>

namespace alpb {

using RF = RingPlusTimesF64;

struct CgState {
	GridSync gs;
	int64_t iterations;
	double residual;
	double tol_abs;
	int converged;
};

} // namespace alpb

#include "cg_rows.cuh"

namespace alpb {

struct CgArgs {
	MergeTables mt;
	const int64_t *offsets;
	const uint32_t *indices;
	const double *values;
	const double *b;
	double *x;
	double2 *pr;   // (r_i, u_i)
	double *u_new, *temp;
	double *r_out; // the first n doubles of the work space: r on return
	double *blk;  // [4][grid] block partials: prelude r.r, prelude b.b, beta, r.r
	int64_t n, max_iter;
	double tol;
	CgState *st;
};

// Warps per block: 16 for systems of few tiles (every warp then holds about
// one tile, so the latency of a phase is that of one tile), 8 otherwise.
// Measured on B200, us per iteration (27-point grids): 32^3 -- 25.4 with 4
// warps, 18.5 with 8, 16.5 with 16; 64^3 -- 58.3, 56.7, 61.1.
constexpr int64_t CG_FEW_TILES = 8192;

// Shared memory of one warp: the tile engine's staging plus the epilogue's
// prefetched vector entries for the rows that end in the tile.
struct CgWarpSmem {
	WarpSmem<RF> tile;
	double p0[WM_TILE];
	double p1[WM_TILE];
};

struct PreludeEpi {
	const CgArgs *a;
	CgWarpSmem *sm;
	int64_t base = 0;
	double acc_rr = 0.0, acc_bb = 0.0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) sm->p0[k] = a->b[i0 + k];
	}
	__device__ __forceinline__ void row(int64_t i, double v, bool has) {
		const double t = has ? 0.0 + v : 0.0;      // temp = 0; temp += A x
		const double bi = sm->p0[i - base];
		const double ri = (0.0 + bi) - t;           // r = 0; r += b; r -= temp
		a->pr[i] = make_double2(ri, 0.0);            // u = 0: gamma = 0 takes u = r
		acc_rr += ri * ri;
		acc_bb += bi * bi;
	}
};

struct GatherU {
	const double2 *pr;
	double gamma;
	// the pairs were written by other blocks before the last barrier: read
	// them through L2 (ld.global.cg) so no stale L1 line can be hit
	__device__ __forceinline__ double operator()(uint32_t j) const {
		const double2 p = __ldcg(pr + j);
		return p.x + gamma * p.y;
	}
};

struct IterEpi {
	const CgArgs *a;
	CgWarpSmem *sm;
	double gamma;
	int64_t base = 0;
	double acc = 0.0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) {
			const double2 p = __ldcg(a->pr + i0 + k);
			sm->p0[k] = p.x;
			sm->p1[k] = p.y;
		}
	}
	__device__ __forceinline__ void row(int64_t i, double v, bool has) {
		const double t = has ? 0.0 + v : 0.0;      // temp = 0; temp += A u
		a->temp[i] = t;
		const double un = sm->p0[i - base] + gamma * sm->p1[i - base];
		a->u_new[i] = un;
		acc += t * un;
	}
};

// Rows are finished by fixed tiles (warp_tile_ordered) and every partial is
// reduced in a fixed order (lane terms in tile order, block_sum, then the
// block partials in block order): the iterates are deterministic for a given
// grid size.
template <int CG_WARPS>
__global__ void __launch_bounds__(32 * CG_WARPS, 24 / CG_WARPS) k_cg(CgArgs a) {
	extern __shared__ __align__(16) unsigned char cg_smem[];
	CgWarpSmem *sm = reinterpret_cast<CgWarpSmem *>(cg_smem);  // one per warp
	__shared__ double red[33];
	CgState *st = a.st;
	int *err = &st->gs.err;
	const int64_t G = gridDim.x;
	const int64_t nt = a.mt.ntiles;
	const int w = threadIdx.x >> 5;
	const int64_t gw = int64_t(blockIdx.x) * CG_WARPS + w, nw = G * CG_WARPS;
	double *blk_rr0 = a.blk, *blk_bb0 = a.blk + G, *blk_beta = a.blk + 2 * G,
		   *blk_rr = a.blk + 3 * G;
	for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < nt;
		 t += G * blockDim.x)
		a.mt.ready[t] = 0;
	if (!grid_sync(&st->gs)) return;
	int32_t epoch = 0;

	// prelude: r = b - A x, u = r (by gamma = 0 below), sigma = r.r, |b|^2
	{
		PreludeEpi epi{&a, &sm[w]};
		PlainX<double> xl{a.x};
		++epoch;
		int64_t t = gw;
		WmMeta g = wm_meta(a.mt, t);
		while (t < nt) {
			const WmMeta next = wm_meta(a.mt, t + nw);
			if (!warp_tile_ordered<RF>(t, g, a.mt, a.offsets, a.indices, a.values, xl, epi, 0,
					sm[w].tile, epoch, err))
				break;
			t += nw;
			g = next;
		}
		const double s1 = block_sum(epi.acc_rr, red);
		const double s2 = block_sum(epi.acc_bb, red);
		if (threadIdx.x == 0) {
			blk_rr0[blockIdx.x] = s1;
			blk_bb0[blockIdx.x] = s2;
		}
	}
	if (!grid_sync(&st->gs)) return;
	double sigma = block_sum_array(blk_rr0, G, red);
	const double bnorm = block_sum_array(blk_bb0, G, red);
	const double tol_abs = a.tol * sqrt(bnorm);

	const int64_t chunk = (a.n + G - 1) / G;
	const int64_t rb = blockIdx.x * chunk;
	const int64_t re = rb + chunk < a.n ? rb + chunk : a.n;
	double gamma = 0.0;
	double rr = 0.0;
	int64_t iter = 0;
	for (;;) {
		++iter;
		// phase A: temp = A u_new, u_new = r + gamma u_old, beta terms
		{
			IterEpi epi{&a, &sm[w], gamma};
			GatherU xl{a.pr, gamma};
			++epoch;
			int64_t t = gw;
			WmMeta g = wm_meta(a.mt, t);
			while (t < nt) {
				const WmMeta next = wm_meta(a.mt, t + nw);
				if (!warp_tile_ordered<RF>(t, g, a.mt, a.offsets, a.indices, a.values, xl, epi, 0,
						sm[w].tile, epoch, err))
					break;
				t += nw;
				g = next;
			}
			const double s = block_sum(epi.acc, red);
			if (threadIdx.x == 0) blk_beta[blockIdx.x] = s;
		}
		if (!grid_sync(&st->gs)) return;
		// phase B: alpha = sigma / beta, x += alpha u, r -= alpha temp, r.r
		const double beta = block_sum_array(blk_beta, G, red);
		const double alpha = sigma / beta;
		double part = 0.0;
		for (int64_t i = rb + threadIdx.x; i < re; i += blockDim.x) {
			const double un = __ldcg(a.u_new + i);
			a.x[i] = a.x[i] + alpha * un;
			const double ri = __ldcg(a.pr + i).x - alpha * __ldcg(a.temp + i);
			a.pr[i] = make_double2(ri, un);
			part += ri * ri;
		}
		part = block_sum(part, red);
		if (threadIdx.x == 0) blk_rr[blockIdx.x] = part;
		if (!grid_sync(&st->gs)) return;
		rr = block_sum_array(blk_rr, G, red);
		if (sqrt(rr) < tol_abs || iter >= a.max_iter) break;
		gamma = rr / sigma;  // alpha = beta / sigma in the reference's naming
		sigma = rr;
	}
	// r out to the first n doubles of the work space, which the pairs occupy:
	// through temp, with a barrier between reading the pairs and overwriting them
	for (int64_t i = rb + threadIdx.x; i < re; i += blockDim.x) a.temp[i] = __ldcg(a.pr + i).x;
	if (!grid_sync(&st->gs)) return;
	for (int64_t i = rb + threadIdx.x; i < re; i += blockDim.x) a.r_out[i] = __ldcg(a.temp + i);
	if (blockIdx.x == 0 && threadIdx.x == 0) {
		st->iterations = iter;
		st->residual = rr;
		st->tol_abs = tol_abs;
		st->converged = sqrt(rr) < tol_abs ? 1 : 0;
	}
}

// Launch shape of k_cg_rows for n rows of at most maxlen nonzeroes.
struct CgRowsShape {
	int L = 1, nb = 0, grid = 0, steps = 0, items = 0, resident = 0, vec_smem = 0;
	size_t smem = 0;
};

// One lane per row gathers best (32 consecutive rows on one line after another:
// 64^3 17 us an iteration, 20 with two lanes a row, 27 with four); more lanes
// only while every other warp would have no item (32^3: four lanes a row).
// Vectors go to shared memory while they leave room for the matrix.
static CgRowsShape cg_rows_shape(int64_t n, int maxlen) {
	CgRowsShape c;
	const size_t cap = CGR_SMEM;
	const int64_t sms = sm_count() < GRID_REDUCE_BLOCKS ? sm_count() : GRID_REDUCE_BLOCKS;
	const int64_t per = (n + sms - 1) / sms;
	if (per > (1 << 24) || maxlen < 1) return c;
	while (c.L < 8 && c.L * 2 <= maxlen && (per * c.L + 31) / 32 * 2 <= CGR_WARPS) c.L *= 2;
	const int H = 32 / c.L;
	c.nb = int((per + H - 1) / H * H);
	c.grid = int((n + c.nb - 1) / c.nb);
	c.steps = (maxlen + c.L - 1) / c.L;
	c.items = c.nb / H;
	const size_t vec = size_t(c.nb) * 32;
	c.vec_smem = vec <= cap * 5 / 8;
	const size_t item = size_t(c.steps) * 32 * 12;
	const size_t left = cap - (c.vec_smem ? vec : 0);
	c.resident = int(left / item < size_t(c.items) ? left / item : size_t(c.items));
	c.smem = (c.vec_smem ? vec : 0) + size_t(c.resident) * item;
	return c;
}

// Entries outside shared memory: 12 bytes each, a second copy of that part of
// the matrix, padded to the longest row.
static size_t cg_rows_ell(const CgRowsShape &c) {
	return size_t(c.grid) * size_t(c.items - c.resident) * size_t(c.steps) * 32;
}

// Largest workspace: after alpb_init the stream-ordered pool keeps it for the next
// solve, so it is bounded.  (To hand one back after every solve costs 10 ms per GB:
// 27-point 160^3, 1.3 GB, 50 iterations 20.2 -> 28.3 ms, k_cg 31.1; 256^3, 5.4 GB,
// 84 -> 142, k_cg 128.)
constexpr size_t CGR_MAX = size_t(8) << 30;

// Whether k_cg_rows is worth its set-up and its padding.  Measured us, k_cg /
// k_cg_rows:
//  - the rewriting takes longer than a few iterations win where most of it goes to
//    memory and rows are long (27-point 64^3, 88 MB: 1 iteration 143 / 180, 2 180 / 192,
//    4 274 / 229; 128^3: 1 627 / 1106, 4 1548 / 1692, 8 2785 / 2470; 256^3: 4 12359 /
//    13250, 50 128344 / 84491; 5-point rows break even at one);
//  - padded entries are read as the others are, and from some size on that is what
//    an iteration costs (8 to 24 random columns a row, half as many again: 1 M rows,
//    288 MB, 2990 / 2867 per 20 iterations, 3 M rows, 864 MB, 9153 / 10522).
static bool cg_rows_pays(const CgRowsShape &c, int64_t nnz, int64_t max_iter) {
	const size_t bytes = cg_rows_ell(c) * 12;
	if (bytes == 0) return true;
	if (bytes > CGR_MAX) return false;
	if (c.steps * c.L > 8 && max_iter < (bytes > (size_t(128) << 20) ? 5 : 3)) return false;
	const double padded = double(c.grid) * c.items * c.steps * 32;
	return bytes <= (size_t(512) << 20) || padded <= 1.25 * double(nnz);
}

// The solve on k_cg_rows; ALPB_UNSUPPORTED (nothing launched) when its
// workspace cannot be had or its blocks cannot be resident together, and the
// caller runs k_cg instead.
template <int L>
static int cg_rows_solve(const CgRowsShape &c, CgRowsArgs a, double *wk, cudaStream_t s,
	CgState *h) {
	static std::atomic<unsigned long long> allowed_in;
	ALPB_CUDA(allow_smem(k_cg_rows<L>, CGR_SMEM, allowed_in));
	if (cooperative_grid(k_cg_rows<L>, CGR_THREADS, c.smem, c.grid) < c.grid) {
		cudaGetLastError();
		return ALPB_UNSUPPORTED;
	}
	const int64_t n = a.n;
	const size_t ell = cg_rows_ell(c);
	// one allocation: state, partials, the items outside shared memory, r
	const size_t head = (sizeof(GridReduce) + sizeof(CgState) + 255) / 256 * 256;
	const size_t bytes = head + ell * 12 + (c.vec_smem ? 0 : size_t(n) * 8);
	unsigned char *ws = nullptr;
	if (cudaMallocAsync(&ws, bytes, s) != cudaSuccess) {
		cudaGetLastError();
		return ALPB_UNSUPPORTED;
	}
	a.gr = reinterpret_cast<GridReduce *>(ws);
	a.st = reinterpret_cast<CgState *>(ws + sizeof(GridReduce));
	a.ell_val = reinterpret_cast<double *>(ws + head);
	a.g_r = a.ell_val + ell;
	a.ell_idx = reinterpret_cast<uint32_t *>(a.g_r + (c.vec_smem ? 0 : n));
	a.pr = reinterpret_cast<double2 *>(wk);
	a.g_u = wk + 2 * n;
	a.g_t = wk + 3 * n;
	a.r_out = wk;
	a.nb = c.nb;
	a.steps = c.steps;
	a.items = c.items;
	a.resident = c.resident;
	a.vec_smem = c.vec_smem;
	ALPB_CUDA(cudaMemsetAsync(ws, 0, head, s));
	void *args[] = {&a};
	const cudaError_t e = cudaLaunchCooperativeKernel((void *) k_cg_rows<L>, dim3(c.grid),
		dim3(CGR_THREADS), args, c.smem, s);
	if (e != cudaSuccess) {
		cudaGetLastError();
		cudaFreeAsync(ws, s);
		if (e == cudaErrorCooperativeLaunchTooLarge) return ALPB_UNSUPPORTED;
		set_error("alpb_cg_solve: %s", cudaGetErrorString(e));
		return ALPB_PANIC;
	}
	ALPB_LAUNCHED();
	ALPB_CUDA(cudaMemcpyAsync(h, a.st, sizeof(CgState), cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(ws, s));
	return ALPB_SUCCESS;
}

// The solve on warp merge tiles (k_cg): any row lengths.  *h is filled once
// the stream has run.
static int cg_tiles_solve(int64_t n, const int64_t *row_ptr, const uint32_t *col_idx,
	const double *values, const double *b, double *x, int64_t max_iter, double tol, double *wk,
	alpb_spmv_plan plan, cudaStream_t s, CgState *h) {
	const bool few = plan->ntiles <= CG_FEW_TILES;
	const int warps = few ? 16 : 8;
	const size_t smem = sizeof(CgWarpSmem) * warps;
	static bool smem_set = false;
	if (!smem_set) {
		ALPB_CUDA(cudaFuncSetAttribute(k_cg<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			int(sizeof(CgWarpSmem) * 16)));
		ALPB_CUDA(cudaFuncSetAttribute(k_cg<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			int(sizeof(CgWarpSmem) * 8)));
		smem_set = true;
	}
	const int grid = few ? solver_grid(k_cg<16>, 32 * 16, plan->ntiles, 16, smem)
						 : solver_grid(k_cg<8>, 32 * 8, plan->ntiles, 8, smem);
	ALPB_CHECK(grid > 0, ALPB_PANIC, "alpb_cg_solve: no cooperative occupancy");
	double *scratch = nullptr;
	CgState *st = nullptr;
	ALPB_CUDA(cudaMallocAsync(&scratch, size_t(4 * grid) * 8, s));
	ALPB_CUDA(cudaMallocAsync(&st, sizeof(CgState), s));
	ALPB_CUDA(cudaMemsetAsync(st, 0, sizeof(CgState), s));
	CgArgs a;
	a.mt = merge_tables(*plan);
	a.offsets = row_ptr;
	a.indices = col_idx;
	a.values = values;
	a.b = b;
	a.x = x;
	a.pr = reinterpret_cast<double2 *>(wk);
	a.u_new = wk + 2 * n;
	a.temp = wk + 3 * n;
	a.r_out = wk;
	a.blk = scratch;
	a.n = n;
	a.max_iter = max_iter;
	a.tol = tol;
	a.st = st;
	void *args[] = {&a};
	ALPB_CUDA(cudaLaunchCooperativeKernel(few ? (void *) k_cg<16> : (void *) k_cg<8>, dim3(grid),
		dim3(32 * warps), args, smem, s));
	ALPB_LAUNCHED();
	ALPB_CUDA(cudaMemcpyAsync(h, st, sizeof(CgState), cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(scratch, s));
	ALPB_CUDA(cudaFreeAsync(st, s));
	return ALPB_SUCCESS;
}

} // namespace alpb

using namespace alpb;

extern "C" int alpb_cg_solve(int64_t n, const int64_t *row_ptr, const uint32_t *col_idx,
	const double *values, const double *b, double *x, int64_t max_iter, double tol,
	int64_t *iterations, double *residual, double *work, alpb_spmv_plan plan, void *stream) {
	ALPB_CHECK(n >= 0, ALPB_ILLEGAL, "alpb_cg_solve: negative size");
	ALPB_CHECK(tol > 0, ALPB_ILLEGAL, "alpb_cg_solve: tolerance must be strictly positive");
	ALPB_CHECK(max_iter > 0, ALPB_ILLEGAL, "alpb_cg_solve: at least one iteration is required");
	ALPB_CHECK(iterations && residual, ALPB_ILLEGAL, "alpb_cg_solve: null output");
	*iterations = 0;
	*residual = INFINITY;
	if (n == 0) return ALPB_SUCCESS;
	cudaStream_t s = as_stream(stream);
	if (plan)
		ALPB_CHECK(plan->m == n && plan->offsets == row_ptr && plan->tile == WM_TILE,
			ALPB_MISMATCH, "alpb_cg_solve: plan was made for another storage");
	alpb_spmv_plan own_plan = nullptr;
	if (!plan) {
		int64_t nnz = 0;
		ALPB_CUDA(cudaMemcpyAsync(&nnz, row_ptr + n, 8, cudaMemcpyDeviceToHost, s));
		ALPB_CUDA(cudaStreamSynchronize(s));
		int rc = plan_create_tiles(&own_plan, n, nnz, row_ptr, ALPB_SCHED_MERGE_PATH, 0, WM_TILE, s);
		if (rc != ALPB_SUCCESS) return rc;
		plan = own_plan;
	}
	// the (r, u) pairs take 16-byte loads: a work space that is not 16-byte
	// aligned is replaced by an internal one
	double *wk = (reinterpret_cast<uintptr_t>(work) & 15) ? nullptr : work;
	double *own_work = nullptr;
	if (!wk) {
		ALPB_CUDA(cudaMallocAsync(&own_work, size_t(4 * n) * 8, s));
		wk = own_work;
	}
	CgState h;
	int rc = ALPB_UNSUPPORTED;
	// short regular rows (the plan's tiles hold whole rows): fixed rows per
	// block.  Measured us per iteration, k_cg -> k_cg_rows, 27-point grids:
	// 10^3 11.6 -> 7.7, 32^3 13.9 -> 7.6, 48^3 26 -> 11, 64^3 47 -> 17,
	// 80^3 78 -> 50, 128^3 311 -> 199
	const CgRowsShape c = plan->tile_d ? cg_rows_shape(n, int(plan->maxlen)) : CgRowsShape{};
	if (c.grid > 0 && n < int64_t(CGR_NONE) && cg_rows_pays(c, plan->nnz, max_iter)) {
		CgRowsArgs a{};
		a.offsets = row_ptr;
		a.indices = col_idx;
		a.values = values;
		a.b = b;
		a.x = x;
		a.n = n;
		a.max_iter = max_iter;
		a.tol = tol;
		rc = c.L == 1 ? cg_rows_solve<1>(c, a, wk, s, &h)
			: c.L == 2 ? cg_rows_solve<2>(c, a, wk, s, &h)
			: c.L == 4 ? cg_rows_solve<4>(c, a, wk, s, &h)
					   : cg_rows_solve<8>(c, a, wk, s, &h);
	}
	if (rc == ALPB_UNSUPPORTED)
		rc = cg_tiles_solve(n, row_ptr, col_idx, values, b, x, max_iter, tol, wk, plan, s, &h);
	if (own_work) ALPB_CUDA(cudaFreeAsync(own_work, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	if (rc != ALPB_SUCCESS) {
		alpb_spmv_plan_destroy(own_plan);
		return rc;
	}
	if (own_plan) alpb_spmv_plan_destroy(own_plan);
	ALPB_CHECK(h.gs.err == 0, ALPB_PANIC, "alpb_cg_solve: a grid barrier or tile wait timed out");
	*iterations = h.iterations;
	*residual = h.residual;
	if (!h.converged) {
		set_error("alpb_cg_solve: not converged after %lld iterations (sqrt(r.r) = %g, tol %g)",
			(long long) h.iterations, sqrt(h.residual), h.tol_abs);
		return ALPB_FAILED;
	}
	return ALPB_SUCCESS;
}
