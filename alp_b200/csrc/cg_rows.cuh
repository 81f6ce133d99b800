// Conjugate gradient on short, regular rows (stencils): the same recurrence as
// k_cg (cg.cu) with the rows of one block fixed for the whole solve.
//
// What bounds a CG iteration on such a system is not HBM: the matrix of a
// 32^3 grid (10 MB) fits the SMs' shared memory, that of a 64^3 grid (82 MB)
// the L2, and an iteration is two dependent grid-wide sums.  So:
//  - one block per SM owns nb consecutive rows; its x, r, direction and A p
//    live in shared memory (in global memory when nb is too large), phase B
//    touches nothing of another block, and only the pairs (r_i, u_i) that
//    phase A gathers are published;
//  - each block rewrites its rows once, at the start, as items of 32 / L rows
//    with L lanes per row, entry s of an item one coalesced line; as many
//    items as fit stay in shared memory, the others stream from a workspace;
//  - the pairs are gathered with plain loads, so the 27 neighbours of
//    consecutive rows share L1 lines (the barrier's fence drops stale ones);
//  - both sums of an iteration ride on the barrier itself (grid_reduce).
#pragma once
#include "common.cuh"
#include "persist.cuh"

namespace alpb {

constexpr int CGR_THREADS = 1024;
constexpr int CGR_WARPS = CGR_THREADS / 32;
constexpr uint32_t CGR_NONE = 0xffffffffu;   // no entry: the row is shorter
constexpr int CGR_BATCH = 8;                 // gathers in flight per lane
// Shared memory of a block: what is left of the SM's 256 KB holds the L1 lines
// of the gathers in flight (64^3, us per iteration: 17.4 with 192 KB, 18.1
// with 226; 40^3 8.2 and 8.2 against 8.8 with 128, which holds less matrix).
constexpr int CGR_SMEM = 192 * 1024;

struct CgRowsArgs {
	const int64_t *offsets;
	const uint32_t *indices;
	const double *values;
	const double *b;
	double *x;
	double2 *pr;          // (r_i, u_i), n
	double *r_out;        // r on return (the memory of pr)
	double *g_r, *g_u, *g_t;   // vectors in global memory when vec_smem == 0
	uint32_t *ell_idx;    // items that do not stay in shared memory:
	double *ell_val;      // [block][items - resident][steps][32]
	GridReduce *gr;
	CgState *st;
	int64_t n, max_iter;
	double tol;
	int nb;               // rows per block
	int steps;            // entries per lane of an item: ceil(longest row / L)
	int items;            // items per block
	int resident;         // of which the first stay in shared memory
	int vec_smem;
};

// The row product of one item for this lane: entries s = 0, 1, ... of lane
// `lane`, fused multiply-adds in that order; then the row's L lanes by tree.
template <int L, bool SM, class XF>
__device__ __forceinline__ double cgr_item(const uint32_t *ix, const double *val, int steps,
	const XF &xf) {
	double acc = 0.0;
	for (int s0 = 0; s0 < steps; s0 += CGR_BATCH) {
		uint32_t j[CGR_BATCH];
		double g[CGR_BATCH], v[CGR_BATCH];
#pragma unroll
		for (int q = 0; q < CGR_BATCH; ++q) {
			j[q] = CGR_NONE;
			if (s0 + q < steps) j[q] = SM ? ix[(s0 + q) * 32] : __ldcg(ix + (s0 + q) * 32);
		}
		if (!SM) {
#pragma unroll
			for (int q = 0; q < CGR_BATCH; ++q)
				v[q] = s0 + q < steps ? __ldcg(val + (s0 + q) * 32) : 0.0;
		}
#pragma unroll
		for (int q = 0; q < CGR_BATCH; ++q) g[q] = j[q] != CGR_NONE ? xf(j[q]) : 0.0;
#pragma unroll
		for (int q = 0; q < CGR_BATCH; ++q)
			if (j[q] != CGR_NONE) acc = fma(SM ? val[(s0 + q) * 32] : v[q], g[q], acc);
	}
#pragma unroll
	for (int o = 1; o < L; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	return acc;
}

template <int L>
__global__ void __launch_bounds__(CGR_THREADS, 1) k_cg_rows(CgRowsArgs a) {
	constexpr int H = 32 / L;   // rows per item
	extern __shared__ __align__(16) unsigned char cgr_smem[];
	__shared__ double red[64];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int sub = lane / L, k = lane % L;
	const int64_t rb = int64_t(blockIdx.x) * a.nb;
	const int rows = int(a.n - rb < a.nb ? a.n - rb : a.nb);
	const int items = (rows + H - 1) / H;
	int *err = &a.st->gs.err;
	double *sm = reinterpret_cast<double *>(cgr_smem);
	double *xs = a.vec_smem ? sm : a.x + rb;
	double *rs = a.vec_smem ? sm + a.nb : a.g_r + rb;
	double *us = a.vec_smem ? sm + 2 * a.nb : a.g_u + rb;
	double *ts = a.vec_smem ? sm + 3 * a.nb : a.g_t + rb;
	const int isz = a.steps * 32;   // entries of an item
	double *sval = sm + (a.vec_smem ? 4 * a.nb : 0);
	uint32_t *sidx = reinterpret_cast<uint32_t *>(sval + size_t(a.resident) * isz);
	const size_t gbase = size_t(blockIdx.x) * size_t(a.items - a.resident) * isz;
	// this lane's entries of item it
	const auto item_val = [&](int it) {
		return it < a.resident ? sval + size_t(it) * isz + lane
							   : a.ell_val + gbase + size_t(it - a.resident) * isz + lane;
	};
	const auto item_idx = [&](int it) {
		return it < a.resident ? sidx + size_t(it) * isz + lane
							   : a.ell_idx + gbase + size_t(it - a.resident) * isz + lane;
	};
	// rewrite the block's rows: a lane reads back only what it writes here
	for (int it = w; it < items; it += CGR_WARPS) {
		const int row = it * H + sub;
		const int64_t o = row < rows ? a.offsets[rb + row] : 0;
		const int len = row < rows ? int(a.offsets[rb + row + 1] - o) : 0;
		double *v = item_val(it);
		uint32_t *ix = item_idx(it);
		for (int s = 0; s < a.steps; ++s) {
			const int q = s * L + k;
			v[s * 32] = q < len ? a.values[o + q] : 0.0;
			ix[s * 32] = q < len ? a.indices[o + q] : CGR_NONE;
		}
	}
	const auto product = [&](int it, const auto &xf) {
		return it < a.resident ? cgr_item<L, true>(item_idx(it), item_val(it), a.steps, xf)
							   : cgr_item<L, false>(item_idx(it), item_val(it), a.steps, xf);
	};

	// prelude: r = b - A x, u = 0 (gamma = 0 takes u = r), r.r and b.b
	unsigned epoch = 0;
	double sigma, bb;
	{
		double prr = 0.0, pbb = 0.0;
		for (int it = w; it < items; it += CGR_WARPS) {
			const double t = product(it, [&](uint32_t j) { return a.x[j]; });
			const int row = it * H + sub;
			if (k == 0 && row < rows) {
				const double bi = a.b[rb + row];
				const double ri = bi - t;
				rs[row] = ri;
				us[row] = 0.0;
				a.pr[rb + row] = make_double2(ri, 0.0);
				prr += ri * ri;
				pbb += bi * bi;
			}
		}
		// the gathers above read x: own rows are copied (and later written)
		// only after every block is past them
		if (!grid_reduce(a.gr, ++epoch, prr, &sigma, red, err)) return;
		if (!grid_reduce(a.gr, ++epoch, pbb, &bb, red, err)) return;
		if (a.vec_smem)
			for (int i = threadIdx.x; i < rows; i += CGR_THREADS) xs[i] = a.x[rb + i];
	}
	const double tol_abs = a.tol * sqrt(bb);
	double gamma = 0.0, rr = 0.0;
	int64_t iter = 0;
	for (;;) {
		++iter;
		// phase A: t = A u, u = r + gamma u_old gathered as pairs; beta = t.u
		double part = 0.0;
		for (int it = w; it < items; it += CGR_WARPS) {
			const double t = product(it, [&](uint32_t j) {
				const double2 p = a.pr[j];
				return p.x + gamma * p.y;
			});
			const int row = it * H + sub;
			if (k == 0 && row < rows) {
				const double un = rs[row] + gamma * us[row];
				us[row] = un;
				ts[row] = t;
				part += t * un;
			}
		}
		double beta;
		if (!grid_reduce(a.gr, ++epoch, part, &beta, red, err)) return;
		// phase B: alpha = sigma / beta, x += alpha u, r -= alpha t, r.r
		const double alpha = sigma / beta;
		part = 0.0;
		for (int i = threadIdx.x; i < rows; i += CGR_THREADS) {
			const double un = us[i];
			xs[i] = xs[i] + alpha * un;
			const double ri = rs[i] - alpha * ts[i];
			rs[i] = ri;
			a.pr[rb + i] = make_double2(ri, un);
			part += ri * ri;
		}
		if (!grid_reduce(a.gr, ++epoch, part, &rr, red, err)) return;
		if (sqrt(rr) < tol_abs || iter >= a.max_iter) break;
		gamma = rr / sigma;  // alpha = beta / sigma in the reference's naming
		sigma = rr;
	}
	// every block is past its last gather: the pairs' memory takes r
	for (int i = threadIdx.x; i < rows; i += CGR_THREADS) {
		a.r_out[rb + i] = rs[i];
		if (a.vec_smem) a.x[rb + i] = xs[i];
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) {
		a.st->iterations = iter;
		a.st->residual = rr;
		a.st->tol_abs = tol_abs;
		a.st->converged = sqrt(rr) < tol_abs ? 1 : 0;
	}
}

} // namespace alpb
