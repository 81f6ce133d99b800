// Fused HPCG: algorithms::hpcg (hpcg/hpcg.hpp:97-223), its multigrid V-cycle
// (hpcg/multigrid_v_cycle.hpp:67-246) and the multi-colour Gauss-Seidel
// smoother (hpcg/red_black_gauss_seidel.hpp:55-123) as device kernels, for
// the system build_hpcg_system makes (hpcg/system_building_utils.hpp:84-150):
// the 3-D 27-point box stencil on every level, levels coarsened by 2 per
// dimension, injection as the coarsening matrix, static colours (row index
// modulo the colour count).
//
// Several right-hand sides are solved together: vectors hold the nrhs values
// of a row side by side (row-major), so every pass over a matrix serves all
// of them.  Each right-hand side keeps its own CG scalars and its own
// convergence test, exactly as separate runs of the algorithm would.
//
// Kernels (all FP64, every sum in a fixed order):
//   k_hpcg_cycle<NRHS>   one V-cycle as one persistent cooperative launch: a
//                        colour step, a restriction or a prolongation between
//                        two grid barriers
//   k_hpcg_rows<NRHS, Op>  the same steps as launches, on levels far larger
//                        than L2
//   k_hpcg_spmm<NRHS>    A p and the block partials of p . A p
//   k_hpcg_dot, k_hpcg_axpby, k_hpcg_update   the CG vector steps, with block
//                        partials of the dot product that follows
//   k_hpcg_finish        the partials summed, then the CG scalars on the device
#include "common.cuh"
#include "persist.cuh"

#include <cmath>
#include <vector>

namespace alpb {

constexpr int HG_BLOCK = 256;
constexpr int HG_ROW = 27;          // entries of a stencil row, at most
constexpr uint32_t HG_NONE = 0xffffffffu;

// Loads of the matrix, which no kernel writes, kept where they stand: ahead of
// the barrier that precedes their use.
__device__ __forceinline__ void hg_load(uint32_t &v, const uint32_t *p) {
	asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
}
__device__ __forceinline__ void hg_load(double &v, const double *p) {
	asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
}
__device__ __forceinline__ void hg_load(int64_t &v, const int64_t *p) {
	asm volatile("ld.global.nc.s64 %0, [%1];" : "=l"(v) : "l"(p));
}

// One row's product by GL lanes: lane (s, k) of the group takes right-hand
// side k = lane % NRHS and the entries s, s + S, ... of the row (at most NE,
// so all of a lane's loads are in flight together: a colour step is one
// dependent chain offsets -> indices -> x, and the serial walk it replaces
// paid that chain once per few entries); the S partial sums are combined by
// an xor tree.
template <int NRHS>
struct HgRow {
	static constexpr int GL = 8 * NRHS < 32 ? 8 * NRHS : 32;
	static constexpr int RPW = 32 / GL;     // rows per warp
	static constexpr int S = GL / NRHS;
	static constexpr int NE = (HG_ROW + S - 1) / S;
	// where a row's entries are: its offset and length (row < 0: none)
	struct At {
		int64_t o;
		int len;
	};
	static __device__ __forceinline__ At at(const int64_t *__restrict__ offsets, int64_t row) {
		At r{0, 0};
		if (row >= 0) {
			int64_t e;
			hg_load(r.o, offsets + row);
			hg_load(e, offsets + row + 1);
			r.len = int(e - r.o);
		}
		return r;
	}
	uint32_t j[NE];
	double v[NE];
	__device__ __forceinline__ void load(const uint32_t *__restrict__ indices,
		const double *__restrict__ values, const At &r) {
		const int s = (threadIdx.x & (GL - 1)) / NRHS;
#pragma unroll
		for (int q = 0; q < NE; ++q) {
			const int e = s + q * S;
			j[q] = HG_NONE;
			v[q] = 0.0;
			if (e < r.len) {
				hg_load(j[q], indices + r.o + e);
				hg_load(v[q], values + r.o + e);
			}
		}
	}
	// sum_e v_e x[j_e], read through L2 (x changes between the barriers of a
	// cycle, and a step reads no line of it twice); after_sum runs once the
	// gathered values are used
	template <class F>
	__device__ __forceinline__ double product(const double *x, F &&after_sum) const {
		const int k = threadIdx.x % NRHS;
		double g[NE], acc = 0.0;
#pragma unroll
		for (int q = 0; q < NE; ++q) g[q] = j[q] != HG_NONE ? __ldcg(x + int64_t(j[q]) * NRHS + k) : 0.0;
#pragma unroll
		for (int q = 0; q < NE; ++q)
			if (j[q] != HG_NONE) acc = fma(v[q], g[q], acc);
		after_sum();
#pragma unroll
		for (int o = NRHS; o < GL; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
		return acc;
	}
	static __device__ __forceinline__ int sub() { return (threadIdx.x & 31) / GL; }
	static __device__ __forceinline__ bool lead() { return (threadIdx.x & (GL - 1)) < NRHS; }
};

// Fine row of coarse point c under injection: coarse (cx, cy, cz) takes the
// fine point (2cx, 2cy, 2cz) (coarsener_generator_iterator,
// ndim_matrix_builders.hpp:412-541; x varies fastest).
struct HgInject {
	int64_t cnx, cny, fnx, fny;
	__device__ __forceinline__ int64_t operator()(int64_t c) const {
		const int64_t cx = c % cnx, cy = (c / cnx) % cny, cz = c / (cnx * cny);
		return 2 * cx + 2 * cy * fnx + 2 * cz * fnx * fny;
	}
};

// One level as the cycle kernel sees it.
struct HgLevelArgs {
	const int64_t *offsets;
	const uint32_t *indices;
	const double *values;
	double *r, *z, *temp;   // temp: null when the smoother is fused
	int64_t n, nx, ny;
};
constexpr int HG_MAX_LEVELS = 16;   // every level halves three dimensions

struct HgCycleArgs {
	HgLevelArgs lv[HG_MAX_LEVELS];
	int l0, l1;              // this launch's levels [l0, l1)
	int part;                // HG_DOWN, HG_UP or HG_WHOLE
	int64_t colors, pre, post;
	double diag;
	GridSync *gs;
	const int32_t *active;   // right-hand sides still iterating: none, no work
};
enum { HG_DOWN, HG_UP, HG_WHOLE };

constexpr int HGC_THREADS = 768;
constexpr int HGC_CLUSTER = 16;     // blocks of a cluster launch

// multi_grid (multigrid_v_cycle.hpp:193-246) on the levels [l0, l1): z = 0 (the
// caller's, on l0); smooth; restrict the residual; recurse; prolong; smooth.  HG_WHOLE ends at
// the coarsest level, which smooths once; HG_DOWN stops after the restriction
// to level l1 and HG_UP begins with the prolongation from it.  A smoother
// (red_black_gauss_seidel.hpp:55-123) is 2 x colors steps, forward then
// backward, each
//   temp = 0 + A[mask] x;  x[mask] = (r - temp + x d) / d
// on the rows c, c + K, ...: in place when no two neighbours share a colour,
// so that no row of the colour reads another's new value; otherwise the
// products are stored first and applied after a barrier.
//
// What bounds it is the chain of steps: 378 of them per cycle on 64^3 with
// three coarser levels, each a few thousand rows at most.  As separate
// launches a step took 17.5 us.  Here it is a barrier, one round of gathers
// and the update; the entries of a warp's next row are in flight, and the
// place of the one after is known, before the barrier, so only x is read
// after it.  CLUSTER: one cluster of blocks with its hardware barrier instead
// of a block per SM with a barrier through L2 -- coarse levels, where the
// barrier is most of a step: 1.0 us there, 1.8 us through L2.  Measured us per
// HPCG iteration, launches -> this: 16^3 with 8 right-hand sides 1451 -> 341,
// 64^3 with 1 2499 -> 971, 64^3 with 8 4088 -> 1508, 128^3 with 8 10576 -> 8377.
// 768 threads leave 80 registers each: two rows' entries in flight do not quite
// fit, and 52 to 132 bytes a thread spill (what that costs was not measured apart).
template <int NRHS, bool CLUSTER>
__global__ void __launch_bounds__(HGC_THREADS, 1) k_hpcg_cycle(HgCycleArgs a) {
	using Row = HgRow<NRHS>;
	using At = typename Row::At;
	if (*a.active == 0) return;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int k = lane % NRHS;
	const int G = gridDim.x;
	// rows and steps in 32 bits: 2^31 stencil rows are more than the memory
	// rows go round the blocks first, so small steps use every SM
	const int nrow = G * (HGC_THREADS / 32) * Row::RPW;
	const int row0 = (w * G + int(blockIdx.x)) * Row::RPW;   // the warp's first
	const int64_t tid = blockIdx.x * int64_t(HGC_THREADS) + threadIdx.x;
	const int64_t nthreads = int64_t(G) * HGC_THREADS;
	const int K = int(a.colors);
	const auto barrier = [&]() {
		if constexpr (CLUSTER) {
			// one fence for the block's writes instead of one per thread
			__syncthreads();
			if (threadIdx.x == 0) asm volatile("fence.acq_rel.cluster;" ::: "memory");
			__syncwarp();
			asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
			asm volatile("barrier.cluster.wait;" ::: "memory");
			return true;
		} else {
			return grid_sync(a.gs);
		}
	};

	// one smoother on level L; false: a barrier gave up
	const auto smooth = [&](const HgLevelArgs &L) {
		// rows t, t + 1, ... of a step's colour belong to the warp's lane groups
		struct Pos {
			int step, t;
		};
		const auto color = [&](int step) { return step < K ? step : 2 * K - 1 - step; };
		const auto row_of = [&](const Pos &p, int sub) {
			const int64_t i = color(p.step) + int64_t(p.t + sub) * K;
			return p.step < 2 * K && i < L.n ? int(i) : -1;
		};
		const auto next = [&](Pos p) {   // the warp's next rows: this step's, else the next one's
			p.t += nrow;
			if (row_of(p, 0) < 0) p = Pos{p.step + 1, row0};
			return p;
		};
		Pos p0{0, row0}, p1 = next(p0);
		int i0 = row_of(p0, Row::sub()), i1 = row_of(p1, Row::sub());
		// One item: the product of p0's rows, entries in `cur`; p1's entries go
		// to `nxt` from their place `at`, and p2's place to `at_next`: after the
		// sum, since gathers that share a scoreboard with later loads wait for
		// those too.  The two sets of registers swap roles from item to item
		// (copying one to the other would wait for the loads just issued).
		const auto item = [&](Row &cur, Row &nxt, const At &at, At &at_next) {
			const Pos p2 = next(p1);
			const int i2 = row_of(p2, Row::sub());
			const int64_t o = int64_t(i0) * NRHS + k;
			const bool mine = i0 >= 0 && Row::lead();
			const double ri = mine ? __ldcg(L.r + o) : 0.0, xi = mine ? __ldcg(L.z + o) : 0.0;
			const double p = cur.product(L.z, [&]() {
				nxt.load(L.indices, L.values, at);
				at_next = Row::at(L.offsets, i2);
			});
			if (mine) {
				if (L.temp) L.temp[o] = p;
				else L.z[o] = (ri - p + xi * a.diag) / a.diag;
			}
			p0 = p1;
			p1 = p2;
			i0 = i1;
			i1 = i2;
		};
		int step = 0;
		// the barriers between this warp's last item of `step` and its next one
		const auto end_of_step = [&]() {
			if (!barrier()) return false;
			if (L.temp) {
				const int64_t c = color(step);
				const int64_t count = c < L.n ? (L.n - 1 - c) / K + 1 : 0;
				for (int64_t q = tid; q < count * NRHS; q += nthreads) {
					const int64_t o = (c + (q / NRHS) * K) * NRHS + q % NRHS;
					L.z[o] = (L.r[o] - L.temp[o] + L.z[o] * a.diag) / a.diag;
				}
				if (!barrier()) return false;
			}
			++step;
			return true;
		};
		Row even, odd;
		At at_odd = Row::at(L.offsets, i1), at_even;
		even.load(L.indices, L.values, Row::at(L.offsets, i0));
		while (step < 2 * K) {
			item(even, odd, at_odd, at_even);
			if (p0.step != step && !end_of_step()) return false;
			if (step == 2 * K) break;
			item(odd, even, at_even, at_odd);
			if (p0.step != step && !end_of_step()) return false;
		}
		return true;
	};

	if (a.part != HG_UP) {
		for (int l = a.l0; l < (a.part == HG_WHOLE ? a.l1 - 1 : a.l1); ++l) {
			const HgLevelArgs &L = a.lv[l], &C = a.lv[l + 1];
			for (int64_t q = 0; q < a.pre; ++q)
				if (!smooth(L)) return;
			// restriction, compute_coarsening (multigrid_v_cycle.hpp:67-86): r_c =
			// r_f - A z at the injected rows, formed only there; the coarse z = 0
			const HgInject inj{C.nx, C.ny, L.nx, L.ny};
			for (int64_t t0 = row0; t0 < C.n; t0 += nrow) {
				const int64_t t = t0 + Row::sub();
				const int64_t f = t < C.n ? inj(t) : -1;
				Row row;
				row.load(L.indices, L.values, Row::at(L.offsets, f));
				const double ax = row.product(L.z, [] {});
				if (f >= 0 && Row::lead()) {
					C.r[t * NRHS + k] = L.r[f * NRHS + k] - ax;
					C.z[t * NRHS + k] = 0.0;
				}
			}
			if (!barrier()) return;
		}
		if (a.part == HG_WHOLE && !smooth(a.lv[a.l1 - 1])) return;
	}
	if (a.part == HG_DOWN) return;
	for (int l = a.part == HG_WHOLE ? a.l1 - 2 : a.l1 - 1; l >= a.l0; --l) {
		const HgLevelArgs &L = a.lv[l], &C = a.lv[l + 1];
		// prolongation, compute_prolongation (multigrid_v_cycle.hpp:88-103): z_f
		// += z_c at the injected rows (the other rows add zero)
		const HgInject inj{C.nx, C.ny, L.nx, L.ny};
		for (int64_t q = tid; q < C.n * NRHS; q += nthreads) {
			const int64_t o = inj(q / NRHS) * NRHS + q % NRHS;
			L.z[o] = L.z[o] + C.z[q];
		}
		if (!barrier()) return;
		for (int64_t q = 0; q < a.post; ++q)
			if (!smooth(L)) return;
	}
}

// ------------------------------------------------ large levels: launches --
// Where x is far larger than L2 a colour step is bound by its gathers from
// memory, and every warp that an SM can hold counts more than the loads each
// has in flight: such levels run a launch per step, 8 lanes per row, lane
// (s, k) of the group walking the entries s, s + S, ... of right-hand side k,
// in 32 registers.  hg_by_launches below says which levels these are, and the
// times of both sides.
constexpr int HG_GROUP = 8;     // lanes per matrix row
template <int NRHS, class Op>
__global__ void __launch_bounds__(HG_BLOCK, 8)
k_hpcg_rows(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const double *__restrict__ values, const double *__restrict__ x, int64_t count, Op op,
	const int32_t *active) {
	if (active && *active == 0) return;   // no right-hand side still iterates
	constexpr int S = HG_GROUP / NRHS;
	constexpr int PARTS = NRHS < 4 ? 1 : NRHS / 2;   // of a lane's sum: 27 terms in one round more
	constexpr int GPW = 32 / HG_GROUP;  // row groups per warp
	const int q = threadIdx.x & (HG_GROUP - 1);
	const int k = q % NRHS, s = q / NRHS;
	const int g = (threadIdx.x & 31) / HG_GROUP;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	// the loop bound is the same for the whole warp, so every lane reaches
	// every shuffle below
	for (int64_t wb = warp * GPW; wb < count; wb += nwarps * GPW) {
		const int64_t idx = wb + g;
		const bool valid = idx < count;
		double acc = 0.0;
		int64_t row = 0;
		if (valid) {
			row = op.row(idx);
			const int64_t b = offsets[row], e = offsets[row + 1];
			double part[PARTS] = {};   // taken in turn
			for (int64_t j = b + s; j < e; j += S) {
				const double t = part[0] + values[j] * x[int64_t(indices[j]) * NRHS + k];
#pragma unroll
				for (int q = 1; q < PARTS; ++q) part[q - 1] = part[q];
				part[PARTS - 1] = t;
			}
#pragma unroll
			for (int q = 0; q < PARTS; ++q) acc += part[q];
		}
#pragma unroll
		for (int o = NRHS; o < HG_GROUP; o <<= 1) {
			const double w = __shfl_xor_sync(0xffffffffu, acc, o);
			acc += w;
		}
		if (valid && s == 0) op.finish(idx, row, k, acc);
	}
}

// One colour step on rows c, c + K, ...: in place, or (temp) the products
// first and k_hpcg_color_update after, as in the cycle kernel.
template <int NRHS>
struct HgColor {
	const double *r;
	double *x;
	double *temp;  // null: fused
	double d;
	int64_t c, K;
	__device__ __forceinline__ int64_t row(int64_t i) const { return c + i * K; }
	__device__ __forceinline__ void finish(int64_t, int64_t row, int k, double acc) const {
		const double t = 0.0 + acc;
		const int64_t at = row * NRHS + k;
		if (temp) {
			temp[at] = t;
		} else {
			const double v = r[at] - t + x[at] * d;
			x[at] = v / d;
		}
	}
};

template <int NRHS>
__global__ void k_hpcg_color_update(const double *r, const double *temp, double *x, double d,
	int64_t c, int64_t K, int64_t count) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count * NRHS;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int64_t at = (c + (i / NRHS) * K) * NRHS + i % NRHS;
		const double v = r[at] - temp[at] + x[at] * d;
		x[at] = v / d;
	}
}

// y = 0 + A x on every row
template <int NRHS>
struct HgSpmm {
	double *y;
	__device__ __forceinline__ int64_t row(int64_t i) const { return i; }
	__device__ __forceinline__ void finish(int64_t, int64_t row, int k, double acc) const {
		y[row * NRHS + k] = 0.0 + acc;
	}
};

// Restriction and prolongation, as in the cycle kernel.
template <int NRHS>
struct HgRestrict {
	const double *r_f;
	double *r_c;
	HgInject inj;
	__device__ __forceinline__ int64_t row(int64_t c) const { return inj(c); }
	__device__ __forceinline__ void finish(int64_t c, int64_t f, int k, double acc) const {
		const double ax = 0.0 + acc;
		r_c[c * NRHS + k] = 0.0 + 1.0 * (r_f[f * NRHS + k] - ax);
	}
};

template <int NRHS>
__global__ void k_hpcg_prolong(double *z_f, const double *z_c, HgInject inj, int64_t count) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count * NRHS;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int64_t c = i / NRHS;
		const int k = int(i % NRHS);
		const int64_t at = inj(c) * NRHS + k;
		z_f[at] = z_f[at] + (0.0 + 1.0 * z_c[i]);
	}
}

// ------------------------------------------------------------ CG pieces --
// Per-right-hand-side sums of a block: thread t holds a term of right-hand
// side t % NRHS (blocks are a multiple of NRHS).  Fixed order: deterministic.
template <int NRHS>
__device__ __forceinline__ void hg_block_partials(double acc, double *partials) {
	__shared__ double sm[HG_BLOCK];
	sm[threadIdx.x] = acc;
	__syncthreads();
	for (int w = HG_BLOCK / 2; w >= NRHS; w >>= 1) {
		if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
		__syncthreads();
	}
	if (threadIdx.x < NRHS) partials[blockIdx.x * NRHS + threadIdx.x] = sm[threadIdx.x];
}

// partials of x_k . y_k (the vector steps return at once where `active` is given
// and no right-hand side still iterates: the host looks every few iterations)
template <int NRHS>
__global__ void __launch_bounds__(HG_BLOCK)
k_hpcg_dot(const double *__restrict__ x, const double *__restrict__ y, int64_t n,
	double *partials, const int32_t *active) {
	if (active && *active == 0) return;
	double acc = 0.0;
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n * NRHS;
		 i += int64_t(gridDim.x) * blockDim.x)
		acc += x[i] * y[i];
	hg_block_partials<NRHS>(acc, partials);
}

// y = 0 + A x on every row (set( y, 0 ); mxv( y, A, x )) and the partials of x . y
template <int NRHS>
__global__ void __launch_bounds__(HG_BLOCK)
k_hpcg_spmm(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const double *__restrict__ values, const double *__restrict__ x, double *__restrict__ y,
	int64_t n, double *partials, const int32_t *active) {
	if (active && *active == 0) return;
	using Row = HgRow<NRHS>;
	const int k = threadIdx.x % NRHS;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t step = ((int64_t(gridDim.x) * blockDim.x) >> 5) * Row::RPW;
	double acc = 0.0;
	for (int64_t i = warp * Row::RPW + Row::sub(); __any_sync(0xffffffffu, i < n); i += step) {
		Row row;
		row.load(indices, values, Row::at(offsets, i < n ? i : -1));
		const double p = row.product(x, [] {});
		if (i < n && Row::lead()) {
			y[i * NRHS + k] = p;
			acc += p * x[i * NRHS + k];
		}
	}
	hg_block_partials<NRHS>(acc, partials);
}

// Device-side CG state of one right-hand side.
struct HgScalars {
	double norm0, norm, rz, rz_old, pap, alpha, beta;
	int64_t iterations;
	int32_t active;
	int32_t pad;
};

template <int NRHS>
__global__ void k_hpcg_axpby(double *out, const double *a, const double *b, const HgScalars *sc,
	int which, int64_t n, const int32_t *active) {
	if (active && *active == 0) return;
	// which 0: out = b - a   (r = b - Ap, eWiseApply with minus)
	//       1: out = beta a + b  (Ap = beta p + z, eWiseMulAdd into a cleared vector)
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n * NRHS;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int k = int(i % NRHS);
		if (which == 0) out[i] = b[i] - a[i];
		else out[i] = sc[k].active ? sc[k].beta * a[i] + b[i] : a[i];  // finished: p kept
	}
}

// x += alpha p; r += -alpha Ap (eWiseMul with the ring, hpcg.hpp:206-207), and
// the partials of r . r
template <int NRHS>
__global__ void __launch_bounds__(HG_BLOCK)
k_hpcg_update(double *x, double *r, const double *p, const double *ap,
	const HgScalars *sc, int64_t n, double *partials, const int32_t *active) {
	if (*active == 0) return;
	double acc = 0.0;
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n * NRHS;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int k = int(i % NRHS);
		double ri = r[i];
		if (sc[k].active) {
			const double al = sc[k].alpha;
			x[i] = x[i] + al * p[i];
			ri = ri + (-al) * ap[i];
			r[i] = ri;
		}
		acc += ri * ri;
	}
	hg_block_partials<NRHS>(acc, partials);
}

__device__ __forceinline__ void hg_scalar_step(HgScalars &s, double dot, int step, int64_t iter,
	int64_t max_iter, double tol) {
	switch (step) {
	case 0:
		s.norm0 = sqrt(dot);
		s.norm = s.norm0;
		s.iterations = 0;
		s.active = 1;
		s.rz = 0.0;
		break;
	case 1:
		if (!s.active) return;
		s.rz_old = s.rz;
		s.rz = dot;
		s.beta = iter == 0 ? 0.0 : s.rz / s.rz_old;
		break;
	case 2:
		if (!s.active) return;
		s.pap = dot;
		s.alpha = s.rz / s.pap;
		break;
	case 3:
		if (!s.active) return;
		s.norm = sqrt(dot);
		s.iterations = iter + 1;
		// do { ... } while( iter < max && norm / norm0 > tol )  (hpcg.hpp:209)
		if (!(s.iterations < max_iter && s.norm / s.norm0 > tol)) s.active = 0;
		break;
	}
}

// The block partials summed in a fixed order (thread t: right-hand side
// t % NRHS, blocks t / NRHS, + HG_BLOCK / NRHS, ..., then a tree), then the
// scalar step, one thread per right-hand side.  step 0: after r.r of the
// initial residual; 1: after r.z; 2: after p.Ap; 3: after the new r.r.
// *active: the right-hand sides still iterating.
template <int NRHS>
__global__ void __launch_bounds__(HG_BLOCK)
k_hpcg_finish(HgScalars *sc, const double *partials, int nblocks, int step, int64_t iter,
	int64_t max_iter, double tol, int32_t *active) {
	__shared__ double dot[HG_BLOCK];
	if (step != 0 && *active == 0) return;   // uniform: only this kernel's end writes it
	double v = 0.0;
	for (int b = threadIdx.x / NRHS; b < nblocks; b += HG_BLOCK / NRHS)
		v += partials[b * NRHS + threadIdx.x % NRHS];
	dot[threadIdx.x] = v;
	__syncthreads();
	for (int w = HG_BLOCK / 2; w >= NRHS; w >>= 1) {
		if (threadIdx.x < w) dot[threadIdx.x] += dot[threadIdx.x + w];
		__syncthreads();
	}
	const int k = threadIdx.x;
	if (k < NRHS) {
		const bool was = step == 0 || sc[k].active;
		hg_scalar_step(sc[k], dot[k], step, iter, max_iter, tol);
		if (step == 0) atomicAdd(active, 1);
		else if (was && !sc[k].active) atomicSub(active, 1);
	}
}

}  // namespace alpb

namespace alpb {

// 1 where two neighbouring rows share a colour (row index modulo K).
__global__ void k_hpcg_color_conflicts(const int64_t *offsets, const uint32_t *indices, int64_t n,
	int64_t K, int32_t *flag) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
		 i += int64_t(gridDim.x) * blockDim.x)
		for (int64_t j = offsets[i]; j < offsets[i + 1]; ++j) {
			const int64_t c = indices[j];
			if (c != i && (c % K) == (i % K)) atomicExch(flag, 1);
		}
}

// ------------------------------------------------- recognising a system --
// Checks of a caller's level against this handle's (alpb_hpcg_match_level);
// each sets *bad on the first difference it sees.
__global__ void k_hg_words_differ(const uint32_t *a, const uint32_t *b, int64_t words,
	int32_t *bad) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < words;
		 i += int64_t(gridDim.x) * blockDim.x)
		if (a[i] != b[i]) {
			*bad = 1;
			return;
		}
}

// every entry assigned and equal to the handle's diagonal value
__global__ void k_hg_check_diag(const double *d, const uint8_t *flags, int64_t n, double diag,
	int32_t *bad) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
		 i += int64_t(gridDim.x) * blockDim.x)
		if ((flags && !flags[i]) || d[i] != diag) {
			*bad = 1;
			return;
		}
}

// colour c of `colors`: assigned (and true) exactly at the rows i = c mod colors
// (build_static_color_masks, hpcg/matrix_building_utils.hpp:131-165)
__global__ void k_hg_check_mask(const uint8_t *vals, const uint8_t *flags, int64_t n,
	int64_t colors, int64_t c, int32_t *bad) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const bool want = i % colors == c;
		const bool has = flags ? flags[i] != 0 : true;
		if (has != want || (has && vals[i] == 0)) {
			*bad = 1;
			return;
		}
	}
}

// the injection coarsener of build_ndims_coarsener_matrix: coarse row c holds
// one 1 at fine column inj(c)
__global__ void k_hg_check_coarsening(const int64_t *off, const uint32_t *idx, const double *val,
	int64_t nc, int64_t fine_n, int64_t cnx, int64_t cny, int64_t fnx, int64_t fny,
	int32_t *bad) {
	for (int64_t c = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; c <= nc;
		 c += int64_t(gridDim.x) * blockDim.x) {
		if (off[c] != c) {
			*bad = 1;
			return;
		}
		if (c == nc) continue;
		const int64_t cx = c % cnx, cy = (c / cnx) % cny, cz = c / (cnx * cny);
		const int64_t f = 2 * cx + 2 * cy * fnx + 2 * cz * fnx * fny;
		if (f >= fine_n || int64_t(idx[c]) != f || val[c] != 1.0) {
			*bad = 1;
			return;
		}
	}
}

struct HgLevel {
	int64_t nx = 0, ny = 0, nz = 0, n = 0, nnz = 0;
	int64_t *offsets = nullptr;
	uint32_t *indices = nullptr;
	double *values = nullptr;
	double *r = nullptr, *z = nullptr, *temp = nullptr;  // n * nrhs each
	bool fused = true;
};

}  // namespace alpb

using namespace alpb;

struct alpb_hpcg_s {
	std::vector<HgLevel> levels;   // [0] is the finest (the system itself)
	int nrhs = 1;
	int64_t colors = 27;
	double diag = 26.0;
	double *p = nullptr, *ap = nullptr;  // CG vectors of the finest level
	double *partials = nullptr;
	HgScalars *scalars = nullptr;
	GridSync *gs = nullptr;      // the cycle kernel's barrier
	int32_t *active = nullptr;   // right-hand sides still iterating
	int cluster_fits = -1;       // coarse levels in one cluster: -1 not asked yet
	int cycle_fits = -1;         // the cycle kernel's blocks all resident: the same
	int dot_blocks = 0;
};

namespace alpb {

// Levels of up to this many values (rows times right-hand sides) run in one
// cluster of blocks.  Measured us per iteration, levels above / below the line
// in the cluster: 32^3 with 8 right-hand sides 971 / 1334, with 1 652 / 609;
// 64^3 with 8 1593 / 1988, with 1 1044 / 1002 (a line at 32,768 values takes
// the better one of each).
constexpr int64_t HG_CLUSTER_VALUES = 32768;

static void hg_cluster_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr) {
	cfg->blockDim = dim3(HGC_THREADS);
	cfg->gridDim = dim3(HGC_CLUSTER);
	attr->id = cudaLaunchAttributeClusterDimension;
	attr->val.clusterDim.x = HGC_CLUSTER;
	attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
	cfg->attrs = attr;
	cfg->numAttrs = 1;
}

// Whether the current device takes the cluster launch (16 blocks of one
// cluster need as many free SMs in one GPC); asked once per handle.
template <int NRHS>
static bool hg_cluster_fits(alpb_hpcg_s *h) {
	if (h->cluster_fits < 0) {
		cudaLaunchConfig_t cfg = {};
		cudaLaunchAttribute attr[1];
		hg_cluster_config(&cfg, attr);
		int n = 0;
		const bool ok = cudaFuncSetAttribute(k_hpcg_cycle<NRHS, true>,
			cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
			cudaOccupancyMaxActiveClusters(&n, k_hpcg_cycle<NRHS, true>, &cfg) == cudaSuccess;
		cudaGetLastError();
		h->cluster_fits = ok && n > 0;
	}
	return h->cluster_fits != 0;
}

// one launch of the cycle kernel over the levels [l0, l1)
template <int NRHS, bool CLUSTER>
static int hg_cycle_part(alpb_hpcg_s *h, HgCycleArgs &a, int l0, int l1, int part,
	cudaStream_t s) {
	a.l0 = l0;
	a.l1 = l1;
	a.part = part;
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	if (CLUSTER) {
		hg_cluster_config(&cfg, attr);
	} else {
		ALPB_CUDA(cudaMemsetAsync(&h->gs->count, 0, sizeof(h->gs->count), s));
		cfg.blockDim = dim3(HGC_THREADS);
		cfg.gridDim = dim3(sm_count());
		attr[0].id = cudaLaunchAttributeCooperative;
		attr[0].val.cooperative = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
	}
	cfg.stream = s;
	ALPB_CUDA(cudaLaunchKernelEx(&cfg, k_hpcg_cycle<NRHS, CLUSTER>, a));
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// Levels whose colour steps hold more than this many warps' worth of rows run a
// launch per step: what the cycle kernel saves is the launch and a step's latency,
// and beyond this the warps that an SM can hold count more.  Measured us per
// iteration, cycle kernel / launches (items per step of the finest level):
//   8 right-hand sides: 128^3 (78 K) 8434 / 9536, 160 x 144^2 (123 K) 12987 / 12875,
//     160^3 (152 K) 15020 / 14338, 192^3 (262 K) 26408 / 24727
//   4: 128^3 (78 K) 6694 / 7069, 144^3 (111 K) 9907 / 9384, 160^3 (152 K) 12205 / 10293
//   2: 160^3 (76 K) 7617 / 7524, 192^3 (131 K) 11983 / 10650; 8 colours 128^3 (131 K)
//     3899 / 3317
// With one right-hand side a warp takes four rows in both, and the cycle kernel
// stays ahead: 256^3 (155 K) 17359 / 19387, 384^3 (524 K) 59445 / 63526; but not where
// a step is two passes: one colour, 96^3 (221 K) 710 / 684.
constexpr int64_t HG_STEP_ITEMS = 100000;

// Whether level L runs by launches (also where the cycle kernel's one block per
// SM cannot be resident; asked once per handle).
template <int NRHS>
static bool hg_by_launches(alpb_hpcg_s *h, const HgLevel &L) {
	if (h->cycle_fits < 0) {
		h->cycle_fits = cooperative_grid(k_hpcg_cycle<NRHS, false>, HGC_THREADS, 0, 0) >= sm_count();
		cudaGetLastError();
	}
	if (!h->cycle_fits) return true;
	const int64_t rows = (L.n + h->colors - 1) / h->colors;
	return (NRHS > 1 || !L.fused) && rows / HgRow<NRHS>::RPW > HG_STEP_ITEMS;
}

template <int NRHS, class Op>
static int hg_rows(const HgLevel &L, const double *x, int64_t count, const Op &op, cudaStream_t s,
	const int32_t *active = nullptr) {
	if (count <= 0) return ALPB_SUCCESS;
	k_hpcg_rows<NRHS, Op><<<grid_for(count * HG_GROUP, HG_BLOCK), HG_BLOCK, 0, s>>>(L.offsets,
		L.indices, L.values, x, count, op, active);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// red_black_gauss_seidel: colours forward, then backward (:96-117)
template <int NRHS>
static int hg_smoother(alpb_hpcg_s *h, HgLevel &L, cudaStream_t s) {
	const int64_t K = h->colors;
	for (int64_t step = 0; step < 2 * K; ++step) {
		const int64_t c = step < K ? step : 2 * K - 1 - step;
		const int64_t count = c < L.n ? (L.n - 1 - c) / K + 1 : 0;
		HgColor<NRHS> op{L.r, L.z, L.fused ? nullptr : L.temp, h->diag, c, K};
		const int rc = hg_rows<NRHS>(L, L.z, count, op, s);
		if (rc != ALPB_SUCCESS) return rc;
		if (!L.fused && count > 0) {
			k_hpcg_color_update<NRHS><<<grid_for(count * NRHS, 256), 256, 0, s>>>(L.r, L.temp, L.z,
				h->diag, c, K, count);
			ALPB_LAUNCHED();
		}
	}
	return ALPB_SUCCESS;
}

// multi_grid from level l down and back up again: a large level by launches,
// the first level that is not large and those below it by the cycle kernel
template <int NRHS>
static int hg_vcycle(alpb_hpcg_s *h, int l, int64_t pre, int64_t post, cudaStream_t s) {
	const int nl = int(h->levels.size());
	HgLevel &L = h->levels[size_t(l)];
	ALPB_CUDA(cudaMemsetAsync(L.z, 0, size_t(L.n) * NRHS * 8, s));
	int rc = ALPB_SUCCESS;
	if (hg_by_launches<NRHS>(h, L)) {
		if (l + 1 == nl) return hg_smoother<NRHS>(h, L, s);
		for (int64_t i = 0; i < pre && rc == ALPB_SUCCESS; ++i) rc = hg_smoother<NRHS>(h, L, s);
		if (rc != ALPB_SUCCESS) return rc;
		HgLevel &C = h->levels[size_t(l) + 1];
		const HgInject inj{C.nx, C.ny, L.nx, L.ny};
		rc = hg_rows<NRHS>(L, L.z, C.n, HgRestrict<NRHS>{L.r, C.r, inj}, s);
		rc = rc ? rc : hg_vcycle<NRHS>(h, l + 1, pre, post, s);
		if (rc != ALPB_SUCCESS) return rc;
		k_hpcg_prolong<NRHS><<<grid_for(C.n * NRHS, 256), 256, 0, s>>>(L.z, C.z, inj, C.n);
		ALPB_LAUNCHED();
		for (int64_t i = 0; i < post && rc == ALPB_SUCCESS; ++i) rc = hg_smoother<NRHS>(h, L, s);
		return rc;
	}
	HgCycleArgs a;
	int coarse = nl;   // first level of the cluster launch
	for (int q = nl - 1; q >= l; --q) {
		const HgLevel &Q = h->levels[size_t(q)];
		a.lv[q] = HgLevelArgs{Q.offsets, Q.indices, Q.values, Q.r, Q.z, Q.fused ? nullptr : Q.temp,
			Q.n, Q.nx, Q.ny};
		if (Q.n * NRHS <= HG_CLUSTER_VALUES && hg_cluster_fits<NRHS>(h)) coarse = q;
	}
	a.colors = h->colors;
	a.pre = pre;
	a.post = post;
	a.diag = h->diag;
	a.gs = h->gs;
	a.active = h->active;
	if (coarse == nl) return hg_cycle_part<NRHS, false>(h, a, l, nl, HG_WHOLE, s);
	if (coarse > l) rc = hg_cycle_part<NRHS, false>(h, a, l, coarse, HG_DOWN, s);
	rc = rc ? rc : hg_cycle_part<NRHS, true>(h, a, coarse, nl, HG_WHOLE, s);
	if (coarse > l) rc = rc ? rc : hg_cycle_part<NRHS, false>(h, a, l, coarse, HG_UP, s);
	return rc;
}

template <int NRHS>
static int hg_finish(alpb_hpcg_s *h, int step, int64_t iter, int64_t max_iter, double tol,
	cudaStream_t s) {
	k_hpcg_finish<NRHS><<<1, HG_BLOCK, 0, s>>>(h->scalars, h->partials, h->dot_blocks, step, iter,
		max_iter, tol, h->active);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

template <int NRHS>
static int hg_dot(alpb_hpcg_s *h, const double *x, const double *y, cudaStream_t s,
	const int32_t *active) {
	k_hpcg_dot<NRHS><<<h->dot_blocks, HG_BLOCK, 0, s>>>(x, y, h->levels[0].n, h->partials, active);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// Ap = A x and the partials of x . Ap: k_hpcg_spmm while a row's entries in flight
// are what counts, a walk over the rows in few registers and a pass for the dot
// product where warps are.  Measured us per iteration without preconditioner, walk /
// k_hpcg_spmm: 8 right-hand sides 48^3 121 / 103, 64^3 147 / 192, 104^3 470 / 751,
// 160^3 1504 / 2544; 4: 80^3 193 / 181, 104^3 285 / 346; 2: 128^3 339 / 337, 160^3
// 596 / 635; 1: 160^3 479 / 362, 256^3 2078 / 1497.
constexpr int64_t HG_WALK = int64_t(1) << 23;   // rows * nrhs^2
template <int NRHS>
static int hg_spmm(alpb_hpcg_s *h, const double *x, cudaStream_t s, const int32_t *active) {
	const HgLevel &L = h->levels[0];
	if (NRHS > 1 && L.n * NRHS * NRHS > HG_WALK) {
		const int rc = hg_rows<NRHS>(L, x, L.n, HgSpmm<NRHS>{h->ap}, s, active);
		return rc ? rc : hg_dot<NRHS>(h, x, h->ap, s, active);
	}
	k_hpcg_spmm<NRHS><<<h->dot_blocks, HG_BLOCK, 0, s>>>(L.offsets, L.indices, L.values, x, h->ap,
		L.n, h->partials, active);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// The host looks whether any right-hand side is left after the first and every
// HG_QUEUE-th iteration: a look takes about 30 us, and the kernels of an iteration
// too many find none and return.
constexpr int64_t HG_QUEUE = 4;

// algorithms::hpcg (hpcg.hpp:97-223) for NRHS right-hand sides at once
template <int NRHS>
static int hg_solve(alpb_hpcg_s *h, const double *b, double *x, bool precondition, int64_t pre,
	int64_t post, int64_t max_iter, double tol, int64_t *iterations, double *residuals,
	cudaStream_t s) {
	HgLevel &L = h->levels[0];
	const int64_t n = L.n;
	const unsigned g = grid_for(n * NRHS, 256);
	ALPB_CUDA(cudaMemsetAsync(h->gs, 0, sizeof(GridSync), s));
	ALPB_CUDA(cudaMemsetAsync(h->active, 0, 4, s));
	// Ap = 0; r = 0; p = x; Ap = A x; r = b - Ap; norm = sqrt(r.r)
	ALPB_CUDA(cudaMemcpyAsync(h->p, x, size_t(n) * NRHS * 8, cudaMemcpyDeviceToDevice, s));
	int rc = hg_spmm<NRHS>(h, x, s, nullptr);
	if (rc != ALPB_SUCCESS) return rc;
	k_hpcg_axpby<NRHS><<<g, 256, 0, s>>>(L.r, h->ap, b, h->scalars, 0, n, nullptr);
	ALPB_LAUNCHED();
	rc = hg_dot<NRHS>(h, L.r, L.r, s, nullptr);
	rc = rc ? rc : hg_finish<NRHS>(h, 0, 0, max_iter, tol, s);
	if (rc != ALPB_SUCCESS) return rc;
	HgScalars hs[NRHS];
	GridSync hgs;
	// a large system's iteration is worth far more than a look at the state
	const int64_t queue = precondition && hg_by_launches<NRHS>(h, L) ? 1 : HG_QUEUE;
	for (int64_t iter = 0;; ++iter) {
		if (precondition) {
			rc = hg_vcycle<NRHS>(h, 0, pre, post, s);
			if (rc != ALPB_SUCCESS) return rc;
		} else {
			ALPB_CUDA(cudaMemcpyAsync(L.z, L.r, size_t(n) * NRHS * 8, cudaMemcpyDeviceToDevice, s));
		}
		// r.z, beta; p = z (first iteration) or p = beta p + z
		rc = hg_dot<NRHS>(h, L.r, L.z, s, h->active);
		rc = rc ? rc : hg_finish<NRHS>(h, 1, iter, max_iter, tol, s);
		if (rc != ALPB_SUCCESS) return rc;
		if (iter == 0) {
			ALPB_CUDA(cudaMemcpyAsync(h->p, L.z, size_t(n) * NRHS * 8, cudaMemcpyDeviceToDevice, s));
		} else {
			// into Ap, then swapped with p (hpcg.hpp:193-196)
			k_hpcg_axpby<NRHS><<<g, 256, 0, s>>>(h->ap, h->p, L.z, h->scalars, 1, n, h->active);
			ALPB_LAUNCHED();
			double *t = h->p;
			h->p = h->ap;
			h->ap = t;
		}
		// Ap = A p; alpha = r.z / p.Ap; x += alpha p; r -= alpha Ap; norm
		rc = hg_spmm<NRHS>(h, h->p, s, h->active);
		rc = rc ? rc : hg_finish<NRHS>(h, 2, iter, max_iter, tol, s);
		if (rc != ALPB_SUCCESS) return rc;
		k_hpcg_update<NRHS><<<h->dot_blocks, HG_BLOCK, 0, s>>>(x, L.r, h->p, h->ap, h->scalars, n,
			h->partials, h->active);
		ALPB_LAUNCHED();
		rc = hg_finish<NRHS>(h, 3, iter, max_iter, tol, s);
		if (rc != ALPB_SUCCESS) return rc;
		if (iter >= 1 && iter % queue != queue - 1 && iter + 1 < max_iter) continue;
		ALPB_CUDA(cudaMemcpyAsync(hs, h->scalars, sizeof(hs), cudaMemcpyDeviceToHost, s));
		ALPB_CUDA(cudaMemcpyAsync(&hgs, h->gs, sizeof(hgs), cudaMemcpyDeviceToHost, s));
		ALPB_CUDA(cudaStreamSynchronize(s));
		ALPB_CHECK(hgs.err == 0, ALPB_PANIC, "alpb_hpcg_solve: a grid barrier timed out");
		bool any = false;
		for (int k = 0; k < NRHS; ++k) any = any || hs[k].active;
		if (!any) break;
	}
	for (int k = 0; k < NRHS; ++k) {
		if (iterations) iterations[k] = hs[k].iterations;
		if (residuals) residuals[k] = hs[k].norm;
	}
	return ALPB_SUCCESS;
}

}  // namespace alpb

extern "C" {

int alpb_hpcg_destroy(alpb_hpcg h) {
	if (!h) return ALPB_SUCCESS;
	for (HgLevel &L : h->levels) {
		cudaFree(L.offsets);
		cudaFree(L.indices);
		cudaFree(L.values);
		cudaFree(L.r);
		cudaFree(L.z);
		cudaFree(L.temp);
	}
	cudaFree(h->p);
	cudaFree(h->ap);
	cudaFree(h->partials);
	cudaFree(h->gs);
	cudaFree(h->active);
	cudaFree(h->scalars);
	delete h;
	return ALPB_SUCCESS;
}

int alpb_hpcg_create(alpb_hpcg *out, int64_t nx, int64_t ny, int64_t nz, double diag,
	double off, int64_t colors, int64_t min_size, int64_t max_levels, int nrhs, void *stream) {
	ALPB_CHECK(out != nullptr, ALPB_ILLEGAL, "alpb_hpcg_create: null handle");
	*out = nullptr;
	ALPB_CHECK(nx > 0 && ny > 0 && nz > 0 && colors > 0 && min_size > 0 && max_levels >= 0,
		ALPB_ILLEGAL, "alpb_hpcg_create: bad sizes");
	ALPB_CHECK(nrhs == 1 || nrhs == 2 || nrhs == 4 || nrhs == 8, ALPB_UNSUPPORTED,
		"alpb_hpcg_create: %d right-hand sides (1, 2, 4 or 8)", nrhs);
	ALPB_CHECK(diag != 0.0, ALPB_ILLEGAL, "alpb_hpcg_create: zero diagonal");
	ALPB_CHECK(nx * ny * nz >= colors, ALPB_ILLEGAL,
		"alpb_hpcg_create: fewer rows than colours");  // build_static_color_masks
	cudaStream_t s = as_stream(stream);
	auto *h = new alpb_hpcg_s();
	h->nrhs = nrhs;
	h->colors = colors;
	h->diag = diag;
	// levels as build_hpcg_system makes them (system_building_utils.hpp:107-147)
	std::vector<int64_t> dims = {nx, ny, nz};
	int64_t min_coarse = std::min(nx, std::min(ny, nz)) / 2;
	h->levels.push_back(HgLevel{});
	h->levels.back().nx = nx;
	h->levels.back().ny = ny;
	h->levels.back().nz = nz;
	int64_t level = 0;
	while (min_coarse >= min_size && level < max_levels) {
		HgLevel c;
		c.nx = h->levels.back().nx / 2;
		c.ny = h->levels.back().ny / 2;
		c.nz = h->levels.back().nz / 2;
		if (c.nx * 2 != h->levels.back().nx || c.ny * 2 != h->levels.back().ny ||
			c.nz * 2 != h->levels.back().nz) {
			alpb_hpcg_destroy(h);
			set_error("alpb_hpcg_create: level sizes must halve exactly");
			return ALPB_ILLEGAL;
		}
		h->levels.push_back(c);
		min_coarse /= 2;
		++level;
	}
	int32_t *flag = nullptr;
	int rc = ALPB_SUCCESS;
	if (cudaMallocAsync(&flag, 4, s) != cudaSuccess) {
		alpb_hpcg_destroy(h);
		set_error("alpb_hpcg_create: out of device memory");
		return ALPB_OUTOFMEM;
	}
	for (HgLevel &L : h->levels) {
		L.n = L.nx * L.ny * L.nz;
		int64_t sizes[4] = {L.nx, L.ny, L.nz, 0};
		if (cudaMalloc(&L.offsets, size_t(L.n + 1) * 8) != cudaSuccess) {
			cudaGetLastError();
			rc = ALPB_OUTOFMEM;
			set_error("alpb_hpcg_create: out of device memory");
			break;
		}
		// first call: row offsets and the nonzero count
		rc = alpb_gen_stencil_crs(3, sizes, diag, off, 1, L.offsets, nullptr, nullptr, &L.nnz,
			stream);
		if (rc != ALPB_SUCCESS) break;
		const size_t vbytes = size_t(L.n) * nrhs * 8;
		if (cudaMalloc(&L.indices, size_t(L.nnz) * 4) != cudaSuccess ||
			cudaMalloc(&L.values, size_t(L.nnz) * 8) != cudaSuccess ||
			cudaMalloc(&L.r, vbytes) != cudaSuccess || cudaMalloc(&L.z, vbytes) != cudaSuccess) {
			cudaGetLastError();
			rc = ALPB_OUTOFMEM;
			set_error("alpb_hpcg_create: out of device memory");
			break;
		}
		rc = alpb_gen_stencil_crs(3, sizes, diag, off, 1, L.offsets, L.indices, L.values, &L.nnz,
			stream);
		if (rc != ALPB_SUCCESS) break;
		// the smoother fuses a colour's product and update when no two
		// neighbours share a colour
		int32_t conflict = 0;
		if (cudaMemsetAsync(flag, 0, 4, s) != cudaSuccess) { rc = ALPB_PANIC; break; }
		k_hpcg_color_conflicts<<<grid_for(L.n, 256), 256, 0, s>>>(L.offsets, L.indices, L.n,
			colors, flag);
		ALPB_LAUNCHED();
		if (cudaMemcpyAsync(&conflict, flag, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
			cudaStreamSynchronize(s) != cudaSuccess) {
			rc = ALPB_PANIC;
			set_error("alpb_hpcg_create: colour check failed");
			break;
		}
		L.fused = conflict == 0;
		if (!L.fused && cudaMalloc(&L.temp, vbytes) != cudaSuccess) {
			cudaGetLastError();
			rc = ALPB_OUTOFMEM;
			set_error("alpb_hpcg_create: out of device memory");
			break;
		}
	}
	cudaFreeAsync(flag, s);
	const int64_t n0 = h->levels[0].n;
	if (rc == ALPB_SUCCESS) {
		h->dot_blocks = int(grid_for(n0 * nrhs, HG_BLOCK, 8));
		if (cudaMalloc(&h->p, size_t(n0) * nrhs * 8) != cudaSuccess ||
			cudaMalloc(&h->ap, size_t(n0) * nrhs * 8) != cudaSuccess ||
			cudaMalloc(&h->partials, size_t(h->dot_blocks) * nrhs * 8) != cudaSuccess ||
			cudaMalloc(&h->gs, sizeof(GridSync)) != cudaSuccess ||
			cudaMalloc(&h->active, 4) != cudaSuccess ||
			cudaMalloc(&h->scalars, size_t(nrhs) * sizeof(HgScalars)) != cudaSuccess) {
			cudaGetLastError();
			rc = ALPB_OUTOFMEM;
			set_error("alpb_hpcg_create: out of device memory");
		}
	}
	if (rc != ALPB_SUCCESS) {
		alpb_hpcg_destroy(h);
		return rc;
	}
	*out = h;
	return ALPB_SUCCESS;
}

int alpb_hpcg_info(alpb_hpcg h, int64_t *levels, int64_t *n_finest, int64_t *nnz_finest,
	int *fused_smoother) {
	ALPB_CHECK(h != nullptr, ALPB_ILLEGAL, "alpb_hpcg_info: null handle");
	if (levels) *levels = int64_t(h->levels.size());
	if (n_finest) *n_finest = h->levels[0].n;
	if (nnz_finest) *nnz_finest = h->levels[0].nnz;
	if (fused_smoother) {
		int all = 1;
		for (const HgLevel &L : h->levels) all &= L.fused ? 1 : 0;
		*fused_smoother = all;
	}
	return ALPB_SUCCESS;
}

int alpb_hpcg_matrix(alpb_hpcg h, int64_t level, const int64_t **offsets,
	const uint32_t **indices, const double **values, int64_t *n, int64_t *nnz) {
	ALPB_CHECK(h != nullptr && level >= 0 && level < int64_t(h->levels.size()), ALPB_ILLEGAL,
		"alpb_hpcg_matrix: no level %lld", (long long) level);
	const HgLevel &L = h->levels[size_t(level)];
	if (offsets) *offsets = L.offsets;
	if (indices) *indices = L.indices;
	if (values) *values = L.values;
	if (n) *n = L.n;
	if (nnz) *nnz = L.nnz;
	return ALPB_SUCCESS;
}

int alpb_hpcg_solve(alpb_hpcg h, const double *b, double *x, int with_preconditioning,
	int64_t presmoother_steps, int64_t postsmoother_steps, int64_t max_iterations,
	double tolerance, int64_t *iterations, double *residuals, void *stream) {
	ALPB_CHECK(h != nullptr && b != nullptr && x != nullptr, ALPB_ILLEGAL,
		"alpb_hpcg_solve: null argument");
	ALPB_CHECK(max_iterations > 0 && presmoother_steps >= 0 && postsmoother_steps >= 0,
		ALPB_ILLEGAL, "alpb_hpcg_solve: bad iteration counts");
	cudaStream_t s = as_stream(stream);
	const bool pc = with_preconditioning != 0;
	switch (h->nrhs) {
	case 1: return hg_solve<1>(h, b, x, pc, presmoother_steps, postsmoother_steps, max_iterations,
		tolerance, iterations, residuals, s);
	case 2: return hg_solve<2>(h, b, x, pc, presmoother_steps, postsmoother_steps, max_iterations,
		tolerance, iterations, residuals, s);
	case 4: return hg_solve<4>(h, b, x, pc, presmoother_steps, postsmoother_steps, max_iterations,
		tolerance, iterations, residuals, s);
	default: return hg_solve<8>(h, b, x, pc, presmoother_steps, postsmoother_steps,
		max_iterations, tolerance, iterations, residuals, s);
	}
}

int alpb_hpcg_match_level(alpb_hpcg h, int64_t level, int64_t n, int64_t nnz,
	const int64_t *offsets, const uint32_t *indices, const double *values, const double *diagonal,
	const uint8_t *diagonal_flags, int64_t colors, const uint8_t *const *mask_values,
	const uint8_t *const *mask_flags, int64_t coarse_nnz, const int64_t *coarse_offsets,
	const uint32_t *coarse_indices, const double *coarse_values, int *matches, void *stream) {
	ALPB_CHECK(h != nullptr && matches != nullptr, ALPB_ILLEGAL,
		"alpb_hpcg_match_level: null argument");
	*matches = 0;
	if (level < 0 || level >= int64_t(h->levels.size())) return ALPB_SUCCESS;
	const HgLevel &L = h->levels[size_t(level)];
	if (n != L.n || nnz != L.nnz || colors != h->colors || !offsets || (nnz && (!indices ||
			!values)) || !diagonal || (colors && (!mask_values || !mask_flags)))
		return ALPB_SUCCESS;
	if (level > 0 && (coarse_nnz != L.n || !coarse_offsets || !coarse_indices || !coarse_values))
		return ALPB_SUCCESS;
	cudaStream_t s = as_stream(stream);
	int32_t *bad = nullptr;
	ALPB_CUDA(cudaMallocAsync(&bad, 4, s));
	ALPB_CUDA(cudaMemsetAsync(bad, 0, 4, s));
	const void *const pa[3] = {offsets, indices, values};
	const void *const pb[3] = {L.offsets, L.indices, L.values};
	const int64_t nw[3] = {2 * (n + 1), nnz, 2 * nnz};   // 4-byte words
	for (int k = 0; k < 3; ++k) {
		if (nw[k] == 0) continue;
		k_hg_words_differ<<<grid_for(nw[k], 256, 2), 256, 0, s>>>(
			static_cast<const uint32_t *>(pa[k]), static_cast<const uint32_t *>(pb[k]), nw[k], bad);
		ALPB_LAUNCHED();
	}
	k_hg_check_diag<<<grid_for(n, 256, 2), 256, 0, s>>>(diagonal, diagonal_flags, n, h->diag,
		bad);
	ALPB_LAUNCHED();
	for (int64_t c = 0; c < colors; ++c) {
		k_hg_check_mask<<<grid_for(n, 256, 2), 256, 0, s>>>(mask_values[c], mask_flags[c], n,
			colors, c, bad);
		ALPB_LAUNCHED();
	}
	if (level > 0) {
		const HgLevel &F = h->levels[size_t(level - 1)];
		k_hg_check_coarsening<<<grid_for(L.n + 1, 256, 2), 256, 0, s>>>(coarse_offsets,
			coarse_indices, coarse_values, L.n, F.n, L.nx, L.ny, F.nx, F.ny, bad);
		ALPB_LAUNCHED();
	}
	int32_t hb = 1;
	ALPB_CUDA(cudaMemcpyAsync(&hb, bad, 4, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(bad, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	*matches = hb == 0 ? 1 : 0;
	return ALPB_SUCCESS;
}

}  // extern "C"
