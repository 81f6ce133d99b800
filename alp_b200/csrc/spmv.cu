// Sparse matrix times dense/sparse vector over a semiring: the replacement of
// internal::vxm_generic + vxm_inner_kernel_gather
// (include/graphblas/reference/blas2.hpp:283-551, 835-1528).
//
// Two schedules gather over a compressed storage whose outer dimension is the
// output (CRS for mxv, CCS for vxm, as the reference does):
//
//  * merge path (dense fast path, merge.cuh): the (rows + nonzeroes) merge
//    list is cut in equal tiles (Merrill & Garland, "Merge-based parallel
//    sparse matrix-vector multiplication", SC'16), so power-law rows cost the
//    same as uniform ones; one launch, sums in a fixed order (deterministic).
//  * vector: short rows of nearly one length stream through shared memory where
//    that is faster (rowstream.cuh, rows_pay), others take W lanes per row; the
//    general path (launch_general: W lanes walking a row, or batched with long
//    rows cut in chunks) carries every ALP semantic of the reference gather:
//    output/input masks (value or structural, inverted), sparse input and
//    output vectors with assigned flags, add_identity, use_index,
//    explicit_zero and the immutable-nonzero shortcut of lor.
#include "common.cuh"
#include "spmv.cuh"
#include "merge.cuh"
#include "wmerge.cuh"
#include "rowstream.cuh"

#include <algorithm>
#include <vector>

namespace alpb {

// ------------------------------------------------------------ plan layout --
// merge-path split of diagonal d: rows consumed i, nonzeroes consumed d - i
__device__ __forceinline__ int64_t merge_search_global(const int64_t *offsets, int64_t m,
	int64_t nnz, int64_t d) {
	int64_t lo = d - nnz > 0 ? d - nnz : 0;
	int64_t hi = d < m ? d : m;
	while (lo < hi) {
		const int64_t pivot = (lo + hi) >> 1;
		// row end of row `pivot` is offsets[pivot + 1]
		if (offsets[pivot + 1] <= d - pivot - 1) lo = pivot + 1; else hi = pivot;
	}
	return lo;
}

__global__ void k_merge_tiles(const int64_t *offsets, int64_t m, int64_t nnz, int64_t ntiles,
	int64_t *tile_row, int64_t tile) {
	for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t <= ntiles;
		 t += int64_t(gridDim.x) * blockDim.x) {
		int64_t d = t * tile;
		if (d > m + nnz) d = m + nnz;
		tile_row[t] = merge_search_global(offsets, m, nnz, d);
	}
}

__global__ void k_row_stats(const int64_t *offsets, int64_t m, unsigned long long *maxlen,
	double *sumsq) {
	int64_t lmax = 0;
	double lsq = 0.0;
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int64_t len = offsets[i + 1] - offsets[i];
		lmax = len > lmax ? len : lmax;
		lsq += double(len) * double(len);
	}
	for (int o = 16; o > 0; o >>= 1) {
		const int64_t om = __shfl_down_sync(0xffffffffu, lmax, o);
		lmax = om > lmax ? om : lmax;
		lsq += __shfl_down_sync(0xffffffffu, lsq, o);
	}
	if ((threadIdx.x & 31) == 0) {
		atomicMax(maxlen, (unsigned long long) lmax);
		atomicAdd(sumsq, lsq);
	}
}

// Spanning-row tables of the merge path (see merge.cuh): for each tile, the
// first tile of its head / tail row when that row crosses tiles, and for the
// first tile of a spanning row the number of tiles it covers.
__global__ void k_merge_tables(const int64_t *offsets, int64_t m, int64_t nnz, int64_t ntiles,
	const int64_t *tile_row, int64_t *head_first, int64_t *tail_first, int32_t *span_len,
	int64_t tile) {
	for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < ntiles;
		 t += int64_t(gridDim.x) * blockDim.x) {
		const int64_t i0 = tile_row[t], i1 = tile_row[t + 1];
		const int64_t d0 = t * tile;
		int64_t d1 = d0 + tile;
		if (d1 > m + nnz) d1 = m + nnz;
		const int64_t j0 = d0 - i0, j1 = d1 - i1;
		head_first[t] = (i1 > i0 && offsets[i0] < j0) ? (i0 + offsets[i0]) / tile : -1;
		int64_t tf = -1;
		if (i1 < m) {
			const int64_t start = offsets[i1] > j0 ? offsets[i1] : j0;
			if (j1 > start) tf = (i1 + offsets[i1]) / tile;
		}
		tail_first[t] = tf;
		span_len[t] = (tf == t) ? int32_t((i1 + offsets[i1 + 1]) / tile - t + 1) : 0;
	}
}

// Row-aligned warp tiles: tile t holds rows [t R, (t+1) R) whole, R chosen so
// that R rows never exceed one tile's items.  No row crosses a tile.
__global__ void k_row_aligned_tiles(const int64_t *offsets, int64_t m, int64_t rows_per_tile,
	int64_t ntiles, int64_t *tile_row, int64_t *tile_d, int64_t *head_first, int64_t *tail_first,
	int32_t *span_len) {
	for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t <= ntiles;
		 t += int64_t(gridDim.x) * blockDim.x) {
		int64_t r = t * rows_per_tile;
		if (r > m) r = m;
		tile_row[t] = r;
		tile_d[t] = r + offsets[r];
		if (t < ntiles) {
			head_first[t] = -1;
			tail_first[t] = -1;
			span_len[t] = 0;
		}
	}
}

// Rows per row-aligned warp tile for rows of at most `maxlen` (mean `mean`)
// nonzeroes, or 0 when whole-row tiles would not stay at least half full.
int64_t aligned_rows_per_tile(double maxlen, double mean, int64_t tile) {
	if (maxlen > double(tile) / 8) return 0;
	const int64_t r = tile / (int64_t(maxlen) + 1);
	return double(r) * (mean + 1.0) >= 0.5 * double(tile) ? r : 0;
}

// Longest row and mean row length of a compressed storage (synchronises).
int row_profile(const int64_t *offsets, int64_t m, double *maxlen, double *sumsq,
	cudaStream_t s) {
	unsigned long long *d_max = nullptr;
	double *d_sq = nullptr;
	ALPB_CUDA(cudaMallocAsync(&d_max, 8, s));
	ALPB_CUDA(cudaMallocAsync(&d_sq, 8, s));
	ALPB_CUDA(cudaMemsetAsync(d_max, 0, 8, s));
	ALPB_CUDA(cudaMemsetAsync(d_sq, 0, 8, s));
	if (m > 0) {
		k_row_stats<<<grid_for(m, 256, 4), 256, 0, s>>>(offsets, m, d_max, d_sq);
		ALPB_LAUNCHED();
	}
	unsigned long long hmax = 0;
	double hsq = 0;
	ALPB_CUDA(cudaMemcpyAsync(&hmax, d_max, 8, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaMemcpyAsync(&hsq, d_sq, 8, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(d_max, s));
	ALPB_CUDA(cudaFreeAsync(d_sq, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	*maxlen = double(hmax);
	if (sumsq) *sumsq = hsq;
	return ALPB_SUCCESS;
}

MergeTables merge_tables(const alpb_spmv_plan_s &p) {
	MergeTables t;
	t.m = p.m;
	t.nnz = p.nnz;
	t.ntiles = p.ntiles;
	t.tile_row = p.tile_row;
	t.head_first = p.head_first;
	t.tail_first = p.tail_first;
	t.span_len = p.span_len;
	t.counter = p.counter;
	t.head_val = p.head_val;
	t.tail_val = p.tail_val;
	t.head_has = p.head_has;
	t.tail_has = p.tail_has;
	t.ready = p.ready;
	t.tile_d = p.tile_d;
	return t;
}

// ------------------------------------------------------- merge-path SpMV --
template <class R>
struct AccumulateY {
	typename R::T *__restrict__ y;
	__device__ __forceinline__ void row(int64_t r, typename R::T v, bool has) {
		if (has) y[r] = R::add(y[r], v);  // foldl( y_r, row sum ), blas2.hpp:534-549
	}
	__device__ __forceinline__ void row_span(int64_t, int64_t r, typename R::T v, bool has) {
		row(r, v, has);
	}
	// the same in two halves (k_wm_fixup)
	__device__ __forceinline__ typename R::T load(int64_t r) const { return y[r]; }
	__device__ __forceinline__ void finish(int64_t r, typename R::T v, typename R::T old) const {
		y[r] = R::add(old, v);
	}
};

template <class R>
__global__ void __launch_bounds__(MP_BLOCK)
k_spmv_merge(MergeTables mt, const int64_t *__restrict__ offsets,
	const uint32_t *__restrict__ indices, const typename R::T *__restrict__ values,
	const typename R::T *__restrict__ x, typename R::T *__restrict__ y, int left) {
	__shared__ MergeSmem<R> sm;
	PlainX<typename R::T> xl{x};
	AccumulateY<R> epi{y};
	for (int64_t t = blockIdx.x; t < mt.ntiles; t += gridDim.x)
		merge_tile<R>(t, mt, offsets, indices, values, xl, epi, left, sm);
}

// Warp-tile merge path (wmerge.cuh): persistent warps, one warp tile at a
// time, no block-wide barrier.
#ifndef ALPB_WM_WARPS
#define ALPB_WM_WARPS 8
#endif
constexpr int WM_WARPS = ALPB_WM_WARPS;  // warps per block
#ifndef ALPB_WM_MIN_BLOCKS
#define ALPB_WM_MIN_BLOCKS 3  // caps registers at 84: three blocks of eight warps per SM
#endif

// y_r = y_r (+) row sum for the rows that end in a warp tile; their old
// values are fetched into the warp's shared memory with the tile, so that
// finishing a row is one store instead of a dependent load and store.
template <class R>
struct WarpAccumulateY {
	using T = typename R::T;
	T *__restrict__ y;
	T *ybuf;            // WM_TILE entries of the warp's shared memory
	int64_t base = 0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) ybuf[k] = y[i0 + k];
	}
	__device__ __forceinline__ void row(int64_t r, T v, bool has) {
		if (has) y[r] = R::add(ybuf[r - base], v);  // foldl( y_r, row sum ), blas2.hpp:534-549
	}
};

template <class R, class XL>
__global__ void __launch_bounds__(32 * WM_WARPS, ALPB_WM_MIN_BLOCKS)
k_spmv_wmerge(MergeTables mt, const int64_t *__restrict__ offsets,
	const uint32_t *__restrict__ indices, const typename R::T *__restrict__ values,
	XL xl, typename R::T *__restrict__ y, int left) {
	__shared__ WarpSmem<R> sm[WM_WARPS];
	__shared__ typename R::T ybuf[WM_WARPS][WM_TILE];
	WarpAccumulateY<R> epi{y, ybuf[threadIdx.x >> 5]};
	const int w = threadIdx.x >> 5;
	const int64_t nw = int64_t(gridDim.x) * WM_WARPS;
	int64_t t = int64_t(blockIdx.x) * WM_WARPS + w;
	WmMeta g = wm_meta(mt, t);
	while (t < mt.ntiles) {
		const WmMeta next = wm_meta(mt, t + nw);
		warp_tile<R, XL, WarpAccumulateY<R>, WarpSmem<R>, WM_LOADS_FIRST | WM_WALK_AHEAD>(t, g, mt,
			offsets, indices, values, xl, epi, left, sm[w]);
		t += nw;
		g = next;
	}
}

// ------------------------------------------------- hot-column cache path --
// The same warp tiles as k_spmv_wmerge, on a plan whose hot_idx marks the
// nonzeroes of its hot columns: one block per SM copies the hot columns'
// x values (gathered once per product into hot_x) into shared memory, and
// the staging loop reads a marked column from there instead of from global
// memory.  Products and sums are those of k_spmv_wmerge, bit for bit.
constexpr uint32_t kHotBit = 0x80000000u;
#ifndef ALPB_HOT_WARPS
#define ALPB_HOT_WARPS 32
#endif
constexpr int HOT_WARPS = ALPB_HOT_WARPS;   // one block of these per SM

template <class T>
struct HotX {
	const T *xs;
	const T *__restrict__ x;
	__device__ __forceinline__ T operator()(uint32_t c) const {
		// the cold columns' x through L2 only: L1 space is left to the misses
		// in flight (with most of the SM's memory given to shared slots, an
		// allocating load held the gathers back measurably at 12 K+ slots)
		return (c & kHotBit) ? xs[c ^ kHotBit] : __ldcg(x + c);
	}
};

// Shared memory of one block: the warps' compact tiles (products, row ends
// and the y of the tile's rows), then the hot-column slots.
template <class R>
struct HotSmem {
	static constexpr size_t warp_bytes = (sizeof(WarpSmemCompact<R>) + 15) / 16 * 16;
	static constexpr size_t x_off = warp_bytes * HOT_WARPS;
	static size_t bytes(int64_t hot_k) { return x_off + size_t(hot_k) * sizeof(typename R::T); }
};

// y_r = y_r (+) row sum, with the y of the tile's rows fetched into the
// compact tile's buffer at the start of the tile (as WarpAccumulateY).
template <class R>
struct HotAccumulateY {
	using T = typename R::T;
	T *__restrict__ y;
	WarpSmemCompact<R> *sm;
	int64_t base = 0;
	__device__ __forceinline__ void begin_tile(int64_t i0, int nrows, int lane) {
		base = i0;
		for (int k = lane; k < nrows; k += 32) sm->y(k) = y[i0 + k];
	}
	__device__ __forceinline__ void row(int64_t r, T v, bool has) {
		if (has) y[r] = R::add(sm->y(int(r - base)), v);  // foldl( y_r, row sum )
	}
};

__global__ void k_col_counts(const uint32_t *__restrict__ idx, int64_t nnz, uint32_t *cnt) {
	for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nnz;
		 k += int64_t(gridDim.x) * blockDim.x)
		atomicAdd(cnt + idx[k], 1u);
}

__global__ void k_hot_remap(const uint32_t *__restrict__ idx, int64_t nnz,
	const int32_t *__restrict__ slot, uint32_t *out) {
	for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nnz;
		 k += int64_t(gridDim.x) * blockDim.x) {
		const uint32_t c = idx[k];
		const int32_t sl = slot[c];
		out[k] = sl >= 0 ? (kHotBit | uint32_t(sl)) : c;
	}
}

template <class T>
__global__ void k_hot_gather(const uint32_t *__restrict__ cols, const T *__restrict__ x,
	T *__restrict__ hx, int64_t k) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < k;
		 i += int64_t(gridDim.x) * blockDim.x)
		hx[i] = x[cols[i]];
}

template <class R>
__global__ void __launch_bounds__(32 * HOT_WARPS, 1)
k_spmv_wmerge_hot(MergeTables mt, const int64_t *__restrict__ offsets,
	const uint32_t *__restrict__ hot_idx, const typename R::T *__restrict__ values,
	const typename R::T *__restrict__ x, const typename R::T *__restrict__ hx, int64_t hot_k,
	typename R::T *__restrict__ y, int left) {
	using T = typename R::T;
	extern __shared__ __align__(16) unsigned char hot_smem[];
	T *xs = reinterpret_cast<T *>(hot_smem + HotSmem<R>::x_off);
	for (int64_t i = threadIdx.x; i < hot_k; i += blockDim.x) xs[i] = hx[i];
	__syncthreads();
	const int w = threadIdx.x >> 5;
	HotX<T> xl{xs, x};
	WarpSmemCompact<R> &mine =
		*reinterpret_cast<WarpSmemCompact<R> *>(hot_smem + HotSmem<R>::warp_bytes * w);
	HotAccumulateY<R> epi{y, &mine};
	const int64_t nw = int64_t(gridDim.x) * HOT_WARPS;
	int64_t t = int64_t(blockIdx.x) * HOT_WARPS + w;
	WmMeta g = wm_meta(mt, t);
	while (t < mt.ntiles) {
		const WmMeta next = wm_meta(mt, t + nw);
		warp_tile<R, HotX<T>, HotAccumulateY<R>, WarpSmemCompact<R>, WM_WALK_AHEAD>(t, g, mt, offsets,
			hot_idx, values, xl, epi, left, mine);
		t += nw;
		g = next;
	}
}

// ---------------------------------------------- boolean lor/land (dense) --
// u_i = u_i OR (OR_k a_ik AND x_j) on the dense fast path.  The lor monoid has
// immutable nonzeroes (grb::has_immutable_nonzeroes, monoid.hpp:139-146): once
// u_i is true no product changes it.  So a row whose u_i is already true is
// skipped, as the reference's gather does (blas2.hpp:351-357), and a row stops
// at its first true product.  OR is idempotent and order-free, so the result
// is the full gather's, bit for bit, whatever order the products run in.
//  * k_lor_head: LOR_W lanes per row over the row's first LOR_HEAD nonzeroes,
//    LOR_W products per round, the group's ballot ends the row;
//  * k_lor_tail: one warp per chunk of LOR_CHUNK nonzeroes of the rest of a
//    long row (the plan's chunk list), skipped when the row is already true.
// Without early exits (x mostly false, as a BFS frontier) every product is
// gathered once, load-balanced by the chunks.
constexpr int LOR_W = 4;
constexpr int LOR_HEAD = 32;
constexpr int LOR_CHUNK = 256;
// general path (k_spmv_vector_general): rows longer than GEN_LONG run in
// chunks of GEN_CHUNK, a lane's loads in batches of GEN_BATCH
constexpr int GEN_LONG = 64;
constexpr int64_t GEN_FEW = int64_t(1) << 15;   // see launch_general
constexpr int GEN_CHUNK = 256;
constexpr int GEN_BATCH = 4;
constexpr int64_t GEN_NARROW = int64_t(1) << 20;   // see launch_general
constexpr int GEN_BATCH_BITS = 8;   // where the flags are bits in shared memory

template <bool VALUED>
__global__ void __launch_bounds__(256)
k_lor_head(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const uint8_t *__restrict__ values, const uint8_t *__restrict__ x, uint8_t *__restrict__ y,
	int64_t m) {
	constexpr int RPW = 32 / LOR_W;
	const int lane = threadIdx.x & (LOR_W - 1);
	const int sub = (threadIdx.x & 31) / LOR_W;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	for (int64_t base = warp * RPW; base < m; base += nwarps * RPW) {
		const int64_t i = base + sub;
		int64_t b = 0, e = 0;
		if (i < m && y[i] == 0) {
			b = offsets[i];
			e = offsets[i + 1];
			if (e > b + LOR_HEAD) e = b + LOR_HEAD;
		}
		bool act = b < e, found = false;
		for (int64_t k0 = b; __any_sync(WM_FULL, act); k0 += LOR_W) {
			bool t = false;
			const int64_t k = k0 + lane;
			if (act && k < e) {
				t = x[__ldcs(indices + k)] != 0;
				if (VALUED) t = t && __ldcs(values + k) != 0;
			}
			const unsigned g = (__ballot_sync(WM_FULL, t) >> (sub * LOR_W)) & ((1u << LOR_W) - 1);
			if (act && g) found = true;
			if (k0 + LOR_W >= e || g) act = false;
		}
		if (found && lane == 0) y[i] = 1;
	}
}

template <bool VALUED>
__global__ void __launch_bounds__(256)
k_lor_tail(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const uint8_t *__restrict__ values, const uint8_t *__restrict__ x, uint8_t *y,
	const int64_t *__restrict__ rows, const int64_t *__restrict__ k0s, int64_t nchunks) {
	const int lane = threadIdx.x & 31;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	for (int64_t c = warp; c < nchunks; c += nwarps) {
		const int64_t i = rows[c];
		// an earlier chunk (or the head) may have set the row: read through L2
		if (__ldcg(y + i) != 0) continue;
		const int64_t k0 = k0s[c];
		int64_t e = offsets[i + 1];
		if (e > k0 + LOR_CHUNK) e = k0 + LOR_CHUNK;
		for (int64_t kb = k0; kb < e; kb += 32) {
			const int64_t k = kb + lane;
			bool t = false;
			if (k < e) {
				t = x[__ldcs(indices + k)] != 0;
				if (VALUED) t = t && __ldcs(values + k) != 0;
			}
			if (__any_sync(WM_FULL, t)) {
				if (lane == 0) y[i] = 1;
				break;
			}
		}
	}
}

// One chunk list of the plan: per row of more than `longer` nonzeroes, its
// nonzeroes from `head` on in chunks of `chunk`, consecutive in the list at a
// position taken from *count (any order of the rows: no result depends on
// it); first and number, when given, list each row's first chunk and its chunks
// at a position from *nrows, listed marks the row.  rows == nullptr: count only.
constexpr int64_t LIST_LAST = int64_t(1) << 62;
struct ChunkList {
	int64_t longer, head, chunk;
	unsigned long long *count, *nrows;
	int64_t *rows, *k0s;
	// the general path's list only: chunks are named by their number in the row
	// (k0s; LIST_LAST marks the last) instead of a place in the storage
	int64_t *first, *number;
	uint32_t *listed;
};
__device__ __forceinline__ void add_row_chunks(const ChunkList &l, int64_t i, int64_t o, int64_t e) {
	if (e - o <= l.longer) return;
	const int64_t b = o + l.head, n = (e - b + l.chunk - 1) / l.chunk;
	const unsigned long long at = atomicAdd(l.count, (unsigned long long) n);
	const unsigned long long r = atomicAdd(l.nrows, 1ull);
	if (!l.rows) return;
	for (int64_t c = 0; c < n; ++c) {
		l.rows[at + c] = i;
		l.k0s[at + c] = l.first ? c | (c + 1 == n ? LIST_LAST : 0) : b + c * l.chunk;
	}
	if (l.first) {
		l.first[r] = int64_t(at);
		l.number[r] = n;
		atomicOr(l.listed + (i >> 5), 1u << (i & 31));
	}
}
__global__ void k_row_chunks(const int64_t *__restrict__ offsets, int64_t m, ChunkList p,
	ChunkList q) {
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m;
		 i += int64_t(gridDim.x) * blockDim.x) {
		const int64_t o = offsets[i], e = offsets[i + 1];
		add_row_chunks(p, i, o, e);
		add_row_chunks(q, i, o, e);
	}
}

static void lists_release(alpb_spmv_plan_s *p) {
	cudaFree(p->lor_row);
	cudaFree(p->lor_k0);
	cudaFree(p->gen_row);   // the general path's five lists
	p->lor_row = p->lor_k0 = p->gen_row = p->gen_c = p->gen_first = p->gen_number = nullptr;
	p->gen_listed = nullptr;
	p->lor_n = -1;
	p->gen_n = p->gen_rows = 0;
}

// the lor path's list (rows beyond their first LOR_HEAD nonzeroes) and the
// general path's (rows of more than GEN_LONG, whole)
static int lists_build(alpb_spmv_plan_s *p, cudaStream_t s) {
	lists_release(p);
	if (p->m == 0) {
		p->lor_n = 0;
		return ALPB_SUCCESS;
	}
	const unsigned grid = grid_for(p->m, 256, 4);
	const size_t listed = size_t(p->m + 31) / 32 * 4;
	unsigned long long *cnt = nullptr, h[4] = {0, 0, 0, 0};  // lor chunks, rows; general chunks, rows
	ALPB_CUDA(cudaMallocAsync(&cnt, sizeof(h), s));
	ALPB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(h), s));
	ChunkList lor{LOR_HEAD, LOR_HEAD, LOR_CHUNK, cnt, cnt + 1};
	ChunkList gen{GEN_LONG, 0, GEN_CHUNK, cnt + 2, cnt + 3};
	k_row_chunks<<<grid, 256, 0, s>>>(p->offsets, p->m, lor, gen);
	ALPB_LAUNCHED();
	ALPB_CUDA(cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	if (h[0] > 0) {
		if (cudaMalloc(&p->lor_row, size_t(h[0]) * 8) != cudaSuccess ||
			cudaMalloc(&p->lor_k0, size_t(h[0]) * 8) != cudaSuccess ||
			(h[2] > 0 && cudaMalloc(&p->gen_row, size_t(h[2] + h[3]) * 16 + listed) != cudaSuccess)) {
			cudaGetLastError();
			cudaFreeAsync(cnt, s);
			cudaStreamSynchronize(s);
			lists_release(p);
			set_error("alpb_spmv_plan_create: out of device memory for the chunk lists");
			return ALPB_OUTOFMEM;
		}
		ALPB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(h), s));
		lor.rows = p->lor_row;
		lor.k0s = p->lor_k0;
		if (h[2] > 0) {   // one allocation
			p->gen_c = p->gen_row + h[2];
			p->gen_first = p->gen_c + h[2];
			p->gen_number = p->gen_first + h[3];
			p->gen_listed = reinterpret_cast<uint32_t *>(p->gen_number + h[3]);
			ALPB_CUDA(cudaMemsetAsync(p->gen_listed, 0, listed, s));
		}
		gen.rows = p->gen_row;
		gen.k0s = p->gen_c;
		gen.first = p->gen_first;
		gen.number = p->gen_number;
		gen.listed = p->gen_listed;
		k_row_chunks<<<grid, 256, 0, s>>>(p->offsets, p->m, lor, gen);
		ALPB_LAUNCHED();
	}
	ALPB_CUDA(cudaFreeAsync(cnt, s));
	p->lor_n = int64_t(h[0]);
	p->gen_n = int64_t(h[2]);
	p->gen_rows = int64_t(h[3]);
	return ALPB_SUCCESS;
}

static int launch_lor(const SpmvArgs &a, const alpb_spmv_plan_s &p, cudaStream_t s) {
	const uint8_t *x = static_cast<const uint8_t *>(a.v);
	const uint8_t *vals = static_cast<const uint8_t *>(a.values);
	uint8_t *y = static_cast<uint8_t *>(a.u);
	const int64_t threads = (a.m_out + 32 / LOR_W - 1) / (32 / LOR_W) * 32;
	if (vals)
		k_lor_head<true><<<grid_for(threads, 256, 8), 256, 0, s>>>(a.offsets, a.indices, vals, x,
			y, a.m_out);
	else
		k_lor_head<false><<<grid_for(threads, 256, 8), 256, 0, s>>>(a.offsets, a.indices, vals, x,
			y, a.m_out);
	ALPB_LAUNCHED();
	if (p.lor_n > 0) {
		if (vals)
			k_lor_tail<true><<<grid_for(p.lor_n * 32, 256, 8), 256, 0, s>>>(a.offsets, a.indices,
				vals, x, y, p.lor_row, p.lor_k0, p.lor_n);
		else
			k_lor_tail<false><<<grid_for(p.lor_n * 32, 256, 8), 256, 0, s>>>(a.offsets, a.indices,
				vals, x, y, p.lor_row, p.lor_k0, p.lor_n);
		ALPB_LAUNCHED();
	}
	return ALPB_SUCCESS;
}

// ------------------------------------------------------ vector schedules --
// Rows are handed out per warp (32/W rows at a time) so that every lane of a
// warp runs the same number of outer iterations and the width-W shuffles
// below always see the full warp.
template <class R, int W>
__global__ void __launch_bounds__(256)
k_spmv_vector_dense(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const typename R::T *__restrict__ values, const typename R::T *__restrict__ x,
	typename R::T *__restrict__ y, int64_t m, int left) {
	using T = typename R::T;
	constexpr int RPW = 32 / W;  // rows per warp step
	const int lane = threadIdx.x & (W - 1);
	const int sub = (threadIdx.x & 31) / W;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	for (int64_t base = warp * RPW; base < m; base += nwarps * RPW) {
		const int64_t i = base + sub;
		T acc = R::zero();
		int64_t b = 0, e = 0;
		if (i < m) {
			b = offsets[i];
			e = offsets[i + 1];
			for (int64_t k = b + lane; k < e; k += W) {
				const T a = values ? __ldcs(values + k) : R::one();
				const T xv = __ldg(x + __ldcs(indices + k));
				acc = R::add(acc, left ? R::mull(xv, a) : R::mulr(a, xv));
			}
		}
#pragma unroll
		for (int o = W / 2; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o, W));
		if (i < m && lane == 0 && e > b) y[i] = R::add(y[i], acc);
	}
}

// warp-aggregated count of newly assigned entries
__device__ __forceinline__ void gen_count(const SpmvArgs &a, int64_t newly) {
	if (!a.u_nnz) return;
	for (int o = 16; o > 0; o >>= 1) newly += __shfl_down_sync(0xffffffffu, newly, o);
	if ((threadIdx.x & 31) == 0 && newly)
		atomicAdd((unsigned long long *) a.u_nnz, (unsigned long long) newly);
}

// General path, all ALP semantics; see the file comment.  Two kernels.
//
// k_spmv_vector_plain: W lanes walk a row, one nonzero of each lane after the
// other, in few registers: many warps hide the chain index -> flag -> value and
// x of each nonzero.  No list, no scratch.  It is the faster one where row
// lengths hardly differ (stencils: neighbouring rows share lines of flags and x,
// and a row is only a few steps; us, this / the other with as many lanes, 27-point
// 130^3 under a mask 181 / 231, from a 50% sparse vector 201 / 280) and it
// serves calls without a plan.
//
// k_spmv_vector_general, for rows of differing lengths: two kinds of work items,
// chunks of long rows, then groups of 32/W rows.  What bounds it is that same
// chain, so a lane issues GEN_BATCH of each load before it uses any, and the row
// lengths: with W lanes on every row, a hub row of 1e5 nonzeroes ran as 1e4
// dependent steps of one lane group while the rest of the chip idled.  Rows of
// more than GEN_LONG nonzeroes are therefore cut in chunks of GEN_CHUNK (the
// plan's list), one warp each, first in the item order; their partials are
// summed in chunk order by k_spmv_general_finish (deterministic).
// Measured, R-MAT: min-plus from a 20% sparse vector, 500,009 vertices,
// 2289 -> 118 us, 78 with the bits and the narrow groups below; lor-land with a
// 5% frontier and 30% visited, 1,000,003 vertices, 474 -> 188, 142 us.
template <class R, int W>
__global__ void __launch_bounds__(256)
k_spmv_vector_plain(SpmvArgs a) {
	using T = typename R::T;
	constexpr int RPW = 32 / W;
	const T *__restrict__ values = reinterpret_cast<const T *>(a.values);
	const T *__restrict__ x = reinterpret_cast<const T *>(a.v);
	T *__restrict__ y = reinterpret_cast<T *>(a.u);
	const bool dense_hint = (a.descr & ALPB_DESC_DENSE) != 0;
	const bool add_identity = (a.descr & ALPB_DESC_ADD_IDENTITY) != 0;
	const bool use_index = (a.descr & ALPB_DESC_USE_INDEX) != 0;
	const bool explicit_zero = (a.descr & ALPB_DESC_EXPLICIT_ZERO) != 0;
	const int lane = threadIdx.x & (W - 1);
	const int sub = (threadIdx.x & 31) / W;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	int64_t newly = 0;
	for (int64_t base = warp * RPW; base < a.m_out; base += nwarps * RPW) {
		const int64_t i = base + sub;
		const bool in_range = i < a.m_out;
		bool row_ok = in_range;
		if (row_ok && a.masked)
			row_ok = a.mask_by_structure
				? (a.u_mask_assigned == nullptr || a.u_mask_assigned[i] != 0)
				: eval_mask(a.u_mask, a.u_mask_assigned, a.u_mask_type, a.descr, i);
		const bool id_row = in_range && add_identity && (a.scatter_sem || row_ok);
		const bool u_has = in_range && (a.u_assigned == nullptr || a.u_assigned[i] != 0);
		// immutable-nonzero shortcut of the gather (blas2.hpp:351-357)
		if (R::immutable && !a.scatter_sem && row_ok && u_has && y[i] != R::zero()) row_ok = false;
		const bool active = row_ok || id_row;
		T acc = R::zero();
		bool set = false;
		if (active) {
			if (id_row && lane == 0 && i < a.n_in) {
				const bool vm_ok = !a.input_masked ||
					eval_mask(a.v_mask, a.v_mask_assigned, a.v_mask_type, a.descr, i);
				if (vm_ok && (dense_hint || a.v_assigned == nullptr || a.v_assigned[i])) {
					acc = a.left ? R::mull(x[i], R::one()) : R::mulr(R::one(), x[i]);
					set = true;
				}
			}
			const int64_t b = row_ok ? a.offsets[i] : 0, e = row_ok ? a.offsets[i + 1] : 0;
			for (int64_t k = b + lane; k < e; k += W) {
				const uint32_t j = a.indices[k];
				if (a.input_masked &&
					!eval_mask(a.v_mask, a.v_mask_assigned, a.v_mask_type, a.descr, j))
					continue;
				if (!dense_hint && a.v_assigned != nullptr && !a.v_assigned[j]) continue;
				const T av = values ? values[k] : R::one();
				const T xv = use_index ? T(j) : x[j];
				acc = R::add(a.left ? R::mull(xv, av) : R::mulr(av, xv), acc);
				set = true;
				if (R::immutable && acc != R::zero()) break;
			}
		}
#pragma unroll
		for (int o = W / 2; o > 0; o >>= 1) {
			acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o, W));
			set = set | (__shfl_down_sync(0xffffffffu, int(set), o, W) != 0);
		}
		const bool ez = explicit_zero && !a.scatter_sem && row_ok;
		if (active && lane == 0 && (ez || set)) {
			if (u_has || dense_hint) {
				y[i] = R::add(y[i], acc);
			} else {
				y[i] = acc;
			}
			if (!u_has && a.u_assigned) {
				a.u_assigned[i] = 1;
				++newly;
			}
		}
	}
	gen_count(a, newly);
}

// Rows of the general path: who takes part, and the row's identity term.  Made
// in two halves: fetch() loads what the row's place says (no load waits for
// another), decide() reads it, one item later in the row loop.
template <class R>
struct GenRow {
	using T = typename R::T;
	int64_t i = -1, b = 0, e = 0;
	uint32_t listed;
	uint8_t mask_has, u_flag;
	T old;
	bool row_ok = false, id_row = false, u_has = false;
	__device__ __forceinline__ void fetch(const SpmvArgs &a, int64_t row,
		const uint32_t *in_list = nullptr) {
		i = row;
		b = e = 0;
		listed = 0;
		mask_has = u_flag = 1;
		old = R::zero();
		if (i < 0) return;
		b = a.offsets[i];
		e = a.offsets[i + 1];
		if (in_list) listed = in_list[i >> 5] >> (i & 31) & 1u;
		if (a.masked && a.u_mask_assigned) mask_has = a.u_mask_assigned[i];
		if (a.u_assigned) u_flag = a.u_assigned[i];
		old = reinterpret_cast<const T *>(a.u)[i];
	}
	// listed rows are somebody else's
	__device__ __forceinline__ void decide(const SpmvArgs &a) {
		row_ok = i >= 0 && listed == 0;
		const bool mine = row_ok;
		if (row_ok && a.masked) {
			bool t = mask_has != 0;
			if (!a.mask_by_structure) {   // as eval_mask
				if (t && !(a.descr & ALPB_DESC_STRUCTURAL) && a.u_mask != nullptr &&
					a.u_mask_type != ALPB_VOID)
					t = mask_value_true(a.u_mask, a.u_mask_type, i);
				if (a.descr & ALPB_DESC_INVERT_MASK) t = !t;
			}
			row_ok = t;
		}
		id_row = mine && (a.descr & ALPB_DESC_ADD_IDENTITY) && (a.scatter_sem || row_ok);
		u_has = mine && u_flag != 0;
		// immutable-nonzero shortcut of the gather (blas2.hpp:351-357)
		if (R::immutable && !a.scatter_sem && row_ok && u_has && old != R::zero()) row_ok = false;
	}
	// the identity's contribution to row i (add_identity), if any
	__device__ __forceinline__ void identity(const SpmvArgs &a, T &acc, bool &set) const {
		if (!id_row || i >= a.n_in) return;
		const T *x = reinterpret_cast<const T *>(a.v);
		const bool vm_ok = !a.input_masked ||
			eval_mask(a.v_mask, a.v_mask_assigned, a.v_mask_type, a.descr, i);
		if (vm_ok && ((a.descr & ALPB_DESC_DENSE) || a.v_assigned == nullptr || a.v_assigned[i])) {
			acc = a.left ? R::mull(x[i], R::one()) : R::mulr(R::one(), x[i]);
			set = true;
		}
	}
	// fold the row's sum into the output; counts a newly assigned entry
	__device__ __forceinline__ void finish(const SpmvArgs &a, T acc, bool set,
		int64_t &newly) const {
		const bool dense_hint = (a.descr & ALPB_DESC_DENSE) != 0;
		const bool ez = (a.descr & ALPB_DESC_EXPLICIT_ZERO) && !a.scatter_sem && row_ok;
		if (!(row_ok || id_row) || !(ez || set)) return;
		reinterpret_cast<T *>(a.u)[i] = u_has || dense_hint ? R::add(old, acc) : acc;
		if (!u_has && a.u_assigned) {
			a.u_assigned[i] = 1;
			++newly;
		}
	}
};

// bits: which inputs take part, one bit each (v_assigned and the input mask
// are then not read); null without BITS.
template <class R, int W, bool BITS = false, int BATCH = BITS ? GEN_BATCH_BITS : GEN_BATCH>
__device__ __forceinline__ void gen_gather(const SpmvArgs &a, int64_t b, int64_t e, int lane,
	typename R::T &acc, bool &set, const uint32_t *bits = nullptr) {
	using T = typename R::T;
	const T *__restrict__ values = reinterpret_cast<const T *>(a.values);
	const T *__restrict__ x = reinterpret_cast<const T *>(a.v);
	const bool use_index = (a.descr & ALPB_DESC_USE_INDEX) != 0;
	const uint8_t *__restrict__ va = (a.descr & ALPB_DESC_DENSE) ? nullptr : a.v_assigned;
	for (int64_t k0 = b + lane; k0 < e; k0 += BATCH * W) {
		uint32_t j[BATCH];
		bool on[BATCH];
		T xv[BATCH], av[BATCH];
#pragma unroll
		for (int q = 0; q < BATCH; ++q) {
			on[q] = k0 + q * W < e;
			j[q] = on[q] ? __ldcs(a.indices + k0 + q * W) : 0u;
		}
		if (BITS) {
#pragma unroll
			for (int q = 0; q < BATCH; ++q)
				if (on[q]) on[q] = (bits[j[q] >> 5] >> (j[q] & 31)) & 1u;
		}
		if (!BITS && a.input_masked) {
#pragma unroll
			for (int q = 0; q < BATCH; ++q)
				if (on[q])
					on[q] = eval_mask(a.v_mask, a.v_mask_assigned, a.v_mask_type, a.descr, j[q]);
		}
		if (!BITS && va) {
#pragma unroll
			for (int q = 0; q < BATCH; ++q)
				if (on[q]) on[q] = va[j[q]] != 0;
		}
#pragma unroll
		for (int q = 0; q < BATCH; ++q) {
			xv[q] = R::zero();
			av[q] = R::one();
			if (on[q]) {
				xv[q] = use_index ? T(j[q]) : x[j[q]];
				if (values) av[q] = values[k0 + q * W];
			}
		}
#pragma unroll
		for (int q = 0; q < BATCH; ++q)
			if (on[q]) {
				acc = R::add(a.left ? R::mull(xv[q], av[q]) : R::mulr(av[q], xv[q]), acc);
				set = true;
			}
		if (R::immutable && acc != R::zero()) break;
	}
}

// The listed long rows: their chunks, and where the chunks' partials go.
// nchunks = 0: the first nlong blocks take a listed row each, without partials
// in memory.  A row's last chunk runs to the row's end and which rows are
// listed is read from the list, so offsets that changed under the plan cost
// time, not right sums.
struct GenChunks {
	int64_t nchunks = 0, nlong = 0;
	const int64_t *row = nullptr, *c = nullptr;             // [chunks] row, number in the row
	const int64_t *first = nullptr, *number = nullptr;      // [nlong] first chunk, chunks
	const uint32_t *listed = nullptr;                       // a bit per row
	uint64_t *val = nullptr;                                // [nchunks] partial sums
	uint8_t *has = nullptr;                                 // [nchunks]
};

// Chunk c of n of a listed row, by one warp: the partial in lane 0, set in all.
template <class R, bool BITS>
__device__ __forceinline__ void gen_chunk(const SpmvArgs &a, const GenRow<R> &row, int64_t c,
	bool last, int wl, typename R::T &acc, bool &set, const uint32_t *bits = nullptr) {
	int64_t k0 = row.b + c * GEN_CHUNK;
	const int64_t end = last || row.e < k0 + GEN_CHUNK ? row.e : k0 + GEN_CHUNK;
	bool go = row.row_ok;
	if (R::immutable && a.probe && go) {   // one nonzero a lane, then the rest
		gen_gather<R, 32, BITS, 1>(a, k0, k0 + 32 < end ? k0 + 32 : end, wl, acc, set, bits);
		go = !__any_sync(0xffffffffu, acc != R::zero());
		k0 += 32;
	}
	if (go) gen_gather<R, 32, BITS>(a, k0, end, wl, acc, set, bits);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o));
	set = __any_sync(0xffffffffu, set);
}

// One listed row by a block of 8 warps, the adds in the order of chunks and
// finish pass: lane c % 32 of the first warp takes the partial of chunk c.
template <class R>
__device__ __forceinline__ void gen_long_row(const SpmvArgs &a, const GenChunks &g, int64_t l,
	int64_t &newly) {
	using T = typename R::T;
	__shared__ T part[8];
	__shared__ uint8_t has[8];
	const int wl = threadIdx.x & 31, w = threadIdx.x >> 5;
	GenRow<R> row;
	row.fetch(a, g.row[g.first[l]]);
	const int64_t n = g.number[l];
	row.decide(a);
	T acc = R::zero();
	bool set = false;
	if (threadIdx.x == 0) row.identity(a, acc, set);
	for (int64_t c0 = 0; c0 < n; c0 += 8) {
		T p = R::zero();
		bool ps = false;
		if (c0 + w < n) gen_chunk<R, false>(a, row, c0 + w, c0 + w == n - 1, wl, p, ps);
		if (wl == 0) {
			part[w] = p;
			has[w] = ps ? 1 : 0;
		}
		__syncthreads();
		const int q = wl - int(c0 & 31);
		if (w == 0 && q >= 0 && q < 8 && has[q]) {
			acc = R::add(acc, part[q]);
			set = true;
		}
		if (__syncthreads_or(R::immutable && acc != R::zero())) break;
	}
	if (w != 0) return;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o));
	set = __any_sync(0xffffffffu, set);
	if (wl == 0) row.finish(a, acc, set, newly);
}

// Which inputs take part (assigned, and let through by the input mask), a bit
// each.
__global__ void k_pack_present(SpmvArgs a, uint32_t *bits) {
	const int64_t n32 = (a.n_in + 31) / 32 * 32;
	const uint8_t *va = (a.descr & ALPB_DESC_DENSE) ? nullptr : a.v_assigned;
	for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < n32;
		 j += int64_t(gridDim.x) * blockDim.x) {
		const bool on = j < a.n_in && (va == nullptr || va[j] != 0) &&
			(!a.input_masked || eval_mask(a.v_mask, a.v_mask_assigned, a.v_mask_type, a.descr, j));
		const unsigned w = __ballot_sync(0xffffffffu, on);
		if ((threadIdx.x & 31) == 0) bits[j >> 5] = w;
	}
}

// How the general kernel runs.  GEN_CHUNKS: flags asked in memory, long rows in
// chunks (or none listed).  GEN_BLOCKS: the same, but the first blocks take a listed
// row each.  GEN_BITS: as GEN_CHUNKS, and every block copies the inputs' bits into its
// shared memory first.  A nonzero then asks shared memory whether its input takes
// part (a warp's 32 random words are about four wavefronts there, and up to 32 in
// L1), and only those that do gather x.
enum { GEN_CHUNKS, GEN_BLOCKS, GEN_BITS };
template <class R, int W, int MODE>
__global__ void __launch_bounds__(MODE == GEN_BITS ? 1024 : 256)
k_spmv_vector_general(SpmvArgs a, GenChunks g, const uint32_t *__restrict__ gbits) {
	using T = typename R::T;
	constexpr bool BITS = MODE == GEN_BITS;
	extern __shared__ __align__(16) uint32_t gen_bits[];
	if (BITS) {
		const int64_t words = (a.n_in + 31) / 32;
		for (int64_t k = threadIdx.x; k < (words + 3) / 4; k += blockDim.x)
			reinterpret_cast<uint4 *>(gen_bits)[k] = reinterpret_cast<const uint4 *>(gbits)[k];
		__syncthreads();
	}
	constexpr int RPW = 32 / W;
	const int wl = threadIdx.x & 31;
	const int lane = threadIdx.x & (W - 1);
	const int sub = wl / W;
	int64_t newly = 0;
	int64_t block = blockIdx.x, nblocks = gridDim.x;
	if constexpr (MODE == GEN_BLOCKS) {
		if (block < g.nlong) {
			gen_long_row<R>(a, g, block, newly);
			gen_count(a, newly);
			return;
		}
		block -= g.nlong;
		nblocks -= g.nlong;
	}
	const int64_t warp = (block * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (nblocks * int64_t(blockDim.x)) >> 5;
	const int64_t items = g.nchunks + (a.m_out + RPW - 1) / RPW;
	int64_t it = warp;
	for (; MODE != GEN_BLOCKS && it < g.nchunks; it += nwarps) {   // one chunk of a long row, the whole warp
		GenRow<R> row;
		row.fetch(a, g.row[it]);
		const int64_t c = g.c[it];
		row.decide(a);
		T acc = R::zero();
		bool set = false;
		gen_chunk<R, BITS>(a, row, c & ~LIST_LAST, (c & LIST_LAST) != 0, wl, acc, set, gen_bits);
		if (wl == 0) {
			store_bits<T>(g.val + it, acc);
			g.has[it] = set ? 1 : 0;
		}
	}
	// groups of rows; what the next group's rows say is fetched before this
	// one's gathers, which then are all an item waits for
	const auto row_of = [&](int64_t t) {
		const int64_t i = (t - g.nchunks) * RPW + sub;
		return t < items && i < a.m_out ? i : int64_t(-1);
	};
	GenRow<R> row, nxt;
	row.fetch(a, row_of(it), g.listed);
	for (; it < items; it += nwarps) {
		nxt.fetch(a, row_of(it + nwarps), g.listed);
		row.decide(a);
		T acc = R::zero();
		bool set = false;
		if (lane == 0) row.identity(a, acc, set);
		if (row.row_ok) {
			int64_t k0 = row.b;
			if (R::immutable && a.probe) {   // one nonzero a lane, then the rest
				gen_gather<R, W, BITS, 1>(a, k0, k0 + W < row.e ? k0 + W : row.e, lane, acc, set,
					gen_bits);
				k0 += W;
			}
			if (!R::immutable || acc == R::zero())
				gen_gather<R, W, BITS>(a, k0, row.e, lane, acc, set, gen_bits);
		}
#pragma unroll
		for (int o = W / 2; o > 0; o >>= 1) {
			acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o, W));
			set = set | (__shfl_down_sync(0xffffffffu, int(set), o, W) != 0);
		}
		if (lane == 0) row.finish(a, acc, set, newly);
		row = nxt;
	}
	gen_count(a, newly);
}

// One warp per long row: its chunks' partials in a fixed order (lane-strided,
// then a shuffle tree), the identity term, the output.
template <class R>
__global__ void __launch_bounds__(256)
k_spmv_general_finish(SpmvArgs a, GenChunks g) {
	using T = typename R::T;
	const int lane = threadIdx.x & 31;
	const int64_t warp = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
	const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
	int64_t newly = 0;
	for (int64_t l = warp; l < g.nlong; l += nwarps) {
		const int64_t c0 = g.first[l];
		GenRow<R> row;
		row.fetch(a, g.row[c0]);
		const int64_t n = g.number[l];
		row.decide(a);
		T acc = R::zero();
		bool set = false;
		if (lane == 0) row.identity(a, acc, set);
		if (row.row_ok)
			for (int64_t c = c0 + lane; c < c0 + n; c += 32)
				if (g.has[c]) {
					acc = R::add(acc, wm_load_slot<T>(g.val + c));
					set = true;
				}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o));
		set = __any_sync(0xffffffffu, set);
		if (lane == 0) row.finish(a, acc, set, newly);
	}
	gen_count(a, newly);
}

// Dense product of a small skewed matrix in one launch: a block per long row
// (more than GEN_LONG nonzeroes), then a lane group per row.  Such a product
// is launch and latency: the merge path's tile walk is a longer chain than
// these two loads, and its crossing rows take a second launch.  Nothing is
// shared between blocks, so a plan may serve several streams at once.
template <class R, int W>
__global__ void __launch_bounds__(256) k_spmv_small(SpmvArgs a, const int64_t *__restrict__ crow,
	const int64_t *__restrict__ first, int64_t nlong) {
	using T = typename R::T;
	__shared__ T part[8];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	T *y = reinterpret_cast<T *>(a.u);
	T acc = R::zero();
	bool set = false;
	if (int64_t(blockIdx.x) < nlong) {
		const int64_t i = crow[first[blockIdx.x]];
		gen_gather<R, 256>(a, a.offsets[i], a.offsets[i + 1], threadIdx.x, acc, set);
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o));
		if (lane == 0) part[w] = acc;
		__syncthreads();
		if (threadIdx.x == 0) {
			for (int k = 1; k < 8; ++k) acc = R::add(acc, part[k]);
			y[i] = R::add(y[i], acc);
		}
		return;
	}
	const int64_t i = ((int64_t(blockIdx.x) - nlong) * 256 + threadIdx.x) / W;
	const int64_t b = i < a.m_out ? a.offsets[i] : 0, e = i < a.m_out ? a.offsets[i + 1] : 0;
	const bool mine = e > b && e - b <= GEN_LONG;
	const T old = mine ? y[i] : R::zero();
	if (mine) gen_gather<R, W>(a, b, e, threadIdx.x & (W - 1), acc, set);
#pragma unroll
	for (int o = W / 2; o > 0; o >>= 1) acc = R::add(acc, __shfl_down_sync(0xffffffffu, acc, o, W));
	if (mine && (threadIdx.x & (W - 1)) == 0) y[i] = R::add(old, acc);
}

// Trivial case of blas2.hpp:1001-1037: the output keeps its values; with
// explicit_zero every unassigned entry becomes the additive identity.
template <class R>
__global__ void k_spmv_trivial(SpmvArgs a) {
	using T = typename R::T;
	T *y = reinterpret_cast<T *>(a.u);
	int64_t newly = 0;
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < a.m_out;
		 i += int64_t(gridDim.x) * blockDim.x) {
		if (a.u_assigned && !a.u_assigned[i]) {
			y[i] = R::zero();
			a.u_assigned[i] = 1;
			++newly;
		}
	}
	if (a.u_nnz) {
		for (int o = 16; o > 0; o >>= 1) newly += __shfl_down_sync(0xffffffffu, newly, o);
		if ((threadIdx.x & 31) == 0 && newly) atomicAdd((unsigned long long *) a.u_nnz,
			(unsigned long long) newly);
	}
}

// --------------------------------------------------------------- drivers --
template <class R>
int launch_merge(const SpmvArgs &a, const alpb_spmv_plan_s &p, cudaStream_t s) {
	using T = typename R::T;
	if (p.ntiles == 0) return ALPB_SUCCESS;
	if (p.tile == WM_TILE && p.hot_on && p.hot_k > 0 && a.indices == p.hot_src) {
		// shared-memory slots (one block per SM)
		const size_t smem = HotSmem<R>::bytes(p.hot_k);
		static size_t smem_set = 0;
		if (smem > smem_set) {
			ALPB_CUDA(cudaFuncSetAttribute(k_spmv_wmerge_hot<R>,
				cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
			smem_set = smem;
		}
		T *hx = reinterpret_cast<T *>(p.hot_x);
		k_hot_gather<T><<<grid_for(p.hot_k, 256), 256, 0, s>>>(p.hot_cols,
			reinterpret_cast<const T *>(a.v), hx, p.hot_k);
		ALPB_LAUNCHED();
		int64_t grid = (p.ntiles + HOT_WARPS - 1) / HOT_WARPS;
		if (grid > sm_count()) grid = sm_count();
		const MergeTables mt = merge_tables(p);
		k_spmv_wmerge_hot<R><<<unsigned(grid), 32 * HOT_WARPS, smem, s>>>(mt, a.offsets,
			p.hot_idx, reinterpret_cast<const T *>(a.values), reinterpret_cast<const T *>(a.v), hx,
			p.hot_k, reinterpret_cast<T *>(a.u), a.left);
		ALPB_LAUNCHED();
		k_wm_fixup<R><<<grid_for((p.ntiles + 31) / 32 * 32, 256), 256, 0, s>>>(mt,
			AccumulateY<R>{reinterpret_cast<T *>(a.u)});
	} else if (p.tile == WM_TILE) {
		const T *values = reinterpret_cast<const T *>(a.values), *x = reinterpret_cast<const T *>(a.v);
		T *u = reinterpret_cast<T *>(a.u);
		const MergeTables mt = merge_tables(p);
		static int blocks_per_sm = 0;
		if (!blocks_per_sm) {
			ALPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm,
				k_spmv_wmerge<R, PlainX<T>>, 32 * WM_WARPS, 0));
			if (blocks_per_sm < 1) blocks_per_sm = 1;
		}
		int64_t grid = (p.ntiles + WM_WARPS - 1) / WM_WARPS;
		const int64_t cap = int64_t(sm_count()) * blocks_per_sm;
		if (grid > cap) grid = cap;
		k_spmv_wmerge<R, PlainX<T>><<<unsigned(grid), 32 * WM_WARPS, 0, s>>>(mt, a.offsets,
			a.indices, values, PlainX<T>{x}, u, a.left);
		ALPB_LAUNCHED();
		// rows crossing tiles: one lane per 32 tiles' worth of first tiles
		k_wm_fixup<R><<<grid_for((p.ntiles + 31) / 32 * 32, 256), 256, 0, s>>>(mt,
			AccumulateY<R>{reinterpret_cast<T *>(a.u)});
	} else {
		k_spmv_merge<R><<<unsigned(p.ntiles), MP_BLOCK, 0, s>>>(merge_tables(p), a.offsets,
			a.indices, reinterpret_cast<const T *>(a.values), reinterpret_cast<const T *>(a.v),
			reinterpret_cast<T *>(a.u), a.left);
	}
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

template <class R, int W>
int launch_vector_dense_w(const SpmvArgs &a, cudaStream_t s) {
	using T = typename R::T;
	const int64_t threads = a.m_out * W;
	k_spmv_vector_dense<R, W><<<grid_for(threads, 256, 8), 256, 0, s>>>(a.offsets, a.indices,
		reinterpret_cast<const T *>(a.values), reinterpret_cast<const T *>(a.v),
		reinterpret_cast<T *>(a.u), a.m_out, a.left);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// The general path asks the inputs' bits in shared memory from GEN_BITS_NNZ
// nonzeroes on, for vectors whose bits fit beside an L1 of some size.  R-MAT,
// us, flags in memory / bits: 500,009 vertices, min-plus, 20% sparse, 118 / 88;
// 100,000 vertices, lor, 36 / 40, min-plus 25 / 27 (packing costs a launch).
constexpr int64_t GEN_BITS_NNZ = int64_t(1) << 21;
constexpr int64_t GEN_BITS_MAX = 200 * 1024 * 8;

// Below this many nonzeroes, in rows of up to GEN_BLOCK_LEN, the listed rows run a
// block each in the one launch: the partials' memory and the finish pass cost a
// small product more than the chip they fill (us, blocks / chunks: R-MAT, min-plus
// from a 20% sparse vector, 20,000 vertices, 0.23 M nonzeroes, 16 / 23, 100,000, 1.4 M,
// 34 / 28; FP64, 4 to 64 rows of 1,000 12 / 16, of 8,000 19 / 16, of 100,000 172 / 18).
constexpr int64_t GEN_SCRATCH_NNZ = int64_t(1) << 20;
constexpr int64_t GEN_BLOCK_LEN = 6144;
static_assert(GEN_SCRATCH_NNZ <= GEN_BITS_NNZ, "the kernel with the bits takes chunks");

// A call under stream capture takes no scratch: its graph would hold allocation
// nodes, and could not be a child graph or run twice at once.
static bool capturing(cudaStream_t s) {
	cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
	cudaGetLastError();   // the legacy stream during another stream's capture
	return true;
}

// Some inputs may not take part.
static bool gen_filtered(const SpmvArgs &a) {
	return a.input_masked || (a.v_assigned && !(a.descr & ALPB_DESC_DENSE));
}

// lists: p's lists are used.
template <class R, int W>
int launch_general_w(const SpmvArgs &a, const alpb_spmv_plan_s *p, bool lists, cudaStream_t s) {
	constexpr int RPW = 32 / W;
	GenChunks g;
	if (lists) {
		g.nlong = p->gen_rows;
		g.row = p->gen_row;
		g.c = p->gen_c;
		g.first = p->gen_first;
		g.number = p->gen_number;
		g.listed = p->gen_listed;
	}
	void *scratch = nullptr;
	uint32_t *bits = nullptr;
	const bool want_bits = gen_filtered(a) && a.nnz >= GEN_BITS_NNZ && a.n_in <= GEN_BITS_MAX;
	const size_t bit_bytes = want_bits ? size_t(a.n_in + 127) / 128 * 16 : 0;
	const int64_t chunks = lists && (a.nnz >= GEN_SCRATCH_NNZ || p->maxlen > GEN_BLOCK_LEN)
		? p->gen_n : 0;
	if ((bit_bytes || chunks) && !capturing(s)) {
		// bits, then the partials of the long rows' chunks: this call's own
		// (calls on other streams may use the same plan); without them the
		// listed rows run a block each and the flags are asked in memory
		if (cudaMallocAsync(&scratch, bit_bytes + size_t(chunks) * 9, s) == cudaSuccess) {
			unsigned char *at = static_cast<unsigned char *>(scratch);
			if (bit_bytes) bits = reinterpret_cast<uint32_t *>(at);
			if (chunks) {
				g.nchunks = chunks;
				g.val = reinterpret_cast<uint64_t *>(at + bit_bytes);
				g.has = reinterpret_cast<uint8_t *>(g.val + chunks);
			}
		} else {
			cudaGetLastError();
			scratch = nullptr;
		}
	}
	const int64_t items = g.nchunks + (a.m_out + RPW - 1) / RPW;
	if (bits) {
		static std::atomic<unsigned long long> allowed_in;
		ALPB_CUDA(allow_smem(k_spmv_vector_general<R, W, GEN_BITS>, GEN_BITS_MAX / 8, allowed_in));
		k_pack_present<<<grid_for(a.n_in, 256), 256, 0, s>>>(a, bits);
		ALPB_LAUNCHED();
		k_spmv_vector_general<R, W, GEN_BITS><<<grid_for(items * 32, 1024, 1), 1024, bit_bytes,
			s>>>(a, g, bits);
	} else if (g.nlong > 0 && g.nchunks == 0) {
		k_spmv_vector_general<R, W, GEN_BLOCKS><<<unsigned(g.nlong + grid_for(items * 32, 256, 8)),
			256, 0, s>>>(a, g, nullptr);
	} else {
		k_spmv_vector_general<R, W, GEN_CHUNKS><<<grid_for(items * 32, 256, 8), 256, 0, s>>>(a, g,
			nullptr);
	}
	ALPB_LAUNCHED();
	if (g.nchunks > 0) {
		k_spmv_general_finish<R><<<grid_for(g.nlong * 32, 256, 8), 256, 0, s>>>(a, g);
		ALPB_LAUNCHED();
	}
	if (scratch) ALPB_CUDA(cudaFreeAsync(scratch, s));
	return ALPB_SUCCESS;
}

template <class R, int W>
int launch_plain_w(const SpmvArgs &a, cudaStream_t s) {
	k_spmv_vector_plain<R, W><<<grid_for(a.m_out * W, 256, 8), 256, 0, s>>>(a);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// Matrices of up to SMALL_NNZ nonzeroes in rows of up to SMALL_ROW take
// k_spmv_small where the merge path is the plan's own choice.  Measured us per
// call (waited for), merge path / this, R-MAT: 4,096 vertices 30.5 / 23.7,
// 10,000 28.4 / 22.8, 20,000 29.9 / 24.0, 30,000 29.4 / 26.3; 60,000 (0.86 M
// nonzeroes) 31 either way.
constexpr int64_t SMALL_NNZ = int64_t(1) << 19;
constexpr int64_t SMALL_ROW = 8192;

template <class R>
int launch_small(const SpmvArgs &a, const alpb_spmv_plan_s &p, cudaStream_t s) {
	const auto go = [&](auto width) {
		constexpr int W = decltype(width)::value;
		const int64_t grid = p.gen_rows + (a.m_out * W + 255) / 256;
		k_spmv_small<R, W><<<unsigned(grid), 256, 0, s>>>(a, p.gen_row, p.gen_first, p.gen_rows);
		ALPB_LAUNCHED();
		return ALPB_SUCCESS;
	};
	return p.mean < 6 ? go(std::integral_constant<int, 4>{}) : go(std::integral_constant<int, 8>{});
}

// f(integral_constant of W)
template <class F>
static int with_width(int W, const F &f) {
	switch (W) {
	case 1: return f(std::integral_constant<int, 1>{});
	case 2: return f(std::integral_constant<int, 2>{});
	case 4: return f(std::integral_constant<int, 4>{});
	case 8: return f(std::integral_constant<int, 8>{});
	case 16: return f(std::integral_constant<int, 16>{});
	default: return f(std::integral_constant<int, 32>{});
	}
}

// The general path.  Which kernel: k_spmv_vector_plain without a plan and, where no
// row is in the lists' way, for rows of nearly one length, small matrices, given
// widths and rows of more than 128.  Measured us, plain / the other, min-plus from a
// 20% sparse vector unless said:
//   lists: R-MAT 100,000 vertices 373 / 28, lognormal rows 300,000 118 / 50 (under a
//   mask, FP64, 2,000,000: 265 / 288); few rows or long ones, FP64 from all inputs:
//   16 rows of 1,000 23 / 12, 1,000 rows of 8,000 278 / 54, 4,000 311 / 167, 16,000 rows
//   of 1,000 119 / 101, 8,000 of up to 1,000 39 / 41, of up to 600 25 / 32; rows that are
//   merely longer than GEN_LONG lose by them (100,000 rows of 200: 82 / 93, 300,000 of
//   0 to 100: 122 / 124, 74 without the lists);
//   random rows without lists, from GEN_NARROW nonzeroes on: mean 16 and 1,000,000 rows
//   110 / 70, mean 30 and 300,000 rows 74 / 45, FP64 up to 300 and 8,000 rows 17 / 19, up
//   to 600 25 / 42; where the inputs' flags do not fit as bits, mean 16 and 3,000,000
//   rows (2 lanes) 314 / 382 (478 / 344 in FP64), mean 30 and 2,000,000 rows 462 / 528:
//   from 8 lanes on the plain one;
//   one length: 27-point 117^3 116 / 274, 5-point 1200^2 37 / 57, rows of 200 as above.
// A lane waits for its row's chain of loads, so from GEN_NARROW nonzeroes on a
// quarter of the lanes per row, and four times the rows in flight, is faster
// (R-MAT with lists, us with 8 / 2 lanes: 1,000,003 vertices, lor, 185 / 144,
// 500,009, min-plus, 90 / 70; 20,000: 15.8 / 17.8); without lists a hub row would
// run on those few.  A width that the caller gave is kept.
static bool gen_no_bits(const SpmvArgs &a) { return gen_filtered(a) && a.n_in > GEN_BITS_MAX; }
template <class R>
int launch_general(const SpmvArgs &a, const alpb_spmv_plan_s *p, int W, cudaStream_t s) {
	const bool lists = p && p->hubs && p->gen_n > 0;
	if (!p || (!lists && (p->steady || p->given_width || a.nnz < GEN_NARROW || p->maxlen > 128 ||
			(W >= 8 && gen_no_bits(a)))))
		return with_width(W, [&](auto w) { return launch_plain_w<R, decltype(w)::value>(a, s); });
	if (!p->given_width && a.nnz >= GEN_NARROW && W >= 4) W /= 4;
	return with_width(W, [&](auto w) {
		return launch_general_w<R, decltype(w)::value>(a, p, lists, s);
	});
}

// Row-streaming kernel of one chunk shape; the block takes as many warps as
// its shared memory holds stages for.
template <class R, int L, int RPL, int U>
static int launch_rows_as(const SpmvArgs &a, int maxlen, cudaStream_t s) {
	using T = typename R::T;
	constexpr int ROWS = 32 / L * RPL;
	const int cap = rs_cap<R>(ROWS, maxlen);
	const size_t warp = size_t(RS_STAGES) * size_t(cap) * (sizeof(T) + 4);
	constexpr size_t room = 220 * 1024;
	int warps = int(room / warp);
	if (warps > RS_MAX_WARPS) warps = RS_MAX_WARPS;
	static std::atomic<unsigned long long> allowed_in;
	ALPB_CUDA(allow_smem(k_spmv_rows<R, L, RPL, U>, room, allowed_in));
	const int64_t chunks = (a.m_out + ROWS - 1) / ROWS;
	const int64_t grid = chunks < sm_count() ? chunks : sm_count();
	const int64_t per = (chunks + grid - 1) / grid;   // chunks of one block
	if (per < warps) warps = int(per);
	k_spmv_rows<R, L, RPL, U><<<unsigned(grid), 32 * warps, warp * warps, s>>>(a.offsets,
		a.indices, reinterpret_cast<const T *>(a.values), reinterpret_cast<const T *>(a.v),
		reinterpret_cast<T *>(a.u), a.m_out, a.nnz, cap, a.left);
	ALPB_LAUNCHED();
	return ALPB_SUCCESS;
}

// Rows of up to 8 nonzeroes: one lane a row, two rows a lane (a chunk of 64
// rows); longer ones: two lanes a row.
template <class R>
static int launch_rows(const SpmvArgs &a, int maxlen, cudaStream_t s) {
	if (maxlen <= 8) return launch_rows_as<R, 1, 2, 5>(a, maxlen, s);
	return launch_rows_as<R, 2, 1, 7>(a, maxlen, s);
}

// Whether k_spmv_rows is the faster one, k_spmv_vector_dense's regular width being
// the other.  Consecutive rows start a row's length apart in shared memory: even
// lengths from 8 on meet in the same banks, and with differing lengths the lanes
// wait for the longest row of the warp and the stages hold less.  The kernel's few
// warps also gather with fewer loads in flight, which shows where the matrix is in
// L2 or little beyond it.  Measured us, this / the other, FP64 unless said (L: row
// length; matrices of diagonals and the stencils, Z: nonzeroes):
//   L 5   8 M 32 / 25 (5-point 1200^2 31 / 25), 16 M 58 / 51, 24 M 82 / 105, 5-point
//         2000^2 74 / 92, 3000^2 160 / 201; int32 8 M 19 / 23, 16 M 45 / 43, 48 M 117 / 168
//   L 8   16 M 73 / 42, 48 M 195 / 181; random columns 78 / 47 (8 M)
//   L 9   24 M 98 / 65, 48 M 189 / 201; pattern 16 M 52 / 45, 48 M 151 / 181
//   L 13  24 M 86 / 69, 48 M 163 / 413; pattern 16 M 36 / 40
//   L 19  8 M 26 / 33, 48 M 138 / 469; L 27 8 M 25 / 36, 48 M 135 / 186 (27-point
//         130^3 165 / 242, int32 126 / 109, pattern 107 / 142); L 63 161 / 218
//   8 to 24 random columns a row, 16 M 151 / 114; pattern 124 / 96
template <class R>
static bool rows_pay(const SpmvArgs &a, const alpb_spmv_plan_s &p) {
	const int64_t len = int64_t(p.maxlen), vb = a.values ? int64_t(sizeof(typename R::T)) : 0;
	if (!p.steady || (len >= 8 && len % 2 == 0)) return false;
	if (len <= 2) return true;
	const double bytes = double(a.nnz) * double(4 + vb) +
		double(a.m_out) * double(8 + 3 * sizeof(typename R::T));
	if (vb == 0) return len != 9 || bytes > 300e6;
	if (vb <= 4) return len <= 7 && (bytes < 110e6 || bytes > 320e6);
	return len > 16 || bytes > (len <= 7 ? 320e6 : 640e6);
}

static int default_width(double mean) {
	int w = 1;
	while (w < 32 && w * 2 <= mean * 0.75 + 1) w *= 2;
	return w;
}

// Lanes per row for regular rows: about a sixth of the mean row length, so a
// warp spans several rows (measured on B200: 2 lanes for the 5-point
// Poisson rows, 4 for the 27-point stencil, each ~1.2-2.5x faster than one
// lane per 1-2 nonzeroes or the merge path).
static int regular_width(double mean) {
	int w = 2;
	while (w < 32 && w * 2 <= mean / 6) w *= 2;
	return w;
}

template <class R>
int run_spmv(const SpmvArgs &a, const alpb_spmv_plan_s *plan, int force_sched, cudaStream_t s) {
	if (a.trivial) {
		if (a.descr & ALPB_DESC_EXPLICIT_ZERO) {
			k_spmv_trivial<R><<<grid_for(a.m_out, 256), 256, 0, s>>>(a);
			ALPB_LAUNCHED();
		}
		return ALPB_SUCCESS;
	}
	const bool fast = a.dense_all && !a.masked && !a.input_masked &&
		!(a.descr & (ALPB_DESC_ADD_IDENTITY | ALPB_DESC_USE_INDEX));
	// A plan's tables and lists are those of the offsets it was made from: with
	// others of the same sizes only its lane width is taken.
	const alpb_spmv_plan_s *p = plan && plan->offsets == a.offsets ? plan : nullptr;
	if constexpr (std::is_same<R, RingLorLandBool>::value) {
		if (fast && !force_sched && p && p->lor_n >= 0) return launch_lor(a, *p, s);
	}
	int sched = force_sched ? force_sched : (p ? p->sched : ALPB_SCHED_VECTOR);
	int W = plan ? plan->vw : default_width(a.m_out ? double(a.nnz) / double(a.m_out) : 1.0);
	if (fast && sched == ALPB_SCHED_MERGE_PATH && p && p->tile_row) {
		if (p->small && p->lor_n >= 0 && !p->hot_on) return launch_small<R>(a, *p, s);
		return launch_merge<R>(a, *p, s);
	}
	// regular short rows: the row-streaming kernel (16-byte copies of the
	// storage's ranges, so its arrays have to start on such a boundary)
	if (fast && p && p->can_rows && (p->rows < 0 ? rows_pay<R>(a, *p) : p->rows != 0) && !(reinterpret_cast<uintptr_t>(a.indices) & 15) &&
		!(reinterpret_cast<uintptr_t>(a.values) & 15))
		return launch_rows<R>(a, int(p->maxlen), s);
	if (!fast) return launch_general<R>(a, p, W, s);
	return with_width(W, [&](auto w) { return launch_vector_dense_w<R, decltype(w)::value>(a, s); });
}

int dispatch_spmv(int ring, const SpmvArgs &a, const alpb_spmv_plan_s *p, int force_sched,
	cudaStream_t s) {
	switch (ring) {
	case ALPB_RING_PLUS_TIMES_F64: return run_spmv<RingPlusTimesF64>(a, p, force_sched, s);
	case ALPB_RING_LOR_LAND_BOOL: return run_spmv<RingLorLandBool>(a, p, force_sched, s);
	case ALPB_RING_MIN_PLUS_I32: return run_spmv<RingMinPlusI32>(a, p, force_sched, s);
	case ALPB_RING_PLUS_PATTERN_F64: return run_spmv<RingPlusPatternF64>(a, p, force_sched, s);
	case ALPB_RING_PLUS_TIMES_I32: return run_spmv<RingPlusTimesI32>(a, p, force_sched, s);
	case ALPB_RING_PLUS_RIGHT_IF_U64: return run_spmv<RingPlusRightIfU64>(a, p, force_sched, s);
	case ALPB_RING_MAX_LEFT_IF_U64: return run_spmv<RingMaxLeftIfU64>(a, p, force_sched, s);
	case ALPB_RING_TIMES_PLUS_F64: return run_spmv<RingTimesPlusF64>(a, p, force_sched, s);
	}
	set_error("alpb_mxv: semiring %d is not instantiated on the device", ring);
	return ALPB_UNSUPPORTED;
}

int ring_value_type(int ring) {
	switch (ring) {
	case ALPB_RING_PLUS_TIMES_F64: return ALPB_FP64;
	case ALPB_RING_LOR_LAND_BOOL: return ALPB_BOOL;
	case ALPB_RING_MIN_PLUS_I32: return ALPB_INT32;
	case ALPB_RING_PLUS_PATTERN_F64: return ALPB_FP64;
	case ALPB_RING_PLUS_TIMES_I32: return ALPB_INT32;
	case ALPB_RING_PLUS_RIGHT_IF_U64: return ALPB_INT64;
	case ALPB_RING_MAX_LEFT_IF_U64: return ALPB_INT64;
	case ALPB_RING_TIMES_PLUS_F64: return ALPB_FP64;
	}
	return -1;
}

int plan_build(alpb_spmv_plan_s *p, const int64_t *offsets, int64_t tile, cudaStream_t s) {
	// row-length profile
	unsigned long long *d_max = nullptr;
	double *d_sq = nullptr;
	ALPB_CUDA(cudaMallocAsync(&d_max, 8, s));
	ALPB_CUDA(cudaMallocAsync(&d_sq, 8, s));
	ALPB_CUDA(cudaMemsetAsync(d_max, 0, 8, s));
	ALPB_CUDA(cudaMemsetAsync(d_sq, 0, 8, s));
	if (p->m > 0) {
		k_row_stats<<<grid_for(p->m, 256, 4), 256, 0, s>>>(offsets, p->m, d_max, d_sq);
		ALPB_LAUNCHED();
	}
	unsigned long long hmax = 0;
	double hsq = 0;
	ALPB_CUDA(cudaMemcpyAsync(&hmax, d_max, 8, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaMemcpyAsync(&hsq, d_sq, 8, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(d_max, s));
	ALPB_CUDA(cudaFreeAsync(d_sq, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	p->maxlen = double(hmax);
	p->mean = p->m ? double(p->nnz) / double(p->m) : 0.0;
	const double var = p->m ? hsq / double(p->m) - p->mean * p->mean : 0.0;
	p->cv = p->mean > 0 ? sqrt(var > 0 ? var : 0.0) / p->mean : 0.0;
	// merge-path tile table
	p->tile = tile;
	const int64_t rpt = tile == WM_TILE ? aligned_rows_per_tile(p->maxlen, p->mean, tile) : 0;
	p->ntiles = rpt ? (p->m + rpt - 1) / rpt : (p->m + p->nnz + tile - 1) / tile;
	if (p->ntiles > 0) {
		ALPB_CHECK(tile != MP_TILE || p->nnz + MP_TILE < (int64_t(1) << 31), ALPB_OVERFLW,
			"alpb_spmv_plan_create: block merge tiles use 32-bit offsets (nnz %lld)",
			(long long) p->nnz);
		const size_t nt = size_t(p->ntiles);
		ALPB_CUDA(cudaMalloc(&p->tile_row, (nt + 1) * 8));
		ALPB_CUDA(cudaMalloc(&p->head_first, nt * 8));
		ALPB_CUDA(cudaMalloc(&p->tail_first, nt * 8));
		ALPB_CUDA(cudaMalloc(&p->span_len, nt * 4));
		ALPB_CUDA(cudaMalloc(&p->counter, nt * 4));
		ALPB_CUDA(cudaMalloc(&p->head_val, nt * 8));
		ALPB_CUDA(cudaMalloc(&p->tail_val, nt * 8));
		ALPB_CUDA(cudaMalloc(&p->head_has, nt));
		ALPB_CUDA(cudaMalloc(&p->tail_has, nt));
		ALPB_CUDA(cudaMalloc(&p->ready, nt * 4));
		ALPB_CUDA(cudaMemsetAsync(p->counter, 0, nt * 4, s));
		ALPB_CUDA(cudaMemsetAsync(p->ready, 0, nt * 4, s));
		if (rpt) {
			ALPB_CUDA(cudaMalloc(&p->tile_d, (nt + 1) * 8));
			k_row_aligned_tiles<<<grid_for(p->ntiles + 1, 256), 256, 0, s>>>(offsets, p->m, rpt,
				p->ntiles, p->tile_row, p->tile_d, p->head_first, p->tail_first, p->span_len);
			ALPB_LAUNCHED();
		} else {
			k_merge_tiles<<<grid_for(p->ntiles + 1, 256), 256, 0, s>>>(offsets, p->m, p->nnz,
				p->ntiles, p->tile_row, tile);
			ALPB_LAUNCHED();
			k_merge_tables<<<grid_for(p->ntiles, 256), 256, 0, s>>>(offsets, p->m, p->nnz, p->ntiles,
				p->tile_row, p->head_first, p->tail_first, p->span_len, tile);
			ALPB_LAUNCHED();
		}
	}
	return ALPB_SUCCESS;
}

} // namespace alpb

using namespace alpb;

extern "C" {

int alpb_spmv_plan_create(alpb_spmv_plan *plan, int64_t m, int64_t nnz, const int64_t *offsets,
	int sched, int vector_width, void *stream) {
	ALPB_CHECK(plan != nullptr, ALPB_ILLEGAL, "alpb_spmv_plan_create: null plan");
	*plan = nullptr;
	cudaStream_t s = as_stream(stream);
	int rc = plan_create_tiles(plan, m, nnz, offsets, sched, vector_width, WM_TILE, s);
	if (rc != ALPB_SUCCESS) return rc;
	rc = lists_build(*plan, s);
	if (rc != ALPB_SUCCESS) {
		alpb_spmv_plan_destroy(*plan);
		*plan = nullptr;
	}
	return rc;
}

} // extern "C"

int alpb::plan_create_tiles(alpb_spmv_plan_s **plan, int64_t m, int64_t nnz,
	const int64_t *offsets, int sched, int vector_width, int64_t tile, cudaStream_t s) {
	*plan = nullptr;
	ALPB_CHECK(m >= 0 && nnz >= 0, ALPB_ILLEGAL, "alpb_spmv_plan_create: negative size");
	ALPB_CHECK(sched >= ALPB_SCHED_AUTO && sched <= ALPB_SCHED_VECTOR, ALPB_ILLEGAL,
		"alpb_spmv_plan_create: schedule %d", sched);
	auto *p = new alpb_spmv_plan_s();
	p->m = m;
	p->nnz = nnz;
	p->offsets = offsets;
	cudaGetDevice(&p->device);
	int rc = plan_build(p, offsets, tile, s);
	if (rc != ALPB_SUCCESS) {
		alpb_spmv_plan_destroy(p);
		return rc;
	}
	// profile heuristic: regular rows -> vector, skewed rows -> merge path
	const bool regular = p->cv < 0.5 && p->maxlen <= 4.0 * p->mean + 32;
	if (vector_width > 0) {
		int w = 1;
		while (w < vector_width && w < 32) w *= 2;
		p->vw = w;
	} else {
		p->vw = regular ? regular_width(p->mean) : default_width(p->mean);
	}
	p->given_width = vector_width > 0;
	// rows of nearly one length (stencils with their boundaries), and rows that no
	// lane group should walk: far longer than the others, long where a group per row
	// leaves the chip idle, or long by themselves.  launch_general has the figures
	p->steady = p->cv < 0.15;
	p->hubs = p->maxlen > 256 && ((!p->steady && p->maxlen >= 8 * p->mean) ||
		p->m * p->vw < GEN_FEW || p->maxlen >= 768);
	p->own_vw = p->vw;
	p->can_small = sched == ALPB_SCHED_AUTO && !regular && nnz <= SMALL_NNZ && p->maxlen <= SMALL_ROW;
	p->small = p->can_small;
	if (sched == ALPB_SCHED_AUTO) sched = regular ? ALPB_SCHED_VECTOR : ALPB_SCHED_MERGE_PATH;
	p->sched = sched;
	p->can_rows = regular && vector_width <= 0 && p->maxlen >= 1 && p->maxlen <= RS_MAX_LEN;
	*plan = p;
	return ALPB_SUCCESS;
}

extern "C" {

int alpb_spmv_plan_destroy(alpb_spmv_plan p) {
	if (!p) return ALPB_SUCCESS;
	cudaFree(p->tile_row);
	cudaFree(p->head_first);
	cudaFree(p->tail_first);
	cudaFree(p->span_len);
	cudaFree(p->counter);
	cudaFree(p->head_val);
	cudaFree(p->tail_val);
	cudaFree(p->head_has);
	cudaFree(p->tail_has);
	cudaFree(p->ready);
	cudaFree(p->tile_d);
	cudaFree(p->hot_idx);
	cudaFree(p->hot_cols);
	cudaFree(p->hot_x);
	lists_release(p);
	delete p;
	return ALPB_SUCCESS;
}

int alpb_spmv_plan_info(alpb_spmv_plan p, int *sched, int *vw, int64_t *tiles) {
	ALPB_CHECK(p != nullptr, ALPB_ILLEGAL, "alpb_spmv_plan_info: null plan");
	if (sched) *sched = p->sched;
	if (vw) *vw = p->vw;
	if (tiles) *tiles = p->ntiles;
	return ALPB_SUCCESS;
}

} // extern "C"

namespace alpb {

// Hot-column slots that fit the shared memory of one block (227 KB) next to
// the warps' tiles, for the value type of `ring`.
template <class R>
static int64_t hot_slots_for() {
	const size_t cap = 227 * 1024;
	return HotSmem<R>::x_off >= cap ? 0
		: int64_t((cap - HotSmem<R>::x_off) / sizeof(typename R::T)) / 1024 * 1024;
}
static int64_t hot_slots_max(int ring) {
	switch (ring) {
	case ALPB_RING_PLUS_TIMES_F64: return hot_slots_for<RingPlusTimesF64>();
	case ALPB_RING_LOR_LAND_BOOL: return hot_slots_for<RingLorLandBool>();
	case ALPB_RING_MIN_PLUS_I32: return hot_slots_for<RingMinPlusI32>();
	case ALPB_RING_PLUS_PATTERN_F64: return hot_slots_for<RingPlusPatternF64>();
	case ALPB_RING_PLUS_TIMES_I32: return hot_slots_for<RingPlusTimesI32>();
	case ALPB_RING_PLUS_RIGHT_IF_U64: return hot_slots_for<RingPlusRightIfU64>();
	case ALPB_RING_MAX_LEFT_IF_U64: return hot_slots_for<RingMaxLeftIfU64>();
	case ALPB_RING_TIMES_PLUS_F64: return hot_slots_for<RingTimesPlusF64>();
	}
	return 0;
}

static void hot_release(alpb_spmv_plan_s *p) {
	cudaFree(p->hot_idx);
	cudaFree(p->hot_cols);
	cudaFree(p->hot_x);
	p->hot_idx = nullptr;
	p->hot_cols = nullptr;
	p->hot_x = nullptr;
	p->hot_k = 0;
	p->hot_on = 0;
	p->hot_src = nullptr;
	p->hot_cover = 0;
}

// Hot-column cache of K slots for the index array `indices` (n columns): the
// K most frequent columns (ties to the smaller column) get the slots in order
// of decreasing frequency.  Column counts are taken on the device; the
// selection runs on the host (n counts) once per plan.
static int hot_build(alpb_spmv_plan_s *p, const uint32_t *indices, int64_t n, int64_t K,
	cudaStream_t s) {
	hot_release(p);
	if (K <= 0 || n <= K || n >= (int64_t(1) << 31) || p->nnz == 0) return ALPB_SUCCESS;
	uint32_t *cnt = nullptr;
	ALPB_CUDA(cudaMallocAsync(&cnt, size_t(n) * 4, s));
	ALPB_CUDA(cudaMemsetAsync(cnt, 0, size_t(n) * 4, s));
	k_col_counts<<<grid_for(p->nnz, 256, 4), 256, 0, s>>>(indices, p->nnz, cnt);
	ALPB_LAUNCHED();
	std::vector<uint32_t> h(static_cast<size_t>(n));
	ALPB_CUDA(cudaMemcpyAsync(h.data(), cnt, size_t(n) * 4, cudaMemcpyDeviceToHost, s));
	ALPB_CUDA(cudaFreeAsync(cnt, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	std::vector<uint32_t> order(static_cast<size_t>(n));
	for (int64_t j = 0; j < n; ++j) order[size_t(j)] = uint32_t(j);
	const auto more = [&h](uint32_t a, uint32_t b) { return h[a] != h[b] ? h[a] > h[b] : a < b; };
	std::partial_sort(order.begin(), order.begin() + K, order.end(), more);
	std::vector<int32_t> slot(static_cast<size_t>(n), -1);
	uint64_t covered = 0;
	for (int64_t k = 0; k < K; ++k) {
		slot[order[size_t(k)]] = int32_t(k);
		covered += h[order[size_t(k)]];
	}
	int32_t *dslot = nullptr;
	ALPB_CUDA(cudaMallocAsync(&dslot, size_t(n) * 4, s));
	ALPB_CUDA(cudaMemcpyAsync(dslot, slot.data(), size_t(n) * 4, cudaMemcpyHostToDevice, s));
	if (cudaMalloc(&p->hot_idx, size_t(p->nnz) * 4) != cudaSuccess ||
		cudaMalloc(&p->hot_cols, size_t(K) * 4) != cudaSuccess ||
		cudaMalloc(&p->hot_x, size_t(K) * 8) != cudaSuccess) {
		cudaGetLastError();
		cudaFreeAsync(dslot, s);
		cudaStreamSynchronize(s);
		hot_release(p);
		set_error("alpb_spmv_autotune: out of device memory for the hot-column cache");
		return ALPB_OUTOFMEM;
	}
	ALPB_CUDA(cudaMemcpyAsync(p->hot_cols, order.data(), size_t(K) * 4, cudaMemcpyHostToDevice, s));
	k_hot_remap<<<grid_for(p->nnz, 256, 4), 256, 0, s>>>(indices, p->nnz, dslot, p->hot_idx);
	ALPB_LAUNCHED();
	ALPB_CUDA(cudaFreeAsync(dslot, s));
	ALPB_CUDA(cudaStreamSynchronize(s));
	p->hot_k = K;
	p->hot_src = indices;
	p->hot_cover = double(covered) / double(p->nnz);
	return ALPB_SUCCESS;
}

} // namespace alpb

extern "C" {

int alpb_spmv_plan_hot(alpb_spmv_plan p, int ring, int64_t n, const uint32_t *indices,
	int64_t slots, void *stream) {
	ALPB_CHECK(p != nullptr, ALPB_ILLEGAL, "alpb_spmv_plan_hot: null plan");
	ALPB_CHECK(ring_value_type(ring) >= 0, ALPB_UNSUPPORTED,
		"alpb_spmv_plan_hot: semiring %d is not instantiated on the device", ring);
	ALPB_CHECK(slots >= 0 && slots <= hot_slots_max(ring), ALPB_ILLEGAL,
		"alpb_spmv_plan_hot: %lld slots (at most %lld for semiring %d)", (long long) slots,
		(long long) hot_slots_max(ring), ring);
	ALPB_CHECK(slots < n || slots == 0, ALPB_ILLEGAL,
		"alpb_spmv_plan_hot: %lld slots for %lld columns", (long long) slots, (long long) n);
	ALPB_CHECK(slots == 0 || (indices != nullptr && n > 0), ALPB_ILLEGAL,
		"alpb_spmv_plan_hot: null indices");
	ALPB_CHECK(slots == 0 || p->tile == WM_TILE, ALPB_UNSUPPORTED,
		"alpb_spmv_plan_hot: the plan has no warp tiles");
	cudaStream_t s = as_stream(stream);
	const int rc = hot_build(p, indices, n, slots, s);
	if (rc != ALPB_SUCCESS) return rc;
	p->hot_on = p->hot_k > 0 ? 1 : 0;
	return ALPB_SUCCESS;
}

int alpb_spmv_plan_hot_info(alpb_spmv_plan p, int64_t *slots, double *cover) {
	ALPB_CHECK(p != nullptr, ALPB_ILLEGAL, "alpb_spmv_plan_hot_info: null plan");
	if (slots) *slots = p->hot_on ? p->hot_k : 0;
	if (cover) *cover = p->hot_on ? p->hot_cover : 0.0;
	return ALPB_SUCCESS;
}

int alpb_spmv_autotune(alpb_spmv_plan p, int ring, int64_t n, const uint32_t *indices,
	const void *values, int value_type, const void *x, void *y_scratch, void *stream) {
	ALPB_CHECK(p != nullptr, ALPB_ILLEGAL, "alpb_spmv_autotune: null plan");
	ALPB_CHECK(value_type == ALPB_VOID || value_type == ring_value_type(ring), ALPB_UNSUPPORTED,
		"alpb_spmv_autotune: value type %d with ring %d", value_type, ring);
	cudaStream_t s = as_stream(stream);
	SpmvArgs a{};
	a.m_out = p->m;
	a.n_in = n;
	a.nnz = p->nnz;
	a.offsets = nullptr;
	a.indices = indices;
	a.values = value_type == ALPB_VOID ? nullptr : values;
	a.v = x;
	a.u = y_scratch;
	a.dense_all = true;
	cudaEvent_t e0, e1;
	ALPB_CUDA(cudaEventCreate(&e0));
	ALPB_CUDA(cudaEventCreate(&e1));
	// candidates: merge path, and vector widths around the mean row length; the
	// same ones whatever an earlier tuning chose
	hot_release(p);
	p->vw = p->own_vw;
	struct Cand { int sched, w; bool rows, small; } cands[8];
	int nc = 0;
	cands[nc++] = {ALPB_SCHED_MERGE_PATH, p->vw, false, false};
	if (p->can_small) cands[nc++] = {ALPB_SCHED_MERGE_PATH, p->vw, false, true};
	if (p->can_rows) cands[nc++] = {ALPB_SCHED_VECTOR, p->vw, true, false};
	for (int w = 2; w <= 32; w *= 2) cands[nc++] = {ALPB_SCHED_VECTOR, w, false, false};
	float best = 1e30f;
	int best_i = 0;
	const int saved_vw = p->vw;
	const int saved_rows = p->rows;
	const bool saved_small = p->small;
	a.offsets = p->offsets;
	for (int c = 0; c < nc; ++c) {
		p->vw = cands[c].w;
		p->rows = cands[c].rows;
		p->small = cands[c].small;
		float total = 0;
		for (int rep = 0; rep < 4; ++rep) {
			ALPB_CUDA(cudaEventRecord(e0, s));
			int rc = dispatch_spmv(ring, a, p, cands[c].sched, s);
			if (rc != ALPB_SUCCESS) {
				p->vw = saved_vw;
				p->rows = saved_rows;
				p->small = saved_small;
				return rc;
			}
			ALPB_CUDA(cudaEventRecord(e1, s));
			ALPB_CUDA(cudaEventSynchronize(e1));
			float ms = 0;
			ALPB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
			if (rep > 0) total += ms;  // first run warms caches
		}
		if (total < best) { best = total; best_i = c; }
	}
	p->sched = cands[best_i].sched;
	p->vw = cands[best_i].sched == ALPB_SCHED_VECTOR ? cands[best_i].w : saved_vw;
	p->rows = cands[best_i].rows;
	p->small = cands[best_i].small;
	// skewed rows on the merge path: try the hot-column cache at four sizes,
	// up to what the shared memory left by the warps' tiles holds
	if (p->sched == ALPB_SCHED_MERGE_PATH && p->tile == WM_TILE && n >= (int64_t(1) << 16) &&
		p->nnz >= (int64_t(1) << 20)) {
		constexpr int NH = 4;
		struct HotCand { int64_t k; } hc[NH] = {{std::min<int64_t>(4096, hot_slots_max(ring))},
			{std::min<int64_t>(8192, hot_slots_max(ring))},
			{std::min<int64_t>(12288, hot_slots_max(ring))}, {hot_slots_max(ring)}};
		int best_c = -1;
		for (int c = 0; c < NH; ++c) {
			if (hc[c].k <= 0 || hc[c].k >= n) continue;
			int rc = hot_build(p, indices, n, hc[c].k, s);
			if (rc != ALPB_SUCCESS) {
				cudaEventDestroy(e0);
				cudaEventDestroy(e1);
				return rc;
			}
			if (p->hot_k == 0) continue;
			p->hot_on = 1;
			float total = 0;
			for (int rep = 0; rep < 4; ++rep) {
				ALPB_CUDA(cudaEventRecord(e0, s));
				rc = dispatch_spmv(ring, a, p, ALPB_SCHED_MERGE_PATH, s);
				if (rc != ALPB_SUCCESS) {
					hot_release(p);
					cudaEventDestroy(e0);
					cudaEventDestroy(e1);
					return rc;
				}
				ALPB_CUDA(cudaEventRecord(e1, s));
				ALPB_CUDA(cudaEventSynchronize(e1));
				float ms = 0;
				ALPB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
				if (rep > 0) total += ms;
			}
			if (total < 0.98f * best) {
				best = total;
				best_c = c;
			}
		}
		hot_release(p);
		if (best_c >= 0) {
			const int rc = hot_build(p, indices, n, hc[best_c].k, s);
			if (rc != ALPB_SUCCESS) return rc;
			p->hot_on = p->hot_k > 0 ? 1 : 0;
		}
	}
	ALPB_CUDA(cudaEventDestroy(e0));
	ALPB_CUDA(cudaEventDestroy(e1));
	p->tuned_ms = best / 3.0f;
	return ALPB_SUCCESS;
}

int alpb_mxv(int ring, uint32_t descr, int form, int64_t m_out, int64_t n_in, int64_t nnz,
	const int64_t *offsets, const uint32_t *indices, const void *values, int value_type,
	void *u, uint8_t *u_assigned, int64_t *u_nnz,
	const void *u_mask, const uint8_t *u_mask_assigned, int u_mask_type, int64_t u_mask_count,
	const void *v, const uint8_t *v_assigned, int64_t v_count,
	const void *v_mask, const uint8_t *v_mask_assigned, int v_mask_type, int64_t v_mask_count,
	alpb_spmv_plan plan, void *stream) {
	ALPB_CHECK(ring_value_type(ring) >= 0, ALPB_UNSUPPORTED,
		"alpb_mxv: semiring %d is not instantiated on the device", ring);
	ALPB_CHECK(value_type == ALPB_VOID || value_type == ring_value_type(ring), ALPB_UNSUPPORTED,
		"alpb_mxv: matrix value type %d does not match semiring %d", value_type, ring);
	ALPB_CHECK(m_out >= 0 && n_in >= 0 && nnz >= 0, ALPB_ILLEGAL, "alpb_mxv: negative size");
	ALPB_CHECK(descr <= 16383u, ALPB_ILLEGAL, "alpb_mxv: descriptor out of range");
	ALPB_CHECK(!(descr & ALPB_DESC_TRANSPOSE_MATRIX), ALPB_ILLEGAL,
		"alpb_mxv: transpose_matrix must be resolved by the caller (storage + handedness)");
	const bool masked = u_mask_count >= 0;
	const bool input_masked = v_mask_count >= 0;
	const bool dense_hint = (descr & ALPB_DESC_DENSE) != 0;
	// dense descriptor on a sparse container is ILLEGAL (blas2.hpp:950-971)
	if (dense_hint) {
		ALPB_CHECK(v_count == n_in, ALPB_ILLEGAL,
			"alpb_mxv: dense descriptor with a sparse input vector");
		ALPB_CHECK(!masked || u_mask_count == m_out, ALPB_ILLEGAL,
			"alpb_mxv: dense descriptor with a sparse output mask");
		ALPB_CHECK(!input_masked || v_mask_count == n_in, ALPB_ILLEGAL,
			"alpb_mxv: dense descriptor with a sparse input mask");
	}
	ALPB_CHECK(m_out == 0 || u != nullptr, ALPB_ILLEGAL, "alpb_mxv: null output");
	ALPB_CHECK(n_in == 0 || v != nullptr || (descr & ALPB_DESC_USE_INDEX), ALPB_ILLEGAL,
		"alpb_mxv: null input");
	ALPB_CHECK(u_assigned == nullptr || u_nnz != nullptr, ALPB_ILLEGAL,
		"alpb_mxv: sparse output needs its nnz counter");
	// overlap checks (blas2.hpp:1040-1052)
	ALPB_CHECK((descr & ALPB_DESC_SAFE_OVERLAP) || u != v || u == nullptr, ALPB_OVERLAP,
		"alpb_mxv: output and input vectors overlap");
	ALPB_CHECK(!masked || u_mask == nullptr || u != u_mask, ALPB_OVERLAP,
		"alpb_mxv: output and mask vectors overlap");
	if (plan) {
		ALPB_CHECK(plan->m == m_out && plan->nnz == nnz, ALPB_MISMATCH,
			"alpb_mxv: plan was made for another storage (%lld x nnz %lld)",
			(long long) plan->m, (long long) plan->nnz);
	}
	SpmvArgs a{};
	a.m_out = m_out;
	a.n_in = n_in;
	a.nnz = nnz;
	a.offsets = offsets;
	a.indices = indices;
	a.values = value_type == ALPB_VOID ? nullptr : values;
	a.u = u;
	a.u_assigned = u_assigned;
	a.u_nnz = u_nnz;
	a.u_mask = u_mask;
	a.u_mask_assigned = u_mask_assigned;
	a.u_mask_type = u_mask == nullptr ? ALPB_VOID : u_mask_type;
	a.v = v;
	a.v_assigned = v_assigned;
	a.v_mask = v_mask;
	a.v_mask_assigned = v_mask_assigned;
	a.v_mask_type = v_mask == nullptr ? ALPB_VOID : v_mask_type;
	a.descr = descr;
	a.left = (form & ALPB_FORM_LEFT) ? 1 : 0;
	a.masked = masked;
	a.input_masked = input_masked;
	a.dense_all = u_assigned == nullptr && (v_assigned == nullptr || dense_hint);
	const bool invert = (descr & ALPB_DESC_INVERT_MASK) != 0;
	a.trivial = v_count == 0 || n_in == 0 || m_out == 0 || nnz == 0 ||
		(masked && u_mask_count == 0 && !invert) || (input_masked && v_mask_count == 0 && !invert);
	// The reference picks its loop by size (blas2.hpp:1108-1132, 1311-1334, the
	// sequential backend's rule): the gather over the output's storage, or the
	// scatter over the input's nonzeroes when that loop is shorter.  The two
	// differ observably, so the same rule selects the semantics here:
	//  - gather with a non-inverted output mask walks the mask's assigned set
	//    and never reads its values (:1256-1301): the mask acts structurally;
	//  - scatter (:617-745, :1135-1213) reads the mask by value, adds the
	//    identity (add_identity) to every processed input index whatever the
	//    mask, and never writes explicit zeroes.
	{
		const int64_t gather_loop = masked ? std::min(m_out, 2 * u_mask_count) : m_out;
		int64_t scatter_loop = dense_hint ? n_in
			: std::min(n_in, (input_masked && !invert) ? 2 * std::min(v_mask_count, v_count)
													   : 2 * v_count);
		if (descr & 8192u) scatter_loop = gather_loop + 1;  // force_row_major
		a.scatter_sem = scatter_loop < gather_loop;
		a.mask_by_structure = masked && !invert && !a.scatter_sem && (form & ALPB_FORM_ROWS);
		if (a.mask_by_structure && u_mask_assigned == nullptr) {
			// a dense mask read by structure selects every row
			a.masked = false;
			a.mask_by_structure = false;
		}
		if (a.scatter_sem) a.dense_all = false;
	}
	// many inputs take part: a row of lor is likely decided by its first nonzeroes
	a.probe = (input_masked && !invert ? std::min(v_mask_count, v_count) : v_count) >= n_in / 4;
	if (m_out == 0) return ALPB_SUCCESS;
	return dispatch_spmv(ring, a, plan, 0, as_stream(stream));
}

} // extern "C"
