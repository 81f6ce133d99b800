// Dense products over short, regular rows (stencils): one lane group per row,
// the matrix streamed through shared memory.
//
// What bounds it is HBM: 12 bytes per nonzero read once, everything else in
// L1 or L2.  W lanes reading a row straight from memory (k_spmv_vector_dense)
// touch a new line per row in every load and hold only a few loads in flight.
// Here a warp owns chunks of consecutive rows, whose indices and values are
// one contiguous range each: it copies them by 16-byte cp.async into its own
// shared-memory stages, RS_STAGES - 1 chunks ahead of the one it sums, so the
// loads are whole lines and their latency hides behind the chunk before.
// Consecutive rows on consecutive lanes gather consecutive x, which the SM's
// L1 serves to all of a stencil's diagonals.  No block-wide barrier, no spin.
#pragma once
#include "common.cuh"

namespace alpb {

// Measured us per product (4 lanes per row before): 27-point 129 x 127 x 131
// 299 -> 164, 5-point 2000^2 92 -> 74; rows_pay (spmv.cu) says where the lanes
// are the faster ones.  27-point with 10 / 14 / 20 warps per SM
// 224 / 185 / 165 (24 are what the registers allow, about 20 what the stages
// of 27-point rows allow), with one / four lanes a row 176 / 193, with three
// stages 193.
constexpr int RS_STAGES = 2;
constexpr int RS_MAX_LEN = 64;       // longest row taken
constexpr int RS_MAX_WARPS = 24;
constexpr int RS_SLACK = 32;         // see rs_cap

__device__ __forceinline__ void rs_copy16(void *dst, const void *src, int bytes) {
	const unsigned d = unsigned(__cvta_generic_to_shared(dst));
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void rs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void rs_wait() {
	asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Copy bytes [beg, end) of src (16-byte aligned, `total` bytes long) to dst,
// which takes byte beg & ~15 first; nothing past the array's end is read.
__device__ __forceinline__ void rs_fetch(unsigned char *dst, const void *src, int64_t beg,
	int64_t end, int64_t total, int lane) {
	const int64_t b0 = beg & ~int64_t(15);
	const unsigned char *p = static_cast<const unsigned char *>(src);
	for (int64_t o = b0 + 16 * lane; o < end; o += 16 * 32)
		rs_copy16(dst + (o - b0), p + o, total - o < 16 ? int(total - o) : 16);
}

// L lanes per row, RPL rows per lane: a chunk is 32 / L * RPL rows.  U: a
// lane's gathers in flight.  A row's sum: each lane's entries in order in
// batches of U, the batches' sums in order, then the row's L lanes by tree.
template <class R, int L, int RPL, int U>
__global__ void __launch_bounds__(32 * RS_MAX_WARPS, 1)
k_spmv_rows(const int64_t *__restrict__ offsets, const uint32_t *__restrict__ indices,
	const typename R::T *__restrict__ values, const typename R::T *__restrict__ x,
	typename R::T *__restrict__ y, int64_t m, int64_t nnz, int cap, int left) {
	using T = typename R::T;
	constexpr int H = 32 / L, ROWS = H * RPL;
	extern __shared__ __align__(16) unsigned char rs_smem[];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nwb = blockDim.x >> 5;
	const int sub = lane / L, k = lane % L;
	const size_t stage = size_t(cap) * (sizeof(T) + 4);
	unsigned char *mine = rs_smem + size_t(w) * RS_STAGES * stage;
	const int64_t chunks = (m + ROWS - 1) / ROWS;
	// chunks go round the blocks first: a small matrix uses every SM
	const int64_t nw = int64_t(gridDim.x) * nwb;
	const int64_t c0 = int64_t(w) * gridDim.x + blockIdx.x;
	// offsets of this lane's rows, loaded one chunk before they are used
	int64_t o[RPL], e[RPL];
	const auto load_rows = [&](int64_t c) {
#pragma unroll
		for (int r = 0; r < RPL; ++r) {
			const int64_t i = c * ROWS + r * H + sub;
			o[r] = e[r] = 0;
			if (c < chunks && i < m) {
				o[r] = offsets[i];
				e[r] = offsets[i + 1];
			}
		}
	};
	// the nonzeroes of the chunk to copy next, loaded one chunk before the copy
	int64_t b = 0, t = 0;
	const auto bounds = [&](int64_t c) {
		if (c < chunks) {
			b = offsets[c * ROWS];
			t = offsets[(c + 1) * ROWS < m ? (c + 1) * ROWS : m];
		}
	};
	// A chunk of more nonzeroes than a stage holds (offsets that changed after
	// the plan took their longest row) is not copied, but read where it stands.
	unsigned direct = 0;   // a bit per stage
	const auto fetch = [&](int64_t c, int s) {
		direct &= ~(1u << s);
		if (c < chunks && t - b > cap - RS_SLACK) {
			direct |= 1u << s;
		} else if (c < chunks) {
			unsigned char *d = mine + s * stage;
			if (values)
				rs_fetch(d, values, b * int64_t(sizeof(T)), t * int64_t(sizeof(T)),
					nnz * int64_t(sizeof(T)), lane);
			rs_fetch(d + size_t(cap) * sizeof(T), indices, b * 4, t * 4, nnz * 4, lane);
		}
		rs_commit();   // an empty group keeps the count
	};
#pragma unroll
	for (int s = 0; s < RS_STAGES - 1; ++s) {
		bounds(c0 + s * nw);
		fetch(c0 + s * nw, s);
	}
	bounds(c0 + (RS_STAGES - 1) * nw);
	load_rows(c0);
	int s = 0;
	for (int64_t c = c0; c < chunks; c += nw) {
		__syncwarp();   // every lane is done with the stage that is refilled
		fetch(c + (RS_STAGES - 1) * nw, s == 0 ? RS_STAGES - 1 : s - 1);
		bounds(c + RS_STAGES * nw);
		T yv[RPL];
		int beg[RPL], len[RPL];
		int64_t ob[RPL];
#pragma unroll
		for (int r = 0; r < RPL; ++r) {
			const int64_t i = c * ROWS + r * H + sub;
			yv[r] = k == 0 && e[r] > o[r] ? y[i] : R::zero();
			ob[r] = o[r];
			len[r] = int(e[r] - o[r]);
		}
		const int64_t first = __shfl_sync(0xffffffffu, o[0], 0);
#pragma unroll
		for (int r = 0; r < RPL; ++r) beg[r] = int(ob[r] - first);
		load_rows(c + nw);
		rs_wait<RS_STAGES - 1>();
		__syncwarp();
		// the stage starts at the 16-byte boundary at or before the first byte
		const T *sv = reinterpret_cast<const T *>(mine + s * stage) +
			(first & (16 / int64_t(sizeof(T)) - 1));
		const uint32_t *si = reinterpret_cast<const uint32_t *>(mine + s * stage +
			size_t(cap) * sizeof(T)) + (first & 3);
#pragma unroll
		for (int r = 0; r < RPL; ++r) {
			T acc = R::zero();
			if (direct >> s & 1u) {
				for (int q = k; q < len[r]; q += L) {
					const T a = values ? values[ob[r] + q] : R::one();
					const T xv = __ldg(x + indices[ob[r] + q]);
					acc = R::add(acc, left ? R::mull(xv, a) : R::mulr(a, xv));
				}
				len[r] = len[r] > 0 ? -1 : 0;   // summed
			}
			for (int q0 = k; q0 < len[r]; q0 += U * L) {
				T xv[U], part = R::zero();
#pragma unroll
				for (int q = 0; q < U; ++q)
					if (q0 + q * L < len[r]) xv[q] = __ldg(x + si[beg[r] + q0 + q * L]);
#pragma unroll
				for (int q = 0; q < U; ++q)
					if (q0 + q * L < len[r]) {
						const T a = values ? sv[beg[r] + q0 + q * L] : R::one();
						part = R::add(part, left ? R::mull(xv[q], a) : R::mulr(a, xv[q]));
					}
				acc = R::add(acc, part);
			}
#pragma unroll
			for (int d = 1; d < L; d <<= 1) acc = R::add(acc, __shfl_xor_sync(0xffffffffu, acc, d));
			if (k == 0 && len[r] != 0) y[c * ROWS + r * H + sub] = R::add(yv[r], acc);
		}
		s = s + 1 == RS_STAGES ? 0 : s + 1;
	}
	rs_wait<0>();
}

// Entries a stage holds: the chunk's rows at most, and the slack of rounding
// its first byte down and its last up to 16 (1-byte values: 15 entries each).
template <class R>
inline int rs_cap(int rows, int maxlen) {
	return (rows * maxlen + RS_SLACK + 15) / 16 * 16;
}

} // namespace alpb
