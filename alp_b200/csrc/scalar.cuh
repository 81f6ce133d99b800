// Reductions to a host scalar in one launch: block partials, the last block to
// leave one sums them and writes the result to mapped host memory.
//
// What bounds such a call on vectors of up to a million entries is not the
// pass over them but what came after it: a second launch whose one thread
// walked the partials (24 us for 489 of them), an allocation and a release,
// and two copies.  The entry points wait for the stream before they return,
// so their scratch is the calling thread's own and is kept: 8 KB in each
// context the thread uses, left to the next thread when it ends.
#pragma once
#include "common.cuh"

#include <new>

namespace alpb {

constexpr int SCALAR_BLOCK = 256;
constexpr int SCALAR_MAX_BLOCKS = 1000;   // partials that fit the scratch

struct ScalarScratch {
	unsigned long long ctx = 0;     // context_id() of the context it lives in
	uint64_t *part = nullptr;       // [SCALAR_MAX_BLOCKS] on the device
	unsigned *arrived = nullptr;    // zero between calls
	uint64_t *host = nullptr;       // the result, as the host reads it
	uint64_t *host_dev = nullptr;   // and as the kernel writes it
};

// The calling thread's scratch in the current context (runtime.cu).
int scalar_scratch(ScalarScratch *out, cudaStream_t s);

// Blocks of a reduction over n entries: four entries per thread (one batch of
// loads) up to the blocks that are resident together.
inline int scalar_grid(int64_t n) {
	int64_t g = (n + SCALAR_BLOCK * 4 - 1) / (SCALAR_BLOCK * 4);
	int64_t cap = int64_t(sm_count()) * 4;
	if (cap > SCALAR_MAX_BLOCKS) cap = SCALAR_MAX_BLOCKS;
	if (g > cap) g = cap;
	return int(g < 1 ? 1 : g);
}

// Operators whose partials may be combined in any grouping; for the others
// (a caller may pass any operator) one thread folds them in block order.
__host__ __device__ __forceinline__ bool scalar_groups(int op) {
	return op == ALPB_OP_ADD || op == ALPB_OP_MUL || op == ALPB_OP_MIN || op == ALPB_OP_MAX ||
		op == ALPB_OP_LOR || op == ALPB_OP_LAND;
}

// acc over the block, in thread 0: warp trees, then warp 0 over the warps.
template <class T, class Op>
__device__ __forceinline__ T scalar_block(T acc, T ident, const Op &op) {
	__shared__ T sm[SCALAR_BLOCK / 32];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	for (int o = 16; o > 0; o >>= 1) acc = op(acc, T(__shfl_down_sync(0xffffffffu, acc, o)));
	__syncthreads();
	if (lane == 0) sm[w] = acc;
	__syncthreads();
	T r = ident;
	if (w == 0) {
		r = lane < SCALAR_BLOCK / 32 ? sm[lane] : ident;
		for (int o = 16; o > 0; o >>= 1) r = op(r, T(__shfl_down_sync(0xffffffffu, r, o)));
	}
	return r;
}

// Every thread of every block calls with its own acc; the last block writes
// init (op) the total to *out.  groups: see scalar_groups.
template <class T, class Op>
__device__ __forceinline__ void scalar_finish(T acc, T ident, T init, bool groups, const Op &op,
	uint64_t *part, unsigned *arrived, uint64_t *out) {
	__shared__ bool last;
	T *p = reinterpret_cast<T *>(part);
	const T mine = scalar_block(acc, ident, op);
	if (threadIdx.x == 0) {
		p[blockIdx.x] = mine;
		__threadfence();
		last = atomicAdd(arrived, 1u) == gridDim.x - 1;
		__threadfence();
	}
	__syncthreads();
	if (!last) return;
	T r = init;
	if (groups) {
		T v = ident;
		for (int b = threadIdx.x; b < int(gridDim.x); b += SCALAR_BLOCK) v = op(v, T(__ldcg(p + b)));
		v = scalar_block(v, ident, op);
		r = op(init, v);
	} else if (threadIdx.x == 0) {
		for (int b = 0; b < int(gridDim.x); ++b) r = op(r, T(__ldcg(p + b)));
	}
	if (threadIdx.x == 0) {
		*arrived = 0;
		*reinterpret_cast<volatile T *>(out) = r;
		__threadfence_system();
	}
}

} // namespace alpb
