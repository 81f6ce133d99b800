// Runtime entry points: init/finalize, error reporting, device memory and
// copies used by the container classes of the grb::b200 backend.
#include "common.cuh"
#include "scalar.cuh"

#include <cuda.h>

#include <cstdarg>
#include <mutex>
#include <new>

namespace alpb {

std::atomic<int64_t> g_launches{0};

static thread_local char t_err[1024] = "";

void set_error(const char *fmt, ...) {
	va_list ap;
	va_start(ap, fmt);
	vsnprintf(t_err, sizeof(t_err), fmt, ap);
	va_end(ap);
}

int sm_count() {
	static int cached[64] = {0};
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
	if (cached[dev] == 0) {
		int v = 0;
		if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
			v = 148;
		cached[dev] = v;
	}
	return cached[dev];
}

size_t type_size(int type) {
	switch (type) {
	case ALPB_VOID: return 0;
	case ALPB_BOOL: return 1;
	case ALPB_INT32: return 4;
	case ALPB_FP64: return 8;
	case ALPB_UINT32: return 4;
	case ALPB_INT64: return 8;
	case ALPB_UINT8: return 1;
	case ALPB_INT8: return 1;
	case ALPB_UINT64: return 8;
	}
	return 0;
}

// The two driver calls are looked up through the runtime, so the library does
// not link the driver library itself.
unsigned long long context_id() {
	typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
	typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long *);
	struct Calls {
		CtxGetCurrentFn current = nullptr;
		CtxGetIdFn id = nullptr;
		Calls() {
			void *f = nullptr, *g = nullptr;
			cudaDriverEntryPointQueryResult q1, q2;
			if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q1) == cudaSuccess &&
				q1 == cudaDriverEntryPointSuccess &&
				cudaGetDriverEntryPoint("cuCtxGetId", &g, cudaEnableDefault, &q2) == cudaSuccess &&
				q2 == cudaDriverEntryPointSuccess) {
				current = reinterpret_cast<CtxGetCurrentFn>(f);
				id = reinterpret_cast<CtxGetIdFn>(g);
			}
			(void) cudaGetLastError();
		}
	};
	static const Calls calls;
	CUcontext ctx = nullptr;
	unsigned long long id = 0;
	if (!calls.id || calls.current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return 0;
	return calls.id(ctx, &id) == CUDA_SUCCESS ? id : 0;
}

// Reduction scratch: a thread holds one per context it reduces in.  A thread that
// ends leaves them for the threads after it, without a call to the runtime (a
// release would invalidate a capture that another thread has under way), so there
// are never more than the threads that reduced at the same time; alpb_finalize
// gives back those of its context that no thread holds.  Addresses of a context
// that is gone are forgotten, never freed: a later context may have given them
// to somebody else.
struct ScalarNode {
	ScalarScratch sc;
	ScalarNode *next = nullptr;
};
static std::mutex g_scalar_mutex;
static ScalarNode *g_scalar_left = nullptr;   // what ended threads left
struct ScalarPool {
	ScalarNode *held = nullptr;
	~ScalarPool() { leave(); }
	void leave() {
		if (!held) return;
		ScalarNode *last = held;
		while (last->next) last = last->next;
		std::lock_guard<std::mutex> lock(g_scalar_mutex);
		last->next = g_scalar_left;
		g_scalar_left = held;
		held = nullptr;
	}
};
static thread_local ScalarPool t_scalar;

// A node of context ctx that an ended thread left, or null.
static ScalarNode *scalar_left(unsigned long long ctx) {
	std::lock_guard<std::mutex> lock(g_scalar_mutex);
	for (ScalarNode **p = &g_scalar_left; *p; p = &(*p)->next)
		if ((*p)->sc.ctx == ctx) {
			ScalarNode *n = *p;
			*p = n->next;
			return n;
		}
	return nullptr;
}

static void scalar_release(ScalarNode *n) {
	if (n->sc.part) cudaFree(n->sc.part);
	if (n->sc.host) cudaFreeHost(n->sc.host);
	delete n;
}

int scalar_scratch(ScalarScratch *out, cudaStream_t s) {
	unsigned long long ctx = context_id();
	if (ctx == 0) {
		ALPB_CUDA(cudaFree(nullptr));   // makes the device's primary context current
		ctx = context_id();
	}
	for (const ScalarNode *p = t_scalar.held; p; p = p->next)
		if (p->sc.ctx == ctx) {
			*out = p->sc;
			return ALPB_SUCCESS;
		}
	ScalarNode *node = scalar_left(ctx);
	if (node) {
		node->next = t_scalar.held;
		t_scalar.held = node;
		*out = node->sc;
		return ALPB_SUCCESS;
	}
	node = new (std::nothrow) ScalarNode;
	ALPB_CHECK(node, ALPB_OUTOFMEM, "reduction scratch: out of host memory");
	ScalarScratch &n = node->sc;
	n.ctx = ctx;
	// allocations of a first call must not disturb a capture that another thread
	// has under way
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
	cudaThreadExchangeStreamCaptureMode(&mode);
	const size_t bytes = size_t(SCALAR_MAX_BLOCKS) * 8 + 8;
	cudaError_t e = cudaMalloc(&n.part, bytes);
	if (e == cudaSuccess) e = cudaMemsetAsync(n.part, 0, bytes, s);
	if (e == cudaSuccess)
		e = cudaHostAlloc(reinterpret_cast<void **>(&n.host), 64, cudaHostAllocMapped);
	if (e == cudaSuccess)
		e = cudaHostGetDevicePointer(reinterpret_cast<void **>(&n.host_dev), n.host, 0);
	if (e == cudaSuccess) e = cudaStreamSynchronize(s);
	if (e != cudaSuccess) {
		cudaGetLastError();
		scalar_release(node);
	}
	cudaThreadExchangeStreamCaptureMode(&mode);
	if (e != cudaSuccess) {
		set_error("reduction scratch: %s", cudaGetErrorString(e));
		return e == cudaErrorMemoryAllocation ? ALPB_OUTOFMEM : ALPB_PANIC;
	}
	n.arrived = reinterpret_cast<unsigned *>(n.part + SCALAR_MAX_BLOCKS);
	node->next = t_scalar.held;
	t_scalar.held = node;
	*out = n;
	return ALPB_SUCCESS;
}

} // namespace alpb

using namespace alpb;

extern "C" {

int alpb_version(void) { return 1; }

const char *alpb_last_error(void) { return t_err; }

int64_t alpb_launch_count(void) { return g_launches.load(); }

int alpb_init(int device) {
	int n = 0;
	ALPB_CUDA(cudaGetDeviceCount(&n));
	ALPB_CHECK(device >= 0 && device < n, ALPB_ILLEGAL, "alpb_init: device %d of %d", device, n);
	ALPB_CUDA(cudaSetDevice(device));
	ALPB_CUDA(cudaFree(nullptr));  // create the primary context now
	// the entry points take their small per-call scratch (block partials,
	// solver state) stream-ordered from the device's default pool: keep what
	// they free in the pool instead of returning it to the driver at every
	// synchronisation, so that repeated calls reuse it
	cudaMemPool_t pool;
	ALPB_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
	uint64_t keep = UINT64_MAX;
	ALPB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
	return ALPB_SUCCESS;
}

int alpb_finalize(void) {
	ALPB_CUDA(cudaDeviceSynchronize());
	t_scalar.leave();
	while (ScalarNode *n = scalar_left(context_id())) scalar_release(n);
	return ALPB_SUCCESS;
}

int alpb_malloc(void **ptr, size_t bytes) {
	ALPB_CHECK(ptr != nullptr, ALPB_ILLEGAL, "alpb_malloc: null out pointer");
	*ptr = nullptr;
	if (bytes == 0) return ALPB_SUCCESS;
	bytes = (bytes + 255) & ~size_t(255);
	cudaError_t e = cudaMalloc(ptr, bytes);
	if (e == cudaErrorMemoryAllocation) {
		cudaGetLastError();
		set_error("alpb_malloc: out of device memory for %zu bytes", bytes);
		return ALPB_OUTOFMEM;
	}
	ALPB_CUDA(e);
	return ALPB_SUCCESS;
}

int alpb_malloc_managed(void **ptr, size_t bytes) {
	ALPB_CHECK(ptr != nullptr, ALPB_ILLEGAL, "alpb_malloc_managed: null out pointer");
	*ptr = nullptr;
	if (bytes == 0) return ALPB_SUCCESS;
	bytes = (bytes + 255) & ~size_t(255);
	cudaError_t e = cudaMallocManaged(ptr, bytes, cudaMemAttachGlobal);
	if (e == cudaErrorMemoryAllocation) {
		cudaGetLastError();
		set_error("alpb_malloc_managed: out of memory for %zu bytes", bytes);
		return ALPB_OUTOFMEM;
	}
	ALPB_CUDA(e);
	return ALPB_SUCCESS;
}

int alpb_prefetch(const void *ptr, size_t bytes, int to_device, void *stream) {
	if (!ptr || bytes == 0) return ALPB_SUCCESS;
	int dev = 0;
	ALPB_CUDA(cudaGetDevice(&dev));
	cudaMemLocation loc;
	loc.type = to_device ? cudaMemLocationTypeDevice : cudaMemLocationTypeHost;
	loc.id = to_device ? dev : 0;
	cudaError_t e = cudaMemPrefetchAsync(ptr, bytes, loc, 0, as_stream(stream));
	if (e != cudaSuccess) {
		// prefetching is a hint: ignore devices without managed-memory support
		cudaGetLastError();
	}
	return ALPB_SUCCESS;
}

int alpb_free(void *ptr) {
	if (ptr) ALPB_CUDA(cudaFree(ptr));
	return ALPB_SUCCESS;
}

int alpb_memcpy_h2d(void *dst, const void *src, size_t bytes, void *stream) {
	if (bytes == 0) return ALPB_SUCCESS;
	ALPB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, as_stream(stream)));
	return ALPB_SUCCESS;
}

int alpb_memcpy_d2h(void *dst, const void *src, size_t bytes, void *stream) {
	if (bytes == 0) return ALPB_SUCCESS;
	ALPB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, as_stream(stream)));
	return ALPB_SUCCESS;
}

int alpb_memcpy_d2d(void *dst, const void *src, size_t bytes, void *stream) {
	if (bytes == 0) return ALPB_SUCCESS;
	ALPB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, as_stream(stream)));
	return ALPB_SUCCESS;
}

int alpb_memset(void *dst, int byte, size_t bytes, void *stream) {
	if (bytes == 0) return ALPB_SUCCESS;
	ALPB_CUDA(cudaMemsetAsync(dst, byte, bytes, as_stream(stream)));
	return ALPB_SUCCESS;
}

int alpb_stream_sync(void *stream) {
	ALPB_CUDA(cudaStreamSynchronize(as_stream(stream)));
	return ALPB_SUCCESS;
}

} // extern "C"
