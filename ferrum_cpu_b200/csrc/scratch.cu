// Device memory of single calls on a caller's stream (CallScratch), and the host-visible status word of a resident weight.
//
// A product on a caller's stream returns before its kernels run, so its scratch can belong neither to the weight (two streams
// would share it) nor to a growing buffer (a capture could not make it). It is taken from a pool per device in the order of
// the stream and given back in that order: calls that may overlap get memory of their own, a captured call becomes an
// allocation node of its graph, and what the pool keeps between calls is bounded by kScratchKept and shared by all weights of
// the device. The pool never makes one stream wait for another. The last weight of a device returns it whole.
#include <mutex>

#include "fc_common.cuh"

namespace fc {

namespace {
struct Pool {
    cudaMemPool_t pool = nullptr;
    int weights = 0;
};
Pool g_pools[64];
std::mutex g_mutex;
}  // namespace

// Made with the first weight of a device, so that a call under stream capture finds it.
int scratch_retain(int device) {
    if (device < 0 || device >= 64) return fail(FC_E_ARG, "device %d out of range", device);
    std::lock_guard<std::mutex> lock(g_mutex);
    Pool& p = g_pools[device];
    if (!p.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        FC_CUDA(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = kScratchKept;
        int no = 0;
        cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            FC_CUDA(e);
        }
        p.pool = pool;
    }
    ++p.weights;
    return FC_OK;
}
void scratch_release(int device) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Pool& p = g_pools[device];
    if (--p.weights == 0) cudaMemPoolTrimTo(p.pool, 0);
}

int CallScratch::take(int device, size_t bytes, cudaStream_t st) {
    st_ = st;
    if (g_debug.withhold_scratch == 1) return FC_OK;
    const cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, g_pools[device].pool, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        p = nullptr;
        return FC_OK;
    }
    FC_CUDA(e);
    return FC_OK;
}
CallScratch::~CallScratch() {
    if (p) cudaFreeAsync(p, st_);
}

int take_planes(CallScratch& scratch, Planes& x, int planes, size_t n, int device, cudaStream_t st) {
    const size_t bytes = (2 * n + 255) & ~(size_t)255;
    FC_TRY(scratch.take(device, planes * bytes, st));
    x.n = planes;
    for (int i = 0; i < planes; ++i) x.p[i] = (char*)scratch.p + i * bytes;
    return FC_OK;
}

int StatusWord::create() {
    void* h = nullptr;
    FC_CUDA(cudaHostAlloc(&h, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
    host = (volatile int*)h;
    *host = 0;
    FC_CUDA(cudaHostGetDevicePointer((void**)&dev, h, 0));
    return FC_OK;
}
void StatusWord::destroy() {
    if (host) cudaFreeHost((void*)host);
    host = nullptr;
    dev = nullptr;
}
int StatusWord::check(const char* what) {
    const int s = *host;
    if (s == 0) return FC_OK;
    *host = 0;
    return fail(FC_E_TIMEOUT, "a bounded wait inside the tensor-core GEMM of %s ran out (status %d)", what, s);
}

}  // namespace fc
