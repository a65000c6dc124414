// Status plumbing shared by every entry point: thread-local error text, CUDA
// error translation, launch counter, cached device properties.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>

#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"
#include "ops.h"
#include "tensor_map.h"

namespace cera {

static thread_local char g_err[512] = "";
static std::atomic<uint64_t> g_launches{0};

int32_t fail(int32_t code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int32_t check_cuda(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return CERA_CUDA_OK;
    const int32_t code = e == cudaErrorMemoryAllocation ? CERA_CUDA_ERR_OOM : CERA_CUDA_ERR_CUDA;
    return fail(code, "%s: %s", what, cudaGetErrorString(e));
}

static uint32_t (*g_status_readers[16])();
static int g_n_status_readers = 0;

bool register_kernel_status(uint32_t (*reader)()) {
    if (g_n_status_readers >= 16) return false;
    g_status_readers[g_n_status_readers++] = reader;
    return true;
}

void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }
uint64_t launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

bool pdl_enabled() {
    static const bool v = [] {
        const char *e = getenv("CERA_CUDA_PDL");
        return !(e && e[0] == '0');
    }();
    return v;
}

int sm_count() {
    static thread_local int cached_dev = -1, cached = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev != cached_dev) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached = n;
        cached_dev = dev;
    }
    return cached;
}

namespace {
constexpr int MAX_DEVICES = 64;
// What the scratch pool keeps while it is in use, and once a weight has been freed: the small products of whatever is left (with nothing kept
// the next call of 64 columns of 4096 x 14336 took 360 us, mapping it again, instead of 115).
constexpr uint64_t POOL_IN_USE = 1ull << 30, POOL_KEPT = 64ull << 20;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[MAX_DEVICES] = {};
}  // namespace

void *scratch_alloc(size_t bytes, cudaStream_t st) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= MAX_DEVICES) return nullptr;
    void *p = nullptr;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        if (cudaMallocAsync(&p, bytes, st) == cudaSuccess) return p;  // the graph's own memory, whatever the pool
        cudaGetLastError();
        return nullptr;
    }
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        if (!g_pools[dev]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            uint64_t keep = POOL_IN_USE;
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // another thread may be capturing
            cudaThreadExchangeStreamCaptureMode(&mode);
            const cudaError_t e = cudaMemPoolCreate(&pool, &props);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            g_pools[dev] = pool;
        }
        pool = g_pools[dev];
    }
    if (cudaMallocFromPoolAsync(&p, bytes, pool, st) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}

void scratch_trim() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= MAX_DEVICES) return;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (g_pools[dev]) cudaMemPoolTrimTo(g_pools[dev], POOL_KEPT);
    cudaGetLastError();
}

int32_t tensor_map_2d(CUtensorMap *map, CUtensorMapDataType type, uint32_t elem_bytes, const void *base, uint64_t rows, uint64_t ld, uint32_t box_cols,
                      uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (PFN_cuTensorMapEncodeTiled_v12000)p;
    }();
    if (!encode) return fail(CERA_CUDA_ERR_CUDA, "the driver offers no cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {ld, rows}, strides[1] = {ld * elem_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows}, es[2] = {1, 1};
    const CUresult r = encode(map, type, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(CERA_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled: error %d for [%llu x %llu]", (int)r, (unsigned long long)rows, (unsigned long long)ld);
    return CERA_CUDA_OK;
}

}  // namespace cera

extern "C" {

const char *cera_cuda_last_error(void) { return cera::g_err; }

int32_t cera_cuda_kernel_status(uint32_t *status_out) {
    if (!status_out) return cera::fail(CERA_CUDA_ERR_BAD_ARG, "kernel_status: null argument");
    uint32_t v = 0;
    for (int i = 0; i < cera::g_n_status_readers; ++i) v |= cera::g_status_readers[i]();
    CERA_CUDA_TRY(cudaGetLastError());
    *status_out = v;
    if (v) return cera::fail(CERA_CUDA_ERR_TIMEOUT, "a bounded device-side wait ran out (status word %u)", v);
    return CERA_CUDA_OK;
}

int32_t cera_cuda_device_count(int32_t *count) {
    if (!count) return cera::fail(CERA_CUDA_ERR_BAD_ARG, "count is null");
    int n = 0;
    CERA_CUDA_TRY(cudaGetDeviceCount(&n));
    *count = n;
    return CERA_CUDA_OK;
}

}  // extern "C"
