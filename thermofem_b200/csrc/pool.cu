// pool.cu -- the library's device memory pool: one stream-ordered CUDA pool
// per device, shared by every context of the process.
//
// A setup allocates and frees a few hundred buffers.  cudaMalloc and cudaFree
// take about 350 us each on a B200 whatever the size (cudaFree waits for the
// device, too), and CUDA's default pool gives every free byte back at each
// synchronisation, so the next allocation maps it again (6.5 ms per GiB).
// From this pool an allocation takes 2 us.
//
// What the pool keeps is bounded: free memory stays with it while a setup
// runs, and at the end of every setup and destroy call pool_trim() returns
// what exceeds kPoolKeep (all of it once the device's last context is gone).
// A cudaMalloc of this process that finds no memory gets what the pool holds
// free (seen on a filled device), so only other processes miss it.
#include <map>
#include <mutex>

#include "common.cuh"

namespace tfb {
namespace {

// Free bytes kept between calls, per device: 2 % of its memory.  (A hierarchy
// set up twice reserves 1.5 GiB in all at 128^3 and 2.7 GiB at 192^3, itself
// included.)
constexpr uint64_t kPoolKeep = uint64_t(4) << 30;

struct DevicePool {
    cudaMemPool_t pool{nullptr};
    cudaStream_t stream{nullptr};  // of frees whose context is gone
    int contexts{0};
};

std::mutex &pool_mutex() {
    static std::mutex *m = new std::mutex;  // never destroyed: buffers may be released at process exit
    return *m;
}
DevicePool &pool_of(int device) {  // pool_mutex() held
    static auto *pools = new std::map<int, DevicePool>;
    DevicePool &p = (*pools)[device];
    if (!p.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cuda_check(cudaMemPoolCreate(&p.pool, &props), "cudaMemPoolCreate");
        uint64_t all = UINT64_MAX;  // trimmed by pool_trim, not at every synchronisation
        cuda_check(cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &all), "pool threshold");
    }
    return p;
}

// Calls of this thread inside the scope leave every stream capture in
// progress alone (giving memory back ends a capture otherwise, also the
// caller's own one around a call that uses temporary arrays).
struct RelaxedCapture {
    cudaStreamCaptureMode mode{cudaStreamCaptureModeRelaxed};
    RelaxedCapture() { swap(); }
    ~RelaxedCapture() { swap(); }
    RelaxedCapture(const RelaxedCapture &) = delete;
    RelaxedCapture &operator=(const RelaxedCapture &) = delete;
    void swap() {
        if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) cudaGetLastError();
    }
};

}  // namespace

void pool_context_opened(int device) {
    std::lock_guard<std::mutex> lock(pool_mutex());
    ++pool_of(device).contexts;
}

void pool_context_closed(int device) noexcept {
    {
        std::lock_guard<std::mutex> lock(pool_mutex());
        try {
            --pool_of(device).contexts;
        } catch (...) {
            return;
        }
    }
    pool_trim(device);
}

void pool_trim(int device) noexcept {
    std::lock_guard<std::mutex> lock(pool_mutex());
    const RelaxedCapture relaxed;
    try {
        DevicePool &p = pool_of(device);
        uint64_t used = 0, reserved = 0;
        if (cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess ||
            cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        const uint64_t keep = used + (p.contexts > 0 ? kPoolKeep : 0);
        if (reserved > keep && cudaMemPoolTrimTo(p.pool, keep) != cudaSuccess) cudaGetLastError();
    } catch (...) {
    }
}

// (cudaFree would give the block back, but leave it counted as used: the bound
// of pool_trim() would rise with every such block)
void pool_free(int device, void *p) noexcept {
    {
        std::lock_guard<std::mutex> lock(pool_mutex());
        const RelaxedCapture relaxed;
        try {
            DevicePool &d = pool_of(device);
            if (!d.stream)
                cuda_check(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking), "cudaStreamCreate");
            cuda_check(cudaFreeAsync(p, d.stream), "cudaFreeAsync");
            cuda_check(cudaStreamSynchronize(d.stream), "cudaFreeAsync");
        } catch (...) {
            cudaGetLastError();
        }
    }
    pool_trim(device);
}

void pool_released(const StreamLife &life) noexcept {
    if (life.open && cudaStreamSynchronize(life.stream) != cudaSuccess) cudaGetLastError();
    pool_trim(life.device);
}

void *pool_allocate(int device, cudaStream_t stream, size_t bytes) {
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(pool_mutex());
        pool = pool_of(device).pool;
    }
    void *p = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, pool, stream);
    if (e == cudaErrorMemoryAllocation) {
        // free blocks too small for this one may hold what is missing
        cudaGetLastError();
        cuda_check(cudaStreamSynchronize(stream), "pool allocation");
        cuda_check(cudaMemPoolTrimTo(pool, 0), "pool trim");
        e = cudaMallocFromPoolAsync(&p, bytes, pool, stream);
    }
    cuda_check(e, "cudaMallocFromPoolAsync");
    return p;
}

bool on_device(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    int device = 0;
    return a.type == cudaMemoryTypeDevice && cudaGetDevice(&device) == cudaSuccess && a.device == device;
}

void wait_for_device() noexcept {
    void *p = nullptr;
    if (cudaMalloc(&p, 256) == cudaSuccess) {
        cudaFree(p);
        return;
    }
    // (a full device)
    cudaGetLastError();
    if (cudaDeviceSynchronize() != cudaSuccess) cudaGetLastError();
}

}  // namespace tfb
