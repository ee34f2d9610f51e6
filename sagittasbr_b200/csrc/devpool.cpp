// devpool.cpp -- device memory of scenes, plans and calls, from one CUDA memory pool per
// device.  A cudaMalloc maps memory anew and a cudaFree waits for the whole device: a
// one-angle sbr_run of a 20k-triangle sphere spent 130 of its 200 us outside its kernels,
// a 181-azimuth one with raster buffers 6 of 19 ms.  The pool keeps up to kKeepOpen
// unused bytes while a scene of the device exists and kKeepIdle afterwards; the rest goes
// back at the next synchronisation (a look at a 20k-triangle sphere 218 -> 111 us, a
// 181-azimuth raster sweep 20.0 -> 14.8 ms, a small scene set-up 2.9 -> 0.34 ms).  Blocks change hands on a stream of the pool's own
// that is waited for before a block is handed out, so callers need no stream order.
#include "devpool.hpp"

#include <mutex>
#include <unordered_map>

namespace sbr {
namespace {

constexpr int kDevices = 64;
constexpr unsigned long long kKeepOpen = 2560ull << 20;  // a chunk of raster buffers fits (plan.cpp)
constexpr unsigned long long kKeepIdle = 64ull << 20;

struct Pool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    int scenes = 0;
    unsigned long long live = 0;                  // bytes handed out
    std::unordered_map<void*, size_t> sizes;
};
std::mutex& g_mu = *new std::mutex;               // never destroyed: scenes may close while the
Pool* const g_pools = new Pool[kDevices];         // process ends

// What the pool may hold before it gives memory back: the blocks in use count as well.
void set_threshold(Pool& P) {
    unsigned long long bytes = P.live + (P.scenes > 0 ? kKeepOpen : kKeepIdle);
    cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &bytes);
}

// The device's pool, made on first use (g_mu is held).
cudaError_t get(int device, Pool** out) {
    if (device < 0 || device >= kDevices) return cudaErrorInvalidDevice;
    Pool& P = g_pools[device];
    if (!P.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool;
        cudaError_t e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        e = cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        P.pool = pool;
        set_threshold(P);
    }
    *out = &P;
    return cudaSuccess;
}

}  // namespace

cudaError_t pool_alloc(int device, void** p, size_t bytes) {
    *p = nullptr;
    if (bytes == 0) bytes = 1;
    std::lock_guard<std::mutex> lock(g_mu);
    Pool* P = nullptr;
    cudaError_t e = get(device, &P);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, P->pool, P->stream);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();  // not sticky; the caller reports it
    if (e != cudaSuccess) return e;
    P->live += bytes;
    P->sizes[*p] = bytes;
    set_threshold(*P);
    return cudaStreamSynchronize(P->stream);
}

void pool_free(int device, void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(g_mu);
    Pool* P = nullptr;
    if (get(device, &P) != cudaSuccess) return;
    const auto it = P->sizes.find(p);
    if (it == P->sizes.end()) return;
    P->live -= it->second;
    P->sizes.erase(it);
    set_threshold(*P);
    cudaFreeAsync(p, P->stream);
}

void pool_open(int device) {
    std::lock_guard<std::mutex> lock(g_mu);
    Pool* P = nullptr;
    if (get(device, &P) == cudaSuccess && P->scenes++ == 0) set_threshold(*P);
}

void pool_close(int device) {
    std::lock_guard<std::mutex> lock(g_mu);
    Pool* P = nullptr;
    if (get(device, &P) != cudaSuccess || --P->scenes > 0) return;
    set_threshold(*P);
    cudaStreamSynchronize(P->stream);
    cudaMemPoolTrimTo(P->pool, P->live + kKeepIdle);
}

}  // namespace sbr
