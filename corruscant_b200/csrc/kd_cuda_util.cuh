// Small CUDA helpers shared by the build and count translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "kd_internal.h"

namespace kd {

struct Error {
    int code;
    char msg[200];
};

[[noreturn]] inline void raise(int code, const char *what, cudaError_t e = cudaSuccess)
{
    Error err;
    err.code = code;
    if (e != cudaSuccess)
        snprintf(err.msg, sizeof err.msg, "%s: %s", what, cudaGetErrorString(e));
    else
        snprintf(err.msg, sizeof err.msg, "%s", what);
    throw err;
}

inline void check(cudaError_t e, const char *what)
{
    if (e != cudaSuccess) raise(e == cudaErrorMemoryAllocation ? KD_ENOMEM : KD_ECUDA, what, e);
}

// Stream-ordered memory pools of their own, per device, beside the default
// pool that every other build and count array comes from (its release
// threshold raised, like the default pool's):
//   kPoolNodes   the node arrays that builds copy to the host.  A node array
//                still being copied while a count runs (deferred builds)
//                would otherwise sit inside a cached block of the default
//                pool that the count's tile-record buffer could have reused.
//   kPoolRecords the counts' tile-record buffers (gigabytes, one per count
//                in flight).  In the default pool, the catalogs and build
//                temporaries of many trees fragment the cached memory, and a
//                count whose record buffer finds no cached block large enough
//                makes the pool map new memory (hundreds of ms for 10 GB).
// Either falls back to the default pool where a pool cannot be made.
enum { kPoolNodes = 0, kPoolRecords = 1 };
inline cudaMemPool_t side_pool(int which)
{
    static std::mutex mu;
    static cudaMemPool_t pools[2][64] = {};
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    cudaMemPool_t def = nullptr;
    if (dev < 0 || dev >= 64 || which < 0 || which > 1) {
        check(cudaDeviceGetDefaultMemPool(&def, dev), "cudaDeviceGetDefaultMemPool");
        return def;
    }
    std::lock_guard<std::mutex> g(mu);
    if (!pools[which][dev]) {
        cudaMemPoolProps props;
        memset(&props, 0, sizeof props);
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) {
            cudaGetLastError();
            check(cudaDeviceGetDefaultMemPool(&def, dev), "cudaDeviceGetDefaultMemPool");
            return def;
        }
        uint64_t thr = UINT64_MAX;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &thr);
        pools[which][dev] = p;
    }
    return pools[which][dev];
}

// Device memory a pool holds but has not handed out (reusable at once).
inline size_t pool_idle_bytes(cudaMemPool_t p)
{
    uint64_t reserved = 0, used = 0;
    if (cudaMemPoolGetAttribute(p, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(p, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved > used ? (size_t)(reserved - used) : 0;
}

// Stream-ordered allocations owned by one call; anything not released to a
// longer-lived owner is freed when the call ends.  A pool of temporaries only
// (nothing of it is kept) takes its small arrays from shared pieces of 1 MB: a
// build of a few thousand points asks for about sixty, at 2 us each with the
// release.
struct Pool {
    static constexpr size_t kPiece = (size_t)1 << 20, kSmall = kPiece / 16;
    cudaStream_t s;
    bool pieces;
    std::vector<void *> ptrs;
    size_t bytes = 0;
    char *piece = nullptr;
    size_t left = 0;
    explicit Pool(cudaStream_t st, bool temporaries = false) : s(st), pieces(temporaries) {}
    template <class T> T *alloc(size_t n)
    {
        const size_t want = ((n ? n : 1) * sizeof(T) + 255) & ~(size_t)255;
        if (!pieces || want > kSmall) return take<T>(n);
        if (want > left) {
            piece = take<char>(kPiece);
            left = kPiece;
        }
        char *const p = piece;
        piece += want;
        left -= want;
        return (T *)p;
    }
    template <class T> T *take(size_t n)
    {
        void *p = nullptr;
        size_t b = (n ? n : 1) * sizeof(T);
        cudaError_t e = cudaMallocAsync(&p, b, s);
        if (e != cudaSuccess) {
            cudaGetLastError();
            raise(KD_ENOMEM, "device allocation failed", e);
        }
        ptrs.push_back(p);
        bytes += b;
        return (T *)p;
    }
    // n elements from a given memory pool (stream-ordered like alloc), or null
    template <class T> T *try_alloc_from(cudaMemPool_t mp, size_t n, cudaError_t *why = nullptr)
    {
        void *p = nullptr;
        size_t b = (n ? n : 1) * sizeof(T);
        cudaError_t e = cudaMallocFromPoolAsync(&p, b, mp, s);
        if (why) *why = e;
        if (e != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ptrs.push_back(p);
        bytes += b;
        return (T *)p;
    }
    template <class T> T *alloc_from(cudaMemPool_t mp, size_t n)
    {
        cudaError_t e;
        T *const p = try_alloc_from<T>(mp, n, &e);
        if (!p) raise(KD_ENOMEM, "device allocation failed", e);
        return p;
    }
    // hand ownership of p to the caller (it will not be freed by ~Pool)
    template <class T> T *keep(T *p)
    {
        for (auto &q : ptrs)
            if (q == (void *)p) q = nullptr;
        return p;
    }
    ~Pool()
    {
        for (void *p : ptrs)
            if (p) cudaFreeAsync(p, s);
    }
};

// One non-blocking stream per API call: calls on different threads do not
// serialise on each other's work.  Up to kIdle streams per device wait, with
// nothing in flight, for a later call: to make and destroy one takes 92 us, and
// tens of ms now and then on a machine whose other GPUs keep the driver busy.
struct Stream {
    static constexpr size_t kIdle = 8;
    struct Idle {
        std::mutex mu;
        std::vector<cudaStream_t> dev[64];
    };
    static Idle &idle()
    {
        static Idle *i = new Idle;  // outlives every thread's calls
        return *i;
    }
    cudaStream_t s = nullptr;
    int dev = 0;
    Stream()
    {
        check(cudaGetDevice(&dev), "cudaGetDevice");
        if (dev < 64) {
            std::lock_guard<std::mutex> g(idle().mu);
            auto &v = idle().dev[dev];
            if (!v.empty()) {
                s = v.back();
                v.pop_back();
                return;
            }
        }
        check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
    }
    ~Stream()
    {
        if (!s) return;
        if (cudaStreamSynchronize(s) == cudaSuccess && dev < 64) {
            std::lock_guard<std::mutex> g(idle().mu);
            auto &v = idle().dev[dev];
            if (v.size() < kIdle) {
                try {
                    v.push_back(s);
                    return;
                } catch (const std::bad_alloc &) {
                }
            }
        }
        cudaStreamDestroy(s);
    }
    Stream(const Stream &) = delete;
    Stream &operator=(const Stream &) = delete;
    void sync() { check(cudaStreamSynchronize(s), "kernel execution"); }
};

// Keep freed device memory cached in the stream-ordered pool so repeated
// builds and counts do not pay for fresh allocations.
void init_device();

inline unsigned blocks_for(long long n, int threads)
{
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 0x7fffffff) b = 0x7fffffff;
    return (unsigned)b;
}

#define KD_LAUNCH_CHECK(what) ::kd::check(cudaGetLastError(), what)

}  // namespace kd
