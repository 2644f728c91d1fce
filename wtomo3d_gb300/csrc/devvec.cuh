// Owning device buffers used throughout the native library.
#pragma once
#include "internal.h"
#include "common.cuh"
#include <vector>

namespace wt3d {

// Memory pool of the current device for per-call temporaries (api.cu): keeps up
// to SCRATCH_KEEP bytes between calls while a handle exists, and gives back what it
// does not use when an allocation of the library fails (scratch_trim) or a caller
// asks (wt3d_scratch_trim).  nullptr where pools cannot be made.
constexpr unsigned long long SCRATCH_KEEP = 16ull << 30;
cudaMemPool_t scratch_pool();
void scratch_trim();

// For checks (wt3d_debug_fail_alloc): whether this allocation of the calling thread is
// the one that is to fail as for lack of memory.
bool alloc_is_to_fail();
inline int no_memory(const char *call, size_t bytes, const char *why)
{
    set_error(std::string(call) + "(" + std::to_string(bytes) + " B): " + why);
    return WT3D_ERR_NOMEM;
}

template <class T>
struct DevVec {
    T *p = nullptr;
    size_t n = 0;
    int alloc(size_t count)
    {
        free();
        if (count == 0) return WT3D_OK;
        if (alloc_is_to_fail()) return no_memory("cudaMalloc", count * sizeof(T), "failed for a check");
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e == cudaErrorMemoryAllocation) {   // what the scratch pool keeps may be enough
            cudaGetLastError();
            scratch_trim();
            e = cudaMalloc(&p, count * sizeof(T));
        }
        if (e != cudaSuccess) {
            cudaGetLastError();   // an allocation failure is not sticky: clear it for later checks
            p = nullptr;
            return no_memory("cudaMalloc", count * sizeof(T), cudaGetErrorString(e));
        }
        n = count;
        return WT3D_OK;
    }
    int upload(const std::vector<T> &v)
    {
        int rc = alloc(v.size());
        if (rc) return rc;
        if (!v.empty() && cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
            set_error("upload failed");
            return WT3D_ERR_CUDA;
        }
        return WT3D_OK;
    }
    void free()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    ~DevVec() { free(); }
    DevVec() = default;
    DevVec(const DevVec &) = delete;
    DevVec &operator=(const DevVec &) = delete;
};

// Waits for a stream at the end of its scope.  Declared before the buffers of a call,
// so that on every way out, errors included, nothing of the call is running any more
// when it returns (its caller may free what it passed in, and buffers released on
// another stream would be given to others while still in use), and the buffers'
// release has been seen, without which the pool cannot be trimmed.
struct StreamDone {
    cudaStream_t st;
    ~StreamDone() { cudaStreamSynchronize(st); }
};

// Stream-ordered device buffer from the scratch pool.  Releasing a cudaMalloc
// buffer with cudaFree waits for the whole device, so a per-call temporary of one
// handle would wait for another handle's factorisation; these buffers are
// released in the order of their own stream instead.  The default pool gives its
// memory back to the driver at every synchronisation and maps it anew at the next
// call, 0.4 + 0.6 ms per GB as measured: 8 ms per solve call on 40^3 whose
// Krylov bases took 1.6 GB.  The stream must outlive the buffer's release.
template <class T>
struct StreamBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t st = nullptr;
    int alloc(size_t count, cudaStream_t s)
    {
        release();
        st = s;
        if (count == 0) return WT3D_OK;
        if (alloc_is_to_fail()) return no_memory("cudaMallocAsync", count * sizeof(T), "failed for a check");
        cudaMemPool_t pool = scratch_pool();
        cudaError_t e = pool ? cudaMallocFromPoolAsync(reinterpret_cast<void **>(&p), count * sizeof(T), pool, s)
                             : cudaMallocAsync(reinterpret_cast<void **>(&p), count * sizeof(T), s);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return no_memory("cudaMallocAsync", count * sizeof(T), cudaGetErrorString(e));
        }
        n = count;
        return WT3D_OK;
    }
    // host vector in (pageable memory: staged before the call returns)
    int upload(const std::vector<T> &v, cudaStream_t s)
    {
        int rc = alloc(v.size(), s);
        if (rc) return rc;
        if (!v.empty() && cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s) != cudaSuccess) {
            set_error("upload failed");
            return WT3D_ERR_CUDA;
        }
        return WT3D_OK;
    }
    void release()
    {
        if (p) cudaFreeAsync(p, st);
        p = nullptr;
        n = 0;
    }
    ~StreamBuf() { release(); }
    StreamBuf() = default;
    StreamBuf(const StreamBuf &) = delete;
    StreamBuf &operator=(const StreamBuf &) = delete;
};

}  // namespace wt3d
