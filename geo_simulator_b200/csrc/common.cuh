// Shared internals of libgeofem: error handling, device buffers, host/device
// pointer staging, the bounded grid barrier and deterministic grid reductions.
#pragma once

#include <cuda/atomic>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "geo_fem.h"

namespace geo {

// ------------------------------------------------------------------ errors
struct Error {
    int code;
    std::string msg;
};

[[noreturn]] inline void fail(int code, const std::string& msg) { throw Error{code, msg}; }

#define GEO_CUDA(expr)                                                                      \
    do {                                                                                    \
        cudaError_t e_ = (expr);                                                            \
        if (e_ != cudaSuccess) {                                                            \
            ::geo::fail(e_ == cudaErrorMemoryAllocation ? GEO_ERR_OUT_OF_MEMORY : GEO_ERR_CUDA, \
                        std::string(#expr) + ": " + cudaGetErrorString(e_));                \
        }                                                                                   \
    } while (0)

#define GEO_CHECK_ARG(cond, msg)                               \
    do {                                                       \
        if (!(cond)) ::geo::fail(GEO_ERR_INVALID_ARG, (msg)); \
    } while (0)

// Device-side error flags (bitwise OR into a device word).
enum : int {
    DEV_ERR_SINGULAR = 1,
    DEV_ERR_TIMEOUT = 2,
    DEV_ERR_BOUNDS = 4,
};

// ------------------------------------------------------------------ device memory
// Caching allocator behind every DevBuf (devmem.cu). A freed block goes back to a
// per-device cache once the device has finished the work queued before the free
// (the wait cudaFree implies, without its unmapping) and is handed out again for a
// request of the same rounded size, so objects created and destroyed call after
// call stop paying cudaMalloc / cudaFree. A cudaMalloc that runs out of memory
// releases the device's cache and is retried once.
void* dev_alloc(size_t bytes);
void dev_free(void* p) noexcept;
void dev_release_cached(int device);  // device < 0: every device

// ------------------------------------------------------------------ buffers
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    explicit DevBuf(size_t count) { alloc(count); }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this != &o) { release(); p = o.p; n = o.n; o.p = nullptr; o.n = 0; }
        return *this;
    }
    ~DevBuf() { release(); }
    void alloc(size_t count) {
        release();
        if (count == 0) return;
        p = static_cast<T*>(dev_alloc(count * sizeof(T)));
        n = count;
    }
    // grow-only reallocation for workspaces
    void ensure(size_t count) {
        if (count > n) alloc(count);
    }
    void release() {
        if (p) dev_free(p);
        p = nullptr;
        n = 0;
    }
    size_t bytes() const { return n * sizeof(T); }
};

// Pinned host staging buffer.
template <class T>
struct HostBuf {
    T* p = nullptr;
    size_t n = 0;
    HostBuf() = default;
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    ~HostBuf() { if (p) cudaFreeHost(p); }
    void ensure(size_t count) {
        if (count <= n) return;
        if (p) cudaFreeHost(p);
        p = nullptr;
        n = 0;
        GEO_CUDA(cudaMallocHost(&p, count * sizeof(T)));
        n = count;
    }
};

// True when p points into memory the GPU of the current device can address as
// device memory (cudaMalloc / managed); false for pageable or pinned host memory.
inline bool is_device_ptr(const void* p) {
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Returns a device pointer holding n elements of src: src itself when it is
// device memory, otherwise a copy staged into tmp (async on stream).
template <class T>
const T* stage_in(const T* src, size_t n, DevBuf<T>& tmp, cudaStream_t s) {
    if (n == 0) return nullptr;
    if (is_device_ptr(src)) return src;
    tmp.ensure(n);
    GEO_CUDA(cudaMemcpyAsync(tmp.p, src, n * sizeof(T), cudaMemcpyHostToDevice, s));
    return tmp.p;
}

// Copies n elements from device src to dst (host or device) on stream s.
template <class T>
void copy_out(T* dst, const T* src, size_t n, cudaStream_t s) {
    if (n == 0) return;
    GEO_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyDefault, s));
}

inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// ------------------------------------------------------------------ device helpers
__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier state in device memory (zeroed before each persistent launch).
struct GridSync {
    unsigned int count;
    unsigned int gen;
    int error;  // DEV_ERR_* bits
    int pad;
};

// Bounded grid-wide barrier for a cooperatively launched (co-resident) grid.
// Every wait is bounded by timeout_ns of %globaltimer; on timeout, or when another
// block already raised an error, the barrier returns false and the caller must
// return from the kernel (all blocks then leave within one timeout).
__device__ __forceinline__ bool grid_barrier(GridSync* gs, unsigned int nblocks,
                                             unsigned long long timeout_ns) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned int, cuda::thread_scope_device> gen(gs->gen);
        cuda::atomic_ref<unsigned int, cuda::thread_scope_device> cnt(gs->count);
        cuda::atomic_ref<int, cuda::thread_scope_device> err(gs->error);
        int ok = 1;
        // thread 0's release (the arrival) and acquire (the new generation) cover the block's
        // other threads through the block barriers on either side
        const unsigned int g = gen.load(cuda::memory_order_relaxed);
        if (cnt.fetch_add(1u, cuda::memory_order_acq_rel) == nblocks - 1) {
            cnt.store(0u, cuda::memory_order_relaxed);
            gen.fetch_add(1u, cuda::memory_order_release);
        } else {
            const unsigned long long t0 = global_timer_ns();
            unsigned int spins = 0;
            while (gen.load(cuda::memory_order_acquire) == g) {
                if ((++spins & 63u) == 0) {
                    if (err.load(cuda::memory_order_relaxed) != 0) { ok = 0; break; }
                    if (global_timer_ns() - t0 > timeout_ns) {
                        err.fetch_or(DEV_ERR_TIMEOUT, cuda::memory_order_relaxed);
                        ok = 0;
                        break;
                    }
                }
                __nanosleep(32);
            }
        }
        if (ok && err.load(cuda::memory_order_relaxed) != 0) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Block-wide sum of K doubles, valid in thread 0 only. blockDim.x must be a multiple
// of 32 and <= 1024. Fixed shuffle tree: deterministic.
template <int K>
__device__ __forceinline__ void block_sum0(double (&v)[K]) {
    __shared__ double red[32][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    __syncthreads();  // an earlier sum may still read red
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = lane < nw ? red[lane][k] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        }
    }
}

// Sum of the per-block partials part[b*K + k] (b < nblocks) in a fixed order, valid in
// thread 0; every block obtains bit-identical totals. Every thread of the block takes
// its share of the partials, several loads in flight: one warp walking them alone
// (19 dependent steps for 592 blocks) cost 3 us more after every reduction.
template <int K>
__device__ __forceinline__ void grid_sum0(const double* part, int nblocks, double (&t)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        if (K == 2) {
            const double2 w = __ldcg(reinterpret_cast<const double2*>(part) + b);
            t[0] += w.x;
            t[K - 1] += w.y;
        } else {
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] += __ldcg(part + (size_t)b * K + k);
        }
    }
    block_sum0<K>(t);
}

// grid_sum0 of partials written before the last grid barrier or ticket, valid in all threads.
template <int K>
__device__ __forceinline__ void grid_total(const double* part, int nblocks, double (&out)[K]) {
    __shared__ double tot[K];
    double t[K];
    grid_sum0<K>(part, nblocks, t);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) tot[k] = t[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = tot[k];
    __syncthreads();
}

// A block's contribution to grid_all_sum: value and epoch, written and read as one word.
struct __align__(16) GridSlot {
    double v;
    unsigned long long epoch;
};
__device__ __forceinline__ void slot_put(GridSlot* s, double v, unsigned long long epoch) {
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n"
                 :: "l"(s), "l"(__double_as_longlong(v)), "l"(epoch) : "memory");
}
__device__ __forceinline__ unsigned long long slot_get(const GridSlot* s, double& v) {
    unsigned long long lo, hi;
    asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(lo), "=l"(hi) : "l"(s) : "memory");
    v = __longlong_as_double((long long)lo);
    return hi;
}

// Grid-wide barrier and sum in one exchange, for a co-resident grid: every block publishes
// its K sums with the running number of the exchange, and its first warp waits for those
// of all blocks and adds them in a fixed order (bit-identical totals everywhere, valid in
// all threads). Against grid_barrier and grid_total it saves the counter that all blocks
// queue at, the wait for its generation, the load of the partials behind it and three of
// five block barriers. slots: [2][stride], stride >= K nblocks, all of it zero before the
// launch; turn counts the exchanges of the kernel and starts at 0. A block reuses a slot
// two exchanges later, when every block has read it. Bounded as grid_barrier; false on
// timeout.
template <int K>
__device__ __forceinline__ bool grid_all_sum(GridSlot* slots, int stride, GridSync* gs, int nblocks,
                                             unsigned long long& turn, unsigned long long timeout_ns, double (&v)[K]) {
    __shared__ double red[2][32][K], tot[2][K];
    __shared__ int s_ok[2];
    const int par = (int)(turn & 1), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GridSlot* mine = slots + par * stride;
    ++turn;
    auto warp_sum = [&]() {
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    };
    warp_sum();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[par][warp][k] = v[k];
    __syncthreads();  // puts the block's work before the release below
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = lane < (int)(blockDim.x >> 5) ? red[par][lane][k] : 0.0;
        warp_sum();
        if (lane == 0) {
            cuda::atomic_thread_fence(cuda::memory_order_release, cuda::thread_scope_device);
#pragma unroll
            for (int k = 0; k < K; ++k) slot_put(mine + k * nblocks + blockIdx.x, v[k], turn);
        }
        bool ok = true;
        unsigned long long t0 = 0;
        unsigned int spins = 0;
        cuda::atomic_ref<int, cuda::thread_scope_device> err(gs->error);
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = 0.0;
        constexpr int kFlight = 5;  // slots per lane and sum in flight: 160 blocks at a time
        for (int b0 = lane; b0 < nblocks && ok; b0 += 32 * kFlight) {
            double w[kFlight][K];
            bool all;
            do {
                all = true;
#pragma unroll
                for (int i = 0; i < kFlight; ++i)
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int b = b0 + 32 * i;
                        w[i][k] = 0.0;
                        if (b < nblocks && slot_get(mine + k * nblocks + b, w[i][k]) != turn) all = false;
                    }
                if (!all && (++spins & 15u) == 0) {
                    const unsigned long long now = global_timer_ns();
                    if (t0 == 0) t0 = now;
                    if (err.load(cuda::memory_order_relaxed) != 0) ok = false;
                    if (now - t0 > timeout_ns) {
                        err.fetch_or(DEV_ERR_TIMEOUT, cuda::memory_order_relaxed);
                        ok = false;
                    }
                }
            } while (!all && ok);
#pragma unroll
            for (int i = 0; i < kFlight; ++i)
#pragma unroll
                for (int k = 0; k < K; ++k) v[k] += w[i][k];
        }
        cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
        ok = __all_sync(0xffffffffu, ok);
        warp_sum();
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) tot[par][k] = v[k];
            s_ok[par] = ok;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = tot[par][k];
    return s_ok[par] != 0;
}

// Block-level partial of K doubles -> part[blockIdx.x*K + k] (thread 0 writes).
template <int K>
__device__ __forceinline__ void store_partial(double* part, double (&v)[K]) {
    block_sum0<K>(v);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) __stcg(part + (size_t)blockIdx.x * K + k, v[k]);
}

}  // namespace geo
