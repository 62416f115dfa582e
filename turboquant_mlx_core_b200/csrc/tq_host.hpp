// Host-side plumbing shared by the C-ABI translation units: RAII device buffers,
// host/device pointer classification, the thread-local error slot and the tq_array
// handle that travels through the `void*` slots of the C interface.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "tq_common.cuh"

namespace tq {

// ---- error slot (one per thread) -----------------------------------------------------
std::string& last_error_slot();
inline void set_last_error(const std::string& m) { last_error_slot() = m; }

// Run `body`, translating exceptions into the error slot.  Returns `ok` or `fail`.
template <typename R, typename F>
R guarded(R ok_unused, R fail, F&& body) {
    (void)ok_unused;
    try {
        return body();
    } catch (const std::exception& e) {
        set_last_error(e.what());
    } catch (...) {
        set_last_error("unknown error");
    }
    return fail;
}

// ---- device selection -------------------------------------------------------------------
int current_device();
int sm_count(int device);
size_t l2_bytes(int device);
// cudaSetDevice only when another device is current (it is not free even as a no-op).
inline void ensure_device(int device) {
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cur != device) TQ_CUDA(cudaSetDevice(device));
}

// ---- pointers ---------------------------------------------------------------------------
// True when the CUDA driver knows `p` as device (or managed) memory.
inline bool is_device_pointer(const void* p) {
    if (!p) return false;
    cudaPointerAttributes attr{};
    cudaError_t e = cudaPointerGetAttributes(&attr, p);
    if (e != cudaSuccess) {
        cudaGetLastError();  // clear the sticky-free error for unregistered host memory on old drivers
        return false;
    }
    return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

// For page-locked host memory (cudaHostAlloc / cudaHostRegister, mapped as usual under unified
// addressing) returns the address a kernel can use for it, else NULL.
inline void* pinned_host_device_alias(const void* p) {
    if (!p) return nullptr;
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return attr.type == cudaMemoryTypeHost ? attr.devicePointer : nullptr;
}

// ---- device memory (tq_memory.cu: released blocks are kept for the next owner) -----------------
inline bool is_legacy_stream(cudaStream_t st) { return st == nullptr || st == cudaStreamLegacy; }
size_t pool_size_class(size_t bytes);
// Whether work put on the stream is captured in a graph.
bool stream_is_capturing(cudaStream_t st);
// A block on `device`, which must be current, for an object that works on `st`.  on_stream: its first use is work put there;
// otherwise the block is idle when the call returns.
void* pool_alloc(size_t bytes, int device, cudaStream_t st, bool on_stream);
// idle: nothing queued anywhere uses the block; otherwise everything that does was put on the legacy default stream.
void pool_release(void* p, size_t bytes, int device, bool idle);
size_t pool_trim();   // the bytes that went back to the driver
struct OutOfMemory : Error {
    using Error::Error;
};
// cudaMalloc, after giving the unused blocks back where memory is short; OutOfMemory where it still is.
void* device_malloc(size_t bytes);
// A zeroed word of page-locked host memory that the device can write.
unsigned int* status_word_take(int device);
// All work that could write the word was put on the legacy default stream, or has ended.
void status_word_return(unsigned int* w, int device);


// Page-locked host memory for the length of one call that waits for its result (kept for the next call).
class PinnedStage {
public:
    explicit PinnedStage(size_t bytes);
    ~PinnedStage();
    PinnedStage(const PinnedStage&) = delete;
    PinnedStage& operator=(const PinnedStage&) = delete;
    template <typename T = void> T* host() const { return static_cast<T*>(p_); }
    template <typename T = void> T* device() const { return static_cast<T*>(alias_); }   // its address for kernels

private:
    void* p_ = nullptr;
    void* alias_ = nullptr;
    size_t bytes_ = 0;
};

// Which streams an object's memory has been used on: what its release has to wait for.
class StreamUse {
public:
    void note(cudaStream_t st) { other_ = other_ || !is_legacy_stream(st); }
    // True when only work on the legacy default stream can be pending.
    bool only_legacy() const { return !other_; }

private:
    bool other_ = false;
};

class DeviceBuffer {
public:
    DeviceBuffer() = default;
    explicit DeviceBuffer(size_t bytes) { resize(bytes); }
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    DeviceBuffer(DeviceBuffer&& o) noexcept { take(o); }
    DeviceBuffer& operator=(DeviceBuffer&& o) noexcept {
        if (this != &o) { release(); take(o); }
        return *this;
    }
    ~DeviceBuffer() { release(); }

    // Without an owner a release waits for the device; with one it follows the owner's record of streams.
    void owned_by(const StreamUse* use) { use_ = use; }
    // Nothing queued uses the contents any more: the release need not wait.
    void set_idle() { idle_ = true; }

    // Grow-only: keeps the allocation when it is already large enough (contents kept
    // only in that case).
    void reserve(size_t bytes) { grow(bytes, nullptr, false); }
    // ... for contents whose first use is work on `st` (or, not on_stream, perhaps on another one after it).
    void reserve(size_t bytes, cudaStream_t st, bool on_stream = true) { grow(bytes, st, on_stream); }
    void resize(size_t bytes) { reserve(bytes); }
    void release() {
        if (p_) {
            const bool legacy = use_ != nullptr && use_->only_legacy();
            if (!idle_ && !legacy) {
                int cur = -1;
                if (cudaGetDevice(&cur) == cudaSuccess && cur != device_) cudaSetDevice(device_);
                cudaDeviceSynchronize();
                if (cur >= 0 && cur != device_) cudaSetDevice(cur);
            }
            pool_release(p_, n_, device_, idle_ || !legacy);
        }
        p_ = nullptr;
        n_ = 0;
        idle_ = false;
    }
    template <typename T = void> T* as() const { return static_cast<T*>(p_); }
    size_t bytes() const { return n_; }

private:
    void grow(size_t bytes, cudaStream_t st, bool on_stream) {
        if (bytes <= n_) return;
        release();
        const int device = current_device();
        p_ = pool_alloc(bytes, device, st, on_stream);
        device_ = device;
        n_ = bytes;
    }
    void take(DeviceBuffer& o) {
        p_ = o.p_; n_ = o.n_; device_ = o.device_; use_ = o.use_; idle_ = o.idle_;
        o.p_ = nullptr;
        o.n_ = 0;
        o.idle_ = false;
    }
    void* p_ = nullptr;
    size_t n_ = 0;
    int device_ = 0;
    const StreamUse* use_ = nullptr;
    bool idle_ = false;
};

// ---- host memory (tq_host_copy.cu) ---------------------------------------------------------------
struct HostCopy {
    void* dst;
    const void* src;
    size_t bytes;
};
// From device memory, behind the work queued on `st`, into host memory of any kind and back; the calls wait for the copies.
void copies_to_host(const HostCopy* copies, int n, cudaStream_t st);
void copies_to_device(const HostCopy* copies, int n, cudaStream_t st);

// A read-only view of caller data on the device: device pointers are used in place,
// host pointers are copied into `staging` on `stream`.
template <typename T>
const T* device_view(const T* p, size_t count, DeviceBuffer& staging, cudaStream_t stream) {
    if (count == 0) return p;
    if (is_device_pointer(p)) return p;
    staging.reserve(count * sizeof(T), stream);
    TQ_CUDA(cudaMemcpyAsync(staging.as<void>(), p, count * sizeof(T), cudaMemcpyHostToDevice, stream));
    return staging.as<T>();
}

}  // namespace tq

// ---- tensor handle ------------------------------------------------------------------------
struct tq_array_s {
    void* data = nullptr;   // device pointer
    int dtype = 0;          // TQ_F32 / TQ_F16 / TQ_U8 / TQ_U32
    int ndim = 0;
    int shape[8] = {0};
    int device = 0;
    bool owns = false;

    size_t count() const {
        size_t n = 1;
        for (int i = 0; i < ndim; ++i) n *= static_cast<size_t>(shape[i]);
        return n;
    }
    static size_t elem_size(int dt) { return dt == 0 || dt == 3 ? 4 : (dt == 1 ? 2 : 1); }
    size_t nbytes() const { return count() * elem_size(dtype); }
};
