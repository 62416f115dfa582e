// Device memory kept between objects.
//
// A new sequence's cache, a scratch buffer of a quantiser call or a layer's planes took a cudaMalloc each and gave the
// memory back with cudaFree, which waits for the whole device: creating a four-layer cache, filling it with an
// 8192-token prompt and releasing it spent 6 to 70 ms in those calls around 0.3 ms of kernels.  Released blocks are
// kept here instead, by device and size class, and handed out again.
//
//   Bounded    at most kKeepBytes of unused memory per device; beyond it the blocks unused for longest go back to the
//              driver first.  A block of more than half the bound is never kept.
//   Given back blocks unused for kKeepSeconds at the next release; everything unused when an allocation of the library fails,
//              and when the program asks for it (tq_release_cached_memory), which it does for another allocator's sake.
//   Threads    one mutex; a block belongs to one owner at a time.
//   Streams    a block may be released while work that uses it is still queued.  The owner says whether all that work
//              was put on the legacy default stream: then an event recorded there marks its end, and the next owner
//              orders itself behind it - on its stream where it names one, on the host otherwise.  An owner that saw
//              any other stream waits for the device before it releases, as cudaFree did.
//   Capture    memory for work on a stream that is being captured comes from cudaMalloc, which the driver allows or refuses
//              by the capture's mode: growing an object inside a capture is not something that a kept block makes work.
#include <chrono>
#include <list>
#include <mutex>

#include "tq_host.hpp"

namespace tq {

namespace {

constexpr size_t kKeepBytes = size_t(512) << 20;
constexpr double kKeepSeconds = 30.0;
constexpr size_t kKeepPinnedBytes = size_t(32) << 20;
constexpr size_t kStatusWords = 512;   // page-locked status words per page

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

struct Block {
    void* p;
    size_t bytes;
    int device;
    cudaEvent_t pending;   // nullptr: nothing queued uses the block
    double since;
};

struct Word {
    unsigned int* host;
    int device;
    cudaEvent_t pending;
};

struct Pinned {
    void* p;
    void* alias;
    size_t bytes;
};

struct Pool {
    std::mutex mu;
    std::vector<Pinned> pinned;   // page-locked staging, the latest last
    size_t pinned_kept = 0;
    std::list<Block> blocks;   // in order of release: the oldest first
    size_t kept[64] = {0};
    std::list<Word> words;
    std::vector<cudaEvent_t> events[64];   // spare events of each device
};

// Never destroyed: the CUDA runtime may be gone when static destructors run.
Pool& pool() {
    static Pool* const p = new Pool();
    return *p;
}

}  // namespace

bool stream_is_capturing(cudaStream_t st) {
    if (is_legacy_stream(st)) return false;   // it cannot be; asking takes 1.5 us
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TQ_CUDA(cudaStreamIsCapturing(st, &cap));
    return cap != cudaStreamCaptureStatusNone;
}

namespace {

// An event recorded on the current device's legacy default stream, nullptr when that failed (the caller then waits).
cudaEvent_t mark_legacy_stream(Pool& P, int device) {
    // While a blocking stream of the device is captured the question fails, and an event would break the capture.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(cudaStreamLegacy, &cap) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    cudaEvent_t e = nullptr;
    if (!P.events[device].empty()) {
        e = P.events[device].back();
        P.events[device].pop_back();
    } else if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (cudaEventRecord(e, nullptr) == cudaSuccess) return e;
    cudaGetLastError();
    cudaEventDestroy(e);
    return nullptr;
}

void free_block(Pool& P, std::list<Block>::iterator it) {
    P.kept[it->device] -= it->bytes;
    cudaFree(it->p);   // waits for the device: the pending work ends first
    if (it->pending) P.events[it->device].push_back(it->pending);
    P.blocks.erase(it);
}

struct DeviceGuard {
    int before = -1;
    explicit DeviceGuard(int device) {
        if (cudaGetDevice(&before) != cudaSuccess) before = -1;
        if (before != device) cudaSetDevice(device);
        else before = -1;
    }
    ~DeviceGuard() {
        if (before >= 0) cudaSetDevice(before);
    }
};

}  // namespace

// Sizes are rounded up to an eighth of their power of two, so that caches of similar lengths share blocks.
size_t pool_size_class(size_t bytes) {
    size_t step = 512;
    while (step * 16 <= bytes) step *= 2;
    return (bytes + step - 1) / step * step;
}

void* pool_alloc(size_t bytes, int device, cudaStream_t st, bool on_stream) {
    const size_t want = pool_size_class(bytes);
    Pool& P = pool();
    if (device < 0 || device >= 64 || stream_is_capturing(st)) return device_malloc(want);
    void* p = nullptr;
    cudaEvent_t pending = nullptr;
    {
        std::lock_guard<std::mutex> lock(P.mu);
        // Newest first: most likely still in the caches, and the oldest get the chance to age.  Of those that the host would
        // have to wait for (the newest, most likely) only if there is no other; work on the legacy stream waits by itself.
        auto found = P.blocks.end();
        for (auto it = P.blocks.end(); it != P.blocks.begin();) {
            --it;
            if (it->bytes != want || it->device != device) continue;
            if (found == P.blocks.end()) found = it;
            if (it->pending == nullptr || (on_stream && is_legacy_stream(st)) || cudaEventQuery(it->pending) == cudaSuccess) {
                found = it;
                break;
            }
            cudaGetLastError();
        }
        if (found != P.blocks.end()) {
            p = found->p;
            pending = found->pending;
            P.kept[device] -= want;
            P.blocks.erase(found);
        }
    }
    if (p == nullptr) return device_malloc(want);
    if (pending != nullptr) {
        // work on the legacy stream is already behind the event
        cudaError_t rc = cudaSuccess;
        if (!on_stream) rc = cudaEventSynchronize(pending);
        else if (!is_legacy_stream(st)) rc = cudaStreamWaitEvent(st, pending, 0);
        {
            std::lock_guard<std::mutex> lock(P.mu);
            P.events[device].push_back(pending);
        }
        if (rc != cudaSuccess) {
            cudaFree(p);
            TQ_CUDA(rc);
        }
    }
    return p;
}

void* device_malloc(size_t bytes) {
    void* p = nullptr;
    cudaError_t rc = cudaMalloc(&p, bytes);
    if (rc == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        pool_trim();
        rc = cudaMalloc(&p, bytes);
    }
    if (rc == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw OutOfMemory("cudaMalloc of " + std::to_string(bytes) + " bytes: " + cudaGetErrorString(rc));
    }
    TQ_CUDA(rc);
    return p;
}

void pool_release(void* p, size_t bytes, int device, bool idle) {
    if (!p) return;
    const size_t size = pool_size_class(bytes);
    Pool& P = pool();
    std::lock_guard<std::mutex> lock(P.mu);
    DeviceGuard guard(device);
    cudaEvent_t e = nullptr;
    const bool keep = device >= 0 && device < 64 && size <= kKeepBytes / 2;
    if (keep && !idle) e = mark_legacy_stream(P, device);
    if (!keep || (!idle && !e)) {
        cudaFree(p);
        cudaGetLastError();
        return;
    }
    const double now = now_s();
    P.blocks.push_back(Block{p, size, device, e, now});
    P.kept[device] += size;
    while (!P.blocks.empty() && now - P.blocks.front().since > kKeepSeconds) free_block(P, P.blocks.begin());
    for (auto it = P.blocks.begin(); P.kept[device] > kKeepBytes && it != P.blocks.end();) {
        auto next = std::next(it);
        if (it->device == device) free_block(P, it);
        it = next;
    }
}

size_t pool_trim() {
    Pool& P = pool();
    std::lock_guard<std::mutex> lock(P.mu);
    size_t freed = 0;
    while (!P.blocks.empty()) {
        DeviceGuard guard(P.blocks.front().device);
        freed += P.blocks.front().bytes;
        free_block(P, P.blocks.begin());
    }
    return freed;
}

unsigned int* status_word_take(int device) {
    Pool& P = pool();
    std::lock_guard<std::mutex> lock(P.mu);
    for (auto it = P.words.begin(); it != P.words.end(); ++it) {
        if (it->device != device) continue;
        if (it->pending) {
            // a kernel that still runs could report through the word: take another one
            if (cudaEventQuery(it->pending) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            P.events[device].push_back(it->pending);
        }
        unsigned int* const w = it->host;
        P.words.erase(it);
        *w = 0u;
        return w;
    }
    unsigned int* page = nullptr;
    TQ_CUDA(cudaMallocHost(&page, kStatusWords * sizeof(unsigned int)));
    for (size_t i = 1; i < kStatusWords; ++i) P.words.push_back(Word{page + i, device, nullptr});
    page[0] = 0u;
    return page;
}

void status_word_return(unsigned int* w, int device) {
    if (!w) return;
    Pool& P = pool();
    std::lock_guard<std::mutex> lock(P.mu);
    DeviceGuard guard(device);
    cudaEvent_t e = device >= 0 && device < 64 ? mark_legacy_stream(P, device) : nullptr;
    if (!e) return;   // 4 bytes stay with the page
    P.words.push_back(Word{w, device, e});
}

PinnedStage::PinnedStage(size_t bytes) {
    size_t want = size_t(64) << 10;
    while (want < bytes) want *= 2;
    Pool& P = pool();
    {
        std::lock_guard<std::mutex> lock(P.mu);
        for (size_t i = P.pinned.size(); i-- > 0;) {
            if (P.pinned[i].bytes != want) continue;
            p_ = P.pinned[i].p;
            alias_ = P.pinned[i].alias;
            bytes_ = want;
            P.pinned.erase(P.pinned.begin() + static_cast<long>(i));
            P.pinned_kept -= want;
            return;
        }
    }
    TQ_CUDA(cudaHostAlloc(&p_, want, cudaHostAllocPortable | cudaHostAllocMapped));
    bytes_ = want;
    alias_ = pinned_host_device_alias(p_);
    if (alias_ == nullptr) {
        cudaFreeHost(p_);
        throw Error("page-locked staging memory is not mapped for the device");
    }
}

PinnedStage::~PinnedStage() {
    if (!p_) return;
    Pool& P = pool();
    {
        std::lock_guard<std::mutex> lock(P.mu);
        if (P.pinned_kept + bytes_ <= kKeepPinnedBytes) {
            P.pinned.push_back(Pinned{p_, alias_, bytes_});
            P.pinned_kept += bytes_;
            return;
        }
    }
    cudaFreeHost(p_);
}

}  // namespace tq
