// Copies of megabytes between the device and pageable host memory: a matrix's code planes out of the quantiser and into a
// layer, a host caller's weights.
//
// The driver copies pageable memory on one thread, through staging of its own, and takes the faults of new pages on the way.  From
// a size on, up to four threads move pieces of 1 MB between the caller's memory and a ring of page-locked ones, each behind its
// own event, while the copy engine is at the next.  The threads live as long as the call.  On a host of 16 cores: 67 MB into
// new pages 13.7 -> 4.8 ms, into old ones 3.2 -> 2.2, out of host memory 4.4 -> 2.4; two planes of 8.4 MB out of the quantiser
// 2.2 -> 0.9 (half of it no longer clearing the pages first).  Smaller copies gain nothing: 17 MB to the device 0.8 and 0.8, 4 MB
// from it 0.2 and 0.2 to 0.5.
#include <algorithm>
#include <atomic>
#include <system_error>
#include <thread>

#include "tq_host.hpp"

namespace tq {

namespace {

constexpr size_t kPiece = size_t(1) << 20;
constexpr int kRing = 8;                                // pieces of staging
constexpr size_t kThreadsToHost = size_t(8) << 20, kThreadsToDevice = size_t(32) << 20;   // bytes from which on threads are used
constexpr int kThreads = 4;

struct Piece {
    uint8_t* dst;
    const uint8_t* src;
    size_t bytes;
};

struct Ring {
    PinnedStage stage{kRing * kPiece};
    cudaEvent_t event[kRing] = {};
    cudaStream_t st;
    explicit Ring(cudaStream_t s) : st(s) {
        for (cudaEvent_t& e : event) TQ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    ~Ring() {
        cudaStreamSynchronize(st);   // (queued copies still read or write the staging)
        for (cudaEvent_t e : event)
            if (e) cudaEventDestroy(e);
    }
    uint8_t* place(size_t i) const { return stage.host<uint8_t>() + (i % kRing) * kPiece; }
};

// All pieces, by the calling thread and as many others as there is use for.
void move_pieces(const std::vector<Piece>& pieces, bool to_device, cudaStream_t st) {
    const size_t n = pieces.size();
    Ring ring(st);
    const int device = current_device();
    std::vector<std::atomic<bool>> issued(n);   // the piece's device copy is queued, its event recorded behind it
    for (auto& f : issued) f.store(false, std::memory_order_relaxed);
    std::atomic<size_t> next{0};
    std::atomic<int> failed{cudaSuccess};
    auto issue = [&](size_t i) {
        const Piece& p = pieces[i];
        cudaError_t rc = to_device ? cudaMemcpyAsync(p.dst, ring.place(i), p.bytes, cudaMemcpyHostToDevice, st)
                                   : cudaMemcpyAsync(ring.place(i), p.src, p.bytes, cudaMemcpyDeviceToHost, st);
        if (rc == cudaSuccess) rc = cudaEventRecord(ring.event[i % kRing], st);
        if (rc != cudaSuccess) failed.store(rc);
        issued[i].store(true, std::memory_order_release);
        return rc == cudaSuccess;
    };
    // Waits until piece i's device copy has ended.  (Its place belongs to whoever does: pieces are taken in order, and the one that
    // issues a copy does so before it takes another piece.)
    auto arrived = [&](size_t i) {
        while (!issued[i].load(std::memory_order_acquire)) {
            if (failed.load() != cudaSuccess) return false;
            std::this_thread::yield();
        }
        const cudaError_t rc = cudaEventSynchronize(ring.event[i % kRing]);
        if (rc != cudaSuccess) failed.store(rc);
        return rc == cudaSuccess;
    };
    auto work = [&] {
        for (size_t i; failed.load() == cudaSuccess && (i = next.fetch_add(1)) < n;) {
            if (to_device) {
                if (i >= kRing && !arrived(i - kRing)) return;
                std::memcpy(ring.place(i), pieces[i].src, pieces[i].bytes);
                if (!issue(i)) return;
            } else {
                if (!arrived(i)) return;
                std::memcpy(pieces[i].dst, ring.place(i), pieces[i].bytes);
                if (i + kRing < n && !issue(i + kRing)) return;
            }
        }
    };
    if (!to_device)
        for (size_t i = 0; i < n && i < kRing; ++i)
            if (!issue(i)) break;
    std::vector<std::thread> helpers;
    const size_t want = std::min<size_t>(std::min<size_t>(kThreads, std::max(1u, std::thread::hardware_concurrency())), n);
    helpers.reserve(want);
    for (size_t t = 1; t < want; ++t) {
        try {
            helpers.emplace_back([&] {
                const cudaError_t rc = cudaSetDevice(device);
                if (rc != cudaSuccess) failed.store(rc);
                else work();
            });
        } catch (const std::system_error&) {
            break;   // fewer threads, then
        }
    }
    work();
    for (std::thread& t : helpers) t.join();
    TQ_CUDA(static_cast<cudaError_t>(failed.load()));
    TQ_CUDA(cudaStreamSynchronize(st));
}

void copy_host(const HostCopy* copies, int n, bool to_device, cudaStream_t st) {
    std::vector<Piece> pieces;
    std::vector<HostCopy> large;
    size_t total = 0;
    for (int i = 0; i < n; ++i) {
        const HostCopy& c = copies[i];
        const void* const host = to_device ? c.src : c.dst;
        if (c.bytes == 0) continue;
        if (c.bytes < kPiece || pinned_host_device_alias(host) != nullptr) {
            TQ_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st));
            continue;
        }
        total += c.bytes;
        large.push_back(c);
        for (size_t at = 0; at < c.bytes; at += kPiece)
            pieces.push_back(Piece{static_cast<uint8_t*>(c.dst) + at, static_cast<const uint8_t*>(c.src) + at, std::min(kPiece, c.bytes - at)});
    }
    if (total >= (to_device ? kThreadsToDevice : kThreadsToHost)) {
        move_pieces(pieces, to_device, st);
        return;
    }
    for (const HostCopy& c : large) TQ_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st));
    TQ_CUDA(cudaStreamSynchronize(st));
}

}  // namespace

void copies_to_host(const HostCopy* copies, int n, cudaStream_t st) { copy_host(copies, n, false, st); }
void copies_to_device(const HostCopy* copies, int n, cudaStream_t st) { copy_host(copies, n, true, st); }

void read_values(void* dst, const void* src, size_t bytes) {
    if (is_device_pointer(src)) TQ_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost));
    else std::memcpy(dst, src, bytes);
}

}  // namespace tq
