// Copies of megabytes between the device and pageable host memory: a matrix's code planes out of the quantiser and into a
// layer, a host caller's weights.
//
// The driver copies pageable memory on one thread, through staging of its own, and takes the faults of new pages on the way.  From
// a size on, up to five threads move pieces of 1 MB between the caller's memory and a ring of page-locked ones, while the copy
// engine is at the next.  The calling thread alone talks to the driver: it queues the pieces' device copies, each with an event
// behind it, and asks those events how far the engine has come, every 128 KB of a piece of its own.  The other threads live as long as the
// call and do nothing but memcpy (a stream handle need not mean the same stream in another thread: cudaStreamPerThread does
// not).  On a host of 16 cores: 67 MB into new pages 13.7 -> 4.8 ms, into old ones 3.2 -> 2.2, out of host memory 4.4 -> 2.2; two planes
// of 8.4 MB out of the quantiser 2.2 -> 0.9 (half of it no longer clearing the pages first).  With a look after whole pieces only, the
// others wait for it: 3000 x 4096 out of the quantiser 1.8 instead of 1.5 ms.  Smaller copies gain nothing: 17 MB to the device 0.8
// and 0.8, 4 MB from it 0.2 and 0.2 to 0.5.
#include <algorithm>
#include <atomic>
#include <thread>

#include "tq_host.hpp"

namespace tq {

namespace {

constexpr size_t kPiece = size_t(1) << 20, kLook = size_t(128) << 10;
constexpr size_t kRing = 16;                            // pieces of staging at most
constexpr size_t kThreadsToHost = size_t(8) << 20, kThreadsToDevice = size_t(32) << 20;   // bytes from which on threads are used
constexpr size_t kThreads = 5;                           // with the calling one
// Three threads, and more from 24 pieces on: what other cores have in their caches is slower to read for the caller afterwards (16 MB of
// planes out of the quantiser and into a layer: 2490 us with five threads, 2200 with three, 2300 with one).
constexpr size_t kPiecesPerThread = 8;

struct Piece {
    uint8_t* dst;
    const uint8_t* src;
    size_t bytes;
};

struct CopyEvent {
    cudaEvent_t e = nullptr;
    CopyEvent() { TQ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); }
    ~CopyEvent() { cudaEventDestroy(e); }
    CopyEvent(const CopyEvent&) = delete;
    CopyEvent& operator=(const CopyEvent&) = delete;
};

// The pieces of a call on their way.  Piece i uses place i % ring_ of the staging; pieces are taken up, queued and found done in order.
class PieceMover {
public:
    PieceMover(const std::vector<Piece>& pieces, bool to_device, cudaStream_t st)
        : pieces_(pieces), n_(pieces.size()), ring_(std::min(kRing, n_)), to_device_(to_device), st_(st), moved_(pieces.size()) {
        for (auto& f : moved_) f.store(false, std::memory_order_relaxed);
        if (to_device_) ready_.store(ring_);
    }
    ~PieceMover() {
        stop_.store(true);
        for (std::thread& t : helpers_) t.join();
        if (arrived_ < queued_) cudaStreamSynchronize(st_);   // (a failure: queued copies still read or write the staging)
    }

    void run() {
        if (!to_device_) queue_copies();
        const size_t want = std::min(std::min(kThreads, static_cast<size_t>(std::max(1u, std::thread::hardware_concurrency()))), std::max<size_t>(3, 1 + n_ / kPiecesPerThread));
        try {
            helpers_.reserve(want);
            while (helpers_.size() + 1 < want)
                helpers_.emplace_back([this] {
                    while (!stop_.load(std::memory_order_relaxed) && next_.load(std::memory_order_relaxed) < n_)
                        if (!move_one(false)) std::this_thread::yield();
                });
        } catch (...) {   // fewer threads, then
        }
        // done: to the device, the last copy has arrived; from it, the last piece is with the caller
        while (to_device_ ? arrived_ < n_ : moved_in_order_ < n_) {
            const bool news = look();
            if (!move_one(true) && !news) std::this_thread::yield();
            while (moved_in_order_ < n_ && moved_[moved_in_order_].load(std::memory_order_acquire)) ++moved_in_order_;
        }
    }

private:
    uint8_t* place(size_t i) const { return stage_.host<uint8_t>() + (i % ring_) * kPiece; }

    // Moves the next piece between the caller's memory and its place, if there is one whose place is ready.  The calling thread looks
    // after the others' pieces on the way: a piece takes up to half a millisecond where the pages are new.
    bool move_one(bool calling_thread) {
        size_t i = next_.load(std::memory_order_relaxed);
        do {
            if (i >= ready_.load(std::memory_order_acquire)) return false;
        } while (!next_.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
        const Piece& p = pieces_[i];
        uint8_t* const dst = to_device_ ? place(i) : p.dst;
        const uint8_t* const src = to_device_ ? p.src : place(i);
        for (size_t at = 0; at < p.bytes; at += kLook) {
            std::memcpy(dst + at, src + at, std::min(kLook, p.bytes - at));
            if (calling_thread) look();
        }
        moved_[i].store(true, std::memory_order_release);
        return true;
    }
    bool look() {
        const bool queued = queue_copies(), arrived = find_arrived();
        return queued || arrived;
    }
    // Queues the device copies that can be: to the device those of the pieces in their places, from it those whose place the piece
    // before has left.
    bool queue_copies() {
        const size_t before = queued_;
        for (; queued_ < n_; ++queued_) {
            if (to_device_ ? !moved_[queued_].load(std::memory_order_acquire)
                           : queued_ >= ring_ && !moved_[queued_ - ring_].load(std::memory_order_acquire))
                break;
            const Piece& p = pieces_[queued_];
            if (to_device_) TQ_CUDA(cudaMemcpyAsync(p.dst, place(queued_), p.bytes, cudaMemcpyHostToDevice, st_));
            else TQ_CUDA(cudaMemcpyAsync(place(queued_), p.src, p.bytes, cudaMemcpyDeviceToHost, st_));
            TQ_CUDA(cudaEventRecord(events_[queued_ % ring_].e, st_));
        }
        return queued_ != before;
    }
    // Looks how many device copies have ended.  (A place's event is recorded anew only behind a copy that was found ended.)
    bool find_arrived() {
        const size_t before = arrived_;
        while (arrived_ < queued_) {
            const cudaError_t rc = cudaEventQuery(events_[arrived_ % ring_].e);
            if (rc == cudaErrorNotReady) {
                cudaGetLastError();
                break;
            }
            TQ_CUDA(rc);
            ++arrived_;
        }
        if (arrived_ != before) ready_.store(to_device_ ? std::min(n_, arrived_ + ring_) : arrived_, std::memory_order_release);
        return arrived_ != before;
    }

    const std::vector<Piece>& pieces_;
    const size_t n_;
    const size_t ring_;
    const bool to_device_;
    const cudaStream_t st_;
    PinnedStage stage_{ring_ * kPiece};
    CopyEvent events_[kRing];
    std::vector<std::atomic<bool>> moved_;   // the piece's memcpy is done
    std::atomic<size_t> next_{0};            // pieces taken up
    std::atomic<size_t> ready_{0};           // pieces that may be: their place is free, or holds them
    std::atomic<bool> stop_{false};
    size_t queued_ = 0, arrived_ = 0, moved_in_order_ = 0;   // (the calling thread's)
    std::vector<std::thread> helpers_;
};

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
    // (on a stream that is being captured the driver's own copy gives the error)
    if (total >= (to_device ? kThreadsToDevice : kThreadsToHost) && !stream_is_capturing(st)) {
        PieceMover(pieces, to_device, st).run();
    } else {
        for (const HostCopy& c : large) TQ_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st));
    }
    TQ_CUDA(cudaStreamSynchronize(st));
}

}  // namespace

void copies_to_host(const HostCopy* copies, int n, cudaStream_t st) { copy_host(copies, n, false, st); }
void copies_to_device(const HostCopy* copies, int n, cudaStream_t st) { copy_host(copies, n, true, st); }

}  // namespace tq
