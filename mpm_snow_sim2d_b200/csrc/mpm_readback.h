// Device-to-host reads through pinned memory.
//
// The getters hand back host arrays that the caller allocated, usually pageable. Into
// memory that has been written before, the driver's copy runs at 19 GB/s, and it is left
// to it. Into fresh memory it falls to 5 GB/s (2 with 4 KB pages), since the one thread that
// moves the data also takes the page faults: 9.6 ms for the positions of 3.8M
// particles. There the copy engine fills a ring of pinned chunks while a few threads
// move finished chunks on: 4.0 ms (chunks of 2 MB move a little faster, of 256 KB slower, but pinning
// memory costs up to 0.8 ms per MB). The ring is for fresh memory only (into written memory it
// takes 474 -> 550 us for 8.5 MB, 1.3 -> 1.45 ms for 24 MB, 2.5 -> 2.6 ms for 46 MB), and it
// is made when reads into fresh memory have come to kRingAfter bytes: what it costs to make, 3
// ms, is what it saves on about 20 MB (a first read of 8.5 MB that makes it: 4 ms, 2.5 without).
// Small fields go through a pinned buffer in one piece, one copy and one wait instead
// of one each (a step and the state of 2.3k particles: 62 us against 147). In between,
// starting threads costs more than they save (a 2 MB picture: 560 us against 220).
//
// Both buffers are shared by every solver and batch of the process, of fixed size,
// made when first needed and freed with the last object that holds a ReadbackUser. One
// read uses them at a time; a second one that finds them taken copies directly.
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include <sys/mman.h>
#include <unistd.h>

#include <cuda_runtime.h>

namespace mpm {

class ReadbackRing {
public:
    static constexpr size_t kChunk = 512u << 10;
    static constexpr int kChunks = 8;
    static constexpr int kThreads = 7;  // besides the caller's
    static constexpr size_t kSmall = 256u << 10, kLarge = 8u << 20, kRingAfter = 40u << 20;

    static ReadbackRing& get() {
        static ReadbackRing ring;
        return ring;
    }

    void add_user() {
        std::lock_guard<std::mutex> lock(count_);
        ++users_;
    }
    void drop_user() {
        std::lock_guard<std::mutex> lock(count_);
        if (--users_ > 0) return;
        std::lock_guard<std::mutex> idle(use_);
        free_all();
    }

    // dst[0 .. bytes) = src (device memory) after the work queued on `stream`;
    // returns when dst is filled.
    cudaError_t read(cudaStream_t stream, const void* src, void* dst, size_t bytes) {
        void* d[1] = {dst};
        const size_t n[1] = {bytes};
        return read_parts(stream, src, d, n, 1);
    }

    // The same for consecutive parts of src, each to its own place (null: skipped).
    cudaError_t read_parts(cudaStream_t stream, const void* src, void* const* dst, const size_t* bytes, int parts) {
        size_t total = 0;
        for (int p = 0; p < parts; ++p) total += bytes[p];
        if (total == 0) return cudaStreamSynchronize(stream);
        const char* s = static_cast<const char*>(src);
        if (total <= kSmall) {
            std::unique_lock<std::mutex> lock(use_, std::try_to_lock);
            if (!lock.owns_lock() || !pin(small_, kSmall)) return direct(stream, src, dst, bytes, parts);
            cudaError_t e = cudaMemcpyAsync(small_, s, total, cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess) return e;
            size_t at = 0;
            for (int p = 0; p < parts; at += bytes[p], ++p)
                if (dst[p]) std::memcpy(dst[p], small_ + at, bytes[p]);
            return cudaSuccess;
        }
        for (int p = 0; p < parts; s += bytes[p], ++p) {
            if (!dst[p] || !bytes[p]) continue;
            std::unique_lock<std::mutex> lock(use_, std::defer_lock);
            cudaError_t e = cudaSuccess;
            bool ring = bytes[p] >= kLarge && untouched(dst[p], bytes[p]) && pageable(dst[p]) && worth_it(bytes[p]);
            if (ring) {
                // wait for the stream before the ring, not while holding it
                if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
                ring = lock.try_lock() && ready();
            }
            e = ring ? pipe(stream, s, static_cast<char*>(dst[p]), bytes[p])
                                       : direct(stream, s, dst + p, bytes + p, 1);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

private:
    std::mutex count_, use_;  // taken in this order
    int users_ = 0;
    char* pin_ = nullptr;    // the ring
    char* small_ = nullptr;
    cudaEvent_t ev_[kChunks] = {};
    int device_ = -1;  // of the events
    std::atomic<bool> made_{false};    // pin_ is there
    std::atomic<size_t> without_{0};   // bytes read into fresh memory without the ring

    bool worth_it(size_t bytes) {
        return made_.load() || without_.fetch_add(bytes) + bytes >= kRingAfter;
    }
    // Whether most of [p, p + bytes) has no memory behind it yet (16 pages asked, 4 us).
    static bool untouched(const void* p, size_t bytes) {
        constexpr int kProbes = 16;
        const size_t page = (size_t)sysconf(_SC_PAGESIZE);
        int missing = 0;
        for (int k = 0; k < kProbes; ++k) {
            const size_t at = (reinterpret_cast<size_t>(p) + bytes / kProbes * k) / page * page;
            unsigned char in = 1;
            if (mincore(reinterpret_cast<void*>(at), page, &in) == 0 && !(in & 1)) ++missing;
        }
        return 2 * missing > kProbes;
    }

    // Pinned memory of the caller's is filled by the copy engine alone (164 MB: 3 ms
    // against 8 through the ring).
    static bool pageable(const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }
    static bool pin(char*& p, size_t bytes) {
        if (p || cudaHostAlloc(reinterpret_cast<void**>(&p), bytes, cudaHostAllocPortable) == cudaSuccess) return true;
        cudaGetLastError();
        p = nullptr;
        return false;
    }
    bool ready() {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || !pin(pin_, kChunk * kChunks)) return false;
        if (device_ != dev) {
            drop_events();
            for (cudaEvent_t& e : ev_)
                if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                    cudaGetLastError();
                    e = nullptr;
                    drop_events();
                    return false;
                }
            device_ = dev;
        }
        made_ = true;
        return true;
    }
    void drop_events() {
        for (cudaEvent_t& e : ev_) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        device_ = -1;
    }
    void free_all() {
        drop_events();
        for (char** p : {&pin_, &small_}) {
            if (*p) cudaFreeHost(*p);
            *p = nullptr;
        }
        made_ = false;
        without_ = 0;
    }

    static cudaError_t direct(cudaStream_t stream, const void* src, void* const* dst, const size_t* bytes, int parts) {
        const char* s = static_cast<const char*>(src);
        for (int p = 0; p < parts; s += bytes[p], ++p) {
            if (!dst[p] || !bytes[p]) continue;
            const cudaError_t e = cudaMemcpyAsync(dst[p], s, bytes[p], cudaMemcpyDeviceToHost, stream);
            if (e != cudaSuccess) return e;
        }
        return cudaStreamSynchronize(stream);
    }

    // Runs job() on the caller's thread and up to `helpers` more.
    template <typename F> static void with_threads(int helpers, F&& job) {
        const int cores = (int)std::thread::hardware_concurrency();
        helpers = std::min(helpers, std::max(cores - 1, 0));
        std::vector<std::thread> team;
        try {
            team.reserve((size_t)helpers);
            for (int t = 0; t < helpers; ++t) team.emplace_back(job);
        } catch (const std::exception&) {  // fewer threads then
        }
        job();
        for (std::thread& t : team) t.join();
    }

    cudaError_t pipe(cudaStream_t stream, const char* src, char* dst, size_t bytes) {
        const int chunks = (int)((bytes + kChunk - 1) / kChunk);
        const std::unique_ptr<char[]> moved(new (std::nothrow) char[chunks]());  // under m
        void* const to = dst;
        if (!moved) return direct(stream, src, &to, &bytes, 1);
        std::mutex m;
        std::condition_variable cv;
        int issued = 0, taken = 0;              // under m
        cudaError_t err = cudaSuccess;          // under m
        auto fail = [&](cudaError_t e) {
            std::lock_guard<std::mutex> l(m);
            if (err == cudaSuccess) err = e;
            cv.notify_all();
        };
        auto move_chunks = [&] {
            cudaError_t e = cudaSetDevice(device_);
            if (e != cudaSuccess) return fail(e);
            for (;;) {
                int c;
                {
                    std::unique_lock<std::mutex> l(m);
                    cv.wait(l, [&] { return err != cudaSuccess || taken >= chunks || issued > taken; });
                    if (err != cudaSuccess || taken >= chunks) return;
                    c = taken++;
                }
                if ((e = cudaEventSynchronize(ev_[c % kChunks])) != cudaSuccess) return fail(e);
                const size_t at = (size_t)c * kChunk;
                std::memcpy(dst + at, pin_ + (size_t)(c % kChunks) * kChunk, std::min(kChunk, bytes - at));
                std::lock_guard<std::mutex> l(m);
                moved[c] = 1;
                cv.notify_all();
            }
        };
        auto issue = [&](int c) {
            const size_t at = (size_t)c * kChunk;
            cudaError_t e = cudaMemcpyAsync(pin_ + (size_t)(c % kChunks) * kChunk, src + at, std::min(kChunk, bytes - at),
                                            cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaEventRecord(ev_[c % kChunks], stream);
            if (e != cudaSuccess) return fail(e);
            std::lock_guard<std::mutex> l(m);
            issued = c + 1;
            cv.notify_all();
        };
        std::atomic<bool> issuer{false};
        with_threads(kThreads, [&] {
            if (issuer.exchange(true)) return move_chunks();
            // the first thread here issues the copies, then helps
            for (int c = 0; c < chunks; ++c) {
                if (c >= kChunks) {
                    std::unique_lock<std::mutex> l(m);
                    // no helper may have started: then move the chunk here
                    if (!moved[c - kChunks] && taken <= c - kChunks) {
                        const int k = taken++;
                        l.unlock();
                        const cudaError_t e = cudaEventSynchronize(ev_[k % kChunks]);
                        if (e != cudaSuccess) return fail(e);
                        const size_t at = (size_t)k * kChunk;
                        std::memcpy(dst + at, pin_ + (size_t)(k % kChunks) * kChunk, std::min(kChunk, bytes - at));
                        l.lock();
                        moved[k] = 1;
                        cv.notify_all();
                    }
                    cv.wait(l, [&] { return err != cudaSuccess || moved[c - kChunks]; });
                    if (err != cudaSuccess) return;
                }
                issue(c);
            }
            move_chunks();
        });
        if (err != cudaSuccess) cudaStreamSynchronize(stream);  // nothing of this read may reach the ring later
        return err;
    }
};

// Holds the ring for the life of a solver or batch.
struct ReadbackUser {
    ReadbackUser() { ReadbackRing::get().add_user(); }
    ~ReadbackUser() { ReadbackRing::get().drop_user(); }
    ReadbackUser(const ReadbackUser&) = delete;
    ReadbackUser& operator=(const ReadbackUser&) = delete;
};

}  // namespace mpm
