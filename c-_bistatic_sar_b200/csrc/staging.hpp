// staging.hpp -- host-device copies of large pageable buffers.
//
// The runtime stages a copy from pageable memory through one pinned buffer with one thread,
// which also takes the page faults of a caller's fresh output array: about 18 GB/s, a third
// of what the link carries.  A Stager does the same with a few threads, each with two pinned
// slots of its own: threads claim chunks, copy between the caller's memory and a slot, and
// enqueue the chunk's transfer on the call's stream, so the copies of some chunks overlap the
// transfers of others.  The batched matched filter of 256 x 4096 complex128 samples, host to
// host (16.8 MB each way), took 1.95 ms and takes 1.1 to 1.3 ms.
//
// One Stager belongs to one context and is used under the context's lock.  It is made at the
// first large copy; its threads end and its pinned memory (kSlotBytes x 2 per thread) is
// freed with the context.  Where threads or pinned memory are not to be had, or the caller's
// memory is pinned already, the plain asynchronous copy runs instead.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace bsar_rt {

class Stager {
public:
    static constexpr size_t kSlotBytes = size_t(1) << 20;
    // Smaller copies gain less than waking the threads costs.  Measured one by one / staged on a
    // 16-thread host: uploads 16.8 MB 0.90 / 0.80-1.3 ms, 134 MB 11.2 / 4.1 ms; downloads into a
    // fresh array, whose page faults the threads share, 2.1 MB 0.16 / 0.14 ms, 16.8 MB
    // 0.94 / 0.50-0.62 ms, 134 MB 27 / 8.2 ms.  In a call that downloads as much right after,
    // the threads are awake for both: the matched filter's 16.8 MB upload staged or not, the
    // call takes 1.09 or 1.55 ms.
    static constexpr size_t kMinUpload = size_t(32) << 20, kMinUploadBack = size_t(8) << 20;
    static constexpr size_t kMinDownload = size_t(2) << 20;
    static constexpr int kMaxThreads = 6;

    // nullptr when the pinned slots cannot be had.
    static std::unique_ptr<Stager> make(int device)
    {
        std::unique_ptr<Stager> s(new Stager(device));
        const int want = std::max(1, std::min<int>(kMaxThreads, (int)std::thread::hardware_concurrency() / 2));
        s->lanes_.reserve(want);
        for (int t = 0; t < want; t++) {
            Lane l;
            const bool ok = cudaMallocHost(&l.mem, 2 * kSlotBytes) == cudaSuccess &&
                            cudaEventCreateWithFlags(&l.ev[0], cudaEventDisableTiming) == cudaSuccess &&
                            cudaEventCreateWithFlags(&l.ev[1], cudaEventDisableTiming) == cudaSuccess;
            s->lanes_.push_back(l);
            if (!ok) {
                cudaGetLastError();
                return nullptr;
            }
        }
        try {
            for (int t = 1; t < want; t++) s->threads_.emplace_back([p = s.get(), t] { p->serve(t); });
        } catch (const std::system_error&) {
            // fewer threads; the lanes beyond them stay unused
        }
        return s;
    }

    ~Stager()
    {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        wake_.notify_all();
        for (auto& t : threads_) t.join();
        for (auto& l : lanes_) {
            for (cudaEvent_t e : l.ev)
                if (e) {
                    cudaEventSynchronize(e);     // the last upload from this slot
                    cudaEventDestroy(e);
                }
            if (l.mem) cudaFreeHost(l.mem);
        }
    }

    Stager(const Stager&) = delete;
    Stager& operator=(const Stager&) = delete;

    // Enqueues the upload; the host buffer is read before the call returns.
    cudaError_t upload(void* dev, const void* host, size_t bytes, cudaStream_t st)
    {
        return run(static_cast<char*>(dev), static_cast<char*>(const_cast<void*>(host)), bytes, st, true);
    }

    // The host buffer is written when the call returns.
    cudaError_t download(void* host, const void* dev, size_t bytes, cudaStream_t st)
    {
        return run(static_cast<char*>(const_cast<void*>(dev)), static_cast<char*>(host), bytes, st, false);
    }

    // Whether a copy of this host buffer gains: at least `least` bytes, and not pinned, managed
    // or mapped.
    static bool wanted(const void* host, size_t bytes, size_t least)
    {
        if (bytes < least) return false;
        cudaPointerAttributes at{};
        if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeUnregistered;
    }

private:
    struct Lane {
        char* mem = nullptr;
        cudaEvent_t ev[2] = {nullptr, nullptr};
    };

    explicit Stager(int device) : device_(device) {}

    cudaError_t run(char* dev, char* host, size_t bytes, cudaStream_t st, bool up)
    {
        {
            std::lock_guard<std::mutex> lk(mu_);
            dev_ = dev;
            host_ = host;
            bytes_ = bytes;
            // four chunks a lane, 256 KB to a whole slot each
            chunk_ = std::min(kSlotBytes, std::max(size_t(256) << 10, (bytes / (4 * lanes_.size()) + 65535) & ~size_t(65535)));
            stream_ = st;
            up_ = up;
            next_.store(0);
            error_.store(cudaSuccess);
            busy_ = (int)threads_.size();
            job_++;
        }
        wake_.notify_all();
        work(lanes_[0]);
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [&] { return busy_ == 0; });
        return (cudaError_t)error_.load();
    }

    void serve(int t)
    {
        cudaSetDevice(device_);
        uint64_t seen = 0;
        std::unique_lock<std::mutex> lk(mu_);
        for (;;) {
            wake_.wait(lk, [&] { return stop_ || job_ != seen; });
            if (stop_) return;
            seen = job_;
            lk.unlock();
            work(lanes_[t]);
            lk.lock();
            if (--busy_ == 0) done_.notify_one();
        }
    }

    void check(cudaError_t e)
    {
        if (e != cudaSuccess) {
            int ok = cudaSuccess;
            error_.compare_exchange_strong(ok, (int)e);
        }
    }

    // Offset of the next chunk to copy, or false when none is left (or a copy failed).
    bool claim(size_t& off, size_t& len)
    {
        if (error_.load() != cudaSuccess) return false;
        off = next_.fetch_add(chunk_);
        if (off >= bytes_) return false;
        len = std::min(chunk_, bytes_ - off);
        return true;
    }

    void work(Lane& l)
    {
        size_t off, len;
        if (up_) {
            for (int s = 0; claim(off, len); s ^= 1) {
                check(cudaEventSynchronize(l.ev[s]));            // the slot's previous transfer
                std::memcpy(l.mem + s * kSlotBytes, host_ + off, len);
                check(cudaMemcpyAsync(dev_ + off, l.mem + s * kSlotBytes, len, cudaMemcpyHostToDevice, stream_));
                check(cudaEventRecord(l.ev[s], stream_));
            }
            return;
        }
        // one transfer ahead of the copy out
        size_t o[2], n[2];
        bool has[2] = {false, false};
        auto start = [&](int s) {
            if (!(has[s] = claim(o[s], n[s]))) return;
            check(cudaEventSynchronize(l.ev[s]));
            check(cudaMemcpyAsync(l.mem + s * kSlotBytes, dev_ + o[s], n[s], cudaMemcpyDeviceToHost, stream_));
            check(cudaEventRecord(l.ev[s], stream_));
        };
        start(0);
        for (int s = 0; has[s]; s ^= 1) {
            start(s ^ 1);
            check(cudaEventSynchronize(l.ev[s]));
            std::memcpy(host_ + o[s], l.mem + s * kSlotBytes, n[s]);
        }
    }

    const int device_;
    std::vector<Lane> lanes_;
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable wake_, done_;
    uint64_t job_ = 0;
    int busy_ = 0;
    bool stop_ = false;
    // the current job
    char *dev_ = nullptr, *host_ = nullptr;
    size_t bytes_ = 0, chunk_ = kSlotBytes;
    cudaStream_t stream_ = nullptr;
    bool up_ = true;
    std::atomic<size_t> next_{0};
    std::atomic<int> error_{cudaSuccess};
};

}  // namespace bsar_rt
