// Copies between pageable host memory and the device, staged through pinned
// slices by a few host threads.
//
// Why: the driver stages a pageable copy with one thread (about 10 GB/s, and
// page faults of fresh result arrays come on top) while the link takes 55 GB/s.
// Each worker copies its own slices into its own pinned buffers and enqueues
// them itself, so workers meet only at the start and the end of a transfer.
// Measured: opening a 972k-triangle mesh (97 MB; the shading half beside the BVH
// build) 11.6 -> 4.5 ms, 1M ray queries (32 MB in, 29 MB out) 8.2 -> 5.0 ms; a 3 MB
// image gradient, still in the caller's cache, 0.5 ms slower.
//
// A process has one copier per device, whatever the number of its renderers: the
// three threads, 8 MB of pinned memory and the events are made when transfers are
// worth it and given back with the last renderer.  It takes one transfer at a
// time, from any thread; a transfer that finds it taken copies plainly, so
// renderers never wait for one another's streams.
// A process forked off has none of the threads: there the copier copies plainly
// and is left alone when its renderers go (a condition variable that vanished
// threads wait on cannot be destroyed).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <unistd.h>

namespace pt {

class HostCopier {
public:
    struct Piece {
        void* device;
        void* host; // (only read by uploads)
        size_t bytes;
    };

    // The copier of a device.
    static std::shared_ptr<HostCopier> of(int device)
    {
        static std::mutex& lock = *new std::mutex; // (outlive every renderer)
        static std::map<int, std::weak_ptr<HostCopier>>& live = *new std::map<int, std::weak_ptr<HostCopier>>;
        std::lock_guard<std::mutex> hold(lock);
        std::shared_ptr<HostCopier> c = live[device].lock();
        if (c == nullptr || c->forked()) {
            c.reset(new HostCopier(device), [](HostCopier* p) {
                if (!p->forked()) {
                    delete p;
                }
            });
            live[device] = c;
        }
        return c;
    }

    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;
    ~HostCopier()
    {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            stop_ = true;
        }
        wake_.notify_all();
        for (std::thread& t : threads_) {
            t.join();
        }
        release();
    }

    // Worth a stream of its own beside other work.
    static bool large(const Piece* p, size_t n)
    {
        size_t total = 0;
        for (size_t i = 0; i < n; ++i) {
            total += p[i].bytes;
        }
        return total >= kBesideBytes;
    }

    // One transfer, ended by finish() or with the object.
    class Transfer {
    public:
        explicit Transfer(HostCopier& c) : c_(c) {}
        Transfer(const Transfer&) = delete;
        Transfer& operator=(const Transfer&) = delete;
        ~Transfer() { finish(); }

        // Starts copying the pieces to the device on stream s; the sources may be
        // changed, and work that reads the copies be put on s, after finish().
        // Transfers too small to gain, from memory that is not pageable or on a
        // stream that cannot be shared with the workers are enqueued at once.
        cudaError_t upload(const Piece* p, size_t n, cudaStream_t s) { return begin(p, n, s, true); }
        // Copies the pieces from the device once the work on s is done; the data is
        // there after finish().
        cudaError_t download(const Piece* p, size_t n, cudaStream_t s) { return begin(p, n, s, false); }

        cudaError_t finish()
        {
            if (!hold_.owns_lock()) {
                return cudaSuccess;
            }
            const cudaError_t e = c_.wait();
            hold_.unlock();
            return e;
        }

    private:
        cudaError_t begin(const Piece* p, size_t n, cudaStream_t s, bool up)
        {
            cudaError_t e = finish();
            size_t total = 0;
            bool staged = s != cudaStreamPerThread && !c_.forked();
            for (size_t i = 0; i < n && e == cudaSuccess; ++i) {
                total += p[i].bytes;
                cudaPointerAttributes a{};
                if (p[i].bytes > 0 && cudaPointerGetAttributes(&a, p[i].host) == cudaSuccess) {
                    staged = staged && a.type == cudaMemoryTypeUnregistered;
                } else {
                    cudaGetLastError();
                }
            }
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            staged = staged && total >= kMinBytes && cudaStreamIsCapturing(s, &cs) == cudaSuccess &&
                cs == cudaStreamCaptureStatusNone && e == cudaSuccess;
            if (staged) {
                hold_ = std::unique_lock<std::mutex>(c_.use_, std::try_to_lock);
                if (hold_.owns_lock()) {
                    if (c_.plain_ < kWorthBytes) {
                        c_.plain_ += total;
                    } else if (c_.ready()) {
                        c_.start(p, n, s, up);
                        return cudaSuccess;
                    }
                    hold_.unlock();
                }
            }
            for (size_t i = 0; i < n && e == cudaSuccess; ++i) {
                if (p[i].bytes > 0) {
                    e = up ? cudaMemcpyAsync(p[i].device, p[i].host, p[i].bytes, cudaMemcpyHostToDevice, s)
                           : cudaMemcpyAsync(p[i].host, p[i].device, p[i].bytes, cudaMemcpyDeviceToHost, s);
                }
            }
            if (e == cudaSuccess && !up) {
                e = cudaStreamSynchronize(s);
            }
            return e;
        }

        HostCopier& c_;
        std::unique_lock<std::mutex> hold_; // of c_.use_, while the copier works on this transfer
    };

private:
    static constexpr size_t kSlice = 1024u << 10; // (256 KB: 5.8 ms for the mesh above, 512: 4.8, 1024: 4.5)
    static constexpr int kWorkers = 4; // the calling thread is one of them
    static constexpr int kBuffers = 2; // per worker: one is filled while the other is in flight
    // Staging gains from about 12 MB on (plain, staged: 131k-ray queries, 4 MB in
    // and out, 1.15, 1.15 ms; 200k 1.8, 1.9; 500k, 16 and 14 MB, 4.05, 3.07; 1M 8.2,
    // 5.0; meshes of 150k triangles, 6 + 9 MB, 1.48, 1.63; 300k, 12 + 18 MB, 2.4, 2.1).
    static constexpr size_t kMinBytes = 12u << 20;
    // The pinned memory and the threads take 4 - 8 ms to make, what staging gains on
    // about this much: made once that much has been copied plainly, so that few
    // transfers never pay for it and many pay once.
    static constexpr size_t kWorthBytes = 96u << 20;
    static constexpr size_t kBesideBytes = 32u << 20;

    bool forked() const { return getpid() != process_; }

    explicit HostCopier(int device) : device_(device) {}

    void start(const Piece* p, size_t n, cudaStream_t s, bool up)
    {
        pieces_.assign(p, p + n);
        stream_ = s;
        up_ = up;
        next_ = 0;
        error_ = cudaSuccess;
        slices_ = 0;
        for (const Piece& q : pieces_) {
            slices_ += (q.bytes + kSlice - 1) / kSlice;
        }
        {
            std::lock_guard<std::mutex> lock(mutex_);
            busy_ = static_cast<int>(threads_.size());
            ++turn_;
        }
        wake_.notify_all();
    }
    // The started transfer's end, with this thread as one of the workers.
    cudaError_t wait()
    {
        work(0);
        std::unique_lock<std::mutex> lock(mutex_);
        done_.wait(lock, [this] { return busy_ == 0; });
        return static_cast<cudaError_t>(error_.load());
    }

    // Threads, pinned memory and events (false: they cannot be had; plain copies).
    bool ready()
    {
        if (state_ != 0) {
            return state_ > 0;
        }
        state_ = -1;
        if (std::thread::hardware_concurrency() <= static_cast<unsigned int>(kWorkers)) {
            return false;
        }
        if (cudaHostAlloc(reinterpret_cast<void**>(&pinned_), kSlice * kBuffers * kWorkers, cudaHostAllocDefault) !=
            cudaSuccess) {
            cudaGetLastError();
            pinned_ = nullptr;
            return false;
        }
        for (cudaEvent_t& ev : events_) {
            if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                ev = nullptr;
                release();
                return false;
            }
        }
        try {
            pieces_.reserve(8);
            threads_.reserve(kWorkers - 1);
            for (int w = 1; w < kWorkers; ++w) {
                threads_.emplace_back([this, w] { loop(w); });
            }
        } catch (...) {
            if (threads_.empty()) {
                release();
                return false;
            }
        }
        state_ = 1;
        return true;
    }

    void release()
    {
        for (cudaEvent_t& ev : events_) {
            if (ev != nullptr) {
                cudaEventSynchronize(ev); // (its buffer may be in flight)
                cudaEventDestroy(ev);
                ev = nullptr;
            }
        }
        if (pinned_ != nullptr) {
            cudaFreeHost(pinned_);
            pinned_ = nullptr;
        }
    }

    void loop(int w)
    {
        cudaSetDevice(device_);
        unsigned long long seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lock(mutex_);
                wake_.wait(lock, [&] { return stop_ || turn_ != seen; });
                if (stop_) {
                    return;
                }
                seen = turn_;
            }
            work(w);
            {
                std::lock_guard<std::mutex> lock(mutex_);
                if (--busy_ == 0) {
                    done_.notify_all();
                }
            }
        }
    }

    void work(int w)
    {
        char* buffers = pinned_ + kSlice * kBuffers * static_cast<size_t>(w);
        cudaEvent_t* events = events_ + kBuffers * w;
        struct Pending {
            char* to = nullptr;
            size_t bytes = 0;
        } pending[kBuffers];
        auto check = [this](cudaError_t e) {
            if (e != cudaSuccess) {
                error_ = static_cast<int>(e);
            }
            return e == cudaSuccess;
        };
        auto land = [&](int b) {
            if (pending[b].to != nullptr && check(cudaEventSynchronize(events[b]))) {
                std::memcpy(pending[b].to, buffers + kSlice * b, pending[b].bytes);
            }
            pending[b].to = nullptr;
        };
        int b = 0;
        for (; error_.load() == static_cast<int>(cudaSuccess); b = (b + 1) % kBuffers) {
            size_t i = next_.fetch_add(1);
            if (i >= slices_) {
                break;
            }
            size_t k = 0;
            for (; i >= (pieces_[k].bytes + kSlice - 1) / kSlice; ++k) {
                i -= (pieces_[k].bytes + kSlice - 1) / kSlice;
            }
            const size_t at = i * kSlice, bytes = std::min(kSlice, pieces_[k].bytes - at);
            char* device = static_cast<char*>(pieces_[k].device) + at;
            char* host = static_cast<char*>(pieces_[k].host) + at;
            char* buffer = buffers + kSlice * b;
            if (up_) {
                // (the buffer's last copy has run)
                if (!check(cudaEventSynchronize(events[b]))) {
                    break;
                }
                std::memcpy(buffer, host, bytes);
                check(cudaMemcpyAsync(device, buffer, bytes, cudaMemcpyHostToDevice, stream_));
            } else {
                land(b);
                if (!check(cudaEventSynchronize(events[b])) ||
                    !check(cudaMemcpyAsync(buffer, device, bytes, cudaMemcpyDeviceToHost, stream_))) {
                    break;
                }
                pending[b].to = host;
                pending[b].bytes = bytes;
            }
            check(cudaEventRecord(events[b], stream_));
        }
        for (int r = 0; r < kBuffers; ++r) {
            land((b + r) % kBuffers);
        }
        if (up_) {
            // (the next transfer, on another stream perhaps, finds the buffers free)
            for (int r = 0; r < kBuffers; ++r) {
                check(cudaEventSynchronize(events[r]));
            }
        }
    }

    const int device_;
    const pid_t process_ = getpid();
    int state_ = 0; // 0 not tried, 1 ready, -1 not available
    size_t plain_ = 0; // bytes copied plainly that could have been staged (up to kWorthBytes and a transfer)
    char* pinned_ = nullptr;
    cudaEvent_t events_[kBuffers * kWorkers] = {};
    std::vector<std::thread> threads_;
    std::mutex use_; // held by the transfer that the copier works on
    std::mutex mutex_;
    std::condition_variable wake_, done_;
    bool stop_ = false;
    unsigned long long turn_ = 0; // transfers started
    int busy_ = 0;                // workers that have not finished the current one
    // the current transfer
    std::vector<Piece> pieces_;
    cudaStream_t stream_ = nullptr;
    bool up_ = true;
    size_t slices_ = 0;
    std::atomic<size_t> next_{0};
    std::atomic<int> error_{0};
};

} // namespace pt
