// Copies between ordinary (pageable) host arrays and the device, by several host threads.
//
// cudaMemcpyAsync on pageable memory stages through the driver on the calling thread: 9 GB/s measured, against 55 GB/s
// of the link and the 41 to 53 GB/s a product on pinned arrays moves. Here the arrays are cut into pieces of 1 MB; each
// worker takes the next piece, copies it into one of its own two pinned buffers and queues the transfer itself, so the
// host copies of eight pieces and the transfers of earlier ones overlap and no thread waits for another one's piece.
//
// The caller publishes segments in order; a segment is done when all of its pieces are queued on (or, device to host,
// have left) its stream. Workers live for one call: nothing runs between calls, no descriptor is inherited by a fork.
// The pinned buffers (16 MB) are kept with the device's pool under the pool's lock. A worker that cannot be started, and
// a piece whose transfer fails, is reported by finish(); fewer workers than asked for do the same work.
//
// Nobody spins for long: a worker without a segment, and the caller that waits for one, sleep on a condition variable after
// HC_SPIN_US, and the workers of a device-to-host segment sleep on an event of the work before it (a product may run for
// much longer than its copies). Only the wait for a piece's own transfer is the driver's usual one.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

namespace b200i {

constexpr size_t HC_PIECE = 1u << 20;
constexpr int HC_WORKERS = 8, HC_SEGMENTS = 24, HC_SPIN_US = 2000;

struct HostStage { // per device, kept: two pinned pieces and their events per worker, and an event per segment to sleep on
    unsigned char *pinned = nullptr;
    cudaEvent_t ev[2 * HC_WORKERS] = {}, before[HC_SEGMENTS] = {};
    bool ready = false;
};

inline cudaError_t host_stage_prepare(HostStage &s) {
    if (s.ready) return cudaSuccess;
    cudaError_t e;
    if (!s.pinned && (e = cudaHostAlloc(reinterpret_cast<void **>(&s.pinned), 2 * HC_WORKERS * HC_PIECE, cudaHostAllocDefault)) != cudaSuccess) {
        s.pinned = nullptr;
        return e;
    }
    for (auto &x : s.ev)
        if (!x && (e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming)) != cudaSuccess) return e;
    for (auto &x : s.before)
        if (!x && (e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming | cudaEventBlockingSync)) != cudaSuccess) return e;
    s.ready = true;
    return cudaSuccess;
}

inline bool host_is_pageable(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

class HostCopier {
  public:
    HostCopier(HostStage &stage, int dev, size_t total_bytes) : stage_(stage), dev_(dev) {
        int want = (int)std::thread::hardware_concurrency() / 2;
        if (want > HC_WORKERS) want = HC_WORKERS;
        const size_t useful = (total_bytes + HC_PIECE - 1) / HC_PIECE;
        if ((size_t)want > useful) want = (int)useful;
        if (want < 1) want = 1;
        for (int i = 0; i < want; i++) {
            try {
                workers_[i] = std::thread(&HostCopier::work, this, i);
                started_++;
            } catch (...) { // no thread, no memory for one: the workers there are do the work; nothing leaves a C entry
                break;
            }
        }
        if (started_ == 0) failed_.store((int)cudaErrorOperatingSystem);
    }
    ~HostCopier() { finish(); }
    HostCopier(const HostCopier &) = delete;
    HostCopier &operator=(const HostCopier &) = delete;

    bool ok() const { return started_ > 0; }
    // host rows of `width` bytes, `pitch` bytes apart, dense on the device
    int add(bool to_device, void *device, void *host, size_t width, size_t pitch, size_t rows, cudaStream_t st) {
        const int i = published_.load(std::memory_order_relaxed);
        if (i >= HC_SEGMENTS) { // never more than the caller's chunks; refused rather than overrun
            fail(cudaErrorInvalidValue);
            return -1;
        }
        Segment &s = seg_[i];
        if (pitch == width) { // one long row
            width *= rows;
            rows = 1;
        }
        s.to_device = to_device;
        s.device = static_cast<unsigned char *>(device);
        s.host = static_cast<unsigned char *>(host);
        s.width = width;
        s.pitch = pitch;
        s.rows = rows;
        s.rows_per_piece = rows == 1 ? 1 : (width >= HC_PIECE ? 1 : HC_PIECE / width);
        s.cuts = rows == 1 || width > HC_PIECE ? (width + HC_PIECE - 1) / HC_PIECE : 1; // pieces of one row
        s.pieces = s.cuts > 1 ? s.cuts * rows : (rows + s.rows_per_piece - 1) / s.rows_per_piece;
        s.stream = st;
        s.next.store(0);
        s.done.store(0);
        if (!to_device) { // what the stream holds now, the product among it, comes before this segment
            const cudaError_t e = cudaEventRecord(stage_.before[i], st);
            if (e != cudaSuccess) {
                fail(e);
                return -1;
            }
        }
        published_.store(i + 1, std::memory_order_release);
        wake(more_);
        return i;
    }
    void wait(int i) { // all pieces of segment i are queued (to the device) or home (from it)
        if (i < 0) return;
        sleep_until(whole_, [&] { return seg_[i].done.load(std::memory_order_acquire) >= seg_[i].pieces || failed_.load() != 0; });
    }
    cudaError_t finish() {
        closed_.store(true, std::memory_order_release);
        wake(more_);
        for (int i = 0; i < started_; i++)
            if (workers_[i].joinable()) workers_[i].join();
        return (cudaError_t)failed_.load();
    }

  private:
    void wake(std::condition_variable &cv) { // after the change itself: a sleeper that missed it holds the mutex until it sleeps
        { std::lock_guard<std::mutex> lock(mu_); }
        cv.notify_all();
    }
    void fail(cudaError_t e) {
        failed_.store((int)e);
        wake(more_);
        wake(whole_);
    }
    template <class Ready>
    void sleep_until(std::condition_variable &cv, Ready ready) {
        const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(HC_SPIN_US);
        while (!ready()) {
            if (std::chrono::steady_clock::now() >= until) {
                std::unique_lock<std::mutex> lock(mu_);
                cv.wait(lock, ready);
                return;
            }
            std::this_thread::yield();
        }
    }
    struct Segment {
        bool to_device;
        unsigned char *device, *host;
        size_t width, pitch, rows, rows_per_piece, cuts, pieces;
        cudaStream_t stream;
        std::atomic<size_t> next{0}, done{0};
    };
    static cudaError_t past(cudaEvent_t ev) { // the work before the event is over
        const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(HC_SPIN_US);
        for (;;) {
            const cudaError_t e = cudaEventQuery(ev);
            if (e != cudaErrorNotReady) return e;
            if (std::chrono::steady_clock::now() >= until) return cudaEventSynchronize(ev);
            std::this_thread::yield();
        }
    }
    void piece(Segment &s, size_t i, int slot) {
        unsigned char *buf = stage_.pinned + (size_t)slot * HC_PIECE;
        cudaEvent_t ev = stage_.ev[slot];
        size_t row0, count, off = 0, len = s.width;
        if (s.cuts > 1) {
            row0 = i / s.cuts;
            count = 1;
            off = (i % s.cuts) * HC_PIECE;
            len = s.width - off < HC_PIECE ? s.width - off : HC_PIECE;
        } else {
            row0 = i * s.rows_per_piece;
            count = s.rows - row0 < s.rows_per_piece ? s.rows - row0 : s.rows_per_piece;
        }
        unsigned char *dp = s.device + row0 * s.width + off, *hp = s.host + row0 * s.pitch + off;
        cudaError_t e = cudaEventSynchronize(ev); // the slot's transfer before this one
        if (e == cudaSuccess && s.to_device) {
            for (size_t r = 0; r < count; r++) std::memcpy(buf + r * len, hp + r * s.pitch, len);
            e = cudaMemcpyAsync(dp, buf, count * len, cudaMemcpyHostToDevice, s.stream);
            if (e == cudaSuccess) e = cudaEventRecord(ev, s.stream);
        } else if (e == cudaSuccess) {
            e = cudaMemcpyAsync(buf, dp, count * len, cudaMemcpyDeviceToHost, s.stream);
            if (e == cudaSuccess) e = cudaEventRecord(ev, s.stream);
            if (e == cudaSuccess) e = past(stage_.before[&s - seg_]); // the transfer is queued, and sleeps behind the product
            if (e == cudaSuccess) e = cudaEventSynchronize(ev);
            if (e == cudaSuccess)
                for (size_t r = 0; r < count; r++) std::memcpy(hp + r * s.pitch, buf + r * len, len);
        }
        if (e != cudaSuccess) fail(e);
    }
    void work(int id) {
        cudaError_t e = cudaSetDevice(dev_);
        if (e != cudaSuccess) {
            fail(e);
            return;
        }
        int turn = 0;
        for (int i = 0;;) {
            if (failed_.load() != 0) return;
            if (i >= published_.load(std::memory_order_acquire)) {
                if (closed_.load(std::memory_order_acquire) && i >= published_.load(std::memory_order_acquire)) return;
                sleep_until(more_, [&] { return i < published_.load(std::memory_order_acquire) || closed_.load(std::memory_order_acquire) || failed_.load() != 0; });
                continue;
            }
            Segment &s = seg_[i];
            const size_t p = s.next.fetch_add(1);
            if (p >= s.pieces) {
                i++;
                continue;
            }
            piece(s, p, 2 * id + (turn ^= 1));
            if (s.done.fetch_add(1, std::memory_order_acq_rel) + 1 == s.pieces) wake(whole_);
        }
    }
    HostStage &stage_;
    int dev_, started_ = 0;
    std::thread workers_[HC_WORKERS];
    Segment seg_[HC_SEGMENTS];
    std::mutex mu_;
    std::condition_variable more_, whole_; // segments to take; a segment done
    std::atomic<int> published_{0}, failed_{0};
    std::atomic<bool> closed_{false};
};

} // namespace b200i
