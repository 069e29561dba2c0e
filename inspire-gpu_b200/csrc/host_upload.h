// host_upload.h -- host-to-device copies of large pageable buffers.
//
// The driver stages a pageable copy through one thread (about 10 GB/s), which
// was most of preprocessing: a 1 GB database took 123 ms, 14 of them kernels.
// Here several threads fill pinned slots and enqueue the copies, so the upload
// runs nearer the PCIe rate (four threads: 60 ms for that database; two 79,
// eight 68).  Buffers that are already pinned (or not host memory) are copied
// directly, and so are those below 128 MB (64 MB: 30 ms of preprocessing either
// way).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "server_internal.h"

namespace ipb {

class HostUpload {
  public:
    // For copies out of the `bytes` bytes at src to the current device.
    HostUpload(const void* src, size_t bytes) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, src) != cudaSuccess) {
            cudaGetLastError();  // not a pointer CUDA knows: pageable
            a.type = cudaMemoryTypeUnregistered;
        }
        if (a.type != cudaMemoryTypeUnregistered || bytes < kMinBytes) return;
        if (cudaGetDevice(&device_) != cudaSuccess) return;
        const size_t n = std::max(1u, std::min(4u, std::thread::hardware_concurrency() / 2));
        pinned_ = std::make_unique<PinnedPages>(n * 2 * kSlot);
        if (!pinned_->p) return;
        try {
            workers_.reserve(n);
            for (size_t i = 0; i < n; ++i) workers_.emplace_back([this, i] { work(i); });
        } catch (const std::system_error&) {  // no more threads: go on with those there are
        }
    }
    ~HostUpload() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();  // each waits for its own copies
    }
    HostUpload(const HostUpload&) = delete;
    HostUpload& operator=(const HostUpload&) = delete;

    // Enqueues the copy on s.  src may change only once s has passed it when it
    // is copied directly, at once otherwise.
    void copy(void* dst, const void* src, size_t bytes, cudaStream_t s) {
        if (workers_.empty()) {
            IPB_CK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
            return;
        }
        std::unique_lock<std::mutex> lk(mu_);
        dst_ = static_cast<uint8_t*>(dst);
        src_ = static_cast<const uint8_t*>(src);
        bytes_ = bytes;
        stream_ = s;
        next_ = 0;
        slots_ = left_ = (bytes + kSlot - 1) / kSlot;
        cv_.notify_all();
        done_.wait(lk, [&] { return left_ == 0; });
        if (err_ != cudaSuccess) cuda_fail(err_, "upload", __FILE__, __LINE__);
    }

  private:
    static constexpr size_t kSlot = (size_t)1 << 20;
    static constexpr size_t kMinBytes = (size_t)128 << 20;

    void work(size_t id) {
        cudaEvent_t ev[2] = {nullptr, nullptr};
        cudaError_t e = cudaSetDevice(device_);
        for (auto& x : ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        int k = 0;
        std::unique_lock<std::mutex> lk(mu_);
        for (;;) {
            cv_.wait(lk, [&] { return stop_ || next_ < slots_; });
            if (next_ >= slots_) break;
            const size_t off = next_++ * kSlot, n = std::min(kSlot, bytes_ - off);
            uint8_t* const dst = dst_ + off;
            const uint8_t* const src = src_ + off;
            const cudaStream_t s = stream_;
            lk.unlock();
            uint8_t* const buf = pinned_->p + (2 * id + k) * kSlot;
            if (e == cudaSuccess) e = cudaEventSynchronize(ev[k]);  // this slot's last copy has left it
            if (e == cudaSuccess) {
                std::memcpy(buf, src, n);
                e = cudaMemcpyAsync(dst, buf, n, cudaMemcpyHostToDevice, s);
            }
            if (e == cudaSuccess) e = cudaEventRecord(ev[k], s);
            k ^= 1;
            lk.lock();
            if (e != cudaSuccess && err_ == cudaSuccess) err_ = e;
            if (--left_ == 0) done_.notify_all();
        }
        lk.unlock();
        for (auto& x : ev)
            if (x) {
                cudaEventSynchronize(x);
                cudaEventDestroy(x);
            }
    }

    int device_ = 0;
    std::unique_ptr<PinnedPages> pinned_;
    std::vector<std::thread> workers_;
    std::mutex mu_;
    std::condition_variable cv_, done_;
    bool stop_ = false;
    uint8_t* dst_ = nullptr;
    const uint8_t* src_ = nullptr;
    size_t bytes_ = 0, next_ = 0, slots_ = 0, left_ = 0;
    cudaStream_t stream_ = nullptr;
    cudaError_t err_ = cudaSuccess;
};

}  // namespace ipb
