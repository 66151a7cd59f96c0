#pragma once
// cudaMalloc-backed bucket pool: HBM buffers instead of the reference's host-visible VMA
// buffers (cpp/include/grilly/buffer_pool.h:18-113).  Same interface: acquire / release /
// upload / download / stats, power-of-two buckets from 256 B to 256 MiB with at most 32 cached
// buffers per bucket (cpp/src/buffer_pool.cpp:64-82,128-175); larger requests are exact-size.
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "grilly/device.h"

namespace grilly {

struct GrillyBuffer {
    void* dptr = nullptr;      // device pointer (HBM)
    size_t size = 0;           // requested bytes
    size_t bucketSize = 0;     // allocated bytes
    bool valid() const { return dptr != nullptr; }
};

struct PoolStats {
    uint64_t hits = 0, misses = 0, allocations = 0, totalAcquired = 0, totalReleased = 0;
};

class BufferPool {
public:
    explicit BufferPool(GrillyDevice& device);
    ~BufferPool();
    BufferPool(const BufferPool&) = delete;

    GrillyBuffer acquire(size_t size);
    void release(GrillyBuffer& buf);
    /// Host -> device copy through the context stream (asynchronous; ordered with launches).
    void upload(const GrillyBuffer& buf, const void* host, size_t bytes);
    /// Device -> host copy; returns after the data is in `host`.
    void download(const GrillyBuffer& buf, void* host, size_t bytes);
    PoolStats stats() const;
    GrillyDevice& device() { return device_; }

    static size_t bucketFor(size_t size);

private:
    GrillyDevice& device_;
    mutable std::mutex mu_;
    std::unordered_map<size_t, std::vector<void*>> free_;
    PoolStats stats_;
};

/// Host arrays of one small call in ONE transfer each way.  A transfer costs some 10 us of driver and link latency whatever its
/// size, which is most of a small call's time: the inputs are packed into one page-locked block, and the result leaves through
/// another.  Reused by the next call on the device, so a call waits for its work (CommandBatch::submit) before it ends.
/// An array of 512 KiB or more is left to the pageable copies (grl_memcpy_h2d / d2h), which take several threads from there on,
/// where packing takes one.  us a call, packed / apart: 4 x 256 x 64 attention (three inputs of 256 KiB) 100 / 102; linear 256 x 256 x 256
/// (inputs and result of 256 KiB) 79 / 86, 128 x 128 x 1000 (two arrays of 500 KiB) 92 / 95; but with one array of 512 KiB to 1 MiB
/// 100 x 256 x 512 82 / 72, 8 x 256 x 900 81 / 66, 256 x 128 x 512 82 / 74, 256 x 200 x 1000 185 / 106.
class SmallCall {
public:
    static constexpr size_t kMaxBytes = 1u << 20;      // inputs together
    static constexpr size_t kMaxArray = 512u << 10;    // each of them, and the result: below this
    static constexpr int kInSlot = 6, kOutSlot = 7;    // GrillyDevice::pinnedStaging
    static bool fits(size_t inputBytes, size_t largestArray) { return inputBytes <= kMaxBytes && largestArray < kMaxArray; }
    explicit SmallCall(BufferPool& pool);
    ~SmallCall();
    SmallCall(const SmallCall&) = delete;
    /// Packs `bytes` from `host`; returns where they will be on the device.  Every input adds up to 256 bytes of alignment.
    void* input(const void* host, size_t bytes);
    void send();                                       // after the last input
    void fetch(const void* device, size_t bytes);      // queue the result's transfer
    void deliver(void* host, size_t bytes) const;      // after CommandBatch::submit

private:
    BufferPool& pool_;
    GrillyBuffer in_;
    size_t used_ = 0;
};

}  // namespace grilly
