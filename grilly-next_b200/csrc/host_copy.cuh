// Copies between pageable host memory and the device through page-locked staging.
//
// cudaMemcpyAsync on pageable memory copies on the calling thread alone: measured (16-core host, PCIe 5) 1 MiB up 82 us and down
// 92 us, 9 MiB 0.5 ms either way, where the link needs 20 and 172 us and a host memcpy of 9 MiB takes 546 us on one thread and 60
// on eight.  So pageable copies go through a ring of page-locked pieces: large pieces are copied by a few threads, and the copy
// of one piece runs beside the transfer of the one before.  Uploads below 512 KiB stay with the driver, which is as fast there.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

struct grl_device;

namespace grl {

// Threads that copy a piece together.  One caller at a time; another one meanwhile copies on its own thread.
class CopyPool {
public:
    static CopyPool& instance();
    // stream: leave the caches alone on the way out (the destination is read by the copy engine next: its reads of lines that
    // sit modified in a core's cache are slow; 9 MiB up 350 us with plain stores, 241 with these)
    void copy(void* dst, const void* src, size_t bytes, bool stream);

private:
    CopyPool();
    ~CopyPool();
    void loop(int id);
    void share(int id) const;
    std::vector<std::thread> threads_;
    std::mutex caller_, mu_;
    std::condition_variable wake_;
    std::atomic<uint32_t> generation_{0};
    std::atomic<int> pending_{0}, sleeping_{0};
    std::atomic<bool> stop_{false};
    int parts_ = 1;
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t bytes_ = 0;
    bool stream_ = false;
};

// The page-locked rings of one device handle: allocated on first use, given back when the handle is closed.  Each has a lock of its
// own, held for a whole copy: a download that waits for the kernels before it does not keep another thread's upload waiting.
struct HostStage {
    static constexpr size_t kPiece = 2u << 20, kShort = 512u << 10;    // the end of a copy that no transfer hides is short
    static constexpr int kSlots = 4;
    struct Ring {
        std::mutex mu;
        char* mem = nullptr;
        cudaEvent_t ev[kSlots] = {};
        bool busy[kSlots] = {};
        int next = 0;
    };
    Ring up, down;
    ~HostStage();
};

// Stream-ordered copies with the semantics of cudaMemcpyAsync on pageable memory: `src` may be reused when the upload returns,
// `dst` is complete when the download returns.
cudaError_t staged_upload(grl_device* dev, void* dst, const void* src, size_t bytes);
// parts: bytes [i * part_bytes, (i + 1) * part_bytes) wait for event i (n_parts 0: for nothing but the stream).
cudaError_t staged_download(grl_device* dev, void* dst, const void* src, size_t bytes, const cudaEvent_t* parts = nullptr, int n_parts = 0,
                            size_t part_bytes = 0);

}  // namespace grl
