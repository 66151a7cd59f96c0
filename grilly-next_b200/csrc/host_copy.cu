// See host_copy.cuh.
#include <immintrin.h>
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"

namespace grl {

namespace {
constexpr size_t kParallelBytes = 512u << 10;   // below this one thread copies faster than the others wake up
constexpr int kSpin = 20000;                    // pauses (some 50 us) a worker looks for the next piece before it sleeps

void copy_range(char* dst, const char* src, size_t n, bool stream) {
    if (!stream || ((uintptr_t)dst & 15)) {
        memcpy(dst, src, n);
        return;
    }
    size_t i = 0;
    for (; i + 64 <= n; i += 64) {
        const __m128i* s = reinterpret_cast<const __m128i*>(src + i);
        __m128i* d = reinterpret_cast<__m128i*>(dst + i);
        const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
        _mm_stream_si128(d, a);
        _mm_stream_si128(d + 1, b);
        _mm_stream_si128(d + 2, c);
        _mm_stream_si128(d + 3, e);
    }
    memcpy(dst + i, src + i, n - i);
    _mm_sfence();
}
}  // namespace

CopyPool& CopyPool::instance() {
    static CopyPool pool;
    return pool;
}

CopyPool::CopyPool() {
    int n = (int)std::thread::hardware_concurrency() / 2;
    if (const char* e = getenv("LOCAL_WORLD_SIZE")) n /= std::max(1, atoi(e));      // one process per GPU: they share the cores
    if (const char* e = getenv("GRILLY_HOST_THREADS")) n = atoi(e);
    parts_ = std::min(8, std::max(1, n));
    for (int i = 1; i < parts_; ++i) threads_.emplace_back([this, i] { loop(i); });
}

CopyPool::~CopyPool() {
    {
        std::lock_guard<std::mutex> lock(mu_);
        stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) t.join();
}

void CopyPool::share(int id) const {
    const size_t per = (bytes_ / parts_ + 4095) & ~(size_t)4095;
    const size_t lo = std::min(bytes_, per * (size_t)id), hi = id + 1 == parts_ ? bytes_ : std::min(bytes_, lo + per);
    if (hi > lo) copy_range(dst_ + lo, src_ + lo, hi - lo, stream_);
}

void CopyPool::loop(int id) {
    uint32_t seen = 0;
    for (;;) {
        for (int i = 0; i < kSpin && generation_.load(std::memory_order_acquire) == seen && !stop_; ++i) _mm_pause();
        if (generation_.load(std::memory_order_acquire) == seen) {
            std::unique_lock<std::mutex> lock(mu_);
            ++sleeping_;
            wake_.wait(lock, [&] { return stop_ || generation_.load(std::memory_order_acquire) != seen; });
            --sleeping_;
        }
        if (stop_) return;
        ++seen;                 // the caller waits for every worker: a generation is never skipped
        share(id);
        pending_.fetch_sub(1, std::memory_order_release);
    }
}

void CopyPool::copy(void* dst, const void* src, size_t bytes, bool stream) {
    if (bytes < kParallelBytes || parts_ == 1 || !caller_.try_lock()) {
        copy_range((char*)dst, (const char*)src, bytes, stream);
        return;
    }
    std::lock_guard<std::mutex> call(caller_, std::adopt_lock);
    dst_ = (char*)dst;
    src_ = (const char*)src;
    bytes_ = bytes;
    stream_ = stream;
    pending_.store(parts_ - 1, std::memory_order_relaxed);
    bool any;
    {
        std::lock_guard<std::mutex> lock(mu_);
        generation_.fetch_add(1, std::memory_order_release);
        any = sleeping_ > 0;
    }
    if (any) wake_.notify_all();
    share(0);
    for (int i = 0; pending_.load(std::memory_order_acquire) > 0; ++i) {
        if (i < kSpin) _mm_pause();
        else std::this_thread::yield();
    }
}

HostStage::~HostStage() {
    for (Ring* r : {&up, &down}) {
        for (cudaEvent_t e : r->ev)
            if (e) cudaEventDestroy(e);
        if (r->mem) cudaFreeHost(r->mem);
    }
}

static cudaError_t open_ring(HostStage::Ring& r) {
    if (r.mem) return cudaSuccess;
    for (cudaEvent_t& e : r.ev)
        if (!e) {
            const cudaError_t rc = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
            if (rc != cudaSuccess) return rc;
        }
    return cudaMallocHost(&r.mem, HostStage::kPiece * HostStage::kSlots);
}

// The next slot of the ring, once the transfer that used it last has completed.
static cudaError_t take_slot(HostStage::Ring& r, int* slot) {
    *slot = r.next;
    r.next = (r.next + 1) % HostStage::kSlots;
    if (!r.busy[*slot]) return cudaSuccess;
    r.busy[*slot] = false;
    return cudaEventSynchronize(r.ev[*slot]);
}

cudaError_t staged_upload(grl_device* dev, void* dst, const void* src, size_t bytes) {
    HostStage& st = dev->stage;
    std::lock_guard<std::mutex> lock(st.up.mu);
    cudaError_t rc = open_ring(st.up);
    for (size_t off = 0, n = 0; off < bytes && rc == cudaSuccess; off += n) {
        n = std::min(off == 0 ? HostStage::kShort : HostStage::kPiece, bytes - off);
        int slot;
        rc = take_slot(st.up, &slot);
        if (rc != cudaSuccess) break;
        char* piece = st.up.mem + (size_t)slot * HostStage::kPiece;
        CopyPool::instance().copy(piece, (const char*)src + off, n, true);
        rc = cudaMemcpyAsync((char*)dst + off, piece, n, cudaMemcpyHostToDevice, dev->stream);
        if (rc == cudaSuccess) rc = cudaEventRecord(st.up.ev[slot], dev->stream);
        st.up.busy[slot] = rc == cudaSuccess;
    }
    return rc;
}

cudaError_t staged_download(grl_device* dev, void* dst, const void* src, size_t bytes, const cudaEvent_t* parts, int n_parts,
                            size_t part_bytes) {
    HostStage& st = dev->stage;
    std::lock_guard<std::mutex> lock(st.down.mu);
    cudaError_t rc = open_ring(st.down);
    // every slot is free between calls: a download leaves none in flight
    auto piece = [&](size_t off) {
        const size_t left = bytes - off, n = left <= HostStage::kShort ? left : std::min(HostStage::kPiece, left - HostStage::kShort);
        return n_parts ? std::min(n, (off / part_bytes + 1) * part_bytes - off) : n;
    };
    size_t issued = 0, done = 0;
    int waited = 0;
    for (int in = 0, out = 0; done < bytes && rc == cudaSuccess; ++out) {
        for (; issued < bytes && in - out < HostStage::kSlots && rc == cudaSuccess; ++in) {
            const size_t n = piece(issued);
            const int slot = in % HostStage::kSlots;
            for (; waited < n_parts && (size_t)waited * part_bytes < issued + n && rc == cudaSuccess; ++waited)
                rc = cudaStreamWaitEvent(dev->stream, parts[waited], 0);
            if (rc != cudaSuccess) break;
            rc = cudaMemcpyAsync(st.down.mem + (size_t)slot * HostStage::kPiece, (const char*)src + issued, n, cudaMemcpyDeviceToHost, dev->stream);
            if (rc == cudaSuccess && issued + n == bytes) queue_status_copy(dev);     // one wait serves the caller's grl_sync too
            if (rc == cudaSuccess) rc = cudaEventRecord(st.down.ev[slot], dev->stream);
            issued += n;
        }
        if (rc != cudaSuccess) break;
        const size_t n = piece(done);
        const int slot = out % HostStage::kSlots;
        rc = cudaEventSynchronize(st.down.ev[slot]);
        if (rc == cudaSuccess) CopyPool::instance().copy((char*)dst + done, st.down.mem + (size_t)slot * HostStage::kPiece, n, false);
        done += n;
    }
    if (rc != cudaSuccess) cudaStreamSynchronize(dev->stream);     // transfers already queued still write to the ring
    return rc;
}

}  // namespace grl
