// Host side of the linear projection: upload -> (cast) -> one kernel -> download.
#include <algorithm>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "grilly/ops/linear.h"

namespace grilly {
namespace ops {

namespace {
// Results from 2.5 MiB up leave in four pieces of whole 64-row tiles.  us a call in one piece / four (K = 768): result of 2 MiB 235 / 260,
// 2.5 MiB 288 / 286, 3.5 MiB 336 / 318, 6 MiB 486 / 453, 16 MiB 935 / 835.  Two pieces: 477 and 870 for the last two; eight: 532 and 820,
// and from 32 to 64 MiB within 3 % of four.
constexpr size_t kPieceBytes = 5u << 19, kPieceRows = 64;
}

void linearEx(CommandBatch& batch, BufferPool& pool, PipelineCache& cache, const float* x, const float* weights,
              const float* bias, float* output, const LinearParams& p, Precision precision) {
    if (!x || !weights || !output) throw std::runtime_error("linear: null tensor pointer");
    if (p.batchSeq == 0 || p.inputDim == 0 || p.outputDim == 0) throw std::runtime_error("linear: empty shape");
    const bool bf16 = precision == Precision::BF16;
    if (bf16 && p.inputDim % 8 != 0) throw std::runtime_error("linear: the bf16 path needs input_dim to be a multiple of 8");
    grl_device* dev = pool.device().handle();
    cache.getOrCreate(std::string(bf16 ? "fnn-linear-tcgen05/" : "fnn-linear/") + std::to_string(p.inputDim));
    const size_t nx = size_t(p.batchSeq) * p.inputDim, nw = size_t(p.outputDim) * p.inputDim, ny = size_t(p.batchSeq) * p.outputDim;
    const bool small = SmallCall::fits((nx + nw + p.outputDim) * 4, std::max({nx, nw, ny}) * 4);
    GrillyBuffer xb, wb, yb = pool.acquire(ny * 4), bb, x16, w16;
    std::vector<grl_event*> events;
    auto releaseAll = [&]() {
        pool.release(xb); pool.release(wb); pool.release(yb); pool.release(bb); pool.release(x16); pool.release(w16);
        for (auto* e : events) grl_event_destroy(e);
    };
    try {
        batch.begin();
        std::optional<SmallCall> block;
        if (small) block.emplace(pool);
        // an input array on the device: packed with the others, or in a buffer of its own
        auto place = [&](GrillyBuffer& buf, const float* host, size_t n) -> const void* {
            if (small) return block->input(host, n * 4);
            buf = pool.acquire(n * 4);
            pool.upload(buf, host, n * 4);
            return buf.dptr;
        };
        const void* xd = place(xb, x, nx);
        const void* wd = place(wb, weights, nw);
        const float* biasDev = p.hasBias && bias ? static_cast<const float*>(place(bb, bias, p.outputDim)) : nullptr;
        if (small) block->send();
        if (bf16) {
            x16 = pool.acquire(nx * 2);
            w16 = pool.acquire(nw * 2);
            check(grl_cast(dev, xd, GRL_F32, x16.dptr, GRL_BF16, nx), "linear: cast");
            check(grl_cast(dev, wd, GRL_F32, w16.dptr, GRL_BF16, nw), "linear: cast");
            xd = x16.dptr;
            wd = w16.dptr;
        }
        // A large result leaves in pieces of rows: the transfer of one piece, which bounds the time, runs beside the product of
        // the next ones.
        const size_t pieces = ny * 4 >= kPieceBytes && p.batchSeq >= 4 * kPieceRows ? 4 : 1;
        const size_t per = (p.batchSeq / pieces + kPieceRows - 1) / kPieceRows * kPieceRows;
        const size_t esz = bf16 ? 2 : 4;
        for (size_t r = 0; r < p.batchSeq; r += per) {
            const size_t rows = std::min(per, size_t(p.batchSeq) - r);
            check(grl_linear(dev, static_cast<const char*>(xd) + r * p.inputDim * esz, wd, biasDev,
                             static_cast<float*>(yb.dptr) + r * p.outputDim, int(rows), int(p.inputDim), int(p.outputDim),
                             bf16 ? GRL_BF16 : GRL_F32), "linear");
            if (pieces > 1) {
                events.push_back(nullptr);
                check(grl_event_create_untimed(&events.back()), "linear: event");
                check(grl_event_record(dev, events.back()), "linear: event");
            }
        }
        if (small) {
            block->fetch(yb.dptr, ny * 4);
        } else if (pieces > 1) {
            grl_device* down = pool.device().downloadQueue();
            check(grl_memcpy_d2h_parts(down, output, yb.dptr, ny * 4, events.data(), int(events.size()), per * p.outputDim * 4),
                  "linear: download");
            events.push_back(nullptr);          // a page-locked output array is still being written: the wait below is for it too
            check(grl_event_create_untimed(&events.back()), "linear: event");
            check(grl_event_record(down, events.back()), "linear: event");
            check(grl_event_wait(dev, events.back()), "linear: event");
        } else {
            check(grl_memcpy_d2h(dev, output, yb.dptr, ny * 4), "linear: download");
        }
        batch.submit();
        if (small) block->deliver(output, ny * 4);
    } catch (...) {
        if (batch.recording()) batch.submitNoWait();
        pool.device().quiesce();   // nothing in flight may still touch the buffers released below
        releaseAll();
        throw;
    }
    releaseAll();
}

void linear(CommandBatch& batch, BufferPool& pool, PipelineCache& cache, const float* x, const float* weights,
            const float* bias, float* output, const LinearParams& p) {
    linearEx(batch, pool, cache, x, weights, bias, output, p, Precision::FP32);
}

void fusedQKVProjection(CommandBatch& batch, BufferPool& pool, PipelineCache& cache, const float* x, const float* wQKV,
                        const float* bQKV, float* output, uint32_t batchSeq, uint32_t hiddenDim, uint32_t numHeads,
                        uint32_t headDim, Precision precision) {
    LinearParams p{batchSeq, hiddenDim, 3 * numHeads * headDim, bQKV ? 1u : 0u};
    linearEx(batch, pool, cache, x, wQKV, bQKV, output, p, precision);
}

}  // namespace ops
}  // namespace grilly
