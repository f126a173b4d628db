// transfer.cu -- pinned slots and plain copies.
#include "transfer.h"

#include <condition_variable>
#include <cstring>
#include <mutex>
#include <vector>

namespace nadia {

namespace {
// Making and freeing pinned memory is refused to a thread (and breaks the
// capture) while another thread captures a graph in the global mode, unless
// this thread says that it does not take part.
struct NoCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    NoCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~NoCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr size_t kCellBytes = 64, kCellBlock = 64 << 10;

struct Pinned {
    std::mutex mu;
    size_t users = 0;
    int device = 0; // whose context the memory was made in
    // the slots, made together
    void *base = nullptr;
    std::vector<void *> free;
    std::condition_variable given;
    // the cells, cut from blocks
    std::vector<void *> blocks;
    std::vector<double *> free_cells;
    size_t cells = 0;

    void *make(size_t bytes) // with mu held
    {
        NoCapture guard;
        void *p = nullptr;
        NADIA_CUDA(cudaGetDevice(&device));
        NADIA_CUDA(cudaHostAlloc(&p, bytes, cudaHostAllocPortable | cudaHostAllocMapped));
        return p;
    }
};
void give_back();
// leaked on purpose: reconstructions destroyed by static destructors still use it
Pinned &pinned()
{
    static Pinned *p = [] {
        when_unused(give_back);
        return new Pinned;
    }();
    return *p;
}

// on a helper thread, some time after the last reconstruction
void give_back()
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    if (P.users > 0) return;
    NoCapture guard;
    if ((P.base || !P.blocks.empty()) && cudaSetDevice(P.device) != cudaSuccess) return;
    if (P.base && P.free.size() == (size_t)kSlots) {
        cudaFreeHost(P.base);
        P.base = nullptr;
        P.free.clear();
    }
    if (P.cells == 0) {
        for (void *b : P.blocks) cudaFreeHost(b);
        P.blocks.clear();
        P.free_cells.clear();
    }
}
} // namespace

PinnedSlots::User::User()
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    ++P.users;
}

PinnedSlots::User::~User()
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    --P.users;
}

void *PinnedSlots::take()
{
    Pinned &P = pinned();
    std::unique_lock<std::mutex> lk(P.mu);
    if (!P.base) {
        void *p = P.make(kSlots * kSlotBytes);
        P.base = p;
        for (int k = 0; k < kSlots; ++k) P.free.push_back((char *)p + k * kSlotBytes);
    }
    P.given.wait(lk, [&] { return !P.free.empty(); });
    void *p = P.free.back();
    P.free.pop_back();
    return p;
}

void PinnedSlots::give(void *p)
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    P.free.push_back(p);
    P.given.notify_one();
}

PinnedCell::PinnedCell()
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    if (P.free_cells.empty()) {
        void *b = P.make(kCellBlock);
        P.blocks.push_back(b);
        for (size_t at = 0; at < kCellBlock; at += kCellBytes)
            P.free_cells.push_back((double *)((char *)b + at));
    }
    p = P.free_cells.back();
    P.free_cells.pop_back();
    ++P.cells;
    *p = 0;
}

PinnedCell::~PinnedCell()
{
    Pinned &P = pinned();
    std::lock_guard<std::mutex> lk(P.mu);
    P.free_cells.push_back(p);
    --P.cells;
}

namespace {
constexpr size_t kRow = 64 << 10;      // plain copies are cut in "rows" of this size
constexpr size_t kSmallCopy = 2 << 20; // below: the driver's own staging (about 16 GB/s)
} // namespace

void await(cudaStream_t st, void *fill, size_t bytes)
{
    {
        NoCapture guard;
        const cudaError_t ready = cudaStreamQuery(st);
        if (ready == cudaSuccess) return; // no wait to hide anything behind
        if (ready == cudaErrorNotReady) (void)cudaGetLastError();
        else NADIA_CUDA(ready);
    }
    if (!fill) {
        NADIA_CUDA(cudaStreamSynchronize(st));
        return;
    }
    constexpr size_t kTouch = 64 << 10, kPage = 4096;
    std::atomic<size_t> next{0};
    std::atomic<bool> over{false};
    cudaError_t e = cudaSuccess;
    const std::thread::id caller = std::this_thread::get_id();
    with_helpers((int)std::min<size_t>(7, bytes / (4 * kTouch)), [&] {
        if (std::this_thread::get_id() == caller) {
            e = cudaStreamSynchronize(st);
            over = true;
            return;
        }
        for (size_t at; !over && (at = next.fetch_add(kTouch)) < bytes;)
            for (size_t k = at; k < std::min(bytes, at + kTouch); k += kPage) {
                volatile char *p = (char *)fill + k;
                *p = *p; // a write, so that the page becomes the array's own
            }
    });
    NADIA_CUDA(e);
}

void to_device(void *d, const void *h, size_t bytes, int device, cudaStream_t st)
{
    if (bytes < kSmallCopy) {
        NADIA_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st));
        NADIA_CUDA(cudaStreamSynchronize(st));
        return;
    }
    in_pieces(device, st, nullptr, 0, (bytes + kRow - 1) / kRow, kRow, [&](CopySlot &slot, size_t r,
                                                                   size_t rows) {
        const size_t at = r * kRow, len = std::min(rows * kRow, bytes - at);
        std::memcpy(slot.p, (const char *)h + at, len);
        NADIA_CUDA(cudaMemcpyAsync((char *)d + at, slot.p, len, cudaMemcpyHostToDevice, st));
        slot.wait(st);
    });
}

void to_host(void *h, const void *d, size_t bytes, int device, cudaStream_t st)
{
    if (bytes < kSmallCopy) {
        NADIA_CUDA(cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, st));
        NADIA_CUDA(cudaStreamSynchronize(st));
        return;
    }
    in_pieces(device, st, h, bytes, (bytes + kRow - 1) / kRow, kRow, [&](CopySlot &slot, size_t r,
                                                                 size_t rows) {
        const size_t at = r * kRow, len = std::min(rows * kRow, bytes - at);
        NADIA_CUDA(cudaMemcpyAsync(slot.p, (const char *)d + at, len, cudaMemcpyDeviceToHost, st));
        slot.wait(st);
        std::memcpy((char *)h + at, slot.p, len);
    });
}

} // namespace nadia
