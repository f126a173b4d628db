// transfer.cu -- pinned slots and plain copies.
#include "transfer.h"

#include <condition_variable>
#include <cstring>
#include <vector>

namespace nadia {

namespace {
// leaked on purpose: reconstructions destroyed by static destructors still use them
std::mutex &slot_mu()
{
    static std::mutex *m = new std::mutex;
    return *m;
}
struct Arena {
    void *base = nullptr;
    std::vector<void *> free;
    std::condition_variable given;
    void release() // with slot_mu held; only when every slot is back
    {
        if (!base || free.size() < (size_t)kSlots) return;
        cudaFreeHost(base);
        base = nullptr;
        free.clear();
    }
};
Arena &arena()
{
    static Arena *a = new Arena;
    return *a;
}
size_t g_users = 0;
} // namespace

PinnedSlots::User::User()
{
    std::lock_guard<std::mutex> lk(slot_mu());
    ++g_users;
}

PinnedSlots::User::~User()
{
    std::lock_guard<std::mutex> lk(slot_mu());
    if (--g_users > 0) return;
    arena().release();
}

void *PinnedSlots::take()
{
    std::unique_lock<std::mutex> lk(slot_mu());
    Arena &A = arena();
    if (!A.base) {
        void *p = nullptr;
        NADIA_CUDA(cudaHostAlloc(&p, kSlots * kSlotBytes, cudaHostAllocPortable));
        A.base = p;
        for (int k = 0; k < kSlots; ++k) A.free.push_back((char *)p + k * kSlotBytes);
    }
    A.given.wait(lk, [&] { return !A.free.empty(); });
    void *p = A.free.back();
    A.free.pop_back();
    return p;
}

void PinnedSlots::give(void *p)
{
    std::lock_guard<std::mutex> lk(slot_mu());
    Arena &A = arena();
    A.free.push_back(p);
    A.given.notify_one();
    if (g_users == 0) A.release();
}

namespace {
// cells are cut from one slot; it is given back with the slots
std::vector<double *> &free_cells()
{
    static std::vector<double *> *v = new std::vector<double *>;
    return *v;
}
std::vector<void *> &cell_slots()
{
    static std::vector<void *> *v = new std::vector<void *>;
    return *v;
}
constexpr size_t kCellBytes = 64;
size_t g_cells = 0;
} // namespace

PinnedCell::PinnedCell()
{
    std::lock_guard<std::mutex> lk(slot_mu());
    if (free_cells().empty()) {
        void *s = nullptr;
        NADIA_CUDA(cudaHostAlloc(&s, 64 << 10, cudaHostAllocPortable | cudaHostAllocMapped));
        cell_slots().push_back(s);
        for (size_t at = 0; at < (64 << 10); at += kCellBytes)
            free_cells().push_back((double *)((char *)s + at));
    }
    p = free_cells().back();
    free_cells().pop_back();
    ++g_cells;
    *p = 0;
}

PinnedCell::~PinnedCell()
{
    std::lock_guard<std::mutex> lk(slot_mu());
    free_cells().push_back(p);
    if (--g_cells > 0) return;
    free_cells().clear();
    for (void *s : cell_slots()) cudaFreeHost(s);
    cell_slots().clear();
}

namespace {
constexpr size_t kRow = 64 << 10;      // plain copies are cut in "rows" of this size
constexpr size_t kSmallCopy = 2 << 20; // below: the driver's own staging (about 16 GB/s)
} // namespace

void to_device(void *d, const void *h, size_t bytes, int device, cudaStream_t st)
{
    if (bytes < kSmallCopy) {
        NADIA_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st));
        NADIA_CUDA(cudaStreamSynchronize(st));
        return;
    }
    in_pieces(device, st, (bytes + kRow - 1) / kRow, kRow, [&](CopySlot &slot, size_t r, size_t rows) {
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
    in_pieces(device, st, (bytes + kRow - 1) / kRow, kRow, [&](CopySlot &slot, size_t r, size_t rows) {
        const size_t at = r * kRow, len = std::min(rows * kRow, bytes - at);
        NADIA_CUDA(cudaMemcpyAsync(slot.p, (const char *)d + at, len, cudaMemcpyDeviceToHost, st));
        slot.wait(st);
        std::memcpy((char *)h + at, slot.p, len);
    });
}

} // namespace nadia
