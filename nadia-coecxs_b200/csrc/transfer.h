// transfer.h -- arrays between host memory and the device.
//
// A caller's arrays are pageable: a copy straight from or to them runs through
// the driver's single staging thread, and a freshly allocated result is
// page-faulted in by that same thread (a 2048^2 complex128 estimate: 14.3 ms,
// 4.7 GB/s on B200 over a link that carries ten times that).  Here an array is
// cut into pieces of whole rows; several threads take piece after piece, each
// through a pinned slot of its own, so one piece's conversion and page faults
// run beside the others' transfers.
#pragma once

#include <algorithm>
#include <exception>
#include <mutex>
#include <thread>

#include "common.h"
#include "helpers.h"

namespace nadia {

constexpr size_t kSlotBytes = 2u << 20; // one pinned slot
constexpr int kSlots = 16;

// Pinned slots of the process, made together at the first transfer; a thread
// that finds none free waits for one.  (Making or freeing pinned memory waits for
// the whole device: with slots made as they ran short, 16 threads reading
// estimates beside a running batch waited for its end.)  They are given back a
// while after the last reconstruction (helpers.h), because making them takes
// longer than a small reconstruction: B200, one 645x475 FP64 or 512^2 FP32
// reconstruction after the other, made, set, stepped once, read and dropped:
// 29 and 38 ms with slots and cells given back with each, 4.7 and 4.9 ms kept.
class PinnedSlots {
public:
    // held by every reconstruction
    struct User {
        HelperUse helpers;
        User();
        ~User();
        User(const User &) = delete;
        User &operator=(const User &) = delete;
    };
    static void *take();
    static void give(void *p);
};

// A few bytes of pinned memory that the device writes and the host reads.
struct PinnedCell {
    double *p; // 0 when made
    PinnedCell();
    ~PinnedCell();
    PinnedCell(const PinnedCell &) = delete;
    PinnedCell &operator=(const PinnedCell &) = delete;
};

struct CopySlot {
    void *p = nullptr;
    cudaEvent_t ev = nullptr;
    CopySlot()
    {
        p = PinnedSlots::take();
        const cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e != cudaSuccess) {
            PinnedSlots::give(p);
            NADIA_CUDA(e);
        }
    }
    ~CopySlot()
    {
        cudaEventSynchronize(ev); // work queued on the slot before an error
        cudaEventDestroy(ev);
        PinnedSlots::give(p);
    }
    CopySlot(const CopySlot &) = delete;
    CopySlot &operator=(const CopySlot &) = delete;
    // waits until what was queued on st by now is done: one piece's copy (the
    // event is polled, as tens of microseconds are too short to sleep)
    void wait(cudaStream_t st)
    {
        NADIA_CUDA(cudaEventRecord(ev, st));
        NADIA_CUDA(cudaEventSynchronize(ev));
    }
};

// Waits for the work queued on st.  Meanwhile helpers bring in the pages of the
// array that a read is about to fill (null: none), which leaves its contents as
// they are; they stop when the wait ends and never wait for it.
void await(cudaStream_t st, void *fill, size_t bytes);

// Calls body(slot, first row, rows) for pieces of `rows` rows of `row_bytes`
// (as they pass through a slot); each piece is done when its call returns.
// The first error of any thread is thrown once all have stopped.  fill: the
// array of `bytes` that a read fills, or null.
//
// The calling thread waits for the work queued on st before any slot is taken,
// so that slots and helpers are held for copies only: a read behind long
// iterations otherwise held eight of the sixteen slots until they ended, and a
// few such reads kept every other reconstruction's transfers waiting (and each
// of their threads polling) although its own stream was idle.  While
// it waits, helpers bring in the pages of a fresh array: B200, reads right behind
// iterations, 2048^2: FP64 3.5 -> 2.1 ms, FP32 2.1 -> 1.8 ms, 512^2 FP32 0.20 ms
// either way.
template <class Body>
void in_pieces(int device, cudaStream_t st, void *fill, size_t bytes, size_t rows, size_t row_bytes,
               Body body)
{
    NADIA_REQUIRE(row_bytes <= kSlotBytes, NADIA_ERR_INVALID, "row too long to transfer");
    if (rows == 0) return;
    await(st, fill, bytes);
    const size_t fit = kSlotBytes / row_bytes;
    // two pieces a thread at least, and pieces worth a thread's start
    const size_t worth = std::max<size_t>(1, (1u << 20) / row_bytes);
    const int most = (int)std::min<size_t>(8, rows / worth + 1);
    const size_t per = std::max<size_t>(1, std::min(fit, (rows + 2 * most - 1) / (2 * most)));
    std::atomic<size_t> next{0};
    std::exception_ptr error;
    std::mutex mu;
    auto work = [&](bool own) {
        try {
            if (!own) NADIA_CUDA(cudaSetDevice(device));
            size_t r = next.fetch_add(per);
            if (r >= rows) return; // the others were quicker
            CopySlot slot;
            for (; r < rows; r = next.fetch_add(per)) {
                body(slot, r, std::min(per, rows - r));
            }
        } catch (...) {
            next = rows;
            std::lock_guard<std::mutex> lk(mu);
            if (!error) error = std::current_exception();
        }
    };
    const std::thread::id caller = std::this_thread::get_id();
    with_helpers(most - 1, [&] { work(std::this_thread::get_id() == caller); });
    if (error) std::rethrow_exception(error);
}

// Calls f(from, to) for parts of 0 .. n-1, several at a time where n is large
// enough to be worth a thread's start.
constexpr size_t kPart = 64 << 10; // values of a part
template <class F>
void in_parts(size_t n, F f)
{
    const size_t parts = (n + kPart - 1) / kPart;
    std::atomic<size_t> next{0};
    with_helpers((int)std::min<size_t>(7, parts - (parts > 0)), [&] {
        for (size_t p; (p = next++) < parts;) f(p * kPart, std::min(n, (p + 1) * kPart));
    });
}

// Copies that are complete when they return, ordered after the work queued on st.
void to_device(void *d, const void *h, size_t bytes, int device, cudaStream_t st);
void to_host(void *h, const void *d, size_t bytes, int device, cudaStream_t st);

} // namespace nadia
