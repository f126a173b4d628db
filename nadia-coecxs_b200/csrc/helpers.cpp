// helpers.cpp -- the host helper threads.
//
// Nobody waits for the helpers to end while the process runs: each ends itself
// when there has been no reconstruction for kHelperLinger.  (They once ended
// with the last reconstruction, by a flag that its destructor raised, joined
// under and lowered; another thread's last reconstruction, gone meanwhile,
// lowered the flag before every helper had seen it, and the join never ended.)
#include "helpers.h"

#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <mutex>
#include <thread>
#include <vector>

#include <pthread.h>

#ifndef NADIA_HELPER_LINGER_MS
#define NADIA_HELPER_LINGER_MS 10000
#endif

namespace nadia {

namespace {
using Clock = std::chrono::steady_clock;
constexpr std::chrono::milliseconds kHelperLinger{NADIA_HELPER_LINGER_MS};
// as many as there are pinned slots; half the cores where those are fewer
constexpr int kMostHelpers = 16;

// one with_helpers call: helpers it still wants, and those at work in it
struct Task {
    const std::function<void()> *f;
    int want, running;
};

struct Helpers {
    std::mutex mu;
    std::condition_variable wake, done;
    std::vector<std::thread> threads; // those at work or asleep
    std::vector<std::thread> ended;   // to be joined, which does not wait
    std::deque<Task *> tasks;
    std::vector<void (*)()> give_back; // by the last helper to end
    int asleep = 0, starting = 0; // helpers not at work
    int wanted = 0;               // those that the tasks still want
    size_t uses = 0;
    Clock::time_point unused_since = Clock::now();
    bool closed = false; // the process (or the library) ends; never lowered
};
// A forked child has none of the threads, and a mutex as it stood: it starts anew.
Helpers *g_helpers = nullptr;
void in_child()
{
    Helpers *h = new Helpers;
    h->uses = g_helpers->uses;
    g_helpers = h;
}
// leaked on purpose: reconstructions destroyed by static destructors still use it
Helpers &helpers()
{
    static const bool made = [] {
        g_helpers = new Helpers;
        return pthread_atfork(nullptr, nullptr, in_child) == 0;
    }();
    (void)made;
    return *g_helpers;
}

void help()
{
    Helpers &h = helpers();
    std::unique_lock<std::mutex> lk(h.mu);
    bool given = false;
    --h.starting;
    for (;;) {
        if (h.closed) return;
        if (h.tasks.empty()) {
            const Clock::time_point until = h.unused_since + kHelperLinger;
            if (h.uses > 0) {
                given = false;
                ++h.asleep;
                h.wake.wait(lk);
                --h.asleep;
                continue;
            }
            if (Clock::now() < until) {
                given = false;
                ++h.asleep;
                h.wake.wait_until(lk, until);
                --h.asleep;
                continue;
            }
            // unused for long enough
            if (h.threads.size() == 1 && !given) {
                const std::vector<void (*)()> fs = h.give_back;
                lk.unlock();
                for (void (*f)() : fs) f();
                lk.lock();
                given = true;
                continue; // unless there is a user again
            }
            for (std::thread &t : h.threads)
                if (t.get_id() == std::this_thread::get_id()) {
                    h.ended.push_back(std::move(t));
                    std::swap(t, h.threads.back());
                    h.threads.pop_back();
                    break;
                }
            return;
        }
        Task *t = h.tasks.front();
        --h.wanted;
        if (--t->want == 0) h.tasks.pop_front();
        ++t->running;
        lk.unlock();
        (*t->f)();
        lk.lock();
        if (--t->running == 0) h.done.notify_all();
    }
}

// one helper more, with h.mu held
void start(Helpers &h)
{
    h.threads.emplace_back(help);
    ++h.starting;
}

// the helpers that have ended, with h.mu held (they hold it no more)
void reap(Helpers &h)
{
    for (std::thread &t : h.ended) t.join();
    h.ended.clear();
}

// no helper outlives the code it runs
struct Close {
    ~Close()
    {
        Helpers &h = helpers();
        std::vector<std::thread> old;
        {
            std::lock_guard<std::mutex> lk(h.mu);
            h.closed = true;
            old.swap(h.threads);
        }
        h.wake.notify_all();
        for (std::thread &t : old) t.join();
        std::lock_guard<std::mutex> lk(h.mu);
        reap(h);
    }
} close_at_end;
} // namespace

HelperUse::HelperUse()
{
    Helpers &h = helpers();
    std::lock_guard<std::mutex> lk(h.mu);
    ++h.uses;
}

HelperUse::~HelperUse()
{
    Helpers &h = helpers();
    {
        std::lock_guard<std::mutex> lk(h.mu);
        if (--h.uses > 0) return;
        h.unused_since = Clock::now();
        try {
            // there is one to give things back
            if (!h.closed && h.threads.empty() && !h.give_back.empty()) start(h);
        } catch (...) {
            // they stay until the next time
        }
    }
    h.wake.notify_all(); // from now on they sleep for a limited time
}

void when_unused(void (*give_back)())
{
    Helpers &h = helpers();
    std::lock_guard<std::mutex> lk(h.mu);
    h.give_back.push_back(give_back);
}

void with_helpers(int extra, const std::function<void()> &f)
{
    static const int most = std::min((int)std::thread::hardware_concurrency() / 2, kMostHelpers);
    extra = std::min(extra, most);
    if (extra <= 0) {
        f();
        return;
    }
    Helpers &h = helpers();
    Task t{&f, extra, 0};
    {
        std::lock_guard<std::mutex> lk(h.mu);
        if (h.closed) {
            t.want = 0;
        } else {
            h.tasks.push_back(&t);
            h.wanted += extra;
            try {
                reap(h);
                while (h.asleep + h.starting < h.wanted && (int)h.threads.size() < most) start(h);
            } catch (...) {
                // fewer helpers then
            }
        }
    }
    if (extra == 1)
        h.wake.notify_one();
    else
        h.wake.notify_all(); // one call of the kernel; there are sixteen at most
    f();
    std::unique_lock<std::mutex> lk(h.mu);
    for (auto it = h.tasks.begin(); it != h.tasks.end(); ++it)
        if (*it == &t) {
            h.tasks.erase(it);
            h.wanted -= t.want;
            break;
        }
    h.done.wait(lk, [&] { return t.running == 0; });
}

} // namespace nadia
