// helpers.h -- the process's host helper threads (no CUDA here).
#pragma once

#include <functional>

namespace nadia {

// Held by every reconstruction: while there is one, the helpers sleep between
// calls; kHelperLinger after the last they end.
class HelperUse {
public:
    HelperUse();
    ~HelperUse();
    HelperUse(const HelperUse &) = delete;
    HelperUse &operator=(const HelperUse &) = delete;
};

// Runs f on the calling thread and on up to `extra` helper threads at once;
// returns when all have returned.  f divides its work among its callers itself
// and does not throw.  The helpers are the process's, shared by all concurrent
// calls and started as calls want them, up to sixteen or half the cores; starting
// threads for each call instead cost about 0.1 ms.
void with_helpers(int extra, const std::function<void()> &f);

// give_back() is called on a helper thread when there has been no reconstruction
// for kHelperLinger: what the process keeps from one reconstruction to the next
// ends there.  Call it once for each function.
void when_unused(void (*give_back)());

} // namespace nadia
