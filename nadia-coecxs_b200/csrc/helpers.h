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
// and does not throw.  The helpers are the process's (half its cores at most,
// shared by all concurrent calls; starting threads for each call instead cost
// about 0.1 ms).
void with_helpers(int extra, const std::function<void()> &f);

} // namespace nadia
