// What the process keeps between reconstructions is given back once, a while
// after the last of them and not while there is one.  Compiled with a linger of
// 200 ms; prints the first thing that is wrong.
#include "helpers.h"

#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

using namespace nadia;

std::atomic<int> given{0};
void give_back() { ++given; }

void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }

bool wait_for(int count)
{
    for (int k = 0; k < 500 && given != count; ++k) nap(10);
    return given == count;
}

#define CHECK(c)                                          \
    do {                                                  \
        if (!(c)) {                                       \
            std::printf("line %d: %s (%d)\n", __LINE__, #c, given.load()); \
            return 1;                                     \
        }                                                 \
    } while (0)

int main()
{
    when_unused(give_back);
    for (int k = 0; k < 5; ++k) { // one after the other
        HelperUse use;
        if (k & 1) with_helpers(3, [] {});
    }
    CHECK(given == 0);
    CHECK(wait_for(1));
    nap(500);
    CHECK(given == 1); // once
    {
        HelperUse use; // no call while there is one
        with_helpers(3, [] {});
        nap(500);
        CHECK(given == 1);
    }
    CHECK(wait_for(2));
    {
        HelperUse use; // without a helper at work
    }
    CHECK(wait_for(3));
    nap(500);
    CHECK(given == 3);
    return 0;
}
