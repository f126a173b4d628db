// Threads that make and drop the last user of the host helper threads while
// others call them; arguments: seconds, working threads, and "fork" to end in a
// forked child too.  Prints the number of rounds; every call's parts are counted.
#include "helpers.h"

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/wait.h>
#include <thread>
#include <unistd.h>
#include <vector>

using namespace nadia;

int main(int argc, char **argv)
{
    const double seconds = argc > 1 ? atof(argv[1]) : 1;
    const auto end = std::chrono::steady_clock::now() + std::chrono::duration<double>(seconds);
    const int workers = argc > 2 ? atoi(argv[2]) : 1;
    std::atomic<long> rounds{0}, wrong{0};
    std::vector<std::thread> ts;
    // those whose reconstruction works
    for (int k = 0; k < workers; ++k)
        ts.emplace_back([&, k] {
            while (std::chrono::steady_clock::now() < end) {
                HelperUse use;
                std::atomic<int> next{0}, done{0};
                with_helpers(7, [&] {
                    while (next++ < 64) ++done;
                });
                if (done != 64) ++wrong;
                ++rounds;
                // so that the count also falls to zero while helpers doze off or end
                if (rounds % 64 == k) std::this_thread::sleep_for(std::chrono::milliseconds(3));
            }
        });
    // those whose constructor refuses its arguments
    for (int k = 0; k < 6; ++k)
        ts.emplace_back([&] {
            while (std::chrono::steady_clock::now() < end) {
                HelperUse use;
            }
        });
    for (std::thread &t : ts) t.join();
    if (argc > 3 && !std::strcmp(argv[3], "fork")) {
        HelperUse *use = new HelperUse; // held across the fork
        with_helpers(7, [] {});
        const pid_t child = fork();
        if (child == 0) {
            std::atomic<int> next{0}, done{0};
            with_helpers(7, [&] {
                while (next++ < 64) ++done;
            });
            delete use;
            std::exit(done == 64 ? 0 : 1); // static destructors run
        }
        int status = 1;
        waitpid(child, &status, 0);
        if (status != 0) ++wrong;
        delete use;
    }
    std::printf("%ld rounds, %ld wrong\n", rounds.load(), wrong.load());
    return wrong == 0 ? 0 : 1;
}
