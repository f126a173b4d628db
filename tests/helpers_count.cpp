// Helper threads are started as calls want them.  Arguments: helpers wanted, calls
// at once.  Prints the threads of the process beside the calling ones.
#include "helpers.h"

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <dirent.h>
#include <thread>
#include <vector>

using namespace nadia;

static int threads()
{
    int n = 0;
    DIR *d = opendir("/proc/self/task");
    while (dirent *e = readdir(d)) n += e->d_name[0] != '.';
    closedir(d);
    return n;
}

int main(int argc, char **argv)
{
    const int extra = argc > 1 ? atoi(argv[1]) : 1, calls = argc > 2 ? atoi(argv[2]) : 1;
    HelperUse use;
    auto nap = [] { std::this_thread::sleep_for(std::chrono::milliseconds(200)); };
    std::vector<std::thread> ts;
    for (int k = 0; k < calls; ++k)
        ts.emplace_back([&] {
            for (int r = 0; r < 3; ++r) with_helpers(extra, nap);
        });
    for (std::thread &t : ts) t.join();
    std::printf("%d\n", threads() - 1);
    return 0;
}
