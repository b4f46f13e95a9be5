// The numbering of short value/regret items over launches, blocks and threads
// (ss_engine.h's cfv_items_per_launch, k_cfv<1>'s index), for
// tests/test_cfv_units_host.py.
//   cfv_units <items> <hands>
// Prints JSON: launches, items covered, and whether the last thread of every
// launch still has a unit of its own sign and an item past the launch's last
// one or its last one.
#include "ss_engine.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>

int main(int argc, char **argv) {
    if (argc != 3) return 2;
    const int n = std::atoi(argv[1]), pairs = (std::atoi(argv[2]) + 1) / 2, most = ssb::cfv_items_per_launch(pairs);
    long long covered = 0;
    int launches = 0, good = 1;
    for (long long left = n; left > 0; left -= most, ++launches) {
        const int now = static_cast<int>(std::min<long long>(left, most));
        const long long threads = static_cast<long long>(now) * pairs;
        const unsigned blocks = static_cast<unsigned>((threads + ssb::kCfvThreads - 1) / ssb::kCfvThreads);
        // the kernel's arithmetic for the first and the last thread
        const int last = static_cast<int>((blocks - 1) * ssb::kCfvThreads + ssb::kCfvThreads - 1);
        good = good && last >= 0 && last / pairs >= now - 1 && last - (last / pairs) * pairs < pairs;
        covered += now;
    }
    std::printf("{\"launches\": %d, \"covered\": %lld, \"good\": %d}\n", launches, covered, good);
    return 0;
}
