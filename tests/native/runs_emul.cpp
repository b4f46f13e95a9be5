// The batch's rule for launches that may go side by side (ss_runs.h) on
// launch lists as a batch builds them, for tests/test_batch_runs.py.
//   runs_emul <players> <bit mask of the players who make decisions>
// Per traverser: a snapshot before the last one's pass, three terminal
// launches of falling weight, and, where the player decides, a value and a
// reach launch.  Prints the ordered list as JSON: [[run, type, traverser,
// weight], ...].
#include "ss_runs.h"

#include <cstdio>
#include <cstdlib>

struct Launch {
    int type, kind, t;
    double w;
};
enum { BUMP, SNAP, TERM, CFV, REACH };

int main(int argc, char **argv) {
    if (argc != 3) return 2;
    const int np = std::atoi(argv[1]), decides = std::atoi(argv[2]);
    std::vector<Launch> q{{BUMP, 0, 0, 0.0}};
    for (int t = 0; t < np; ++t) {
        if (t == np - 1) q.push_back({SNAP, 0, t, 0.0});
        for (int k = 0; k < 3; ++k) q.push_back({TERM, k, t, 10.0 * (np - t) - k});
        if (decides >> t & 1) {
            q.push_back({CFV, 0, t, 0.0});
            q.push_back({REACH, 0, t, 0.0});
        }
    }
    auto terminal = [](const Launch &L) { return L.type == TERM; };
    ssb::order_runs(&q, terminal, [](const Launch &L) { return L.w; });
    int run = 0;
    std::printf("[");
    for (size_t i = 0; i < q.size(); ++run) {
        const size_t j = ssb::run_end(q, i, terminal);
        for (; i < j; ++i) std::printf("%s[%d, %d, %d, %g]", i ? ", " : "", run, q[i].type, q[i].t, q[i].w);
    }
    std::printf("]\n");
    return 0;
}
