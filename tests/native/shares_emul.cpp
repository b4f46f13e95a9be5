// A job cut over host threads (ss_shares.h) where threads run out, for
// tests/test_shares_host.py.
//   shares_emul <shares> <threads that can be had> <0: no thread, 1: no memory>
// Prints how often each share ran.
#include "ss_shares.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <system_error>
#include <utility>

static int g_have = 0, g_made = 0, g_memory = 0;

struct Scarce {
    std::thread t;
    Scarce() = default;
    template <class... A>
    explicit Scarce(A &&...a) {
        if (g_made == g_have) {
            if (g_memory) throw std::bad_alloc();
            throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        }
        ++g_made;
        t = std::thread(std::forward<A>(a)...);
    }
    Scarce(Scarce &&) = default;
    Scarce &operator=(Scarce &&) = default;
    void join() { t.join(); }
};

int main(int argc, char **argv) {
    if (argc != 4) return 2;
    const int n = std::atoi(argv[1]);
    g_have = std::atoi(argv[2]);
    g_memory = std::atoi(argv[3]);
    std::atomic<int> ran[8] = {};
    ssb::run_shares<8, Scarce>(n, [&](int i) { ++ran[i]; });
    for (int i = 0; i < 8; ++i) std::printf("%d ", ran[i].load());
    std::printf("\n");
    return 0;
}
