// The three-opponent mass by contraction and its second sum
// (poker-solver_b200/csrc/ss_triple.cuh) on ranges whose weight lies on hands
// that the traverser blocks, against enumeration in long double, for
// tests/test_triple_skew_host.py.
//   triple_skew <seed> <deck> <hands per player> <weight of the others> <player> [repeat third]
// Every traverser hand holds card 0.  The given opponent's hands with card 0
// weigh U(0.5, 1), its others that times the given weight; the other two
// opponents' U(0, 1).  Prints JSON: the largest relative error of a mass, the
// smallest mass over the product of the ranges' sums, and hands whose exact
// zero is wrong.
#include "ss_triple.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <utility>
#include <vector>

using namespace ssb::tri;

int main(int argc, char **argv) {
    if (argc < 6) return 2;
    std::mt19937 rng(static_cast<unsigned>(std::atoi(argv[1])));
    const int n = std::atoi(argv[2]), nh = std::atoi(argv[3]);
    const double rest = std::atof(argv[4]);
    const int skewed = std::atoi(argv[5]);
    const bool repeat = argc > 6 && std::atoi(argv[6]) != 0;
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const int HS = (nh + 31) / 32 * 32;
    std::vector<std::vector<int>> code(4, std::vector<int>(HS, 0));
    std::vector<std::vector<float>> r(3, std::vector<float>(HS, 0.f));
    std::vector<int> H(4, nh);
    H[3] = std::min(nh, n - 1);
    for (int p = 0; p < 4; ++p) {
        std::vector<std::pair<int, int>> all;
        for (int a = 0; a < n; ++a)
            for (int b = a + 1; b < n; ++b)
                if (p < 3 || a == 0) all.push_back({a, b});
        std::shuffle(all.begin(), all.end(), rng);
        for (int h = 0; h < H[p]; ++h) {
            int a = all[h % all.size()].first, b = all[h % all.size()].second;
            if (p == 2 && repeat && h % 4 == 3) a = (code[2][h - 1] >> 20) & 63, b = (code[2][h - 1] >> 26) & 63;
            code[p][h] = (a << 20) | (b << 26);
            if (p == 3) continue;
            const double u = U(rng);
            r[p][h] = static_cast<float>(p != skewed ? u : (0.5 + 0.5 * u) * (a == 0 ? 1.0 : rest));
        }
    }
    std::vector<int> pair[3];
    for (int p = 0; p < 3; ++p) {
        pair[p].assign(52 * 52, HS);
        for (int h = 0; h < nh; ++h) {
            const int a = (code[p][h] >> 20) & 63, b = (code[p][h] >> 26) & 63;
            pair[p][a * 52 + b] = pair[p][b * 52 + a] = h;
        }
    }
    std::vector<double> mem(doubles(n), std::nan(""));
    const Tables t = tables(mem.data(), n);
    std::vector<unsigned long long> mA(kVS), mB(kVS);
    std::vector<int> nA(kVS), nB(kVS), nW(kVS), nD(kVS);
    std::vector<long long> s(4);
    const Counts k{mA.data(), mB.data(), nA.data(), nB.data(), nW.data(), nD.data(), s.data()};
    phase_gather(0, 1, t, r[0].data(), r[1].data(), r[2].data(), pair[0].data(), pair[1].data(), pair[2].data(), HS,
                 !repeat);
    if (repeat) phase_gather_third(0, 1, t, r[2].data(), code[2].data(), nh);
    phase_products(0, 1, t);
    phase_vectors(0, 1, t);
    phase_scalars(0, 1, t);
    phase_masks(0, 1, t, k);
    phase_counts(0, 1, t, k);

    auto mask = [&](int p, int h) { return 1ull << ((code[p][h] >> 20) & 63) | 1ull << ((code[p][h] >> 26) & 63); };
    double worst = 0.0, least = 1.0;
    int zero_bad = 0;
    for (int h = 0; h < H[3]; ++h) {
        const unsigned long long m0 = mask(3, h);
        long double want = 0.0L;
        for (int x = 0; x < nh; ++x) {
            if (mask(0, x) & m0) continue;
            for (int y = 0; y < nh; ++y) {
                if (mask(1, y) & (m0 | mask(0, x))) continue;
                long double z = 0.0L;
                for (int w = 0; w < nh; ++w)
                    if (!(mask(2, w) & (m0 | mask(0, x) | mask(1, y)))) z += r[2][w];
                want += static_cast<long double>(r[0][x]) * r[1][y] * z;
            }
        }
        const int a = (code[3][h] >> 20) & 63, b = (code[3][h] >> 26) & 63;
        double m = hand_mass(a, b, t);
        if (std::fabs(m) <= zero_bound(t)) {
            m = 0.0;
            for (int j = 0; j < nh; ++j) m += tuple_mass(a, b, t, k, r[2][j], code[2][j]);
        }
        if (want == 0.0L) {
            zero_bad += m != 0.0;
            continue;
        }
        worst = std::max(worst, static_cast<double>(std::fabs((m - want) / want)));
        least = std::min(least, static_cast<double>(want) / (t.sc[FA] * t.sc[FB] * t.sc[FC]));
    }
    std::printf("{\"worst\": %.3e, \"least\": %.3e, \"zero_bad\": %d}\n", worst, least, zero_bad);
    return 0;
}
