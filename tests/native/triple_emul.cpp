// Runs the block phases of the three-opponent mass by contraction
// (poker-solver_b200/csrc/ss_triple.cuh) on the host, each phase over 384
// emulated threads in kernel order, and compares every traverser hand with
// enumeration of the disjoint opponent tuples, for tests/test_triple_host.py.
//   triple_emul <seed> <deck> <hands per player> <zero fraction> <repeat third> [zero player]
// Hands are random distinct pairs over the dense deck; about a tenth of every
// range touches the board (dense index 63); weights U(0, 1), the given share
// zeroed (all of the zero player's); with repeat third, the third opponent
// holds every fourth combo twice.  Prints JSON: the largest error relative to
// the product of the ranges' sums, and hands whose exact zero is wrong.
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
    const double zero = std::atof(argv[4]);
    const bool repeat = std::atoi(argv[5]) != 0;
    const int none = argc > 6 ? std::atoi(argv[6]) : -1;
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const int HS = (nh + 31) / 32 * 32;
    std::vector<std::vector<int>> code(4, std::vector<int>(HS, 0));
    std::vector<std::vector<float>> r(3, std::vector<float>(HS, 0.f));
    for (int p = 0; p < 4; ++p) {
        std::vector<std::pair<int, int>> all;
        for (int a = 0; a < n; ++a)
            for (int b = a + 1; b < n; ++b) all.push_back({a, b});
        std::shuffle(all.begin(), all.end(), rng);
        for (int h = 0; h < nh; ++h) {
            int a = all[h % all.size()].first, b = all[h % all.size()].second, blocked = 0;
            if (p == 2 && repeat && h % 4 == 3) a = (code[2][h - 1] >> 20) & 63, b = (code[2][h - 1] >> 26) & 63;
            if (U(rng) < 0.1) {
                (U(rng) < 0.5 ? a : b) = 63;
                blocked = 1;
            }
            if (a == 63 || b == 63) blocked = 1;
            code[p][h] = (blocked << 16) | (a << 20) | (b << 26);
            if (p < 3) r[p][h] = p == none || U(rng) < zero ? 0.f : static_cast<float>(U(rng));
        }
    }
    std::vector<int> pair[3];
    for (int p = 0; p < 3; ++p) {
        pair[p].assign(52 * 52, HS);
        for (int h = 0; h < nh; ++h) {
            if (code[p][h] & 0x10000) continue;
            const int a = (code[p][h] >> 20) & 63, b = (code[p][h] >> 26) & 63;
            pair[p][a * 52 + b] = pair[p][b * 52 + a] = h;
        }
    }
    std::vector<double> mem(doubles(n), std::nan(""));   // whatever a phase reads, a phase has written
    const Tables t = tables(mem.data(), n);
    std::vector<unsigned long long> mA(kVS), mB(kVS);
    std::vector<int> nA(kVS), nB(kVS), nW(kVS), nD(kVS);
    std::vector<long long> s(4);
    const Counts k{mA.data(), mB.data(), nA.data(), nB.data(), nW.data(), nD.data(), s.data()};
    const int nt = 384;
    for (int i = 0; i < nt; ++i)
        phase_gather(i, nt, t, r[0].data(), r[1].data(), r[2].data(), pair[0].data(), pair[1].data(), pair[2].data(),
                     HS, !repeat);
    if (repeat)
        for (int i = 0; i < nt; ++i) phase_gather_third(i, nt, t, r[2].data(), code[2].data(), nh);
    for (int i = 0; i < nt; ++i) phase_products(i, nt, t);
    for (int i = 0; i < nt; ++i) phase_vectors(i, nt, t);
    for (int i = 0; i < nt; ++i) phase_scalars(i, nt, t);
    for (int i = 0; i < nt; ++i) phase_masks(i, nt, t, k);
    for (int i = 0; i < nt; ++i) phase_counts(i, nt, t, k);

    auto mask = [&](int p, int h) {
        const int a = (code[p][h] >> 20) & 63, b = (code[p][h] >> 26) & 63;
        return (a < 63 ? 1ull << a : 0ull) | (b < 63 ? 1ull << b : 0ull);
    };
    std::vector<std::vector<std::pair<unsigned long long, double>>> live(3);
    for (int p = 0; p < 3; ++p)
        for (int h = 0; h < nh; ++h)
            if (!(code[p][h] & 0x10000) && r[p][h] > 0.f) live[p].push_back({mask(p, h), r[p][h]});
    const double scale = std::max(1e-300, t.sc[FA] * t.sc[FB] * t.sc[FC]);
    double worst = 0.0;
    int zero_bad = 0, zeros = 0;
    for (int h = 0; h < nh; ++h) {
        const unsigned long long m0 = mask(3, h);
        double want = 0.0;
        for (auto &x : live[0]) {
            if (x.first & m0) continue;
            for (auto &y : live[1]) {
                if (y.first & (m0 | x.first)) continue;
                double z = 0.0;
                for (auto &w : live[2])
                    if (!(w.first & (m0 | x.first | y.first))) z += w.second;
                want += x.second * y.second * z;
            }
        }
        const int a = std::min((code[3][h] >> 20) & 63, n), b = std::min((code[3][h] >> 26) & 63, n);
        const double m = hand_mass(a, b, t);
        worst = std::max(worst, std::fabs(m - want) / scale);
        bool any = false;
        for (int j = 0; j < nh && !any; ++j) any = tuple_with(a, b, k, r[2][j], code[2][j]);
        zeros += !any;
        zero_bad += any != (want > 0.0);
        if (want == 0.0 && std::fabs(m) > zero_bound(t)) ++zero_bad;   // the kernel would not look
    }
    std::printf("{\"worst\": %.3e, \"zeros\": %d, \"zero_bad\": %d}\n", worst, zeros, zero_bad);
    return 0;
}
