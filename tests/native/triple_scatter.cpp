// The opponents' matrices written hand by hand (phase_clear, phase_scatter)
// against the pair tables' (phase_gather) of poker-solver_b200/csrc/ss_triple.cuh,
// for tests/test_triple_scatter_host.py.
//   triple_scatter <seed> <deck> <hands> <zero fraction> <repeat third>
// Prints the number of cells and row masks that differ.
#include "ss_triple.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <utility>
#include <vector>

using namespace ssb::tri;

int main(int argc, char **argv) {
    if (argc != 6) return 2;
    std::mt19937 rng(static_cast<unsigned>(std::atoi(argv[1])));
    const int n = std::atoi(argv[2]), nh = std::atoi(argv[3]);
    const double zero = std::atof(argv[4]);
    const bool repeat = std::atoi(argv[5]) != 0;
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::vector<std::pair<int, int>> all;
    for (int a = 0; a < n; ++a)
        for (int b = a + 1; b < n; ++b) all.push_back({a, b});
    int H[3], HS = 32;
    std::vector<int> code[3], pair[3];
    std::vector<float> r[3];
    for (int p = 0; p < 3; ++p) {
        H[p] = std::min<int>(nh + p, static_cast<int>(all.size()));
        HS = std::max(HS, (H[p] + 31) / 32 * 32);
    }
    for (int p = 0; p < 3; ++p) {
        std::shuffle(all.begin(), all.end(), rng);
        code[p].assign(HS, 0);
        r[p].assign(HS, 0.f);
        pair[p].assign(52 * 52, HS);
        for (int h = 0; h < H[p]; ++h) {
            std::pair<int, int> x = all[h];
            if (p == 2 && repeat && h % 3 == 2) x = all[h - 1];
            const int blocked = U(rng) < 0.1;
            if (U(rng) < 0.5) std::swap(x.first, x.second);
            code[p][h] = (blocked << 16) | (x.first << 20) | (x.second << 26);
            r[p][h] = U(rng) < zero ? 0.f : static_cast<float>(U(rng)) + 1e-3f;
            if (!blocked) pair[p][x.first * 52 + x.second] = pair[p][x.second * 52 + x.first] = h;
        }
    }
    std::vector<double> m0(doubles(n), 7.0), m1(doubles(n), 9.0);
    const Tables t0 = tables(m0.data(), n), t1 = tables(m1.data(), n);
    phase_gather(0, 1, t0, r[0].data(), r[1].data(), r[2].data(), pair[0].data(), pair[1].data(), pair[2].data(), HS,
                 !repeat);
    const int nt = 384;
    const float *const rr[3] = {r[0].data(), r[1].data(), r[2].data()};
    const int *const cc[3] = {code[0].data(), code[1].data(), code[2].data()};
    for (int i = 0; i < nt; ++i) phase_clear(i, nt, t1);
    for (int i = 0; i < nt; ++i) phase_scatter(i, nt, t1, rr, cc, H, !repeat);
    if (repeat) {
        for (int i = 0; i < nt; ++i) phase_gather_third(i, nt, t0, rr[2], cc[2], H[2]);
        for (int i = 0; i < nt; ++i) phase_gather_third(i, nt, t1, rr[2], cc[2], H[2]);
    }
    int bad = 0;
    for (int x = 0; x <= n; ++x) {
        for (int y = 0; y <= n; ++y) {
            const int at = x * t0.S + y;
            bad += std::memcmp(t0.A + at, t1.A + at, 8) != 0;
            bad += std::memcmp(t0.B + at, t1.B + at, 8) != 0;
            bad += std::memcmp(t0.C + at, t1.C + at, 8) != 0;
        }
        for (int i = 0; i < 3; ++i) bad += t0.m[i * kVS + x] != t1.m[i * kVS + x];
    }
    std::printf("%d\n", bad);
    return 0;
}
