// ss_triple.cuh -- card-removal mass of three counted opponents for every
// traverser hand (folds and leaves of 4+ player subgames), by contraction.
//
// With symmetric combo matrices A, B, C (zero diagonal) of the three
// opponents' reach over the dense deck, the mass of pairwise disjoint hands
// (o1, o2, o3) is, by inclusion-exclusion over the cards that two of them
// share (u = row sums, F = sum u / 2, Q_XY = u_X . u_Y, d_XY(x) =
// sum_y X[x][y] Y[x][y], E_XY = sum d_XY / 2),
//   F_A F_B F_C + F_C (E_AB - Q_AB) + F_B (E_AC - Q_AC) + F_A (E_BC - Q_BC)
//   + 2 sum_x u_A u_B u_C + u_A C u_B + u_C B u_A + u_C A u_B
//   - 2 sum_x (u_A d_BC + u_B d_AC + u_C d_AB)
//   + 2 sum_xy A B C - tr(A B C).
// For a traverser hand {a, b} it is the same expression on the matrices with
// rows and columns a, b removed (primed).  F', Q', E', the elementwise sum
// and the trace follow from tables of the full matrices in O(1); the sums
// over x run over the deck with u'(x) = u(x) - X[x][a] - X[x][b],
// (C' u_B')(x) = (C u_B)(x) - (C B)[x][a] - (C B)[x][b] - C[x][a] u_B'(a) -
// C[x][b] u_B'(b), and the like: O(deck) per hand.  (Conditioning on the
// third opponent's hand, ss_cr3.cuh, takes O(hands) evaluations of the
// two-opponent form instead.)
//
// A board card of the traverser's hand maps to the dummy index n (the deck
// size), whose rows, columns and vector entries are zero.  Rows are S = n + 1
// rounded up to odd doubles, so rows and columns both read without bank
// conflicts across consecutive cards.
//
// Each phase is a function of (thread index, thread count) whose work items
// are independent within the phase; the kernel separates phases with block
// barriers, and a host build runs them one after another.
#pragma once

#if defined(__CUDACC__)
#define SSB_TRI_HD __host__ __device__ __forceinline__
#else
#define SSB_TRI_HD inline
#endif

namespace ssb {
namespace tri {

// per-card vectors, then the scalars (one array, fixed order)
enum Vec : int { UA, UB, UC, DAB, DAC, DBC, AUB, BUA, AUC, CUA, BUC, CUB, HH, TABC, TCAB, TACB, N_VEC };
enum Scal : int { FA, FB, FC, QAB, QAC, QBC, EAB, EAC, EBC, SH, TR, N_SCAL };
constexpr int kVS = 56;   // stride of a per-card vector (n <= 52 plus the dummy)

struct Tables {
    double *A, *B, *C, *AB, *CB;   // [S][S]
    double *v;                     // [N_VEC][kVS]
    double *sc;                    // [N_SCAL]
    unsigned long long *m;         // [3][kVS]: nonzero cells of each row of A, B, C
    int n, S;
};

SSB_TRI_HD constexpr int stride(int n) { return (n + 1) | 1; }
SSB_TRI_HD constexpr int doubles(int n) { return 5 * stride(n) * stride(n) + N_VEC * kVS + N_SCAL + 1 + 3 * kVS; }

SSB_TRI_HD Tables tables(double *mem, int n) {
    Tables t;
    t.n = n;
    t.S = stride(n);
    const int m = t.S * t.S;
    t.A = mem;
    t.B = mem + m;
    t.C = mem + 2 * m;
    t.AB = mem + 3 * m;
    t.CB = mem + 4 * m;
    t.v = mem + 5 * m;
    t.sc = t.v + N_VEC * kVS;
    t.m = reinterpret_cast<unsigned long long *>(t.sc + N_SCAL + 1);
    return t;
}

// phase 1: the matrices of the opponents' hands with reach, written hand by
// hand over cleared ones (3 x 1128 hands at most; looking every pair of cards
// up took 9 K cycles of a block).  The first two ranges repeat no combo.
// Without `third` (a third range that does) C is left to phase_gather_third.
// t.m: the nonzero cells of each row.
SSB_TRI_HD void phase_clear(int tid, int nt, const Tables &t) {
    for (int i = tid; i < 3 * t.S * t.S; i += nt) t.A[i] = 0.0;   // A, B, C lie in a row
    for (int i = tid; i < 3 * kVS; i += nt) t.m[i] = 0ull;
}
SSB_TRI_HD void mark(unsigned long long *row, int x) {
#if defined(__CUDA_ARCH__)
    atomicOr(reinterpret_cast<unsigned *>(row) + (x >> 5), 1u << (x & 31));   // (64 bits would be a loop)
#else
    *row |= 1ull << x;
#endif
}
template <class T>
SSB_TRI_HD void phase_scatter(int tid, int nt, const Tables &t, const T *const r[3], const int *const code[3],
                              const int H[3], bool third) {
    const int n = H[0] + H[1] + (third ? H[2] : 0);
#pragma unroll 4
    for (int i = tid; i < n; i += nt) {
        const int o = i < H[0] ? 0 : i < H[0] + H[1] ? 1 : 2;
        const int h = i - (o > 0 ? H[0] : 0) - (o > 1 ? H[1] : 0);
        const int c = (o == 0 ? code[0] : o == 1 ? code[1] : code[2])[h];
        const T v = (o == 0 ? r[0] : o == 1 ? r[1] : r[2])[h];
        if ((c & 0x10000) || v == T(0) || (o == 2 && !(v > T(0)))) continue;   // touches the board, or nothing to add
        const int x = (c >> 20) & 63, y = (c >> 26) & 63;
        double *M = o == 0 ? t.A : o == 1 ? t.B : t.C;
        M[x * t.S + y] = M[y * t.S + x] = static_cast<double>(v);
        mark(t.m + o * kVS + x, y);
        mark(t.m + o * kVS + y, x);
    }
}
// The same from the pair tables ([52][52] dense pair -> range index, HS if
// none), row by row: what the host checks hold the scatter against.
template <class T>
SSB_TRI_HD void phase_gather(int tid, int nt, const Tables &t, const T *r1, const T *r2, const T *r3,
                             const int *pair1, const int *pair2, const int *pair3, int HS, bool third) {
    for (int x = tid; x <= t.n; x += nt) {
        for (int i = 0; i < 3; ++i) t.m[i * kVS + x] = 0ull;
        for (int y = 0; y <= t.n; ++y) {
            double v[3] = {0.0, 0.0, 0.0};
            if (x < t.n && y < t.n) {
                const int j1 = pair1[x * 52 + y], j2 = pair2[x * 52 + y], j3 = third ? pair3[x * 52 + y] : HS;
                if (j1 < HS) v[0] = static_cast<double>(r1[j1]);
                if (j2 < HS) v[1] = static_cast<double>(r2[j2]);
                if (j3 < HS && r3[j3] > T(0)) v[2] = static_cast<double>(r3[j3]);
            }
            t.A[x * t.S + y] = v[0];
            t.B[x * t.S + y] = v[1];
            t.C[x * t.S + y] = v[2];
            for (int i = 0; i < 3; ++i) t.m[i * kVS + x] |= static_cast<unsigned long long>(v[i] != 0.0) << y;
        }
    }
}

// phase 1 continued, for a third range that repeats a combo: its hands add up
// in hand order, one item per row
template <class T>
SSB_TRI_HD void phase_gather_third(int tid, int nt, const Tables &t, const T *r3, const int *code3, int H3) {
    for (int x = tid; x < t.n; x += nt)
        for (int h = 0; h < H3; ++h) {
            const int code = code3[h];
            if ((code & 0x10000) || !(r3[h] > T(0))) continue;   // touches the board, or nothing to add
            const int p = (code >> 20) & 63, q = (code >> 26) & 63;
            if (p != x && q != x) continue;
            const int o = p == x ? q : p;
            t.C[x * t.S + o] += static_cast<double>(r3[h]);
            t.m[2 * kVS + x] |= 1ull << o;
        }
}

// sum of f(0) .. f(n - 1) in four interleaved partial sums (a chain of n
// dependent FP64 additions is the latency of a phase)
template <class F>
SSB_TRI_HD double sum4(int n, F f) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int x = 0;
#pragma unroll 2
    for (; x + 3 < n; x += 4) {
        s0 += f(x);
        s1 += f(x + 1);
        s2 += f(x + 2);
        s3 += f(x + 3);
    }
    for (; x < n; ++x) s0 += f(x);
    return (s0 + s1) + (s2 + s3);
}

SSB_TRI_HD int low_bit(unsigned long long m) {
#if defined(__CUDA_ARCH__)
    return __ffsll(static_cast<long long>(m)) - 1;
#else
    return __builtin_ctzll(m);
#endif
}

// phase 2: row sums, and AB = A B, CB = C B in 4 x 4 cells per item (A and C
// are symmetric: row k is column k), each cell summed over k in order, without
// the k whose cells are all zero in one operand's tile (sparse ranges)
SSB_TRI_HD void phase_products(int tid, int nt, const Tables &t) {
    const int n = t.n, S = t.S, nt4 = (n + 3) / 4;
    for (int q = tid; q < 2 * nt4 * nt4; q += nt) {
        const bool second = q >= nt4 * nt4;
        const int r = second ? q - nt4 * nt4 : q;
        const double *M = second ? t.C : t.A;
        const unsigned long long *mM = t.m + (second ? 2 : 0) * kVS, *mB = t.m + kVS;
        double *P = second ? t.CB : t.AB;
        int ii[4], jj[4];
        unsigned long long rows = 0ull, cols = 0ull;
        for (int i = 0; i < 4; ++i) {   // past the deck: the dummy's zeros
            ii[i] = r / nt4 * 4 + i < n ? r / nt4 * 4 + i : n;
            jj[i] = r % nt4 * 4 + i < n ? r % nt4 * 4 + i : n;
            rows |= mM[ii[i]];
            cols |= mB[jj[i]];
        }
        double acc[4][4] = {};
        for (unsigned long long m = rows & cols; m; m &= m - 1) {
            const int k = low_bit(m);
            double x[4], y[4];
            for (int i = 0; i < 4; ++i) {
                x[i] = M[k * S + ii[i]];
                y[i] = t.B[k * S + jj[i]];
            }
            for (int i = 0; i < 4; ++i)
                for (int j = 0; j < 4; ++j) acc[i][j] += x[i] * y[j];
        }
        for (int i = 0; i < 4; ++i)
            for (int j = 0; j < 4; ++j)
                if (ii[i] < n && jj[j] < n) P[ii[i] * S + jj[j]] = acc[i][j];
    }
    // the row sums, on the threads that had the fewest tiles
    for (int i = nt - 1 - tid; i < 3 * n; i += nt) {
        const int c = i % n;
        const double *M = (i < n ? t.A : i < 2 * n ? t.B : t.C) + c * S;
        t.v[(i < n ? UA : i < 2 * n ? UB : UC) * kVS + c] = sum4(n, [&](int x) { return M[x]; });
    }
    for (int i = tid; i < N_VEC; i += nt) t.v[i * kVS + n] = 0.0;
    for (int i = tid; i <= n; i += nt) t.AB[n * S + i] = t.AB[i * S + n] = t.CB[n * S + i] = t.CB[i * S + n] = 0.0;
}

// phase 3: the other per-card vectors, one item per (vector, card)
SSB_TRI_HD void phase_vectors(int tid, int nt, const Tables &t) {
    const int n = t.n, S = t.S;
    for (int i = tid; i < 10 * n; i += nt) {
        const int g = i / n, c = i - g * n;
        if (g < 6) {
            const double *M = (g == 0 || g == 2 ? t.A : g == 1 || g == 4 ? t.B : t.C) + c * S;
            const double *u = t.v + (g == 0 || g == 5 ? UB : g == 1 || g == 3 ? UA : UC) * kVS;
            t.v[(AUB + g) * kVS + c] = sum4(n, [&](int x) { return M[x] * u[x]; });
        } else if (g == 6) {
            const double *a = t.A + c * S, *b = t.B + c * S, *d = t.C + c * S;
            t.v[DAC * kVS + c] = sum4(n, [&](int x) { return a[x] * d[x]; });
            t.v[HH * kVS + c] = sum4(n, [&](int x) { return a[x] * b[x] * d[x]; });
            t.v[DAB * kVS + c] = t.AB[c * S + c];
            t.v[DBC * kVS + c] = t.CB[c * S + c];
        } else {
            // (A B C), (C A B) and (A C B) at [c][c]
            const double *M = (g == 9 ? t.A : t.C) + c * S;
            const double *P = g == 9 ? t.CB : t.AB;
            const int at = g == 7 ? c * S : c, step = g == 7 ? 1 : S;
            t.v[(g == 7 ? TABC : g == 8 ? TCAB : TACB) * kVS + c] =
                sum4(n, [&](int x) { return M[x] * P[at + x * step]; });
        }
    }
}

// phase 4: the scalars, each in sum4's order; on the device four lanes take the
// four partial sums (one thread per scalar: 3 K cycles of waiting for it)
SSB_TRI_HD void phase_scalars(int tid, int nt, const Tables &t) {
    auto term = [&](int k, int c) {
        const int p = k == QAB || k == QAC ? UA : k == QBC ? UB : -1, q = k == QAB ? UB : UC;
        const int one = k < 3 ? UA + k : k >= EAB && k <= EBC ? DAB + (k - EAB) : k == SH ? HH : TABC;
        return p >= 0 ? t.v[p * kVS + c] * t.v[q * kVS + c] : t.v[one * kVS + c];
    };
    auto put = [&](int k, double s) { t.sc[k] = k < 3 || (k >= EAB && k <= EBC) ? 0.5 * s : s; };
#if defined(__CUDA_ARCH__)
    const int part = tid & 3, n4 = t.n & ~3;
    for (int base = (tid >> 5) * 8; base < N_SCAL; base += nt >> 2) {
        const int k = base + ((tid & 31) >> 2);
        double s = 0.0;
        if (k < N_SCAL) {
#pragma unroll 4
            for (int c = part; c < n4; c += 4) s += term(k, c);
            if (part == 0)
                for (int c = n4; c < t.n; ++c) s += term(k, c);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (part == 0 && k < N_SCAL) put(k, s);
    }
#else
    for (int k = tid; k < N_SCAL; k += nt) put(k, sum4(t.n, [&](int c) { return term(k, c); }));
#endif
}

// The mass of one traverser hand with dense cards (a, b): the sums over the
// deck's cards x0, x0 + step, ... (few hands: several lanes per hand), then the
// rest from their totals.
struct Part {
    double acc, ACab, ACba;   // AC = A C at [a][b] and [b][a]
};
SSB_TRI_HD Part hand_part(int a, int b, const Tables &t, int x0, int step) {
    const int S = t.S;
    const double *v = t.v;
    const double Aab = t.A[a * S + b], Bab = t.B[a * S + b];
    const double Aa = v[UA * kVS + a] - Aab, Ab = v[UA * kVS + b] - Aab;
    const double Ba = v[UB * kVS + a] - Bab, Bb = v[UB * kVS + b] - Bab;
    double acc = 0.0, ACab = 0.0, ACba = 0.0;
#pragma unroll 2
    for (int x = x0; x < t.n; x += step) {
        const double Xa = t.A[x * S + a], Xb = t.A[x * S + b];
        const double Ya = t.B[x * S + a], Yb = t.B[x * S + b];
        const double Za = t.C[x * S + a], Zb = t.C[x * S + b];
        ACab += Xa * Zb;
        ACba += Xb * Za;
        const bool out = x == a || x == b;
        const double al = out ? 0.0 : v[UA * kVS + x] - Xa - Xb;
        const double be = out ? 0.0 : v[UB * kVS + x] - Ya - Yb;
        const double ga = out ? 0.0 : v[UC * kVS + x] - Za - Zb;
        // (C' u_B')(x), (B' u_A')(x) + (A' u_B')(x), and d'_BC, d'_AC, d'_AB at x
        const double cb = v[CUB * kVS + x] - (t.CB[x * S + a] + t.CB[x * S + b]) - Za * Ba - Zb * Bb;
        const double ba = (v[BUA * kVS + x] + v[AUB * kVS + x]) - (t.AB[a * S + x] + t.AB[b * S + x]) -
                          (t.AB[x * S + a] + t.AB[x * S + b]) - Ya * Aa - Yb * Ab - Xa * Ba - Xb * Bb;
        const double dbc = v[DBC * kVS + x] - Ya * Za - Yb * Zb;
        const double dac = v[DAC * kVS + x] - Xa * Za - Xb * Zb;
        const double dab = v[DAB * kVS + x] - Xa * Ya - Xb * Yb;
        acc += al * (2.0 * (be * ga - dbc) + cb) + ga * (ba - 2.0 * dab) - 2.0 * (be * dac);
    }
    return Part{acc, ACab, ACba};
}
SSB_TRI_HD double hand_finish(int a, int b, const Tables &t, const Part &part) {
    const int S = t.S;
    const double *v = t.v, *sc = t.sc;
    const double acc = part.acc, ACab = part.ACab, ACba = part.ACba;
    const double Aab = t.A[a * S + b], Bab = t.B[a * S + b], Cab = t.C[a * S + b];
    const double Aa = v[UA * kVS + a] - Aab, Ab = v[UA * kVS + b] - Aab;
    const double Ba = v[UB * kVS + a] - Bab, Bb = v[UB * kVS + b] - Bab;
    const double Ca = v[UC * kVS + a] - Cab, Cb = v[UC * kVS + b] - Cab;
    const double ABs = t.AB[a * S + b] + t.AB[b * S + a], CBab = t.CB[a * S + b], CBba = t.CB[b * S + a];
    auto at2 = [&](int k) { return v[k * kVS + a] + v[k * kVS + b]; };
    const double fa = sc[FA] - at2(UA) + Aab, fb = sc[FB] - at2(UB) + Bab, fc = sc[FC] - at2(UC) + Cab;
    const double qab = sc[QAB] - (at2(AUB) + at2(BUA)) + (at2(DAB) + ABs) - (Aa * Ba + Ab * Bb);
    const double qac = sc[QAC] - (at2(AUC) + at2(CUA)) + (at2(DAC) + (ACab + ACba)) - (Aa * Ca + Ab * Cb);
    const double qbc = sc[QBC] - (at2(BUC) + at2(CUB)) + (at2(DBC) + (CBab + CBba)) - (Ba * Ca + Bb * Cb);
    const double eab = sc[EAB] - at2(DAB) + Aab * Bab;
    const double eac = sc[EAC] - at2(DAC) + Aab * Cab;
    const double ebc = sc[EBC] - at2(DBC) + Bab * Cab;
    const double h = sc[SH] - 2.0 * at2(HH) + 2.0 * (Aab * Bab * Cab);
    const double tr = sc[TR] - at2(TABC) - at2(TCAB) + ABs * Cab - at2(TACB) + Aab * (CBab + CBba) + Bab * (ACab + ACba);
    return fa * fb * fc + fc * (eab - qab) + fb * (eac - qac) + fa * (ebc - qbc) + acc + 2.0 * h - tr;
}

SSB_TRI_HD double hand_mass(int a, int b, const Tables &t) { return hand_finish(a, b, t, hand_part(a, b, t, 0, 1)); }

// Up to this bound a computed mass is summed again by conditioning on the
// third opponent's hand (pair_mass): the contraction subtracts what hands that
// share a card with the traverser add to the sums, so its error is a few
// hundred roundings of F_A F_B F_C (below 1e-13 of that product), whatever is
// left of it.  At 1e-6 of the product that is 1e-7 of the mass at most (3e-12
// was seen at 8e-6, 120 hands).  Conditioning leaves those hands out instead, so a
// third range whose weight lies on cards of the traverser's costs no digits;
// it also finds the empty sets, whose mass is exactly 0.
SSB_TRI_HD double zero_bound(const Tables &t) { return 1e-6 * t.sc[FA] * t.sc[FB] * t.sc[FC]; }

// The mass of the first two opponents' pairs of disjoint hands that avoid the
// four cards {a, b, x, y}: the two-opponent form, D2 in ss_cr3.cuh.
SSB_TRI_HD double pair_mass(int a, int b, int x, int y, const Tables &t) {
    const int s[4] = {a, b, x, y};
    const double *v = t.v;
    double fa = t.sc[FA], fb = t.sc[FB], q = t.sc[QAB], e = t.sc[EAB];
    for (int i = 0; i < 4; ++i) {
        const int c = s[i];
        double ua = v[UA * kVS + c], ub = v[UB * kVS + c];
        fa -= ua;
        fb -= ub;
        q -= v[AUB * kVS + c] + v[BUA * kVS + c];
        e -= v[DAB * kVS + c];
        for (int j = 0; j < 4; ++j) {
            const double A = t.A[c * t.S + s[j]], B = t.B[c * t.S + s[j]];
            ua -= A;
            ub -= B;
            q += t.AB[c * t.S + s[j]];
            if (j > i) {
                fa += A;
                fb += B;
                e += A * B;
            }
        }
        q -= ua * ub;
    }
    return fa * fb - q + e;
}

// Whether a tuple of positive reach is disjoint and avoids {a, b} (exact):
// tuple_with asks it for one hand of the third opponent, by the two-opponent
// count on the positive cells of A and B (row masks mA, mB; row and vector
// counts as in the mass).  Only hands near zero mass come here.
struct Counts {
    unsigned long long *mA, *mB;   // [kVS]
    int *nA, *nB, *nW, *nD;        // [kVS]: row counts, (I_B n_A + I_A n_B), common cells
    long long *s;                  // F_A, F_B, Q, E
};
SSB_TRI_HD int popc(unsigned long long x) {
#if defined(__CUDA_ARCH__)
    return __popcll(x);
#else
    return __builtin_popcountll(x);
#endif
}
SSB_TRI_HD void phase_masks(int tid, int nt, const Tables &t, const Counts &k) {
    auto put = [&](int c, unsigned long long a, unsigned long long b) {
        k.mA[c] = a;
        k.mB[c] = b;
        k.nA[c] = popc(a);
        k.nB[c] = popc(b);
        k.nD[c] = popc(a & b);
    };
#if defined(__CUDA_ARCH__)
    const int lane = tid & 31;   // a warp per row
    for (int c = tid >> 5; c <= t.n; c += nt >> 5) {
        unsigned long long a = 0ull, b = 0ull;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int x = half * 32 + lane;
            a |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, x < t.n && t.A[c * t.S + x] > 0.0)) << (32 * half);
            b |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, x < t.n && t.B[c * t.S + x] > 0.0)) << (32 * half);
        }
        if (lane == 0) put(c, a, b);
    }
#else
    for (int c = tid; c <= t.n; c += nt) {
        unsigned long long a = 0ull, b = 0ull;
        for (int x = 0; x < t.n; ++x) {
            a |= static_cast<unsigned long long>(t.A[c * t.S + x] > 0.0) << x;
            b |= static_cast<unsigned long long>(t.B[c * t.S + x] > 0.0) << x;
        }
        put(c, a, b);
    }
#endif
}
SSB_TRI_HD void phase_counts(int tid, int nt, const Tables &t, const Counts &k) {
    // whole numbers, below 52^3
    auto w = [&](int c, int x) {
        return x >= t.n ? 0 : ((k.mB[c] >> x) & 1ull ? k.nA[x] : 0) + ((k.mA[c] >> x) & 1ull ? k.nB[x] : 0);
    };
    auto total = [&](int i, int c) {
        return c >= t.n ? 0 : i == 0 ? k.nA[c] : i == 1 ? k.nB[c] : i == 2 ? k.nA[c] * k.nB[c] : k.nD[c];
    };
    auto put = [&](int i, int s) { k.s[i] = i == 2 ? s : s / 2; };
#if defined(__CUDA_ARCH__)
    const int lane = tid & 31;   // a warp per sum
    for (int c = tid >> 5; c <= t.n + 4; c += nt >> 5) {
        const bool row = c <= t.n;
        const int i = c - t.n - 1;
        const int s = __reduce_add_sync(0xffffffffu, row ? w(c, lane) + w(c, lane + 32) : total(i, lane) + total(i, lane + 32));
        if (lane > 0) continue;
        if (row)
            k.nW[c] = s;
        else
            put(i, s);
    }
#else
    for (int c = tid; c <= t.n; c += nt) {
        int s = 0;
        for (int x = 0; x < t.n; ++x) s += w(c, x);
        k.nW[c] = s;
    }
    if (tid == nt - 1)
        for (int i = 0; i < 4; ++i) {
            int s = 0;
            for (int c = 0; c < t.n; ++c) s += total(i, c);
            put(i, s);
        }
#endif
}
template <class T>
SSB_TRI_HD bool tuple_with(int a, int b, const Counts &k, T r, int code) {
    if ((code & 0x10000) || !(r > T(0))) return false;
    const int s[4] = {a, b, (code >> 20) & 63, (code >> 26) & 63};
    if (s[2] == a || s[2] == b || s[3] == a || s[3] == b) return false;
    // pairs of the first two opponents avoiding the four cards
    long long fa = k.s[0], fb = k.s[1], q = k.s[2], e = k.s[3];
    for (int i = 0; i < 4; ++i) {
        const int c = s[i];
        int na = k.nA[c], nb = k.nB[c];
        fa -= na;
        fb -= nb;
        q -= k.nW[c];
        e -= k.nD[c];
        for (int j = 0; j < 4; ++j) {
            const int f = s[j];
            const int ab = static_cast<int>((k.mA[c] >> f) & 1ull), bb = static_cast<int>((k.mB[c] >> f) & 1ull);
            na -= ab;
            nb -= bb;
            q += popc(k.mA[c] & k.mB[f]);
            if (j > i) {
                fa += ab;
                fb += bb;
                e += ab & bb;
            }
        }
        q -= static_cast<long long>(na) * nb;
    }
    return fa * fb - q + e > 0;
}

// what one hand of the third opponent adds to the mass of {a, b}; exactly 0
// without a tuple
template <class T>
SSB_TRI_HD double tuple_mass(int a, int b, const Tables &t, const Counts &k, T r, int code) {
    if (!tuple_with(a, b, k, r, code)) return 0.0;
    return static_cast<double>(r) * pair_mass(a, b, (code >> 20) & 63, (code >> 26) & 63, t);
}

}  // namespace tri
}  // namespace ssb
