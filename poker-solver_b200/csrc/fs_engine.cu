// fs_engine.cu -- the multi-street two-player solver on the GPU.
//
// The reference (flop_solve.cu:974-1270) keeps reach and values per node for
// every hand, re-runs regret matching over all decision nodes and
// re-propagates the opponent's reach through every level for each traverser,
// and launches one kernel per tree level and kind with a host sync per
// iteration.  Here the street solver's machinery carries over:
//   * reach is stored per sequence (one row per decision edge): a chance node
//     deals a card but changes no player's reach, so it is transparent, and a
//     player's reach is re-propagated once per iteration, after its own
//     regret update (k_reach, regret matching fused in);
//   * values are written only for terminals and the traverser's decision
//     nodes; an edge's value is the sum of its frontier rows -- through the
//     opponent's decisions and through chance nodes, whose average becomes a
//     weight 1 / cards dealt folded into each frontier row when it is written
//     (the items' `scale`), so k_cfv sums rows unchanged;
//   * terminals: sums per card and in strength order over the opponent's reach
//     row, then O(1) per traverser hand; one warp per terminal with the ranges'
//     tables or the river board's in the block's shared memory, one block per
//     terminal where a launch has few;
//   * strengths and the tables by strength: once per solve for every river
//     board of the tree on the device (k_fs_tables), instead of once per
//     showdown node;
//   * iterations are captured as CUDA graphs with the counter on the device.
// fs_solve_gpu_extract_all reads the average strategy of every node and the
// last traverser's values at every node (terminals, both players' decisions,
// chance averages) from the same solve: the strategy of the last pass is kept
// for the read-out.
#include "fs_engine.h"
#include "ss_kernels.h"
#include "ss_rank.cuh"
#include "ss_stage.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>

namespace ssb {
namespace fs {

// ---------------------------------------------------------------------------
// planner
// ---------------------------------------------------------------------------

namespace {

bool fail(const std::string &m) {
    set_error("fs: " + m);
    return false;
}

bool validate(const FSTreeData &td, FsPlan &P) {
    if (!td.nodes || !td.children || td.num_nodes < 1) return fail("tree has no nodes");
    for (int p = 0; p < 2; ++p) {
        if (td.num_hands[p] < 0 || td.num_hands[p] > FS_MAX_HANDS) return fail("num_hands must be 0..200");
        P.H[p] = td.num_hands[p];
        for (int h = 0; h < P.H[p]; ++h) {
            const int a = td.hands[p][h][0], b = td.hands[p][h][1];
            if (a < 0 || a > 51 || b < 0 || b > 51 || a == b) return fail("hands must be two distinct cards 0..51");
        }
    }
    P.max_h = std::max(P.H[0], P.H[1]);
    if (P.max_h == 0) return fail("both ranges are empty");
    for (int i = 0; i < td.num_nodes; ++i) {
        const FSNode &n = td.nodes[i];
        if (n.num_board < 3 || n.num_board > 5) return fail("node board must hold 3..5 cards");
        if (n.type == FS_NODE_DECISION || n.type == FS_NODE_CHANCE) {
            if (n.num_children < 1 || n.first_child < 0 || n.first_child + n.num_children > td.num_children_total)
                return fail("node " + std::to_string(i) + " has bad children");
            if (n.type == FS_NODE_DECISION && (n.num_children > FS_MAX_ACTIONS || n.player < 0 || n.player > 1))
                return fail("decision node " + std::to_string(i) + " needs a player and 1..6 actions");
            for (int a = 0; a < n.num_children; ++a) {
                const int c = td.children[n.first_child + a];
                if (c <= 0 || c >= td.num_nodes) return fail("child id out of range");
            }
        } else if (n.type == FS_NODE_FOLD) {
            if (n.player < 0 || n.player > 1 || n.num_children != 0) return fail("fold node without a winner");
        } else if (n.type == FS_NODE_SHOWDOWN) {
            if (n.num_board != 5 || n.num_children != 0) return fail("showdown before the river");
        } else {
            return fail("unknown node type");
        }
        for (int b = 0; b < n.num_board; ++b)
            if (n.board_cards[b] < 0 || n.board_cards[b] > 51) return fail("board card out of range");
    }
    if (td.nodes[0].type != FS_NODE_DECISION) return fail("node 0 must be a decision node");
    return true;
}

}  // namespace

int build_plan(const FSTreeData &td, FsPlan *out) {
    FsPlan &P = *out;
    if (!validate(td, P)) return SS_ERR_INVALID;
    const int N = td.num_nodes;
    P.N = N;
    P.HS = (P.max_h + 31) / 32 * 32;
    const FSNode *nd = td.nodes;
    auto child = [&](int x, int a) { return td.children[nd[x].first_child + a]; };
    // breadth-first order; every node reached once
    std::vector<int> order{0}, parent(N, -2), pact(N, -1), depth(N, 0);
    parent[0] = -1;
    for (size_t q = 0; q < order.size(); ++q) {
        const int x = order[q];
        if (nd[x].type != FS_NODE_DECISION && nd[x].type != FS_NODE_CHANCE) continue;
        for (int a = 0; a < nd[x].num_children; ++a) {
            const int c = child(x, a);
            if (parent[c] != -2) {
                set_error("fs: node " + std::to_string(c) + " is reached twice: not a tree");
                return SS_ERR_INVALID;
            }
            parent[c] = x;
            pact[c] = a;
            depth[c] = depth[x] + 1;
            order.push_back(c);
        }
    }
    if (static_cast<int>(order.size()) != N) {
        set_error("fs: some nodes are not reachable from node 0");
        return SS_ERR_INVALID;
    }
    P.root_player = nd[0].player;
    P.root_na = nd[0].num_children;
    P.first_edge.assign(N, -1);
    P.edge_node.clear();
    for (int x : order)
        if (nd[x].type == FS_NODE_DECISION) {
            P.first_edge[x] = static_cast<int>(P.edge_node.size());
            for (int a = 0; a < nd[x].num_children; ++a) P.edge_node.push_back(x);
        }
    P.E = static_cast<int>(P.edge_node.size());
    const int E = P.E;
    for (int i = 0; i < N; ++i)
        if (nd[i].type == FS_NODE_DECISION) P.dec_nodes.push_back(i);
    // each player's sequence (reach row) and own-decision depth at every node
    std::vector<int> last(2 * static_cast<size_t>(N)), pdepth(2 * static_cast<size_t>(N), 0);
    for (int x : order)
        for (int p = 0; p < 2; ++p) {
            if (x == 0) {
                last[p] = E + p;
                continue;
            }
            const int par = parent[x];
            const bool acted = nd[par].type == FS_NODE_DECISION && nd[par].player == p;
            last[2 * x + p] = acted ? P.first_edge[par] + pact[x] : last[2 * par + p];
            pdepth[2 * x + p] = pdepth[2 * par + p] + (acted ? 1 : 0);
        }
    for (int p = 0; p < 2; ++p)
        for (int x : order) {
            if (nd[x].type != FS_NODE_DECISION || nd[x].player != p) continue;
            const int lev = pdepth[2 * x + p];
            if (static_cast<int>(P.reach_levels[p].size()) <= lev) P.reach_levels[p].resize(lev + 1);
            ReachItem it;
            it.first_edge = P.first_edge[x];
            it.na = nd[x].num_children;
            it.parent_row = last[2 * x + p];
            it.frozen = -1;
            P.reach_levels[p][lev].push_back(it);
        }
    // frontiers: through the other player's decisions and through chance nodes
    P.fr_off.assign(E + 1, 0);
    std::vector<int> stack;
    for (int e = 0; e < E; ++e) {
        const int x = P.edge_node[e], p = nd[x].player;
        stack.assign(1, child(x, e - P.first_edge[x]));
        while (!stack.empty()) {
            const int y = stack.back();
            stack.pop_back();
            const bool pass = nd[y].type == FS_NODE_CHANCE || (nd[y].type == FS_NODE_DECISION && nd[y].player != p);
            if (!pass) {
                P.fr_items.push_back(y);
                continue;
            }
            for (int a = nd[y].num_children - 1; a >= 0; --a) stack.push_back(child(y, a));
        }
        P.fr_off[e + 1] = static_cast<int>(P.fr_items.size());
    }
    // per traverser: the chance weight of every node within its frontier
    // (1 below a traverser decision, divided by the cards at each chance node)
    std::vector<double> w(N);
    for (int t = 0; t < 2; ++t) {
        for (int x : order) {
            if (x == 0) {
                w[x] = 1.0;
                continue;
            }
            const int par = parent[x];
            w[x] = nd[par].type == FS_NODE_DECISION && nd[par].player == t ? 1.0
                   : nd[par].type == FS_NODE_CHANCE ? w[par] / nd[par].num_children
                                                    : w[par];
        }
        // value / regret levels: height in own decisions, bottom-up
        std::vector<int> height(N, 0);
        P.cfv_levels[t].clear();
        for (int q = N - 1; q >= 0; --q) {
            const int x = order[q];
            if (nd[x].type != FS_NODE_DECISION || nd[x].player != t) continue;
            int h = 0;
            const int fe = P.first_edge[x];
            for (int k = P.fr_off[fe]; k < P.fr_off[fe + nd[x].num_children]; ++k) {
                const int y = P.fr_items[k];
                if (nd[y].type == FS_NODE_DECISION) h = std::max(h, height[y] + 1);
            }
            height[x] = h;
            if (static_cast<int>(P.cfv_levels[t].size()) <= h) P.cfv_levels[t].resize(h + 1);
            CfvItem it;
            it.first_edge = fe;
            it.na = nd[x].num_children;
            it.frozen = -1;
            it.node = x;
            it.scale = static_cast<float>(w[x]);
            inline_frontier(it, P.fr_off, P.fr_items);
            P.cfv_levels[t][h].push_back(it);
        }
        P.cfv_nlong[t].assign(P.cfv_levels[t].size(), 0);
        for (size_t l = 0; l < P.cfv_levels[t].size(); ++l) {
            P.cfv_nlong[t][l] = order_cfv_level(P.cfv_levels[t][l], [&](const CfvItem &it) {
                return P.fr_off[it.first_edge + it.na] - P.fr_off[it.first_edge];
            });
        }
    }
    // river boards of the showdowns, and the terminal items
    const float half_start = static_cast<float>(nd[0].pot) * 0.5f;   // flop_solve.cu:755
    std::vector<int> board_row(N, -1);
    {
        std::vector<long long> keys;
        for (int x = 0; x < N; ++x)
            if (nd[x].type == FS_NODE_SHOWDOWN) {
                long long k = 0;
                for (int b = 0; b < 5; ++b) k = k * 64 + nd[x].board_cards[b];
                keys.push_back(k);
            }
        std::vector<long long> uk = keys;
        std::sort(uk.begin(), uk.end());
        uk.erase(std::unique(uk.begin(), uk.end()), uk.end());
        for (long long k : uk)   // card b is base-64 digit 4 - b
            for (int b = 0; b < 5; ++b) P.sboards.push_back(static_cast<int>((k >> (6 * (4 - b))) & 63));
        for (int x = 0; x < N; ++x)
            if (nd[x].type == FS_NODE_SHOWDOWN) {
                long long k = 0;
                for (int b = 0; b < 5; ++b) k = k * 64 + nd[x].board_cards[b];
                board_row[x] = static_cast<int>(std::lower_bound(uk.begin(), uk.end(), k) - uk.begin());
            }
    }
    // each board's first showdown item
    P.bstart.assign(P.sboards.size() / 5 + 1, 0);
    int n_fold = 0;
    for (int x = 0; x < N; ++x) {
        n_fold += nd[x].type == FS_NODE_FOLD;
        if (board_row[x] >= 0) ++P.bstart[board_row[x] + 1];
    }
    for (size_t b = 1; b < P.bstart.size(); ++b) P.bstart[b] += P.bstart[b - 1];
    for (int t = 0; t < 2; ++t) {
        // chance weights for traverser t again (the loop above kept t = 1's)
        for (int x : order) {
            if (x == 0) {
                w[x] = 1.0;
                continue;
            }
            const int par = parent[x];
            w[x] = nd[par].type == FS_NODE_DECISION && nd[par].player == t ? 1.0
                   : nd[par].type == FS_NODE_CHANCE ? w[par] / nd[par].num_children
                                                    : w[par];
        }
        // folds first, then showdowns by river board (one launch each)
        P.term[t].resize(static_cast<size_t>(n_fold) + P.bstart.back());
        int fold_at = 0;
        std::vector<int> sd_at(P.bstart);
        for (int x = 0; x < N; ++x) {
            const FSNode &n = nd[x];
            if (n.type != FS_NODE_FOLD && n.type != FS_NODE_SHOWDOWN) continue;
            FsTermItem it;
            std::memset(&it, 0, sizeof(it));
            it.node = x;
            it.kind = n.type == FS_NODE_FOLD ? 0 : 1;
            it.opp_row = last[2 * x + (1 - t)];
            it.sboard = board_row[x];
            if (n.type == FS_NODE_FOLD) {
                const int winner = n.player, loser = 1 - winner;
                it.payoff = t == winner ? half_start + static_cast<float>(n.bets[loser])
                                        : -(half_start + static_cast<float>(n.bets[t]));
            }
            it.half_pot = static_cast<float>(n.pot) * 0.5f;
            it.scale = static_cast<float>(w[x]);
            it.nb = n.num_board;
            for (int b = 0; b < n.num_board; ++b) it.board[b] = n.board_cards[b];
            P.term[t][n.type == FS_NODE_FOLD ? fold_at++ : n_fold + sd_at[board_row[x]]++] = it;
        }
        P.nfold[t] = n_fold;
    }
    // hands, and per player the hands holding each card (folds)
    const int HSi = P.HS;
    P.hand_cards.assign(2 * static_cast<size_t>(HSi), -1);
    for (int p = 0; p < 2; ++p)
        for (int h = 0; h < P.H[p]; ++h) P.hand_cards[p * HSi + h] = td.hands[p][h][0] | (td.hands[p][h][1] << 8);
    P.f_coff.assign(2 * 53, 0);
    P.f_clist.assign(2 * 2 * static_cast<size_t>(HSi), 0);
    for (int p = 0; p < 2; ++p) {
        std::vector<std::vector<int>> byc(52);
        for (int h = 0; h < P.H[p]; ++h) {
            byc[td.hands[p][h][0]].push_back(h);
            byc[td.hands[p][h][1]].push_back(h);
        }
        int at = 0;
        for (int c = 0; c < 52; ++c) {
            P.f_coff[p * 53 + c] = at;
            for (int h : byc[c]) P.f_clist[p * 2 * HSi + at++] = h;
        }
        P.f_coff[p * 53 + 52] = at;
    }
    // each hand's combo in the opponent's range (where combos repeat, the last)
    P.f_same.assign(2 * static_cast<size_t>(HSi), -1);
    for (int p = 0; p < 2; ++p) {
        std::vector<int> of(52 * 52, -1);
        P.dup[p] = 0;
        for (int h = 0; h < P.H[p]; ++h) {
            const int a = td.hands[p][h][0], b = td.hands[p][h][1];
            if (of[a * 52 + b] >= 0) P.dup[p] = 1;
            of[a * 52 + b] = of[b * 52 + a] = h;
        }
        for (int h = 0; h < P.H[1 - p]; ++h)
            P.f_same[(1 - p) * HSi + h] = of[td.hands[1 - p][h][0] * 52 + td.hands[1 - p][h][1]];
    }
    // read-out levels: BFS depth, deepest first
    int maxd = 0;
    for (int x = 0; x < N; ++x) maxd = std::max(maxd, depth[x]);
    P.depth_off.assign(maxd + 2, 0);
    std::vector<std::vector<int>> byd(maxd + 1);
    for (int x : order) byd[depth[x]].push_back(x);
    for (int d = maxd; d >= 0; --d) {
        P.depth_nodes.insert(P.depth_nodes.end(), byd[d].begin(), byd[d].end());
        P.depth_off[maxd - d + 1] = static_cast<int>(P.depth_nodes.size());
    }
    return SS_OK;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

namespace {

constexpr int kFsThreads = 256;

struct FsTables {
    const int *hand_cards;                    // [2][HS]
    const int *f_coff, *f_clist;              // [2][53], [2][2 HS]
    const int *f_same;                        // [2][HS]: the opponent's hand of the same two cards, -1 if none
    int dup[2];                               // the player's range repeats a combo
    const unsigned *sd_str;                   // [nsb][2][HS]
    const int *sd_ord, *sd_hpos, *sd_coff, *sd_clist;
    int HS, H0, H1;
};

// The showdown tables of every river board (layouts in fs_engine.h), one block
// per board, straight into device memory: 7-card strengths, then positions,
// card lists and the traverser's bounds by counting over the at most 200 hands
// of each player in shared memory (200 broadcast reads per entry).  On the
// host the same tables (2,352 boards, 200 hands: 34 MB) took 300 ms of sorting
// and the copy; here they are not worth a mention beside one iteration.
struct FsTableOut {
    unsigned *str;
    int *ord, *hpos, *coff, *clist;
};
__global__ void __launch_bounds__(kFsThreads) k_fs_tables(const int *__restrict__ boards,
                                                         const int *__restrict__ hand_cards, FsTableOut O, int HS,
                                                         int H0, int H1) {
    __shared__ unsigned st[2][FS_MAX_HANDS];
    __shared__ int cd[2][FS_MAX_HANDS];
    __shared__ short pos[2][FS_MAX_HANDS];
    __shared__ int off[2][53];
    const int tid = threadIdx.x;
    const size_t row = static_cast<size_t>(blockIdx.x) * 2;
    const size_t hs = static_cast<size_t>(HS);
    const int H[2] = {H0, H1};
    int bd[5];
    for (int i = 0; i < 5; ++i) bd[i] = __ldg(boards + 5 * blockIdx.x + i);
    static_assert(FS_MAX_HANDS <= kFsThreads, "one thread per hand");
    for (int p = 0; p < 2; ++p)
        if (tid < H[p]) {
            const int code = __ldg(hand_cards + p * HS + tid);
            const int c[7] = {bd[0], bd[1], bd[2], bd[3], bd[4], code & 0xff, (code >> 8) & 0xff};
            bool repeat = false;
            for (int i = 0; i < 7; ++i)
                for (int j = i + 1; j < 7; ++j) repeat |= c[i] == c[j];
            const unsigned v = repeat ? 0u : rank7(c);
            st[p][tid] = v;
            cd[p][tid] = code;
            O.str[(row + p) * hs + tid] = v;
        }
    __syncthreads();
    // positions by ascending strength, ties in hand order
    for (int p = 0; p < 2; ++p)
        if (tid < H[p]) {
            const unsigned v = st[p][tid];
            int k = 0;
            for (int j = 0; j < H[p]; ++j) k += st[p][j] < v || (st[p][j] == v && j < tid);
            pos[p][tid] = static_cast<short>(k);
            O.ord[(row + p) * hs + k] = tid;
        }
    // hands per card
    if (tid < 2 * 52) {
        const int p = tid / 52, c = tid - p * 52;
        int n = 0;
        for (int j = 0; j < H[p]; ++j) n += (cd[p][j] & 0xff) == c || ((cd[p][j] >> 8) & 0xff) == c;
        off[p][c + 1] = n;
    }
    __syncthreads();
    if (tid < 2) {
        off[tid][0] = 0;
        for (int c = 0; c < 52; ++c) off[tid][c + 1] += off[tid][c];
    }
    __syncthreads();
    if (tid < 2 * 53) O.coff[row * 53 + tid] = off[tid / 53][tid % 53];
    for (int p = 0; p < 2; ++p)
        if (tid < H[p]) {
            // this hand's place in the lists of its two cards (as the opponent)
            const int c1 = cd[p][tid] & 0xff, c2 = (cd[p][tid] >> 8) & 0xff, k = pos[p][tid];
            int k1 = 0, k2 = 0;
            for (int j = 0; j < H[p]; ++j) {
                const int x = cd[p][j] & 0xff, y = (cd[p][j] >> 8) & 0xff;
                const bool before = pos[p][j] < k;
                k1 += before && (x == c1 || y == c1);
                k2 += before && (x == c2 || y == c2);
            }
            O.clist[(row + p) * 2 * hs + off[p][c1] + k1] = k;
            O.clist[(row + p) * 2 * hs + off[p][c2] + k2] = k;
            // its bounds among the opponent's hands (as the traverser)
            const int o = 1 - p;
            const unsigned v = st[p][tid];
            int lo = 0, hi = 0, l1 = 0, h1 = 0, l2 = 0, h2 = 0;
            for (int j = 0; j < H[o]; ++j) {
                const int x = cd[o][j] & 0xff, y = (cd[o][j] >> 8) & 0xff;
                const bool w = st[o][j] < v, we = st[o][j] <= v;
                const bool on1 = x == c1 || y == c1, on2 = x == c2 || y == c2;
                lo += w;
                hi += we;
                l1 += w && on1;
                h1 += we && on1;
                l2 += w && on2;
                h2 += we && on2;
            }
            reinterpret_cast<int4 *>(O.hpos)[(row + p) * hs + tid] =
                make_int4(lo | (hi << 16), c1 | (c2 << 8), l1 | (h1 << 16), l2 | (h2 << 16));
        }
}

// Terminals, where a launch has many: one warp per terminal and no block
// barriers (a block per terminal spends its time waiting at three of them: 764 us
// for 113,488 folds, 640 us for 152,880 showdowns of 200 hands; a warp each 182
// and 374 us).  What the terminals of a block share
// sits in shared memory: the ranges' tables (folds), one river board's tables
// (showdowns).  Every sum keeps a fixed order: positions or hands in runs per
// lane, lists in list order.
constexpr int kFsWarps = kFsThreads / 32;
constexpr int kFsRun = (FS_MAX_HANDS + 31) / 32;   // hands or positions per lane

// Folds (flop_solve.cu:731-779): payoff x the opponent's reach over hands
// sharing no card with the traverser's hand {a, b} or with the node's board.
// Per terminal: the opponent's hands the board leaves; per card c their sums
// u(c), and F in all; then per traverser hand
//   mass = F - u(a) - u(b) + (the opponent's reach on the combo {a, b}),
// the last term by the table of equal combos (or, in a range that repeats a
// combo, from the opponent's list of card a).  The same sums over 0/1
// count the opponent hands with positive reach; none gives exactly 0, as the
// reference's sum of zeros does.
__global__ void __launch_bounds__(kFsThreads) k_fs_fold(const FsTermItem *__restrict__ items, int n, int trav,
                                                       const float *__restrict__ reach, FsTables T,
                                                       float *__restrict__ out, int scaled) {
    __shared__ unsigned long long mask_o[FS_MAX_HANDS];
    __shared__ short list[2 * FS_MAX_HANDS], off[53], same_t[FS_MAX_HANDS];
    __shared__ unsigned char ca[FS_MAX_HANDS], cb[FS_MAX_HANDS];
    __shared__ double r_w[kFsWarps][FS_MAX_HANDS];
    __shared__ double u_w[kFsWarps][52];
    __shared__ int cu_w[kFsWarps][52];
    const int opp = 1 - trav;
    const int Ho = opp == 0 ? T.H0 : T.H1, Ht = trav == 0 ? T.H0 : T.H1;
    const size_t hs = static_cast<size_t>(T.HS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool dup = T.dup[opp] != 0;
    if (tid < Ho) {
        const int code = T.hand_cards[opp * T.HS + tid];
        mask_o[tid] = (1ull << (code & 0xff)) | (1ull << ((code >> 8) & 0xff));
    }
    if (tid < Ht) {
        const int code = T.hand_cards[trav * T.HS + tid];
        ca[tid] = static_cast<unsigned char>(code & 0xff);
        cb[tid] = static_cast<unsigned char>((code >> 8) & 0xff);
        same_t[tid] = static_cast<short>(T.f_same[trav * T.HS + tid]);
    }
    if (tid < 53) off[tid] = static_cast<short>(T.f_coff[opp * 53 + tid]);
    for (int k = tid; k < 2 * Ho; k += kFsThreads) list[k] = static_cast<short>(T.f_clist[opp * 2 * T.HS + k]);
    __syncthreads();
    double *r_o = r_w[warp], *u = u_w[warp];
    int *cu = cu_w[warp];
    for (int i = blockIdx.x * kFsWarps + warp; i < n; i += gridDim.x * kFsWarps) {
        const FsTermItem I = items[i];
        unsigned long long board = 0ull;
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (k < I.nb) board |= 1ull << I.board[k];
        const float *row = reach + static_cast<size_t>(I.opp_row) * hs;
        float x[kFsRun];
#pragma unroll
        for (int g = 0; g < kFsRun; ++g) x[g] = g * 32 + lane < Ho ? row[g * 32 + lane] : 0.f;
        double F = 0.0;
        int CF = 0;
#pragma unroll
        for (int g = 0; g < kFsRun; ++g) {
            const int o = g * 32 + lane;
            const bool on = o < Ho && !(mask_o[o] & board);
            double f = on ? static_cast<double>(x[g]) : 0.0;
            if (o < Ho) r_o[o] = f;
            CF += __popc(__ballot_sync(0xffffffffu, f > 0.0));
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) f += __shfl_xor_sync(0xffffffffu, f, k);
            F += f;
        }
        __syncwarp();
        for (int c = lane; c < 52; c += 32) {
            double s = 0.0;
            int m = 0;
            for (int k = off[c]; k < off[c + 1]; ++k) {
                const double r = r_o[list[k]];
                s += r;
                m += r > 0.0 ? 1 : 0;
            }
            u[c] = s;
            cu[c] = m;
        }
        __syncwarp();
        const float sc = scaled ? I.scale : 1.0f;
        float *dst = out + static_cast<size_t>(I.node) * hs;
        for (int h = lane; h < Ht; h += 32) {
            const int a = ca[h], b = cb[h];
            double same = 0.0;
            int csame = 0;
            if (!dup) {
                const int o = same_t[h];
                if (o >= 0) {
                    same = r_o[o];
                    csame = same > 0.0 ? 1 : 0;
                }
            } else {
                for (int k = off[a]; k < off[a + 1]; ++k) {
                    const int o = list[k];
                    if (!(mask_o[o] >> b & 1ull)) continue;
                    same += r_o[o];
                    csame += r_o[o] > 0.0 ? 1 : 0;
                }
            }
            const int cnt = CF - cu[a] - cu[b] + csame;
            const double mass = cnt == 0 ? 0.0 : F - u[a] - u[b] + same;
            dst[h] = static_cast<float>(mass) * I.payoff * sc;
        }
        __syncwarp();
    }
}

// Showdowns (flop_solve.cu:781-833): +-half_pot per opponent hand that is
// weaker / stronger, ties 0, hands the board blocks 0.  With the opponent's
// hands in ascending strength on this river board, W = the reach below the
// traverser hand's strength and L = above it, each less the opponent hands
// holding one of its two cards (their own prefix sums along each card's
// list); value = (W - L) x half_pot, FP64 sums.  The same on 0/1 counts
// gives exactly 0 where no positive-reach opponent hand wins or loses.
// A river board's terminals [bstart[b], bstart[b + 1]) are consecutive items,
// shared by `split` blocks (a tree from the turn or the river on has few boards
// with many terminals each).
//
// Bound by shared-memory wavefronts, so the zero test keeps no counts beside
// the sums: a W or L above 1e-9 of the opponent's whole reach cannot be the
// rounding of an empty set (a few hundred roundings of 1e-16), an exact 0 is
// the answer either way, and only what lies between is looked up exactly, as
// 7 words of positive positions against the card masks of the board.
struct FsSdWarp {
    double P[FS_MAX_HANDS + 1];
    double PC[2 * FS_MAX_HANDS + 52];
    float x[FS_MAX_HANDS];
};
constexpr size_t fs_sd_smem() {
    return FS_MAX_HANDS * sizeof(int4) + kFsWarps * sizeof(FsSdWarp) + 52 * kFsRun * sizeof(unsigned) +
           (FS_MAX_HANDS + 2 * FS_MAX_HANDS + 64 + FS_MAX_HANDS) * sizeof(short) + 16;
}
__global__ void __launch_bounds__(kFsThreads) k_fs_showdown(const FsTermItem *__restrict__ items,
                                                           const int *__restrict__ bstart, int split, int trav,
                                                           const float *__restrict__ reach, FsTables T,
                                                           float *__restrict__ out, int scaled) {
    extern __shared__ __align__(16) char smem[];
    int4 *hpos = reinterpret_cast<int4 *>(smem);                               // [Ht]
    FsSdWarp *all = reinterpret_cast<FsSdWarp *>(hpos + FS_MAX_HANDS);
    unsigned *cmask = reinterpret_cast<unsigned *>(all + kFsWarps);             // [52][kFsRun] positions holding a card
    short *ord = reinterpret_cast<short *>(cmask + 52 * kFsRun);                // [Ho], -1 where the board blocks it
    short *list = ord + FS_MAX_HANDS, *off = list + 2 * FS_MAX_HANDS;           // [2 Ho], [53]
    short *live = off + 64;                                                     // [Ht]
    const int opp = 1 - trav;
    const int Ho = opp == 0 ? T.H0 : T.H1, Ht = trav == 0 ? T.H0 : T.H1;
    const size_t hs = static_cast<size_t>(T.HS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int board = blockIdx.x / split, share = blockIdx.x - board * split;
    const int first = bstart[board] + share * kFsWarps, end = bstart[board + 1];
    if (first >= end) return;
    const size_t bo = static_cast<size_t>(board) * 2 + opp, bt = static_cast<size_t>(board) * 2 + trav;
    for (int i = tid; i < 52 * kFsRun; i += kFsThreads) cmask[i] = 0u;
    if (tid < Ho) {
        const int o = T.sd_ord[bo * hs + tid];
        ord[tid] = static_cast<short>(T.sd_str[bo * hs + o] == 0u ? -1 : o);
    }
    if (tid < Ht) {
        hpos[tid] = reinterpret_cast<const int4 *>(T.sd_hpos)[bt * hs + tid];
        live[tid] = T.sd_str[bt * hs + tid] != 0u;
    }
    if (tid < 53) off[tid] = static_cast<short>(T.sd_coff[bo * 53 + tid]);
    for (int k = tid; k < 2 * Ho; k += kFsThreads) list[k] = static_cast<short>(T.sd_clist[bo * 2 * hs + k]);
    __syncthreads();
    // position k is bit k / kFsRun of word k % kFsRun (the warp's ballots below)
    if (tid < 52)
        for (int k = off[tid]; k < off[tid + 1]; ++k) cmask[tid * kFsRun + list[k] % kFsRun] |= 1u << (list[k] / kFsRun);
    __syncthreads();
    FsSdWarp &W = all[warp];
    for (int i = first + warp; i < end; i += split * kFsWarps) {
        const FsTermItem &I = items[i];
        const float *row = reach + static_cast<size_t>(I.opp_row) * hs;
        // the opponent's reach by position (0 where the board blocks the
        // hand): each lane a run of consecutive positions
        const int k0 = lane * kFsRun;
        float x[kFsRun];
        unsigned live_k[kFsRun];
#pragma unroll
        for (int j = 0; j < kFsRun; ++j) {
            const int o = k0 + j < Ho ? ord[k0 + j] : -1;
            x[j] = o >= 0 ? row[o] : 0.f;
        }
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < kFsRun; ++j) {
            live_k[j] = __ballot_sync(0xffffffffu, x[j] > 0.f);
            if (k0 + j < Ho) {
                W.x[k0 + j] = x[j];
                s += static_cast<double>(x[j]);
            }
        }
        // prefix sums over positions: lane totals scanned across the warp
        // (fixed order), then along each lane's run
        double incl = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += v;
        }
        double run = incl - s;
#pragma unroll
        for (int j = 0; j < kFsRun; ++j)
            if (k0 + j < Ho) {
                W.P[k0 + j] = run;
                run += static_cast<double>(x[j]);
            }
        const double total = __shfl_sync(0xffffffffu, incl, 31);
        if (lane == 31) W.P[Ho] = incl;
        __syncwarp();
        // per card: prefix sums along the opponent's hands holding it
        for (int c = lane; c < 52; c += 32) {
            const int b0 = off[c], b1 = off[c + 1];
            double q = 0.0;
            W.PC[b0 + c] = 0.0;
            for (int k = b0; k < b1; ++k) {
                q += static_cast<double>(W.x[list[k]]);
                W.PC[k + c + 1] = q;
            }
        }
        __syncwarp();
        // whether an opponent hand of positive reach at a position in
        // [from, to) holds neither c1 nor c2
        auto any_in = [&](int c1, int c2, int from, int to) {
            unsigned hit = 0u;
#pragma unroll
            for (int j = 0; j < kFsRun; ++j) {
                const int nf = max(0, (from - j + kFsRun - 1) / kFsRun), nt = max(0, (to - j + kFsRun - 1) / kFsRun);
                const unsigned in = ((nt >= 32 ? 0u : 1u << nt) - 1u) & ~((nf >= 32 ? 0u : 1u << nf) - 1u);
                hit |= live_k[j] & in & ~cmask[c1 * kFsRun + j] & ~cmask[c2 * kFsRun + j];
            }
            return hit != 0u;
        };
        bool odd = false;   // a negative or NaN reach voids the bound: look everything up
#pragma unroll
        for (int j = 0; j < kFsRun; ++j) odd |= !(x[j] >= 0.f);
        const double zb = __any_sync(0xffffffffu, odd) ? __longlong_as_double(0x7ff0000000000000ll) : 1e-9 * total;
        const float sc = scaled ? I.scale : 1.0f;
        const double half_pot = static_cast<double>(I.half_pot);
        float *dst = out + static_cast<size_t>(I.node) * hs;
        for (int h = lane; h < Ht; h += 32) {
            float v = 0.f;
            if (live[h]) {
                const int4 hp = hpos[h];
                const int lo = hp.x & 0xffff, hi = hp.x >> 16;
                const int c1 = hp.y & 0xff, c2 = (hp.y >> 8) & 0xff;
                const int b1 = off[c1] + c1, e1 = off[c1 + 1] + c1;
                const int b2 = off[c2] + c2, e2 = off[c2 + 1] + c2;
                const int l1lo = hp.z & 0xffff, l1hi = hp.z >> 16, l2lo = hp.w & 0xffff, l2hi = hp.w >> 16;
                double w = W.P[lo] - W.PC[b1 + l1lo] - W.PC[b2 + l2lo];
                double l = (total - W.P[hi]) - (W.PC[e1] - W.PC[b1 + l1hi]) - (W.PC[e2] - W.PC[b2 + l2hi]);
                if (w != 0.0 && !(fabs(w) > zb) && !any_in(c1, c2, 0, lo)) w = 0.0;
                if (l != 0.0 && !(fabs(l) > zb) && !any_in(c1, c2, hi, Ho)) l = 0.0;
                v = static_cast<float>((w - l) * half_pot);
            }
            dst[h] = v * sc;
        }
        __syncwarp();
    }
}

// The same values (same sums, same order) by a block per terminal, for launches
// of few of them, which wait for one terminal and not for all: the hands and
// the cards of a terminal are spread over the block, and nothing is brought to
// shared memory but what the terminal computes.
__global__ void __launch_bounds__(kFsThreads) k_fs_fold_few(const FsTermItem *__restrict__ items, int trav,
                                                           const float *__restrict__ reach, FsTables T,
                                                           float *__restrict__ out, int scaled) {
    __shared__ double r_o[FS_MAX_HANDS];
    __shared__ double u[52], tot[kFsWarps];
    __shared__ int cu[52], ctot[kFsWarps];
    const FsTermItem I = items[blockIdx.x];
    const int opp = 1 - trav;
    const int Ho = opp == 0 ? T.H0 : T.H1, Ht = trav == 0 ? T.H0 : T.H1;
    const size_t hs = static_cast<size_t>(T.HS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int *cl = T.f_clist + opp * 2 * T.HS, *coff = T.f_coff + opp * 53;
    double f = 0.0;
    if (tid < Ho) {
        const int code = T.hand_cards[opp * T.HS + tid];
        const float r = reach[static_cast<size_t>(I.opp_row) * hs + tid];
        bool blocked = false;
        for (int k = 0; k < I.nb; ++k) blocked |= (code & 0xff) == I.board[k] || ((code >> 8) & 0xff) == I.board[k];
        f = blocked ? 0.0 : static_cast<double>(r);
        r_o[tid] = f;
    }
    const int hc = tid < Ht ? T.hand_cards[trav * T.HS + tid] : 0, so = tid < Ht ? T.f_same[trav * T.HS + tid] : -1;
    const int n = __popc(__ballot_sync(0xffffffffu, f > 0.0));
    for (int k = 16; k > 0; k >>= 1) f += __shfl_xor_sync(0xffffffffu, f, k);
    if (lane == 0) {
        tot[warp] = f;
        ctot[warp] = n;
    }
    __syncthreads();
    if (tid < 52) {
        double s = 0.0;
        int m = 0;
        for (int k = coff[tid]; k < coff[tid + 1]; ++k) {
            const double r = r_o[cl[k]];
            s += r;
            m += r > 0.0 ? 1 : 0;
        }
        u[tid] = s;
        cu[tid] = m;
    }
    __syncthreads();
    static_assert(FS_MAX_HANDS <= kFsThreads, "a thread per hand");
    if (tid >= Ht) return;
    double F = 0.0;
    int CF = 0;
    for (int w = 0; w < kFsRun; ++w) {
        F += tot[w];
        CF += ctot[w];
    }
    const int a = hc & 0xff, b = (hc >> 8) & 0xff;
    double same = 0.0;
    int csame = 0;
    if (!T.dup[opp]) {
        same = so >= 0 ? r_o[so] : 0.0;
        csame = same > 0.0 ? 1 : 0;
    } else {
        for (int k = coff[a]; k < coff[a + 1]; ++k) {
            const int o = cl[k], oc = T.hand_cards[opp * T.HS + o];
            if ((oc & 0xff) != b && ((oc >> 8) & 0xff) != b) continue;
            same += r_o[o];
            csame += r_o[o] > 0.0 ? 1 : 0;
        }
    }
    const int cnt = CF - cu[a] - cu[b] + csame;
    const double mass = cnt == 0 ? 0.0 : F - u[a] - u[b] + same;
    out[static_cast<size_t>(I.node) * hs + tid] = static_cast<float>(mass) * I.payoff * (scaled ? I.scale : 1.0f);
}

__global__ void __launch_bounds__(kFsThreads) k_fs_showdown_few(const FsTermItem *__restrict__ items, int trav,
                                                               const float *__restrict__ reach, FsTables T,
                                                               float *__restrict__ out, int scaled) {
    __shared__ double P[FS_MAX_HANDS + 1], PC[2 * FS_MAX_HANDS + 52];
    __shared__ int Pn[FS_MAX_HANDS + 1], PCn[2 * FS_MAX_HANDS + 52];   // the same sums over positive reach
    __shared__ float x_s[32 * kFsRun];
    const FsTermItem &I = items[blockIdx.x];
    const int opp = 1 - trav;
    const int Ho = opp == 0 ? T.H0 : T.H1, Ht = trav == 0 ? T.H0 : T.H1;
    const size_t hs = static_cast<size_t>(T.HS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t bo = static_cast<size_t>(I.sboard) * 2 + opp, bt = static_cast<size_t>(I.sboard) * 2 + trav;
    const int *coff = T.sd_coff + bo * 53;
    // the opponent's reach by position (0 where the board blocks the hand)
    if (tid < 32 * kFsRun) {
        const int o = tid < Ho ? T.sd_ord[bo * hs + tid] : -1;
        x_s[tid] = o >= 0 && T.sd_str[bo * hs + o] != 0u ? reach[static_cast<size_t>(I.opp_row) * hs + o] : 0.f;
    }
    const bool live = tid < Ht && T.sd_str[bt * hs + tid] != 0u;
    const int4 hp = live ? reinterpret_cast<const int4 *>(T.sd_hpos)[bt * hs + tid] : make_int4(0, 0, 0, 0);
    static_assert(32 * kFsRun <= kFsThreads && FS_MAX_HANDS <= kFsThreads, "a thread per hand");
    __syncthreads();
    if (warp == 0) {
        const int k0 = lane * kFsRun;
        double s = 0.0;
        int n = 0;
#pragma unroll
        for (int j = 0; j < kFsRun; ++j) {
            s += static_cast<double>(x_s[k0 + j]);
            n += x_s[k0 + j] > 0.f ? 1 : 0;
        }
        double incl = s;
        int nincl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, d);
            const int m = __shfl_up_sync(0xffffffffu, nincl, d);
            if (lane >= d) {
                incl += v;
                nincl += m;
            }
        }
        double run = incl - s;
        int nrun = nincl - n;
#pragma unroll
        for (int j = 0; j < kFsRun; ++j)
            if (k0 + j < Ho) {
                P[k0 + j] = run;
                Pn[k0 + j] = nrun;
                run += static_cast<double>(x_s[k0 + j]);
                nrun += x_s[k0 + j] > 0.f ? 1 : 0;
            }
        if (lane == 31) {
            P[Ho] = incl;
            Pn[Ho] = nincl;
        }
    } else if (tid >= 64 && tid < 64 + 52) {
        const int c = tid - 64, b0 = coff[c], b1 = coff[c + 1];
        const int *cl = T.sd_clist + bo * 2 * hs;
        double q = 0.0;
        int m = 0;
        PC[b0 + c] = 0.0;
        PCn[b0 + c] = 0;
        for (int k = b0; k < b1; ++k) {
            const float v = x_s[cl[k]];
            q += static_cast<double>(v);
            m += v > 0.f ? 1 : 0;
            PC[k + c + 1] = q;
            PCn[k + c + 1] = m;
        }
    }
    __syncthreads();
    if (tid >= Ht) return;
    float v = 0.f;
    if (live) {
        const int lo = hp.x & 0xffff, hi = hp.x >> 16;
        const int c1 = hp.y & 0xff, c2 = (hp.y >> 8) & 0xff;
        const int b1 = coff[c1] + c1, e1 = coff[c1 + 1] + c1;
        const int b2 = coff[c2] + c2, e2 = coff[c2 + 1] + c2;
        const int l1lo = hp.z & 0xffff, l1hi = hp.z >> 16, l2lo = hp.w & 0xffff, l2hi = hp.w >> 16;
        double w = P[lo] - PC[b1 + l1lo] - PC[b2 + l2lo];
        double l = (P[Ho] - P[hi]) - (PC[e1] - PC[b1 + l1hi]) - (PC[e2] - PC[b2 + l2hi]);
        if (Pn[lo] - PCn[b1 + l1lo] - PCn[b2 + l2lo] == 0) w = 0.0;
        if ((Pn[Ho] - Pn[hi]) - (PCn[e1] - PCn[b1 + l1hi]) - (PCn[e2] - PCn[b2 + l2hi]) == 0) l = 0.0;
        v = static_cast<float>((w - l) * static_cast<double>(I.half_pot));
    }
    out[static_cast<size_t>(I.node) * hs + tid] = v * (scaled ? I.scale : 1.0f);
}

// Terminals of a launch up to which each has a block.  Microseconds per launch
// by block / by warp, 200 hands: folds 3.6 / 5.6 at 4, 5.1 / 6.1 at 292, 6.3 /
// 6.1 at 484, 40 / 13.9 at 5,596; showdowns 3.7 / 9.5 at 5, 8.6 / 15.4 at 1,296,
// 18.2 / 21.1 at 3,792, 30.7 / 30.0 at 6,480, 72 / 63 at 16,656.  40 hands: folds
// 4.4 / 4.4 at 292, showdowns 9.3 / 9.6 at 3,120, 17.2 / 13.4 at 6,480.
constexpr int kFsFewFolds = 2 * 148, kFsFewShowdowns = 4096;
// blocks that share a river board's showdowns: as many as it takes to have two
// per SM, while a warp gets a terminal or more
inline int fs_split(int showdowns, int boards) {
    return std::max(1, std::min((2 * 148 + boards - 1) / boards, showdowns / (boards * kFsWarps)));
}

// the regret-matched strategy of every decision node of player p into
// sig [E][HS] (the read-out keeps the last pass's strategy)
__global__ void k_fs_sigma(const float *__restrict__ R, const int *__restrict__ edge_first,
                           const int *__restrict__ edge_na, int E, int HS, int H, float *__restrict__ sig) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= E * HS) return;
    const int e = i / HS, h = i - e * HS;
    if (h >= H) return;
    const int fe = edge_first[e], na = edge_na[e];
    float sum = 0.f;
    for (int a = 0; a < na; ++a) {
        const float r = R[static_cast<size_t>(fe + a) * HS + h];
        sum += r > 0.f ? r : 0.f;
    }
    const float r = R[i];
    sig[i] = sum > 0.f ? (r > 0.f ? r : 0.f) * (1.0f / sum) : 1.0f / static_cast<float>(na);
}

// one level of the read-out: every node's value for traverser t from its
// children (terminals were written by k_fs_fold / k_fs_showdown): the traverser's decisions
// weight by its last-pass strategy, the opponent's sum, chance nodes average
// (flop_solve.cu:835-892 order: children in order, then the division)
__global__ void k_fs_value_level(const FSNode *__restrict__ nodes, const int *__restrict__ children,
                                 const int *__restrict__ lev, int n, const int *__restrict__ first_edge,
                                 const float *__restrict__ sig, int trav, int HS, int H, float *__restrict__ val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * HS) return;
    const int x = lev[i / HS], h = i % HS;
    if (h >= H) return;
    const FSNode nd = nodes[x];
    if (nd.type != FS_NODE_DECISION && nd.type != FS_NODE_CHANCE) return;
    const size_t hs = static_cast<size_t>(HS);
    float v = 0.f;
    for (int a = 0; a < nd.num_children; ++a) {
        const float cv = val[static_cast<size_t>(children[nd.first_child + a]) * hs + h];
        if (nd.type == FS_NODE_DECISION && nd.player == trav)
            v += sig[static_cast<size_t>(first_edge[x] + a) * hs + h] * cv;
        else
            v += cv;
    }
    if (nd.type == FS_NODE_CHANCE) v = v / static_cast<float>(nd.num_children);
    val[static_cast<size_t>(x) * hs + h] = v;
}

#define FCK(call)                                                                     \
    do {                                                                              \
        cudaError_t e_ = (call);                                                      \
        if (e_ != cudaSuccess) {                                                      \
            set_error(std::string("CUDA: ") + cudaGetErrorString(e_) + " at " #call); \
            return e_ == cudaErrorMemoryAllocation ? SS_ERR_NOMEM : SS_ERR_CUDA;      \
        }                                                                             \
    } while (0)

struct Blob {
    std::vector<char> host;
    size_t add(const void *src, size_t bytes) {
        size_t off = (host.size() + 255) & ~static_cast<size_t>(255);
        host.resize(off + bytes);
        if (bytes && src) std::memcpy(host.data() + off, src, bytes);
        return off;
    }
    template <class T>
    size_t add(const std::vector<T> &v) {
        return add(v.data(), v.size() * sizeof(T));
    }
};

// one solve's device state and launch lists
class Solve {
  public:
    FsPlan P;
    cudaStream_t stream = nullptr;
    char *dbase = nullptr, *dtab = nullptr;
    float *dstate = nullptr;
    int *diter = nullptr;
    float *dsnap = nullptr;
    float *dsig = nullptr, *dval = nullptr;   // read-out
    DevCtx c{};
    const ReachItem *reach_items[2] = {};
    std::vector<std::pair<int, int>> reach_lv[2], cfv_lv[2];
    const CfvItem *cfv_items[2] = {};
    const FsTermItem *term_items[2] = {};
    const int *hand_cards = nullptr, *edge_first = nullptr, *edge_na = nullptr, *depth_nodes = nullptr;
    FsTables tab{};
    const int *bstart = nullptr;
    FSNode *dnodes = nullptr;
    int *dchildren = nullptr;
    const int *dfirst_edge = nullptr;
    cudaGraphExec_t gblock = nullptr;
    int block_iters = 10;

    ~Solve() {
        if (gblock) cudaGraphExecDestroy(gblock);
        if (stream) {
            for (void *p : {static_cast<void *>(dbase), static_cast<void *>(dtab), static_cast<void *>(dstate),
                            static_cast<void *>(diter), static_cast<void *>(dsnap), static_cast<void *>(dsig),
                            static_cast<void *>(dval), static_cast<void *>(dnodes), static_cast<void *>(dchildren)})
                if (p) cudaFreeAsync(p, stream);
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
    }

    int init(const FSTreeData &td) {
        int rc = build_plan(td, &P);
        if (rc != SS_OK) return rc;
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
            set_error("no CUDA device");
            return SS_ERR_NO_DEVICE;
        }
        FCK(cudaSetDevice(0));
        FCK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        const size_t HS = static_cast<size_t>(P.HS), E = static_cast<size_t>(P.E), N = static_cast<size_t>(P.N);
        Blob b;
        size_t o_reach[2], o_cfv[2], o_term[2];
        for (int p = 0; p < 2; ++p) {
            std::vector<ReachItem> all;
            for (auto &lv : P.reach_levels[p]) {
                reach_lv[p].push_back({static_cast<int>(all.size()), static_cast<int>(lv.size())});
                all.insert(all.end(), lv.begin(), lv.end());
            }
            o_reach[p] = b.add(all);
            std::vector<CfvItem> call;
            for (auto &lv : P.cfv_levels[p]) {
                cfv_lv[p].push_back({static_cast<int>(call.size()), static_cast<int>(lv.size())});
                call.insert(call.end(), lv.begin(), lv.end());
            }
            o_cfv[p] = b.add(call);
            o_term[p] = b.add(P.term[p]);
        }
        std::vector<int> ef(E), ena(E);
        for (size_t e = 0; e < E; ++e) {
            ef[e] = P.first_edge[P.edge_node[e]];
            ena[e] = td.nodes[P.edge_node[e]].num_children;
        }
        const size_t o_fro = b.add(P.fr_off), o_fri = b.add(P.fr_items), o_hc = b.add(P.hand_cards),
                     o_ef = b.add(ef), o_ena = b.add(ena), o_dn = b.add(P.depth_nodes), o_fe = b.add(P.first_edge),
                     o_fco = b.add(P.f_coff), o_fcl = b.add(P.f_clist), o_sbd = b.add(P.sboards), o_fsm = b.add(P.f_same), o_bst = b.add(P.bstart);
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&dbase), std::max<size_t>(b.host.size(), 256), stream));
        FCK(stage_upload(dbase, b.host.data(), b.host.size(), stream));
        for (int p = 0; p < 2; ++p) {
            reach_items[p] = reinterpret_cast<const ReachItem *>(dbase + o_reach[p]);
            cfv_items[p] = reinterpret_cast<const CfvItem *>(dbase + o_cfv[p]);
            term_items[p] = reinterpret_cast<const FsTermItem *>(dbase + o_term[p]);
        }
        hand_cards = reinterpret_cast<const int *>(dbase + o_hc);
        tab.hand_cards = hand_cards;
        tab.f_coff = reinterpret_cast<const int *>(dbase + o_fco);
        tab.f_clist = reinterpret_cast<const int *>(dbase + o_fcl);
        // the showdown tables: [boards][2 players][...], made on the device
        const size_t rows = P.sboards.size() / 5 * 2;
        if (rows > 0) {
            FsTableOut O{};
            size_t at = 0;
            auto take = [&](size_t ints) {
                const size_t off = at;
                at += (ints * sizeof(int) + 255) / 256 * 256;
                return off;
            };
            const size_t t_str = take(rows * HS), t_ord = take(rows * HS), t_hpos = take(rows * HS * 4),
                         t_coff = take(rows * 53), t_clist = take(rows * 2 * HS);
            FCK(cudaMallocAsync(reinterpret_cast<void **>(&dtab), at, stream));
            O.str = reinterpret_cast<unsigned *>(dtab + t_str);
            O.ord = reinterpret_cast<int *>(dtab + t_ord);
            O.hpos = reinterpret_cast<int *>(dtab + t_hpos);
            O.coff = reinterpret_cast<int *>(dtab + t_coff);
            O.clist = reinterpret_cast<int *>(dtab + t_clist);
            k_fs_tables<<<static_cast<unsigned>(rows / 2), kFsThreads, 0, stream>>>(
                reinterpret_cast<const int *>(dbase + o_sbd), hand_cards, O, P.HS, P.H[0], P.H[1]);
            FCK(cudaGetLastError());
            tab.sd_str = O.str;
            tab.sd_ord = O.ord;
            tab.sd_hpos = O.hpos;
            tab.sd_coff = O.coff;
            tab.sd_clist = O.clist;
        }
        tab.f_same = reinterpret_cast<const int *>(dbase + o_fsm);
        tab.dup[0] = P.dup[0];
        tab.dup[1] = P.dup[1];
        bstart = reinterpret_cast<const int *>(dbase + o_bst);
        tab.HS = P.HS;
        tab.H0 = P.H[0];
        tab.H1 = P.H[1];
        edge_first = reinterpret_cast<const int *>(dbase + o_ef);
        edge_na = reinterpret_cast<const int *>(dbase + o_ena);
        depth_nodes = reinterpret_cast<const int *>(dbase + o_dn);
        dfirst_edge = reinterpret_cast<const int *>(dbase + o_fe);
        // state: regrets, strategy sums, reach (weights in the last 2 rows), values
        const size_t nR = E * HS, nReach = (E + 2) * HS, nVal = N * HS;
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&dstate), (2 * nR + nReach + nVal) * sizeof(float), stream));
        FCK(cudaMemsetAsync(dstate, 0, (2 * nR + nReach + nVal) * sizeof(float), stream));
        c.R = dstate;
        c.S = c.R + nR;
        c.reach = c.S + nR;
        c.val = c.reach + nReach;
        std::vector<float> w(2 * HS, 0.f);
        for (int p = 0; p < 2; ++p)
            for (int h = 0; h < P.H[p]; ++h) w[p * HS + h] = td.weights[p][h];
        FCK(cudaMemcpyAsync(c.reach + E * HS, w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice, stream));
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&diter), sizeof(int), stream));
        FCK(cudaMemsetAsync(diter, 0, sizeof(int), stream));
        const int nrs = P.root_na * std::max(1, P.H[P.root_player]);
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&dsnap), nrs * sizeof(float), stream));
        FCK(cudaMemsetAsync(dsnap, 0, nrs * sizeof(float), stream));
        c.fr_off = reinterpret_cast<const int *>(dbase + o_fro);
        c.fr_items = reinterpret_cast<const int *>(dbase + o_fri);
        c.iter = diter;
        c.HS = P.HS;
        c.np = 2;
        c.H[0] = P.H[0];
        c.H[1] = P.H[1];
        FCK(cudaStreamSynchronize(stream));   // host staging must outlive the copies
        // all regrets 0: uniform play
        for (int p = 0; p < 2; ++p) FCK(reach(p));
        return SS_OK;
    }

    cudaError_t reach(int p) {
        for (auto &lv : reach_lv[p]) {
            cudaError_t e = launch_reach(c, reach_items[p] + lv.first, lv.second, P.H[p], stream);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    cudaError_t terms(int t, float *out, int scaled) {
        const int nf = P.nfold[t], ns = static_cast<int>(P.term[t].size()) - nf, boards = static_cast<int>(P.bstart.size()) - 1;
        if (nf > 0 && nf <= kFsFewFolds) {
            k_fs_fold_few<<<nf, kFsThreads, 0, stream>>>(term_items[t], t, c.reach, tab, out, scaled);
        } else if (nf > 0) {
            // eight resident blocks per SM, each over many terminals
            const int grid = std::min((nf + kFsWarps - 1) / kFsWarps, 8 * 148);
            k_fs_fold<<<grid, kFsThreads, 0, stream>>>(term_items[t], nf, t, c.reach, tab, out, scaled);
        }
        if (ns > 0 && ns <= kFsFewShowdowns) {
            k_fs_showdown_few<<<ns, kFsThreads, 0, stream>>>(term_items[t] + nf, t, c.reach, tab, out, scaled);
        } else if (ns > 0) {
            cudaError_t e = cudaFuncSetAttribute(k_fs_showdown, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(fs_sd_smem()));
            if (e != cudaSuccess) return e;
            k_fs_showdown<<<boards * fs_split(ns, boards), kFsThreads, fs_sd_smem(), stream>>>(
                term_items[t] + nf, bstart, fs_split(ns, boards), t, c.reach, tab, out, scaled);
        }
        return cudaGetLastError();
    }

    // one iteration: per traverser terminals, values and regrets bottom-up,
    // then its reach; the root strategy is taken before the last traverser's
    // pass (the reference's last regret matching)
    cudaError_t iteration(bool keep_sigma) {
        cudaError_t e = launch_bump(diter, 1, stream);
        for (int t = 0; t < 2 && e == cudaSuccess; ++t) {
            if (t == 1) {
                e = launch_root_strategy(c, P.first_edge[0], P.root_na, -1, P.H[P.root_player], dsnap, stream);
                if (e == cudaSuccess && keep_sigma && P.E > 0) {
                    const int n = P.E * P.HS;
                    k_fs_sigma<<<(n + 255) / 256, 256, 0, stream>>>(c.R, edge_first, edge_na, P.E, P.HS, P.H[1], dsig);
                    e = cudaGetLastError();
                }
            }
            if (e == cudaSuccess) e = terms(t, c.val, 1);
            for (size_t l = 0; l < cfv_lv[t].size() && e == cudaSuccess; ++l)
                e = launch_cfv(c, cfv_items[t] + cfv_lv[t][l].first, cfv_lv[t][l].second, P.cfv_nlong[t][l], P.H[t],
                               stream);
            if (e == cudaSuccess) e = reach(t);
        }
        return e;
    }

    int run(int iters, bool keep_sigma_last) {
        int done = 0;
        const int graph_part = keep_sigma_last ? iters - 1 : iters;
        if (graph_part >= block_iters) {
            cudaGraph_t g = nullptr;
            FCK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
            cudaError_t body = cudaSuccess;
            for (int i = 0; i < block_iters && body == cudaSuccess; ++i) body = iteration(false);
            cudaError_t e = cudaStreamEndCapture(stream, &g);
            if (body != cudaSuccess) {
                if (g) cudaGraphDestroy(g);
                FCK(body);
            }
            FCK(e);
            e = cudaGraphInstantiate(&gblock, g, 0);
            cudaGraphDestroy(g);
            FCK(e);
            for (; done + block_iters <= graph_part; done += block_iters) FCK(cudaGraphLaunch(gblock, stream));
        }
        for (; done < iters; ++done) FCK(iteration(keep_sigma_last && done == iters - 1));
        FCK(cudaStreamSynchronize(stream));
        return SS_OK;
    }

    // the last traverser's value at every node under the last pass's strategy
    int readout() {
        const int t = 1;
        FCK(terms(t, dval, 0));
        const int L = static_cast<int>(P.depth_off.size()) - 1;
        for (int l = 0; l < L; ++l) {
            const int n = P.depth_off[l + 1] - P.depth_off[l];
            const int tot = n * P.HS;
            k_fs_value_level<<<(tot + 255) / 256, 256, 0, stream>>>(dnodes, dchildren, depth_nodes + P.depth_off[l], n,
                                                                   dfirst_edge, dsig, t, P.HS, P.H[t], dval);
            FCK(cudaGetLastError());
        }
        FCK(cudaStreamSynchronize(stream));
        return SS_OK;
    }
};

}  // namespace

int solve(FSTreeData *td, int iterations, FSOutput *out, bool extract) {
    std::memset(out, 0, sizeof(*out));
    if (!td) {
        set_error("fs_solve_gpu: no tree");
        return SS_ERR_INVALID;
    }
    if (iterations < 1) {
        set_error("fs_solve_gpu: max_iterations must be >= 1");
        return SS_ERR_INVALID;
    }
    Solve s;
    int rc = s.init(*td);
    if (rc != SS_OK) return rc;
    const FsPlan &P = s.P;
    const size_t HS = static_cast<size_t>(P.HS), N = static_cast<size_t>(P.N), mh = static_cast<size_t>(P.max_h);
    if (extract) {
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&s.dsig), std::max<size_t>(1, P.E * HS) * sizeof(float), s.stream));
        FCK(cudaMemsetAsync(s.dsig, 0, std::max<size_t>(1, P.E * HS) * sizeof(float), s.stream));
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&s.dval), N * HS * sizeof(float), s.stream));
        FCK(cudaMemsetAsync(s.dval, 0, N * HS * sizeof(float), s.stream));
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&s.dnodes), N * sizeof(FSNode), s.stream));
        FCK(cudaMemcpyAsync(s.dnodes, td->nodes, N * sizeof(FSNode), cudaMemcpyHostToDevice, s.stream));
        FCK(cudaMallocAsync(reinterpret_cast<void **>(&s.dchildren),
                            std::max(1, td->num_children_total) * sizeof(int), s.stream));
        FCK(cudaMemcpyAsync(s.dchildren, td->children, td->num_children_total * sizeof(int), cudaMemcpyHostToDevice,
                            s.stream));
    }
    rc = s.run(iterations, extract);
    if (rc != SS_OK) return rc;
    const int nrh = P.H[P.root_player];
    FSOutput o{};
    o.root_num_actions = P.root_na;
    o.root_player = P.root_player;
    o.root_strategy = static_cast<float *>(std::malloc(std::max(1, P.root_na * nrh) * sizeof(float)));
    if (!o.root_strategy) {
        set_error("fs_solve_gpu: out of host memory");
        return SS_ERR_NOMEM;
    }
    FCK(cudaMemcpy(o.root_strategy, s.dsnap, P.root_na * nrh * sizeof(float), cudaMemcpyDeviceToHost));
    if (extract) {
        rc = s.readout();
        if (rc != SS_OK) {
            free_output(&o);
            return rc;
        }
        o.max_hands = P.max_h;
        o.all_avg_strategies = static_cast<float *>(std::calloc(N * FS_MAX_ACTIONS * mh, sizeof(float)));
        o.all_cfv = static_cast<float *>(std::malloc(std::max<size_t>(1, N * mh) * sizeof(float)));
        std::vector<float> S(P.E * HS), V(N * HS);
        if (!o.all_avg_strategies || !o.all_cfv) {
            free_output(&o);
            set_error("fs_solve_gpu_extract_all: out of host memory");
            return SS_ERR_NOMEM;
        }
        FCK(cudaMemcpy(S.data(), s.c.S, S.size() * sizeof(float), cudaMemcpyDeviceToHost));
        FCK(cudaMemcpy(V.data(), s.dval, V.size() * sizeof(float), cudaMemcpyDeviceToHost));
        for (size_t x = 0; x < N; ++x)
            for (size_t h = 0; h < mh; ++h) o.all_cfv[x * mh + h] = h < static_cast<size_t>(P.H[1]) ? V[x * HS + h] : 0.f;
        // normalised strategy sums at every decision node (flop_solve.cu:1516-1540)
        for (int x : P.dec_nodes) {
            const FSNode &n = td->nodes[x];
            const int fe = P.first_edge[x], na = n.num_children;
            float *dst = o.all_avg_strategies + static_cast<size_t>(x) * FS_MAX_ACTIONS * mh;
            for (int h = 0; h < P.H[n.player]; ++h) {
                float sum = 0.f;
                for (int a = 0; a < na; ++a) {
                    const float v = S[(fe + a) * HS + h];
                    sum += v > 0.f ? v : 0.f;
                }
                for (int a = 0; a < na; ++a) {
                    const float v = S[(fe + a) * HS + h];
                    dst[a * mh + h] = sum > 0.f ? (v > 0.f ? v * (1.0f / sum) : 0.f) : 1.0f / static_cast<float>(na);
                }
            }
        }
        // turn roots: the decision children of the flop-ending chance nodes
        std::vector<int> roots, cards;
        for (int x = 0; x < P.N; ++x) {
            const FSNode &n = td->nodes[x];
            if (n.type != FS_NODE_CHANCE || n.num_board != 3) continue;
            for (int a = 0; a < n.num_children; ++a) {
                const int ch = td->children[n.first_child + a];
                if (td->nodes[ch].type == FS_NODE_DECISION) {
                    roots.push_back(ch);
                    cards.push_back(td->nodes[ch].board_cards[3]);
                }
            }
        }
        o.turn_root_indices = static_cast<int *>(std::malloc(std::max<size_t>(1, roots.size()) * sizeof(int)));
        o.turn_root_cards = static_cast<int *>(std::malloc(std::max<size_t>(1, roots.size()) * sizeof(int)));
        if (!o.turn_root_indices || !o.turn_root_cards) {
            free_output(&o);
            set_error("fs_solve_gpu_extract_all: out of host memory");
            return SS_ERR_NOMEM;
        }
        std::copy(roots.begin(), roots.end(), o.turn_root_indices);
        std::copy(cards.begin(), cards.end(), o.turn_root_cards);
        o.num_turn_roots = static_cast<int>(roots.size());
    }
    *out = o;
    return SS_OK;
}

void free_output(FSOutput *o) {
    if (!o) return;
    std::free(o->root_strategy);
    std::free(o->root_ev);
    std::free(o->all_avg_strategies);
    std::free(o->all_cfv);
    std::free(o->turn_root_indices);
    std::free(o->turn_root_cards);
    std::memset(o, 0, sizeof(*o));
}

}  // namespace fs
}  // namespace ssb
