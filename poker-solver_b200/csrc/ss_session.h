// ss_session.h -- a resident subgame on one GPU (internal).
//
// The Session owns the plan, the device tables and state, and the CUDA graphs
// of one subgame; the batched and served forms (ss_batch.cu) drive many
// sessions with merged launches.
#pragma once

#include "ss_kernels.h"

#include <cuda_runtime.h>

#include <cstring>
#include <string>
#include <utility>
#include <vector>

namespace ssb {

// tuple visits of the enumeration kernel that one solve may spend
constexpr double kEnumLimitPerIter = 4e9;
constexpr double kEnumLimitTotal = 2e11;

enum ProfClass { PC_REACH = 0, PC_CFV, PC_FILL, PC_CR1, PC_CR2, PC_SD1, PC_ENUM, PC_OTHER };
inline int term_class(int kind) {
    switch (kind) {
        case TK_ZERO:
        case TK_LEAF0: return PC_FILL;
        case TK_CR1:
        case TK_CR1D: return PC_CR1;
        case TK_CR2: return PC_CR2;
        case TK_SD1:
        case TK_SD2:
        case TK_SD3: return PC_SD1;
        case TK_CR3:   // the class of terminals with three or more counted opponents
        default: return PC_ENUM;
    }
}

// A small subgame that is launched kernel by kernel (Session::crowded): one of
// more node-hand pairs (nodes x both ranges) than this level by level, a smaller
// one with its tree passes.  Eight sessions at once, microseconds per iteration
// of one with tree passes / by level: 6.4 / 18 (51 nodes, 2,162 hands: 110 K
// pairs), 14.9 / 24 (141, 2,162: 305 K), 32 / 22.6 (1,081, 2,256: 2.4 M).
constexpr double kLevelsAbove = 6e5;
// threads of its tree passes then: two blocks per SM
constexpr int kTreeBeside = 512;

// iterations of a captured graph where `iters` are run, at most `most`
int graph_length(int iters, int most);

class Session {
  public:
    Plan P;
    int device = 0;
    int graph_iters = 10;
    int iterations = 0;
    cudaStream_t stream = nullptr;
    char *dbase = nullptr;    // static tables
    float *dstate = nullptr;  // R, S, reach, val
    float *dleaf = nullptr;
    float *dsmall = nullptr;  // root strategy snapshot + root values
    int *diter = nullptr;
    size_t nR = 0, nReach = 0, nVal = 0, n_rs = 0;
    int frozen_root = -1;
    DevCtx c{};
    const ReachItem *reach_items[SS_MAX_PLAYERS] = {};
    std::vector<std::pair<int, int>> reach_lv[SS_MAX_PLAYERS];
    const CfvItem *cfv_items[SS_MAX_PLAYERS] = {};
    std::vector<std::pair<int, int>> cfv_lv[SS_MAX_PLAYERS];
    TreeRef tree[SS_MAX_PLAYERS] = {};
    SmallRef small{};         // small heads-up subgames: iterations in one cooperative kernel
    int small_blocks = 0;     // its grid; 0: the captured iterations run
    unsigned small_fault = 0; // its fault word as last read: set until the state is reset
    int sms = 0;
    cudaEvent_t ev_done = nullptr;   // after the iterations queued last (small subgames)
    bool in_flight = false;          // it was recorded and not yet seen to be reached (under the list's lock)
    const TermItem *term_items[SS_MAX_PLAYERS][TK_COUNT] = {};
    const int *term_heads[SS_MAX_PLAYERS][TK_COUNT] = {};   // null for kinds without P.term_heads
    const int *root_fr[SS_MAX_PLAYERS] = {};
    const int *dec_fe = nullptr, *dec_na = nullptr, *dec_pl = nullptr;
    std::vector<int> dec_na_host, dec_player_host;   // per decision node (index order): actions, acting player
    // per (player, level) / (traverser, kind) minimum bytes, for the profile
    std::vector<double> reach_bytes[SS_MAX_PLAYERS], cfv_bytes[SS_MAX_PLAYERS];
    double term_bytes[SS_MAX_PLAYERS][TK_COUNT] = {};
    cudaGraphExec_t graph = nullptr;   // graph_len iterations
    int graph_len = 0;
    int direct_done = 0;               // iterations launched without a graph while there was none
    // best response state (allocated on first use, ensure_br)
    std::vector<float> host_w;          // range weights [np][HS]
    double *dbr = nullptr;              // reach_d [E + np][HS], val_d [N + 1][HS]
    char *dbr_tab = nullptr;            // edge -> decision index, deal item, row list, scalars
    float *davg_br = nullptr;           // profile in the output layout
    const int *br_edge_di = nullptr;    // in dbr_tab: [E] decision index of each edge's node
    const TermItem *br_deal = nullptr;  // in dbr_tab: the deal-mass item (val_d row N)
    const int *br_row = nullptr;        // in dbr_tab: {N}
    double *br_sc = nullptr;            // in dbr_tab: root sums (nashconv_from_sums layout)
    TermItem deal{};
    int deal_kind = TK_ENUM;

    // profiling hook: when set, every launch is preceded by an event record
    struct Mark {
        int cls;
        double bytes;
        int items;
        cudaEvent_t ev;
    };
    std::vector<Mark> *marks = nullptr;
    std::vector<SSLaunchRecord> last_launches;   // per launch of the last profiled iteration

    // terminal kinds of one pass write disjoint value rows and only read
    // reach: in the captured iteration all but one run on side streams
    // (fork / join through events), so short kinds overlap the long one
    cudaStream_t side[TK_COUNT] = {};
    cudaEvent_t ev_fork = nullptr, ev_join[TK_COUNT] = {};

    ~Session() {
        leave_flights();
        if (graph) cudaGraphExecDestroy(graph);
        for (int k = 0; k < TK_COUNT; ++k) {
            if (side[k]) cudaStreamDestroy(side[k]);
            if (ev_join[k]) cudaEventDestroy(ev_join[k]);
        }
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (stream) {
            if (dbase) cudaFreeAsync(dbase, stream);
            if (dstate) cudaFreeAsync(dstate, stream);
            if (dleaf) cudaFreeAsync(dleaf, stream);
            if (dsmall) cudaFreeAsync(dsmall, stream);
            if (diter) cudaFreeAsync(diter, stream);
            if (dbr) cudaFreeAsync(dbr, stream);
            if (dbr_tab) cudaFreeAsync(dbr_tab, stream);
            if (davg_br) cudaFreeAsync(davg_br, stream);
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
    }

    cudaError_t mark(int cls, double bytes, int items = 0) {
        if (!marks) return cudaSuccess;
        Mark m{cls, bytes, items, nullptr};
        cudaError_t e = cudaEventCreate(&m.ev);
        if (e != cudaSuccess) return e;
        marks->push_back(m);
        // an external record becomes an event-record node of the captured graph
        return cudaEventRecordWithFlags(m.ev, stream, cudaEventRecordExternal);
    }

    // player p's reach levels from level `from` on
    cudaError_t reach(int p, size_t from = 0) {
        for (size_t l = from; l < reach_lv[p].size(); ++l) {
            cudaError_t e = mark(PC_REACH, reach_bytes[p][l], reach_lv[p][l].second);
            if (e == cudaSuccess)
                e = launch_reach(c, reach_items[p] + reach_lv[p][l].first, reach_lv[p][l].second,
                                 P.H[p], stream);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    // A small subgame is launched kernel by kernel only beside others (crowded),
    // so what counts there is the time on all SMs together: level by level, which
    // is spread over short blocks, unless the tree pass is short.
    bool levels() const { return small_blocks > 0 && P.node_hands > kLevelsAbove; }

    // Where traverser t has two-way showdowns, its one-opponent folds and zero
    // rows ride in their launch (rivers: tens of short blocks of each kind), as
    // long as that launch has large blocks.
    bool light(int t, int k) const {
        const size_t n = P.term[t][TK_SD1].size();
        return !levels() && n > 0 && n <= kSd1Few && (k == TK_SD1 || k == TK_CR1 || k == TK_ZERO);
    }

    // traverser t's terminals of kind k (grouped kinds: one block per head)
    cudaError_t terms(int t, int k, cudaStream_t s) {
        if (light(t, k))
            return launch_terms_light(c, term_items[t][TK_SD1], static_cast<int>(P.term[t][TK_SD1].size()),
                                      term_items[t][TK_CR1], static_cast<int>(P.term[t][TK_CR1].size()),
                                      term_items[t][TK_ZERO], static_cast<int>(P.term[t][TK_ZERO].size()), t, s);
        return launch_terms(c, k, term_items[t][k], static_cast<int>(P.term[t][k].size()), t, s, nullptr,
                            term_heads[t][k], static_cast<int>(P.term_heads[t][k].size()));
    }

    // The terminal launches of traverser t's pass, their bytes, and the one
    // with the most work, which stays on the session stream (relative block
    // times of full-range rivers and turns); returns their number.
    int launch_kinds(int t, int kinds[TK_COUNT], int *main_k, double by[TK_COUNT]) const {
        int nk = 0;
        double main_w = 0;
        for (int k = 0; k < TK_COUNT; ++k) {
            const int n = static_cast<int>(P.term[t][k].size());
            const int lk = light(t, k) ? static_cast<int>(TK_SD1) : k;
            by[lk] += term_bytes[t][k];
            if (n == 0 || lk != k) continue;
            kinds[nk++] = k;
            const double w = n * (k == TK_SD3 || k == TK_CR3 ? 64.0 : k == TK_SD2 || k == TK_ENUM ? 16.0 : 1.0);
            if (*main_k < 0 || w > main_w) {
                *main_k = k;
                main_w = w;
            }
        }
        return nk;
    }

    // the side streams and events that a captured iteration forks onto, made
    // when the first one is captured
    cudaError_t ensure_side() {
        cudaError_t e = cudaSuccess;
        for (int t = 0; t < P.np; ++t) {
            int kinds[TK_COUNT], main_k = -1;
            double by[TK_COUNT] = {};
            const int nk = launch_kinds(t, kinds, &main_k, by);
            if (nk <= 1) continue;
            if (!ev_fork) e = cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming);
            for (int i = 0; i < nk && e == cudaSuccess; ++i) {
                const int k = kinds[i];
                if (k == main_k || side[k]) continue;
                e = cudaStreamCreateWithFlags(&side[k], cudaStreamNonBlocking);
                if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev_join[k], cudaEventDisableTiming);
            }
            if (e != cudaSuccess) return e;
        }
        return e;
    }

    // traverser t's part of iteration *iter + iter_add
    cudaError_t pass(int t, bool snapshot_root, int iter_add) {
        cudaError_t e = cudaSuccess;
        if (snapshot_root) {
            e = mark(PC_OTHER, 0);
            if (e == cudaSuccess)
                e = launch_root_strategy(c, P.first_edge[0], P.root_na, frozen_root,
                                         P.H[P.root_player], dsmall, stream);
            if (e != cudaSuccess) return e;
        }
        int kinds[TK_COUNT], main_k = -1;
        double by[TK_COUNT] = {};
        const int nk = launch_kinds(t, kinds, &main_k, by);
        if (marks || nk <= 1) {
            // one kind after the other (the profile times each class)
            for (int i = 0; i < nk; ++i) {
                const int k = kinds[i];
                e = mark(term_class(k), by[k], static_cast<int>(P.term[t][k].size()));
                if (e == cudaSuccess) e = terms(t, k, stream);
                if (e != cudaSuccess) return e;
            }
        } else {
            e = cudaEventRecord(ev_fork, stream);
            for (int i = 0; i < nk && e == cudaSuccess; ++i) {
                const int k = kinds[i];
                if (k == main_k) continue;
                e = cudaStreamWaitEvent(side[k], ev_fork, 0);
                if (e == cudaSuccess) e = terms(t, k, side[k]);
                if (e == cudaSuccess) e = cudaEventRecord(ev_join[k], side[k]);
            }
            if (e == cudaSuccess) e = terms(t, main_k, stream);
            for (int i = 0; i < nk && e == cudaSuccess; ++i)
                if (kinds[i] != main_k) e = cudaStreamWaitEvent(stream, ev_join[kinds[i]], 0);
            if (e != cudaSuccess) return e;
        }
        // the large value/regret levels, then the small levels of values and
        // reach in one launch, then the large reach levels
        const TreePass &T = P.tree[t];
        const bool tree_pass = tree[t].n_stages > 0 && !levels();
        double tree_by = 0;
        int items = 0;
        for (size_t l = 0; l < cfv_lv[t].size(); ++l) {
            if (tree_pass && static_cast<int>(l) >= T.cfv_from) {
                tree_by += cfv_bytes[t][l];
                items += cfv_lv[t][l].second;
                continue;
            }
            e = mark(PC_CFV, cfv_bytes[t][l], cfv_lv[t][l].second);
            if (e == cudaSuccess)
                e = launch_cfv(c, cfv_items[t] + cfv_lv[t][l].first, cfv_lv[t][l].second, P.cfv_nlong[t][l],
                               P.H[t], stream, nullptr, -1, iter_add);
            if (e != cudaSuccess) return e;
        }
        if (tree_pass) {
            for (int l = 0; l < T.reach_to; ++l) tree_by += reach_bytes[t][l];
            e = mark(PC_CFV, tree_by, items);
            if (e == cudaSuccess) e = launch_tree(c, tree[t], P.H[t], stream, iter_add);
            if (e != cudaSuccess) return e;
        }
        return reach(t, tree_pass ? static_cast<size_t>(T.reach_to) : 0);
    }

    // iteration *iter + iter_add
    cudaError_t iteration(bool last, int iter_add) {
        cudaError_t e = cudaSuccess;
        for (int t = 0; t < P.np && e == cudaSuccess; ++t) e = pass(t, last && t == P.np - 1, iter_add);
        return e;
    }

    // `iters` iterations launched one by one; the last one's root strategy is
    // kept for the output
    cudaError_t direct(int iters, bool last) {
        cudaError_t e = ensure_side();
        for (int i = 0; i < iters && e == cudaSuccess; ++i) e = iteration(last && i == iters - 1, i + 1);
        if (e == cudaSuccess) e = mark(PC_OTHER, 0);
        if (e == cudaSuccess) e = launch_bump(diter, iters, stream);
        return e;
    }

    cudaError_t capture(int iters, bool last, cudaGraphExec_t *exec) {
        cudaGraph_t g = nullptr;
        cudaError_t e = ensure_side();
        if (e == cudaSuccess) e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return e;
        const cudaError_t body = direct(iters, last);
        e = cudaStreamEndCapture(stream, &g);
        if (body != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return body;
        }
        if (e != cudaSuccess) return e;
        e = cudaGraphInstantiate(exec, g, 0);
        cudaGraphDestroy(g);
        return e;
    }

    int init(const Problem &pb, const SolveConfig &cfg);
    int ensure_br();
    int exploitability(const float *host_avg, double *pct, double *nash, double *br, double *cur,
                       double *deal_mass);
    void nashconv_from_sums(const double *sc, double *pct, double *nash, double *br, double *cur,
                            double *deal_mass) const;
    int reset();
    int run(int iters);
    int run_launches(int iters);      // iterations kernel by kernel
    bool crowded();                   // small subgames: whether its grid does not fit beside those in flight
    int join_flights();               // marks what was just queued as in flight
    void leave_flights();
    int output(SSOutput *out);
    int sync();
    int small_fault_error();          // the error of a session whose wait ran out
    cudaError_t fetch_small_fault();  // queues the read of the fault word (small sessions)
    int profile(SSKernelProfile *prof);
    int profile_launches(SSLaunchRecord *rec, int max_records, int *num_records) const;
};

}  // namespace ssb
