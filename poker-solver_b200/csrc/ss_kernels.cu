// ss_kernels.cu -- sm_100a kernels of the single-street Linear-CFR solver.
//
// Per-hand kernels, over rows of HS floats (HS a multiple of 32): reach in
// units of one work item and 256 hands, four to a block, four consecutive hands
// per thread (128-bit loads and stores); values and regrets one pair of hands
// per thread, items back to back; the small levels near the root in one launch
// with eight hands per block (k_tree); a small heads-up subgame's whole
// iterations in one cooperative kernel (k_small_solve).
//
// Per-terminal kernels: one block per terminal node (several for a long
// showdown sweep or a large range).  The block stages the
// counted opponents' reach at that node in shared memory as 52x52 combo
// matrices (or as a strength-sorted vector for showdowns), reduces them to
// per-card aggregates, and then evaluates the exact card-removal formula for
// every traverser hand in O(1) (plus one small matrix product for two
// opponents).  The reference enumerates opponent tuples per traverser hand
// instead (street_solve.cu:704-1130), which is O(H^k).
#include "ss_kernels.h"

#include <algorithm>
#include <cstddef>
#include <cstdlib>
#include "ss_cr3.cuh"
#include "ss_triple.cuh"

namespace ssb {

// Device fault word: a kernel that gives up a bounded wait on the tensor
// cores, or gets a block it was not built for, records it here instead of
// trapping; the host reads and clears it after a solve (read_device_fault).
__device__ unsigned g_ss_fault = 0;

namespace {

constexpr unsigned kFaultTcInput = 1u;   // k_term_cr2_tc: a subgame outside its path
constexpr unsigned kFaultTcWait = 2u;    // k_term_cr2_tc: the MMA completion wait ran out

constexpr int MS = 52;  // shared-memory row stride of a 52x52 combo matrix (16-byte rows)

// Programmatic dependent launch: the kernels of an iteration are launched
// with it (pdl_launch), so a kernel's blocks are scheduled while the kernel
// before it in the stream drains.  Every kernel starts here:
// griddepcontrol.wait returns once the preceding kernel has completed and its
// writes are visible (at once when there is no programmatic predecessor).
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t pdl_launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                       A &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
// pdl_launch(kernel, grid, block, shared bytes, stream, kernel arguments...),
// returning its error from the enclosing function
#define SSB_LAUNCH(...)                                      \
    do {                                                     \
        const cudaError_t le_ = pdl_launch(__VA_ARGS__);     \
        if (le_ != cudaSuccess) return le_;                  \
    } while (0)

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float get(const float4 &v, int i) {
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Regret matching for 4 hands at one node (street_solve.cu:596-613): positive
// regrets normalised by their sum (multiplied by the float reciprocal), uniform
// when no regret is positive; an A3-frozen node plays its frozen action for
// every hand (street_solve.cu:641-643).  The reference's pruning branch only
// maps regrets below -1e4 to 0, which the positive part already does.
// r receives the raw regrets.
__device__ __forceinline__ void regret_match4(const float *__restrict__ R, size_t HS, int fe,
                                              int na, int frozen, int h0,
                                              float r[SS_MAX_ACTIONS][4],
                                              float sig[SS_MAX_ACTIONS][4]) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
        if (a < na) {
            const float4 v = ld4(R + static_cast<size_t>(fe + a) * HS + h0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                r[a][i] = get(v, i);
                sum[i] += r[a][i] > 0.f ? r[a][i] : 0.f;
            }
        }
    }
    const float uni = 1.0f / static_cast<float>(na);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool pos = sum[i] > 0.f;
        const float inv = pos ? 1.0f / sum[i] : 0.f;
#pragma unroll
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
            if (a < na) {
                float s = pos ? (r[a][i] > 0.f ? r[a][i] : 0.f) * inv : uni;
                if (frozen >= 0) s = (a == frozen) ? 1.0f : 0.0f;
                sig[a][i] = s;
            }
        }
    }
}

// regret-matched (and frozen) strategy of one node, out[na][H]
// (street_solve.cu:1564-1573), by nt threads
__device__ __forceinline__ void root_strategy(const float *__restrict__ R, size_t HS, int fe, int na, int frozen, int H,
                                              float *out, int tid, int nt) {
    for (int h0 = tid * 4; h0 < H; h0 += nt * 4) {
        float r[SS_MAX_ACTIONS][4], sig[SS_MAX_ACTIONS][4];
        regret_match4(R, HS, fe, na, frozen, h0, r, sig);
        for (int a = 0; a < na; ++a)
            for (int i = 0; i < 4; ++i)
                if (h0 + i < H) out[static_cast<size_t>(a) * H + h0 + i] = sig[a][i];
    }
}

// --------------------------------------------------------------------------
// reach: reach[first_edge + a] = reach[parent_row] * sigma_a
// (street_solve.cu:650-683, stored per sequence instead of per node)
// --------------------------------------------------------------------------
// Batched form: a subgame that has left the batch keeps its items in the
// captured launches; their blocks return at once.  Every block serves one
// subgame, so the test is block-uniform (ahead of any barrier).
__device__ __forceinline__ bool retired(const DevCtx *ctxs, int sg) { return ctxs && !ctxs[sg].live; }

// reach rows of 4 hands at an item of at most A actions (regret_match4's
// strategy, formed action by action)
template <int A>
__device__ __forceinline__ void reach_item(const float *__restrict__ R, float *__restrict__ reach, size_t HS,
                                           const ReachItem &I, int h0) {
    float4 r[A];
    const float4 pr = ld4(reach + static_cast<size_t>(I.parent_row) * HS + h0);
#pragma unroll
    for (int a = 0; a < A; ++a)
        if (a < I.na) r[a] = ld4(R + static_cast<size_t>(I.first_edge + a) * HS + h0);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int a = 0; a < A; ++a)
        if (a < I.na) {
            sum.x += r[a].x > 0.f ? r[a].x : 0.f;
            sum.y += r[a].y > 0.f ? r[a].y : 0.f;
            sum.z += r[a].z > 0.f ? r[a].z : 0.f;
            sum.w += r[a].w > 0.f ? r[a].w : 0.f;
        }
    const float uni = 1.0f / static_cast<float>(I.na);
    const float4 inv = make_float4(sum.x > 0.f ? 1.0f / sum.x : 0.f, sum.y > 0.f ? 1.0f / sum.y : 0.f,
                                   sum.z > 0.f ? 1.0f / sum.z : 0.f, sum.w > 0.f ? 1.0f / sum.w : 0.f);
#pragma unroll
    for (int a = 0; a < A; ++a)
        if (a < I.na) {
            auto sigma = [&](float ra, float s, float i) {
                if (I.frozen >= 0) return a == I.frozen ? 1.0f : 0.0f;
                return s > 0.f ? (ra > 0.f ? ra : 0.f) * i : uni;
            };
            st4(reach + static_cast<size_t>(I.first_edge + a) * HS + h0,
                make_float4(pr.x * sigma(r[a].x, sum.x, inv.x), pr.y * sigma(r[a].y, sum.y, inv.y),
                            pr.z * sigma(r[a].z, sum.z, inv.z), pr.w * sigma(r[a].w, sum.w, inv.w)));
        }
}

// Four (item, chunk) units of 64 threads per block: a block per unit was
// bound by block launches on trees of many items (96,432 items of 200 hands,
// 340 MB: 146 us so, 97 us now).
constexpr int kReachUnits = 4;
__global__ void __launch_bounds__(kHandThreads *kReachUnits, 5) k_reach(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                                    const ReachItem *__restrict__ items, int units,
                                                                    int nchunk, int H, int p) {
    wait_prior_grid();
    const int unit = blockIdx.x * kReachUnits + threadIdx.x / kHandThreads;
    if (unit >= units) return;
    const int it = unit / nchunk;
    const int ch = unit - it * nchunk;
    const int h0 = (ch * kHandThreads + threadIdx.x % kHandThreads) * 4;
    const ReachItem I = items[it];
    if (retired(ctxs, I.sg)) return;
    // context fields in registers (a reference to either the parameter or a
    // batch entry would send every field read through local memory)
    float *R, *reach;
    int HSi, Hp;
    if (ctxs) {
        const DevCtx &c = ctxs[I.sg];
        R = c.R, reach = c.reach, HSi = c.HS, Hp = c.H[p];
    } else {
        R = c0.R, reach = c0.reach, HSi = c0.HS, Hp = H;
    }
    if (h0 >= Hp) return;
    const size_t HS = static_cast<size_t>(HSi);
    if (I.na <= 4)
        reach_item<4>(R, reach, HS, I, h0);
    else
        reach_item<SS_MAX_ACTIONS>(R, reach, HS, I, h0);
}

// --------------------------------------------------------------------------
// cfv: value, regret and strategy-sum update at traverser nodes
// (street_solve.cu:1155-1175): v = sum_a sigma_a ev_a; r_a = (r_a + (ev_a - v))
// * t/(t+1); s_a += t * sigma_a; ev_a = sum of val over frontier(edge a).
// Each thread owns 2 hands.  S == 1: it walks whole frontiers, eight row
// loads in flight.  S > 1 (items with long frontiers, which are few): the S
// warps of a block share one hand chunk and each sums every S-th frontier
// row; warp 0 adds the S partial sums in a fixed order and updates.
// --------------------------------------------------------------------------
__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void st2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
// a float2 load kept as a separate L1-cached access (not merged with an
// earlier load of the same address, so the value need not stay in registers)
__device__ __forceinline__ float2 ld2_l1(const float *p) {
    float2 v;
    asm volatile("ld.global.ca.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void add2(float2 &a, float2 b) {
    a.x += b.x;
    a.y += b.y;
}

// context fields of the value/regret kernel, copied into registers (see Cr2View)
struct CfvView {
    float *R, *S, *val;
    const int *fr_off, *fr_items, *iter;
    int HS, H;
};
__device__ __forceinline__ CfvView cfv_view(const DevCtx &c, int H) {
    return CfvView{c.R, c.S, c.val, c.fr_off, c.fr_items, c.iter, c.HS, H};
}


// the first 32 bytes of a CfvItem (the inline frontier rows follow), read
// with two 16-byte loads
struct CfvHead {
    int first_edge, na, frozen, node, sg;
    float scale;
    int nfr, fr_bnd;
};
static_assert(sizeof(CfvItem) == 64 && offsetof(CfvItem, nfr) == 24 && offsetof(CfvItem, fr) == 32,
              "CfvItem layout read by cfv_head");
__device__ __forceinline__ CfvHead cfv_head(const CfvItem *p) {
    const int4 a = __ldg(reinterpret_cast<const int4 *>(p)), b = __ldg(reinterpret_cast<const int4 *>(p) + 1);
    return CfvHead{a.x, a.y, a.z, a.w, b.x, __int_as_float(b.y), b.z, b.w};
}

__device__ __forceinline__ void cfv_short(const CfvView &V, const CfvHead &I, const CfvItem *item,
                                          const float *__restrict__ val, int h0, int iter_add) {
    constexpr int kA = 4;
    const size_t HS = static_cast<size_t>(V.HS);
    const int4 *fp = reinterpret_cast<const int4 *>(item) + 2;
    const int4 f0 = __ldg(fp), f1 = __ldg(fp + 1);
    float *Rh = V.R + static_cast<size_t>(I.first_edge) * HS + h0, *Sh = V.S + static_cast<size_t>(I.first_edge) * HS + h0;
    float2 r[kA], sm[kA], x[kCfvInline];
#pragma unroll
    for (int a = 0; a < kA; ++a)
        if (a < I.na) {
            r[a] = ld2(Rh + a * HS);
            sm[a] = ld2(Sh + a * HS);
        }
    const int rows[kCfvInline] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
    for (int i = 0; i < kCfvInline; ++i)
        x[i] = i < I.nfr ? ld2(val + static_cast<size_t>(rows[i]) * HS) : make_float2(0.f, 0.f);
    const int t = *V.iter + iter_add;
    const float d = static_cast<float>(t) / (static_cast<float>(t) + 1.0f);
    const float w = static_cast<float>(t);
    float2 ev[kA];
#pragma unroll
    for (int a = 0; a < kA; ++a) ev[a] = make_float2(0.f, 0.f);
    const unsigned bnd = static_cast<unsigned>(I.fr_bnd);
#pragma unroll
    for (int i = 0; i < kCfvInline; ++i)
        if (i < I.nfr) {
            int e = 0;   // the edge of row i: the edges whose last row (nibble) is before it
#pragma unroll
            for (int a = 0; a < kA - 1; ++a) e += i > static_cast<int>((bnd >> (4 * a)) & 15u) ? 1 : 0;
#pragma unroll
            for (int a = 0; a < kA; ++a)
                if (e == a) add2(ev[a], x[i]);
        }
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int a = 0; a < kA; ++a)
        if (a < I.na) {
            s0 += r[a].x > 0.f ? r[a].x : 0.f;
            s1 += r[a].y > 0.f ? r[a].y : 0.f;
        }
    const float uni = 1.0f / static_cast<float>(I.na);
    const float inv0 = s0 > 0.f ? 1.0f / s0 : 0.f, inv1 = s1 > 0.f ? 1.0f / s1 : 0.f;
    auto sigma = [&](int a, float ra, float sum, float inv) {
        if (I.frozen >= 0) return a == I.frozen ? 1.0f : 0.0f;
        return sum > 0.f ? (ra > 0.f ? ra : 0.f) * inv : uni;
    };
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int a = 0; a < kA; ++a)
        if (a < I.na) {
            v0 += sigma(a, r[a].x, s0, inv0) * ev[a].x;
            v1 += sigma(a, r[a].y, s1, inv1) * ev[a].y;
        }
#pragma unroll
    for (int a = 0; a < kA; ++a)
        if (a < I.na) {
            float2 nr, ns;
            nr.x = (r[a].x + (ev[a].x - v0)) * d;
            nr.y = (r[a].y + (ev[a].y - v1)) * d;
            ns.x = sm[a].x + w * sigma(a, r[a].x, s0, inv0);
            ns.y = sm[a].y + w * sigma(a, r[a].y, s1, inv1);
            st2(Rh + a * HS, nr);
            st2(Sh + a * HS, ns);
        }
    st2(V.val + static_cast<size_t>(I.node) * HS + h0, make_float2(v0 * I.scale, v1 * I.scale));
}

// A S == 1 item of at most kCfvShort actions whose frontier is held in it
// (the bulk of a tree: its lowest level) loads all it needs at once -- value,
// regret and strategy-sum rows -- and keeps them in registers (the general
// form reads the regrets three times through L1): 96,432 items of 200 hands
// 345 -> 245 us with the back-to-back hand pairs.
constexpr int kCfvShort = 4;
template <int S>
__global__ void __launch_bounds__(kCfvThreads, 8) k_cfv(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                     const CfvItem *__restrict__ items, int n, int nchunk, int Hl,
                                                     int trav, int iter_add) {
    wait_prior_grid();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // S == 1: nchunk hand pairs per item, one per thread, items back to back
    // (64-hand chunks per warp left a quarter of the lanes idle at 200 hands);
    // S > 1: a block per (item, 64 hands)
    const int unit = S == 1 ? blockIdx.x * kCfvThreads + threadIdx.x : blockIdx.x;
    const int it = unit / nchunk;
    const int ch = unit - it * nchunk;
    if (S == 1 && it >= n) return;
    const CfvHead I = cfv_head(items + it);
    if (retired(ctxs, I.sg)) return;
    const CfvView V = ctxs ? cfv_view(ctxs[I.sg], ctxs[I.sg].H[trav]) : cfv_view(c0, Hl);
    const int h0 = S == 1 ? ch * 2 : ch * 64 + lane * 2;
    const bool act = h0 < V.H;
    if (S == 1 && !act) return;
    const size_t HS = static_cast<size_t>(V.HS);
    const float *val = V.val + h0;
    if constexpr (S == 1) {
        if (I.nfr > 0 && I.na <= kCfvShort) {
            cfv_short(V, I, items + it, val, h0, iter_add);
            return;
        }
    }
    const int *__restrict__ fr = V.fr_items;
    // the regret and strategy-sum rows are needed after the frontier sums:
    // start bringing them into L1 now (no registers held)
    if (act && (S == 1 || warp == 0)) {
#pragma unroll
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
            if (a < I.na) {
                const size_t off = static_cast<size_t>(I.first_edge + a) * HS + h0;
                asm volatile("prefetch.global.L1 [%0];" ::"l"(V.R + off));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(V.S + off));
            }
        }
    }
    float2 ev[SS_MAX_ACTIONS];
#pragma unroll
    for (int a = 0; a < SS_MAX_ACTIONS; ++a) ev[a] = make_float2(0.f, 0.f);
    if constexpr (S == 1) {
        if (I.nfr > 0) {
            // a short frontier held in the item: its rows load at once, with
            // no index loads before them; each row adds to its edge in row order
            const unsigned bnd = static_cast<unsigned>(I.fr_bnd);
            static_assert(kCfvInline == 8, "two 16-byte loads of inline rows");
            const int4 *fp = reinterpret_cast<const int4 *>(items + it) + 2;
            const int4 f0 = __ldg(fp), f1 = __ldg(fp + 1);
            const int rows[kCfvInline] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
            float2 x[kCfvInline];
#pragma unroll
            for (int i = 0; i < kCfvInline; ++i)
                x[i] = i < I.nfr ? ld2(val + static_cast<size_t>(rows[i]) * HS) : make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kCfvInline; ++i) {
                if (i < I.nfr) {
                    int e = 0;   // the edge of row i: the edges whose last row (nibble) is before it
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS - 1; ++a)
                        e += i > static_cast<int>((bnd >> (4 * a)) & 15u) ? 1 : 0;
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                        if (e == a) add2(ev[a], x[i]);
                }
            }
        } else {
            // the frontiers of all edges are one contiguous run of rows: walk
            // it eight rows at a time across edge boundaries (short frontiers,
            // one row per edge at the lowest level, would otherwise leave one
            // load in flight); each row adds to its edge in row order
            const int fe = I.first_edge;
            int bnd[SS_MAX_ACTIONS];
#pragma unroll
            for (int a = 0; a < SS_MAX_ACTIONS; ++a) bnd[a] = a < I.na ? V.fr_off[fe + a + 1] : 0x7fffffff;
            const int k0 = V.fr_off[fe], kend = V.fr_off[fe + I.na];
            for (int k = k0; k < kend; k += 8) {
                float2 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    x[i] = k + i < kend ? ld2(val + static_cast<size_t>(__ldg(fr + k + i)) * HS)
                                        : make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (k + i < kend) {
                        int e = 0;
#pragma unroll
                        for (int a = 0; a < SS_MAX_ACTIONS - 1; ++a) e += k + i >= bnd[a] ? 1 : 0;
#pragma unroll
                        for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                            if (e == a) add2(ev[a], x[i]);
                    }
                }
            }
        }
    } else {
#pragma unroll
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
            if (a < I.na && act) {
                float2 e = make_float2(0.f, 0.f);
                int k = V.fr_off[I.first_edge + a] + warp;
                const int k1 = V.fr_off[I.first_edge + a + 1];
                for (; k + 7 * S < k1; k += 8 * S) {
                    float2 x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = ld2(val + static_cast<size_t>(__ldg(fr + k + i * S)) * HS);
#pragma unroll
                    for (int i = 0; i < 8; ++i) add2(e, x[i]);
                }
                if (k < k1) {
                    // the last (< 8) rows of this warp, loaded together; the
                    // missing ones add +0, so the sum is the row-order sum
                    float2 x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        x[i] = k + i * S < k1 ? ld2(val + static_cast<size_t>(__ldg(fr + k + i * S)) * HS)
                                              : make_float2(0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) add2(e, x[i]);
                }
                ev[a] = e;
            }
        }
    }
    if constexpr (S > 1) {
        __shared__ float2 part[S][SS_MAX_ACTIONS][32];
#pragma unroll
        for (int a = 0; a < SS_MAX_ACTIONS; ++a)
            if (a < I.na) part[warp][a][lane] = ev[a];
        __syncthreads();
        if (warp != 0 || !act) return;
#pragma unroll
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
            if (a < I.na) {
                float2 e = part[0][a][lane];
#pragma unroll
                for (int w = 1; w < S; ++w) add2(e, part[w][a][lane]);
                ev[a] = e;
            }
        }
    }
    // the regrets are read three times (sum, value, update) instead of being
    // held in registers; the rereads hit L1
    const float *Rh = V.R + static_cast<size_t>(I.first_edge) * HS + h0;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
        if (a < I.na) {
            const float2 r = ld2_l1(Rh + a * HS);
            s0 += r.x > 0.f ? r.x : 0.f;
            s1 += r.y > 0.f ? r.y : 0.f;
        }
    }
    const float uni = 1.0f / static_cast<float>(I.na);
    const float inv0 = s0 > 0.f ? 1.0f / s0 : 0.f, inv1 = s1 > 0.f ? 1.0f / s1 : 0.f;
    // strategy of action a (regret matching, A3 freeze)
    auto sigma = [&](int a, float ra, float sum, float inv) {
        if (I.frozen >= 0) return a == I.frozen ? 1.0f : 0.0f;
        return sum > 0.f ? (ra > 0.f ? ra : 0.f) * inv : uni;
    };
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
        if (a < I.na) {
            const float2 r = ld2_l1(Rh + a * HS);
            v0 += sigma(a, r.x, s0, inv0) * ev[a].x;
            v1 += sigma(a, r.y, s1, inv1) * ev[a].y;
        }
    }
    const int t = *V.iter + iter_add;
    const float d = static_cast<float>(t) / (static_cast<float>(t) + 1.0f);
    const float w = static_cast<float>(t);
#pragma unroll
    for (int a = 0; a < SS_MAX_ACTIONS; ++a) {
        if (a < I.na) {
            const size_t off = static_cast<size_t>(I.first_edge + a) * HS + h0;
            const float2 r = ld2_l1(Rh + a * HS);
            const float2 sm = ld2(V.S + off);
            float2 nr, ns;
            nr.x = (r.x + (ev[a].x - v0)) * d;
            nr.y = (r.y + (ev[a].y - v1)) * d;
            ns.x = sm.x + w * sigma(a, r.x, s0, inv0);
            ns.y = sm.y + w * sigma(a, r.y, s1, inv1);
            st2(V.R + off, nr);
            st2(V.S + off, ns);
        }
    }
    // scale 1 on a single street (exact: the row equals v); below chance
    // nodes the row carries their 1 / cards weights for the parent's frontier
    st2(V.val + static_cast<size_t>(I.node) * HS + h0, make_float2(v0 * I.scale, v1 * I.scale));
}

// --------------------------------------------------------------------------
// One player's value/regret levels (bottom-up) and reach levels (top-down)
// near the root in one launch.  No hand depends on another here, so a block
// owns 8 hands (one 32-byte sector of every row) and walks the levels between
// its own barriers: a launch per level costs about 3.6 us of dependent-launch
// latency, a stage of this kernel about one chain of loads.  Threads are
// (slot, hand) pairs: in a value stage a slot sums one row chain into shared
// memory, then a slot updates one item; in a reach stage a slot takes one
// item.  Summation orders and expressions are those of k_cfv and k_reach.
// What is left is the latency of the row loads, so everything that no kernel
// writes (the pass's tables) comes to shared memory before the wait for the
// previous kernel where it fits (kResident), the next chain's rows are loaded
// while the last one's are added, and regret rows are prefetched into L1.
// --------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// The stages of one pass for hands [first, first + kTreeHands); tab: its blob
// (shared or global memory), part: the tile's partial sums in shared memory.
// Iteration t.  Every thread of the block takes part.
__device__ __forceinline__ void tree_pass(const DevCtx &c, const TreeRef &T, const char *tab, float *part, int first,
                                          int H, int t) {
    const TreeStage *stages = reinterpret_cast<const TreeStage *>(tab);
    const TreeItem *items = reinterpret_cast<const TreeItem *>(tab + T.o_items);
    const int2 *chains = reinterpret_cast<const int2 *>(tab + T.o_chains);
    const int4 *reach_items = reinterpret_cast<const int4 *>(tab + T.o_reach);
    const int *rows = reinterpret_cast<const int *>(tab + T.o_rows);
    const int hand = threadIdx.x & (kTreeHands - 1), slot = threadIdx.x / kTreeHands;
    const int slots = blockDim.x / kTreeHands;
    const int h = first + hand;
    const bool act = h < H;
    const size_t HS = static_cast<size_t>(c.HS);
    const float *val = c.val + h;
    float *R = c.R + h, *S = c.S + h, *reach = c.reach + h;
    const float d = static_cast<float>(t) / (static_cast<float>(t) + 1.0f);
    const float w = static_cast<float>(t);
    for (int si = 0; si < T.n_stages; ++si) {
        const int4 sa = *reinterpret_cast<const int4 *>(stages + si);
        if (sa.x == TS_VALUE) {
            const int c0 = sa.w, c1 = stages[si].c1;
            if (act) {
                // this slot's first item: its regret and strategy-sum rows
                if (sa.y + slot < sa.z) {
                    const TreeItem &I = items[sa.y + slot];
                    const size_t off = static_cast<size_t>(I.first_edge) * HS;
                    for (int a = 0; a < I.na; ++a) {
                        prefetch_l1(R + off + a * HS);
                        prefetch_l1(S + off + a * HS);
                    }
                }
                // rows i .. i + 7 of a chain (+0 past its end: the sum is the row-order sum)
                auto load8 = [&](int2 C, int i, float x[8]) {
                    const int n = C.y >> 4, st = C.y & 15;
                    const int *fr = rows + C.x;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        x[j] = i + j < n ? val[static_cast<size_t>(fr[(i + j) * st]) * HS] : 0.f;
                };
                float x[8];
                int ch = c0 + slot;
                int2 C = ch < c1 ? chains[ch] : make_int2(0, 0);
                load8(C, 0, x);
                while (ch < c1) {
                    const int nx = ch + slots;
                    const int2 Cn = nx < c1 ? chains[nx] : make_int2(0, 0);
                    float y[8];
                    load8(Cn, 0, y);
                    float e = 0.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) e += x[j];
                    for (int i = 8; i < C.y >> 4; i += 8) {
                        load8(C, i, x);
#pragma unroll
                        for (int j = 0; j < 8; ++j) e += x[j];
                    }
                    part[(ch - c0) * kTreeHands + hand] = e;
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = y[j];
                    C = Cn;
                    ch = nx;
                }
            }
            __syncthreads();
            if (act) {
                for (int it = sa.y + slot; it < sa.z; it += slots) {
                    const int4 I0 = reinterpret_cast<const int4 *>(items + it)[0];
                    const int4 I1 = reinterpret_cast<const int4 *>(items + it)[1];
                    const int na = I0.y, frozen = I0.z, split = I1.z;
                    const float *pp = part + I1.y * kTreeHands + hand;
                    float *Rh = R + static_cast<size_t>(I0.x) * HS, *Sh = S + static_cast<size_t>(I0.x) * HS;
                    float r[SS_MAX_ACTIONS], ev[SS_MAX_ACTIONS], sm[SS_MAX_ACTIONS];
                    float sum = 0.f;
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                        if (a < na) {
                            r[a] = Rh[a * HS];
                            sm[a] = Sh[a * HS];
                        }
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                        if (a < na) {
                            float e = pp[a * split * kTreeHands];
                            if (split > 1)
                                for (int k = 1; k < kCfvSplit; ++k) e += pp[(a * split + k) * kTreeHands];
                            ev[a] = e;
                            sum += r[a] > 0.f ? r[a] : 0.f;
                        }
                    const float uni = 1.0f / static_cast<float>(na);
                    const float inv = sum > 0.f ? 1.0f / sum : 0.f;
                    auto sigma = [&](int a) {
                        if (frozen >= 0) return a == frozen ? 1.0f : 0.0f;
                        return sum > 0.f ? (r[a] > 0.f ? r[a] : 0.f) * inv : uni;
                    };
                    float v = 0.f;
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                        if (a < na) v += sigma(a) * ev[a];
#pragma unroll
                    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                        if (a < na) {
                            Rh[a * HS] = (r[a] + (ev[a] - v)) * d;
                            Sh[a * HS] = sm[a] + w * sigma(a);
                        }
                    c.val[static_cast<size_t>(I0.w) * HS + h] = v * __int_as_float(I1.x);
                }
            }
        } else if (act) {
            for (int it = sa.y + slot; it < sa.z; it += slots) {
                const int4 I = reach_items[it];   // first_edge, na, parent_row, frozen
                const float *Rh = R + static_cast<size_t>(I.x) * HS;
                float *out = reach + static_cast<size_t>(I.x) * HS;
                const float pr = reach[static_cast<size_t>(I.z) * HS];
                float r[SS_MAX_ACTIONS], sum = 0.f;
#pragma unroll
                for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                    if (a < I.y) {
                        r[a] = Rh[a * HS];
                        sum += r[a] > 0.f ? r[a] : 0.f;
                    }
                const float uni = 1.0f / static_cast<float>(I.y);
                const bool pos = sum > 0.f;
                const float inv = pos ? 1.0f / sum : 0.f;
#pragma unroll
                for (int a = 0; a < SS_MAX_ACTIONS; ++a)
                    if (a < I.y) {
                        float s = pos ? (r[a] > 0.f ? r[a] : 0.f) * inv : uni;
                        if (I.w >= 0) s = (a == I.w) ? 1.0f : 0.0f;
                        out[a * HS] = pr * s;
                    }
            }
        }
        // the stage's value and reach rows are read by other slots of the
        // block in the next stages, and its partial sums are overwritten
        __syncthreads();
    }
}

template <bool kResident>
__global__ void __launch_bounds__(kTreeThreads, 1) k_tree(DevCtx c, TreeRef T, int H, int iter_add) {
    extern __shared__ __align__(16) char smem[];
    const char *tab = T.blob;
    if constexpr (kResident) {
        int4 *dst = reinterpret_cast<int4 *>(smem + static_cast<size_t>(T.max_chains) * kTreeHands * sizeof(float));
        const int4 *src = reinterpret_cast<const int4 *>(T.blob);
        for (int i = threadIdx.x; i < T.bytes / 16; i += blockDim.x) dst[i] = __ldg(src + i);
        tab = reinterpret_cast<const char *>(dst);
    }
    wait_prior_grid();
    if constexpr (kResident) __syncthreads();
    tree_pass(c, T, tab, reinterpret_cast<float *>(smem), blockIdx.x * kTreeHands, H, *c.iter + iter_add);
}

// --------------------------------------------------------------------------
// terminals
// --------------------------------------------------------------------------

// per-hand factor: fold payoff, or the leaf value of this traverser hand
__device__ __forceinline__ float term_factor(const DevCtx &c, const TermItem &I, int h) {
    return I.leaf_off >= 0 ? c.leaf_values[I.leaf_off + h] : I.payoff;
}

// The terminal kernels serve the CFR iterations (T = float: reach and values
// in FP32, per-node aggregates in FP64) and the best response (T = double).
template <class T> __device__ __forceinline__ const T *reach_rows(const DevCtx &c);
template <> __device__ __forceinline__ const float *reach_rows<float>(const DevCtx &c) { return c.reach; }
template <> __device__ __forceinline__ const double *reach_rows<double>(const DevCtx &c) { return c.reach_d; }
template <class T> __device__ __forceinline__ T *val_rows(const DevCtx &c);
template <> __device__ __forceinline__ float *val_rows<float>(const DevCtx &c) { return c.val; }
template <> __device__ __forceinline__ double *val_rows<double>(const DevCtx &c) { return c.val_d; }

// value rows of terminals with no opponent coupling: zero, or the factor itself
// (a leaf without a live opponent, street_solve.cu:1062-1065)
template <class T>
__global__ void __launch_bounds__(kHandThreads) k_term_fill(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                            const TermItem *__restrict__ items, int nchunk,
                                                            int trav, int zero) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const int ch = blockIdx.x - it * nchunk;
    const int h0 = (ch * kHandThreads + threadIdx.x) * 4;
    const TermItem I = items[it];
    if (retired(ctxs, I.sg)) return;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    if (h0 >= c.HS) return;
    const int Ht = c.H[trav];
    T *out = val_rows<T>(c) + static_cast<size_t>(I.node) * c.HS + h0;
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (zero || h0 + i >= Ht) ? T(0) : static_cast<T>(term_factor(c, I, h0 + i));
}

// Scatter one opponent's reach at a terminal into a 52x52 combo matrix
// (row stride MS): M[a][b] = M[b][a] = reach of the opponent's hand {a, b}.
// Board-blocked hands never count (street_solve.cu:755-757).  A range that
// holds some combo twice accumulates atomically; otherwise each cell has one
// writer and plain stores suffice.
template <class T>
__device__ __forceinline__ void scatter_combo(const DevCtx &c, int opp, int row, T *M) {
    const T *r = reach_rows<T>(c) + static_cast<size_t>(row) * c.HS;
    const int *code = c.hand_code + static_cast<size_t>(opp) * c.HS;
    const int Ho = c.H[opp];
    const bool dup = c.dup[opp] != 0;
    for (int j = threadIdx.x; j < Ho; j += blockDim.x) {
        const int hc = code[j];
        if (hc & 0x10000) continue;
        const int a = hc & 0xff, b = (hc >> 8) & 0xff;
        const T x = r[j];
        if (dup) {
            atomicAdd(&M[a * MS + b], x);
            atomicAdd(&M[b * MS + a], x);
        } else {
            M[a * MS + b] = x;
            M[b * MS + a] = x;
        }
    }
}

__device__ __forceinline__ int bit(unsigned long long m, int b) { return static_cast<int>((m >> b) & 1ull); }

template <class T>
__device__ __forceinline__ void zero_matrix(T *M) {
    float4 *m4 = reinterpret_cast<float4 *>(M);
    const int n = 52 * MS * static_cast<int>(sizeof(T)) / 16;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// four consecutive matrix entries (16-byte aligned)
__device__ __forceinline__ void load4(const double *p, double v[4]) {
    const double2 x = *reinterpret_cast<const double2 *>(p);
    const double2 y = *reinterpret_cast<const double2 *>(p + 2);
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void load4(const float *p, float v[4]) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void store4(double *p, const double v[4]) {
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void store4(float *p, const float v[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// Row pass over a combo matrix, one warp per card row r: the row sum u(r) in
// FP64 and the 64-bit mask of the row's positive cells.  The masks give the
// exact number of compatible positive-reach opponent tuples through the same
// inclusion-exclusion as the sums; where that number is 0 the value is
// exactly 0, as in the reference, which only adds positive products
// (street_solve.cu:810-812).  Without it rounding residue of the closed form
// would turn into a pure strategy under regret matching where the reference
// plays uniformly.
template <class T>
__device__ __forceinline__ void row_stats(const T *M, int r, int lane, double *sum_out,
                                          unsigned long long *mask_out, double *x0, double *x1) {
    const T a = M[r * MS + lane];
    const T b = lane + 32 < 52 ? M[r * MS + lane + 32] : T(0);
    const unsigned lo = __ballot_sync(0xffffffffu, a > T(0));
    const unsigned hi = __ballot_sync(0xffffffffu, b > T(0));
    *sum_out = warp_sum(static_cast<double>(a) + static_cast<double>(b));
    *mask_out = static_cast<unsigned long long>(lo) | (static_cast<unsigned long long>(hi) << 32);
    *x0 = a;
    *x1 = b;
}

template <class T>
__device__ __forceinline__ void store_value(T *out, int h, double v) { out[h] = static_cast<T>(v); }

// shared-memory carve-up of the terminal kernels (dynamic, 16-byte aligned)
struct Carve {
    char *p;
    template <class U>
    __device__ __forceinline__ U *take(int n) {
        U *r = reinterpret_cast<U *>(p);
        p += (static_cast<size_t>(n) * sizeof(U) + 15) & ~static_cast<size_t>(15);
        return r;
    }
};

template <class T>
constexpr size_t cr1_smem() {
    return 52 * MS * sizeof(T) + 52 * 8 + 52 * 8 + 64;
}

// One counted opponent: mass(h) = F - u(c1) - u(c2) + f(h), F the opponent's
// total reach, u(c) its reach on hands holding card c, f(h) its reach on the
// traverser's own combo.  Folds: payoff * mass (street_solve.cu:745-761);
// leaves: leaf value * mass (:1047-1066).  This form scatters the opponent's
// reach into a cleared 52x52 matrix (atomically), so it serves ranges that
// hold some combo more than once; k_term_cr1 below covers the others.
template <class T>
__global__ void __launch_bounds__(kTermThreads) k_term_cr1_dup(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                           const TermItem *__restrict__ items, int trav) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    Carve cv{smem};
    T *M = cv.take<T>(52 * MS);
    double *u = cv.take<double>(52);
    unsigned long long *B = cv.take<unsigned long long>(52);
    double *F = cv.take<double>(1);
    int *npos = cv.take<int>(1);
    const TermItem I = items[blockIdx.x];
    if (retired(ctxs, I.sg)) return;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    zero_matrix(M);
    __syncthreads();
    scatter_combo(c, I.opp_player[0], I.opp_row[0], M);
    __syncthreads();
    for (int r = warp; r < 52; r += blockDim.x / 32) {
        double s, x0, x1;
        unsigned long long m;
        row_stats(M, r, lane, &s, &m, &x0, &x1);
        if (lane == 0) {
            u[r] = s;
            B[r] = m;
        }
    }
    __syncthreads();
    if (warp == 0) {
        double s = u[lane] + (lane + 32 < 52 ? u[lane + 32] : 0.0);
        int n = __popcll(B[lane]) + (lane + 32 < 52 ? __popcll(B[lane + 32]) : 0);
        s = warp_sum(s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
        if (lane == 0) {
            *F = 0.5 * s;
            *npos = n / 2;
        }
    }
    __syncthreads();
    const int Ht = c.H[trav];
    const int *tc = c.hand_code + static_cast<size_t>(trav) * c.HS;
    T *out = val_rows<T>(c) + static_cast<size_t>(I.node) * c.HS;
    const double Fv = *F;
    const int np_ = *npos;
    for (int h = tid; h < c.HS; h += blockDim.x) {
        double v = 0.0;
        if (h < Ht) {
            const int hc = tc[h];
            const int a = hc & 0xff, b = (hc >> 8) & 0xff;
            const unsigned long long Ba = B[a], Bb = B[b];
            const int live = np_ - __popcll(Ba) - __popcll(Bb) + bit(Ba, b);
            if (live > 0) {
                const double z = Fv - u[a] - u[b] + static_cast<double>(M[a * MS + b]);
                v = static_cast<double>(term_factor(c, I, h)) * z;
            }
        }
        store_value(out, h, v);
    }
}

// Per-card terms of the two-opponent closed form over the dense deck (the
// non-board cards, renumbered 0 .. deck-1): FP64 sums and integer counts of
// positive-reach cells.  Entry 52 stays zero and stands for a board card of
// the traverser.  The tensor-core form packs the sums per card (Cr2Card);
// k_term_cr2 keeps one array per field.
struct alignas(16) Cr2Card {
    double u1, u2;      // per-card reach sums of opponents 1 and 2
    double g;           // u1 u2 + w - 2 d, w = (M2 u1 + M1 u2)(c), d = sum_b M1[c][b] M2[c][b]
    double d;
};
struct alignas(16) Cr2Cnt {
    int n1, n2;         // positive-reach cells of the card's row in M1, M2
    int pad0, pad1;
};
// block scalars: F_i = sum u_i / 2, QD = D - Q with Q = sum u1 u2, D = sum d / 2,
// and the same on the 0/1 positive-reach matrices
struct Cr2Scalars {
    double F1, F2, QD;
    int IF1, IF2, IQD, pad;
};
constexpr int kCr2Off = 52;   // index of the zero per-card entry
constexpr int kMaxHS = 1344;  // largest row stride: 1326 combos rounded up to 32

// dynamic shared memory of the two-opponent kernel for row stride HS: M1, M2,
// P (whose space first stages the two opponents' reach rows), the first
// terminal's leaf row, per-card terms, staged group items
template <class T>
constexpr size_t cr2_smem(int HS) {
    return 3 * 52 * MS * sizeof(T) + (static_cast<size_t>(HS) + 4) * sizeof(T) + 3 * 56 * sizeof(double) + 53 * sizeof(Cr2Cnt) +
           53 * 16 + 5 * 48 * 4 + sizeof(Cr2Scalars) + 3 * kTermGroupMax * 4 + 8 * 16;
}

// asynchronous global -> shared copies (cp.async): 16-byte chunks and 4-byte words
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One opponent's staged reach as a symmetric matrix over the dense deck:
// M[a][b] = M[b][a] = reach of the hand {a, b}; board-blocked hands never
// count (street_solve.cu:755-757).  This form serves ranges that hold some
// combo twice (accumulated atomically into a cleared matrix).
template <class T>
__device__ __forceinline__ void scatter_dense(const int *__restrict__ code, int Ho, const T *r, T *M) {
    for (int j = threadIdx.x; j < Ho; j += blockDim.x) {
        const int hc = __ldg(code + j);
        if (hc & 0x10000) continue;
        const int a = (hc >> 20) & 63, b = (hc >> 26) & 63;
        const T x = r[j];
        atomicAdd(&M[a * MS + b], x);
        atomicAdd(&M[b * MS + a], x);
    }
}

// The same matrices gathered instead (ranges without a repeated combo): each
// thread fills 4-column chunks of rows 0 .. Dp-1 through the player's table of
// range indices per dense-card pair (missing pairs index the zero kept after
// the staged row), so every cell is written once, with 16-byte stores and no
// clearing pass.  Cells outside rows and columns 0 .. Dp-1 are left unset;
// nothing reads them.
template <class T>
__device__ __forceinline__ void gather_dense(const int *__restrict__ tab, const T *r, T *M, int Dp) {
    const int chunk = threadIdx.x & 15, c0 = chunk * 4;
    if (c0 >= Dp) return;
    for (int row = threadIdx.x >> 4; row < Dp; row += kTermThreads / 16) {
        const int4 ix = __ldg(reinterpret_cast<const int4 *>(tab + row * 52 + c0));
        const T v[4] = {r[ix.x], r[ix.y], r[ix.z], r[ix.w]};
        store4(M + row * MS + c0, v);
    }
}

// The fields of a subgame context that the two-opponent kernel reads, copied
// into registers.  (A reference bound to either the kernel parameter or a
// batch entry would give the parameter a generic address, and every field
// read would then go through local memory.)
template <class T>
struct Cr2View {
    const T *reach;
    T *val;
    const int *code_t, *code0, *code1;   // hand codes of the traverser and the two opponents
    const int *tab0, *tab1;              // dense-pair tables of the two opponents
    const int *x0, *x1;                  // each traverser hand's index in the two opponents' ranges
    const float *leaf;
    int HS, deck, Ht, H0, H1;
    bool dup;
};
template <class T>
__device__ __forceinline__ Cr2View<T> cr2_view(const DevCtx &c, int trav, int o0, int o1) {
    Cr2View<T> v;
    v.reach = reach_rows<T>(c);
    v.val = val_rows<T>(c);
    v.code_t = c.hand_code + static_cast<size_t>(trav) * c.HS;
    v.code0 = c.hand_code + static_cast<size_t>(o0) * c.HS;
    v.code1 = c.hand_code + static_cast<size_t>(o1) * c.HS;
    v.tab0 = c.pair_idx + static_cast<size_t>(o0) * 52 * 52;
    v.tab1 = c.pair_idx + static_cast<size_t>(o1) * 52 * 52;
    v.x0 = c.cross_idx + (static_cast<size_t>(trav) * c.np + o0) * c.HS;
    v.x1 = c.cross_idx + (static_cast<size_t>(trav) * c.np + o1) * c.HS;
    v.leaf = c.leaf_values;
    v.HS = c.HS;
    v.deck = c.deck;
    v.Ht = c.H[trav];
    v.H0 = c.H[o0];
    v.H1 = c.H[o1];
    v.dup = (c.dup[o0] | c.dup[o1]) != 0;
    return v;
}

// TF32 split of the tensor-core product below: x = hi + lo, hi = x truncated
// to TF32 (10 explicit mantissa bits), lo = the exact FP32 remainder rounded
// to TF32 (half away from zero on the bit pattern).  hi*hi + hi*lo + lo*hi
// then carries about 21 significant bits, close to the FP32 product.
__device__ __forceinline__ void split_tf32(float x, unsigned &hi, unsigned &lo) {
    hi = __float_as_uint(x) & 0xffffe000u;                                        // truncated: x - hi is exact
    lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xffffe000u;     // rounded remainder
}
// d += a b, one m16n8k8 TF32 tile (A row-major 16x8, B column-major 8x8)
__device__ __forceinline__ void mma_tf32(float d[4], const unsigned a[4], const unsigned b[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// P = M1 M2 over a dense deck of at most 48 cards on the tensor cores: warp w
// (0..5) owns rows 16 (w / 2) .. +15 and columns 24 (w % 2) .. +23 (three
// 8-column tiles); six k-steps of 8.  Operand fragments are read from the
// FP32 matrices in shared memory (row stride 52 keeps the A-fragment loads
// free of bank conflicts) and split into TF32 pairs in registers.
// Also leaves rsum[h][r] = sum of row r over column half h and csum[s][c] =
// sum of column c over row strip s (FP32, deterministic order).
__device__ __forceinline__ void product_mma48(const float *M1, const float *M2, float *P, float *rsum, float *csum,
                                              int warp, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const int m0 = (warp >> 1) * 16, n0 = (warp & 1) * 24;
    float acc[3][4] = {};
#pragma unroll
    for (int k0 = 0; k0 < 48; k0 += 8) {
        unsigned ah[4], al[4];
        split_tf32(M1[(m0 + g) * MS + k0 + t], ah[0], al[0]);
        split_tf32(M1[(m0 + g + 8) * MS + k0 + t], ah[1], al[1]);
        split_tf32(M1[(m0 + g) * MS + k0 + t + 4], ah[2], al[2]);
        split_tf32(M1[(m0 + g + 8) * MS + k0 + t + 4], ah[3], al[3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int n = n0 + j * 8 + g;
            unsigned bh[2], bl[2];
            split_tf32(M2[(k0 + t) * MS + n], bh[0], bl[0]);
            split_tf32(M2[(k0 + t + 4) * MS + n], bh[1], bl[1]);
            mma_tf32(acc[j], al, bh);
            mma_tf32(acc[j], ah, bl);
            mma_tf32(acc[j], ah, bh);
        }
    }
    float ra = 0.f, rb = 0.f;   // this lane's share of rows m0 + g and m0 + g + 8
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int n = n0 + j * 8 + 2 * t;
        *reinterpret_cast<float2 *>(&P[(m0 + g) * MS + n]) = make_float2(acc[j][0], acc[j][1]);
        *reinterpret_cast<float2 *>(&P[(m0 + g + 8) * MS + n]) = make_float2(acc[j][2], acc[j][3]);
        ra += acc[j][0] + acc[j][1];
        rb += acc[j][2] + acc[j][3];
    }
    // row sums over this warp's 24 columns and column sums over its 16 rows
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        ra += __shfl_xor_sync(0xffffffffu, ra, o);
        rb += __shfl_xor_sync(0xffffffffu, rb, o);
    }
    if (t == 0) {
        rsum[(warp & 1) * 48 + m0 + g] = ra;
        rsum[(warp & 1) * 48 + m0 + g + 8] = rb;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        float c0 = acc[j][0] + acc[j][2], c1 = acc[j][1] + acc[j][3];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            c0 += __shfl_xor_sync(0xffffffffu, c0, o);
            c1 += __shfl_xor_sync(0xffffffffu, c1, o);
        }
        if (g == 0) {
            csum[(warp >> 1) * 48 + n0 + j * 8 + 2 * t] = c0;
            csum[(warp >> 1) * 48 + n0 + j * 8 + 2 * t + 1] = c1;
        }
    }
}

// column sums and positive-cell masks of M1 (s < Dp) or M2 (s >= Dp): four
// independent partial sums in T (Dp is a multiple of 4; FP32 keeps the
// relative error near 1e-7), added in FP64 in a fixed order
template <class T>
__device__ __forceinline__ void column_stats(const T *M1, const T *M2, int s, int Dp, double *cu1, double *cu2,
                                             ulonglong2 *Bm) {
    const bool second = s >= Dp;
    const int col = second ? s - Dp : s;
    const T *M = (second ? M2 : M1) + col;
    T u[4] = {T(0), T(0), T(0), T(0)};
    unsigned long long B = 0ull;
    for (int r = 0; r < Dp; r += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const T x = M[(r + i) * MS];
            u[i] += x;
            B |= static_cast<unsigned long long>(x > T(0)) << (r + i);
        }
    }
    const double tot = (static_cast<double>(u[0]) + static_cast<double>(u[1])) +
                       (static_cast<double>(u[2]) + static_cast<double>(u[3]));
    if (second) {
        cu2[col] = tot;
        Bm[col].y = B;
    } else {
        cu1[col] = tot;
        Bm[col].x = B;
    }
}

// 4x4 tile (rows i0.., columns j0..) of P = M1 M2; M1 is symmetric, so row k
// of M1 is its column k.
template <class T>
__device__ __forceinline__ void product_tile(const T *M1, const T *M2, T *P, int i0, int j0, int Dp) {
    T acc[4][4] = {};
#pragma unroll 4
    for (int k = 0; k < Dp; ++k) {
        T xs[4], ys[4];
        load4(&M1[k * MS + i0], xs);
        load4(&M2[k * MS + j0], ys);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += xs[i] * ys[j];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) P[(i0 + i) * MS + j0 + j] = acc[i][j];
}

// Number of opponent pairs with positive reach that are disjoint from each
// other and from the traverser hand (a, b): the two-opponent formula on the
// 0/1 positive-reach matrices, whose entries are the bits of the card masks
// (row c of M_i = bits of Bm[c]).  The per-card term ng(c) = n1 n2 + nw - 2 nd
// with nw(c) = (I2 n1 + I1 n2)(c) is summed here over the set bits, since the
// count is only needed for the few hands whose mass is near zero.
__device__ __forceinline__ int card_ng(const ulonglong2 *Bm, const Cr2Cnt *cnt, int c) {
    const ulonglong2 Bc = Bm[c];
    int nw = 0;
    for (unsigned long long m = Bc.y; m; m &= m - 1) nw += cnt[__ffsll(static_cast<long long>(m)) - 1].n1;
    for (unsigned long long m = Bc.x; m; m &= m - 1) nw += cnt[__ffsll(static_cast<long long>(m)) - 1].n2;
    return cnt[c].n1 * cnt[c].n2 + nw - 2 * __popcll(Bc.x & Bc.y);
}
__device__ __noinline__ int pair_count(const ulonglong2 *Bm, const Cr2Cnt *cnt, int a, int b, int IF1, int IF2,
                                      int IQD) {
    const ulonglong2 Ba = Bm[a], Bb = Bm[b];
    const int n1a = cnt[a].n1, n1b = cnt[b].n1, n2a = cnt[a].n2, n2b = cnt[b].n2;
    const int j1 = bit(Ba.x, b), j2 = bit(Ba.y, b);
    return (IF1 - n1a - n1b + j1) * (IF2 - n2a - n2b + j2) + IQD + card_ng(Bm, cnt, a) + card_ng(Bm, cnt, b) -
           j2 * (n1a + n1b) - j1 * (n2a + n2b) + 3 * j1 * j2 - (__popcll(Ba.x & Bb.y) + __popcll(Bb.x & Ba.y));
}

// Two counted opponents (1, 2) with combo matrices M1, M2 over the dense
// deck, per-card sums u_i = M_i 1, d(c) = sum_b M1[c][b] M2[c][b],
// w = M2 u1 + M1 u2, P = M1 M2, F_i = sum u_i / 2, Q = sum u1 u2, D = sum d / 2.
// For a traverser hand (a, b), m_i = M_i[a][b], A_i = F_i - u_i(a) - u_i(b) + m_i,
// the mass of opponent pairs disjoint from each other and from (a, b) is
//   A1 A2 - Q + u1(a)u2(a) + u1(b)u2(b) + w(a) + w(b)
//   - m2 (u1(a) + u1(b)) - m1 (u2(a) + u2(b)) - 2 (d(a) + d(b)) + 3 m1 m2
//   - P[a][b] - P[b][a] + D
// (inclusion-exclusion over shared cards), equal to the reference odometer
// sum of street_solve.cu:771-823 / :1079-1127 for two opponents.
//
// Exact zeros: the reference only adds positive reach products, so a hand
// with no compatible positive-reach pair gets exactly 0.  Every term above is
// at most a few F1 F2 in size and the product P carries FP32 accuracy, so a
// computed mass above 1e-4 F1 F2 cannot come from an empty set of pairs; at or
// below it the kernel counts the compatible positive-reach pairs exactly (the
// same formula on the 0/1 positive-reach matrices, via 64-bit card masks) and
// writes 0 when there are none.
//
// One block per group of terminals sharing both opponents' reach rows: the
// masses are computed once and multiplied by each terminal's factor.  A
// chain of groups on the same first-opponent row (TermItem::chain) runs in
// one block, one group after the other: the first opponent's matrix, its
// column sums and masks are built once for the chain.
// Phases per group: cp.async staging of the reach rows (both for the
// chain's first group; the next group's second-opponent row is staged while
// this group's mass is computed); gather (or clear + scatter for ranges that
// repeat a combo); P (tensor cores) alongside per-column sums and masks;
// per-card FP64 terms and block scalars; per-hand mass and one output row
// per terminal (the leaf factors read one hand ahead from global memory).
template <class T>
__global__ void __launch_bounds__(kTermThreads, sizeof(T) == 4 ? 5 : 2) k_term_cr2(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                              const TermItem *__restrict__ items,
                                                              const int *__restrict__ heads, int trav) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    const TermItem *I0 = items + (heads ? __ldg(heads + blockIdx.x) : static_cast<int>(blockIdx.x));
    // followers are written by their group's leader, chained groups by the chain's head
    if (I0->follow || I0->chained) return;
    if (retired(ctxs, I0->sg)) return;
    const int o0 = I0->opp_player[0], o1 = I0->opp_player[1];
    const Cr2View<T> V = ctxs ? cr2_view<T>(ctxs[I0->sg], trav, o0, o1) : cr2_view<T>(c0, trav, o0, o1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int HS = V.HS;
    const int Dp = (V.deck + 3) & ~3;
    const int hc_first = tid < V.Ht ? __ldg(V.code_t + tid) : 0;   // this thread's first hand code
    // shared memory was provisioned for c0's row stride (the largest of a batch)
    if (HS > c0.HS || V.deck > 52) return;
    Carve cv{smem};
    T *M1 = cv.take<T>(52 * MS);
    T *M2 = cv.take<T>(52 * MS);
    T *P = cv.take<T>(52 * MS);
    // per-card terms, one array per field (a hand reads three of them at two
    // cards; separate arrays keep those reads free of bank conflicts)
    double *cu1 = cv.take<double>(56), *cu2 = cv.take<double>(56), *cg = cv.take<double>(56);
    Cr2Cnt *cnt = cv.take<Cr2Cnt>(53);
    ulonglong2 *Bm = cv.take<ulonglong2>(53);   // positive-cell masks of M1 (x) and M2 (y) per card
    float *rsum = cv.take<float>(2 * 48);       // tensor-core path: partial row / column sums of P
    float *csum = cv.take<float>(3 * 48);
    Cr2Scalars *sc = cv.take<Cr2Scalars>(1);
    int *gnode = cv.take<int>(kTermGroupMax);
    int *gleaf = cv.take<int>(kTermGroupMax);
    float *gpay = cv.take<float>(kTermGroupMax);
    // the second opponent's staged reach row, followed by a zero (last: every
    // other offset is a constant); the next group's row lands here while
    // this group's mass is computed.  The first opponent's row is staged in
    // P's space (P is written after the gather).
    T *r2 = cv.take<T>(HS + 16 / sizeof(T));
    T *r1 = P;
    bool mma = false;
    if constexpr (sizeof(T) == 4) mma = Dp <= 48;
    const int Ht = V.Ht;
    const int *__restrict__ tc = V.code_t;

    // staging: a group's second-opponent reach row (16-byte chunks; rows
    // start on 128-byte boundaries), the first opponent's row with with_first
    auto stage_rows = [&](const TermItem *G, bool with_first) {
        constexpr int per = 16 / sizeof(T);
        const T *s1 = V.reach + static_cast<size_t>(G->opp_row[0]) * HS;
        const T *s2 = V.reach + static_cast<size_t>(G->opp_row[1]) * HS;
        for (int i = tid * per; i < HS; i += kTermThreads * per) {
            if (with_first) cp_async16(r1 + i, s1 + i);
            cp_async16(r2 + i, s2 + i);
        }
    };
    // a group's items' fields
    auto stage_items = [&](const TermItem *G) {
        if (tid <= G->gextra) {
            const TermItem &I = G[tid];
            gnode[tid] = I.node;
            gleaf[tid] = I.leaf_off;
            gpay[tid] = I.payoff;
        }
    };
    auto gather_second = [&]() {
        if (V.dup)
            scatter_dense(V.code1, V.H1, r2, M2);
        else
            gather_dense(V.tab1, r2, M2, Dp);
    };

    // the chain's first group: both opponents' matrices
    stage_rows(I0, true);
    stage_items(I0);
    if (tid == 0) {
        r1[HS] = T(0);
        r2[HS] = T(0);
    }
    if (V.dup) {
        zero_matrix(M1);
        zero_matrix(M2);
    }
    cp_async_wait_all();
    __syncthreads();
    if (V.dup)
        scatter_dense(V.code0, V.H0, r1, M1);
    else
        gather_dense(V.tab0, r1, M1, Dp);
    gather_second();
    __syncthreads();

    const TermItem *G = I0;
    const int nchain = I0->chain;
    for (int q = 0;; ++q) {
        const bool first = q == 0;
        const int ng = G->gextra + 1;

        // phase A: P = M1 M2 (tensor cores when the deck fits 48 cards, else
        // 4x4 SIMT tiles); per-column reach sums and positive-cell masks (the
        // first opponent's for the chain's first group only: they stay in
        // cu1 and Bm[].x)
        if (mma) {
            if constexpr (sizeof(T) == 4) {
                if (warp < 6) product_mma48(M1, M2, P, rsum, csum, warp, lane);
            }
            // columns: warps 6-7 take 0..63, warp 0 (after its MMA tiles) 64..95
            const int s = tid >= 6 * 32 ? tid - 6 * 32 : tid < 32 ? 64 + tid : 2 * 52;
            if (s < 2 * Dp && (first || s >= Dp)) column_stats(M1, M2, s, Dp, cu1, cu2, Bm);
        } else {
            const int nt = Dp >> 2;
            if (tid < nt * nt) product_tile(M1, M2, P, (tid / nt) * 4, (tid % nt) * 4, Dp);
            const int s = kTermThreads - 1 - tid;
            if (s < 2 * Dp && (first || s >= Dp)) column_stats(M1, M2, s, Dp, cu1, cu2, Bm);
        }
        __syncthreads();
        // the chain's next group: its second-opponent row is brought in while
        // this group's mass is computed (the gather of this group's is done)
        if (q < nchain) stage_rows(G + ng, false);

        // phase B: per-card terms (w from the row and column sums of P, d from its
        // diagonal: P = M1 M2 with symmetric M1, M2 gives rowsum = M1 u2,
        // colsum = M2 u1, P[c][c] = d(c)); entries beyond the deck are zeroed;
        // the last warp forms the block scalars
        if (tid < Dp) {
            const int col = tid;
            double w;
            if (mma) {
                w = (static_cast<double>(rsum[col]) + static_cast<double>(rsum[48 + col])) +
                    ((static_cast<double>(csum[col]) + static_cast<double>(csum[48 + col])) +
                     static_cast<double>(csum[96 + col]));
            } else {
                w = 0.0;
                for (int b = 0; b < Dp; ++b)
                    w += static_cast<double>(P[col * MS + b]) + static_cast<double>(P[b * MS + col]);
            }
            const double d = P[col * MS + col];
            cg[col] = cu1[col] * cu2[col] + w - 2.0 * d;
            const ulonglong2 Bc = Bm[col];
            cnt[col] = Cr2Cnt{__popcll(Bc.x), __popcll(Bc.y), 0, 0};
        } else if (tid <= kCr2Off) {
            cu1[tid] = 0.0;
            cu2[tid] = 0.0;
            cg[tid] = 0.0;
            cnt[tid] = Cr2Cnt{0, 0, 0, 0};
            Bm[tid] = make_ulonglong2(0ull, 0ull);
        } else if (warp == kTermThreads / 32 - 1) {
            double a1 = 0.0, a2 = 0.0, qq = 0.0, e = 0.0;
            int n1 = 0, n2 = 0, nq = 0, nd = 0;
            for (int k = lane; k < Dp; k += 32) {
                const double u1 = cu1[k], u2 = cu2[k];
                a1 += u1;
                a2 += u2;
                qq += u1 * u2;
                e += static_cast<double>(P[k * MS + k]);
                const ulonglong2 B = Bm[k];
                const int p1 = __popcll(B.x), p2 = __popcll(B.y);
                n1 += p1;
                n2 += p2;
                nq += p1 * p2;
                nd += __popcll(B.x & B.y);
            }
            a1 = warp_sum(a1);
            a2 = warp_sum(a2);
            qq = warp_sum(qq);
            e = warp_sum(e);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                n1 += __shfl_xor_sync(0xffffffffu, n1, o);
                n2 += __shfl_xor_sync(0xffffffffu, n2, o);
                nq += __shfl_xor_sync(0xffffffffu, nq, o);
                nd += __shfl_xor_sync(0xffffffffu, nd, o);
            }
            if (lane == 0) *sc = Cr2Scalars{0.5 * a1, 0.5 * a2, 0.5 * e - qq, n1 / 2, n2 / 2, nd / 2 - nq, 0};
        }
        __syncthreads();

        // phase C: card-removal mass of every traverser hand, written out as
        // factor x mass for every terminal of the group
        const Cr2Scalars S = *sc;
        const double zmin = 1e-4 * S.F1 * S.F2;
        const bool none = !(S.F1 > 0.0 && S.F2 > 0.0);   // an opponent without positive reach: all zero
        const int gl0 = gleaf[0];
        const float gp0 = gpay[0];
        T *out0 = V.val + static_cast<size_t>(gnode[0]) * HS;
        // the next hand's code is loaded one iteration ahead (the first one at
        // the start of the block), so the loop does not wait on it
        int hc_next = hc_first;
        float f_next = tid < Ht ? (gl0 >= 0 ? __ldg(V.leaf + gl0 + tid) : gp0) : 0.f;
        for (int h = tid; h < HS; h += kTermThreads) {
            const int hc = hc_next;
            const float f0 = f_next;
            hc_next = h + kTermThreads < Ht ? __ldg(tc + h + kTermThreads) : 0;
            f_next = h + kTermThreads < Ht ? (gl0 >= 0 ? __ldg(V.leaf + gl0 + h + kTermThreads) : gp0) : 0.f;
            double v = 0.0;
            if (h < Ht && !none) {
                const int a = min((hc >> 20) & 63, kCr2Off), b = min((hc >> 26) & 63, kCr2Off);
                const bool on = (a < kCr2Off) && (b < kCr2Off);
                const double ua1 = cu1[a], ua2 = cu2[a], ub1 = cu1[b], ub2 = cu2[b];
                const double m1 = on ? static_cast<double>(M1[a * MS + b]) : 0.0;
                const double m2 = on ? static_cast<double>(M2[a * MS + b]) : 0.0;
                const double pp = on ? static_cast<double>(P[a * MS + b] + P[b * MS + a]) : 0.0;
                const double A1 = S.F1 - ua1 - ub1 + m1;
                const double A2 = S.F2 - ua2 - ub2 + m2;
                v = A1 * A2 + S.QD + cg[a] + cg[b] - m2 * (ua1 + ub1) - m1 * (ua2 + ub2) + 3.0 * m1 * m2 - pp;
                if (fabs(v) <= zmin && pair_count(Bm, cnt, a, b, S.IF1, S.IF2, S.IQD) <= 0) v = 0.0;
            }
            out0[h] = static_cast<T>(static_cast<double>(f0) * v);
            for (int g = 1; g < ng; ++g) {
                const float f = h >= Ht ? 0.f : gleaf[g] >= 0 ? __ldg(V.leaf + gleaf[g] + h) : gpay[g];
                V.val[static_cast<size_t>(gnode[g]) * HS + h] = static_cast<T>(static_cast<double>(f) * v);
            }
        }
        if (q == nchain) break;
        // the chain's next group: its second-opponent matrix replaces the
        // last one once every thread is done with the shared state
        G += ng;
        __syncthreads();
        stage_items(G);
        if (V.dup) zero_matrix(M2);
        cp_async_wait_all();
        __syncthreads();
        gather_second();
        __syncthreads();
    }
}

#include "ss_cr2_tc.cuh"

template <class T>
__host__ __device__ constexpr size_t cr1_gather_smem(int HS) {
    return ((static_cast<size_t>(HS) + 4) * sizeof(T) + static_cast<size_t>(HS) * 4 + 64 * 8 + 64 * 4 +
            3 * kTermGroupMax * 4 + 2 * 16 + 8 * 16 + 15) / 16 * 16;
}

// One counted opponent over the dense deck, for ranges without a repeated
// combo: u(c) and f(h) are read from the staged reach row through the
// opponent's pair table (row c of the table lists the opponent's hands
// holding card c), so no matrix is built.  Exact zeros: the number of
// compatible positive-reach opponent hands N - n(a) - n(b) + [f(h) > 0]
// decides a value of exactly 0.  One block per group of terminals sharing the
// opponent's reach row (the traverser's own continuation choices).
// The work of kTermThreads threads (tid) with their own barrier (sync).
template <class T, class Sync>
__device__ __forceinline__ void cr1_terminal(const DevCtx &c0, const DevCtx *__restrict__ ctxs,
                                             const TermItem *__restrict__ I0, int trav, char *smem, int tid,
                                             Sync sync) {
    if (I0->follow) return;   // written by the block of its group's first item
    if (retired(ctxs, I0->sg)) return;
    const int ng = I0->gextra + 1;
    const int o = I0->opp_player[0];
    const Cr2View<T> V = ctxs ? cr2_view<T>(ctxs[I0->sg], trav, o, o) : cr2_view<T>(c0, trav, o, o);
    const int HS = V.HS;
    if (HS > c0.HS || V.deck > 52) return;   // shared memory was provisioned for c0's row stride
    const int lane = tid & 31;
    const int Dp = (V.deck + 3) & ~3;
    Carve cv{smem};
    T *r = cv.take<T>(HS + 4);                 // staged reach row, r[HS] = 0 for missing pairs
    float *leaf0 = cv.take<float>(HS);
    double *u = cv.take<double>(64);
    int *nz = cv.take<int>(64);
    int *gnode = cv.take<int>(kTermGroupMax);
    int *gleaf = cv.take<int>(kTermGroupMax);
    float *gpay = cv.take<float>(kTermGroupMax);
    {
        const T *src = V.reach + static_cast<size_t>(I0->opp_row[0]) * HS;
        constexpr int per = 16 / sizeof(T);
        for (int q = tid * per; q < HS; q += kTermThreads * per) cp_async16(r + q, src + q);
        const int lo = I0->leaf_off;
        if (lo >= 0) {
            const float *ls = V.leaf + lo;
            for (int h = tid; h < V.Ht; h += kTermThreads) cp_async4(leaf0 + h, ls + h);
        }
        if (tid < ng) {
            const TermItem &I = I0[tid];
            gnode[tid] = I.node;
            gleaf[tid] = I.leaf_off;
            gpay[tid] = I.payoff;
        }
        if (tid == 0) r[HS] = T(0);
        if (tid < 64) {
            u[tid] = 0.0;
            nz[tid] = 0;
        }
    }
    cp_async_wait_all();
    sync();
    // per card c: u(c) and the count of positive-reach hands holding c, four
    // lanes per card (a quarter of the table row each, shuffles in a fixed order)
    {
        const int col = tid >> 2, part = tid & 3, q = Dp >> 2;
        double s = 0.0;
        int n = 0;
        if (col < Dp) {
            const int *row = V.tab0 + col * 52 + part * q;
            for (int b = 0; b < q; ++b) {
                const T x = r[__ldg(row + b)];
                s += static_cast<double>(x);
                n += x > T(0) ? 1 : 0;
            }
        }
#pragma unroll
        for (int k = 1; k < 4; k <<= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, k);
            n += __shfl_xor_sync(0xffffffffu, n, k);
        }
        if (part == 0 && col < Dp) {
            u[col] = s;
            nz[col] = n;
        }
    }
    sync();
    double F;
    int N;
    {
        double s = (lane < Dp ? u[lane] : 0.0) + (lane + 32 < Dp ? u[lane + 32] : 0.0);
        int n = (lane < Dp ? nz[lane] : 0) + (lane + 32 < Dp ? nz[lane + 32] : 0);
        s = warp_sum(s);
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) n += __shfl_xor_sync(0xffffffffu, n, k);
        F = 0.5 * s;
        N = n / 2;
    }
    const int Ht = V.Ht;
    const int *__restrict__ tc = V.code_t;
    const bool leaf_first = gleaf[0] >= 0;
    const float gp0 = gpay[0];
    T *out0 = V.val + static_cast<size_t>(gnode[0]) * HS;
    for (int h = tid; h < HS; h += kTermThreads) {
        double v = 0.0;
        if (h < Ht) {
            const int hc = __ldg(tc + h);
            const int a = min((hc >> 20) & 63, kCr2Off), b = min((hc >> 26) & 63, kCr2Off);
            const T f = r[__ldg(V.x0 + h)];   // 0 for a hand touching the board (index HS)
            const int live = N - nz[a] - nz[b] + (f > T(0) ? 1 : 0);
            if (live > 0) v = F - u[a] - u[b] + static_cast<double>(f);
        }
        const float f0 = h >= Ht ? 0.f : leaf_first ? leaf0[h] : gp0;
        out0[h] = static_cast<T>(static_cast<double>(f0) * v);
        for (int g = 1; g < ng; ++g) {
            const float f = h >= Ht ? 0.f : gleaf[g] >= 0 ? __ldg(V.leaf + gleaf[g] + h) : gpay[g];
            V.val[static_cast<size_t>(gnode[g]) * HS + h] = static_cast<T>(static_cast<double>(f) * v);
        }
    }
}

template <class T>
__global__ void __launch_bounds__(kTermThreads) k_term_cr1(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                           const TermItem *__restrict__ items, int trav) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    cr1_terminal<T>(c0, ctxs, items + blockIdx.x, trav, smem, threadIdx.x, [] { __syncthreads(); });
}

template <class T>
constexpr size_t sd1_smem() {
    return 1326 * sizeof(T) + 1327 * 8 + 52 * 53 * 8 + 52 * 4 + 8 * 8 + 52 * 8 + 64;
}

// Showdown against one live opponent (street_solve.cu:886-903): with W, T, L
// the opponent reach on compatible hands that are weaker, tied and stronger,
// value = (pot - bet) W + (pot/2 - bet) T - bet L.  Combos are ranked once per board; the
// block builds the opponent's reach in rank order, its prefix sums P and
// per-card prefix sums PC[c], and then for a traverser combo (c1, c2) with
// tie group [lo, hi):
//   W = P[lo] - PC[c1][<lo] - PC[c2][<lo]
//   T = P[hi] - P[lo] - (PC[c1][<hi] - PC[c1][<lo]) - (PC[c2][<hi] - PC[c2][<lo]) + f(h)
//   S = P[end] - PC[c1][end] - PC[c2][end] + f(h)
// A traverser hand with no compatible positive-reach opponent hand gets
// exactly 0 (positive-reach masks per card, as in the two-opponent kernels).
//
// NT = kSd1Threads is for few showdowns, whose launch waits for one block: eight
// warps scan the rank positions while the other 24 take the cards' lists, and
// every table that no kernel writes is read before the wait for the previous
// kernel where a register can hold it.  (Not of a member that has left the
// batch: its tables are freed.  The live flag is written by a copy, which the
// kernels' order cannot overtake.)  NT = kTermThreads is for many, where five
// small blocks per SM do more than two large ones: one step after the other,
// the reach scattered hand by hand (a narrow range touches its own hands, not
// every position).  Same sums in the same order.
constexpr int kSd1Threads = 1024;
constexpr int kSd1Scan = 256;   // threads of the rank-order scan (fixes its summation order)
template <int NT, class T>
__device__ __forceinline__ void sd1_terminal(const DevCtx &c0, const DevCtx *__restrict__ ctxs,
                                             const TermItem *__restrict__ item, int trav, char *smem) {
    Carve cv{smem};
    T *Rr = cv.take<T>(1326);
    double *Pp = cv.take<double>(1327);
    double *PC = cv.take<double>(52 * 53);
    int *clen = cv.take<int>(52);
    double *wsum = cv.take<double>(kSd1Scan / 32);
    unsigned long long *B = cv.take<unsigned long long>(52);
    const TermItem I = *item;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nc = c.ncomb, HS = c.HS, Ht = c.H[trav];
    const int o = I.opp_player[0];
    const bool dup = c.dup[o] != 0;
    const int *ph = c.pos_hand + static_cast<size_t>(o) * nc;
    const int *tpos = c.sd_pos + static_cast<size_t>(trav) * HS;
    const bool gone = retired(ctxs, I.sg);
    constexpr bool kFew = NT > kSd1Scan;
    const int ph0 = kFew && !gone && tid < nc ? __ldg(ph + tid) : -1;
    const int q0 = kFew && !gone && tid < Ht ? __ldg(tpos + tid) : -1;
    wait_prior_grid();
    if (gone) return;
    const T *r = reach_rows<T>(c) + static_cast<size_t>(I.opp_row[0]) * HS;
    if (kFew && !dup) {
        // the opponent's reach by rank position, gathered
        for (int q = tid; q < nc; q += NT) {
            const int j = q == tid ? ph0 : __ldg(ph + q);
            Rr[q] = j >= 0 ? r[j] : T(0);
        }
    } else {
        for (int i = tid; i < nc; i += NT) Rr[i] = T(0);
        __syncthreads();
        const int *pos = c.sd_pos + static_cast<size_t>(o) * HS;
        for (int j = tid; j < c.H[o]; j += NT) {
            const int q = pos[j];
            if (q < 0) continue;
            if (dup)
                atomicAdd(&Rr[q], r[j]);
            else
                Rr[q] = r[j];
        }
    }
    __syncthreads();
    if (!kFew || warp < kSd1Scan / 32) {
        // exclusive prefix over rank positions: each thread scans a contiguous chunk
        const int per = (nc + kSd1Scan - 1) / kSd1Scan;
        const int b0 = tid * per, b1 = min(nc, b0 + per);
        double local = 0.0;
        for (int i = b0; i < b1; ++i) local += Rr[i];
        double incl = local;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, incl, k);
            if (lane >= k) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        asm volatile("bar.sync 1, %0;" ::"n"(kSd1Scan) : "memory");
        double base = 0.0;
        for (int w = 0; w < warp; ++w) base += wsum[w];
        double run = base + incl - local;
        for (int i = b0; i < b1; ++i) {
            Pp[i] = run;
            run += Rr[i];
        }
        if (tid == kSd1Scan - 1) {
            double tot = 0.0;
            for (int w = 0; w < kSd1Scan / 32; ++w) tot += wsum[w];
            Pp[nc] = tot;
        }
    }
    if (!kFew || warp >= kSd1Scan / 32) {
        // per card: exclusive prefix sums over its combos in rank order, and
        // the mask of partner cards whose combo holds positive reach
        constexpr int kFirst = kFew ? kSd1Scan / 32 : 0;
        for (int card = warp - kFirst; card < 52; card += NT / 32 - kFirst) {
            const short *L = c.sd_card_list + card * 52;
            const short *Pt = c.sd_card_partner + card * 52;
            const int i0 = 2 * lane, i1 = 2 * lane + 1;
            const int q0c = i0 < 52 ? L[i0] : -1, q1c = i1 < 52 ? L[i1] : -1;
            const T f0 = q0c >= 0 ? Rr[q0c] : T(0), f1 = q1c >= 0 ? Rr[q1c] : T(0);
            const double v0 = f0, v1 = f1;
            const double pair = v0 + v1;
            double incl = pair;
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                const double y = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += y;
            }
            const double ex = incl - pair;
            const int len =
                __popc(__ballot_sync(0xffffffffu, q0c >= 0)) + __popc(__ballot_sync(0xffffffffu, q1c >= 0));
            if (i0 <= len) PC[card * 53 + i0] = ex;
            if (i1 <= len) PC[card * 53 + i1] = ex + v0;
            unsigned long long m = 0ull;
            if (f0 > T(0)) m |= 1ull << Pt[i0];
            if (f1 > T(0)) m |= 1ull << Pt[i1];
            const unsigned lo = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(m));
            const unsigned hi = __reduce_or_sync(0xffffffffu, static_cast<unsigned>(m >> 32));
            if (lane == 0) {
                clen[card] = len;
                B[card] = static_cast<unsigned long long>(lo) | (static_cast<unsigned long long>(hi) << 32);
            }
        }
    }
    __syncthreads();
    // positive-reach hands of the opponent (every warp for itself)
    const int np_ = (__reduce_add_sync(0xffffffffu, __popcll(B[lane]) + (lane + 32 < 52 ? __popcll(B[lane + 32]) : 0))) / 2;
    T *out = val_rows<T>(c) + static_cast<size_t>(I.node) * HS;
    // payoff per class with the reference's float coefficients (win pot - bet,
    // tie pot * 0.5 - bet, loss -bet): a coefficient that is exactly 0 drops
    // its class exactly, as in the reference's sum
    const double cw = static_cast<double>(I.pot - I.bet), ct = static_cast<double>(I.pot * 0.5f - I.bet);
    const double cl = -static_cast<double>(I.bet);
    for (int h = tid; h < HS; h += NT) {
        double v = 0.0;
        const int q = kFew && h == tid ? q0 : h < Ht ? __ldg(tpos + h) : -1;
        if (q >= 0) {
            const SdCombo s = c.sd_combo[q];
            const unsigned long long B1 = B[s.c1], B2 = B[s.c2];
            if (np_ - __popcll(B1) - __popcll(B2) + bit(B1, s.c2) > 0) {
                const double *p1 = PC + s.c1 * 53, *p2 = PC + s.c2 * 53;
                const double self = Rr[q];
                const double W = Pp[s.lo] - p1[s.l1lo] - p2[s.l2lo];
                const double Tt = (Pp[s.hi] - Pp[s.lo]) - (p1[s.l1hi] - p1[s.l1lo]) -
                                  (p2[s.l2hi] - p2[s.l2lo]) + self;
                const double L = (Pp[nc] - Pp[s.hi]) - (p1[clen[s.c1]] - p1[s.l1hi]) - (p2[clen[s.c2]] - p2[s.l2hi]);
                v = cw * W + ct * Tt + cl * L;
            }
        }
        store_value(out, h, v);
    }
}

template <int NT, class T>
__global__ void __launch_bounds__(NT, NT == kSd1Threads ? 2 : 5) k_term_sd1(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                                          const TermItem *__restrict__ items, int trav) {
    extern __shared__ __align__(16) char smem[];
    sd1_terminal<NT, T>(c0, ctxs, items + blockIdx.x, trav, smem);
}

// Two-way showdowns, one-opponent folds and zero rows of a river in one
// launch: one block per showdown, then one per four folds (256 threads each,
// their own barriers), then one per four zero rows.  A river has tens of
// each, so a launch of its own costs each kind more than its work: on side
// streams of the captured iteration they also doubled the graph's build and
// release time.
constexpr int kLightGroups = kSd1Threads / kTermThreads;
__global__ void __launch_bounds__(kSd1Threads, 2) k_term_light(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                               const TermItem *__restrict__ sd1, int n_sd1,
                                                               const TermItem *__restrict__ cr1, int n_cr1,
                                                               const TermItem *__restrict__ zero, int n_zero,
                                                               int trav) {
    extern __shared__ __align__(16) char smem[];
    int b = blockIdx.x;
    if (b < n_sd1) {
        sd1_terminal<kSd1Threads, float>(c0, ctxs, sd1 + b, trav, smem);
        return;
    }
    wait_prior_grid();
    b -= n_sd1;
    const int group = threadIdx.x / kTermThreads, tid = threadIdx.x % kTermThreads;
    const int cr1_blocks = (n_cr1 + kLightGroups - 1) / kLightGroups;
    if (b < cr1_blocks) {
        const int i = b * kLightGroups + group;
        if (i < n_cr1)
            cr1_terminal<float>(c0, ctxs, cr1 + i, trav, smem + group * cr1_gather_smem<float>(c0.HS), tid, [group] {
                asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kTermThreads) : "memory");
            });
        return;
    }
    const int i = (b - cr1_blocks) * kLightGroups + group;
    if (i >= n_zero) return;
    const TermItem &I = zero[i];
    if (retired(ctxs, I.sg)) return;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    float *out = c.val + static_cast<size_t>(I.node) * c.HS;
    for (int h = tid; h < c.HS; h += kTermThreads) out[h] = 0.f;
}

// --------------------------------------------------------------------------
// Many iterations of a small heads-up subgame in one cooperative launch: the
// terminals of a traverser spread over the blocks, a grid barrier, the
// traverser's tree (8 hands per block), a grid barrier, and so on.
//
// Such an iteration is bound by the latency of its chain of dependent steps.
// As launches it was four kernels of 7-8 us, and in this form with the tree in
// global memory still 8 us a phase: each level's values and regrets made a
// round trip through L2 (4,000 cycles a level).  So a block keeps what only
// its own hands touch in shared memory for the whole launch -- regrets,
// strategy sums, the pass's values and reach -- beside the tables that no
// kernel writes; what crosses the blocks is the reach rows (to the other
// player's terminals) and the terminal rows, one L2 round trip each per phase.
// Summation orders and expressions are those of the separate kernels.
// Per iteration: heads-up river of 51 nodes and 1081 hands 34.9 us as launches,
// 18.0 so (with four items per block 19.5: terminals 4.5 us, tree 3.3 us, two
// barriers 1.5 us each, twice); 141 nodes and 90 hands 35.5 -> 19.7; turn of
// 1,081 nodes and 1128 hands 59 -> 38.9.
// --------------------------------------------------------------------------
constexpr int kSmallThreads = kSd1Threads;

// All blocks of the (cooperative) grid; count starts at 0 and grows by
// gridDim.x per barrier.  False when the wait ran out: the fault word is set
// and the caller returns.
__device__ bool grid_barrier(unsigned *count, unsigned *fault, unsigned limit) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned before;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(count) : "memory");
        const unsigned target = (before / gridDim.x + 1u) * gridDim.x;
        unsigned now = before + 1u, polls = 0;
        while (static_cast<int>(now - target) < 0 && polls++ < limit)
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(count) : "memory");
        ok = static_cast<int>(now - target) >= 0;
        if (!ok) atomicOr(fault, 1u);
    }
    __syncthreads();
    return ok != 0;
}

// Tables of one traverser's terminals in shared memory.
struct SmallHand {         // a traverser hand at showdowns and folds
    unsigned a, b, c;      // a: rank position | lo << 11; b: hi | c1 << 11 | c2 << 17 | unranked << 31;
};                         // c: l1lo | l1hi << 6 | l2lo << 12 | l2hi << 18
// (beside them: the player's hand at each rank position as short, -1 if none;
// per card the rank positions of its combos as short, -1 past them, and their
// number; per traverser hand dense a | dense b << 6 | its index
// in the opponent's range << 12; the player's hand of each dense-card pair as
// short, HS if none)

__host__ __device__ constexpr size_t small_fold_space(int HS) { return (static_cast<size_t>(HS) + 4) * sizeof(float) + 64 * 12 + 64; }

SmallLayout small_layout(const SmallRef &s, int HS, int ncomb, const int *H) {
    SmallLayout L{};
    unsigned at = 0;
    auto take = [&](size_t bytes) {
        const unsigned off = at;
        at += static_cast<unsigned>((bytes + 15) / 16 * 16);
        return off;
    };
    const bool river = s.n_sd1[0] + s.n_sd1[1] > 0, folds = s.n_cr1[0] + s.n_cr1[1] > 0;
    const size_t row = kTreeHands * sizeof(float);
    for (int p = 0; p < 2; ++p) L.tab[p] = take(s.tree[p].bytes);
    for (int p = 0; p < 2; ++p) L.sd[p] = take(river ? H[p] * sizeof(SmallHand) : 0);
    for (int p = 0; p < 2; ++p) L.pos_hand[p] = take(river ? ncomb * sizeof(short) : 0);
    L.list = take(river ? 52 * 52 * sizeof(short) : 0);
    L.clen = take(river ? 52 * sizeof(int) : 0);
    for (int p = 0; p < 2; ++p) L.fold[p] = take(folds ? H[p] * sizeof(unsigned) : 0);
    for (int p = 0; p < 2; ++p) L.pair[p] = take(folds ? 52 * 52 * sizeof(short) : 0);
    for (int p = 0; p < 2; ++p) L.R[p] = take(s.tree[p].n_edges * row);
    for (int p = 0; p < 2; ++p) L.S[p] = take(s.tree[p].n_edges * row);
    // the phases' own space: a showdown, four folds, or a pass's rows and reach
    size_t work = 0;
    if (river) work = std::max(work, sd1_smem<float>());
    if (folds) work = std::max(work, kLightGroups * small_fold_space(HS));
    for (int p = 0; p < 2; ++p)
        work = std::max(work, (static_cast<size_t>(s.tree[p].n_rows) + s.tree[p].n_edges) * row);
    L.phase = take(work);
    L.total = at;
    return L;
}

// One two-way showdown (sd1_terminal on the tables in shared memory).
__device__ __forceinline__ void small_sd1(const DevCtx &c, const SmallHand *hands, const short *pos_hand,
                                          const short *card_list, const int *clen, const TermItem &I, int trav,
                                          char *smem) {
    Carve cv{smem};
    float *Rr = cv.take<float>(1326);
    double *Pp = cv.take<double>(1327);
    double *PC = cv.take<double>(52 * 53);
    double *wsum = cv.take<double>(kSd1Scan / 32);
    int *wpos = cv.take<int>(kSmallThreads / 32);   // positions of positive reach, per warp
    int *npos = cv.take<int>(52);                   // and per card
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kRounds = (kMaxHS + kSmallThreads - 1) / kSmallThreads;   // positions, hands per thread
    const int nc = c.ncomb, HS = c.HS, Ht = c.H[trav], opp = 1 - trav;
    const float *r = c.reach + static_cast<size_t>(I.opp_row[0]) * HS;
    if (!c.dup[opp]) {
        float x[kRounds];
#pragma unroll
        for (int k = 0; k < kRounds; ++k) {
            const int q = tid + k * kSmallThreads, j = q < nc ? pos_hand[q] : -1;
            x[k] = j >= 0 ? r[j] : 0.f;
        }
        int pos = 0;
#pragma unroll
        for (int k = 0; k < kRounds; ++k) {
            pos += __popc(__ballot_sync(0xffffffffu, x[k] > 0.f));
            if (tid + k * kSmallThreads < nc) Rr[tid + k * kSmallThreads] = x[k];
        }
        if (lane == 0) wpos[warp] = pos;
    } else {
        for (int i = tid; i < nc; i += kSmallThreads) Rr[i] = 0.f;
        __syncthreads();
        const int *pos = c.sd_pos + static_cast<size_t>(opp) * HS;
        for (int j = tid; j < c.H[opp]; j += kSmallThreads)
            if (pos[j] >= 0) atomicAdd(&Rr[pos[j]], r[j]);
        __syncthreads();
        int n = 0;
        for (int q = warp * 32; q < nc; q += kSmallThreads)
            n += __popc(__ballot_sync(0xffffffffu, q + lane < nc && Rr[q + lane] > 0.f));
        if (lane == 0) wpos[warp] = n;
    }
    __syncthreads();
    if (warp < kSd1Scan / 32) {
        // each thread's run of at most kRun positions in registers
        constexpr int kRun = (1326 + kSd1Scan - 1) / kSd1Scan;
        const int per = (nc + kSd1Scan - 1) / kSd1Scan, b0 = tid * per;
        double x[kRun], local = 0.0;
#pragma unroll
        for (int i = 0; i < kRun; ++i) x[i] = i < per && b0 + i < nc ? static_cast<double>(Rr[b0 + i]) : 0.0;
        local = x[0];
#pragma unroll
        for (int i = 1; i < kRun; ++i)
            if (i < per) local += x[i];
        double incl = local;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, incl, k);
            if (lane >= k) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        asm volatile("bar.sync 1, %0;" ::"n"(kSd1Scan) : "memory");
        double ws[kSd1Scan / 32], base = 0.0, tot = 0.0;
#pragma unroll
        for (int w = 0; w < kSd1Scan / 32; ++w) ws[w] = wsum[w];
#pragma unroll
        for (int w = 0; w < kSd1Scan / 32; ++w) {
            if (w == warp) base = tot;
            tot += ws[w];
        }
        double run = base + incl - local;
#pragma unroll
        for (int i = 0; i < kRun; ++i) {
            if (i < per) {
                if (b0 + i < nc) Pp[b0 + i] = run;
                run += x[i];
            }
        }
        if (tid == kSd1Scan - 1) Pp[nc] = tot;
    } else {
        // this warp's cards side by side (one at a time is a chain of
        // shuffles and FP64 additions per card)
        constexpr int kCardWarps = (kSmallThreads - kSd1Scan) / 32, kCards = (52 + kCardWarps - 1) / kCardWarps;
        const int i0 = 2 * lane, i1 = 2 * lane + 1, c0 = warp - kSd1Scan / 32;
        double v0[kCards], pair[kCards], incl[kCards];
#pragma unroll
        for (int k = 0; k < kCards; ++k) {
            const int card = c0 + k * kCardWarps;
            const bool on = card < 52 && i0 < 52;   // i1 = i0 + 1 < 52 as well
            const short2 q = on ? *reinterpret_cast<const short2 *>(card_list + card * 52 + i0) : make_short2(-1, -1);
            const float f0 = q.x >= 0 ? Rr[q.x] : 0.f, f1 = q.y >= 0 ? Rr[q.y] : 0.f;
            v0[k] = f0;
            pair[k] = incl[k] = static_cast<double>(f0) + static_cast<double>(f1);
            const int n = __popc(__ballot_sync(0xffffffffu, f0 > 0.f)) + __popc(__ballot_sync(0xffffffffu, f1 > 0.f));
            if (lane == 0 && card < 52) npos[card] = n;
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            double y[kCards];
#pragma unroll
            for (int k = 0; k < kCards; ++k) y[k] = __shfl_up_sync(0xffffffffu, incl[k], d);
#pragma unroll
            for (int k = 0; k < kCards; ++k)
                if (lane >= d) incl[k] += y[k];
        }
#pragma unroll
        for (int k = 0; k < kCards; ++k) {
            const int card = c0 + k * kCardWarps;
            if (card >= 52) continue;
            const int len = clen[card];
            const double ex = incl[k] - pair[k];
            if (i0 <= len) PC[card * 53 + i0] = ex;
            if (i1 <= len) PC[card * 53 + i1] = ex + v0[k];
        }
    }
    __syncthreads();
    const int N = __reduce_add_sync(0xffffffffu, wpos[lane]);
    const double total = Pp[nc];
    float *out = c.val + static_cast<size_t>(I.node) * HS;
    const double cw = static_cast<double>(I.pot - I.bet), ct = static_cast<double>(I.pot * 0.5f - I.bet);
    const double cl = -static_cast<double>(I.bet);
    double v[kRounds];
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
        const int h = tid + k * kSmallThreads;
        v[k] = 0.0;
        const SmallHand e = h < Ht ? hands[h] : SmallHand{0u, 1u << 31, 0u};
        if (!(e.b >> 31)) {
            const int q = e.a & 2047, lo = e.a >> 11, hi = e.b & 2047;
            const int c1 = e.b >> 11 & 63, c2 = e.b >> 17 & 63;
            const int l1lo = e.c & 63, l1hi = e.c >> 6 & 63, l2lo = e.c >> 12 & 63, l2hi = e.c >> 18 & 63;
            const double *p1 = PC + c1 * 53, *p2 = PC + c2 * 53;
            const float self = Rr[q];
            const double W = Pp[lo] - p1[l1lo] - p2[l2lo];
            const double Tt = (Pp[hi] - Pp[lo]) - (p1[l1hi] - p1[l1lo]) - (p2[l2hi] - p2[l2lo]) + static_cast<double>(self);
            const double L = (total - Pp[hi]) - (p1[clen[c1]] - p1[l1hi]) - (p2[clen[c2]] - p2[l2hi]);
            const double x = cw * W + ct * Tt + cl * L;
            // a hand without a compatible hand of positive reach gets exactly 0
            if (N - npos[c1] - npos[c2] + (self > 0.f ? 1 : 0) > 0) v[k] = x;
        }
    }
#pragma unroll
    for (int k = 0; k < kRounds; ++k)
        if (tid + k * kSmallThreads < HS) store_value(out, tid + k * kSmallThreads, v[k]);
}

// One group of one-opponent folds or leaves (cr1_terminal on the tables in
// shared memory) by kTermThreads threads with barrier `bar`.
__device__ __forceinline__ void small_cr1(const DevCtx &c, const unsigned *hands, const short *pair,
                                          const TermItem *__restrict__ I0, int trav, char *smem, int tid, int bar) {
    constexpr int kRounds = (kMaxHS + kTermThreads - 1) / kTermThreads;
    auto sync = [bar] { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kTermThreads) : "memory"); };
    const int ng = I0->gextra + 1, lane = tid & 31;
    const int HS = c.HS, Ht = c.H[trav], Dp = (c.deck + 3) & ~3;
    Carve cv{smem};
    float *r = cv.take<float>(HS + 4);
    double *u = cv.take<double>(64);
    int *nz = cv.take<int>(64);
    const float *src = c.reach + static_cast<size_t>(I0->opp_row[0]) * HS;
    for (int q = tid * 4; q < HS; q += kTermThreads * 4) cp_async16(r + q, src + q);
    // an item's factors of this thread's hands, loaded well before their use
    auto factors = [&](const TermItem &I, float f[kRounds]) {
        const int lo = __ldg(&I.leaf_off);
        const float pay = __ldg(&I.payoff);
#pragma unroll
        for (int k = 0; k < kRounds; ++k) {
            const int h = tid + k * kTermThreads;
            f[k] = h >= Ht ? 0.f : lo >= 0 ? __ldg(c.leaf_values + lo + h) : pay;
        }
    };
    float f[kRounds];
    factors(*I0, f);
    if (tid == 0) r[HS] = 0.f;
    if (tid < 64) {
        u[tid] = 0.0;
        nz[tid] = 0;
    }
    cp_async_wait_all();
    sync();
    {
        const int col = tid >> 2, part = tid & 3, q = Dp >> 2;
        double s = 0.0;
        int n = 0;
        if (col < Dp) {
            const short *row = pair + col * 52 + part * q;
            for (int b = 0; b < q; ++b) {
                const float x = r[row[b]];
                s += static_cast<double>(x);
                n += x > 0.f ? 1 : 0;
            }
        }
#pragma unroll
        for (int k = 1; k < 4; k <<= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, k);
            n += __shfl_xor_sync(0xffffffffu, n, k);
        }
        if (part == 0 && col < Dp) {
            u[col] = s;
            nz[col] = n;
        }
    }
    sync();
    double F;
    int N;
    {
        double s = (lane < Dp ? u[lane] : 0.0) + (lane + 32 < Dp ? u[lane + 32] : 0.0);
        int n = (lane < Dp ? nz[lane] : 0) + (lane + 32 < Dp ? nz[lane + 32] : 0);
        s = warp_sum(s);
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) n += __shfl_xor_sync(0xffffffffu, n, k);
        F = 0.5 * s;
        N = n / 2;
    }
    double v[kRounds];
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
        const int h = tid + k * kTermThreads;
        v[k] = 0.0;
        if (h < Ht) {
            const unsigned e = hands[h];
            const int a = e & 63, b = e >> 6 & 63;
            const float x = r[e >> 12];
            const int live = N - nz[a] - nz[b] + (x > 0.f ? 1 : 0);
            if (live > 0) v[k] = F - u[a] - u[b] + static_cast<double>(x);
        }
    }
    for (int g = 0; g < ng; ++g) {
        float *out = c.val + static_cast<size_t>(__ldg(&I0[g].node)) * HS;
        float fn[kRounds];
        if (g + 1 < ng)
            factors(I0[g + 1], fn);
        else
            for (int k = 0; k < kRounds; ++k) fn[k] = 0.f;
#pragma unroll
        for (int k = 0; k < kRounds; ++k) {
            const int h = tid + k * kTermThreads;
            if (h < HS) out[h] = static_cast<float>(static_cast<double>(f[k]) * v[k]);
            f[k] = fn[k];
        }
    }
}

// One player's values and regrets bottom-up, then its reach top-down, for hand
// h of the block's 8 (act: a hand of the range): rv holds the frontier rows,
// rs the reach of the local edges, weight the hand's range weight.  Iteration
// t; node values also go to global memory with `keep`.
//
// A warp per item, a lane per (action, hand): one thread walking an item's
// actions was a chain of some 300 dependent instructions, 6,000 cycles a
// level.  The sums over actions run in action order on shuffled operands, the
// same in every lane of a hand.
__device__ __forceinline__ void whole_pass(const DevCtx &c, const WholeRef &T, const char *tab, float *R, float *S,
                                           float *rv, float *rs, int h, bool act, float weight, int t, bool keep) {
    const WholeItem *items = reinterpret_cast<const WholeItem *>(tab);
    const WholeReach *reach = reinterpret_cast<const WholeReach *>(tab + T.o_reach);
    const short *edge_end = reinterpret_cast<const short *>(tab + T.o_end);
    const int *rows = reinterpret_cast<const int *>(tab + T.o_rows);
    const int *voff = reinterpret_cast<const int *>(tab + T.o_voff), *roff = reinterpret_cast<const int *>(tab + T.o_roff);
    const int hand = threadIdx.x & (kTreeHands - 1), warp = threadIdx.x >> 5;
    const int a4 = (threadIdx.x & 31) / kTreeHands;   // this lane's actions: a4 and a4 + 4
    constexpr int kWarps = kSmallThreads / 32, kSlots = kSmallThreads / kTreeHands;
    static_assert(kTreeHands == 8 && SS_MAX_ACTIONS == 8, "a warp covers four actions of eight hands, twice");
    const size_t HS = static_cast<size_t>(c.HS);
    const float d = static_cast<float>(t) / (static_cast<float>(t) + 1.0f);
    const float w = static_cast<float>(t);
    if (act) {
        const float *val = c.val + h;
        constexpr int kAhead = 8;   // rows in flight per thread
        for (int i0 = threadIdx.x / kTreeHands; i0 < T.n_rows; i0 += kAhead * kSlots) {
            int row[kAhead];
            float x[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) row[k] = i0 + k * kSlots < T.n_rows ? rows[i0 + k * kSlots] : -1;
#pragma unroll
            for (int k = 0; k < kAhead; ++k) x[k] = row[k] >= 0 ? val[static_cast<size_t>(row[k]) * HS] : 0.f;
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (row[k] >= 0) rv[(i0 + k * kSlots) * kTreeHands + hand] = x[k];
        }
    }
    __syncthreads();
    // the strategy of this lane's actions from their regrets
    auto strategy = [&](const float r[2], int na, int frozen, float uniform, float sig[2]) {
        float rp[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) rp[j] = a4 + 4 * j < na && r[j] > 0.f ? r[j] : 0.f;
        // past the node's actions rp is +0, which changes no sum
        float x[4], sum = 0.f;
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = __shfl_sync(0xffffffffu, rp[0], a * kTreeHands + hand);
#pragma unroll
        for (int a = 0; a < 4; ++a) sum += x[a];
        if (na > 4) {
#pragma unroll
            for (int a = 0; a < 4; ++a) x[a] = __shfl_sync(0xffffffffu, rp[1], a * kTreeHands + hand);
#pragma unroll
            for (int a = 0; a < 4; ++a) sum += x[a];
        }
        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            sig[j] = sum > 0.f ? rp[j] * inv : uniform;
            if (frozen >= 0) sig[j] = a4 + 4 * j == frozen ? 1.0f : 0.0f;
        }
    };
    for (int l = 0; l < T.value_levels; ++l) {
        for (int it = voff[l] + warp; it < voff[l + 1]; it += kWarps) {
            const WholeItem I = items[it];
            const int na = I.na;
            float r[2] = {0.f, 0.f}, ev[2] = {0.f, 0.f}, sig[2], sm[2] = {0.f, 0.f};
            float *Rh = R + (I.edge0 + a4) * kTreeHands + hand, *Sh = S + (I.edge0 + a4) * kTreeHands + hand;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (j == 1 && na <= 4) break;
                const int a = a4 + 4 * j;
                if (a >= na) continue;
                r[j] = Rh[4 * j * kTreeHands];
                sm[j] = Sh[4 * j * kTreeHands];
                int k = a ? edge_end[I.edge0 + a - 1] : I.row0;
                const int end = edge_end[I.edge0 + a];
                const float *x = rv + hand;
                if (I.split == 1) {
                    float e = 0.f;
                    for (; k + 3 < end; k += 4) {
                        const float x0 = x[k * kTreeHands], x1 = x[(k + 1) * kTreeHands];
                        const float x2 = x[(k + 2) * kTreeHands], x3 = x[(k + 3) * kTreeHands];
                        e += x0;
                        e += x1;
                        e += x2;
                        e += x3;
                    }
                    for (; k < end; ++k) e += x[k * kTreeHands];
                    ev[j] = e;
                } else {
                    // four interleaved chains, added in order
                    static_assert(kCfvSplit == 4, "four chains");
                    float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
                    for (; k < end; k += 4) {
                        q0 += x[k * kTreeHands];
                        if (k + 1 < end) q1 += x[(k + 1) * kTreeHands];
                        if (k + 2 < end) q2 += x[(k + 2) * kTreeHands];
                        if (k + 3 < end) q3 += x[(k + 3) * kTreeHands];
                    }
                    ev[j] = q0 + q1 + q2 + q3;
                }
            }
            strategy(r, na, I.frozen, I.uniform, sig);
            // past the node's actions ev is +0, whose products add nothing
            float v = 0.f;
            auto add4 = [&](float sj, float ej) {
                float sa[4], ea[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    sa[a] = __shfl_sync(0xffffffffu, sj, a * kTreeHands + hand);
                    ea[a] = __shfl_sync(0xffffffffu, ej, a * kTreeHands + hand);
                }
#pragma unroll
                for (int a = 0; a < 4; ++a) v += sa[a] * ea[a];
            };
            add4(sig[0], ev[0]);
            if (na > 4) add4(sig[1], ev[1]);
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if ((j == 0 || na > 4) && a4 + 4 * j < na) {
                    Rh[4 * j * kTreeHands] = (r[j] + (ev[j] - v)) * d;
                    Sh[4 * j * kTreeHands] = sm[j] + w * sig[j];
                }
            v *= I.scale;
            if (a4 == 0) {
                if (I.row >= 0) rv[I.row * kTreeHands + hand] = v;
                if (keep && act) c.val[static_cast<size_t>(I.node) * HS + h] = v;
            }
        }
        __syncthreads();
    }
    for (int l = 0; l < T.reach_levels; ++l) {
        for (int it = roff[l] + warp; it < roff[l + 1]; it += kWarps) {
            const WholeReach I = reach[it];
            const int na = I.na;
            const float pr = I.parent >= 0 ? rs[I.parent * kTreeHands + hand] : weight;
            float r[2] = {0.f, 0.f}, sig[2];
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if ((j == 0 || na > 4) && a4 + 4 * j < na) r[j] = R[(I.edge0 + a4 + 4 * j) * kTreeHands + hand];
            strategy(r, na, I.frozen, I.uniform, sig);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int a = a4 + 4 * j;
                if ((j == 1 && na <= 4) || a >= na) continue;
                const float x = pr * sig[j];
                rs[(I.edge0 + a) * kTreeHands + hand] = x;
                if (act) c.reach[static_cast<size_t>(I.first_edge + a) * HS + h] = x;
            }
        }
        if (l + 1 < T.reach_levels) __syncthreads();   // a grid barrier follows the last
    }
}

__global__ void __launch_bounds__(kSmallThreads, 1) k_small_solve(const __grid_constant__ DevCtx c,
                                                                const __grid_constant__ SmallRef s, int iters,
                                                                int snapshot) {
    extern __shared__ __align__(16) char smem[];
    const size_t HS = static_cast<size_t>(c.HS);
    const bool river = s.n_sd1[0] + s.n_sd1[1] > 0, folds = s.n_cr1[0] + s.n_cr1[1] > 0;
    const int hand = threadIdx.x & (kTreeHands - 1), h = blockIdx.x * kTreeHands + hand;
    // an earlier launch gave up: its rows are no state to go on from.  (One thread
    // asks for the block: this launch's own blocks may set the word meanwhile, and
    // the named barriers below count on every thread.)
    if (__syncthreads_or(threadIdx.x == 0 && *s.fault != 0u)) return;
    float weight0 = 0.f, weight1 = 0.f;
    // tables and the block's rows
    for (int p = 0; p < 2; ++p) {
        const int4 *src = reinterpret_cast<const int4 *>(s.tree[p].blob);
        for (int i = threadIdx.x; i < s.tree[p].bytes / 16; i += kSmallThreads)
            reinterpret_cast<int4 *>(smem + s.at.tab[p])[i] = __ldg(src + i);
        if (river) {
            for (int q = threadIdx.x; q < c.ncomb; q += kSmallThreads)
                reinterpret_cast<short *>(smem + s.at.pos_hand[p])[q] = static_cast<short>(__ldg(c.pos_hand + static_cast<size_t>(p) * c.ncomb + q));
            for (int i = threadIdx.x; i < c.H[p]; i += kSmallThreads) {
                const int q = __ldg(c.sd_pos + p * HS + i);
                SmallHand e{0u, 1u << 31, 0u};
                if (q >= 0) {
                    const SdCombo &k = c.sd_combo[q];
                    e.a = static_cast<unsigned>(q) | static_cast<unsigned>(k.lo) << 11;
                    e.b = static_cast<unsigned>(k.hi) | static_cast<unsigned>(k.c1) << 11 | static_cast<unsigned>(k.c2) << 17;
                    e.c = static_cast<unsigned>(k.l1lo) | static_cast<unsigned>(k.l1hi) << 6 |
                          static_cast<unsigned>(k.l2lo) << 12 | static_cast<unsigned>(k.l2hi) << 18;
                }
                reinterpret_cast<SmallHand *>(smem + s.at.sd[p])[i] = e;
            }
        }
        if (folds) {
            for (int i = threadIdx.x; i < 52 * 52; i += kSmallThreads)
                reinterpret_cast<short *>(smem + s.at.pair[p])[i] = static_cast<short>(__ldg(c.pair_idx + p * 52 * 52 + i));
            for (int i = threadIdx.x; i < c.H[p]; i += kSmallThreads) {
                const int hc = __ldg(c.hand_code + p * HS + i);
                const unsigned a = min((hc >> 20) & 63, kCr2Off), b = min((hc >> 26) & 63, kCr2Off);
                const unsigned x = __ldg(c.cross_idx + (static_cast<size_t>(p) * c.np + (1 - p)) * HS + i);
                reinterpret_cast<unsigned *>(smem + s.at.fold[p])[i] = a | b << 6 | x << 12;
            }
        }
    }
    {
        const float *own = c.reach + static_cast<size_t>(s.tree[0].n_edges + s.tree[1].n_edges) * HS + h;
        if (h < c.H[0]) weight0 = own[0];
        if (h < c.H[1]) weight1 = own[HS];
    }
    if (river)
        for (int i = threadIdx.x; i < 52 * 52; i += kSmallThreads)
            reinterpret_cast<short *>(smem + s.at.list)[i] = __ldg(c.sd_card_list + i);
    if (river && threadIdx.x < 52) {
        int n = 0;
        while (n < 52 && __ldg(c.sd_card_list + threadIdx.x * 52 + n) >= 0) ++n;
        reinterpret_cast<int *>(smem + s.at.clen)[threadIdx.x] = n;
    }
    __syncthreads();
    // the block's regrets and strategy sums, in and (at the end) out
    auto rows = [&](bool out) {
        for (int p = 0; p < 2; ++p) {
            const int *edge_row = reinterpret_cast<const int *>(smem + s.at.tab[p] + s.tree[p].o_edge);
            float *R = reinterpret_cast<float *>(smem + s.at.R[p]), *S = reinterpret_cast<float *>(smem + s.at.S[p]);
            if (h < c.H[p])
                for (int e = threadIdx.x / kTreeHands; e < s.tree[p].n_edges; e += kSmallThreads / kTreeHands) {
                    const size_t g = static_cast<size_t>(edge_row[e]) * HS + h;
                    if (out) {
                        c.R[g] = R[e * kTreeHands + hand];
                        c.S[g] = S[e * kTreeHands + hand];
                    } else {
                        R[e * kTreeHands + hand] = c.R[g];
                        S[e * kTreeHands + hand] = c.S[g];
                    }
                }
        }
    };
    rows(false);
    __shared__ TermItem first_sd1[2];
    if (threadIdx.x < 2 && static_cast<int>(blockIdx.x) < s.n_sd1[threadIdx.x])
        first_sd1[threadIdx.x] = s.sd1[threadIdx.x][blockIdx.x];
    const int base = *c.iter;
    const int group = threadIdx.x / kTermThreads, tid = threadIdx.x % kTermThreads;
    // the first fold or leaf of either traverser is the same every iteration
    int first_cr1[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int j = static_cast<int>(blockIdx.x) - s.n_sd1[t], i = j + group * s.cr1_jobs[t];
        first_cr1[t] = j >= 0 && i < s.n_cr1[t] ? __ldg(s.cr1_head[t] + i) : 0;
    }
    char *work = smem + s.at.phase;
    __syncthreads();
    for (int it = 1; it <= iters; ++it) {
        for (int t = 0; t < 2; ++t) {
            const int n_sd1 = s.n_sd1[t], n_cr1 = s.n_cr1[t], n_zero = s.n_zero[t];
            const int cr1_jobs = s.cr1_jobs[t];
            const int jobs = n_sd1 + cr1_jobs + (n_zero + kLightGroups - 1) / kLightGroups;
            for (int job = blockIdx.x; job < jobs; job += gridDim.x) {
                if (job < n_sd1) {
                    // the block's first showdown is the same every iteration
                    small_sd1(c, reinterpret_cast<const SmallHand *>(smem + s.at.sd[t]),
                              reinterpret_cast<const short *>(smem + s.at.pos_hand[1 - t]),
                              reinterpret_cast<const short *>(smem + s.at.list),
                              reinterpret_cast<const int *>(smem + s.at.clen), job == static_cast<int>(blockIdx.x) ? first_sd1[t] : s.sd1[t][job], t, work);
                } else if (job < n_sd1 + cr1_jobs) {
                    const int i = job - n_sd1 + group * cr1_jobs;
                    if (i < n_cr1)
                        small_cr1(c, reinterpret_cast<const unsigned *>(smem + s.at.fold[t]),
                                  reinterpret_cast<const short *>(smem + s.at.pair[1 - t]),
                                  s.cr1[t] + (job == static_cast<int>(blockIdx.x) ? first_cr1[t] : __ldg(s.cr1_head[t] + i)), t,
                                  work + group * small_fold_space(c.HS), tid, group + 1);
                } else {
                    const int i = (job - n_sd1 - cr1_jobs) * kLightGroups + group;
                    if (i < n_zero) {
                        float *out = c.val + static_cast<size_t>(s.zero[t][i].node) * HS;
                        for (int k = tid; k < c.HS; k += kTermThreads) out[k] = 0.f;
                    }
                }
                if (job + static_cast<int>(gridDim.x) < jobs) __syncthreads();   // the next job's space
            }
            if (!grid_barrier(s.barrier, s.fault, s.polls)) return;
            float *R = reinterpret_cast<float *>(smem + s.at.R[t]), *S = reinterpret_cast<float *>(smem + s.at.S[t]);
            // the root strategy before the last traverser's pass
            if (snapshot && it == iters && t == 1) {
                const int p = c.root_player;
                const int *edge_row = reinterpret_cast<const int *>(smem + s.at.tab[p] + s.tree[p].o_edge);
                const float *Rp = reinterpret_cast<const float *>(smem + s.at.R[p]);
                int e = 0;   // the root's first local edge
                while (e < s.tree[p].n_edges && edge_row[e] != c.root_fe) ++e;
                if (threadIdx.x < kTreeHands && h < c.H[p]) {
                    float sum = 0.f;
                    for (int a = 0; a < c.root_na; ++a) {
                        const float r = Rp[(e + a) * kTreeHands + hand];
                        sum += r > 0.f ? r : 0.f;
                    }
                    const float inv = sum > 0.f ? 1.0f / sum : 0.f;
                    for (int a = 0; a < c.root_na; ++a) {
                        const float r = Rp[(e + a) * kTreeHands + hand];
                        float x = sum > 0.f ? (r > 0.f ? r : 0.f) * inv : 1.0f / static_cast<float>(c.root_na);
                        if (c.root_frozen >= 0) x = a == c.root_frozen ? 1.0f : 0.0f;
                        c.snap[static_cast<size_t>(a) * c.H[p] + h] = x;
                    }
                }
                __syncthreads();
            }
            float *rv = reinterpret_cast<float *>(work);
            whole_pass(c, s.tree[t], smem + s.at.tab[t], R, S, rv, rv + s.tree[t].n_rows * kTreeHands, h, h < c.H[t],
                       t ? weight1 : weight0, base + it, it == iters);
            if (!grid_barrier(s.barrier, s.fault, s.polls)) return;
        }
    }
    rows(true);
    if (blockIdx.x == 0 && threadIdx.x == 0) *const_cast<int *>(c.iter) = base + iters;
}

// ---------------------------------------------------------------------------
// Three-way showdown (two live opponents), street_solve.cu:936-1002: the
// traverser (strength s) against opponents 1, 2 on disjoint hands o1, o2
// wins pot / (1 + number of opponents tying s) - bet if neither opponent is
// stronger, else loses bet.  With D(X, Y) the mass of opponent pairs
// (o1 in X, o2 in Y) disjoint from each other and from the hand, and L / E
// the opponents' hands weaker than / tying s, the classes are W2 = D(L, L)
// (win), T1 = D(E, L) + D(L, E) (two-way tie), T2 = D(E, E) (three-way tie)
// and the rest of Z = D(all, all) (loss).
// D(X, Y) is the two-opponent card-removal closed form on matrices holding
// only X's and Y's hands.  The kernel sweeps the combos in rank order and
// keeps that form's aggregates (P = M1 M2, u_i, w, d, F_i, Q, D; FP64) for
// the opponents' hands added so far; per tie group of the traverser's hands
// it reads A = D(L, L) before the group and C = D(L+E, L+E) after adding
// both opponents' group hands, and sums D(L, E) over opponent 2's group
// hands and D(E, L) over opponent 1's directly (each term an exact four-card
// removal for the other opponent).  With Z read after the sweep:
//   W2 = A, T1 = D(E, L) + D(L, E), T2 = C - A - T1, lose = Z - C,
//   value = (pot - bet) W2 + (pot/2 - bet) T1 + (pot/3 - bet) T2 - bet lose,
// and T2 = 0 exactly when opponent 2 holds nothing in the group (C is then
// B = D(L+E, L), and C - B the empty class).
// Adding a hand changes two rows (or columns) of P, two card sums and every
// w entry, so each phase gives threads fixed ownership (P cells by column
// and row residue, one card's u / d / w, the scalars, matrix cells), each
// accumulating its share of the phase's hands in registers: no atomics, a
// fixed summation order.  The sweep of a terminal is cut into runs of tie
// groups of about equal cost, one block each, starting from a directly
// computed state (the product P as 3x3 FP64 tiles over all 256 threads).
// C of a group and A of the next are read in one phase (the same state); the
// tie sums of a traverser hand are split over eight lanes.
// ---------------------------------------------------------------------------
constexpr int SD2_S = 49;   // row stride of the sweep's card matrices (odd: conflict-free columns)
constexpr int SD2_N = 48;   // cards a matrix covers (dense indices; a river deck has 47)
constexpr int SD2_W = (1326 + 31) / 32;   // words of a position mask
// live positions (of the opponent with more) up to which a sweep takes the sparse form.  A
// river's 40 three-way showdowns, dense -> sparse form: 61 -> 48 us at 200 hands, 65.5 -> 65.5
// at 400, 66 -> 72 at 550, 74 -> 110 at all 1,081 (walking masks costs more than testing values)
constexpr int SD2_SPARSE = 400;
static_assert(kTermThreads == 256, "the sweep's thread roles assume 256 threads");

// the opponents' reach by rank position; after the sweep the same space holds
// the positive-reach masks, counts and scalars of the exact-zero test
template <class T>
__host__ __device__ constexpr size_t sd2_reach_bytes(int ncomb) {
    return 2 * static_cast<size_t>(ncomb) * sizeof(T) > 53 * sizeof(ulonglong2) + 53 * sizeof(Cr2Cnt) + sizeof(Cr2Scalars)
               ? 2 * static_cast<size_t>(ncomb) * sizeof(T)
               : 53 * sizeof(ulonglong2) + 53 * sizeof(Cr2Cnt) + sizeof(Cr2Scalars);
}

// dynamic shared memory for runs of at most `span` rank positions: P, M1, M2,
// u1, u2, w, d, scalars, per-position classes of the run, reach (masks), the
// cards of each position, the traverser's hand at each position of the run,
// the last positive position; 16 bytes of alignment slack per carve
template <class T>
constexpr size_t sd2_smem(int span, int ncomb) {
    return SD2_S * SD2_S * 8 + 2 * SD2_S * SD2_S * sizeof(T) + 4 * 64 * 8 + 8 * 8 + static_cast<size_t>(span) * 32 +
           sd2_reach_bytes<T>(ncomb) + static_cast<size_t>(ncomb) * 2 + static_cast<size_t>(span) * 2 + 16 +
           2 * SD2_W * 4 + 2 * 48 * 8 + 17 * 16;
}
// Rank positions of any board.  The attribute that allows a launch its shared
// memory is one per kernel, for all host threads: it is set to what the largest
// launch takes, never to this launch's size, which another thread's may exceed
// by the time that it launches.
constexpr int kMaxSpan = 1326;
static_assert(sd2_smem<double>(kMaxSpan, kMaxSpan) <= 227 * 1024, "one block fits");

struct Sd2State {
    double *P, *u1, *u2, *w, *d, *sc;   // sc: F1, F2, Q, D
    // the positions where each opponent's reach is not 0 (bit q % 32 of word q / 32): sparse
    // ranges walk these, and a group where an opponent has none costs it no phase
    unsigned *on1, *on2;
    unsigned long long *row1, *row2;    // direct states: the cells of each matrix row that are not 0
};

// the first position >= q of `on` below hi, or hi (dense: q itself; the caller
// skips the zeros)
template <bool SP>
__device__ __forceinline__ int sd2_next(const unsigned *on, int q, int hi) {
    if (!SP) return q;
    while (q < hi) {
        const unsigned m = on[q >> 5] >> (q & 31);
        if (m) return min(hi, q + __ffs(static_cast<int>(m)) - 1);
        q = (q | 31) + 1;
    }
    return hi;
}

__device__ __forceinline__ int sd2_c1(unsigned short e) { return e & 255; }
__device__ __forceinline__ int sd2_c2(unsigned short e) { return e >> 8; }

// D(., .) of the hand (a, b) on the current sweep state (the two-opponent
// closed form, see k_term_cr2)
// Written with explicit round-to-nearest operations (no contraction into
// FMAs), so two evaluations on the same state agree bit for bit wherever they
// are inlined: the class masses below are differences of such evaluations and
// must come out exactly 0 when the class is empty and the states coincide.
template <class T>
__device__ __forceinline__ double sd2_mass(Sd2State st, const T *M1, const T *M2, int a, int b) {
    const double u1a = st.u1[a], u1b = st.u1[b], u2a = st.u2[a], u2b = st.u2[b];
    const double m1 = static_cast<double>(M1[a * SD2_S + b]), m2 = static_cast<double>(M2[a * SD2_S + b]);
    const double pp = __dadd_rn(st.P[a * SD2_S + b], st.P[b * SD2_S + a]);
    const double ga = __dsub_rn(__dadd_rn(__dmul_rn(u1a, u2a), st.w[a]), __dmul_rn(2.0, st.d[a]));
    const double gb = __dsub_rn(__dadd_rn(__dmul_rn(u1b, u2b), st.w[b]), __dmul_rn(2.0, st.d[b]));
    const double A1 = __dadd_rn(__dsub_rn(__dsub_rn(st.sc[0], u1a), u1b), m1);
    const double A2 = __dadd_rn(__dsub_rn(__dsub_rn(st.sc[1], u2a), u2b), m2);
    double z = __dmul_rn(A1, A2);
    z = __dadd_rn(z, __dsub_rn(st.sc[3], st.sc[2]));
    z = __dadd_rn(z, __dadd_rn(ga, gb));
    z = __dsub_rn(z, __dmul_rn(m2, __dadd_rn(u1a, u1b)));
    z = __dsub_rn(z, __dmul_rn(m1, __dadd_rn(u2a, u2b)));
    z = __dadd_rn(z, __dmul_rn(3.0, __dmul_rn(m1, m2)));
    return __dsub_rn(z, pp);
}

// Add the hands of opponent `who` (0 or 1) at rank positions [lo, hi) to the
// sweep state.  R: that opponent's reach by rank position; Mo: that
// opponent's matrix, Mx: the other's (symmetric); uo / ux: their card sums.
template <bool SP, class T>
__device__ __forceinline__ void sd2_add(Sd2State st, const unsigned short *dd, const T *R, T *Mo, const T *Mx,
                                        double *uo, const double *ux, int who, int lo, int hi) {
    const int tid = threadIdx.x;
    const unsigned *on = who == 0 ? st.on1 : st.on2;
    if (tid < 4 * SD2_N) {
        // P = M1 M2: opponent 1's hand {x, y} adds r Mx[y][.] to row x and
        // r Mx[x][.] to row y; opponent 2's adds the same to columns x, y.
        // Thread (part, j) owns column (row) j of the rows (columns) x with
        // x % 4 == part: the four suits of a rank fall to different threads.
        const int part = tid / SD2_N, j = tid - part * SD2_N;
        for (int q = sd2_next<SP>(on, lo, hi); q < hi; q = sd2_next<SP>(on, q + 1, hi)) {
            const T rt = R[q];
            if (!SP && rt == T(0)) continue;
            const double r = static_cast<double>(rt);
            const unsigned short e = dd[q];
            const int x = sd2_c1(e), y = sd2_c2(e);
            if ((x & 3) == part) {
                double *p = who == 0 ? st.P + x * SD2_S + j : st.P + j * SD2_S + x;
                *p += r * static_cast<double>(Mx[y * SD2_S + j]);
            }
            if ((y & 3) == part) {
                double *p = who == 0 ? st.P + y * SD2_S + j : st.P + j * SD2_S + y;
                *p += r * static_cast<double>(Mx[x * SD2_S + j]);
            }
        }
        return;
    }
    // Warps 6 and 7.  Card c: this opponent's card sum u(c), d(c) = sum_b
    // M1[c][b] M2[c][b] and w(c) = (M2 u1 + M1 u2)(c): the hand changes Mo at
    // (x, y) and uo at x, y.  The lane after the last card takes F (this
    // opponent's total), Q = sum u1 u2 and D = sum d / 2 in the same steps (a
    // branch of its own, and one for Mo's cells, ran after the cards': 500
    // cycles per hand where the other warps took 200 to 250).
    const int c = tid - 4 * SD2_N;
    const bool all = c == SD2_N;
    if (c <= SD2_N) {
        double du = 0.0, dd_c = 0.0, dw = 0.0;
        if (all) {
            du = st.sc[who];
            dw = st.sc[2];
            dd_c = st.sc[3];
        }
        for (int q = sd2_next<SP>(on, lo, hi); q < hi; q = sd2_next<SP>(on, q + 1, hi)) {
            const T rt = R[q];
            if (!SP && rt == T(0)) continue;
            const double r = static_cast<double>(rt);
            const unsigned short e = dd[q];
            const int x = sd2_c1(e), y = sd2_c2(e);
            const bool mine = all || c == x || c == y;
            const double mx = static_cast<double>(Mx[(all ? y : c) * SD2_S + x]);
            const double my = static_cast<double>(Mx[(all ? x : c) * SD2_S + y]);
            const double uy = ux[c == x || all ? y : x];
            dw = fma(r, all ? ux[x] + uy : mx + my, dw);
            if (mine) {
                du += r;
                dd_c = fma(r, c == y ? mx : my, dd_c);
                if (!all) dw = fma(r, uy, dw);
            }
        }
        if (all) {
            st.sc[who] = du;
            st.sc[2] = dw;
            st.sc[3] = dd_c;
        } else {
            uo[c] += du;
            st.d[c] += dd_c;
            st.w[c] += dw;
        }
    }
    if (c < 32)
        for (int q = lo + c; q < hi; q += 32) {
            const T r = R[q];
            if (r == T(0)) continue;
            const unsigned short e = dd[q];
            const int x = sd2_c1(e), y = sd2_c2(e);
            Mo[x * SD2_S + y] = r;
            Mo[y * SD2_S + x] = r;
        }
}

// The sweep state for the opponents' hands at rank positions [0, qend),
// computed directly (not by adding them one tie group at a time): the two
// matrices, P = M1 M2 as FP64 3x3 tiles over the 48-card box, the card sums,
// d = diag P, w = column sums + row sums of P, and the scalars, each summed
// in a fixed order.  The caller syncs before; this syncs after.
template <bool SP, class T>
__device__ __forceinline__ void sd2_direct_state(Sd2State st, T *M1, T *M2, const T *R1, const T *R2,
                                                 const unsigned short *dd, int qend) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (qend == 0) {
        // no hands: every aggregate is zero (the same for every thread of the
        // block, so the early return passes no barrier unevenly)
        for (int i = tid; i < SD2_S * SD2_S; i += kTermThreads) {
            M1[i] = T(0);
            M2[i] = T(0);
            st.P[i] = 0.0;
        }
        if (tid < 64) {
            st.u1[tid] = 0.0;
            st.u2[tid] = 0.0;
            st.w[tid] = 0.0;
            st.d[tid] = 0.0;
        }
        if (tid < 8) st.sc[tid] = 0.0;
        __syncthreads();
        return;
    }
    for (int i = tid; i < SD2_S * SD2_S; i += kTermThreads) {
        M1[i] = T(0);
        M2[i] = T(0);
    }
    if (SP && tid < SD2_N) st.row1[tid] = st.row2[tid] = 0ull;
    __syncthreads();
    for (int q = tid; q < qend; q += kTermThreads) {
        const unsigned short e = dd[q];
        const int x = sd2_c1(e), y = sd2_c2(e);
        const T r1 = R1[q], r2 = R2[q];
        if (r1 != T(0)) {
            M1[x * SD2_S + y] = r1;
            M1[y * SD2_S + x] = r1;
            if (SP) {
                atomicOr(&st.row1[x], 1ull << y);
                atomicOr(&st.row1[y], 1ull << x);
            }
        }
        if (r2 != T(0)) {
            M2[x * SD2_S + y] = r2;
            M2[y * SD2_S + x] = r2;
            if (SP) {
                atomicOr(&st.row2[x], 1ull << y);
                atomicOr(&st.row2[y], 1ull << x);
            }
        }
    }
    __syncthreads();
    {
        const int i0 = (tid >> 4) * 3, j0 = (tid & 15) * 3;
        double acc[3][3] = {};
        // sparse: without the k whose three cells of M1 or of M2 are 0 (their
        // terms are exact +0)
        unsigned long long m = 0ull;
        if (SP)
            m = (st.row1[i0] | st.row1[i0 + 1] | st.row1[i0 + 2]) & (st.row2[j0] | st.row2[j0 + 1] | st.row2[j0 + 2]);
        for (int k = 0; k < SD2_N; ++k) {
            if (SP) {
                if (!m) break;
                k = __ffsll(static_cast<long long>(m)) - 1;
                m &= m - 1;
            }
            double xs[3], ys[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                xs[i] = static_cast<double>(M1[(i0 + i) * SD2_S + k]);
                ys[i] = static_cast<double>(M2[k * SD2_S + j0 + i]);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) acc[i][j] += xs[i] * ys[j];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) st.P[(i0 + i) * SD2_S + j0 + j] = acc[i][j];
    }
    __syncthreads();
    if (tid < SD2_N) {
        const int c = tid;
        double u = 0.0;
#pragma unroll 12
        for (int r = 0; r < SD2_N; ++r) u += static_cast<double>(M1[r * SD2_S + c]);
        st.u1[c] = u;
        st.d[c] = st.P[c * SD2_S + c];
    } else if (tid >= 64 && tid < 64 + SD2_N) {
        const int c = tid - 64;
        double u = 0.0;
#pragma unroll 12
        for (int r = 0; r < SD2_N; ++r) u += static_cast<double>(M2[r * SD2_S + c]);
        st.u2[c] = u;
    } else if (tid >= 128 && tid < 128 + SD2_N) {
        const int c = tid - 128;
        double w = 0.0;   // (M2 u1)(c) = sum_r P[r][c]
#pragma unroll 12
        for (int r = 0; r < SD2_N; ++r) w += st.P[r * SD2_S + c];
        st.w[c] = w;
    }
    __syncthreads();
    if (tid < SD2_N) {
        const int c = tid;
        double w = 0.0;   // (M1 u2)(c) = sum_r P[c][r]
#pragma unroll 12
        for (int r = 0; r < SD2_N; ++r) w += st.P[c * SD2_S + r];
        st.w[c] += w;
    } else if (warp == kTermThreads / 32 - 1) {
        double f1 = 0.0, f2 = 0.0, q = 0.0, e = 0.0;
        for (int c = lane; c < SD2_N; c += 32) {
            f1 += st.u1[c];
            f2 += st.u2[c];
            q += st.u1[c] * st.u2[c];
            e += st.d[c];
        }
        f1 = warp_sum(f1);
        f2 = warp_sum(f2);
        q = warp_sum(q);
        e = warp_sum(e);
        if (lane == 0) {
            st.sc[0] = 0.5 * f1;
            st.sc[1] = 0.5 * f2;
            st.sc[2] = q;
            st.sc[3] = 0.5 * e;
        }
    }
    __syncthreads();
}

// For the traverser's hands at positions [lo, hi) (a tie group), on the state
// before the group: T1 = D(L, E) + D(E, L), summing over
// opponent 2's group hands (opponent 1's weaker hands avoiding four cards)
// and over opponent 1's (opponent 2's avoiding four cards); whether opponent 2
// holds any group hand.  Eight lanes per hand, each taking every eighth group
// position, combined in a fixed order.  Classes of position q at
// cls[4 (q - base)]: A = D(L, L), T1, opponent 2 present, C; A and C are
// sd2_phase_mass's.
template <bool SP, class T>
__device__ __forceinline__ void sd2_phase_a(Sd2State st, const T *M1, const T *M2, const T *R1, const T *R2,
                                            const unsigned short *dd, const short *pt, double *cls, int base,
                                            int lo, int hi) {
    const int l8 = threadIdx.x & 7, team = threadIdx.x >> 3;
    const int tbit = threadIdx.x & 24;   // the team's first lane in its warp
    for (int q0 = lo; q0 < hi; q0 += kTermThreads / 8) {
        const int q = q0 + team;
        const bool mine = q < hi && pt[q - base] >= 0;   // the same for all lanes of a team
        double t1 = 0.0;
        bool any2 = false;
        int a = 0, b = 0;
        if (mine) {
            const unsigned short e = dd[q];
            a = sd2_c1(e);
            b = sd2_c2(e);
            const double F1 = st.sc[0], F2 = st.sc[1];
            const double u1a = st.u1[a], u1b = st.u1[b], u2a = st.u2[a], u2b = st.u2[b];
            const double m1ab = static_cast<double>(M1[a * SD2_S + b]), m2ab = static_cast<double>(M2[a * SD2_S + b]);
            double dle = 0.0, del = 0.0;
            // this lane's group positions: lo + l8 and every eighth after it
            // (sparse: those of them where an opponent has reach, 32 at a time)
            const unsigned eighth = 0x01010101u << ((lo + l8) & 7);
            int base2 = lo & ~31, q2 = lo + l8 - 8;
            unsigned m = SP ? (st.on1[base2 >> 5] | st.on2[base2 >> 5]) & eighth & (~0u << (lo & 31)) : 0u;
            for (;;) {
                if (SP) {
                    while (!m && (base2 += 32) < hi) m = (st.on1[base2 >> 5] | st.on2[base2 >> 5]) & eighth;
                    if (!m) break;
                    q2 = base2 + __ffs(static_cast<int>(m)) - 1;
                    m &= m - 1;
                } else {
                    q2 += 8;
                }
                if (q2 >= hi) break;
                const T r1 = R1[q2], r2 = R2[q2];
                any2 = any2 || r2 != T(0);
                if (!SP && r1 == T(0) && r2 == T(0)) continue;
                const unsigned short e2 = dd[q2];
                const int x = sd2_c1(e2), y = sd2_c2(e2);
                if (x == a || x == b || y == a || y == b) continue;
                if (r2 != T(0))
                    dle += static_cast<double>(r2) *
                           (F1 - u1a - u1b - st.u1[x] - st.u1[y] + m1ab + static_cast<double>(M1[a * SD2_S + x]) +
                            static_cast<double>(M1[a * SD2_S + y]) + static_cast<double>(M1[b * SD2_S + x]) +
                            static_cast<double>(M1[b * SD2_S + y]) + static_cast<double>(M1[x * SD2_S + y]));
                if (r1 != T(0))
                    del += static_cast<double>(r1) *
                           (F2 - u2a - u2b - st.u2[x] - st.u2[y] + m2ab + static_cast<double>(M2[a * SD2_S + x]) +
                            static_cast<double>(M2[a * SD2_S + y]) + static_cast<double>(M2[b * SD2_S + x]) +
                            static_cast<double>(M2[b * SD2_S + y]) + static_cast<double>(M2[x * SD2_S + y]));
            }
            t1 = dle + del;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t1 += __shfl_xor_sync(0xffffffffu, t1, o);
        const unsigned bal = __ballot_sync(0xffffffffu, any2);
        if (mine && l8 == 0) {
            double *k4 = cls + 4 * (q - base);
            k4[1] = t1;
            k4[2] = ((bal >> tbit) & 0xffu) ? 1.0 : 0.0;
        }
    }
}

// mass on the current state for the traverser's hands at [lo, hi), into
// class slot k; thread `first` takes the first hand, so that a short group's
// masses fall to warps that its T1 leaves idle
template <class T>
__device__ __forceinline__ void sd2_phase_mass(Sd2State st, const T *M1, const T *M2, const unsigned short *dd,
                                               const short *pt, double *cls, int base, int lo, int hi, int k, int first) {
    for (int q = lo + ((threadIdx.x - first) & (kTermThreads - 1)); q < hi; q += kTermThreads)
        if (pt[q - base] >= 0) cls[4 * (q - base) + k] = sd2_mass(st, M1, M2, sd2_c1(dd[q]), sd2_c2(dd[q]));
}

// The sweep over a block's runs: segments [s0, s1), the first at `sg`, then the
// state of every hand.
// Groups are short and their phases wait on one another, so a block's time is
// its barriers and the serial walk over a group's hands, not arithmetic.  With
// few live hands (SP: at most SD2_SPARSE) most groups hold none of an opponent:
// such a group takes no phase and no barrier, walks touch live positions only,
// and the products skip terms that are exact zeros.  The order of what is
// summed is the same either way, so both give the same bits.  207 three-way
// showdowns of a 4-player river with 66 of 101 hands live: 300 -> 129 us.
template <bool SP, class T>
__device__ __forceinline__ void sd2_run(const Sd2State &st, T *M1, T *M2, const T *R1, const T *R2,
                                        const unsigned short *dd, const short *pt, double *cls,
                                        const int4 *__restrict__ seg4, int4 sg, int s0, int s1, int run_hi, int nc) {
    const int run_lo = sg.x;
    constexpr int kMassA = 5 * 32, kMassC = 7 * 32;   // first threads of the masses
    // the runs start from the state of every hand ranked below them
    sd2_direct_state<SP>(st, M1, M2, R1, R2, dd, run_lo);

    // segment entries come from global memory a step ahead of their use
    int4 nsg = s0 + 1 < s1 ? __ldg(seg4 + s0 + 1) : make_int4(0, 0, 0, 0);
    // reads: the state has been read since the last barrier, so the next hands
    // added wait for one
    bool reads = false;
    if (sg.z) {
        sd2_phase_a<SP>(st, M1, M2, R1, R2, dd, pt, cls, run_lo, sg.x, sg.y);
        sd2_phase_mass(st, M1, M2, dd, pt, cls, run_lo, sg.x, sg.y, 0, kMassA);
        reads = true;
    }
    for (int si = s0; si < s1; ++si) {
        const int lo = sg.x, hi = sg.y;
        const bool has = sg.z != 0, nhas = si + 1 < s1 && nsg.z != 0;
        const bool any1 = sd2_next<SP>(st.on1, lo, hi) < hi, any2 = sd2_next<SP>(st.on2, lo, hi) < hi;
        if ((any1 || any2) && reads) {
            __syncthreads();
            reads = false;
        }
        if (any1) {
            sd2_add<SP>(st, dd, R1, M1, M2, st.u1, st.u2, 0, lo, hi);
            __syncthreads();
        }
        if (any2) {
            sd2_add<SP>(st, dd, R2, M2, M1, st.u2, st.u1, 1, lo, hi);
            __syncthreads();
        }
        // C of this group and A of the next group: the same state
        if (has) sd2_phase_mass(st, M1, M2, dd, pt, cls, run_lo, lo, hi, 3, kMassC);
        if (nhas) {
            sd2_phase_mass(st, M1, M2, dd, pt, cls, run_lo, nsg.x, nsg.y, 0, kMassA);
            sd2_phase_a<SP>(st, M1, M2, R1, R2, dd, pt, cls, run_lo, nsg.x, nsg.y);
        }
        reads = reads || has || nhas;
        sg = nsg;   // the next segment's entry is loaded a full step before its use
        if (si + 2 < s1) nsg = __ldg(seg4 + si + 2);
    }
    if (reads) __syncthreads();
    // the whole state, unless these runs end the rank order and have it
    if (run_hi < nc) sd2_direct_state<SP>(st, M1, M2, R1, R2, dd, nc);
}

// One block per 2^lgm consecutive runs of a terminal's sweep (grid: items x
// kSd2Chunks / 2^lgm).  With bmap (batches), block b serves item bmap[b].x,
// run group bmap[b].y, with that item's own lgm (its subgame's solo choice).
template <class T>
__global__ void __launch_bounds__(kTermThreads, 4) k_term_sd2(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                              const TermItem *__restrict__ items, int trav, int lgm,
                                                              const int2 *__restrict__ bmap) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    int it_idx, grp;
    if (bmap) {
        const int2 m = bmap[blockIdx.x];
        it_idx = m.x;
        grp = m.y;
        lgm = items[it_idx].kind_detail;
    } else {
        const int per = kSd2Chunks >> lgm;
        it_idx = blockIdx.x / per;
        grp = blockIdx.x % per;
    }
    const TermItem I = items[it_idx];
    if (retired(ctxs, I.sg)) return;
    const int o1 = I.opp_player[0], o2 = I.opp_player[1];
    const T *reach;
    T *val;
    const int *pos_hand, *seg, *sd_pos;
    const SdCombo *cb;
    int HS, nc, Ht, s0, s1, span;
    {
        const DevCtx &c = ctxs ? ctxs[I.sg] : c0;   // read once into registers below
        reach = reach_rows<T>(c);
        val = val_rows<T>(c);
        pos_hand = c.pos_hand;
        seg = c.sd_seg;
        sd_pos = c.sd_pos;
        cb = c.sd_combo;
        HS = c.HS;
        nc = c.ncomb;
        span = c.sd_span[lgm];
        Ht = c.H[trav];
        const int *ch = c.sd_chunk + static_cast<size_t>(trav) * (kSd2Chunks + 1);
        s0 = ch[grp << lgm];
        s1 = ch[(grp + 1) << lgm];
    }
    // the launch provisioned shared memory for c0's rank table and run span
    // (the largest of a batch); a block needing more must not run
    if (HS > c0.HS || nc > c0.ncomb || span > c0.sd_span[lgm]) return;
    if (s0 >= s1) return;   // an unused run (the player has few tie groups)
    const int4 *seg4 = reinterpret_cast<const int4 *>(seg);   // {lo, hi, holds a traverser hand, 0}
    int4 sg = __ldg(seg4 + s0);
    const int run_lo = sg.x, run_hi = __ldg(seg + 4 * (s1 - 1) + 1);
    const int tid = threadIdx.x, lane = tid & 31;
    Carve cv{smem};
    Sd2State st;
    st.P = cv.take<double>(SD2_S * SD2_S);
    T *M1 = cv.take<T>(SD2_S * SD2_S);
    T *M2 = cv.take<T>(SD2_S * SD2_S);
    st.u1 = cv.take<double>(64);
    st.u2 = cv.take<double>(64);
    st.w = cv.take<double>(64);
    st.d = cv.take<double>(64);
    st.sc = cv.take<double>(8);
    st.row1 = cv.take<unsigned long long>(SD2_N);
    st.row2 = cv.take<unsigned long long>(SD2_N);
    st.on1 = cv.take<unsigned>(SD2_W);
    st.on2 = cv.take<unsigned>(SD2_W);
    double *cls = cv.take<double>(4 * span);   // per position of the run: A, T1, opponent 2 present, C
    char *rbuf = cv.take<char>(static_cast<int>(sd2_reach_bytes<T>(nc)));
    T *R1 = reinterpret_cast<T *>(rbuf);
    T *R2 = R1 + nc;
    unsigned short *dd = cv.take<unsigned short>(nc);
    short *pt = cv.take<short>(span);   // the traverser's hand at each position of the run, -1 if none
    int *last_pos = cv.take<int>(4);

    // opponents' reach and the cards by rank position, and the last position
    // holding positive reach of either opponent
    bool odd = false;   // a reach that is not finite: no term may be skipped
    if (tid == 0) *last_pos = -1;
    if (tid < 64) {
        st.u1[tid] = 0.0;
        st.u2[tid] = 0.0;
        st.w[tid] = 0.0;
        st.d[tid] = 0.0;
    }
    __syncthreads();
    {
        const T *ra = reach + static_cast<size_t>(I.opp_row[0]) * HS;
        const T *rb = reach + static_cast<size_t>(I.opp_row[1]) * HS;
        const int *pa = pos_hand + static_cast<size_t>(o1) * nc, *pb = pos_hand + static_cast<size_t>(o2) * nc;
        int lp = -1;
#pragma unroll 4
        for (int q0 = 0; q0 < nc; q0 += kTermThreads) {
            const int q = q0 + tid;
            const int ha = q < nc ? __ldg(pa + q) : -1, hb = q < nc ? __ldg(pb + q) : -1;
            const T x = ha >= 0 ? ra[ha] : T(0), y = hb >= 0 ? rb[hb] : T(0);
            odd = odd || !(x - x == T(0)) || !(y - y == T(0));
            const unsigned m1 = __ballot_sync(0xffffffffu, x != T(0)), m2 = __ballot_sync(0xffffffffu, y != T(0));
            if (q >= nc) continue;
            if (lane == 0) {
                st.on1[q >> 5] = m1;
                st.on2[q >> 5] = m2;
            }
            R1[q] = x;
            R2[q] = y;
            dd[q] = static_cast<unsigned short>(cb[q].d1 | (cb[q].d2 << 8));
            if (x > T(0) || y > T(0)) lp = q;
        }
        atomicMax(last_pos, lp);
        const int *ph_t = pos_hand + static_cast<size_t>(trav) * nc + run_lo;
        for (int k = tid; k < run_hi - run_lo; k += kTermThreads) pt[k] = static_cast<short>(__ldg(ph_t + k));
    }
    odd = __syncthreads_or(odd);
    int live = 0;
    for (int i = lane; i < (nc + 31) / 32; i += 32) live += max(__popc(st.on1[i]), __popc(st.on2[i]));
    const bool sparse = !odd && __reduce_add_sync(0xffffffffu, live) <= SD2_SPARSE;
    if (sparse)
        sd2_run<true>(st, M1, M2, R1, R2, dd, pt, cls, seg4, sg, s0, s1, run_hi, nc);
    else
        sd2_run<false>(st, M1, M2, R1, R2, dd, pt, cls, seg4, sg, s0, s1, run_hi, nc);

    // all hands added: Z, and the exact positive-pair count for hands whose
    // mass is within the error bound of zero (masks over the 47-card matrices,
    // in the reach space)
    ulonglong2 *Bm = reinterpret_cast<ulonglong2 *>(rbuf);
    Cr2Cnt *cnt = reinterpret_cast<Cr2Cnt *>(rbuf + 53 * sizeof(ulonglong2));
    Cr2Scalars *sc2 = reinterpret_cast<Cr2Scalars *>(rbuf + 53 * sizeof(ulonglong2) + 53 * sizeof(Cr2Cnt));
    if (tid < 2 * 64) {
        const int col = tid & 63;
        const T *M = tid < 64 ? M1 : M2;
        unsigned long long B = 0ull;
        if (col < SD2_S - 2)
            for (int r = 0; r < SD2_S - 2; ++r) B |= static_cast<unsigned long long>(M[r * SD2_S + col] > T(0)) << r;
        if (col <= kCr2Off) {
            if (tid < 64)
                Bm[col].x = B;
            else
                Bm[col].y = B;
        }
    }
    __syncthreads();
    if (tid <= kCr2Off) cnt[tid] = Cr2Cnt{__popcll(Bm[tid].x), __popcll(Bm[tid].y), 0, 0};
    __syncthreads();
    if (tid < 32) {
        int n1 = 0, n2 = 0, nq = 0, nd = 0;
        for (int k = lane; k <= kCr2Off; k += 32) {
            n1 += cnt[k].n1;
            n2 += cnt[k].n2;
            nq += cnt[k].n1 * cnt[k].n2;
            nd += __popcll(Bm[k].x & Bm[k].y);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n1 += __shfl_xor_sync(0xffffffffu, n1, o);
            n2 += __shfl_xor_sync(0xffffffffu, n2, o);
            nq += __shfl_xor_sync(0xffffffffu, nq, o);
            nd += __shfl_xor_sync(0xffffffffu, nd, o);
        }
        if (lane == 0) *sc2 = Cr2Scalars{0.0, 0.0, 0.0, n1 / 2, n2 / 2, nd / 2 - nq, 0};
    }
    __syncthreads();
    const Cr2Scalars S2 = *sc2;
    const double zmin = 1e-4 * st.sc[0] * st.sc[1];
    // payoff per class with the reference's float coefficients (pot / winners
    // - bet, or -bet): a coefficient that is exactly 0 drops its class exactly
    const double cw = static_cast<double>(I.pot - I.bet), c1 = static_cast<double>(I.pot / 2.0f - I.bet);
    const double c2 = static_cast<double>(I.pot / 3.0f - I.bet), cl = -static_cast<double>(I.bet);
    T *out = val + static_cast<size_t>(I.node) * HS;
    const int lastp = *last_pos;
    // the traverser's hands at this run's positions
    for (int q = run_lo + tid; q < run_hi; q += kTermThreads) {
        const int h = pt[q - run_lo];
        if (h < 0) continue;
        const unsigned short e = dd[q];
        const int a = sd2_c1(e), b = sd2_c2(e);
        const double Z = sd2_mass(st, M1, M2, a, b);
        const double *k4 = cls + 4 * (q - run_lo);
        const double A = k4[0], T1 = k4[1], C = k4[3];
        // no positive-reach opponent hand ranked above the group: the loss
        // class is empty, exactly (Z and C may come from different runs)
        const double L = __ldg(&cb[q].hi) > lastp ? 0.0 : Z - C;
        const double T2 = k4[2] != 0.0 ? (C - A) - T1 : 0.0;
        double v = cw * A + c1 * T1 + c2 * T2 + cl * L;
        if (fabs(Z) <= zmin && pair_count(Bm, cnt, a, b, S2.IF1, S2.IF2, S2.IQD) <= 0) v = 0.0;
        out[h] = static_cast<T>(v);
    }
    // the first block of the terminal also writes the hands without a rank
    // position (board-blocked) and the padding
    if (grp == 0) {
        const int *tp = sd_pos + static_cast<size_t>(trav) * HS;
        for (int h = tid; h < HS; h += kTermThreads)
            if (h >= Ht || __ldg(tp + h) < 0) out[h] = T(0);
    }
}

// Exact enumeration of opponent hand tuples, with the reference validity
// rules and payoffs (street_solve.cu:771-823 fold, :936-1002 showdown,
// :1079-1127 leaf).  One warp per (terminal, traverser hand): the tuple space
// (the opponents' hands in odometer order, the last opponent fastest) is cut
// into 32 contiguous runs, one per lane; each lane walks its run with an
// odometer and adds the positive products in FP64, and the lanes' sums are
// combined in a fixed order.  A block of 4 warps serves 4 hands; the blocks
// of a terminal stride over the subgame's hands.  Cost is the product of the
// opponents' range sizes; the planner only routes small cases here.
constexpr int kEnumWarps = 4;
template <class T>
__global__ void __launch_bounds__(32 * kEnumWarps) k_term_enum(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                               const TermItem *__restrict__ items, int nchunk,
                                                               int trav) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const int ch = blockIdx.x - it * nchunk;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TermItem I = items[it];
    if (retired(ctxs, I.sg)) return;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    T *out = val_rows<T>(c) + static_cast<size_t>(I.node) * c.HS;
    const T *reach = reach_rows<T>(c);
    const int Ht = c.H[trav], HSs = c.HS;
    const size_t HS = static_cast<size_t>(HSs);
    const int k = I.k;
    const bool sd = I.kind_detail == 2;
    int radix[SS_MAX_PLAYERS - 1] = {1, 1, 1, 1, 1};
    long long ntup = 1;
    for (int i = 0; i < k; ++i) {
        radix[i] = c.H[I.opp_player[i]];
        ntup *= radix[i];
    }
    const long long per = (ntup + 31) / 32;
    const double tb = static_cast<double>(static_cast<T>(I.bet));
    for (int hb = ch; hb * kEnumWarps < HSs; hb += nchunk) {
        const int h = hb * kEnumWarps + warp;
        if (h >= HSs) break;
        if (h >= Ht) {
            if (lane == 0) out[h] = T(0);
            continue;
        }
        const int hc = c.hand_code[trav * HS + h];
        const int t0 = hc & 0xff, t1 = (hc >> 8) & 0xff;
        unsigned hs = 0;
        if (sd) {
            hs = c.strength[trav * HS + h];
            if (hs == 0) {
                if (lane == 0) out[h] = T(0);
                continue;
            }
        }
        // this lane's run of tuples [q0, q1), its first tuple's digits (an
        // opponent without hands leaves no tuple at all)
        const long long q0 = lane * per, q1 = q0 + per < ntup ? q0 + per : ntup;
        int idx[SS_MAX_PLAYERS - 1] = {0, 0, 0, 0, 0};
        if (q0 < q1) {
            long long q = q0;
            for (int i = k - 1; i >= 0; --i) {
                idx[i] = static_cast<int>(q % radix[i]);
                q /= radix[i];
            }
        }
        double total = 0.0;
        for (long long q = q0; q < q1; ++q) {
            int cards[SS_MAX_PLAYERS - 1][2];
            unsigned os[SS_MAX_PLAYERS - 1];
            T prod = T(1);
            bool ok = true;
            for (int i = 0; i < k && ok; ++i) {
                const int p = I.opp_player[i], o = idx[i];
                const int code = c.hand_code[p * HS + o];
                const int a0 = code & 0xff, a1 = (code >> 8) & 0xff;
                cards[i][0] = a0;
                cards[i][1] = a1;
                if (t0 == a0 || t0 == a1 || t1 == a0 || t1 == a1) { ok = false; break; }
                if (sd) {
                    os[i] = c.strength[p * HS + o];
                    if (os[i] == 0) { ok = false; break; }
                } else if (code & 0x10000) {
                    ok = false;
                    break;
                }
                prod *= reach[static_cast<size_t>(I.opp_row[i]) * HS + o];
                for (int j = 0; j < i; ++j)
                    if (a0 == cards[j][0] || a0 == cards[j][1] || a1 == cards[j][0] || a1 == cards[j][1]) {
                        ok = false;
                        break;
                    }
            }
            if (ok && prod > T(0)) {
                if (!sd) {
                    total += static_cast<double>(prod);
                } else {
                    unsigned best = hs;
                    for (int i = 0; i < k; ++i) best = os[i] > best ? os[i] : best;
                    if (hs < best) {
                        total += static_cast<double>(prod) * (-tb);
                    } else {
                        int wins = 1;
                        for (int i = 0; i < k; ++i) wins += os[i] == best ? 1 : 0;
                        // the reference's float payoff pot / winners - bet
                        const double pay = static_cast<double>(static_cast<T>(I.pot) / static_cast<T>(wins) -
                                                               static_cast<T>(I.bet));
                        total += static_cast<double>(prod) * pay;
                    }
                }
            }
            for (int j = k - 1; j >= 0; --j) {
                if (++idx[j] < radix[j]) break;
                idx[j] = 0;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0)
            out[h] = sd ? static_cast<T>(total) : static_cast<T>(static_cast<double>(term_factor(c, I, h)) * total);
    }
}

// Folds and leaves with three counted opponents (4+ player subgames): the
// card-removal mass by contraction (ss_triple.cuh), in FP64: O(deck) per
// traverser hand over tables of O(deck^2), where conditioning on the third
// opponent's hand took O(hands) two-opponent evaluations.  One block per
// (group of terminals on the same reach rows, share of the hands); its first
// item's blocks write every member's row, each with its own factor.  Bound by
// the FP64 pipe and shared memory: per hand and card 34 FP64 operations and
// 23 shared-memory wavefronts per warp, beside two 48 x 48 products per block.
// A hand whose mass is small beside the product of the three sums is summed
// again by conditioning, to keep its digits, and 0 when it has no tuple (the
// reference adds only positive products).
//
// 384 threads take the 1128 hands of a turn in three rounds of 98 %, and the
// tables of a 48-card deck (105 KB) leave two blocks per SM (512 and 576
// threads spill: 1.4x slower).  Measured on the 4-player turn (5,681 nodes,
// 2,696 terminals), a mean launch of 60 iterations by conditioning on every
// third hand and now: 8.35 and 0.69 ms at full ranges, 390 and 224 us at 200
// hands, 158 and 133 us at 60, 118 and 104 us at 24, where the tables are the
// work (165 and 133 us at 60 and 24 while every pair of cards was looked up).
constexpr int kCr3Threads = 384;
static_assert(kMaxHS <= 14 * (kCr3Threads / 4), "a thread's rounds fit a mask");
// blocks a launch is brought to by sharing a group's hands between blocks (each
// builds the tables): two per SM
constexpr int kCr3Blocks = 2 * 148;
constexpr size_t cr3_smem(int deck) {
    return static_cast<size_t>(tri::doubles(deck)) * sizeof(double) + 2 * tri::kVS * sizeof(unsigned long long) +
           4 * tri::kVS * sizeof(int) + 4 * sizeof(long long) + 8 * 16;
}

template <class T>
__global__ void __launch_bounds__(kCr3Threads, 2) k_term_cr3(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                            const TermItem *__restrict__ items, int nchunk,
                                                            int trav) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    const int it = blockIdx.x / nchunk;
    const int ch = blockIdx.x - it * nchunk;
    const TermItem *I0 = items + it;
    if (I0->follow) return;   // written by the blocks of its group's first item
    if (retired(ctxs, I0->sg)) return;
    const int ng = I0->gextra + 1;
    const DevCtx &c = ctxs ? ctxs[I0->sg] : c0;
    const int HS = c.HS, Ht = c.H[trav], n = c.deck;
    // shared memory was provisioned for c0's deck (the largest of a batch)
    if (HS > kMaxHS || n > c0.deck || (ch > 0 && ch * kCr3Threads >= HS)) return;
    const int tid = threadIdx.x;
    Carve cv{smem};
    const tri::Tables t = tri::tables(cv.take<double>(tri::doubles(n)), n);
    tri::Counts k;
    k.mA = cv.take<unsigned long long>(tri::kVS);
    k.mB = cv.take<unsigned long long>(tri::kVS);
    k.nA = cv.take<int>(tri::kVS);
    k.nB = cv.take<int>(tri::kVS);
    k.nW = cv.take<int>(tri::kVS);
    k.nD = cv.take<int>(tri::kVS);
    k.s = cv.take<long long>(4);
    const int o1 = I0->opp_player[0], o2 = I0->opp_player[1], o3 = I0->opp_player[2];
    const T *reach = reach_rows<T>(c);
    const size_t hs = static_cast<size_t>(HS);
    const T *r1 = reach + static_cast<size_t>(I0->opp_row[0]) * hs;
    const T *r2 = reach + static_cast<size_t>(I0->opp_row[1]) * hs;
    const T *r3 = reach + static_cast<size_t>(I0->opp_row[2]) * hs;
    const int *code3 = c.hand_code + static_cast<size_t>(o3) * hs;
    const int H3 = c.H[o3];
    const bool dup3 = c.dup[o3] != 0;
    tri::phase_clear(tid, kCr3Threads, t);
    __syncthreads();
    {
        const T *const r[3] = {r1, r2, r3};
        const int *const code[3] = {c.hand_code + static_cast<size_t>(o1) * hs, c.hand_code + static_cast<size_t>(o2) * hs, code3};
        const int H[3] = {c.H[o1], c.H[o2], H3};
        tri::phase_scatter(tid, kCr3Threads, t, r, code, H, !dup3);
    }
    __syncthreads();
    if (dup3) {
        tri::phase_gather_third(tid, kCr3Threads, t, r3, code3, H3);
        __syncthreads();
    }
    tri::phase_products(tid, kCr3Threads, t);
    __syncthreads();
    tri::phase_vectors(tid, kCr3Threads, t);
    __syncthreads();
    tri::phase_scalars(tid, kCr3Threads, t);
    __syncthreads();
    // an opponent without positive reach: every mass is 0
    const bool none = t.sc[tri::FA] == 0.0 || t.sc[tri::FB] == 0.0 || t.sc[tri::FC] == 0.0;
    const double zb = tri::zero_bound(t);
    const int *code_t = c.hand_code + static_cast<size_t>(trav) * hs;
    auto dense = [&](int hc, int shift) {
        const int d = (hc >> shift) & 63;
        return d < n ? d : n;
    };
    T *val = val_rows<T>(c);
    auto write = [&](int h, double m) {
        for (int g = 0; g < ng; ++g) {
            const TermItem &Ig = I0[g];
            val[static_cast<size_t>(Ig.node) * hs + h] =
                h < Ht ? static_cast<T>(static_cast<double>(term_factor(c, Ig, h)) * m) : T(0);
        }
    };
    // lanes per hand: a range too small for the block's threads splits each
    // hand's sum over the deck
    const int lanes = Ht * 4 <= kCr3Threads ? 4 : Ht * 2 <= kCr3Threads ? 2 : 1;
    const int per = kCr3Threads / lanes, mine = tid / lanes, part = tid % lanes;   // hands per round
    const int first = ch * per, step = nchunk * per;
    unsigned near = 0;   // this thread's hands (by round) to sum again
    int round = 0;
#pragma unroll 1
    for (int h0 = first; h0 < HS; h0 += step, ++round) {
        const int h = h0 + mine;
        const bool live = h < Ht && !none;
        const int hc = live ? __ldg(code_t + h) : 0, a = dense(hc, 20), b = dense(hc, 26);
        tri::Part p{0.0, 0.0, 0.0};
        if (live) p = tri::hand_part(a, b, t, part, lanes);
        for (int k = 1; k < lanes; k <<= 1) {
            p.acc += __shfl_xor_sync(0xffffffffu, p.acc, k);
            p.ACab += __shfl_xor_sync(0xffffffffu, p.ACab, k);
            p.ACba += __shfl_xor_sync(0xffffffffu, p.ACba, k);
        }
        if (part != 0 || h >= HS) continue;
        const double m = live ? tri::hand_finish(a, b, t, p) : 0.0;
        if (live && fabs(m) <= zb) near |= 1u << round;
        write(h, m);
    }
    if (!__syncthreads_or(near != 0)) return;
    // a warp per hand to sum again, 32 third-opponent hands at a time;
    // the list of those hands takes C's space
    int *n_near = reinterpret_cast<int *>(t.C);
    unsigned short *list = reinterpret_cast<unsigned short *>(n_near + 4);
    static_assert(kMaxHS * 2 + 16 <= 47 * 47 * 8, "the list fits C's space");
    if (tid == 0) *n_near = 0;
    tri::phase_masks(tid, kCr3Threads, t, k);
    __syncthreads();
    for (int r = 0; near >> r; ++r)
        if (near >> r & 1u) list[atomicAdd(n_near, 1)] = static_cast<unsigned short>(first + r * step + mine);
    tri::phase_counts(tid, kCr3Threads, t, k);
    __syncthreads();
    const int lane = tid & 31;
    for (int i = tid >> 5; i < *n_near; i += kCr3Threads / 32) {
        const int h = list[i], hc = __ldg(code_t + h), a = dense(hc, 20), b = dense(hc, 26);
        double m = 0.0;
        for (int j = lane; j < H3; j += 32) m += tri::tuple_mass(a, b, t, k, r3[j], __ldg(code3 + j));
        m = warp_sum(m);
        if (lane == 0) write(h, m);
    }
}

// Four-way showdowns (three live opponents): the traverser's class masses
// (ss_cr3.cuh) in FP64.  One block per (terminal, 256 rank positions).  The
// block builds the tables of the first two opponents' full matrices once
// (every tuple's mass, for the loss class and the exact zero), then walks the
// tie groups that hold one of its traverser hands with the tables of the
// weaker parts, and adds the third opponent's hands by class.  A class mass
// within rounding of 0 takes its exact tuple count (0: exactly 0).
//
// A block is a chain of short phases between barriers, so what bounds it is
// their latency: loads that wait on loads, and warps with nothing to do.  So
// the block's rank positions (hands, reach, cards, groups) are read once into
// shared memory, the table gathers have all their loads in flight together,
// and a warp takes one (hand, pair of classes) at a time, of the hands that
// are there and not of the positions, all pairs that read the same tables in
// one round.  Blocks come chunk by chunk: the last chunk, the shortest, runs
// last.  Measured per launch, 4-player rivers: 73 terminals with 66 of 101
// hands live 410 -> 143 us, 13 with 390 of 600 live 1.9 -> 1.2 ms, 9 at full
// ranges 4.1 -> 3.4 ms; before, one thread listed the third opponent's hands
// and warps took one pair of classes at a time, position by position.
constexpr int kSd3Positions = 1081;   // C(47, 2): rank positions on every river board
constexpr int kSd3Warps = kTermThreads / 32;
// a tie group whose tying parts hold at most this many positive-reach hands
// of each of the first two opponents takes the sparse steps (grown weaker
// parts, tying pairs evaluated directly); a longer one rebuilds tables
constexpr int kSd3MaxE = 64;
// a table build in units of one D2 evaluation (the sparse steps' cost model)
constexpr double kSd3BuildCost = 3000.0;
template <class T>
constexpr size_t sd3_smem(int HS) {
    return (4 * cr3::kS * cr3::kS + 4 * cr3::kS + 8) * sizeof(double) + 4 * cr3::kS * sizeof(int) +
           2 * cr3::kS * sizeof(unsigned long long) + 8 * sizeof(long long) +
           static_cast<size_t>(HS) * (sizeof(double) + 2 * sizeof(short)) +
           kTermThreads * (2 * sizeof(T) + 3 * sizeof(short) + 3) +
           4 * kSd3Warps * (sizeof(double) + sizeof(long long)) + 2 * kSd3MaxE * sizeof(cr3::EHand) +
           (4 * kSd3Warps + 4) * sizeof(int) + 4 * 16;
}
static_assert(2 * kSd3MaxE * sizeof(cr3::EHand) == kTermThreads * sizeof(double), "the masses share the lists' space");
static_assert(sd3_smem<float>(kMaxHS) <= (228 * 1024 - 2 * 1024) / 2, "two blocks per SM");

template <class T>
__global__ void __launch_bounds__(kTermThreads, 2) k_term_sd3(DevCtx c0, const DevCtx *__restrict__ ctxs,
                                                             const TermItem *__restrict__ items, int nchunk,
                                                             int trav) {
    wait_prior_grid();
    extern __shared__ __align__(16) char smem[];
    const int n_items = gridDim.x / nchunk;
    const int ch = blockIdx.x / n_items;
    const int it = blockIdx.x - ch * n_items;
    const TermItem I = items[it];
    if (retired(ctxs, I.sg)) return;
    const DevCtx &c = ctxs ? ctxs[I.sg] : c0;
    const int HS = c.HS;
    if (HS > c0.HS || c.deck > cr3::kS - 1) return;
    const size_t hs = static_cast<size_t>(HS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T *out = val_rows<T>(c) + static_cast<size_t>(I.node) * hs;
    const int *tpos = c.sd_pos + static_cast<size_t>(trav) * hs;
    // the first chunk writes the hands without a rank position and the padding
    if (ch == 0)
        for (int h = tid; h < HS; h += kTermThreads)
            if (h >= c.H[trav] || tpos[h] < 0) out[h] = T(0);
    const int nc = c.ncomb;
    const int q0 = ch * kTermThreads;
    if (q0 >= nc) return;
    const int qend = min(q0 + kTermThreads, nc);
    Carve cv{smem};
    cr3::Tables t;
    t.A = cv.take<double>(cr3::kS * cr3::kS);
    t.B = cv.take<double>(cr3::kS * cr3::kS);
    t.P = cv.take<double>(cr3::kS * cr3::kS);
    t.PT = cv.take<double>(cr3::kS * cr3::kS);
    t.uA = cv.take<double>(cr3::kS);
    t.uB = cv.take<double>(cr3::kS);
    t.w = cv.take<double>(cr3::kS);
    t.d = cv.take<double>(cr3::kS);
    t.sc = cv.take<double>(8);
    t.iuA = cv.take<int>(cr3::kS);
    t.iuB = cv.take<int>(cr3::kS);
    t.iw = cv.take<int>(cr3::kS);
    t.id = cv.take<int>(cr3::kS);
    t.mA = cv.take<unsigned long long>(cr3::kS);
    t.mB = cv.take<unsigned long long>(cr3::kS);
    t.isc = cv.take<long long>(8);
    // per warp: the two class partials of one (hand, slice); two sets, so that
    // a round's sums are read while the next round writes
    double *part = cv.take<double>(4 * kSd3Warps);
    long long *partc = cv.take<long long>(4 * kSd3Warps);
    // the block's rank positions: the first two opponents' reach (0: no hand)
    // and dense cards, the tie group's end; the traverser's dense cards
    T *pr1 = cv.take<T>(kTermThreads);
    T *pr2 = cv.take<T>(kTermThreads);
    unsigned short *pxy1 = cv.take<unsigned short>(kTermThreads);
    unsigned short *pxy2 = cv.take<unsigned short>(kTermThreads);
    short *phi = cv.take<short>(kTermThreads);
    unsigned char *ga = cv.take<unsigned char>(kTermThreads);
    unsigned char *gb = cv.take<unsigned char>(kTermThreads);
    // the positions that hold a traverser hand: in order, as a mask, and how
    // many before each of its words
    unsigned char *gl = cv.take<unsigned char>(kTermThreads);
    unsigned *hm = cv.take<unsigned>(kSd3Warps + 1);
    int *hp = cv.take<int>(kSd3Warps + 1);
    int *wc = cv.take<int>(kSd3Warps);
    // the current tie group's tying hands of the first two opponents, and their numbers
    cr3::EHand *elist1 = cv.take<cr3::EHand>(kSd3MaxE);
    cr3::EHand *elist2 = cv.take<cr3::EHand>(kSd3MaxE);
    double *tot = reinterpret_cast<double *>(elist1);   // (before the groups) every tuple's mass, by position
    int *en = cv.take<int>(2);
    t.r3 = cv.take<double>(HS);   // (the third opponent's range may hold a combo twice)
    t.xy = cv.take<unsigned short>(HS);
    short *p3 = cv.take<short>(HS);
    const T *reach = reach_rows<T>(c);
    const int o1 = I.opp_player[0], o2 = I.opp_player[1], o3 = I.opp_player[2];
    cr3::Opp3<T> in;
    in.r1 = reach + static_cast<size_t>(I.opp_row[0]) * hs;
    in.r2 = reach + static_cast<size_t>(I.opp_row[1]) * hs;
    in.r3 = reach + static_cast<size_t>(I.opp_row[2]) * hs;
    in.pair1 = c.pair_idx + static_cast<size_t>(o1) * 52 * 52;
    in.pair2 = c.pair_idx + static_cast<size_t>(o2) * 52 * 52;
    in.code3 = c.hand_code + static_cast<size_t>(o3) * hs;
    in.H3 = c.H[o3];
    in.HS = HS;
    in.deck = c.deck;
    const int *code1 = c.hand_code + static_cast<size_t>(o1) * hs, *code2 = c.hand_code + static_cast<size_t>(o2) * hs;
    const int *ph1 = c.pos_hand + static_cast<size_t>(o1) * nc, *ph2 = c.pos_hand + static_cast<size_t>(o2) * nc;
    const int *posA = c.sd_pos + static_cast<size_t>(o1) * hs;
    const int *posB = c.sd_pos + static_cast<size_t>(o2) * hs;
    const int *pre1 = c.pos_prefix + static_cast<size_t>(o1) * (nc + 1);
    const int *pre2 = c.pos_prefix + static_cast<size_t>(o2) * (nc + 1);
    // this thread's rank position: the traverser's hand there, the first two
    // opponents' hands, the tie group
    cr3::Sd3Thread st;
    cr3::sd3_thread_init(q0 + tid, qend, c.pos_hand + static_cast<size_t>(trav) * nc,
                         c.hand_code + static_cast<size_t>(trav) * hs, c.sd_combo, st);
    {
        const int q = q0 + tid;
        const int h1 = q < qend ? ph1[q] : -1, h2 = q < qend ? ph2[q] : -1;
        pr1[tid] = h1 >= 0 ? in.r1[h1] : T(0);
        pr2[tid] = h2 >= 0 ? in.r2[h2] : T(0);
        const int e1 = h1 >= 0 ? code1[h1] : 0, e2 = h2 >= 0 ? code2[h2] : 0;
        pxy1[tid] = static_cast<unsigned short>(((e1 >> 20) & 63) | (((e1 >> 26) & 63) << 8));
        pxy2[tid] = static_cast<unsigned short>(((e2 >> 20) & 63) | (((e2 >> 26) & 63) << 8));
        phi[tid] = q < qend ? static_cast<short>(c.sd_combo[q].hi) : 0;
        ga[tid] = static_cast<unsigned char>(st.a);
        gb[tid] = static_cast<unsigned char>(st.b);
        const unsigned m = __ballot_sync(0xffffffffu, st.h >= 0);
        if (lane == 0) hm[warp] = m;
        if (tid == 0) hm[kSd3Warps] = 0u;
    }
    __syncthreads();
    if (tid <= kSd3Warps) {
        int n = 0;
        for (int w = 0; w < tid; ++w) n += __popc(hm[w]);
        hp[tid] = n;
    }
    __syncthreads();
    const int nhand = hp[kSd3Warps];
    if (nhand == 0) return;   // no row of this block's positions to write
    // how many traverser hands the block has below its position j
    auto rank_at = [&](int j) { return hp[j >> 5] + __popc(hm[j >> 5] & ((1u << (j & 31)) - 1u)); };
    const int myrank = rank_at(tid);
    if (st.h >= 0) gl[myrank] = static_cast<unsigned char>(tid);
    // the third opponent's positive-reach live hands in hand order
    int n3 = 0;
    for (int base = 0; base < in.H3; base += kTermThreads) {
        const int h = base + tid;
        int code = 0x10000, p = -1;
        T r = T(0);
        if (h < in.H3) {
            code = in.code3[h];
            p = c.sd_pos[static_cast<size_t>(o3) * hs + h];
            r = in.r3[h];
        }
        const bool ok = !(code & 0x10000) && p >= 0 && r > T(0);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) wc[warp] = __popc(m);
        __syncthreads();
        int at = n3 + __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < kSd3Warps; ++w) {
            if (w < warp) at += wc[w];
            n3 += wc[w];
        }
        if (ok) {
            t.r3[at] = static_cast<double>(r);
            t.xy[at] = static_cast<unsigned short>(((code >> 20) & 63) | (((code >> 26) & 63) << 8));
            p3[at] = static_cast<short>(p);
        }
        __syncthreads();
    }
    if (tid == 0) t.isc[4] = n3;
    constexpr int kAll = 1 << 30;
    auto build = [&](int lo1, int hi1, int lo2, int hi2, bool first) {
        cr3::gather_dev(tid, in, t, posA, lo1, hi1, posB, lo2, hi2);
        __syncthreads();
        if (first && tid == kTermThreads - 1) {   // (this warp has no part of the product)
            double f3 = 0.0;
#pragma unroll 8
            for (int k = 0; k < n3; ++k) f3 += t.r3[k];
            t.sc[4] = f3;
        }
        cr3::build_step1(tid, t);
        __syncthreads();
        cr3::build_step2(tid, t);
        __syncthreads();
    };
    build(0, kAll, 0, kAll, true);
    // Every tuple's mass per traverser hand, the third opponent's hands added
    // in their order: `lanes` threads per hand evaluate as many of its terms,
    // then each adds all of them in turn.
    {
        const double zb = cr3::zero_bound(t);
        int lanes = 32;
        while (lanes > 1 && lanes * nhand > kTermThreads) lanes >>= 1;
        const int hc = tid / lanes, l = tid - hc * lanes;
        const bool on = hc < nhand;
        const int j = on ? gl[hc] : 0, a = ga[j], b = gb[j];
        const cr3::HandPart part_ab = cr3::hand_part(a, b, t);
        double sum = 0.0;
        for (int k0 = 0; k0 < n3; k0 += lanes) {
            const int k = k0 + l;
            double v = 0.0;
            if (on && k < n3) {
                const int x = t.xy[k] & 0xff, y = t.xy[k] >> 8;
                if (x != a && x != b && y != a && y != b) v = cr3::d2_at(part_ab, a, b, x, y, t);
            }
            if (lanes == 1) {
                sum = fma(t.r3[k0], v, sum);
            } else {
                for (int i = 0; i < lanes; ++i) {
                    const double vi = __shfl_sync(0xffffffffu, v, i, lanes);
                    if (k0 + i < n3) sum = fma(t.r3[k0 + i], vi, sum);
                }
            }
        }
        const bool near = on && fabs(sum) <= zb;
        if (__any_sync(0xffffffffu, near)) {
            long long n = 0;
            if (near) {
                const cr3::HandCount cab = cr3::hand_count_part(a, b, t);
                for (int k = l; k < n3; k += lanes) {
                    const int x = t.xy[k] & 0xff, y = t.xy[k] >> 8;
                    if (x != a && x != b && y != a && y != b) n += cr3::c2_at(cab, a, b, x, y, t);
                }
            }
            for (int o = lanes >> 1; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
            if (near && n == 0) sum = 0.0;
        }
        if (on && l == 0) tot[j] = sum;
    }
    __syncthreads();
    st.total = tot[tid];   // written, and used, where st.h >= 0
    // The tie groups meeting [q0, qend), the same walk in every thread.  A
    // class mass of a (hand, pair of the first two opponents' parts) is a sum
    // over the third opponent's list: slices of that list over `per` warps,
    // lanes splitting a slice, and the hand's owner thread combines its warps'
    // partials in warp order.
    // the weaker parts' tables (positions [0, t_hi) of the first two
    // opponents), grown group by group while the groups' tying parts are short
    bool t_valid = false;
    int t_hi = 0;
    int buf = 0;
    int glo = c.sd_combo[q0].lo;   // the first group may begin below the block's positions
    for (int g = q0; g < qend;) {
        const int lo = glo, hi = phi[g - q0];
        glo = hi;
        const int j0 = max(lo, q0) - q0, ng = min(hi, qend) - q0 - j0;
        const int k0 = rank_at(j0), nmine = rank_at(j0 + ng) - k0;   // the block's traverser hands in the group
        if (k0 == nhand) break;   // none here or above
        if (nmine == 0 && !t_valid) {
            g = hi;
            continue;
        }
        const int mine_at = st.h >= 0 && st.glo == lo ? myrank - k0 : -1;   // this thread's hand among them
        const bool any = nmine > 0;
        __syncthreads();
        // the group's tying hands of the first two opponents with positive
        // reach, in rank order (warp 0: first opponent, warp 1: second)
        if (warp < 2) {
            const int *ph = warp == 0 ? ph1 : ph2;
            const T *rr = warp == 0 ? in.r1 : in.r2;
            const int *code = warp == 0 ? code1 : code2;
            const T *pr = warp == 0 ? pr1 : pr2;
            const unsigned short *pxy = warp == 0 ? pxy1 : pxy2;
            cr3::EHand *E = warp == 0 ? elist1 : elist2;
            int n = 0;
            for (int base = lo; base < hi; base += 32) {
                const int q = base + lane;
                T rv = T(0);
                int x = 0, y = 0;
                if (q >= q0 && q < qend) {
                    rv = q < hi ? pr[q - q0] : T(0);
                    x = pxy[q - q0] & 0xff;
                    y = pxy[q - q0] >> 8;
                } else {   // a group reaching past the block's positions
                    const int hh = q < hi ? ph[q] : -1;
                    if (hh >= 0) {
                        rv = rr[hh];
                        const int hc = code[hh];
                        x = (hc >> 20) & 63;
                        y = (hc >> 26) & 63;
                    }
                }
                const bool ok = rv > T(0);
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                const int at = n + __popc(bal & ((1u << lane) - 1u));
                if (ok && at < kSd3MaxE) E[at] = cr3::EHand{static_cast<double>(rv), x, y};
                n += __popc(bal);
            }
            if (lane == 0) en[warp] = n;
        }
        __syncthreads();
        const int n1 = en[0], n2 = en[1];
        const bool small = n1 <= kSd3MaxE && n2 <= kSd3MaxE;
        if (any) {
            // LL from the weaker parts' tables (grown along the walk, or built
            // here); a pair with a tying part is evaluated directly from them
            // when that costs less than building its own tables (direct: a
            // six-card one-opponent mass per tying hand and third-opponent
            // hand; built: a table build shared by the group's hands, then one
            // D2 per third-opponent hand) -- sparse ranges go direct, full
            // ranges build; the direct pairs run first, while the tables
            // still hold the weaker parts
            if (!(t_valid && t_hi == lo)) {
                build(0, lo, 0, lo, false);
                t_valid = true;
                t_hi = lo;
            }
            const double work = static_cast<double>(nmine) * static_cast<double>(n3);
            auto go_direct = [&](int pr) {
                if (!small) return false;
                const double terms = pr == 1 ? n1 : pr == 2 ? n2 : 0.125 * n1 * n2;
                return work * (0.8 * terms) <= kSd3BuildCost + work;
            };
            // an opponent without a hand in its part of a pair: no tuple, both
            // class masses exactly 0 (what the tables and the exact count
            // would give), nothing to do
            const int w1 = pre1[lo] - pre1[0], e1 = pre1[hi] - pre1[lo];
            const int w2 = pre2[lo] - pre2[0], e2 = pre2[hi] - pre2[lo];
            // pairs to take from the weaker parts' tables, and to build (two
            // bits each, in order)
            unsigned now = 0u, later = 0u;
            int n_now = 0, n_later = 0;
            for (int pr = 0; pr < 4; ++pr) {
                if (((pr & 1) ? e1 : w1) == 0 || ((pr & 2) ? e2 : w2) == 0) continue;
                if (pr == 0 || go_direct(pr))
                    now |= static_cast<unsigned>(pr) << (2 * n_now++);
                else
                    later |= static_cast<unsigned>(pr) << (2 * n_later++);
            }
            const int per = ng >= kSd3Warps ? 1 : kSd3Warps / ng;   // warps per (hand, pair)
            const int ipr = kSd3Warps / per;                          // (hand, pair) items per round
            const int r = warp / per, sl = warp - r * per;
            // the class masses of n_pairs pairs: LL and built pairs (`built`)
            // from the tables, tying pairs directly
            auto walk = [&](unsigned pairs, int n_pairs, bool built) {
                const int n_work = n_pairs * nmine;
                const double zb = cr3::zero_bound(t);
                bool near = false;
                int near_pr = 0;
                for (int base = 0; base < n_work; base += ipr) {
                    const int item = base + r;
                    double o[2] = {0.0, 0.0};
                    long long n[2] = {0, 0};
                    if (r < ipr && item < n_work) {
                        const int pi = item / nmine, j = gl[k0 + item - pi * nmine];
                        const int pr = static_cast<int>(pairs >> (2 * pi)) & 3;
                        const int a = ga[j], b = gb[j];
                        const bool direct = pr > 0 && !built;
                        if (direct)
                            cr3::e_pair_slice(pr, a, b, t, elist1, n1, elist2, n2, p3, lo, hi, sl * 32 + lane,
                                              per * 32, o, n);
                        else
                            cr3::hand_mass_cls_slice(a, b, t, p3, lo, hi, sl * 32 + lane, per * 32, o, n, false);
                        for (int off = 16; off > 0; off >>= 1) {
                            o[0] += __shfl_xor_sync(0xffffffffu, o[0], off);
                            o[1] += __shfl_xor_sync(0xffffffffu, o[1], off);
                        }
                        // one warp holds all of a hand's sum: the exact count at once
                        const bool near0 = !direct && per == 1 && fabs(o[0]) <= zb;
                        const bool near1 = !direct && per == 1 && fabs(o[1]) <= zb;
                        if (near0 || near1) {
                            double none[2];
                            cr3::hand_mass_cls_slice(a, b, t, p3, lo, hi, lane, 32, none, n, true);
                        }
                        if (direct || near0 || near1)
                            for (int off = 16; off > 0; off >>= 1) {
                                n[0] += __shfl_xor_sync(0xffffffffu, n[0], off);
                                n[1] += __shfl_xor_sync(0xffffffffu, n[1], off);
                            }
                        if (near0 && n[0] == 0) o[0] = 0.0;
                        if (near1 && n[1] == 0) o[1] = 0.0;
                    }
                    double *ps = part + buf * 2 * kSd3Warps;
                    long long *cs = partc + buf * 2 * kSd3Warps;
                    if (lane == 0) {
                        ps[2 * warp] = o[0];
                        ps[2 * warp + 1] = o[1];
                        cs[2 * warp] = n[0];
                        cs[2 * warp + 1] = n[1];
                    }
                    __syncthreads();
                    if (mine_at >= 0)
                        for (int pi = 0; pi < n_pairs; ++pi) {
                            const int at = pi * nmine + mine_at - base;
                            if (at < 0 || at >= ipr) continue;
                            const int pr = static_cast<int>(pairs >> (2 * pi)) & 3;
                            double m0 = 0.0, m1 = 0.0;
                            long long c0 = 0, c1 = 0;
                            for (int k = 0; k < per; ++k) {
                                m0 += ps[2 * (at * per + k)];
                                m1 += ps[2 * (at * per + k) + 1];
                                c0 += cs[2 * (at * per + k)];
                                c1 += cs[2 * (at * per + k) + 1];
                            }
                            if (pr > 0 && !built) {
                                if (c0 == 0) m0 = 0.0;
                                if (c1 == 0) m1 = 0.0;
                            } else if (per > 1 && (fabs(m0) <= zb || fabs(m1) <= zb)) {
                                near = true;
                                near_pr = pr;
                            }
#pragma unroll
                            for (int p = 0; p < 4; ++p)
                                if (p == pr) {
                                    st.m[p][0] = m0;
                                    st.m[p][1] = m1;
                                }
                        }
                    buf ^= 1;
                }
                // a sum split over warps: the exact counts in a second pass
                // (at most one of the pairs is from the tables: the first)
                if (per > 1 && __syncthreads_or(near)) {
                    for (int base = 0; base < nmine; base += ipr) {
                        long long n[2] = {0, 0};
                        if (r < ipr && base + r < nmine) {
                            const int j = gl[k0 + base + r];
                            double none[2];
                            cr3::hand_mass_cls_slice(ga[j], gb[j], t, p3, lo, hi, sl * 32 + lane, per * 32, none, n,
                                                     true);
                            for (int off = 16; off > 0; off >>= 1) {
                                n[0] += __shfl_xor_sync(0xffffffffu, n[0], off);
                                n[1] += __shfl_xor_sync(0xffffffffu, n[1], off);
                            }
                        }
                        long long *cs = partc + buf * 2 * kSd3Warps;
                        if (lane == 0) {
                            cs[2 * warp] = n[0];
                            cs[2 * warp + 1] = n[1];
                        }
                        __syncthreads();
                        const int at = mine_at - base;
                        if (near && at >= 0 && at < ipr) {
                            long long c0 = 0, c1 = 0;
                            for (int k = 0; k < per; ++k) {
                                c0 += cs[2 * (at * per + k)];
                                c1 += cs[2 * (at * per + k) + 1];
                            }
#pragma unroll
                            for (int p = 0; p < 4; ++p)
                                if (p == near_pr) {
                                    if (fabs(st.m[p][0]) <= zb && c0 == 0) st.m[p][0] = 0.0;
                                    if (fabs(st.m[p][1]) <= zb && c1 == 0) st.m[p][1] = 0.0;
                                }
                        }
                        buf ^= 1;
                    }
                }
            };
            if (n_now > 0) walk(now, n_now, false);
            for (int i = 0; i < n_later; ++i) {
                const int pr = static_cast<int>(later >> (2 * i)) & 3;
                int lo1, hi1, lo2, hi2;
                cr3::sd3_pair_bounds(pr, lo, hi, &lo1, &hi1, &lo2, &hi2);
                __syncthreads();
                build(lo1, hi1, lo2, hi2, false);
                t_valid = false;   // the pair's tables replace the weaker parts'
                walk(static_cast<unsigned>(pr), 1, true);
            }
        }
        // advance the weaker parts' tables past this group: its tying hands
        // join the first opponent's side, then the second's
        if (t_valid && t_hi == lo) {
            if (!small) {
                t_valid = false;
            } else {
                if (n1 > 0) {
                    cr3::add_hands(tid, kTermThreads, t, 0, elist1, n1);
                    __syncthreads();
                }
                if (n2 > 0) {
                    cr3::add_hands(tid, kTermThreads, t, 1, elist2, n2);
                    __syncthreads();
                }
                t_hi = hi;
            }
        }
        g = hi;
    }
    if (st.h >= 0) out[st.h] = static_cast<T>(cr3::sd3_thread_value(st, I.pot, I.bet));
}

// --------------------------------------------------------------------------
// best response (FP64): exploitability of an average-strategy profile
// avg[(di * 8 + a) * max_h + h] (the SSOutput layout)
// --------------------------------------------------------------------------

__device__ __forceinline__ double avg_sigma(const float *avg, int di, int a, int h, int max_h, int frozen) {
    if (frozen >= 0) return a == frozen ? 1.0 : 0.0;
    return static_cast<double>(avg[(static_cast<size_t>(di) * SS_MAX_ACTIONS + a) * max_h + h]);
}

// reach of one player under the average strategy
__global__ void __launch_bounds__(128) k_br_reach(DevCtx c, const ReachItem *__restrict__ items, int nchunk,
                                                  int H, const float *__restrict__ avg,
                                                  const int *__restrict__ edge_di, int max_h) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const int h = (blockIdx.x - it * nchunk) * blockDim.x + threadIdx.x;
    if (h >= H) return;
    const ReachItem I = items[it];
    const size_t HS = static_cast<size_t>(c.HS);
    const int di = edge_di[I.first_edge];
    const double pr = c.reach_d[static_cast<size_t>(I.parent_row) * HS + h];
    for (int a = 0; a < I.na; ++a)
        c.reach_d[static_cast<size_t>(I.first_edge + a) * HS + h] = pr * avg_sigma(avg, di, a, h, max_h, I.frozen);
}

// value of the traverser's nodes: mode 0 follows the profile, mode 1 takes
// the best action (a pure best response per information set; a frozen node
// keeps its frozen action)
__global__ void __launch_bounds__(128) k_br_value(DevCtx c, const CfvItem *__restrict__ items, int nchunk,
                                                  int H, const float *__restrict__ avg,
                                                  const int *__restrict__ edge_di, int max_h, int mode) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const int h = (blockIdx.x - it * nchunk) * blockDim.x + threadIdx.x;
    if (h >= H) return;
    const CfvItem I = items[it];
    const size_t HS = static_cast<size_t>(c.HS);
    const int di = edge_di[I.first_edge];
    double v = mode == 1 ? -1e300 : 0.0;
    double vf = 0.0;
    for (int a = 0; a < I.na; ++a) {
        double e = 0.0;
        for (int k = c.fr_off[I.first_edge + a]; k < c.fr_off[I.first_edge + a + 1]; ++k)
            e += c.val_d[static_cast<size_t>(c.fr_items[k]) * HS + h];
        if (mode == 1) {
            v = e > v ? e : v;
            if (a == I.frozen) vf = e;
        } else {
            v += avg_sigma(avg, di, a, h, max_h, I.frozen) * e;
        }
    }
    if (mode == 1 && I.frozen >= 0 && I.frozen < I.na) v = vf;
    c.val_d[static_cast<size_t>(I.node) * HS + h] = v;
}

// out = sum over hands h < H of weight(h) * (sum over rows of val_d[row][h]);
// the weights are the traverser's range (reach_d row weight_row); with
// skip_blocked, hands touching the board do not count.  One block, fixed
// reduction order.
__global__ void __launch_bounds__(1024) k_br_root(DevCtx c, const int *__restrict__ rows, int n, int H,
                                                  int weight_row, int trav, int skip_blocked, double *out) {
    wait_prior_grid();
    __shared__ double part[32];
    const size_t HS = static_cast<size_t>(c.HS);
    double acc = 0.0;
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        if (skip_blocked && (c.hand_code[trav * HS + h] & 0x10000)) continue;
        double s = 0.0;
        for (int k = 0; k < n; ++k) s += c.val_d[static_cast<size_t>(rows[k]) * HS + h];
        acc += c.reach_d[static_cast<size_t>(weight_row) * HS + h] * s;
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) *out = v;
    }
}

// Batched best response: the kernels above with every item reading its own
// subgame's context (its FP64 rows, profile and tables); blocks of subgames
// that have left the batch return at once.
__global__ void __launch_bounds__(128) k_avg_many(const DevCtx *__restrict__ ctxs,
                                                  const AvgItem *__restrict__ items, int nchunk) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const AvgItem I = items[it];
    if (!ctxs[I.sg].live) return;
    const DevCtx &c = ctxs[I.sg];
    const int h = (blockIdx.x - it * nchunk) * blockDim.x + threadIdx.x;
    const int max_h = c.max_h;
    if (h >= max_h) return;
    const int fe = c.dec_fe[I.di], na = c.dec_na[I.di], p = c.dec_pl[I.di];
    float *o = c.avg_br + static_cast<size_t>(I.di) * SS_MAX_ACTIONS * max_h;
    if (h >= c.H[p]) {
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) o[static_cast<size_t>(a) * max_h + h] = 0.f;
        return;
    }
    float v[SS_MAX_ACTIONS];
    float sum = 0.f;
    for (int a = 0; a < na; ++a) {
        float x = c.S[static_cast<size_t>(fe + a) * c.HS + h];
        x = x < 0.f ? 0.f : x;
        v[a] = x;
        sum += x;
    }
    const float inv = sum > 0.f ? 1.0f / sum : 1.0f / static_cast<float>(na);
    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
        o[static_cast<size_t>(a) * max_h + h] = a < na ? (sum > 0.f ? v[a] * inv : inv) : 0.f;
}

__global__ void __launch_bounds__(128) k_br_reach_many(const DevCtx *__restrict__ ctxs,
                                                       const ReachItem *__restrict__ items, int nchunk, int p) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const ReachItem I = items[it];
    if (!ctxs[I.sg].live) return;
    const DevCtx &c = ctxs[I.sg];
    const int h = (blockIdx.x - it * nchunk) * blockDim.x + threadIdx.x;
    if (h >= c.H[p]) return;
    const size_t HS = static_cast<size_t>(c.HS);
    const int di = c.edge_di[I.first_edge];
    const double pr = c.reach_d[static_cast<size_t>(I.parent_row) * HS + h];
    for (int a = 0; a < I.na; ++a)
        c.reach_d[static_cast<size_t>(I.first_edge + a) * HS + h] = pr * avg_sigma(c.avg_br, di, a, h, c.max_h, I.frozen);
}

__global__ void __launch_bounds__(128) k_br_value_many(const DevCtx *__restrict__ ctxs,
                                                       const CfvItem *__restrict__ items, int nchunk, int trav,
                                                       int mode) {
    wait_prior_grid();
    const int it = blockIdx.x / nchunk;
    const CfvItem I = items[it];
    if (!ctxs[I.sg].live) return;
    const DevCtx &c = ctxs[I.sg];
    const int h = (blockIdx.x - it * nchunk) * blockDim.x + threadIdx.x;
    if (h >= c.H[trav]) return;
    const size_t HS = static_cast<size_t>(c.HS);
    const int di = c.edge_di[I.first_edge];
    double v = mode == 1 ? -1e300 : 0.0;
    double vf = 0.0;
    for (int a = 0; a < I.na; ++a) {
        double e = 0.0;
        for (int k = c.fr_off[I.first_edge + a]; k < c.fr_off[I.first_edge + a + 1]; ++k)
            e += c.val_d[static_cast<size_t>(c.fr_items[k]) * HS + h];
        if (mode == 1) {
            v = e > v ? e : v;
            if (a == I.frozen) vf = e;
        } else {
            v += avg_sigma(c.avg_br, di, a, h, c.max_h, I.frozen) * e;
        }
    }
    if (mode == 1 && I.frozen >= 0 && I.frozen < I.na) v = vf;
    c.val_d[static_cast<size_t>(I.node) * HS + h] = v;
}

// one block per item, same fixed reduction order as k_br_root
__global__ void __launch_bounds__(1024) k_br_root_many(const DevCtx *__restrict__ ctxs,
                                                       const RootItem *__restrict__ items, double *out) {
    wait_prior_grid();
    __shared__ double part[32];
    const RootItem I = items[blockIdx.x];
    if (!ctxs[I.sg].live) return;
    const DevCtx &c = ctxs[I.sg];
    const size_t HS = static_cast<size_t>(c.HS);
    const int H = c.H[I.trav];
    double acc = 0.0;
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        if (I.skip_blocked && (c.hand_code[I.trav * HS + h] & 0x10000)) continue;
        double s = 0.0;
        for (int k = 0; k < I.n; ++k) s += c.val_d[static_cast<size_t>(I.rows[k]) * HS + h];
        acc += c.reach_d[static_cast<size_t>(I.weight_row) * HS + h] * s;
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) out[I.slot] = v;
    }
}

// batched form: advance the iteration counter of every listed subgame
__global__ void k_bump_many(const DevCtx *__restrict__ ctxs, const int *__restrict__ sgs, int n) {
    wait_prior_grid();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && ctxs[sgs[i]].live) *const_cast<int *>(ctxs[sgs[i]].iter) += 1;
}

// batched form: root strategy snapshot (regret matching of the root node)
// of every listed subgame, one block per subgame, into its ctx.snap
__global__ void __launch_bounds__(128) k_snapshot_many(const DevCtx *__restrict__ ctxs,
                                                       const int *__restrict__ sgs) {
    wait_prior_grid();
    const DevCtx &c = ctxs[sgs[blockIdx.x]];
    if (!c.live) return;
    root_strategy(c.R, static_cast<size_t>(c.HS), c.root_fe, c.root_na, c.root_frozen, c.H[c.root_player], c.snap,
                  threadIdx.x, blockDim.x);
}

__global__ void k_bump(int *iter, int by) {
    wait_prior_grid();
    *iter += by;
}

// out[h] = sum over rows of val[row][h]
__global__ void __launch_bounds__(kHandThreads) k_sum_rows(DevCtx c, const int *__restrict__ rows, int n,
                                                           float *out, int H) {
    wait_prior_grid();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= H) return;
    float s = 0.f;
    for (int k = 0; k < n; ++k) s += c.val[static_cast<size_t>(rows[k]) * c.HS + h];
    out[h] = s;
}

__global__ void __launch_bounds__(kHandThreads) k_root_strategy(DevCtx c, int fe, int na, int frozen,
                                                                int H, float *out) {
    wait_prior_grid();
    root_strategy(c.R, static_cast<size_t>(c.HS), fe, na, frozen, H, out, blockIdx.x * blockDim.x + threadIdx.x,
                  gridDim.x * blockDim.x);
}

// normalised strategy sums of every decision node in the output layout
// [num_dec][8][max_h] (street_solve.cu:1589-1612)
__global__ void __launch_bounds__(128) k_avg_strategy(DevCtx c, const int *__restrict__ dec_fe,
                                                      const int *__restrict__ dec_na,
                                                      const int *__restrict__ dec_player, int nchunk,
                                                      int max_h, float *out) {
    wait_prior_grid();
    const int di = blockIdx.x / nchunk;
    const int h = (blockIdx.x - di * nchunk) * blockDim.x + threadIdx.x;
    if (h >= max_h) return;
    const int fe = dec_fe[di], na = dec_na[di], p = dec_player[di];
    float *o = out + static_cast<size_t>(di) * SS_MAX_ACTIONS * max_h;
    if (h >= c.H[p]) {
        for (int a = 0; a < SS_MAX_ACTIONS; ++a) o[static_cast<size_t>(a) * max_h + h] = 0.f;
        return;
    }
    float v[SS_MAX_ACTIONS];
    float sum = 0.f;
    for (int a = 0; a < na; ++a) {
        float x = c.S[static_cast<size_t>(fe + a) * c.HS + h];
        x = x < 0.f ? 0.f : x;
        v[a] = x;
        sum += x;
    }
    const float inv = sum > 0.f ? 1.0f / sum : 1.0f / static_cast<float>(na);
    for (int a = 0; a < SS_MAX_ACTIONS; ++a)
        o[static_cast<size_t>(a) * max_h + h] = a < na ? (sum > 0.f ? v[a] * inv : inv) : 0.f;
}

inline int chunks(int H) { return (H + kHandsPerBlock - 1) / kHandsPerBlock; }

// The tensor-core form of the two-opponent terminals serves dense decks of
// at most 48 cards (turn and river boards) without repeated combos; c is the
// launch's context (for a batch: the largest deck and the OR of every
// member's repeated-combo flags).  It is taken only with SSB_CR2_TENSOR=1 in
// the environment: measured on the 3-player turn it is slower than the
// mma.sync form (0.70 vs 0.55 ms of two-opponent terminals per iteration) --
// its operand space (55 KB per block) leaves four blocks per SM instead of
// five, and a block's time is set by its serial phases, not the product.
bool tensor_product_serves(const DevCtx &c) {
    static const bool on = [] {
        const char *v = std::getenv("SSB_CR2_TENSOR");
        return v && v[0] == '1';
    }();
    if (!on || c.deck <= 0 || c.deck > kTcRows) return false;
    for (int p = 0; p < SS_MAX_PLAYERS; ++p)
        if (c.dup[p]) return false;
    return true;
}

}  // namespace

bool cr2_tensor_form(const DevCtx &c) { return tensor_product_serves(c); }

cudaError_t read_device_fault(unsigned *code, cudaStream_t s) {
    *code = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(code, g_ss_fault, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && *code) {
        static const unsigned zero = 0;
        e = cudaMemcpyToSymbolAsync(g_ss_fault, &zero, sizeof(unsigned), 0, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    return e;
}

cudaError_t launch_reach(const DevCtx &c, const ReachItem *items, int n, int H, cudaStream_t s,
                         const DevCtx *ctxs, int player) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    const int nc = chunks(H), units = n * nc;
    SSB_LAUNCH(k_reach, (units + kReachUnits - 1) / kReachUnits, kHandThreads * kReachUnits, 0, s, c, ctxs, items, units,
               nc, H, player);
    return cudaGetLastError();
}

cudaError_t launch_cfv(const DevCtx &c, const CfvItem *items, int n, int n_long, int H, cudaStream_t s,
                       const DevCtx *ctxs, int trav, int iter_add) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    n_long = n_long < 0 ? 0 : n_long > n ? n : n_long;
    const int n_short = n - n_long;
    const int pairs = (H + 1) / 2, most = cfv_items_per_launch(pairs);
    for (long long at = 0; at < n_short; at += most) {
        const int now = static_cast<int>(std::min<long long>(n_short - at, most));
        const long long threads = static_cast<long long>(now) * pairs;
        SSB_LAUNCH(k_cfv<1>, static_cast<unsigned>((threads + kCfvThreads - 1) / kCfvThreads), kCfvThreads, 0, s, c, ctxs,
                   items + at, now, pairs, H, trav, iter_add);
    }
    if (n_long > 0) {
        const int nc = (H + 63) / 64;
        static_assert(32 * kCfvSplit == kCfvThreads, "the split form fills one block of kCfvThreads");
        SSB_LAUNCH(k_cfv<kCfvSplit>, n_long * nc, kCfvThreads, 0, s, c, ctxs, items + n_short, n_long, nc, H, trav,
                   iter_add);
    }
    return cudaGetLastError();
}

cudaError_t launch_tree(const DevCtx &c, const TreeRef &t, int H, cudaStream_t s, int iter_add) {
    if (t.n_stages <= 0 || H <= 0) return cudaSuccess;
    const unsigned grid = static_cast<unsigned>((H + kTreeHands - 1) / kTreeHands);
    size_t sm = static_cast<size_t>(t.max_chains) * kTreeHands * sizeof(float);
    if (t.bytes <= kTreeResident) {
        sm += static_cast<size_t>(t.bytes);
        const cudaError_t e = cudaFuncSetAttribute(k_tree<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   kTreeResident + kTreeChains * kTreeHands * 4);
        if (e != cudaSuccess) return e;
        SSB_LAUNCH(k_tree<true>, grid, t.threads, sm, s, c, t, H, iter_add);
    } else {
        SSB_LAUNCH(k_tree<false>, grid, t.threads, sm, s, c, t, H, iter_add);
    }
    return cudaGetLastError();
}

// The grid: a block per 8 hands and per terminal job, at most one per SM.  The
// groups of folds or leaves are dealt one by one to as many blocks as that leaves
// within what the hands ask for, or half the SMs if that is more (so that two
// sessions run side by side), up to four to a block at a time.  Groups, not items:
// the three other continuation choices of a leaf follow its first, and items
// taken four by four left three of four thread groups idle.  Microseconds per
// iteration in fours of items and so: heads-up turn of 1,081 nodes 42.2 and
// 38.9, river of 51 nodes and 1,081 hands 19.7 and 18.0.
int small_solve_blocks(const DevCtx &c, SmallRef *ref) {
    SmallRef &s = *ref;
    int dev = 0, coop = 0, sms = 0, optin = 0, per_sm = 0;
    s.at = small_layout(s, c.HS, c.ncomb, c.H);
    const size_t sm = s.at.total;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        sm > static_cast<size_t>(optin - 1024) ||
        cudaFuncSetAttribute(k_small_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_small_solve, kSmallThreads, sm) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        return 0;
    }
    int widest = 1;
    for (int t = 0; t < 2; ++t) {
        const int zeros = (s.n_zero[t] + kLightGroups - 1) / kLightGroups;
        const int most = std::max((std::max(c.H[0], c.H[1]) + kTreeHands - 1) / kTreeHands, sms / 2);
        const int fewest = (s.n_cr1[t] + kLightGroups - 1) / kLightGroups;
        s.cr1_jobs[t] = std::max(fewest, std::min(s.n_cr1[t], most - s.n_sd1[t] - zeros));
        const int jobs = s.n_sd1[t] + s.cr1_jobs[t] + zeros;
        const int chunks = (c.H[t] + kTreeHands - 1) / kTreeHands;
        if (chunks > sms) return 0;   // a block owns 8 hands for the whole launch
        widest = std::max({widest, jobs, chunks});
    }
    return std::min(widest, sms);
}

cudaError_t launch_small_solve(const DevCtx &c, const SmallRef &s, int blocks, int iters, bool snapshot,
                               cudaStream_t st) {
    // the barrier counts from 0 in every launch (after a fault, too)
    const cudaError_t e = cudaMemsetAsync(s.barrier, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    DevCtx ctx = c;
    SmallRef ref = s;
    int n = iters, snap = snapshot ? 1 : 0;
    void *args[] = {&ctx, &ref, &n, &snap};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_small_solve), dim3(blocks), dim3(kSmallThreads),
                                       args, s.at.total, st);
}

template <class T>
cudaError_t launch_terms_t(const DevCtx &c, int kind, const TermItem *items, int n, int trav,
                           cudaStream_t s, const DevCtx *ctxs, const int *heads = nullptr, int n_heads = 0) {
    if (n <= 0 || (heads && n_heads <= 0)) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    switch (kind) {
        case TK_ZERO:
        case TK_LEAF0: {
            const int nc = chunks(c.HS);
            SSB_LAUNCH(k_term_fill<T>, n * nc, kHandThreads, 0, s, c, ctxs, items, nc, trav, kind == TK_ZERO);
            break;
        }
        case TK_CR1: {
            const size_t sm = cr1_gather_smem<T>(c.HS);
            if (sm > 48 * 1024)
                e = cudaFuncSetAttribute(k_term_cr1<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(cr1_gather_smem<T>(kMaxHS)));
            if (e != cudaSuccess) return e;
            SSB_LAUNCH(k_term_cr1<T>, n, kTermThreads, sm, s, c, ctxs, items, trav);
            break;
        }
        case TK_CR1D:
            SSB_LAUNCH(k_term_cr1_dup<T>, n, kTermThreads, cr1_smem<T>(), s, c, ctxs, items, trav);
            break;
        case TK_CR2: {
            // c.HS: the row stride (the largest of a batch); the staging of two
            // reach rows in the product's space needs HS <= kMaxHS
            if (c.HS > kMaxHS) return cudaErrorInvalidValue;
            if constexpr (sizeof(T) == 4) {
                if (tensor_product_serves(c)) {
                    e = cudaFuncSetAttribute(k_term_cr2_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(cr2_tc_smem(kMaxHS)));
                    if (e != cudaSuccess) return e;
                    SSB_LAUNCH(k_term_cr2_tc, n, kTermThreads, cr2_tc_smem(c.HS), s, c, ctxs, items, trav);
                    break;
                }
            }
            const size_t sm = cr2_smem<T>(c.HS);
            if (sm > 48 * 1024)
                e = cudaFuncSetAttribute(k_term_cr2<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(cr2_smem<T>(kMaxHS)));
            if (e != cudaSuccess) return e;
            SSB_LAUNCH(k_term_cr2<T>, heads ? n_heads : n, kTermThreads, sm, s, c, ctxs, items, heads, trav);
            break;
        }
        case TK_SD1:
            static_assert(sd1_smem<T>() <= 48 * 1024, "no attribute needed");
            if (n <= kSd1Few)
                SSB_LAUNCH((k_term_sd1<kSd1Threads, T>), n, kSd1Threads, sd1_smem<T>(), s, c, ctxs, items, trav);
            else
                SSB_LAUNCH((k_term_sd1<kTermThreads, T>), n, kTermThreads, sd1_smem<T>(), s, c, ctxs, items, trav);
            break;
        case TK_SD2: {
            // runs per block: about two waves of four blocks per SM at most
            const int lgm = sd2_merge_of(n);
            const size_t sm = sd2_smem<T>(c.sd_span[lgm], c.ncomb);
            e = cudaFuncSetAttribute(k_term_sd2<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(sd2_smem<T>(kMaxSpan, kMaxSpan)));
            if (e != cudaSuccess) return e;
            SSB_LAUNCH(k_term_sd2<T>, n * (kSd2Chunks >> lgm), kTermThreads, sm, s, c, ctxs, items, trav, lgm, nullptr);
            break;
        }
        case TK_ENUM: {
            // blocks per terminal: one per 4 hands, at most 16 (they stride
            // over a larger range; a batch's c.HS is its largest row stride)
            const int nc = std::min((c.HS + kEnumWarps - 1) / kEnumWarps, 16);
            SSB_LAUNCH(k_term_enum<T>, n * nc, 32 * kEnumWarps, 0, s, c, ctxs, items, nc, trav);
            break;
        }
        case TK_SD3: {
            // the grid covers the 1081 rank positions of a river board
            if (c.HS > kMaxHS || c.ncomb > kSd3Positions) return cudaErrorInvalidValue;
            const int nc = (kSd3Positions + kTermThreads - 1) / kTermThreads;
            e = cudaFuncSetAttribute(k_term_sd3<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(sd3_smem<T>(kMaxHS)));
            if (e != cudaSuccess) return e;
            SSB_LAUNCH(k_term_sd3<T>, n * nc, kTermThreads, sd3_smem<T>(c.HS), s, c, ctxs, items, nc, trav);
            break;
        }
        case TK_CR3: {
            if (c.HS > kMaxHS || c.deck < 0 || c.deck > 52) return cudaErrorInvalidValue;
            const int rounds = (c.HS + kCr3Threads - 1) / kCr3Threads;
            const int nc = std::min(rounds, std::max(1, kCr3Blocks / n));
            e = cudaFuncSetAttribute(k_term_cr3<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(cr3_smem(52)));
            if (e != cudaSuccess) return e;
            SSB_LAUNCH(k_term_cr3<T>, n * nc, kCr3Threads, cr3_smem(c.deck), s, c, ctxs, items, nc, trav);
            break;
        }
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_terms(const DevCtx &c, int kind, const TermItem *items, int n, int trav,
                         cudaStream_t s, const DevCtx *ctxs, const int *heads, int n_heads) {
    return launch_terms_t<float>(c, kind, items, n, trav, s, ctxs, heads, n_heads);
}

cudaError_t launch_terms_light(const DevCtx &c, const TermItem *sd1, int n_sd1, const TermItem *cr1, int n_cr1,
                               const TermItem *zero, int n_zero, int trav, cudaStream_t s, const DevCtx *ctxs) {
    const int grid = n_sd1 + (n_cr1 + kLightGroups - 1) / kLightGroups + (n_zero + kLightGroups - 1) / kLightGroups;
    if (grid <= 0) return cudaSuccess;
    const size_t sm = std::max(sd1_smem<float>(), n_cr1 > 0 ? kLightGroups * cr1_gather_smem<float>(c.HS) : 0);
    if (sm > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_term_light, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(std::max(sd1_smem<float>(), kLightGroups * cr1_gather_smem<float>(kMaxHS))));
        if (e != cudaSuccess) return e;
    }
    SSB_LAUNCH(k_term_light, grid, kSd1Threads, sm, s, c, ctxs, sd1, n_sd1, cr1, n_cr1, zero, n_zero, trav);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_sd2_mapped_t(const DevCtx &c, const TermItem *items, const int2 *bmap, int nblocks, int lg_max,
                                int trav, cudaStream_t s, const DevCtx *ctxs) {
    if (nblocks <= 0) return cudaSuccess;
    const size_t sm = sd2_smem<T>(c.sd_span[lg_max], c.ncomb);
    cudaError_t e = cudaFuncSetAttribute(k_term_sd2<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sd2_smem<T>(kMaxSpan, kMaxSpan)));
    if (e != cudaSuccess) return e;
    SSB_LAUNCH(k_term_sd2<T>, nblocks, kTermThreads, sm, s, c, ctxs, items, trav, 0, bmap);
    return cudaGetLastError();
}

cudaError_t launch_sd2_mapped(const DevCtx &c, const TermItem *items, const int2 *bmap, int nblocks, int lg_max,
                              int trav, cudaStream_t s, const DevCtx *ctxs, bool fp64) {
    return fp64 ? launch_sd2_mapped_t<double>(c, items, bmap, nblocks, lg_max, trav, s, ctxs)
                : launch_sd2_mapped_t<float>(c, items, bmap, nblocks, lg_max, trav, s, ctxs);
}

cudaError_t launch_terms_fp64(const DevCtx &c, int kind, const TermItem *items, int n, int trav,
                              cudaStream_t s, const DevCtx *ctxs) {
    return launch_terms_t<double>(c, kind, items, n, trav, s, ctxs);
}

cudaError_t launch_avg_many(const DevCtx *ctxs, const AvgItem *items, int n, int max_h, cudaStream_t s) {
    if (n <= 0 || max_h <= 0) return cudaSuccess;
    const int nc = (max_h + 127) / 128;
    SSB_LAUNCH(k_avg_many, n * nc, 128, 0, s, ctxs, items, nc);
    return cudaGetLastError();
}

cudaError_t launch_br_reach_many(const DevCtx *ctxs, const ReachItem *items, int n, int H, int player,
                                 cudaStream_t s) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    const int nc = (H + 127) / 128;
    SSB_LAUNCH(k_br_reach_many, n * nc, 128, 0, s, ctxs, items, nc, player);
    return cudaGetLastError();
}

cudaError_t launch_br_value_many(const DevCtx *ctxs, const CfvItem *items, int n, int H, int trav, int mode,
                                 cudaStream_t s) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    const int nc = (H + 127) / 128;
    SSB_LAUNCH(k_br_value_many, n * nc, 128, 0, s, ctxs, items, nc, trav, mode);
    return cudaGetLastError();
}

cudaError_t launch_br_root_many(const DevCtx *ctxs, const RootItem *items, int n, double *out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    SSB_LAUNCH(k_br_root_many, n, 1024, 0, s, ctxs, items, out);
    return cudaGetLastError();
}

cudaError_t launch_bump(int *iter, int by, cudaStream_t s) {
    SSB_LAUNCH(k_bump, 1, 1, 0, s, iter, by);
    return cudaGetLastError();
}

cudaError_t launch_sum_rows(const DevCtx &c, const int *rows, int n, float *out, int H,
                            cudaStream_t s) {
    if (H <= 0) return cudaSuccess;
    SSB_LAUNCH(k_sum_rows, (H + kHandThreads - 1) / kHandThreads, kHandThreads, 0, s, c, rows, n, out, H);
    return cudaGetLastError();
}

cudaError_t launch_root_strategy(const DevCtx &c, int first_edge, int na, int frozen, int H,
                                 float *out, cudaStream_t s) {
    if (H <= 0) return cudaSuccess;
    SSB_LAUNCH(k_root_strategy, (H + kHandsPerBlock - 1) / kHandsPerBlock, kHandThreads, 0, s,
               c, first_edge, na, frozen, H, out);
    return cudaGetLastError();
}

cudaError_t launch_avg_strategy(const DevCtx &c, const int *dec_fe, const int *dec_na,
                                const int *dec_player, int num_dec, int max_h, float *out,
                                cudaStream_t s) {
    if (num_dec <= 0) return cudaSuccess;
    const int nc = (max_h + 127) / 128;
    SSB_LAUNCH(k_avg_strategy, num_dec * nc, 128, 0, s, c, dec_fe, dec_na, dec_player, nc, max_h, out);
    return cudaGetLastError();
}

cudaError_t launch_br_reach(const DevCtx &c, const ReachItem *items, int n, int H, const float *avg,
                            const int *edge_di, int max_h, cudaStream_t s) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    const int nc = (H + 127) / 128;
    SSB_LAUNCH(k_br_reach, n * nc, 128, 0, s, c, items, nc, H, avg, edge_di, max_h);
    return cudaGetLastError();
}

cudaError_t launch_br_value(const DevCtx &c, const CfvItem *items, int n, int H, const float *avg,
                            const int *edge_di, int max_h, int mode, cudaStream_t s) {
    if (n <= 0 || H <= 0) return cudaSuccess;
    const int nc = (H + 127) / 128;
    SSB_LAUNCH(k_br_value, n * nc, 128, 0, s, c, items, nc, H, avg, edge_di, max_h, mode);
    return cudaGetLastError();
}

cudaError_t launch_br_root(const DevCtx &c, const int *rows, int n, int H, int weight_row, int trav,
                           int skip_blocked, double *out, cudaStream_t s) {
    SSB_LAUNCH(k_br_root, 1, 1024, 0, s, c, rows, n, H, weight_row, trav, skip_blocked, out);
    return cudaGetLastError();
}

cudaError_t launch_bump_many(const DevCtx *ctxs, const int *sgs, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    SSB_LAUNCH(k_bump_many, (n + 127) / 128, 128, 0, s, ctxs, sgs, n);
    return cudaGetLastError();
}

cudaError_t launch_snapshot_many(const DevCtx *ctxs, const int *sgs, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    SSB_LAUNCH(k_snapshot_many, n, 128, 0, s, ctxs, sgs);
    return cudaGetLastError();
}

}  // namespace ssb
