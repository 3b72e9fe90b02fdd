// Link construction on the GPU: the dual-tree traversal of
// CAutoRefine::RefineMutual / RefineSelf (Solver/Autorefine.cpp:3096-3235,
// 2115-2229) and the bucketing of the emitted pairs by destination node
// (the link lists of CAutoRefine::RecurseIndex, Solver/Autorefine.cpp:1173-1220).
//
// Traversal. Every root pair (one per conductor pair, then one per internal
// element for the self interactions, in the host traversal's order) starts a
// binary recursion tree: a pair either links (a leaf of the recursion tree)
// or is replaced by two pairs, the children of one side. The frontier is
// expanded one level per launch; the two children of a split pair are placed
// next to each other, wherever in the next level the warp's atomic puts them,
// and every split pair remembers where. A bottom-up pass counts the links
// under every frontier item and a top-down pass hands out depth-first
// positions (an exclusive scan over the roots, then parent offset / parent
// offset + left child count): the emitted pairs come out in exactly the order
// of the recursive host traversal, in whatever order a level holds its pairs.
//
// Buckets. Pair k = (a, b) gives the entries (dest a, src b) and (dest b,
// src a); a stable LSD radix sort on the destination (8-bit digits, warp
// match for the stable rank) keeps every row in emission order, which is the
// host builder's stable counting sort.
//
// This file is compiled with -fmad=false so that fcg_link_decision rounds
// every operation the way the host builder (-ffp-contract=off) does: the
// device takes exactly the host's decisions and produces the same arrays.
#include <cuda_runtime.h>

#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <chrono>
#include <string>
#include <vector>

#include "fc_potential.h"
#include "pair32.cuh"
#include "fcg_internal.hpp"
#include "scan.cuh"
#include "../host/model.hpp"

namespace fcg {

using namespace devscan;
using namespace pair32;

namespace {


static_assert(sizeof(Element) == 96, "element record layout");

// ------------------------------------------------------------------ traversal
// FP32 pre-test of every pair (pair32.cuh), FP64 for the undecided ones.

// fcg_link_decision in FP32, or -1 when only the FP64 test can tell
__device__ int decide32(const Element &A, const Element &B, float e, float inv_max_area, float inv_max_side) {
    bool leaf1 = (A.type & FCG_IS_LEAF) != 0, leaf2 = (B.type & FCG_IS_LEAF) != 0;
    if (leaf1 && leaf2) return 0;
    float dx = A.c[0] - B.c[0], dy = A.c[1] - B.c[1], dz = A.c[2] - B.c[2];  // fcg_fsub's float values
    float r = sqrtf(dx * dx + dy * dy + dz * dz);
    double rm = A.maxside > B.maxside ? A.maxside : B.maxside;
    float rho = r / (float)rm;
    if (!(r > 1e-10f) || !(fabsf(rho - 2.0f) > 1e-5f)) return -1;
    bool quad = rho < 2.0f;
    float c1, e1, c2, e2;
    if (!weight32(A, B, dx, dy, dz, r, quad, inv_max_area, inv_max_side, c1, e1)) return -1;
    if (!weight32(B, A, -dx, -dy, -dz, r, quad, inv_max_area, inv_max_side, c2, e2)) return -1;
    int t1 = side_test(c1, e1, e), t2 = side_test(c2, e2, e);
    if (t1 != 1 && t2 != 1) {
        if (t1 == 0 && t2 == 0) return 0;
        return -1;
    }
    if (!leaf1 && leaf2) return 1;
    if (leaf1 && !leaf2) return 2;
    return A.area > B.area ? 1 : 2;
}

// a level's counts on the device: pairs split, pairs for the FP64 test
struct LevelCount {
    unsigned long long splits, listed;
};

// The children of a warp's split pairs (f = 1 or 2: pair i splits its first
// or second element; 0 a link; -1 none of this kernel's) into the next level,
// at places that one atomic hands out; rank[i] says where (r: entries 2 r and
// 2 r + 1; -1: a link).
__device__ __forceinline__ void emit_children(LevelCount *count, int64_t ne, int64_t i, int f, int2 pr, uint16_t rl,
                                              const Element *__restrict__ el, int32_t *__restrict__ rank, int64_t next_cap,
                                              int2 *__restrict__ next, uint16_t *__restrict__ next_level, unsigned *bad) {
    const unsigned split = __ballot_sync(0xffffffffu, f > 0);
    if (f == 0) rank[i] = -1;
    if (!split) return;
    const int64_t r = warp_claim(&count->splits, __popc(split)) + __popc(split & ((1u << (threadIdx.x & 31)) - 1u));
    if (f <= 0) return;
    int2 c0 = pr, c1 = pr;
    if (f == 1) {
        c0.x = el[pr.x].left;
        c1.x = el[pr.x].right;
    } else {
        c0.y = el[pr.y].left;
        c1.y = el[pr.y].right;
    }
    // a split side always has two children; anything else is a corrupt hierarchy
    if (c0.x < 0 || c0.y < 0 || c1.x < 0 || c1.y < 0 || c0.x >= ne || c0.y >= ne || c1.x >= ne || c1.y >= ne) {
        atomicAdd(bad, 1u);
        c0 = c1 = make_int2(0, 0);
    }
    rank[i] = (int32_t)r;
    if (2 * r + 1 < next_cap) {  // always: the next level has room for two children of every pair
        next[2 * r] = c0;
        next[2 * r + 1] = c1;
        next_level[2 * r] = rl;
        next_level[2 * r + 1] = rl;
    }
}

// One level of the traversal: every pair is decided in FP32 where that is
// certain (0 link, 1 split the first element, 2 the second) and its children
// placed at once; the others are listed for k_link_level64. The pairs of this
// level: n0, or twice the splits of the level before (read on the device, so
// that several small levels run without the host).
__global__ void __launch_bounds__(128) k_link_level(int64_t n0, const LevelCount *__restrict__ prev, const int2 *__restrict__ pairs,
                                                    const uint16_t *__restrict__ root_level, int depth, int64_t ne,
                                                    const Element *__restrict__ el, float e, float inv_max_area, float inv_max_side,
                                                    int32_t *__restrict__ rank, int64_t next_cap, int2 *__restrict__ next,
                                                    uint16_t *__restrict__ next_level, LevelCount *count, int32_t *__restrict__ listed,
                                                    int *max_level, unsigned *bad) {
    const int64_t n = prev ? 2 * (int64_t)prev->splits : n0;
    const int lane = threadIdx.x & 31;
    int lvl = 0;
    // whole warps stay in the loop while their first pair exists (ballots below)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i - lane < n; i += (int64_t)gridDim.x * blockDim.x) {
        int f = -1;
        bool undecided = false;
        int2 pr = make_int2(0, 0);
        uint16_t rl = 0;
        if (i < n) {
            pr = pairs[i];
            rl = root_level[i];
            lvl = max(lvl, (int)rl + depth);
            f = decide32(el[pr.x], el[pr.y], e, inv_max_area, inv_max_side);
            undecided = f < 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, undecided);
        if (m) {
            const int64_t at = warp_claim(&count->listed, __popc(m)) + __popc(m & ((1u << lane) - 1u));
            if (undecided) listed[at] = (int32_t)i;
        }
        emit_children(count, ne, i, f, pr, rl, el, rank, next_cap, next, next_level, bad);
    }
    for (int o = 16; o > 0; o >>= 1) lvl = max(lvl, __shfl_xor_sync(0xffffffffu, lvl, o));
    if (lane == 0 && lvl) atomicMax(max_level, lvl);
}

// The FP64 test (the host builder's own code) for the level's listed pairs: two
// lanes a pair, one for each direction's weight, whose arithmetic does not
// change when the two elements swap places (7.8 -> 5.2 us a level of a small
// model; 25 levels of 10.8 million pairs 457 -> 278, 27 of 28 million 618 -> 370).
__global__ void __launch_bounds__(128) k_link_level64(const int2 *__restrict__ pairs, const uint16_t *__restrict__ root_level, int64_t ne,
                                                      const Element *__restrict__ el, double eps, double max_side, double max_area,
                                                      int32_t *__restrict__ rank, int64_t next_cap, int2 *__restrict__ next,
                                                      uint16_t *__restrict__ next_level, LevelCount *count,
                                                      const int32_t *__restrict__ listed, unsigned *bad) {
    const int64_t m = (int64_t)count->listed;
    const int odd = threadIdx.x & 1;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t - (threadIdx.x & 31) < 2 * m; t += (int64_t)gridDim.x * blockDim.x) {
        int f = -1;
        int64_t i = 0;
        int2 pr = make_int2(0, 0);
        uint16_t rl = 0;
        double c = 0.0;
        if (t < 2 * m) {
            i = listed[t >> 1];
            pr = pairs[i];
            rl = root_level[i];
            const Element &A = el[odd ? pr.y : pr.x], &B = el[odd ? pr.x : pr.y];
            fcg_d3 dist;
            double rdist, rmax;
            fcg_pair_span(A, B, &dist, &rdist, &rmax);
            c = fcg_one_way(A, B, dist, rdist, rmax, 1.0, max_side, max_area);
        }
        const double c2 = __shfl_xor_sync(0xffffffffu, c, 1);
        if (t < 2 * m && !odd) {
            const Element &A = el[pr.x], &B = el[pr.y];
            const bool link = (A.type & B.type & FCG_IS_LEAF) || !(c > eps || c2 > eps);
            f = link ? 0 : fcg_link_side(A, B);
        }
        emit_children(count, ne, i, f, pr, rl, el, rank, next_cap, next, next_level, bad);
    }
}

// links under every item (bottom-up; the deepest level has only links)
__global__ void k_count(int64_t n, const int32_t *__restrict__ rank, const long long *__restrict__ cnt_next, long long *cnt) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t r = rank[i];
        cnt[i] = r < 0 ? 1 : cnt_next[2 * (int64_t)r] + cnt_next[2 * (int64_t)r + 1];
    }
}

// depth-first positions (top-down); `next` holds the next level's counts and
// receives its offsets (each pair of entries is touched by its parent only)
__global__ void k_place(int64_t n, const int2 *__restrict__ pairs, const int32_t *__restrict__ rank, const long long *__restrict__ off,
                        long long *next, int2 *out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t r = rank[i];
        long long o = off[i];
        if (r < 0) {
            out[o] = pairs[i];
        } else {
            long long c0 = next[2 * (int64_t)r];
            next[2 * (int64_t)r] = o;
            next[2 * (int64_t)r + 1] = o + c0;
        }
    }
}

// ------------------------------------------------------------------ buckets
// pair k -> entries 2k (dest a, src b) and 2k+1 (dest b, src a); node degrees
__global__ void k_entries(int64_t P, const int2 *__restrict__ pairs, const int32_t *__restrict__ node_of,
                          unsigned long long *ent, int *deg) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < P; k += (int64_t)gridDim.x * blockDim.x) {
        int2 pr = pairs[k];
        unsigned a = (unsigned)node_of[pr.x], b = (unsigned)node_of[pr.y];
        ent[2 * k] = ((unsigned long long)a << 32) | b;
        ent[2 * k + 1] = ((unsigned long long)b << 32) | a;
        atomicAdd(deg + a, 1);
        atomicAdd(deg + b, 1);
    }
}

// ------------------------------------------------------------------ host side
constexpr size_t kMaxGroup = 24;       // levels launched at a time (the bound doubles: at most 18)
constexpr int64_t kNoWait = 1 << 18;  // pairs up to which levels are launched without knowing their size
// Pairs of room that the levels held may have beyond their sizes: a level is
// made for twice the pairs of the one before, and about half of them split. Up to
// this much (32 MB) it stays; then levels are copied to arrays of their sizes,
// since all of them are held until the placement, whose counts and emitted
// pairs (12 bytes a pair test, next to 12 of the levels) are the peak of the
// build (127 million pair tests: 4745 -> 3159 MB).
constexpr int64_t kUnusedPairs = 4 << 20;

struct Level {
    int64_t n = 0, room = 0, rank_room = 0;  // pairs, and what `pairs` and `rank` have room for
    int2 *pairs = nullptr;
    uint16_t *root_level = nullptr;
    int32_t *rank = nullptr;
    long long *cnt = nullptr;
};


}  // namespace

#define LB_CK(x)                                                                                     \
    do {                                                                                             \
        cudaError_t e_ = (x);                                                                        \
        if (e_ != cudaSuccess) {                                                                     \
            err = std::string("device link construction: ") + cudaGetErrorString(e_);               \
            cudaGetLastError();                                                                      \
            return e_ == cudaErrorMemoryAllocation ? FCG_OUT_OF_MEMORY : FCG_DEVICE_ERROR;           \
        }                                                                                            \
    } while (0)

int link_build_device(DeviceContext &ctx, const Element *el, int64_t ne, const LinkRoots &roots, bool on_device,
                      int64_t n_nodes, double eps, double max_side, double max_area, std::vector<int64_t> &link_ptr,
                      std::vector<int32_t> &link_src, int &max_level, std::string &err,
                      std::shared_ptr<int32_t> *device_src) {
    LB_CK(cudaSetDevice(ctx.device));
    Bufs B;
    LB_CK(cudaStreamCreateWithFlags(&B.s, cudaStreamNonBlocking));
    cudaStream_t s = B.s;
    const int sms = ctx.sm_count > 0 ? ctx.sm_count : 1;
    link_ptr.assign((size_t)n_nodes + 1, 0);
    link_src.clear();
    max_level = 0;
    const int64_t n_roots = roots.n;
    if (n_roots == 0 || n_nodes == 0) return FCG_NORMAL_END;

    const Element *d_el = el;
    const int32_t *d_node_of = roots.node_of.get();
    long long *d_scalars;  // [0] scan total, [1] spare
    int *d_max_level;
    unsigned *d_bad;
    LevelCount *d_count;  // per level of a group
    int32_t *d_listed = nullptr;
    int64_t listed_room = 0;
    const bool trace = getenv("FCG_TRACE") != nullptr;
    const auto t_begin = std::chrono::steady_clock::now();
    LB_CK(B.alloc(&d_count, kMaxGroup));
    LB_CK(B.alloc(&d_scalars, 2));
    LB_CK(B.alloc(&d_max_level, 1));
    LB_CK(B.alloc(&d_bad, 1));
    if (!on_device) {
        Element *up;
        int32_t *up_of;
        LB_CK(B.alloc(&up, (size_t)ne));
        LB_CK(B.alloc(&up_of, (size_t)ne));
        LB_CK(cudaMemcpyAsync(up, el, (size_t)ne * sizeof(Element), cudaMemcpyHostToDevice, s));
        LB_CK(cudaMemcpyAsync(up_of, d_node_of, (size_t)ne * sizeof(int32_t), cudaMemcpyHostToDevice, s));
        d_el = up;
        d_node_of = up_of;
    }
    LB_CK(cudaMemsetAsync(d_max_level, 0, sizeof(int), s));
    LB_CK(cudaMemsetAsync(d_bad, 0, sizeof(unsigned), s));

    // roots
    std::vector<Level> lv(1);
    {
        Level &L0 = lv[0];
        L0.n = n_roots;
        const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
        L0.room = n_roots;
        LB_CK(B.alloc(&L0.pairs, (size_t)n_roots));
        LB_CK(B.alloc(&L0.root_level, (size_t)n_roots));
        LB_CK(cudaMemcpyAsync(L0.pairs, roots.pairs.get(), (size_t)n_roots * sizeof(int2), kind, s));
        LB_CK(cudaMemcpyAsync(L0.root_level, roots.level.get(), (size_t)n_roots * sizeof(uint16_t), kind, s));
    }

    // frontier expansion, one level per launch. A level has at most twice the
    // pairs of the one before: the host waits for the counts only when that
    // bound has grown past kNoWait pairs since it last knew them.
    long long n_tests = 0, n_fp64 = 0;
    // an array of n elements in the place of a larger one
    auto shrink = [&](auto *&p, int64_t &room, int64_t n) -> cudaError_t {
        if (room <= n) return cudaSuccess;
        room = n;
        auto *old = p;
        cudaError_t e = B.alloc(&p, (size_t)n);
        if (e == cudaSuccess) e = cudaMemcpyAsync(p, old, (size_t)n * sizeof(*p), cudaMemcpyDeviceToDevice, s);
        B.release(old);
        return e;
    };
    for (bool more = true; more;) {
        const size_t first = lv.size() - 1;  // its size is known
        int64_t bound = lv[first].n;
        size_t d = first;
        LB_CK(cudaMemsetAsync(d_count, 0, kMaxGroup * sizeof(LevelCount), s));
        do {
            if (bound > (1ll << 30)) {
                err = "model too large for 32-bit link indices";
                return FCG_OUT_OF_MEMORY;
            }
            if (bound > listed_room) {
                B.release(d_listed);
                listed_room = std::max<int64_t>(bound, kNoWait);
                LB_CK(B.alloc(&d_listed, (size_t)listed_room));
            }
            lv[d].rank_room = bound;
            LB_CK(B.alloc(&lv[d].rank, (size_t)bound));
            Level nx;
            nx.n = nx.room = 2 * bound;
            LB_CK(B.alloc(&nx.pairs, (size_t)nx.n));
            LB_CK(B.alloc(&nx.root_level, (size_t)nx.n));
            const Level &L = lv[d];
            LevelCount *count = d_count + (d - first);
            k_link_level<<<grid_stride(bound, sms, 128), 128, 0, s>>>(
                L.n, d > first ? count - 1 : nullptr, L.pairs, L.root_level, (int)d, ne, d_el, (float)eps, (float)(1.0 / max_area),
                (float)(1.0 / max_side), L.rank, nx.n, nx.pairs, nx.root_level, count, d_listed, d_max_level, d_bad);
            k_link_level64<<<grid_stride(bound, sms, 128), 128, 0, s>>>(L.pairs, L.root_level, ne, d_el, eps, max_side, max_area, L.rank,
                                                                       nx.n, nx.pairs, nx.root_level, count, d_listed, d_bad);
            LB_CK(cudaGetLastError());
            lv.push_back(nx);
            d++;
            bound *= 2;
        } while (bound <= kNoWait && d - first < kMaxGroup);
        std::vector<LevelCount> counts(d - first);
        LB_CK(cudaMemcpyAsync(counts.data(), d_count, counts.size() * sizeof(LevelCount), cudaMemcpyDeviceToHost, s));
        LB_CK(cudaStreamSynchronize(s));
        for (size_t q = first; q < d; q++) {
            const long long sp = (long long)counts[q - first].splits;
            if (sp > (1ll << 29)) {
                err = "model too large for 32-bit link indices";
                return FCG_OUT_OF_MEMORY;
            }
            n_tests += lv[q].n;
            n_fp64 += (long long)counts[q - first].listed;
            B.release(lv[q].root_level);
            lv[q + 1].n = 2 * sp;
            if (sp == 0) {  // the traversal ended at level q
                for (size_t u = q + 1; u <= d; u++) {
                    B.release(lv[u].pairs);
                    B.release(lv[u].root_level);
                    B.release(lv[u].rank);
                }
                lv.resize(q + 1);
                more = false;
                break;
            }
        }
        // the levels with the most unused room first: each costs an allocation and a copy
        int64_t unused = 0;
        for (const Level &L : lv) unused += L.room - L.n;
        for (int64_t least = kUnusedPairs / 16; unused > kUnusedPairs; least = 1)
            for (Level &L : lv) {
                if (L.room - L.n < least) continue;
                unused -= L.room - L.n;
                LB_CK(shrink(L.pairs, L.room, L.n));
                LB_CK(shrink(L.rank, L.rank_room, L.n));
            }
    }
    B.release(d_listed);
    unsigned bad = 0;
    LB_CK(cudaMemcpyAsync(&bad, d_bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    LB_CK(cudaMemcpyAsync(&max_level, d_max_level, sizeof(int), cudaMemcpyDeviceToHost, s));
    LB_CK(cudaStreamSynchronize(s));
    if (bad) {
        err = "device link construction: a split element without two children (" + std::to_string(bad) + " pairs)";
        return FCG_GENERIC_ERROR;
    }
    if (trace)
        fprintf(stderr, "[fcg links] %zu levels, %lld pair tests, %lld (%.2f %%) by the FP64 test\n", lv.size(), n_tests, n_fp64,
                n_tests ? 100.0 * (double)n_fp64 / (double)n_tests : 0.0);

    auto t_mark = std::chrono::steady_clock::now();
    auto mark = [&](const char *what) {
        if (!trace) return;
        auto now = std::chrono::steady_clock::now();
        fprintf(stderr, "[fcg links]   %-28s %9.3f ms\n", what, std::chrono::duration<double, std::milli>(now - t_mark).count());
        t_mark = now;
    };
    if (trace) fprintf(stderr, "[fcg links]   traversal                    %9.3f ms\n",
                       std::chrono::duration<double, std::milli>(t_mark - t_begin).count());
    // links under every item, deepest level first
    long long *cnt_all;
    LB_CK(B.alloc(&cnt_all, (size_t)n_tests));
    {
        long long *at = cnt_all;
        for (Level &L : lv) {
            L.cnt = at;
            at += L.n;
        }
    }
    for (size_t d = lv.size(); d-- > 0;) {
        Level &L = lv[d];
        const long long *cn = d + 1 < lv.size() ? lv[d + 1].cnt : nullptr;
        k_count<<<grid_stride(L.n, sms), 256, 0, s>>>(L.n, L.rank, cn, L.cnt);
        LB_CK(cudaGetLastError());
    }
    // depth-first positions: scan over the roots, then parent to children
    long long P = 0;
    {
        Level &L0 = lv[0];
        unsigned tiles = grid_tiles(L0.n);
        long long *sums;
        LB_CK(B.alloc(&sums, tiles));
        k_scan_tiles<<<tiles, kThreads, 0, s>>>(L0.n, L0.cnt, sums);
        k_scan_sums<<<1, 1024, 0, s>>>(tiles, sums, d_scalars);
        k_scan_apply<<<tiles, kThreads, 0, s>>>(L0.n, L0.cnt, L0.cnt, sums);
        LB_CK(cudaGetLastError());
        LB_CK(cudaMemcpyAsync(&P, d_scalars, sizeof(long long), cudaMemcpyDeviceToHost, s));
        LB_CK(cudaStreamSynchronize(s));
        B.release(sums);
    }
    if (2 * P > 0x7fffffffLL) {
        err = "model too large for 32-bit link indices";
        return FCG_OUT_OF_MEMORY;
    }
    int2 *emitted;
    LB_CK(B.alloc(&emitted, (size_t)P));
    for (size_t d = 0; d < lv.size(); d++) {
        Level &L = lv[d];
        long long *next = d + 1 < lv.size() ? lv[d + 1].cnt : nullptr;
        k_place<<<grid_stride(L.n, sms), 256, 0, s>>>(L.n, L.pairs, L.rank, L.cnt, next, emitted);
        LB_CK(cudaGetLastError());
    }
    for (Level &L : lv) {
        B.release(L.pairs);
        B.release(L.rank);
    }
    B.release(cnt_all);

    // rows: entries, degrees -> link_ptr, stable radix sort by destination
    const int64_t nent = 2 * P;
    unsigned long long *ent, *ent2 = nullptr;
    int *deg;
    int64_t *d_ptr;
    int32_t *d_src;
    LB_CK(B.alloc(&ent, (size_t)nent));
    LB_CK(B.alloc(&deg, (size_t)n_nodes));
    LB_CK(B.alloc(&d_ptr, (size_t)n_nodes + 1));
    LB_CK(B.alloc(&d_src, (size_t)nent));
    LB_CK(cudaMemsetAsync(deg, 0, (size_t)n_nodes * sizeof(int), s));
    if (P > 0) k_entries<<<grid_stride(P, sms), 256, 0, s>>>(P, emitted, d_node_of, ent, deg);
    LB_CK(cudaGetLastError());
    B.release(emitted);
    {
        unsigned tiles = grid_tiles(n_nodes);
        long long *sums;
        LB_CK(B.alloc(&sums, tiles));
        k_scan_tiles<<<tiles, kThreads, 0, s>>>(n_nodes, deg, sums);
        k_scan_sums<<<1, 1024, 0, s>>>(tiles, sums, (long long *)(d_ptr + n_nodes));
        k_scan_apply<<<tiles, kThreads, 0, s>>>(n_nodes, deg, d_ptr, sums);
        LB_CK(cudaGetLastError());
        B.release(sums);
    }
    B.release(deg);
    if (nent > 0) {
        int bits = 0;
        while (bits < 32 && ((int64_t)1 << bits) < n_nodes) bits++;
        int passes = std::max(1, (bits + 7) / 8);
        unsigned tiles = grid_tiles(nent);
        int64_t nh = (int64_t)tiles * kDigits;
        int *hist;
        long long *hsums;
        unsigned htiles = grid_tiles(nh);
        LB_CK(B.alloc(&hist, (size_t)nh));
        LB_CK(B.alloc(&hsums, htiles));
        if (passes > 1) LB_CK(B.alloc(&ent2, (size_t)nent));
        unsigned long long *src = ent, *dst = ent2;
        for (int pass = 0; pass < passes; pass++) {
            int shift = 32 + 8 * pass;
            bool last = pass == passes - 1;
            k_radix_hist<<<tiles, kThreads, 0, s>>>(nent, src, shift, hist);
            k_scan_tiles<<<htiles, kThreads, 0, s>>>(nh, hist, hsums);
            k_scan_sums<<<1, 1024, 0, s>>>(htiles, hsums, d_scalars + 1);
            k_scan_apply<<<htiles, kThreads, 0, s>>>(nh, hist, hist, hsums);
            k_radix_scatter<<<tiles, kThreads, 0, s>>>(nent, src, shift, hist, last ? nullptr : dst, last ? d_src : nullptr);
            LB_CK(cudaGetLastError());
            std::swap(src, dst);
        }
    }
    if (trace) {
        LB_CK(cudaStreamSynchronize(s));
        mark("placement and row sort");
    }
    LB_CK(cudaMemcpyAsync(link_ptr.data(), d_ptr, ((size_t)n_nodes + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    if (device_src) {
        *device_src = B.hand_over(d_src);
        link_src.clear();
    } else {
        link_src.resize((size_t)nent);
        mark("host link array");
        if (nent > 0) LB_CK(cudaMemcpyAsync(link_src.data(), d_src, (size_t)nent * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    }
    LB_CK(cudaStreamSynchronize(s));
    mark("download");
    if (link_ptr[(size_t)n_nodes] != nent) {
        err = "device link construction: row offsets do not add up to the link count";
        return FCG_GENERIC_ERROR;
    }
    return FCG_NORMAL_END;
}

}  // namespace fcg
