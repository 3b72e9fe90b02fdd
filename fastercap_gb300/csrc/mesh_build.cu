// Adaptive mesh refinement on the GPU: CAutoRefine::DiscretizeMutual /
// DiscretizeSelf (Solver/Autorefine.cpp:2638-2795) with CAutoPanel::Subdivide
// (Solver/AutoPanel.cpp:382-523).
//
// The refined mesh does not depend on the order in which element pairs are
// examined. A pair's test (fcg_mesh_decision) reads only the two elements'
// own geometry, never whether they already have children, and a split
// always bisects the same element the same way (fcg_subdivide) and only once.
// So the mesh is the closure of: refine every conductor pair from the two
// conductors' top elements (`selfc` off); refine the two children of every
// internal element, including every element split along the way (`selfc`
// on). The host builder reaches that closure depth first; here the pairs
// advance one level per step:
//   level    decide every frontier pair (FP32 where certain, else, from a
//            list, by the host builder's own FP64 code); non-split pairs update
//            the largest achieved weight; a split pair is listed for the next
//            step, and the first one to split a leaf gives it the ids of its
//            halves
//   grow     the halves of every leaf given ids (its two halves are a pair of
//            the next frontier, with `selfc`), and every listed pair's two
//            children pairs.
// Places in the next frontier and element ids come from one atomic per warp
// and 32 pairs: no scans, and the host only waits where the next levels' sizes
// have no useful bound.
// The element ids differ from the host builder's (creation order), but the
// tree, and so the flattened model, is the same. Recursion levels are those
// of the host recursion: a conductor pair starts at level 1, the self pair of
// an element at depth s of its conductor's tree at level s + 2.
//
// Compiled with -fmad=false so that every decision and every bisection
// rounds the way the host builder (-ffp-contract=off) does.
#include <cuda_runtime.h>

#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <string>
#include <vector>

#include "fc_potential.h"
#include "pair32.cuh"
#include "fcg_internal.hpp"
#include "scan.cuh"
#include "../host/model.hpp"

namespace fcg {

using namespace devscan;

namespace {

constexpr int kMaxMeshLevel = 4096;           // the host recursion's limit
constexpr uint16_t kSelfBit = kMeshSelfPair;  // frontier meta: self pass
constexpr uint16_t kLevelMask = 0x7fff;       // frontier meta: recursion level
constexpr int64_t kMaxFrontier = 1ll << 30;   // pairs held at once
constexpr int64_t kNoWait = 1 << 18;          // pairs up to which levels are launched without knowing their size
constexpr int kMaxGroup = 24;                 // levels launched at a time (the bound triples: at most 12)

static_assert(sizeof(Element) == 96, "element record layout");

// ---- FP32 pre-test of the mesh decision (fcg_mesh_decision), see pair32.cuh

// geometric normal (fcg_geo_normal) in FP32 and a bound on each component's
// distance to the FP64 path's value; false when a super node's Newell modulus
// is within rounding of the normalisation cut-off
__device__ __forceinline__ bool geo_normal32(const pair32::PairElement &e, float &x, float &y, float &z, float &err) {
    if (!(e.type & FCG_IS_SUPER_NODE)) {
        x = e.n[0]; y = e.n[1]; z = e.n[2];
        err = 0.0f;
        return true;
    }
    float n[3];
    n[0] = n[1] = n[2] = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; i++) {  // the float sums of fcg_newell_normal, same operations
        int j = i + 1 > 2 ? 0 : i + 1;
        const float *a = e.v + 3 * i, *b = e.v + 3 * j;
        n[0] += (a[1] - b[1]) * (a[2] + b[2]);
        n[1] += (a[2] - b[2]) * (a[0] + b[0]);
        n[2] += (a[0] - b[0]) * (a[1] + b[1]);
    }
    float m = sqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    const float cut = (float)FCG_PANEL_EPS;
    if (!(fabsf(m - cut) > 1e-5f * cut)) return false;
    if (m > cut) {
        x = n[0] / m; y = n[1] / m; z = n[2] / m;
        err = 16.0f * pair32::kU;  // unit components: a few roundings each
    } else {
        x = n[0]; y = n[1]; z = n[2];
        err = 0.0f;  // the same float sums, unnormalised
    }
    return true;
}

// fcg_mesh_decision in FP32: 1 / 2 refine (split the larger-area element),
// 0 no refinement (c1, c2 and their bounds e1, e2 are the pair's weights),
// -1 only the FP64 test can tell, -2 a near pair, left alone without `near`
__device__ __forceinline__ int mesh_decide32(pair32::PairElement &A, pair32::PairElement &B, bool near, bool selfc, float e, float mesh_curv, float inv_max_area,
                             float inv_max_side, float &c1, float &e1, float &c2, float &e2) {
    using namespace pair32;
    float dx = A.c[0] - B.c[0], dy = A.c[1] - B.c[1], dz = A.c[2] - B.c[2];  // fcg_fsub's float values
    float r = sqrtf(dx * dx + dy * dy + dz * dz);
    double rm = A.maxside > B.maxside ? A.maxside : B.maxside;
    float rho = r / (float)rm;
    if (!(r > 1e-10f) || !(fabsf(rho - 2.0f) > 1e-5f)) return -1;
    bool quad = rho < 2.0f;
    if (quad && !near) return -2;
    if (quad || (selfc && ((A.type | B.type) & FCG_IS_SUPER_NODE))) {
        A.vertices();
        B.vertices();
    }
    float cc = 1.0f, cc_err = 0.0f;
    if (selfc) {
        float ax, ay, az, ae, bx, by, bz, be;
        if (!geo_normal32(A, ax, ay, az, ae) || !geo_normal32(B, bx, by, bz, be)) return -1;
        float na = fabsf(ax) + fabsf(ay) + fabsf(az), nb = fabsf(bx) + fabsf(by) + fabsf(bz);
        float dot = ax * bx + ay * by + az * bz;
        float dot_err = ae * nb + be * na + 8.0f * kU * (na * nb);
        cc = (mesh_curv - 1.0f) * (dot + 1.0f) + 1.0f;
        cc_err = (mesh_curv - 1.0f) * dot_err + 8.0f * kU * fabsf(cc) + 8.0f * kU * fabsf(mesh_curv - 1.0f) * (fabsf(dot) + 1.0f);
        if (!(cc - cc_err > 0.0f)) return -1;
    }
    float w1, w1e, w2, w2e;
    if (!weight32(A, B, dx, dy, dz, r, quad, inv_max_area, inv_max_side, w1, w1e)) return -1;
    if (!weight32(B, A, -dx, -dy, -dz, r, quad, inv_max_area, inv_max_side, w2, w2e)) return -1;
    // c = w / cc with the bounds of both factors
    c1 = w1 / cc;
    c2 = w2 / cc;
    e1 = (w1e + c1 * cc_err) / (cc - cc_err) + 8.0f * kU * c1;
    e2 = (w2e + c2 * cc_err) / (cc - cc_err) + 8.0f * kU * c2;
    if (!isfinite(e1) || !isfinite(e2)) return -1;
    int t1 = side_test(c1, e1, e), t2 = side_test(c2, e2, e);
    if (t1 == 1 || t2 == 1) return A.area > B.area ? 1 : 2;
    if (t1 == 0 && t2 == 0) return 0;
    return -1;
}

// what the levels know of one another, on the device
struct LevelHead {
    unsigned long long n, ne;                        // frontier pairs, elements
    unsigned long long n_split, n_leaves, n_listed;  // pairs split, leaves bisected, pairs for the FP64 test
};

// a level's lists of split pairs (the side that splits in the sign of the
// first id), of bisected leaves and of pairs for the FP64 test
struct LevelLists {
    int2 *split_pairs;
    uint16_t *split_meta;
    int32_t *leaves, *listed;
};

// A warp's split pairs (f = 1 or 2: the pair splits its first or second
// element, a leaf when `leaf` is set) into the level's list; the first to
// split a leaf gives it the ids of its halves.
__device__ __forceinline__ void emit_splits(LevelHead *head, int64_t ne, int f, bool leaf, int2 pr, uint16_t m, Element *el, int *claim,
                                            const LevelLists &ls) {
    const unsigned split = __ballot_sync(0xffffffffu, f != 0);
    if (!split) return;
    const int x = f == 1 ? pr.x : pr.y;
    const bool mine = f && leaf && atomicExch(&claim[x], 1) == 0;
    const unsigned first = __ballot_sync(0xffffffffu, mine), below = (1u << (threadIdx.x & 31)) - 1u;
    const int64_t rs = warp_claim(&head->n_split, __popc(split)) + __popc(split & below);
    if (first) {
        const int64_t rl = warp_claim(&head->n_leaves, __popc(first)) + __popc(first & below);
        if (mine) {
            ls.leaves[rl] = x;
            el[x].left = (int32_t)(ne + 2 * rl);
            el[x].right = (int32_t)(ne + 2 * rl + 1);
        }
    }
    if (f) {
        ls.split_pairs[rs] = make_int2(f == 2 ? ~pr.x : pr.x, pr.y);
        ls.split_meta[rs] = m;
    }
}

// One level's decisions in FP32 where that is certain. Pairs the FP32 test
// cannot decide are listed for the FP64 test, and so are the kept pairs that
// may hold the largest weight of the model: a kept pair whose upper bound is
// below the largest lower bound already seen cannot (that pair's exact weight
// is at least its lower bound), so only pairs near the running maximum take
// the FP64 test for it. `lo_bits` holds that running lower bound (bits of a
// non-negative double). With pre32 unset every pair takes the FP64 test.
// A pair nearer than twice the larger side needs quadratures, some ten times
// the instructions of a far one, and one such lane holds its warp: where a warp
// has several rounds, near pairs wait in its queue until 32 of them run
// together (one round: at once, the queue would only add a round). Levels of
// 42 / 120 million pairs in all 2720 / 6335 -> 2063 / 4575 us with the 16-byte
// loads of PairElement (without the queue 2420 / 5880, the queue alone 2435 /
// 5320); a small level 11.7 -> 7.7. What is left is the FP64 pipe (areas and
// sides; 55 % active in the longest level) and latency at 24 warps an SM: 20 (no
// spills) 2277 / 5265, 32 2111 / 4504. Four pairs a lane with one claim
// (218 -> 300 us a level of 4M pairs) and one claim a CTA (2842 / 7243) were
// slower. A small level is bound by its launches: three kernels a level and a
// wait for the host every few levels, instead of nine and one each: a 528-panel
// model's refinement 1.74 -> 0.96 ms, its links 1.49 -> 0.90 ms.
__global__ void __launch_bounds__(128, 6) k_mesh_level(LevelHead *__restrict__ head, const int2 *__restrict__ pairs,
                                                       const uint16_t *__restrict__ meta, Element *el, int *claim, int pre32, float e,
                                                       float mesh_curv, float inv_max_area, float inv_max_side, const LevelLists ls,
                                                       unsigned long long *lo_bits, int *max_level, unsigned *too_deep) {
    __shared__ int32_t queue[4][64];
    const int64_t n = (int64_t)head->n, ne = (int64_t)head->ne, stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    int32_t *q = queue[threadIdx.x >> 5];
    const bool direct = n <= stride;  // a warp has one round at most
    int lvl_max = 0, waiting = 0;
    // whole warps stay in the loop (ballots below)
    for (int64_t next = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31);;) {
        const bool near = waiting >= 32 || (waiting > 0 && next >= n);
        if (!near && next >= n) break;
        int64_t i = n;
        if (near) {
            const int take = min(waiting, 32);
            waiting -= take;
            if (lane < take) i = q[waiting + lane];
        } else {
            i = next + lane;
            next += stride;
        }
        int f = 0;
        bool leaf = false;
        double lo = 0.0;
        int2 pr = make_int2(0, 0);
        uint16_t m = 0;
        if (i < n) {
            pr = pairs[i];
            m = meta[i];
            const int lvl = m & kLevelMask;
            lvl_max = max(lvl_max, lvl);
            if (lvl > kMaxMeshLevel) {
                atomicOr(too_deep, 1u);
            } else if (pre32) {
                pair32::PairElement A(el[pr.x]), B(el[pr.y]);
                float c1 = 0, e1 = 0, c2 = 0, e2 = 0;
                f = mesh_decide32(A, B, near || direct, (m & kSelfBit) != 0, e, mesh_curv, inv_max_area, inv_max_side, c1, e1, c2, e2);
                leaf = ((f == 1 ? A.type : B.type) & FCG_IS_LEAF) != 0;
                if (f == 0) {
                    // a kept pair: may its exact weight be the model's largest?
                    float hi = 0.0f, l = 0.0f;
                    if (!(A.type & FCG_IS_SUPER_NODE)) { hi = c1 + e1; l = c1 - e1; }
                    if (!(B.type & FCG_IS_SUPER_NODE)) { hi = fmaxf(hi, c2 + e2); l = fmaxf(l, c2 - e2); }
                    const double cur = __longlong_as_double((long long)*(volatile unsigned long long *)lo_bits);
                    if (hi > 0.0f && (double)hi >= cur) {
                        f = -1;
                        if (l > 0.0f) lo = (double)l;
                    }
                }
            } else {
                f = -1;
            }
        }
        const unsigned later = __ballot_sync(0xffffffffu, f == -2);  // none in a round from the queue
        if (f == -2) q[waiting + __popc(later & ((1u << lane) - 1u))] = (int32_t)i;
        waiting += __popc(later);
        __syncwarp();
        const unsigned listed = __ballot_sync(0xffffffffu, f == -1);
        if (listed) {
            const int64_t at = warp_claim(&head->n_listed, __popc(listed)) + __popc(listed & ((1u << lane) - 1u));
            if (f == -1) ls.listed[at] = (int32_t)i;
            for (int o = 16; o > 0; o >>= 1) lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            if (lane == 0 && lo > 0.0) atomicMax(lo_bits, (unsigned long long)__double_as_longlong(lo));
        }
        emit_splits(head, ne, max(f, 0), leaf, pr, m, el, claim, ls);
    }
    for (int o = 16; o > 0; o >>= 1) lvl_max = max(lvl_max, __shfl_xor_sync(0xffffffffu, lvl_max, o));
    if (lane == 0 && lvl_max) atomicMax(max_level, lvl_max);
}

// The FP64 test (the host builder's own code) of the level's listed pairs: the
// decision and, for kept pairs, the exact weights behind the model's largest.
// Two lanes a pair, one for each direction's weight (fcg_mesh_decision's, whose
// arithmetic does not change when the two elements swap places): most levels
// list few pairs, and the chain of one lane's FP64 instructions is what they
// wait for: 16.5 -> 10.1 us a level of a 528-panel model, 654 -> 392 in 25
// levels of 42 million pairs, 626 -> 371 in 29 of 120 million.
__global__ void __launch_bounds__(128) k_mesh_level64(LevelHead *__restrict__ head, const int2 *__restrict__ pairs,
                                                      const uint16_t *__restrict__ meta, Element *el, int *claim, double mesh_eps,
                                                      double mesh_curv, double max_side, double max_area, const LevelLists ls,
                                                      unsigned long long *max_eps_bits) {
    const int64_t cnt = (int64_t)head->n_listed, ne = (int64_t)head->ne;
    // largest weight of the pairs this thread kept, as the bits of a
    // non-negative double (their order is the values' order)
    unsigned long long eps_max = 0;
    const int odd = threadIdx.x & 1;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t - (threadIdx.x & 31) < 2 * cnt; t += (int64_t)gridDim.x * blockDim.x) {
        int f = 0;
        bool leaf = false;
        int2 pr = make_int2(0, 0);
        uint16_t m = 0;
        double c = 0.0;
        if (t < 2 * cnt) {
            const int64_t i = ls.listed[t >> 1];
            pr = pairs[i];
            m = meta[i];
            const Element &A = el[odd ? pr.y : pr.x], &B = el[odd ? pr.x : pr.y];
            fcg_d3 dist;
            double rdist, rmax;
            fcg_pair_span(A, B, &dist, &rdist, &rmax);
            c = fcg_one_way(A, B, dist, rdist, rmax, fcg_curv_coeff(A, B, (m & kSelfBit) != 0, mesh_curv), max_side, max_area);
        }
        const double c2 = __shfl_xor_sync(0xffffffffu, c, 1);
        if (t < 2 * cnt) {
            if (c > mesh_eps || c2 > mesh_eps) {
                if (!odd) {
                    f = el[pr.x].area > el[pr.y].area ? 1 : 2;
                    leaf = (el[f == 1 ? pr.x : pr.y].type & FCG_IS_LEAF) != 0;
                }
            } else if (!(el[odd ? pr.y : pr.x].type & FCG_IS_SUPER_NODE) && c == c) {
                eps_max = max(eps_max, (unsigned long long)__double_as_longlong(c));
            }
        }
        emit_splits(head, ne, f, leaf, pr, m, el, claim, ls);
    }
    for (int o = 16; o > 0; o >>= 1) eps_max = max(eps_max, __shfl_xor_sync(0xffffffffu, eps_max, o));
    if ((threadIdx.x & 31) == 0 && eps_max) atomicMax(max_eps_bits, eps_max);
}

// The next frontier: the children of every split pair (2 r, 2 r + 1), then the
// halves of every bisected leaf, which are made here; and the next level's head.
__global__ void __launch_bounds__(256) k_mesh_grow(LevelHead *__restrict__ head, Element *el, int32_t *depth,
                                                   const LevelLists ls, int2 *__restrict__ next, uint16_t *__restrict__ next_meta) {
    const int64_t ns = (int64_t)head->n_split, nlv = (int64_t)head->n_leaves, ne = (int64_t)head->ne;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        head[1].n = (unsigned long long)(2 * ns + nlv);
        head[1].ne = (unsigned long long)(ne + 2 * nlv);
    }
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ns + nlv; t += (int64_t)gridDim.x * blockDim.x) {
        if (t < ns) {
            int2 p = ls.split_pairs[t];
            const bool second = p.x < 0;
            if (second) p.x = ~p.x;
            int2 c0 = p, c1 = p;
            if (second) {
                c0.y = el[p.y].left;
                c1.y = el[p.y].right;
            } else {
                c0.x = el[p.x].left;
                c1.x = el[p.x].right;
            }
            const uint16_t m = ls.split_meta[t];
            const uint16_t m1 = (uint16_t)((m & kSelfBit) | (uint16_t)min((m & kLevelMask) + 1, (int)kLevelMask));
            next[2 * t] = c0;
            next[2 * t + 1] = c1;
            next_meta[2 * t] = m1;
            next_meta[2 * t + 1] = m1;
        } else {
            const int64_t k = t - ns;
            const int32_t x = ls.leaves[k], l = (int32_t)(ne + 2 * k), r = l + 1;
            Element Lc, Rc;
            fcg_subdivide(el[x], Lc, Rc);
            el[l] = Lc;
            el[r] = Rc;
            const int32_t d = depth[x];
            depth[l] = d + 1;
            depth[r] = d + 1;
            el[x].type = (uint8_t)(el[x].type & ~FCG_IS_LEAF);
            next[2 * ns + k] = make_int2(l, r);
            next_meta[2 * ns + k] = (uint16_t)(kSelfBit | (uint16_t)min(d + 2, (int)kLevelMask));
        }
    }
}

}  // namespace

#define MB_CK(x)                                                                                     \
    do {                                                                                             \
        cudaError_t e_ = (x);                                                                        \
        if (e_ != cudaSuccess) {                                                                     \
            err = std::string("device mesh refinement: ") + cudaGetErrorString(e_);                  \
            cudaGetLastError();                                                                      \
            return e_ == cudaErrorMemoryAllocation ? FCG_OUT_OF_MEMORY : FCG_DEVICE_ERROR;           \
        }                                                                                            \
    } while (0)

int mesh_refine_device(DeviceContext &ctx, std::vector<Element> &el, const std::vector<int32_t> &depth,
                       const std::vector<int32_t> &root_a, const std::vector<int32_t> &root_b,
                       const std::vector<uint16_t> &root_meta, double mesh_eps, double mesh_curv, double max_side,
                       double max_area, int64_t keep_from, std::shared_ptr<Element> &kept, int64_t &n_kept,
                       double &max_mesh_eps, int &max_level, std::string &err) {
    MB_CK(cudaSetDevice(ctx.device));
    Bufs B;
    MB_CK(cudaStreamCreateWithFlags(&B.s, cudaStreamNonBlocking));
    cudaStream_t s = B.s;
    const int sms = ctx.sm_count > 0 ? ctx.sm_count : 1;
    const bool trace = getenv("FCG_TRACE") != nullptr;
    // FCG_MESH_FP64=1: every pair through the FP64 test (no FP32 pre-test)
    const bool fp64_only = getenv("FCG_MESH_FP64") != nullptr;
    int64_t ne = (int64_t)el.size();
    int64_t cap = std::max<int64_t>(2 * ne, ne + (1 << 20));
    Element *d_el;
    int32_t *d_depth;
    int *d_claim;
    LevelHead *d_head;
    unsigned long long *d_max_eps, *d_lo_bits;
    int *d_max_level;
    unsigned *d_too_deep;
    MB_CK(B.alloc(&d_el, (size_t)cap));
    MB_CK(B.alloc(&d_depth, (size_t)cap));
    MB_CK(B.alloc(&d_claim, (size_t)cap));
    MB_CK(B.alloc(&d_head, (size_t)kMaxGroup + 1));
    MB_CK(B.alloc(&d_max_eps, 1));
    MB_CK(B.alloc(&d_lo_bits, 1));
    MB_CK(B.alloc(&d_max_level, 1));
    MB_CK(B.alloc(&d_too_deep, 1));
    MB_CK(cudaMemcpyAsync(d_el, el.data(), (size_t)ne * sizeof(Element), cudaMemcpyHostToDevice, s));
    MB_CK(cudaMemcpyAsync(d_depth, depth.data(), (size_t)ne * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    MB_CK(cudaMemsetAsync(d_claim, 0, (size_t)cap * sizeof(int), s));
    MB_CK(cudaMemsetAsync(d_max_eps, 0, sizeof(unsigned long long), s));
    MB_CK(cudaMemsetAsync(d_lo_bits, 0, sizeof(unsigned long long), s));
    MB_CK(cudaMemsetAsync(d_max_level, 0, sizeof(int), s));
    MB_CK(cudaMemsetAsync(d_too_deep, 0, sizeof(unsigned), s));

    int64_t n = (int64_t)root_a.size();
    // two frontiers, and the split pairs and bisected leaves of a level
    int2 *pairs[2] = {nullptr, nullptr};
    uint16_t *meta[2] = {nullptr, nullptr};
    LevelLists ls = {nullptr, nullptr, nullptr, nullptr};
    int64_t room[2] = {0, 0}, list_room = 0;
    auto frontier = [&](int f, int64_t need) -> cudaError_t {
        if (need <= room[f]) return cudaSuccess;
        B.release(pairs[f]);
        B.release(meta[f]);
        room[f] = std::max<int64_t>(need, 1 << 16);
        cudaError_t e = B.alloc(&pairs[f], (size_t)room[f]);
        return e == cudaSuccess ? B.alloc(&meta[f], (size_t)room[f]) : e;
    };
    auto lists = [&](int64_t need) -> cudaError_t {
        if (need <= list_room) return cudaSuccess;
        B.release(ls.split_pairs);
        B.release(ls.split_meta);
        B.release(ls.leaves);
        B.release(ls.listed);
        list_room = std::max<int64_t>(need, 1 << 16);
        cudaError_t e = B.alloc(&ls.split_pairs, (size_t)list_room);
        if (e == cudaSuccess) e = B.alloc(&ls.split_meta, (size_t)list_room);
        if (e == cudaSuccess) e = B.alloc(&ls.leaves, (size_t)list_room);
        return e == cudaSuccess ? B.alloc(&ls.listed, (size_t)list_room) : e;
    };
    // room for elements: the arrays grow, keeping the first `have`
    auto elements = [&](int64_t have, int64_t need) -> cudaError_t {
        if (need <= cap) return cudaSuccess;
        const int64_t ncap = std::max<int64_t>(2 * cap, need);
        Element *el2;
        int32_t *depth2;
        int *claim2;
        cudaError_t e = B.alloc(&el2, (size_t)ncap);
        if (e == cudaSuccess) e = B.alloc(&depth2, (size_t)ncap);
        if (e == cudaSuccess) e = B.alloc(&claim2, (size_t)ncap);
        if (e == cudaSuccess) e = cudaMemcpyAsync(el2, d_el, (size_t)have * sizeof(Element), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(depth2, d_depth, (size_t)have * sizeof(int32_t), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(claim2, d_claim, (size_t)have * sizeof(int), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(claim2 + have, 0, (size_t)(ncap - have) * sizeof(int), s);
        if (e != cudaSuccess) return e;
        B.release(d_el);
        B.release(d_depth);
        B.release(d_claim);
        d_el = el2;
        d_depth = depth2;
        d_claim = claim2;
        cap = ncap;
        return cudaSuccess;
    };
    {
        std::vector<int2> h((size_t)n);
        for (int64_t i = 0; i < n; i++) h[(size_t)i] = make_int2(root_a[(size_t)i], root_b[(size_t)i]);
        MB_CK(frontier(0, n));
        MB_CK(cudaMemcpyAsync(pairs[0], h.data(), (size_t)n * sizeof(int2), cudaMemcpyHostToDevice, s));
        MB_CK(cudaMemcpyAsync(meta[0], root_meta.data(), (size_t)n * sizeof(uint16_t), cudaMemcpyHostToDevice, s));
        MB_CK(cudaStreamSynchronize(s));  // the host vector goes out of scope
    }
    long long tests = 0, steps = 0;
    int cur = 0;
    auto grid_of = [&](int64_t items, int per) {
        return (unsigned)std::max<int64_t>(std::min<int64_t>((items + per - 1) / per, (int64_t)sms * 16), 1);
    };
    while (n > 0) {
        // levels are launched without waiting while the bound on their size
        // (every pair split, each by a leaf's bisection: three next pairs, two
        // elements) stays below kNoWait; above it the host waits for a level's
        // counts before it makes room for the next
        std::vector<LevelHead> heads(kMaxGroup + 1, LevelHead{0, 0, 0, 0, 0});
        heads[0].n = (unsigned long long)n;
        heads[0].ne = (unsigned long long)ne;
        MB_CK(cudaMemcpyAsync(d_head, heads.data(), heads.size() * sizeof(LevelHead), cudaMemcpyHostToDevice, s));
        int64_t bound = n, ne_bound = ne;
        int g = 0;
        bool waited = false;
        do {
            LevelHead *head = d_head + g;
            MB_CK(lists(bound));
            k_mesh_level<<<grid_of(bound, 128), 128, 0, s>>>(head, pairs[cur], meta[cur], d_el, d_claim,
                                                                       fp64_only ? 0 : 1, (float)mesh_eps, (float)mesh_curv,
                                                                       (float)(1.0 / max_area), (float)(1.0 / max_side), ls,
                                                                       d_lo_bits, d_max_level, d_too_deep);
            k_mesh_level64<<<grid_of(bound, 128), 128, 0, s>>>(head, pairs[cur], meta[cur], d_el, d_claim, mesh_eps, mesh_curv,
                                                              max_side, max_area, ls, d_max_eps);
            int64_t next_bound = 3 * bound, grow = 2 * bound;
            if (next_bound > kNoWait) {
                unsigned deep = 0;
                MB_CK(cudaMemcpyAsync(heads.data(), d_head, (size_t)(g + 1) * sizeof(LevelHead), cudaMemcpyDeviceToHost, s));
                MB_CK(cudaMemcpyAsync(&deep, d_too_deep, sizeof deep, cudaMemcpyDeviceToHost, s));
                MB_CK(cudaStreamSynchronize(s));
                const LevelHead &h = heads[(size_t)g];
                waited = true;
                next_bound = (int64_t)(2 * h.n_split + h.n_leaves);
                grow = (int64_t)(2 * h.n_leaves);
                ne_bound = (int64_t)h.ne;
                if (deep || next_bound > kMaxFrontier || ne_bound + grow > 0x7fffffffLL) {
                    err = "mesh refinement recursion too deep (touching or overlapping panels?)";
                    return FCG_GENERIC_ERROR;
                }
            }
            MB_CK(frontier(cur ^ 1, next_bound));
            MB_CK(elements(ne_bound, ne_bound + grow));
            k_mesh_grow<<<grid_of(waited ? std::max<int64_t>(next_bound, 1) : 2 * bound, 256), 256, 0, s>>>(
                head, d_el, d_depth, ls, pairs[cur ^ 1], meta[cur ^ 1]);
            MB_CK(cudaGetLastError());
            cur ^= 1;
            bound = next_bound;
            ne_bound += grow;
            steps++;
            g++;
        } while (!waited && bound <= kNoWait && g < kMaxGroup);
        heads.resize((size_t)g + 1);
        if (waited) {
            // the last level's counts are known, and with them the next's size: one
            // wait a level, not two (180 thousand elements 5.4 -> 4.2 ms)
            heads.back().n = (unsigned long long)bound;
            heads.back().ne = (unsigned long long)ne_bound;
        } else {
            unsigned deep = 0;
            MB_CK(cudaMemcpyAsync(heads.data(), d_head, heads.size() * sizeof(LevelHead), cudaMemcpyDeviceToHost, s));
            MB_CK(cudaMemcpyAsync(&deep, d_too_deep, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
            MB_CK(cudaStreamSynchronize(s));
            if (deep) {
                err = "mesh refinement recursion too deep (touching or overlapping panels?)";
                return FCG_GENERIC_ERROR;
            }
        }
        for (size_t q = 0; q + 1 < heads.size(); q++) tests += (long long)heads[q].n;
        n = (int64_t)heads.back().n;
        ne = (int64_t)heads.back().ne;
    }
    unsigned long long eps_bits = 0;
    MB_CK(cudaMemcpyAsync(&eps_bits, d_max_eps, sizeof(eps_bits), cudaMemcpyDeviceToHost, s));
    MB_CK(cudaMemcpyAsync(&max_level, d_max_level, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (ne >= keep_from) {
        el.clear();
        // to its size: the room for growth, at least 2^20 elements, would stay
        // through the flattening and the links, whose memory is the build's peak
        for (int f = 0; f < 2; f++) {
            B.release(pairs[f]);
            B.release(meta[f]);
        }
        B.release(ls.split_pairs);
        B.release(ls.split_meta);
        B.release(ls.leaves);
        B.release(ls.listed);
        B.release(d_depth);
        B.release(d_claim);
        Element *fit;
        MB_CK(B.alloc(&fit, (size_t)ne));
        MB_CK(cudaMemcpyAsync(fit, d_el, (size_t)ne * sizeof(Element), cudaMemcpyDeviceToDevice, s));
        B.release(d_el);
        d_el = fit;
    } else {
        el.resize((size_t)ne);
        MB_CK(cudaMemcpyAsync(el.data(), d_el, (size_t)ne * sizeof(Element), cudaMemcpyDeviceToHost, s));
    }
    MB_CK(cudaStreamSynchronize(s));
    if (ne >= keep_from) {
        kept = B.hand_over(d_el);
        n_kept = ne;
    }
    double me;
    memcpy(&me, &eps_bits, sizeof me);
    max_mesh_eps = me;
    if (trace) fprintf(stderr, "[fcg mesh] %lld steps, %lld pair tests, %lld elements\n", steps, tests, (long long)ne);
    return FCG_NORMAL_END;
}

}  // namespace fcg
