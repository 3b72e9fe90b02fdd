// Flattening of a refined element hierarchy on the GPU: the node order of
// CAutoRefine::RecurseIndex (Solver/Autorefine.cpp:1173-1220; every
// conductor's tree in post-order, conductors in solver order), the node
// arrays in that order and the root pairs of the link traversal.
//
// Every element's place follows from the leaf counts on the way to its
// conductor's root alone: a tree with m leaves has 2 m - 1 nodes and m - 1
// internal ones, so the nodes, leaves and internal nodes (the self pairs'
// pre-order) before a subtree are sums over the left siblings met on the way
// up, and a sibling's count is the parent's less the node's own. Three
// kernels, none of them a level at a time:
//   parents  the parent of every element, and which side it hangs on
//   leaves   leaf counts: a thread per leaf climbs, the second to arrive at a
//            node adds up its children and goes on
//   place    a thread per element climbs to its root and writes where it goes
// and one that writes the node arrays, a thread per node. All are bound by
// the latency of a climb (some 25 levels of L2 reads) and then by the 200
// bytes a node that are read and written.
//
// 180 / 323 thousand elements: walks, numbering, root pairs and arrays took
// 7.0 / 11.0 ms on the host; here they take 0.20 / 0.21 ms, or 1.1 / 1.7 ms
// with the node arrays' download. The elements stay on the device between
// refinement and links (0.6 / 1.0 ms less), and a problem made from node
// arrays in device memory has no upload (1.1 / 1.9 -> 0.3 / 0.4 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "fc_potential.h"
#include "fcg_internal.hpp"
#include "scan.cuh"
#include "../host/model.hpp"

namespace fcg {

using namespace devscan;

namespace {

static_assert(sizeof(Element) == 96, "element record layout");

constexpr uint32_t kNoParent = 0xffffffffu;  // else 2 parent + (1 for a right child)

struct NodeArrays {
    uint8_t *type, *maxside_idx, *leaf_diel;
    int32_t *left, *right, *cond, *leaf_node;
    int64_t *leaf_first, *leaf_count;
    float *vert, *cent, *norm;
    double *area, *maxside;
};

__global__ void k_tree_parents(int64_t ne, const Element *__restrict__ el, uint32_t *parent) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ne; i += (int64_t)gridDim.x * blockDim.x) {
        if (el[i].type & FCG_IS_LEAF) continue;
        parent[el[i].left] = 2u * (uint32_t)i;
        parent[el[i].right] = 2u * (uint32_t)i + 1u;
    }
}

__global__ void k_tree_leaves(int64_t ne, const Element *__restrict__ el, const uint32_t *__restrict__ parent, int *arrived,
                              int32_t *leaves) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ne; i += (int64_t)gridDim.x * blockDim.x) {
        if (!(el[i].type & FCG_IS_LEAF)) continue;
        __stcg(leaves + i, 1);
        for (uint32_t p = parent[i]; p != kNoParent; p = parent[p >> 1]) {
            __threadfence();
            if (atomicAdd(arrived + (p >> 1), 1) == 0) break;  // the sibling's climber goes on
            __threadfence();
            const Element &e = el[p >> 1];
            __stcg(leaves + (p >> 1), __ldcg(leaves + e.left) + __ldcg(leaves + e.right));
        }
    }
}

__global__ void k_tree_tops(int nc, const int32_t *__restrict__ tops, const int32_t *__restrict__ leaves, int32_t *top_of,
                            int32_t *cnt) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        top_of[tops[k]] = k;
        cnt[k] = leaves[tops[k]];
    }
}

// top_of[id] = conductor of a root element, -1 elsewhere; off[3 k ..] = first
// node, first leaf and first root pair of conductor k
__global__ void k_tree_place(int64_t ne, int nc, const Element *__restrict__ el, const uint32_t *__restrict__ parent,
                             const int32_t *__restrict__ leaves, const int32_t *__restrict__ top_of,
                             const int64_t *__restrict__ off, int32_t *node_of, int32_t *post, NodeArrays a, int2 *roots,
                             uint16_t *root_level, int *max_depth) {
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < ne; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        int depth = 0;
        if (i < ne) {
            const int32_t m = leaves[i];
            int32_t x = (int32_t)i, mx = m, leaf0 = 0, inner0 = 0;
            int64_t node0 = 0;
            for (uint32_t p = parent[x]; p != kNoParent; p = parent[x]) {
                x = (int32_t)(p >> 1);
                const int32_t mp = leaves[x];
                if (p & 1u) {
                    leaf0 += mp - mx;
                    inner0 += mp - mx - 1;
                    node0 += 2 * (int64_t)(mp - mx) - 1;
                }
                inner0++;
                depth++;
                mx = mp;
            }
            const int k = top_of[x];
            if (k < 0) {  // in no conductor's tree
                node_of[i] = -1;
                depth = 0;
            } else {
                const int64_t node = off[3 * k] + node0 + 2 * (int64_t)m - 2;
                node_of[i] = (int32_t)node;
                post[node] = (int32_t)i;
                a.cond[node] = k;
                a.leaf_first[node] = off[3 * k + 1] + leaf0;
                a.leaf_count[node] = m;
                const Element &e = el[i];
                if (e.type & FCG_IS_LEAF) {
                    a.left[node] = a.right[node] = -1;
                } else {
                    a.right[node] = (int32_t)(node - 1);
                    a.left[node] = (int32_t)(node - 2 * (int64_t)leaves[e.right]);
                    // after the conductor's pairs with the later ones, in pre-order
                    const int64_t r = off[3 * k + 2] + (nc - 1 - k) + inner0;
                    roots[r] = make_int2(e.left, e.right);
                    root_level[r] = (uint16_t)min(depth + 2, 0xffff);
                }
            }
        }
        depth = __reduce_max_sync(0xffffffffu, depth);
        if ((threadIdx.x & 31) == 0 && depth > 0) atomicMax(max_depth, depth);
    }
}

// the conductors' pairs (k, j > k), at recursion level 1
__global__ void k_tree_pairs(int nc, const int32_t *__restrict__ tops, const int64_t *__restrict__ off, int2 *roots,
                             uint16_t *root_level) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (int64_t)nc * nc; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / nc), j = (int)(t % nc);
        if (j <= k) continue;
        const int64_t r = off[3 * k + 2] + (j - k - 1);
        roots[r] = make_int2(tops[k], tops[j]);
        root_level[r] = 1;
    }
}

__global__ void k_tree_nodes(int64_t n_nodes, const Element *__restrict__ el, const int32_t *__restrict__ post, NodeArrays a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_nodes; i += (int64_t)gridDim.x * blockDim.x) {
        const Element e = el[post[i]];
        for (int c = 0; c < 9; c++) a.vert[9 * i + c] = e.v[c];
        for (int c = 0; c < 3; c++) a.cent[3 * i + c] = e.c[c];
        for (int c = 0; c < 3; c++) a.norm[3 * i + c] = e.n[c];
        a.type[i] = e.type;
        a.area[i] = e.area;
        a.maxside[i] = e.maxside;
        a.maxside_idx[i] = e.maxside_idx;
        if (e.type & FCG_IS_LEAF) {
            const int64_t j = a.leaf_first[i];
            a.leaf_node[j] = (int32_t)i;
            a.leaf_diel[j] = (e.type & FCG_IS_DIEL) ? 0 : e.diel;
        }
    }
}

}  // namespace

#define TF_CK(x)                                                                                     \
    do {                                                                                             \
        cudaError_t e_ = (x);                                                                        \
        if (e_ != cudaSuccess) {                                                                     \
            err = std::string("device model layout: ") + cudaGetErrorString(e_);                     \
            cudaGetLastError();                                                                      \
            return e_ == cudaErrorMemoryAllocation ? FCG_OUT_OF_MEMORY : FCG_DEVICE_ERROR;           \
        }                                                                                            \
    } while (0)

int tree_flatten_device(DeviceContext &ctx, const Element *d_el, int64_t ne, const std::vector<int32_t> &tops, bool keep_nodes,
                        Model &M, std::vector<int64_t> &cond_leaves, LinkRoots &out, int &max_depth, std::string &err) {
    TF_CK(cudaSetDevice(ctx.device));
    Bufs B;
    TF_CK(cudaStreamCreateWithFlags(&B.s, cudaStreamNonBlocking));
    cudaStream_t s = B.s;
    const int sms = ctx.sm_count > 0 ? ctx.sm_count : 1;
    const int nc = (int)tops.size();
    uint32_t *d_parent;
    int *d_arrived, *d_max_depth;
    int32_t *d_leaves, *d_top_of, *d_tops, *d_cnt;
    int64_t *d_off;
    TF_CK(B.alloc(&d_parent, (size_t)ne));
    TF_CK(B.alloc(&d_arrived, (size_t)ne));
    TF_CK(B.alloc(&d_leaves, (size_t)ne));
    TF_CK(B.alloc(&d_top_of, (size_t)ne));
    TF_CK(B.alloc(&d_tops, (size_t)nc));
    TF_CK(B.alloc(&d_cnt, (size_t)nc));
    TF_CK(B.alloc(&d_off, 3 * (size_t)nc));
    TF_CK(B.alloc(&d_max_depth, 1));
    TF_CK(cudaMemsetAsync(d_parent, 0xff, (size_t)ne * sizeof(uint32_t), s));
    TF_CK(cudaMemsetAsync(d_arrived, 0, (size_t)ne * sizeof(int), s));
    TF_CK(cudaMemsetAsync(d_top_of, 0xff, (size_t)ne * sizeof(int32_t), s));
    TF_CK(cudaMemsetAsync(d_max_depth, 0, sizeof(int), s));
    TF_CK(cudaMemcpyAsync(d_tops, tops.data(), (size_t)nc * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    const unsigned ge = grid_stride(ne, sms), gc = grid_stride(nc, sms);
    k_tree_parents<<<ge, 256, 0, s>>>(ne, d_el, d_parent);
    k_tree_leaves<<<ge, 256, 0, s>>>(ne, d_el, d_parent, d_arrived, d_leaves);
    k_tree_tops<<<gc, 256, 0, s>>>(nc, d_tops, d_leaves, d_top_of, d_cnt);
    TF_CK(cudaGetLastError());
    std::vector<int32_t> cnt((size_t)nc);
    TF_CK(cudaMemcpyAsync(cnt.data(), d_cnt, (size_t)nc * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    TF_CK(cudaStreamSynchronize(s));

    std::vector<int64_t> off(3 * (size_t)nc);
    int64_t Nn = 0, Np = 0, nr = 0;
    cond_leaves.assign((size_t)nc, 0);
    for (int k = 0; k < nc; k++) {
        off[3 * (size_t)k] = Nn;
        off[3 * (size_t)k + 1] = Np;
        off[3 * (size_t)k + 2] = nr;
        cond_leaves[(size_t)k] = cnt[(size_t)k];
        Nn += 2 * (int64_t)cnt[(size_t)k] - 1;
        Np += cnt[(size_t)k];
        nr += (nc - 1 - k) + (int64_t)cnt[(size_t)k] - 1;
    }
    if (Nn > 0x7fffffffLL) {
        err = "model too large for 32-bit link indices";
        return FCG_OUT_OF_MEMORY;
    }
    NodeArrays a;
    int32_t *d_node_of, *d_post;
    int2 *d_roots;
    uint16_t *d_level;
    const size_t nn = (size_t)Nn, np = (size_t)Np;
    TF_CK(B.alloc(&d_node_of, (size_t)ne));
    TF_CK(B.alloc(&d_post, nn));
    TF_CK(B.alloc(&d_roots, (size_t)nr));
    TF_CK(B.alloc(&d_level, (size_t)nr));
    TF_CK(B.alloc(&a.type, nn));
    TF_CK(B.alloc(&a.maxside_idx, nn));
    TF_CK(B.alloc(&a.leaf_diel, np));
    TF_CK(B.alloc(&a.left, nn));
    TF_CK(B.alloc(&a.right, nn));
    TF_CK(B.alloc(&a.cond, nn));
    TF_CK(B.alloc(&a.leaf_node, np));
    TF_CK(B.alloc(&a.leaf_first, nn));
    TF_CK(B.alloc(&a.leaf_count, nn));
    TF_CK(B.alloc(&a.vert, 9 * nn));
    TF_CK(B.alloc(&a.cent, 3 * nn));
    TF_CK(B.alloc(&a.norm, 3 * nn));
    TF_CK(B.alloc(&a.area, nn));
    TF_CK(B.alloc(&a.maxside, nn));
    TF_CK(cudaMemcpyAsync(d_off, off.data(), off.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s));
    k_tree_place<<<ge, 256, 0, s>>>(ne, nc, d_el, d_parent, d_leaves, d_top_of, d_off, d_node_of, d_post, a, d_roots, d_level,
                                    d_max_depth);
    k_tree_pairs<<<grid_stride((int64_t)nc * nc, sms), 256, 0, s>>>(nc, d_tops, d_off, d_roots, d_level);
    k_tree_nodes<<<grid_stride(Nn, sms), 256, 0, s>>>(Nn, d_el, d_post, a);
    TF_CK(cudaGetLastError());

    M.n_nodes = Nn;
    M.n_panels = Np;
    if (!keep_nodes) {  // the vectors are made while the kernels run
        auto download = [&](auto &v, const auto *d, size_t n) -> cudaError_t {
            v.resize(n);
            return cudaMemcpyAsync(v.data(), d, n * sizeof(*d), cudaMemcpyDeviceToHost, s);
        };
        TF_CK(download(M.type, a.type, nn));
        TF_CK(download(M.maxside_idx, a.maxside_idx, nn));
        TF_CK(download(M.leaf_diel, a.leaf_diel, np));
        TF_CK(download(M.left, a.left, nn));
        TF_CK(download(M.right, a.right, nn));
        TF_CK(download(M.cond, a.cond, nn));
        TF_CK(download(M.leaf_node, a.leaf_node, np));
        TF_CK(download(M.leaf_first, a.leaf_first, nn));
        TF_CK(download(M.leaf_count, a.leaf_count, nn));
        TF_CK(download(M.vert, a.vert, 9 * nn));
        TF_CK(download(M.cent, a.cent, 3 * nn));
        TF_CK(download(M.norm, a.norm, 3 * nn));
        TF_CK(download(M.area, a.area, nn));
        TF_CK(download(M.maxside, a.maxside, nn));
    }
    TF_CK(cudaMemcpyAsync(&max_depth, d_max_depth, sizeof(int), cudaMemcpyDeviceToHost, s));
    TF_CK(cudaStreamSynchronize(s));
    if (keep_nodes) {
        std::unique_ptr<DeviceNodes> d(new DeviceNodes());
        auto keep = [&](auto *q) {
            d->owned.push_back(B.hand_over(q));
            return q;
        };
        d->type = keep(a.type);
        d->leaf_diel = keep(a.leaf_diel);
        d->left = keep(a.left);
        d->right = keep(a.right);
        d->leaf_first = keep(a.leaf_first);
        d->leaf_count = keep(a.leaf_count);
        d->vert = keep(a.vert);
        d->cent = keep(a.cent);
        d->norm = keep(a.norm);
        d->area = keep(a.area);
        d->maxside = keep(a.maxside);
        M.d_nodes = std::move(d);
    }
    out.n = nr;
    out.pairs = B.hand_over((int32_t *)d_roots);
    out.level = B.hand_over(d_level);
    out.node_of = B.hand_over(d_node_of);
    return FCG_NORMAL_END;
}

int tree_nodes_to_host(DeviceContext &ctx, Model &M, std::string &err) {
    TF_CK(cudaSetDevice(ctx.device));
    Bufs B;  // its stream
    TF_CK(cudaStreamCreateWithFlags(&B.s, cudaStreamNonBlocking));
    const DeviceNodes &d = *M.d_nodes;
    const size_t nn = (size_t)M.n_nodes, np = (size_t)M.n_panels;
    auto download = [&](auto &v, const auto *q, size_t n) -> cudaError_t {
        v.resize(n);
        return cudaMemcpyAsync(v.data(), q, n * sizeof(*q), cudaMemcpyDeviceToHost, B.s);
    };
    TF_CK(download(M.type, d.type, nn));
    TF_CK(download(M.leaf_diel, d.leaf_diel, np));
    TF_CK(download(M.left, d.left, nn));
    TF_CK(download(M.right, d.right, nn));
    TF_CK(download(M.leaf_first, d.leaf_first, nn));
    TF_CK(download(M.leaf_count, d.leaf_count, nn));
    TF_CK(download(M.vert, d.vert, 9 * nn));
    TF_CK(download(M.cent, d.cent, 3 * nn));
    TF_CK(download(M.norm, d.norm, 3 * nn));
    TF_CK(download(M.area, d.area, nn));
    TF_CK(download(M.maxside, d.maxside, nn));
    TF_CK(cudaStreamSynchronize(B.s));
    M.d_nodes.reset();
    return FCG_NORMAL_END;
}

}  // namespace fcg
