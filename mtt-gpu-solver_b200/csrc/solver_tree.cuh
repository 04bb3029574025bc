// solver_tree.cuh — the arithmetic of the CFR sweeps on float4 hand groups and
// the whole-tree sweep kernel, shared by the heads-up and four-player solvers.
#pragma once
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>
#include <system_error>
#include <thread>
#include <vector>

#include "mtt_bulk.cuh"
#include "mtt_common.h"

namespace mtt {

__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) {
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
// Starts a fetch of the line holding p into L2 (no register is written, so
// every row of a work item can be requested before its first use).
__device__ __forceinline__ void pf_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
}

__device__ __forceinline__ float4 max04(float4 a) {
    return make_float4(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f), fmaxf(a.z, 0.f), fmaxf(a.w, 0.f));
}
// Regret matching: pos / sum, or uniform where nothing is positive.  A zero
// numerator would take the division's long special-case path, and under CFR+
// a large share of the regrets is exactly 0, so those skip the division (the
// quotient is 0 either way).  rm1 divides in line with the zeros replaced,
// rm1b branches around the division: on the 1,024-subgame river batch the
// forward levels took 224 -> 167 us (175 with rm1b) and the backward levels
// 566 -> 515 us (543 with rm1, whose temporaries spill there).
__device__ __forceinline__ float rm1(float pos, float sum, float invA) {
    const bool some = sum > 1e-7f, in = pos > 0.f;
    const float d = some ? sum : 1.f;
    const float q = __fdiv_rn(in ? pos : d, d);
    return some ? (in ? q : 0.f) : invA;
}
__device__ __forceinline__ float rm1b(float pos, float sum, float invA) {
    float q = sum > 1e-7f ? 0.f : invA;
    if (sum > 1e-7f && pos > 0.f) q = __fdiv_rn(pos, sum);
    return q;
}
__device__ __forceinline__ float4 rm4(float4 pos, float4 sum, float invA) {
    return make_float4(rm1(pos.x, sum.x, invA), rm1(pos.y, sum.y, invA), rm1(pos.z, sum.z, invA),
                       rm1(pos.w, sum.w, invA));
}
__device__ __forceinline__ float4 rm4b(float4 pos, float4 sum, float invA) {
    return make_float4(rm1b(pos.x, sum.x, invA), rm1b(pos.y, sum.y, invA), rm1b(pos.z, sum.z, invA),
                       rm1b(pos.w, sum.w, invA));
}
__device__ __forceinline__ float4 fma4(float4 a, float4 b, float4 c) {
    return make_float4(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y), __fmaf_rn(a.z, b.z, c.z),
                       __fmaf_rn(a.w, b.w, c.w));
}
__device__ __forceinline__ float cfrplus1(float r, float inst) { return fmaxf(0.0f, __fadd_rn(r, inst)); }
__device__ __forceinline__ float dcfr1(float r, float inst, float dpos, float dneg) {
    return __fadd_rn(__fmul_rn(r, r > 0.0f ? dpos : dneg), inst);
}

// ------------------------------------------------------------- whole-tree sweeps
// Between two terminal passes every value of a hand depends on that hand
// alone: its counterfactual values come up the tree from its own terminals,
// its regrets and strategy follow, and its reach goes down the tree again.  So
// where a subgame deals no card and its tree is small enough, one CTA takes
// one player's slice of 4 to 32 hands through the whole tree: it stages the
// slice's regret and strategy-sum rows, terminal values and reach in shared
// memory (asynchronous 16-byte copies, all in flight at once), walks the
// backward levels and then the forward levels of the new strategy there, with
// a block barrier between levels instead of a launch, and writes every result
// as it is formed.  An iteration of alternating updates is then four launches
// (terminals and tree, per player) instead of one per level, kernel class and
// player: a 39-node spot's iteration took 61.6 us by levels (47.3 once zero
// regrets skip their divisions) and takes 26.4 us.  Bound by the chain of
// levels; the arithmetic of a node and hand is that of k_bwd and k_fwd, in the
// same order, so the results are the same bit for bit.
struct alignas(16) TreeSeg {   // one player of one subgame
    long long reach;      // arena float offset of the player's part of node 0's reach slot
    long long cfv;        // the same in the value region
    long long rows;       // R/S float offset of the player's rows
    int h4, hs4;          // float4 groups of the player; slot stride in float4
    int n_rows, n_nodes;
    int node0, n_dec;     // decision nodes, in backward order
    int int0, n_int;      // integers: [nb + 1 backward bounds][nf + 1 forward bounds][own nodes in forward order]
                          // [terminals][value slot of every node, two a word]
    int nb, nf, n_own, n_term;
    int pad[2];
};
static_assert(sizeof(TreeSeg) == 80, "TreeSeg is 80 bytes");
struct TreeCta {          // one CTA: hands [4 g0, 4 (g0 + G)) of a TreeSeg, G = 1 << lg lanes
    int seg, g0, lg, pad;
};
// A decision node: first child; node | reach id << 16; node whose slot holds
// the player's reach; actions | acts << 5 | first regret row << 6.  Reach ids
// number the slots the player writes: 0 the root, 1 + row + k child k of the
// own node with that first row.
using TreeNode = int4;
struct TreeArgs {
    float *arena, *R, *S;
    const float* iter_tab;
    int* iter;            // [0] iteration, [1] CTAs done, [2] last iteration of the run
    const TreeCta* ctas;
    const TreeSeg* segs;
    const int* ints;
    const TreeNode* nodes;
    int n;                // CTAs of all the launches that close the iteration (TR_NEXT)
    int flags;            // TR_*
};
enum { TR_BWD = 1, TR_FWD = 2, TR_LAST = 4, TR_NEXT = 8 };   // TR_LAST: no forward part in the run's last iteration
constexpr int TREE_THREADS = 256, TREE_MAX_NODES = 1 << 16;

// float4 slots a lane: regret rows, sums, values and reach.  With simultaneous
// updates the sums are added by the forward part, so sums and reach take the
// place of the values once the backward part is done with them.
// A decision node's value takes the slot of its first child, which only it
// reads, so values need a slot per terminal.
__host__ __device__ inline int tree_slots(int n_rows, int n_term, bool sim) {
    const int sr = 2 * n_rows + 1;
    return n_rows + (sim ? (sr > n_term ? sr : n_term) : sr + n_term);
}
__host__ __device__ inline int tree_smem_bytes(int n_rows, int n_term, int n_dec, int n_int, int lg, bool sim) {
    return (tree_slots(n_rows, n_term, sim) << lg) * 16 + n_dec * 16 + (n_int + 3) / 4 * 16;
}

template <int ALGO>
__device__ __forceinline__ float4 upd_regret(float4 rk, float4 qk, float4 v, float dpos, float dneg) {
    if (ALGO == MTT_ALGO_DCFR)
        return make_float4(dcfr1(rk.x, __fsub_rn(qk.x, v.x), dpos, dneg), dcfr1(rk.y, __fsub_rn(qk.y, v.y), dpos, dneg),
                           dcfr1(rk.z, __fsub_rn(qk.z, v.z), dpos, dneg), dcfr1(rk.w, __fsub_rn(qk.w, v.w), dpos, dneg));
    return make_float4(cfrplus1(rk.x, __fsub_rn(qk.x, v.x)), cfrplus1(rk.y, __fsub_rn(qk.y, v.y)),
                       cfrplus1(rk.z, __fsub_rn(qk.z, v.z)), cfrplus1(rk.w, __fsub_rn(qk.w, v.w)));
}
template <int ALGO>
__device__ __forceinline__ float4 upd_sum(float4 sv, float4 r, float4 wr, float4 sg, float dstr) {
    return ALGO == MTT_ALGO_DCFR ? fma4(r, sg, mul4(sv, f4(dstr))) : fma4(wr, sg, sv);
}

// One node of one hand group, its rows and child values G float4 apart in
// shared memory: the acting player's update (returns the node's value) and the
// reach of its children.  A: the action count, with every row read before any
// is used, or 0: na actions.
template <int A, int ALGO, bool SIM>
__device__ __forceinline__ float4 tree_update(float4* rs, const float4* ss, const float4* V, const uint16_t* slot, float4 r,
                                              float4* R, float4* S, int na, int lg, int H4, const float4& tb) {
    const int n = A ? A : na;
    const float invA = __fdiv_rn(1.0f, (float)n);
    const float4 wr = mul4(r, f4(tb.x));
    float4 sum = f4(0.f), v = f4(0.f);
    if constexpr (A > 0) {
        float4 rk[A], qk[A], sg[A];
#pragma unroll
        for (int k = 0; k < A; ++k) { rk[k] = rs[k << lg]; qk[k] = V[(int)slot[k] << lg]; }
#pragma unroll
        for (int k = 0; k < A; ++k) sum = add4(sum, max04(rk[k]));
#pragma unroll
        for (int k = 0; k < A; ++k) sg[k] = rm4(max04(rk[k]), sum, invA);
#pragma unroll
        for (int k = 0; k < A; ++k) {
            v = fma4(sg[k], qk[k], v);
            if (!SIM) S[(size_t)k * H4] = upd_sum<ALGO>(ss[k << lg], r, wr, sg[k], tb.w);
        }
#pragma unroll
        for (int k = 0; k < A; ++k) {
            const float4 x = upd_regret<ALGO>(rk[k], qk[k], v, tb.y, tb.z);
            R[(size_t)k * H4] = x;
            rs[k << lg] = x;
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < n; ++k) sum = add4(sum, max04(rs[k << lg]));
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            const float4 sg = rm4(max04(rs[k << lg]), sum, invA);
            v = fma4(sg, V[(int)slot[k] << lg], v);
            if (!SIM) S[(size_t)k * H4] = upd_sum<ALGO>(ss[k << lg], r, wr, sg, tb.w);
        }
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            const float4 x = upd_regret<ALGO>(rs[k << lg], V[(int)slot[k] << lg], v, tb.y, tb.z);
            R[(size_t)k * H4] = x;
            rs[k << lg] = x;
        }
    }
    return v;
}

template <int A, int ALGO, bool SIM>
__device__ __forceinline__ void tree_reach(const float4* rs, const float4* ss, float4 r, float4* P, float4* ch, float4* S,
                                           int na, int lg, int H4, int HS4, const float4& tb) {
    const int n = A ? A : na;
    const float invA = __fdiv_rn(1.0f, (float)n);
    const float4 wr = mul4(r, f4(tb.x));
    float4 sum = f4(0.f);
    auto put = [&](int k, float4 sg) {
        const float4 x = mul4(r, sg);
        P[k << lg] = x;
        ch[(size_t)k * HS4] = x;
        if (SIM) S[(size_t)k * H4] = upd_sum<ALGO>(ss[k << lg], r, wr, sg, tb.w);
    };
    if constexpr (A > 0) {
        float4 rk[A];
#pragma unroll
        for (int k = 0; k < A; ++k) rk[k] = max04(rs[k << lg]);
#pragma unroll
        for (int k = 0; k < A; ++k) sum = add4(sum, rk[k]);
#pragma unroll
        for (int k = 0; k < A; ++k) rk[k] = rm4(rk[k], sum, invA);
#pragma unroll
        for (int k = 0; k < A; ++k) put(k, rk[k]);
    } else {
#pragma unroll 1
        for (int k = 0; k < n; ++k) sum = add4(sum, max04(rs[k << lg]));
#pragma unroll 1
        for (int k = 0; k < n; ++k) put(k, rm4(max04(rs[k << lg]), sum, invA));
    }
}

// SIM: both players are updated from one terminal pass; the strategy sums are
// then added by the forward part (of the next iteration), else by the backward
// part.
template <int ALGO, bool SIM>
__global__ void __launch_bounds__(TREE_THREADS, 2) k_tree(TreeArgs t) {
    extern __shared__ __align__(16) float4 tree_smem[];
    const TreeCta c = t.ctas[blockIdx.x];
    const TreeSeg sg = t.segs[c.seg];
    const int tid = threadIdx.x, lg = c.lg, G = 1 << lg, groups = TREE_THREADS >> lg;
    const int lane = tid & (G - 1), grp = tid >> lg, g = c.g0 + lane;
    const int H4 = sg.h4, HS4 = sg.hs4, n_rows = sg.n_rows;
    const bool live = g < H4;
    float4* const Rs = tree_smem + lane;                              // regret rows
    float4* const Ss = Rs + (n_rows << lg);                           // strategy sums
    float4* const P = Ss + (n_rows << lg);                            // reach by id
    float4* const V = SIM ? Ss : P + ((n_rows + 1) << lg);            // values by slot
    TreeNode* const nodes = reinterpret_cast<TreeNode*>(tree_smem + (tree_slots(n_rows, sg.n_term, SIM) << lg));
    int* const blev = reinterpret_cast<int*>(nodes + sg.n_dec);
    int* const flev = blev + sg.nb + 1;
    int* const own = flev + sg.nf + 1;
    int* const term = own + sg.n_own;
    const uint16_t* const slot = reinterpret_cast<const uint16_t*>(term + sg.n_term);
    for (int i = tid; i < sg.n_dec; i += TREE_THREADS) nodes[i] = t.nodes[sg.node0 + i];
    for (int i = tid; i < sg.n_int; i += TREE_THREADS) blev[i] = t.ints[sg.int0 + i];
    float4* const reach = reinterpret_cast<float4*>(t.arena + sg.reach) + g;
    float4* const cfv = reinterpret_cast<float4*>(t.arena + sg.cfv) + g;
    float4* const R = reinterpret_cast<float4*>(t.R + sg.rows) + g;
    float4* const S = reinterpret_cast<float4*>(t.S + sg.rows) + g;
    __syncthreads();
    // the tree's description is written once, before any solve; all else
    // belongs to the kernels before
    grid_dep_trigger();
    grid_dep_wait();
    const int iter = t.iter[0];
    const bool bwd = t.flags & TR_BWD;
    const bool fwd = (t.flags & TR_FWD) && !((t.flags & TR_LAST) && iter >= t.iter[2]);
    if (live) {
        for (int i = grp; i < n_rows; i += groups) {
            copy_async16(Rs + (i << lg), R + (size_t)i * H4);
            if (!SIM && bwd) copy_async16(Ss + (i << lg), S + (size_t)i * H4);
        }
        if (bwd)
            for (int i = grp; i < sg.n_term; i += groups)
                copy_async16(V + (i << lg), cfv + (size_t)term[i] * HS4);
        if (!SIM && bwd)
            for (int i = grp; i < sg.n_own; i += groups) {
                const TreeNode nd = nodes[own[i]];
                copy_async16(P + ((int)((unsigned)nd.y >> 16) << lg), reach + (size_t)nd.z * HS4);
            }
        if (!SIM && !bwd && grp == 0) copy_async16(P, reach);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (bwd) {
        const float4 tb = *reinterpret_cast<const float4*>(t.iter_tab + 4 * (size_t)(iter - 1));
        for (int l = 0; l < sg.nb; ++l) {
            const int hi = blev[l + 1];
            for (int i = blev[l] + grp; live && i < hi; i += groups) {
                const TreeNode nd = nodes[i];
                const int na = nd.w & 31, self = nd.y & 0xFFFF;
                const uint16_t* const cs = slot + nd.x;
                float4 v = f4(0.f);
                if (nd.w & 32) {
                    const int row = (int)((unsigned)nd.w >> 6);
                    const float4 r = SIM ? f4(0.f) : P[(int)((unsigned)nd.y >> 16) << lg];
#define TREE_CALL(A) \
    v = tree_update<A, ALGO, SIM>(Rs + (row << lg), Ss + (row << lg), V, cs, r, R + (size_t)row * H4, S + (size_t)row * H4, na, lg, \
                                  H4, tb)
                    switch (na) {
                        case 2: TREE_CALL(2); break;
                        case 3: TREE_CALL(3); break;
                        case 4: TREE_CALL(4); break;
                        default: TREE_CALL(0); break;
                    }
#undef TREE_CALL
                } else {
#pragma unroll 4
                    for (int k = 0; k < na; ++k) v = add4(v, V[(int)cs[k] << lg]);
                }
                V[(int)cs[0] << lg] = v;
                cfv[(size_t)self * HS4] = v;
            }
            __syncthreads();
        }
    }
    if (fwd) {
        if (SIM) {                     // every CTA thread is past the values
            if (live) {
                for (int i = grp; i < n_rows; i += groups) copy_async16(Ss + (i << lg), S + (size_t)i * H4);
                if (grp == 0) copy_async16(P, reach);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
        // the sums of simultaneous updates are weighted by the iteration they open
        const float4 tb = SIM ? *reinterpret_cast<const float4*>(t.iter_tab + 4 * (size_t)(iter - (bwd ? 0 : 1))) : f4(0.f);
        for (int l = 0; l < sg.nf; ++l) {
            const int hi = flev[l + 1];
            for (int i = flev[l] + grp; live && i < hi; i += groups) {
                const TreeNode nd = nodes[own[i]];
                const int na = nd.w & 31, row = (int)((unsigned)nd.w >> 6);
                const float4 r = P[(int)((unsigned)nd.y >> 16) << lg];
#define TREE_CALL(A) \
    tree_reach<A, ALGO, SIM>(Rs + (row << lg), Ss + (row << lg), r, P + ((1 + row) << lg), reach + (size_t)nd.x * HS4, \
                             S + (size_t)row * H4, na, lg, H4, HS4, tb)
                switch (na) {
                    case 2: TREE_CALL(2); break;
                    case 3: TREE_CALL(3); break;
                    case 4: TREE_CALL(4); break;
                    default: TREE_CALL(0); break;
                }
#undef TREE_CALL
            }
            if (l + 1 < sg.nf) __syncthreads();
        }
    }
    // the last CTA of the closing launches opens the next iteration: every CTA has read this one's number
    if ((t.flags & TR_NEXT) && tid == 0 && atomicAdd(t.iter + 1, 1) == t.n - 1) {
        t.iter[1] = 0;
        t.iter[0] = iter + 1;
    }
}

// What build_seg needs of node k: decision nodes only carry player, na, first,
// row; src is the node whose slot holds the player's reach.
struct TreeShapeNode {
    bool dec;
    int player, na, first, row, src, depth;
};

// Host arrays of the whole-tree sweeps.
struct TreeHost {
    std::vector<TreeSeg> segs;
    std::vector<int> sub;            // subgame of each segment
    std::vector<int> ints;
    std::vector<TreeNode> nodes;
    void append(const TreeHost& o) {
        for (TreeSeg g : o.segs) {
            g.node0 += (int)nodes.size();
            g.int0 += (int)ints.size();
            segs.push_back(g);
        }
        sub.insert(sub.end(), o.sub.begin(), o.sub.end());
        ints.insert(ints.end(), o.ints.begin(), o.ints.end());
        nodes.insert(nodes.end(), o.nodes.begin(), o.nodes.end());
    }
};

// Their device copies, parts of one allocation.
struct TreeDev {
    TreeNode* nodes = nullptr;
    TreeSeg* segs = nullptr;
    int* ints = nullptr;
};

// fn(0) .. fn(n - 1), about `ns` nanoseconds in all, on up to 16 host threads
// with 200 us each or more (starting one takes some 30).
template <typename Fn>
inline void on_threads(int n, long long ns, Fn fn) {
    const int nt = (int)std::min<long long>({n, (long long)std::thread::hardware_concurrency(), 16, ns / 200000});
    std::atomic<int> next{0};
    auto run = [&]() { for (int i; (i = next.fetch_add(1)) < n;) fn(i); };
    std::vector<std::thread> th;
    try {
        for (int t = 1; t < nt; ++t) th.emplace_back(run);
    } catch (const std::system_error&) {       // no more threads to be had: those there are share the work
    }
    run();
    for (std::thread& x : th) x.join();
}

// What a slice of one player's tree needs of shared memory, at most one level
// per node.  No slice fits where two nodes share regret rows: a level launch
// adds both nodes' sums to them, one level after the other, while a slice
// stages the sums once and numbers its reach by row.
struct TreeSize {
    int n_rows = 0, n_term = 0, n_dec = 0, n_int = 0;
    bool shared = false;
    int bytes(int lg, bool sim) const {        // of 4 << lg hands
        return shared ? INT_MAX : tree_smem_bytes(n_rows, n_term, n_dec, n_int, lg, sim);
    }
};
template <typename Node>
inline TreeSize tree_size(int n_nodes, int n_rows, int q, Node node) {
    TreeSize z;
    int own = 0;
    std::vector<char> used(n_rows, 0);
    for (int k = 0; k < n_nodes; ++k) {
        const TreeShapeNode nd = node(k);
        z.n_dec += nd.dec;
        if (!nd.dec || nd.player != q) continue;
        ++own;
        for (int a = 0; a < nd.na; ++a) {
            z.shared |= used[nd.row + a] != 0;
            used[nd.row + a] = 1;
        }
    }
    z.n_rows = n_rows;
    z.n_term = n_nodes - z.n_dec;
    z.n_int = 2 * (z.n_dec + 1) + own + z.n_term + (n_nodes + 1) / 2;
    return z;
}

// One player's view of a chance-free tree: the backward order (all decision
// nodes, deepest level first) and the forward order (the player's own, by how
// many of them lie above), each level sorted by role and action count so that
// a warp's nodes take the same path.  g: offsets, sizes and rows filled in.
template <typename Node>
inline void build_tree_seg(TreeHost& L, TreeSeg g, int sub, int q, Node node) {
    const int n = g.n_nodes;
    std::vector<TreeShapeNode> nd(n);
    for (int k = 0; k < n; ++k) nd[k] = node(k);
    g.node0 = (int)L.nodes.size();
    g.int0 = (int)L.ints.size();
    std::vector<int> above(n, 0), id(n, 0), pos(n, 0), order;
    for (int k = 0; k < n; ++k) {
        if (!nd[k].dec) continue;
        const bool own = nd[k].player == q;
        for (int c = 0; c < nd[k].na; ++c) {
            above[nd[k].first + c] = above[k] + (own ? 1 : 0);
            if (own) id[nd[k].first + c] = 1 + nd[k].row + c;
        }
        order.push_back(k);
    }
    auto key = [&](int k) { return (nd[k].player == q ? 32 : 0) | nd[k].na; };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return nd[x].depth != nd[y].depth ? nd[x].depth > nd[y].depth : key(x) < key(y);
    });
    g.n_dec = (int)order.size();
    for (int i = 0; i < g.n_dec; ++i) {
        const int k = order[i];
        if (i == 0 || nd[k].depth != nd[order[i - 1]].depth) { L.ints.push_back(i); ++g.nb; }
        const bool own = nd[k].player == q;
        L.nodes.push_back(make_int4(nd[k].first, (int)((unsigned)k | (unsigned)id[nd[k].src] << 16), nd[k].src,
                                    (int)((unsigned)key(k) | (own ? (unsigned)nd[k].row << 6 : 0u))));
        pos[k] = i;
    }
    L.ints.push_back(g.n_dec);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return above[x] != above[y] ? above[x] < above[y] : key(x) < key(y);
    });
    std::vector<int> own;
    int last = -1;
    for (int k : order) {
        if (nd[k].player != q) continue;
        if (above[k] != last) { L.ints.push_back((int)own.size()); ++g.nf; last = above[k]; }
        own.push_back(pos[k]);
    }
    L.ints.push_back((int)own.size());
    g.n_own = (int)own.size();
    L.ints.insert(L.ints.end(), own.begin(), own.end());
    std::vector<uint16_t> slot(n + (n & 1), 0);
    for (int k = 0; k < n; ++k)
        if (!nd[k].dec) { slot[k] = (uint16_t)g.n_term++; L.ints.push_back(k); }
    for (int k = n - 1; k >= 0; --k)               // children follow their parents
        if (nd[k].dec) slot[k] = slot[nd[k].first];
    for (int k = 0; k < n; k += 2) L.ints.push_back((int)((unsigned)slot[k] | (unsigned)slot[k + 1] << 16));
    g.n_int = (int)L.ints.size() - g.int0;
    L.segs.push_back(g);
    L.sub.push_back(sub);
}

}  // namespace mtt
