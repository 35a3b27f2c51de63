// Warp-level PUCT select with virtual loss, plus the backup / release kernels that undo the claims.
//
// Drop-in for the reference's only native library, src/puct/puct_gpu_v3_cpp.cu: the exported launcher
// puct_select_winner_recalc_launch has the same 21 arguments (:450-481) and puct_cpp_cuda_error_string the same
// meaning (:483-485), so the reference's ctypes binding (src/puct/puct_gpu_v3_cpp.py:84-156) can load this library
// instead.  Semantics followed (not the code): one warp = one traversal of its tree; per level the progressive-widening
// quota ceil(c_pw * N^alpha) (:150-157), an expansion ticket by atomicAdd (:219-233), the score
// W/N + cpuct * P * sqrt(N_parent_eff) / (1 + N + inflight) (:171-180), ties broken by edge id rotated by the warp id
// (:50-71), the winner claimed with atomicCAS(inflight, seen, seen + 1) and at most two evaluations (:235-275), the
// path entry (node << 8) | edge (:436), the packed result reason << 25 | kind << 22 | slot << 14 | node (:38-41),
// and the rollback of every claim of the traversal when it fails (:206-217).
//
// What is done differently: a traversal is a chain of dependent loads from gigabytes of edge arrays, and a warp that is alone
// on its scheduler takes 4 to 5 cycles for every instruction of the chain between two of them, so a level is built to cost
// ONE memory round trip and few instructions.  Every lane keeps child / prior / W / N / inflight of its edges in
// registers; as soon as the winner is known, the child's node record and ALL the child's edges are requested, then the claim
// (atomicCAS) is sent; and the claim's answer is looked at only when the child's own winner has been worked out, right before
// anything else is claimed, so that its round trip is not waited for.  A lost claim goes back to the level it was made on
// and reads that level's edges again.  Sums, maxima and the tie-break use the warp-reduce instructions (redux.sync); the
// edge number of the winner names the lane that holds it.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/puct_b200.h"
#include "select_math.cuh"

namespace puct {

using namespace select_math;

constexpr int NODE_TERMINAL = -1;
constexpr int OUTSIDE = -2;   // in place of a node's record: the node does not exist
constexpr int NODE_LIMIT = 16384, NODE_MASK = 0x3FFF, EDGE_LIMIT = 256;
constexpr int KIND_SHIFT = 22, SLOT_SHIFT = 14, REASON_SHIFT = 25;
enum Kind { INVALID = 0, EXPAND = 1, TERMINAL = 2, DEPTH_LIMIT = 3, BUSY = 4 };
enum Reason {
    R_UNSET = 0, R_OK_EXPAND = 1, R_OK_TERMINAL = 2, R_OK_DEPTH_LIMIT = 3, R_BUSY_EXPAND_INFLIGHT = 4,
    R_BUSY_WINNER_RECALC = 5, R_INVALID_SHAPE = 10, R_INVALID_NODE_INFO = 11, R_INVALID_NO_VALID_EDGE = 14,
    R_INVALID_CHILD_OOB = 15, R_INVALID_UNKNOWN = 16
};
constexpr int MAX_EVALUATIONS = 2;
constexpr int NO_EDGE = 0x7FFFFFFF;
// what root_kernel leaves in the place of a path's length where the traversal goes on: at the child in the place of its result, from
// the root
constexpr int FROM_CHILD = -1, FROM_ROOT = -2;

__device__ __forceinline__ int pack(int kind, int node, int slot, int reason) {
    return (reason << REASON_SHIFT) | (kind << KIND_SHIFT) | (slot << SLOT_SHIFT) | node;
}

// undo the claims of the first `depth` path entries of this warp
__device__ __forceinline__ void rollback(const int *path, int depth, int lane, int *edge_inflight, long long tree_edges_base,
                                         int node_cnt, int edges, int amount) {
    __syncwarp();   // lane 0 wrote the entries
    for (int d = lane; d < depth; d += 32) {
        const int enc = path[d];
        const int parent = enc >> 8, slot = enc & 0xFF;
        if (parent >= 0 && parent < node_cnt && slot < edges)
            atomicSub(&edge_inflight[tree_edges_base + (long long)parent * edges + slot], amount);
    }
}

// The edges of one node as seen by one lane (edge lane + 32 k in slot k).  Slots beyond the array's `edges` keep harmless values.
template <int EPL>
struct EdgeRegs {
    const int *child_of, *n_of;   // of this tree
    const float *prior_of, *w_of;
    int *inflight_of;
    float prior[EPL], w[EPL];
    int n[EPL], inflight[EPL], child[EPL];

    __device__ __forceinline__ void init(long long tree_edges, const int *edge_child_id, const float *edge_prior, const float *edge_W,
                                         const int *edge_N, int *edge_inflight) {
        child_of = edge_child_id + tree_edges;
        prior_of = edge_prior + tree_edges;
        w_of = edge_W + tree_edges;
        n_of = edge_N + tree_edges;
        inflight_of = edge_inflight + tree_edges;
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            prior[k] = w[k] = 1.f;
            n[k] = 1;
            inflight[k] = 0;
            child[k] = -1;
        }
    }

    // requests all `edges` slots of a node, expanded or not (the arrays are dense, so the addresses are valid): this is done
    // before the node's record has arrived, i.e. before the number of expanded edges is known
    __device__ __forceinline__ void request(int node, int lane, int edges) {
        const unsigned first = (unsigned)(node * edges + lane) * 4u;   // < 2^24
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (lane + 32 * k < edges) {
                n[k] = *at(n_of, first + 128u * k);
                inflight[k] = *(volatile const int *)at(inflight_of, first + 128u * k);
                prior[k] = *at(prior_of, first + 128u * k);
                w[k] = *at(w_of, first + 128u * k);
                child[k] = *at(child_of, first + 128u * k);
            }
    }
};

// Scores of the expanded edges (LOWEST_INF: none, as for NaN and -inf); returns the best
template <int EPL>
__device__ __forceinline__ float score_edges(const EdgeRegs<EPL> &r, float (&score)[EPL], float cpuct, float sqrt_parent, int n_exp, int lane) {
    float my_best = LOWEST_INF;
    bool plain = true;
#pragma unroll
    for (int k = 0; k < EPL; k++) {
        const bool visited = r.n[k] > 0;
        const float up = cpuct * r.prior[k] * sqrt_parent;
        const int tries = r.n[k] + r.inflight[k] + 1;
        const float mean = Count(visited ? r.n[k] : 1).divides(r.w[k]);
        const float v = (visited ? mean : 0.0f) + Count(tries).divides(up);
        plain = plain && (unsigned)((tries - 1) | r.n[k]) < (1u << 22) && Count::plain(r.w[k], up);
        score[k] = v;
    }
    if (!plain) {   // counts of millions, or values no network gives
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            const float q = r.n[k] > 0 ? r.w[k] / (float)r.n[k] : 0.0f;
            score[k] = q + cpuct * r.prior[k] * sqrt_parent / (float)(r.n[k] + r.inflight[k] + 1);
        }
    }
#pragma unroll
    for (int k = 0; k < EPL; k++) {
        score[k] = lane + 32 * k < n_exp && score[k] >= LOWEST ? score[k] : LOWEST_INF;
        my_best = fmaxf(my_best, score[k]);
    }
    return max_of_warp(my_best);
}

template <int EPL>
__device__ __forceinline__ int parent_count(const EdgeRegs<EPL> &r, int n_exp, int lane) {
    int partial = 0;
#pragma unroll
    for (int k = 0; k < EPL; k++)
        if (lane + 32 * k < n_exp) partial += r.n[k] + r.inflight[k];
    return max(__reduce_add_sync(FULL, partial), 1);
}

// EPL: edges per lane, ceil(edges / 32) rounded up to 1, 2, 4 or 8 (registers follow it).
//
// Traversal i = tree * warps + w is block i, a single warp.  The reference puts the `warps` traversals of a tree into one block
// (src/puct/puct_gpu_v3_cpp.cu:472-473); with 8 traversals per tree most of them lose the claim at the root and leave after
// two evaluations, and a block of 8 warps then keeps its 6 idle warp slots until its last traversal has gone all the way
// down.  Small blocks give the slots back at once; the traversals of a tree still start together (their blocks are
// neighbours in the grid).  As many blocks as an SM can hold (32) with up to 64 edges.
// WIDENING: c_pw is not zero.
//
// RESUMED: root_kernel has been here; see there.
template <int EPL, bool WIDENING, bool RESUMED>
__global__ void __launch_bounds__(32, EPL <= 2 ? 32 : (EPL == 4 ? 24 : 16))
select_kernel(float cpuct, float c_pw, float alpha_pw, int soft_winner, const int *edge_child_id,
              const float *edge_prior, const float *edge_W, const int *edge_N,
              int *edge_inflight, int *node_expand_inflight, const int *node_expanded,
              const int *tree_nodes, int *out_selected_node, int *out_path_eids, int *out_path_len, int nodes,
              int edges, int warps, int path_depth, int vl, int trees) {
    let_the_next_kernel_come();
    const unsigned block = block_after_the_kernel_before();
    const int lane = threadIdx.x;
    int tree, wid, traversal;
    if (RESUMED) {   // the traversals that go on are the first of their trees, but for ties: they start first, the others leave at once
        wid = block / trees;
        tree = block - wid * trees;
        traversal = tree * warps + wid;
    } else {
        traversal = block;
        tree = traversal / warps;
        wid = traversal - tree * warps;
    }
    const int state = RESUMED ? out_path_len[traversal] : FROM_ROOT;
    if (RESUMED && state >= 0) return;
    int *path = out_path_eids + (long long)traversal * path_depth;
    const long long tree_nodes_base = (long long)tree * nodes;
    const long long tree_edges_base = tree_nodes_base * edges;
    const int node_cnt = tree_nodes[tree];
    if (!(path_depth >= 1 && nodes > 0 && node_cnt > 0 && node_cnt <= nodes && node_cnt <= NODE_LIMIT && edges > 0 &&
          edges <= EDGE_LIMIT)) {
        if (lane == 0) {
            out_selected_node[traversal] = pack(INVALID, NODE_MASK, 0, R_INVALID_SHAPE);
            out_path_len[traversal] = 0;
        }
        return;
    }
    const int *expanded = node_expanded + tree_nodes_base;
    EdgeRegs<EPL> r;
    r.init(tree_edges_base, edge_child_id, edge_prior, edge_W, edge_N, edge_inflight);
    int *inflight_of_tree = edge_inflight + tree_edges_base;
    int node = 0, depth = 0;
    bool outside = false;      // the child that was picked does not exist
    if (RESUMED && state == FROM_CHILD) {
        node = out_selected_node[traversal];
        depth = 1;
        outside = (unsigned)node >= (unsigned)node_cnt;
    }
    const int start = outside ? 0 : node;
    int info = expanded[start];
    r.request(start, lane, edges);
    if (outside) info = OUTSIDE;
    float sqrt_parent = 0.f;
    int attempt = 0;           // evaluations of this level that ended with a lost claim
    // the claim made on the level above, until its answer is needed
    bool pending = false;
    int up_node = 0, up_info = 0, up_edge = 0, up_attempt = 0, up_seen = 0, up_old = 0;   // the last two: the owner's lane
    float up_sqrt = 0.f;
    int my_seen = 0, my_child = -1;    // of the lane's best edge

    // arg-max over the expanded edges (two or more); NO_EDGE: no edge has a score (NaN and -inf are none)
    auto arg_max = [&](int n_exp) {
        // ties go to the edge closest after `rot` = wid modulo n_exp (small numbers: the product with the reciprocal truncates
        // right)
        const int rot = wid - n_exp * (int)(((float)wid + 0.5f) * reciprocal((float)n_exp));
        float score[EPL];
        const float top = score_edges(r, score, cpuct, sqrt_parent, n_exp, lane);
        if (top == LOWEST_INF) return NO_EDGE;
        // the bits are compared: +0 is above -0
        if (EPL <= 2) {
            const unsigned low = __ballot_sync(FULL, __float_as_uint(score[0]) == __float_as_uint(top)), behind = low >> rot;   // rot < 32
            const unsigned high = EPL == 2 ? __ballot_sync(FULL, __float_as_uint(score[EPL - 1]) == __float_as_uint(top)) : 0u;
            const int best = behind ? rot + __ffs(behind) - 1 : (high ? 31 + __ffs(high) : __ffs(low) - 1);
            my_seen = EPL == 2 && best >= 32 ? r.inflight[EPL - 1] : r.inflight[0];
            my_child = EPL == 2 && best >= 32 ? r.child[EPL - 1] : r.child[0];
            return best;
        }
        int my_tie = NO_EDGE;
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            const int e = lane + 32 * k;
            const int tie = e >= rot ? e - rot : e - rot + n_exp;
            if (__float_as_uint(score[k]) == __float_as_uint(top) && tie < my_tie) {
                my_tie = tie;
                my_seen = r.inflight[k];
                my_child = r.child[k];
            }
        }
        const int tie = (int)__reduce_min_sync(FULL, (unsigned)my_tie);
        return tie + rot >= n_exp ? tie + rot - n_exp : tie + rot;
    };
    auto quota_of = [&](int parent_eff) {
        const float quota = (alpha_pw == 0.5f) ? c_pw * root_of_count(parent_eff) : c_pw * powf((float)parent_eff, alpha_pw);
        return quota >= (float)edges ? edges : max(1, (int)ceilf(quota));
    };
    // (no claim made: up_old == up_seen everywhere)
    auto claim_held = [&]() { return __any_sync(FULL, lane == (up_edge & 31) && up_old == up_seen) != 0; };
    // claims edge `best` of `node` and goes on to its child, whose data is requested first
    auto descend = [&](int best, bool only) {
        const int owner = best & 31;
        const int child = __shfl_sync(FULL, my_child, owner);
        outside = (unsigned)child >= (unsigned)node_cnt;
        up_info = info;
        const int there = outside ? 0 : child;
        info = *at(expanded, (unsigned)there * 4u);
        r.request(there, lane, edges);
        if (outside) info = OUTSIDE;
        int *count = inflight_of_tree + (node * edges + best);
        if (only) {
            if (lane == 0) atomicAdd(count, vl);
            up_old = up_seen;
        } else {
            // predicated, so that nothing behind it waits for the answer
            up_seen = my_seen;
            asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %4, %5;\n\t@p atom.global.cas.b32 %0, [%1], %2, %3;\n\t}"
                         : "+r"(up_old) : "l"(count), "r"(my_seen), "r"(my_seen + vl), "r"(lane), "r"(owner) : "memory");
        }
        pending = !only;
        up_node = node;
        up_edge = best;
        if (lane == 0) path[depth] = (node << 8) | best;
        node = child;
        depth++;
    };

    const unsigned several = edges - 1;   // info - 2 below it: two edges or more, and no more than there are
    // A claim's answer takes longer than the next level's data out of L2: a traversal that is alone in its tree looks at it
    // only when it is about to make the next claim.  Where others compete for the tree a lost claim is noticed before the level
    // below is worked out for nothing.
    const bool alone = warps == 1;
    int result, result_len = 0;
    for (;;) {
        // ---- the usual level: two or more edges, no room for another, a score, and the claim of the level above held
        if (attempt == 0) while ((unsigned)(info - 2) < several && depth < path_depth) {
            if (!alone && !claim_held()) break;
            const int parent_eff = parent_count(r, info, lane);
            sqrt_parent = root_of_count(parent_eff);
            if (WIDENING && quota_of(parent_eff) > info) break;
            const int best = arg_max(info);
            if (best == NO_EDGE || (alone && !claim_held())) break;
            up_attempt = 0;
            up_sqrt = sqrt_parent;
            descend(best, false);
        }
        // ---- anything else.  The claim of the level above has to hold first
        if (pending) {
            pending = false;
            bool held = claim_held();
            if (!held && up_attempt + 1 >= MAX_EVALUATIONS && soft_winner != 0) {
                if (lane == 0) atomicAdd(inflight_of_tree + (up_node * edges + up_edge), vl);
                held = true;
            }
            if (!held) {
                // somebody else moved the winner's count
                depth--;
                node = up_node;
                if (up_attempt + 1 >= MAX_EVALUATIONS) {
                    rollback(path, depth, lane, edge_inflight, tree_edges_base, node_cnt, edges, vl);
                    result = pack(BUSY, node, 0, R_BUSY_WINNER_RECALC);
                    break;
                }
                info = up_info;
                attempt = up_attempt + 1;
                sqrt_parent = up_sqrt;
                outside = false;
                r.request(node, lane, edges);
                continue;
            }
        }
        const int n_exp = info;
        const bool at_end = outside || info < 0 || info > edges || depth >= path_depth;
        int allowed = 1, best = NO_EDGE;
        if (!at_end && (n_exp != 1 || WIDENING)) {
            const int parent_eff = parent_count(r, n_exp, lane);
            if (attempt == 0) sqrt_parent = root_of_count(parent_eff);   // another evaluation keeps the parent's count
            if (WIDENING) allowed = quota_of(parent_eff);
            if (n_exp > 1) best = arg_max(n_exp);
        }
        if (at_end) {
            if (outside) {
                rollback(path, depth, lane, edge_inflight, tree_edges_base, node_cnt, edges, vl);
                result = pack(INVALID, NODE_MASK, 0, R_INVALID_CHILD_OOB);
            } else if (info == NODE_TERMINAL) {
                result = pack(TERMINAL, node, 0, R_OK_TERMINAL);
                result_len = depth + 1;
            } else if (info < 0 || info > edges) {
                rollback(path, depth, lane, edge_inflight, tree_edges_base, node_cnt, edges, vl);
                result = pack(INVALID, NODE_MASK, 0, R_INVALID_NODE_INFO);
            } else {
                result = pack(DEPTH_LIMIT, node, 0, R_OK_DEPTH_LIMIT);
                result_len = depth + 1;
            }
            break;
        }
        if (allowed > n_exp && attempt == 0) {
            // room for a new child: take a ticket unless the tickets in flight already fill the quota
            int slot = -1;
            if (lane == 0) {
                int *tickets = &node_expand_inflight[tree_nodes_base + node];
                if (n_exp + *tickets < allowed) {
                    const int s = n_exp + atomicAdd(tickets, 1);
                    if (s < allowed) slot = s;
                    else atomicSub(tickets, 1);
                }
            }
            slot = __shfl_sync(FULL, slot, 0);
            if (slot >= 0) {
                result = pack(EXPAND, node, slot, R_OK_EXPAND);
                result_len = depth + 1;
                break;
            }
            if (n_exp == 0) {
                rollback(path, depth, lane, edge_inflight, tree_edges_base, node_cnt, edges, vl);
                result = pack(BUSY, node, 0, R_BUSY_EXPAND_INFLIGHT);
                break;
            }
        }
        // ---- go on to an existing child
        const bool only = n_exp == 1;
        if (only) {
            best = 0;
            my_child = r.child[0];
        } else if (best == NO_EDGE) {
            rollback(path, depth, lane, edge_inflight, tree_edges_base, node_cnt, edges, vl);
            result = pack(INVALID, NODE_MASK, 0, R_INVALID_NO_VALID_EDGE);
            break;
        }
        up_attempt = attempt;
        up_sqrt = sqrt_parent;
        descend(best, only);
        attempt = 0;
    }
    if (lane == 0) {
        out_selected_node[traversal] = result;
        out_path_len[traversal] = result_len;
    }
}

// The root for all traversals of a tree, by one warp.  Traversals that start together see the same counts, so there is one
// evaluation to make, not one each; those that want the same edge want it at the same time, and the first of them has it.  The others
// evaluate once more and, under the strict rule, are BUSY if they lose again: with eight traversals a tree six of them, whose warps
// did nothing but that.  The traversals that hold a claim (and those of a root that is not the usual one: two edges
// or more, a score) go on in select_kernel<., ., RESUMED>.  4096 trees x 64 edges x 16 levels x 8 traversals: 95 us in one kernel, see
// roots_first.
constexpr int ROOT_WARPS = 4;
template <int EPL>
__global__ void __launch_bounds__(ROOT_WARPS * 32)
root_kernel(float cpuct, int soft_winner, const int *edge_child_id, const float *edge_prior,
            const float *edge_W, const int *edge_N, int *edge_inflight, const int *node_expanded,
            const int *tree_nodes, int *out_selected_node, int *out_path_eids, int *out_path_len, int trees, int nodes, int edges,
            int warps, int path_depth, int vl) {
    let_the_next_kernel_come();
    const unsigned block = block_after_the_kernel_before();
    const int lane = threadIdx.x & 31, tree = block * ROOT_WARPS + (threadIdx.x >> 5);
    if (tree >= trees) return;
    const bool mine = lane < warps;   // lane w: traversal w
    const long long traversal = (long long)tree * warps + lane;
    const int node_cnt = tree_nodes[tree];
    const long long tree_edges = (long long)tree * nodes * edges;
    int n_exp = 0;
    EdgeRegs<EPL> r;
    r.init(tree_edges, edge_child_id, edge_prior, edge_W, edge_N, edge_inflight);
    if (path_depth >= 1 && nodes > 0 && node_cnt > 0 && node_cnt <= nodes && node_cnt <= NODE_LIMIT && edges > 0 && edges <= EDGE_LIMIT) {
        n_exp = node_expanded[(long long)tree * nodes];
        r.request(0, lane, edges);
    }
    bool usual = n_exp >= 2 && n_exp <= edges;
    float sqrt_parent = 0.f;
    if (usual) sqrt_parent = root_of_count(parent_count(r, n_exp, lane));
    bool open = mine;          // the traversal has no claim and no result yet
    for (int evaluation = 1; usual && evaluation <= MAX_EVALUATIONS; evaluation++) {
        if (evaluation > 1) {
            __syncwarp();   // the claims just made, each by a lane of its own, are seen
            r.request(0, lane, edges);
        }
        float score[EPL];
        const float top = score_edges(r, score, cpuct, sqrt_parent, n_exp, lane);
        if (top == LOWEST_INF) {
            if (evaluation == 1) usual = false;
            else if (open) {
                out_selected_node[traversal] = pack(INVALID, NODE_MASK, 0, R_INVALID_NO_VALID_EDGE);
                out_path_len[traversal] = 0;
                open = false;
            }
            break;
        }
        // every lane its own traversal's edge: the first of those with the top score from edge wid modulo n_exp on
        unsigned even[EPL];
#pragma unroll
        for (int k = 0; k < EPL; k++) even[k] = __ballot_sync(FULL, __float_as_uint(score[k]) == __float_as_uint(top));
        const int rot = lane % n_exp;
        int best = NO_EDGE, first = NO_EDGE;
#pragma unroll
        for (int k = EPL - 1; k >= 0; k--) {
            if (even[k] == 0u) continue;
            first = 32 * k + __ffs(even[k]) - 1;
            const unsigned behind = rot >= 32 * k + 32 ? 0u : (rot > 32 * k ? even[k] >> (rot - 32 * k) << (rot - 32 * k) : even[k]);
            if (behind != 0u) best = 32 * k + __ffs(behind) - 1;
        }
        if (best == NO_EDGE) best = first;
        // its count and its child, out of the lane that holds them
        int seen = 0, child = 0;
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            const int c = __shfl_sync(FULL, r.inflight[k], best & 31), to = __shfl_sync(FULL, r.child[k], best & 31);
            if (k == best >> 5) {
                seen = c;
                child = to;
            }
        }
        const unsigned same = __match_any_sync(FULL, open ? best : -1);
        bool held = false;
        if (open && __ffs(same) - 1 == lane) held = atomicCAS(&r.inflight_of[best], seen, seen + vl) == seen;
        if (open && !held && evaluation == MAX_EVALUATIONS && soft_winner != 0) {
            atomicAdd(&r.inflight_of[best], vl);
            held = true;
        }
        if (held) {
            out_path_eids[traversal * path_depth] = best;   // node 0
            out_selected_node[traversal] = child;
            out_path_len[traversal] = FROM_CHILD;
            open = false;
        }
        if (!__any_sync(FULL, open)) break;
    }
    if (open) {
        out_selected_node[traversal] = pack(BUSY, 0, 0, R_BUSY_WINNER_RECALC);
        out_path_len[traversal] = usual ? 0 : FROM_ROOT;
    }
}

// Whether a launch's roots are done by root_kernel first: where more traversals will find no place at a root, all but two of
// a tree, than a quarter over what the device holds at once of them (32, 24 or 16 warps an SM).  Fewer cost less than the second
// launch, 5 us.  Microseconds of the select, one kernel / two (trees x edges x levels x traversals a tree):
//   4096 x 64 x 16 x 8 95 / 68, x 4 74 / 68   2500 x 64 x 12 x 8 58 / 45   1000 x 64 x 12 x 8 33 / 30   2500 x 19 x 12 x 8 45 / 36
//   4096 x 8 x 16 x 8 76 / 46   3000 x 100 x 8 x 8 82 / 48   1500 x 200 x 6 x 8 76 / 43, x 4 54 / 43;   not taken: 4096 x 64 x 16 x 2
//   64 / 68   2500 x 64 x 12 x 4 44 / 45   700 x 64 x 12 x 8 29 / 29   500 x 100 x 8 x 8 27 / 27
static bool roots_first(int trees, int edges, int warps) {
    const int warps_of_sm = edges <= 64 ? 32 : (edges <= 128 ? 24 : 16);
    return warps > 2 && edges >= 2 && edges <= EDGE_LIMIT && 4LL * trees * (warps - 2) > 5LL * warps_of_sm * sm_count();
}

// Turns the claims of finished traversals into statistics (v3 edge layout; the reference has this step only for its
// older node-inflight layout, src/puct/puct_gpu_v2.py:847-927): per path edge inflight -= virtual_loss, N += 1,
// W += value; an EXPAND result also returns its ticket.  With values == NULL only the claims are released
// (src/puct/test_puct_gpu_v3.py:274-332).
__global__ void backup_kernel(int virtual_loss, float *edge_W, int *edge_N, int *edge_inflight, int *node_expand_inflight,
                              const int *tree_nodes, const int *out_selected_node,
                              const int *out_path_eids, const int *out_path_len,
                              const float *path_edge_values, int traversals, int nodes, int edges, int warps,
                              int path_depth, int log2_lanes) {
    const BackupLane at_work(block_after_the_kernel_before(), traversals, log2_lanes);
    const int out_ix = at_work.traversal;
    if (out_ix < 0) return;
    const int tree = out_ix / warps;
    const int raw = out_selected_node[out_ix];
    const int plen = out_path_len[out_ix];
    const int node_cnt = tree_nodes[tree];
    if (node_cnt <= 0 || node_cnt > nodes || node_cnt > NODE_LIMIT) return;
    if (raw < 0) return;
    const int kind = (raw >> KIND_SHIFT) & 7;
    if (kind == INVALID || kind == BUSY) return;
    if (plen <= 0) return;
    const long long tree_edges_base = (long long)tree * nodes * edges;
    const int *path = out_path_eids + (long long)out_ix * path_depth;
    for (int d = at_work.lane; d < plen - 1; d += 1 << log2_lanes) {
        const int enc = path[d];
        const float value = path_edge_values ? path_edge_values[(long long)out_ix * path_depth + d] : 0.f;
        if (enc < 0) continue;
        const int parent = enc >> 8, slot = enc & 0xFF;
        if (parent < node_cnt && slot < edges) {
            const long long ix = tree_edges_base + (long long)parent * edges + slot;
            atomicSub(&edge_inflight[ix], virtual_loss);
            if (path_edge_values) {
                atomicAdd(&edge_N[ix], 1);
                atomicAdd(&edge_W[ix], value);
            }
        }
    }
    if (at_work.lane == 0 && kind == EXPAND) {
        const int leaf = raw & NODE_MASK;
        if (leaf < node_cnt) atomicSub(&node_expand_inflight[(long long)tree * nodes + leaf], 1);
    }
}

static int launch_select(float cpuct, float c_pw, float alpha_pw, int soft_winner, int virtual_loss, const int *edge_child_id,
                         const float *edge_prior, const float *edge_W, const int *edge_N, int *edge_inflight,
                         int *node_expand_inflight, const int *node_expanded, const int *tree_nodes, int *out_selected_node,
                         int *out_path_eids, int *out_path_len, int trees, int nodes, int edges, int warps, int path_depth,
                         cudaStream_t stream) {
    const unsigned grid = (unsigned)((long long)trees * warps);
    if (c_pw == 0.0f && roots_first(trees, edges, warps)) {
#define PUCT_LAUNCH(E)                                                                                                     \
    do {                                                                                                                  \
        select_math::launch_behind(root_kernel<E>, ((unsigned)trees + ROOT_WARPS - 1) / ROOT_WARPS, ROOT_WARPS * 32, stream, cpuct, soft_winner, edge_child_id, edge_prior, edge_W, edge_N, edge_inflight,       \
                                                    node_expanded, tree_nodes, out_selected_node, out_path_eids,           \
                                                    out_path_len, trees, nodes, edges, warps, path_depth, virtual_loss);   \
        select_math::launch_behind(select_kernel<E, false, true>, grid, 32, stream,                                                            \
            cpuct, c_pw, alpha_pw, soft_winner, edge_child_id, edge_prior, edge_W, edge_N, edge_inflight,                  \
            node_expand_inflight, node_expanded, tree_nodes, out_selected_node, out_path_eids, out_path_len, nodes, edges, \
            warps, path_depth, virtual_loss, trees);                                                                   \
    } while (0)
        if (edges <= 32) PUCT_LAUNCH(1);
        else if (edges <= 64) PUCT_LAUNCH(2);
        else if (edges <= 128) PUCT_LAUNCH(4);
        else PUCT_LAUNCH(8);
#undef PUCT_LAUNCH
        return (int)cudaGetLastError();
    }
#define PUCT_LAUNCH_AS(E, W)                                                                                              \
    select_math::launch_behind(select_kernel<E, W, false>, grid, 32, stream, cpuct, c_pw, alpha_pw, soft_winner, edge_child_id, edge_prior, edge_W,     \
                                                 edge_N, edge_inflight, node_expand_inflight, node_expanded, tree_nodes,    \
                                                 out_selected_node, out_path_eids, out_path_len, nodes, edges, warps,       \
                                                 path_depth, virtual_loss, trees)
#define PUCT_LAUNCH(E)                        \
    do {                                      \
        if (c_pw != 0.0f) PUCT_LAUNCH_AS(E, true); \
        else PUCT_LAUNCH_AS(E, false);        \
    } while (0)
    if (edges <= 32) PUCT_LAUNCH(1);
    else if (edges <= 64) PUCT_LAUNCH(2);
    else if (edges <= 128) PUCT_LAUNCH(4);
    else PUCT_LAUNCH(8);   // more than 256 edges: the kernel itself reports the invalid shape
#undef PUCT_LAUNCH
#undef PUCT_LAUNCH_AS
    return (int)cudaGetLastError();
}

}  // namespace puct

// Same arguments and meaning as puct_select_winner_recalc_launch of src/puct/puct_gpu_v3_cpp.cu:450-481.
extern "C" int puct_select_winner_recalc_launch(float cpuct, float c_pw, float alpha_pw, int soft_winner, const int *edge_child_id,
                                                const float *edge_prior, const float *edge_W, const int *edge_N,
                                                int *edge_inflight, int *node_expand_inflight, const int *node_expanded,
                                                const int *tree_nodes, int *out_selected_node, int *out_path_eids,
                                                int *out_path_len, int trees, int nodes, int edges, int warps, int path_depth,
                                                void *stream) {
    if (trees <= 0 || warps <= 0 || warps > 32) return (int)cudaErrorInvalidValue;
    return puct::launch_select(cpuct, c_pw, alpha_pw, soft_winner, 1, edge_child_id, edge_prior, edge_W, edge_N, edge_inflight,
                                  node_expand_inflight, node_expanded, tree_nodes, out_selected_node, out_path_eids,
                                  out_path_len, trees, nodes, edges, warps, path_depth, (cudaStream_t)stream);
}

// The same select with a virtual-loss weight other than 1 (an extension: the reference's select always claims 1).
extern "C" int puct_select_virtual_loss_launch(float cpuct, float c_pw, float alpha_pw, int soft_winner, int virtual_loss,
                                               const int *edge_child_id, const float *edge_prior, const float *edge_W,
                                               const int *edge_N, int *edge_inflight, int *node_expand_inflight,
                                               const int *node_expanded, const int *tree_nodes, int *out_selected_node,
                                               int *out_path_eids, int *out_path_len, int trees, int nodes, int edges, int warps,
                                               int path_depth, void *stream) {
    if (trees <= 0 || warps <= 0 || warps > 32 || virtual_loss < 1) return (int)cudaErrorInvalidValue;
    return puct::launch_select(cpuct, c_pw, alpha_pw, soft_winner, virtual_loss, edge_child_id, edge_prior, edge_W, edge_N,
                                  edge_inflight, node_expand_inflight, node_expanded, tree_nodes, out_selected_node,
                                  out_path_eids, out_path_len, trees, nodes, edges, warps, path_depth, (cudaStream_t)stream);
}

// Backup of finished traversals (path_edge_values: float[trees][warps][path_depth], already seen from the side of the
// player who took the edge) or, with path_edge_values == NULL, release of their claims only.
extern "C" int puct_backup_launch(int virtual_loss, float *edge_W, int *edge_N, int *edge_inflight, int *node_expand_inflight,
                                  const int *tree_nodes, const int *out_selected_node, const int *out_path_eids,
                                  const int *out_path_len, const float *path_edge_values, int trees, int nodes, int edges,
                                  int warps, int path_depth, void *stream) {
    if (trees <= 0 || warps <= 0 || warps > 32) return (int)cudaErrorInvalidValue;
    if ((long long)trees * warps > 0x7FFFFFFF) return (int)cudaErrorInvalidValue;
    const select_math::BackupGrid g(trees * warps, path_depth);
    select_math::launch_behind(puct::backup_kernel, g.blocks, g.THREADS, (cudaStream_t)stream, virtual_loss, edge_W, edge_N, edge_inflight, node_expand_inflight,
                                                                          tree_nodes, out_selected_node, out_path_eids, out_path_len,
                                                                          path_edge_values, trees * warps, nodes, edges, warps,
                                                                          path_depth, g.log2_lanes);
    return (int)cudaGetLastError();
}

extern "C" const char *puct_select_kernel_name(float c_pw, int trees, int edges, int warps) {
    return c_pw == 0.0f && puct::roots_first(trees, edges, warps) ? "puct::root_kernel + puct::select_kernel" : "puct::select_kernel";
}

// Same meaning as puct_cpp_cuda_error_string of src/puct/puct_gpu_v3_cpp.cu:483-485.
extern "C" const char *puct_cpp_cuda_error_string(int code) { return cudaGetErrorString(static_cast<cudaError_t>(code)); }
