// The two older PUCT select kernels of the reference and their backup, for trees whose virtual visits are kept per
// child NODE (node_inflight[tree, node]) instead of per edge:
//   preclaim      _select_kernel_native        src/puct/puct_gpu_v2.py:573-697   every candidate child gets +1 before it is
//                                              scored, the losers give theirs back
//   counter-CAS   _select_kernel_winner_recalc src/puct/puct_gpu_v2.py:700-840   the winner alone is claimed, by
//                                              compare-and-swap on the counter; a claim that met other visits is given
//                                              back once and the choice repeated without that edge
//   backup        _backup_kernel_native        src/puct/puct_gpu_v2.py:847-927
// Semantics followed, not the code.  Results are packed (kind << 22) | (slot << 14) | node without reason bits, a failed
// traversal rolls its path back and reports INVALID (there is no BUSY kind in this layout), path entries are
// (parent << 8) | slot.
//
// What is done differently: one traversal per block of one warp (see puct_select.cu), up to 8 edges a lane held in registers,
// and a level made of as few dependent memory round trips as the layout allows.  All edge arrays of a child and its record
// are requested together as soon as the child is known; then the children's visit counters follow, one more round trip:
// preclaim takes them from its own visits (an atomic add returns the count before it), without reading them first where nobody
// else visits the tree and progressive widening cannot end the traversal there (a child that several edges of the node lead to
// gets several visits of the one traversal, which are taken out of the parent's count again); counter-CAS claims with the count
// it has read and looks at the answer when the child's own edges have arrived.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/puct_b200.h"
#include "select_math.cuh"

namespace puct_v2 {

using namespace select_math;

constexpr int NODE_TERMINAL = -1;
constexpr int NODE_LIMIT = 16384, NODE_MASK = 0x3FFF, EDGE_LIMIT = 256;
constexpr int KIND_SHIFT = 22, SLOT_SHIFT = 14;
enum Kind { INVALID = 0, EXPAND = 1, TERMINAL = 2, DEPTH_LIMIT = 3 };
constexpr int PACKED_INVALID = (INVALID << KIND_SHIFT) | NODE_MASK;
constexpr int MAX_CLAIM_RETRY = 8;   // compare-and-swap attempts before the claim falls back to an atomic add (:328-347)
constexpr int MAX_RECALC = 2;        // evaluations of a level by the counter-CAS variant (:528-560)
constexpr int NO_EDGE = 0x7FFFFFFF;

__device__ __forceinline__ int pack(int kind, int node, int slot) { return (kind << KIND_SHIFT) | (slot << SLOT_SHIFT) | node; }

__device__ __forceinline__ unsigned ordered(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// a counter that can take a visit: not a corrupt (negative) one, nor one at its largest value (:328-347)
__device__ __forceinline__ bool claimable(int count) { return (unsigned)count < 0x7FFFFFFFu; }

// give back the visit of every child on the first `depth` path entries (:291-311)
__device__ __forceinline__ void rollback(const int *path, int depth, int lane, const int *edge_child_id, int *node_inflight,
                                         long long tree_nodes_base, long long tree_edges_base, int node_cnt, int edges) {
    __syncwarp();   // lane 0 wrote the entries
    for (int d = lane; d < depth; d += 32) {
        const int enc = path[d];
        if (enc < 0) continue;
        const int parent = enc >> 8, slot = enc & 0xFF;
        if (parent < node_cnt && slot < edges) {
            const int child = edge_child_id[tree_edges_base + (long long)parent * edges + slot];
            if (child >= 0 && child < node_cnt) atomicSub(&node_inflight[tree_nodes_base + child], 1);
        }
    }
}

// The edges of one node as seen by one lane (edge lane + 32 k in slot k) with the visits of their children.  Slots beyond the
// array's `edges` keep harmless values.
template <int EPL>
struct EdgeRegs {
    const int *child_of, *n_of;   // of this tree
    const float *prior_of, *w_of;
    float prior[EPL], w[EPL];
    int n[EPL], child[EPL], visits[EPL];

    __device__ __forceinline__ void init(long long tree_edges, const int *edge_child_id, const float *edge_prior, const float *edge_W,
                                         const int *edge_N) {
        child_of = edge_child_id + tree_edges;
        prior_of = edge_prior + tree_edges;
        w_of = edge_W + tree_edges;
        n_of = edge_N + tree_edges;
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            prior[k] = w[k] = 1.f;
            n[k] = 1;
            visits[k] = 0;
            child[k] = -1;
        }
    }

    // all `edges` slots of a node, expanded or not: before the number of expanded edges is known
    __device__ __forceinline__ void request(int node, int lane, int edges) {
        const unsigned first = (unsigned)(node * edges + lane) * 4u;   // < 2^24
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (lane + 32 * k < edges) {
                child[k] = *at(child_of, first + 128u * k);
                n[k] = *at(n_of, first + 128u * k);
                prior[k] = *at(prior_of, first + 128u * k);
                w[k] = *at(w_of, first + 128u * k);
            }
    }

    // edges that do not lead anywhere are marked by child = -1
    __device__ __forceinline__ void drop_invalid(int lane, int n_exp, int node_cnt) {
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (lane + 32 * k >= n_exp || (unsigned)child[k] >= (unsigned)node_cnt) child[k] = -1;
    }

    __device__ __forceinline__ void read_visits(const int *node_inflight) {
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (child[k] >= 0) visits[k] = *(volatile const int *)&node_inflight[child[k]];
    }

    // Whether the `n_exp` children, taken round in a circle, rise but for one place: then they all differ.  So they do where the
    // children of a node were made one after the other or all at once.  About 5 instructions an edge slot, in the shadow of the
    // visits' answers: select and release 16.2 -> 16.6 us with 1000 trees x 82 edges x 9 levels, 28.4 -> 29.3 with 4096 x 64 x 12;
    // reading the counters in front of the visits instead takes 19.5 and 30.6.
    __device__ __forceinline__ bool children_ascend(int lane, int n_exp) const {
        int next[EPL], rises = 0;
        const int first = __shfl_sync(FULL, child[0], 0);
#pragma unroll
        for (int k = 0; k < EPL; k++) next[k] = __shfl_sync(FULL, child[k], (lane + 1) & 31);
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            const int e = lane + 32 * k;
            const int after = e + 1 == n_exp ? first : (lane == 31 ? (k + 1 < EPL ? next[k + 1 < EPL ? k + 1 : k] : -1) : next[k]);
            rises += after > child[k] ? 1 : 0;   // none from -1 to -1, behind the last child
        }
        return __reduce_add_sync(FULL, rises) >= n_exp - 1;
    }

    __device__ __forceinline__ int parent_count() const {   // :418-427
        int partial = 0;
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (child[k] >= 0) partial += n[k] + visits[k];
        return max(__reduce_add_sync(FULL, partial), 1);
    }

    // order-preserving keys of the scores; 0: no edge there, or a NaN, which never wins
    __device__ __forceinline__ void keys(float cpuct, float sqrt_parent, unsigned *key) const {
        float score[EPL];
        bool plain = true;
#pragma unroll
        for (int k = 0; k < EPL; k++) {
            const bool visited = n[k] > 0;
            const float up = cpuct * prior[k] * sqrt_parent;
            const int tries = n[k] + visits[k] + 1;
            const float mean = Count(visited ? n[k] : 1).divides(w[k]);
            score[k] = (visited ? mean : 0.0f) + Count(tries).divides(up);
            plain = plain && (child[k] < 0 || ((unsigned)((tries - 1) | n[k]) < (1u << 22) && Count::plain(w[k], up)));
        }
        if (!plain) {   // counts of millions, or values no network gives
#pragma unroll
            for (int k = 0; k < EPL; k++) {
                const float q = n[k] > 0 ? w[k] / (float)n[k] : 0.0f;
                score[k] = q + cpuct * prior[k] * sqrt_parent / (float)(n[k] + visits[k] + 1);
            }
        }
#pragma unroll
        for (int k = 0; k < EPL; k++) key[k] = child[k] >= 0 && score[k] == score[k] ? ordered(score[k]) : 0u;
    }
};

__device__ __forceinline__ int widening_quota(float c_pw, float alpha_pw, int parent_eff, int edges) {   // :237-262
    const float quota = (alpha_pw == 0.5f) ? c_pw * root_of_count(parent_eff) : c_pw * powf((float)parent_eff, alpha_pw);
    return quota >= (float)edges ? edges : max(1, (int)ceilf(quota));
}

// ticket per node: distinct slots for traversals that expand the same node together (:397-414); -1: no room left
__device__ __forceinline__ int expansion_ticket(int *tickets, int n_exp, int allowed, int lane) {
    int slot = -1;
    if (lane == 0) {
        const int s = n_exp + atomicAdd(tickets, 1);
        if (s < allowed) slot = s;
        else atomicSub(tickets, 1);
    }
    return __shfl_sync(FULL, slot, 0);
}

// PRECLAIM: true = _select_kernel_native, false = the counter-CAS variant.  WIDENING: c_pw is not zero; for preclaim it stands
// for reading the visits before making any, so it is set for several traversals per tree too (a traversal that is alone in its
// tree learns from its own visits what it would read before them).
template <bool PRECLAIM, int EPL, bool WIDENING>
__global__ void __launch_bounds__(32, EPL <= 2 ? 32 : (EPL == 4 ? 24 : 16))
select_kernel(float cpuct, float c_pw, float alpha_pw, const int *edge_child_id, const float *edge_prior,
              const float *edge_W, const int *edge_N, int *node_inflight_all, int *node_expand_inflight,
              const int *node_expanded, const int *tree_nodes, int *out_selected_node, int *out_path_eids,
              int *out_path_len, int nodes, int edges, int warps, int path_depth) {
    let_the_next_kernel_come();
    const unsigned block = block_after_the_kernel_before();
    const int lane = threadIdx.x;
    const int traversal = block;
    const int tree = traversal / warps;
    const int wid = traversal - tree * warps;
    int *path = out_path_eids + (long long)traversal * path_depth;
    int result = PACKED_INVALID, result_len = 0;
    const int node_cnt = tree_nodes[tree];
    const bool shape_ok = path_depth >= 1 && nodes > 0 && node_cnt > 0 && node_cnt <= nodes && node_cnt <= NODE_LIMIT && edges > 0 &&
                          edges <= EDGE_LIMIT;
    const long long tree_nodes_base = (long long)tree * nodes;
    const long long tree_edges_base = tree_nodes_base * edges;
    int *node_inflight = node_inflight_all + tree_nodes_base;
    const int *expanded = node_expanded + tree_nodes_base;
    EdgeRegs<EPL> r;
    int node = 0, depth = 0, info = 0;
    if (shape_ok) {
        r.init(tree_edges_base, edge_child_id, edge_prior, edge_W, edge_N);
        info = expanded[0];
        r.request(0, lane, edges);
    }
    // counter-CAS: the claim made on the level above, until its answer is needed, and what a second choice there needs
    bool pending = false;
    int up_node = 0, up_info = 0, up_best = 0, up_child = 0, up_seen = 0, up_old = 0, up_attempt = 0;
    int attempt = 0, skip = -1;
    float sqrt_parent = 0.f, up_sqrt = 0.f;
    while (shape_ok) {
        if (!PRECLAIM && pending) {
            pending = false;
            // compare-and-swap old -> old + 1 on the child's counter; `conflict` = somebody was there already
            int claim = 0;   // bit 0: held, bit 1: conflict
            if (lane == (up_best & 31)) {
                int *counter = node_inflight + up_child;
                bool can_claim = true, got = claimable(up_seen) && up_old == up_seen;
                int old = up_old;
                if (got) old = up_seen;
                for (int t = 1; t < MAX_CLAIM_RETRY && !got; t++) {
                    if (!claimable(old)) {
                        can_claim = false;
                        break;
                    }
                    const int now = atomicCAS(counter, old, old + 1);
                    got = now == old;
                    if (!got) old = now;
                }
                if (!got && can_claim) {
                    old = atomicAdd(counter, 1);
                    got = true;
                }
                claim = (got ? 1 : 0) | ((got && old > 0) ? 2 : 0);
            }
            claim = __shfl_sync(FULL, claim, up_best & 31);
            if (!(claim & 1)) {
                rollback(path, depth - 1, lane, edge_child_id, node_inflight_all, tree_nodes_base, tree_edges_base, node_cnt, edges);
                break;
            }
            if ((claim & 2) && up_info > 1 && up_attempt + 1 < MAX_RECALC) {
                // given back once, and the choice repeated without that edge (:528-560)
                if (lane == 0) atomicSub(node_inflight + up_child, 1);
                __syncwarp();
                depth--;
                node = up_node;
                info = up_info;
                attempt = up_attempt + 1;
                skip = up_best;
                sqrt_parent = up_sqrt;
                r.request(node, lane, edges);
            }
        }
        if (depth >= path_depth) {
            result = pack(DEPTH_LIMIT, node, 0);
            result_len = depth + 1;
            break;
        }
        if (info == NODE_TERMINAL) {
            result = pack(TERMINAL, node, 0);
            result_len = depth + 1;
            break;
        }
        if (info < 0 || info > edges) {
            rollback(path, depth, lane, edge_child_id, node_inflight_all, tree_nodes_base, tree_edges_base, node_cnt, edges);
            break;
        }
        const int n_exp = info;
        r.drop_invalid(lane, n_exp, node_cnt);
        if (!PRECLAIM || (WIDENING && n_exp != 0)) r.read_visits(node_inflight);
        if (attempt == 0) {
            int allowed = 1;   // the preclaim kernel lets a node without children expand exactly one (:646)
            if (WIDENING && (!PRECLAIM || n_exp != 0)) allowed = widening_quota(c_pw, alpha_pw, r.parent_count(), edges);
            if (allowed > n_exp) {
                const int slot = expansion_ticket(&node_expand_inflight[tree_nodes_base + node], n_exp, allowed, lane);
                if (slot >= 0) {
                    result = pack(EXPAND, node, slot);
                    result_len = depth + 1;
                } else {
                    rollback(path, depth, lane, edge_child_id, node_inflight_all, tree_nodes_base, tree_edges_base, node_cnt, edges);
                }
                break;
            }
        }
        unsigned key[EPL];
        int best = NO_EDGE, my_child = -1, my_seen = 0;
        if (PRECLAIM) {
            // every candidate's child is visited first, scored with the count it had before, then the losers leave (:448-483)
            if (WIDENING) sqrt_parent = root_of_count(r.parent_count());   // of the counts read before the visits
#pragma unroll
            for (int k = 0; k < EPL; k++)
                if (r.child[k] >= 0) r.visits[k] = atomicAdd(node_inflight + r.child[k], 1);
            if (!WIDENING) {
                int parent_eff;
                if (r.children_ascend(lane, n_exp)) {
                    parent_eff = r.parent_count();
                } else {
                    // Where m edges lead to one child, every visit but the first has met those before it: the m answers hold
                    // m (m - 1) / 2 visits of this traversal's own.  By as many the counter, now that all are made, exceeds
                    // answer + 1, summed over the m edges.
                    __syncwarp();
                    int partial = 0;
#pragma unroll
                    for (int k = 0; k < EPL; k++)
                        if (r.child[k] >= 0)
                            partial += r.n[k] + 2 * r.visits[k] + 1 - *(volatile const int *)&node_inflight[r.child[k]];
                    parent_eff = max(__reduce_add_sync(FULL, partial), 1);
                }
                sqrt_parent = root_of_count(parent_eff);
            }
        } else if (attempt == 0) {
            sqrt_parent = root_of_count(r.parent_count());
        }
        r.keys(cpuct, sqrt_parent, key);
        {
            // ties: preclaim, the edge closest after the warp's index; counter-CAS, the lowest edge (:110-119)
            const int rot = !PRECLAIM || wid < n_exp ? (PRECLAIM ? wid : 0) : (n_exp > 0 ? wid % n_exp : 0);
            unsigned my_key = 0;
            int my_tie = NO_EDGE;
#pragma unroll
            for (int k = 0; k < EPL; k++) {
                const int e = lane + 32 * k;
                const int tie = e >= rot ? e - rot : e - rot + n_exp;
                if (key[k] != 0u && (PRECLAIM || e != skip) && (key[k] > my_key || (key[k] == my_key && tie < my_tie))) {
                    my_key = key[k];
                    my_tie = tie;
                    my_child = r.child[k];
                    my_seen = r.visits[k];
                }
            }
            const unsigned top = __reduce_max_sync(FULL, my_key);
            const unsigned tie = __reduce_min_sync(FULL, my_key == top ? (unsigned)my_tie : (unsigned)NO_EDGE);
            if (top != 0u) best = (int)tie + rot >= n_exp ? (int)tie + rot - n_exp : (int)tie + rot;
        }
        const bool again = !PRECLAIM && best == NO_EDGE && skip >= 0;
        if (again) {
            best = skip;   // only the edge given back is left: take it after all (:533-536)
            my_child = up_child;
            my_seen = *(volatile int *)(node_inflight + up_child);
        }
        const int child = best == NO_EDGE ? -1 : __shfl_sync(FULL, my_child, best & 31);
        int next_info = 0;
        const int now = node;
        if (PRECLAIM) {
            // the losers' children, before the registers take the next level's edges
            int loser[EPL];
#pragma unroll
            for (int k = 0; k < EPL; k++) loser[k] = lane + 32 * k != best ? r.child[k] : -1;
            if (child >= 0) {
                next_info = expanded[child];
                r.request(child, lane, edges);
            }
#pragma unroll
            for (int k = 0; k < EPL; k++)
                if (loser[k] >= 0) atomicSub(node_inflight + loser[k], 1);
        } else if (child >= 0) {
            next_info = expanded[child];
            r.request(child, lane, edges);
            // predicated, so that nothing behind it waits for the answer; a count that cannot take a visit is only read
            asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %4, %5;\n\t@p atom.global.cas.b32 %0, [%1], %2, %3;\n\t}"
                         : "+r"(up_old) : "l"(node_inflight + child), "r"(my_seen), "r"(claimable(my_seen) ? my_seen + 1 : my_seen), "r"(lane),
                           "r"(best & 31) : "memory");
            pending = true;
            up_node = node;
            up_info = info;
            up_best = best;
            up_child = child;
            up_seen = my_seen;
            up_attempt = attempt;
            up_sqrt = sqrt_parent;
        }
        if (child < 0) {
            rollback(path, depth, lane, edge_child_id, node_inflight_all, tree_nodes_base, tree_edges_base, node_cnt, edges);
            break;
        }
        if (lane == 0) path[depth] = (now << 8) | best;
        node = child;
        info = next_info;
        attempt = 0;
        skip = -1;
        depth++;
    }
    if (lane == 0) {
        out_selected_node[traversal] = result;
        out_path_len[traversal] = result_len;
    }
}

// _backup_kernel_native (:847-927): per path edge the child's visit is given back, the edge gets N += 1 and W += value;
// an EXPAND result returns its ticket.  With values == NULL only the visits and the ticket are released.
__global__ void backup_kernel(int virtual_loss, const int *edge_child_id, float *edge_W, int *edge_N,
                              int *node_inflight, int *node_expand_inflight, const int *tree_nodes,
                              const int *out_selected_node, const int *out_path_eids,
                              const int *out_path_len, const float *path_edge_values, int traversals, int nodes,
                              int edges, int warps, int path_depth, int log2_lanes) {
    const BackupLane at_work(block_after_the_kernel_before(), traversals, log2_lanes);
    const int traversal = at_work.traversal;
    if (traversal < 0) return;
    const int tree = traversal / warps;
    const int raw = out_selected_node[traversal];
    const int plen = out_path_len[traversal];
    const int node_cnt = tree_nodes[tree];
    if (node_cnt <= 0 || node_cnt > nodes || node_cnt > NODE_LIMIT) return;
    if (raw < 0 || (raw >> KIND_SHIFT) == INVALID) return;
    if (plen <= 0) return;
    const long long tree_nodes_base = (long long)tree * nodes, tree_edges_base = tree_nodes_base * edges;
    const int *path = out_path_eids + (long long)traversal * path_depth;
    for (int d = at_work.lane; d < plen - 1; d += 1 << log2_lanes) {
        const int enc = path[d];
        const float value = path_edge_values ? path_edge_values[(long long)traversal * path_depth + d] : 0.f;
        if (enc < 0) continue;
        const int parent = enc >> 8, slot = enc & 0xFF;
        if (parent < node_cnt && slot < edges) {
            const long long ix = tree_edges_base + (long long)parent * edges + slot;
            const int child = edge_child_id[ix];
            if (child >= 0 && child < node_cnt) atomicSub(&node_inflight[tree_nodes_base + child], virtual_loss);
            if (path_edge_values) {
                atomicAdd(&edge_N[ix], 1);
                atomicAdd(&edge_W[ix], value);
            }
        }
    }
    if (at_work.lane == 0 && (raw >> KIND_SHIFT) == EXPAND) {
        const int leaf = raw & NODE_MASK;
        if (leaf < node_cnt) atomicSub(&node_expand_inflight[tree_nodes_base + leaf], 1);
    }
}

}  // namespace puct_v2

// variant 0: preclaim (the reference's _select_kernel_native), 1: counter-CAS (_select_kernel_winner_recalc of
// src/puct/puct_gpu_v2.py).  Array shapes as for puct_select_winner_recalc_launch, with node_inflight int32[trees][nodes]
// in place of the per-edge counters.
extern "C" int puct_v2_select_launch(int variant, float cpuct, float c_pw, float alpha_pw, const int *edge_child_id,
                                     const float *edge_prior, const float *edge_W, const int *edge_N, int *node_inflight,
                                     int *node_expand_inflight, const int *node_expanded, const int *tree_nodes,
                                     int *out_selected_node, int *out_path_eids, int *out_path_len, int trees, int nodes, int edges,
                                     int warps, int path_depth, void *stream) {
    if (trees <= 0 || warps <= 0 || warps > 32 || (variant != 0 && variant != 1)) return (int)cudaErrorInvalidValue;
    const unsigned grid = (unsigned)((long long)trees * warps);
    const cudaStream_t s = (cudaStream_t)stream;
#define PUCT_V2_LAUNCH(P, E, W)                                                                                              \
    select_math::launch_behind(puct_v2::select_kernel<P, E, W>, grid, 32, s, cpuct, c_pw, alpha_pw, edge_child_id, edge_prior, edge_W, edge_N,    \
                                                        node_inflight, node_expand_inflight, node_expanded, tree_nodes,      \
                                                        out_selected_node, out_path_eids, out_path_len, nodes, edges, warps, \
                                                        path_depth)
#define PUCT_V2_LAUNCH_EDGES(P, W)             \
    do {                                       \
        if (edges <= 32) PUCT_V2_LAUNCH(P, 1, W);       \
        else if (edges <= 64) PUCT_V2_LAUNCH(P, 2, W);  \
        else if (edges <= 128) PUCT_V2_LAUNCH(P, 4, W); \
        else PUCT_V2_LAUNCH(P, 8, W);                   \
    } while (0)
    if (variant == 0 && (c_pw != 0.0f || warps > 1)) PUCT_V2_LAUNCH_EDGES(true, true);
    else if (variant == 0) PUCT_V2_LAUNCH_EDGES(true, false);
    else if (c_pw != 0.0f) PUCT_V2_LAUNCH_EDGES(false, true);
    else PUCT_V2_LAUNCH_EDGES(false, false);
#undef PUCT_V2_LAUNCH_EDGES
#undef PUCT_V2_LAUNCH
    return (int)cudaGetLastError();
}

extern "C" int puct_v2_backup_launch(int virtual_loss, const int *edge_child_id, float *edge_W, int *edge_N, int *node_inflight,
                                     int *node_expand_inflight, const int *tree_nodes, const int *out_selected_node,
                                     const int *out_path_eids, const int *out_path_len, const float *path_edge_values, int trees,
                                     int nodes, int edges, int warps, int path_depth, void *stream) {
    if (trees <= 0 || warps <= 0 || warps > 32) return (int)cudaErrorInvalidValue;
    if ((long long)trees * warps > 0x7FFFFFFF) return (int)cudaErrorInvalidValue;
    const select_math::BackupGrid g(trees * warps, path_depth);
    select_math::launch_behind(puct_v2::backup_kernel, g.blocks, g.THREADS, (cudaStream_t)stream, virtual_loss, edge_child_id, edge_W, edge_N, node_inflight,
                                                                             node_expand_inflight, tree_nodes, out_selected_node,
                                                                             out_path_eids, out_path_len, path_edge_values,
                                                                             trees * warps, nodes, edges, warps, path_depth,
                                                                             g.log2_lanes);
    return (int)cudaGetLastError();
}
