// Decoupled-UCT (DUCT) select and backup for simultaneous-move games: two players, A actions each (A <= 16), a child
// per joint action.  NO COUNTERPART IN THE REFERENCE: src/puct holds only the single-agent PUCT select; the benchmark
// configuration "DUCT 2 x 8 joint actions" names a variant the reference does not implement, so the semantics below are
// this library's own (stated in include/duct_b200.h and restated on the CPU in oracle/duct_oracle.py) and parity is
// unpinned by construction.  The conventions of the PUCT select are kept where they apply: path entries (node << 8) | slot,
// packed results reason << 25 | kind << 22 | slot << 14 | node, virtual loss claimed on the way down and returned by the backup.
//
// A level costs one memory round trip: the lanes of a traversal hold the statistics of one action each and, next to them,
// their share of the node's A*A child ids, all requested together with the node's terminal flag; when both players have
// picked, the child is known from a register, and its data is requested before the claims' answers are waited for.
// A warp runs as many traversals as fit: 8 lanes a player (two traversals) up to 8 actions, 4 lanes (four) up to 4; fewer
// warps then share the issue slots and more traversals are on the device at once.  4096 trees x 8 traversals x 16 levels, 8
// actions: 275 us with a traversal per warp and the claims waited for, 157 us so.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/duct_b200.h"
#include "select_math.cuh"

namespace duct {

using namespace select_math;

constexpr int MAX_ACTIONS = 16, NODE_LIMIT = 16384;
constexpr int KIND_SHIFT = 22, SLOT_SHIFT = 14, REASON_SHIFT = 25;
constexpr int CHILD_NONE = -1, CHILD_CLAIMED = -2;
enum Kind { INVALID = 0, EXPAND = 1, TERMINAL = 2, DEPTH_LIMIT = 3, BUSY = 4 };
enum Reason { R_UNSET = 0, R_OK_EXPAND = 1, R_OK_TERMINAL = 2, R_OK_DEPTH_LIMIT = 3, R_BUSY_EXPAND_INFLIGHT = 4,
              R_INVALID_SHAPE = 10, R_INVALID_CHILD_OOB = 15 };
constexpr int MAX_EVALUATIONS = 3;  // arg-max evaluations of a player at one node before its pick is claimed regardless

__device__ __forceinline__ int pack(int kind, int node, int slot, int reason) {
    return (reason << REASON_SHIFT) | (kind << KIND_SHIFT) | (slot << SLOT_SHIFT) | node;
}

__device__ __forceinline__ unsigned ordered(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// score of one action of one player; every operation rounds once, in this order (the CPU restatement does the same)
__device__ __forceinline__ float score(float cpuct, float prior, float w, int n, int inflight, int virtual_loss, float sqrt_total) {
    const int n_eff = n + virtual_loss * inflight;
    const float w_eff = __fsub_rn(w, (float)(virtual_loss * inflight));  // a traversal in flight counts as a loss
    const float up = __fmul_rn(__fmul_rn(cpuct, prior), sqrt_total);
    if ((unsigned)n_eff < (1u << 22) && Count::plain(w_eff, up)) {
        const float q = Count(max(n_eff, 1)).divides(w_eff);
        return __fadd_rn(n_eff > 0 ? q : 0.f, Count(n_eff + 1).divides(up));
    }
    const float q = n_eff > 0 ? __fdiv_rn(w_eff, (float)n_eff) : 0.f;
    return __fadd_rn(q, __fdiv_rn(up, (float)(1 + n_eff)));
}

// Blocks of eight warps: the traversals of a tree start on one SM together, as they did with a block per tree, and meet each
// other's claims in the same way (blocks of two warps: 4096 trees x 8 traversals 150 instead of 157 us).
constexpr int WARPS_PER_BLOCK = 8;

// LANES lanes per player, action = lane within them; 2 * LANES lanes per traversal, the traversals of a warp side by side
template <int LANES>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32)
select_kernel(float cpuct, int virtual_loss, int *child_all, const float *__restrict__ node_prior, const float *__restrict__ node_w,
              const int *__restrict__ node_n, int *node_inflight_all, const int *__restrict__ node_terminal,
              const int *__restrict__ tree_nodes, int *out_selected, int *out_path, int *out_len, int trees, int nodes, int A, int warps,
              int path_depth) {
    constexpr int GROUP = 2 * LANES, PER_WARP = 32 / GROUP;
    constexpr int SLOTS = (LANES * LANES + GROUP - 1) / GROUP;   // child ids a lane may hold
    const int lane = threadIdx.x & 31;
    const int sub = lane & (GROUP - 1), base = lane & ~(GROUP - 1);   // lane within the traversal, its first lane
    const int player = sub / LANES, action = sub & (LANES - 1);
    // the traversals of a warp belong to neighbouring trees (those of one tree would lose each other's claims in step)
    const int unit = (int)blockIdx.x * WARPS_PER_BLOCK + (int)(threadIdx.x >> 5);
    const int first_tree = unit / warps * PER_WARP, wid = unit % warps;
    const bool exists = first_tree + lane / GROUP < trees;
    const int tree = exists ? first_tree + lane / GROUP : 0;
    const int out = tree * warps + wid;
    int *path = out_path + (long long)out * path_depth;
    const int node_cnt = tree_nodes[tree];
    const bool has_action = action < A;
    const int joints = A * A;
    const long long tree_nodes_base = (long long)tree * nodes;
    const long long stats_base = tree_nodes_base * 2 * A;
    int *child_of = child_all + tree_nodes_base * joints;
    int *inflight_of = node_inflight_all + stats_base;
    const float *prior_of = node_prior + stats_base, *w_of = node_w + stats_base;
    const int *n_of = node_n + stats_base, *terminal_of = node_terminal + tree_nodes_base;

    float prior = 0.f, w = 0.f;
    int n = 0, inflight = 0, terminal = 0, kids[SLOTS];
    // everything a level needs, requested together
    auto request = [&](int at_node) {
        const int s = at_node * 2 * A + player * A + action;
        if (has_action) {
            prior = prior_of[s];
            w = w_of[s];
            n = n_of[s];
            inflight = *(volatile const int *)&inflight_of[s];
        }
#pragma unroll
        for (int k = 0; k < SLOTS; k++) {
            const int j = sub + GROUP * k;
            if (j < joints) kids[k] = *(volatile const int *)&child_of[at_node * joints + j];
        }
        terminal = terminal_of[at_node];
    };
    // gives back the claims of the first `count` path entries of the traversal
    auto rollback = [&](int count) {
        for (int d = sub; d < count; d += GROUP) {
            const int enc = path[d];
            const int joint = enc & 0xFF, s0 = (enc >> 8) * 2 * A;
            atomicSub(&inflight_of[s0 + joint / A], virtual_loss);
            atomicSub(&inflight_of[s0 + A + joint % A], virtual_loss);
        }
    };
    int node = 0, depth = 0, result = pack(INVALID, 0, 0, R_UNSET);
    bool going = exists;
    if (exists && (node_cnt <= 0 || node_cnt > nodes)) {
        result = pack(INVALID, 0, 0, R_INVALID_SHAPE);
        going = false;
    }
#pragma unroll
    for (int k = 0; k < SLOTS; k++) kids[k] = CHILD_NONE;
    if (going) request(0);
    while (__any_sync(FULL, going)) {
        if (going && terminal) {
            result = pack(TERMINAL, node, 0, R_OK_TERMINAL);
            going = false;
        } else if (going && depth >= path_depth) {
            result = pack(DEPTH_LIMIT, node, 0, R_OK_DEPTH_LIMIT);
            going = false;
        }
        // ---- each player's arg-max over its own marginal statistics.  The winner is claimed with a compare-and-swap on the count
        // it was scored with: if another traversal claimed it meanwhile, the counts in flight are read again and the arg-max
        // is redone, so that traversals started together spread over the actions as they would one after the other; the
        // last evaluation claims unconditionally.
        const int s = node * 2 * A + player * A + action;
        bool open = going;          // this player has no claim yet
        int pick = 0, from = -1;    // `from`: the child whose data has been requested
        const int here = node;
        float my_prior = prior, my_w = w;
        int my_n = n, my_inflight = inflight, my_kids[SLOTS];
#pragma unroll
        for (int k = 0; k < SLOTS; k++) my_kids[k] = kids[k];
        int joint = 0, kid = CHILD_NONE;
        for (int evaluation = 1; __any_sync(FULL, open); evaluation++) {
            int total = has_action ? my_n + virtual_loss * my_inflight : 0;
#pragma unroll
            for (int o = 1; o < LANES; o <<= 1) total += __shfl_xor_sync(FULL, total, o);
            const float sqrt_total = root_of_count(max(total, 1));
            const unsigned key = has_action ? ordered(score(cpuct, my_prior, my_w, my_n, my_inflight, virtual_loss, sqrt_total)) : 0u;
            unsigned best = key;
#pragma unroll
            for (int o = 1; o < LANES; o <<= 1) best = max(best, __shfl_xor_sync(FULL, best, o));
            const unsigned tied = __ballot_sync(FULL, has_action && key == best) >> (base + player * LANES);
            if (open) pick = __ffs(tied & ((1u << LANES) - 1u)) - 1;   // lowest action on ties
            const int other = __shfl_xor_sync(FULL, pick, LANES);
            joint = player ? other * A + pick : pick * A + other;
            int held[SLOTS];   // slot joint / GROUP, found by halves (an index would send the array to local memory)
#pragma unroll
            for (int k = 0; k < SLOTS; k++) held[k] = my_kids[k];
#pragma unroll
            for (int half = SLOTS / 2, bit = SLOTS / 2 * GROUP; half > 0; half /= 2, bit /= 2)
#pragma unroll
                for (int k = 0; k < half; k++) held[k] = (joint & bit) ? held[k + half] : held[k];
            kid = __shfl_sync(FULL, held[0], base + (joint & (GROUP - 1)));
            // the child's data travels together with the claims
            if (going && kid >= 0 && kid < node_cnt && kid != from) {
                request(kid);
                from = kid;
            }
            bool claimed = true;
            if (open && action == pick) {
                if (evaluation < MAX_EVALUATIONS) claimed = atomicCAS(&inflight_of[s], my_inflight, my_inflight + virtual_loss) == my_inflight;
                else atomicAdd(&inflight_of[s], virtual_loss);
            }
            const unsigned lost = __ballot_sync(FULL, !claimed) >> (base + player * LANES);
            open = open && (lost & ((1u << LANES) - 1u)) != 0u;
            if (open && has_action) my_inflight = *(volatile const int *)&inflight_of[s];
        }
        if (going) {
            if (sub == 0) path[depth] = (here << 8) | joint;
            depth++;
        }
        __syncwarp();   // the rollbacks below read the entry
        if (going && kid >= node_cnt) {
            rollback(depth);
            result = pack(INVALID, here, joint, R_INVALID_CHILD_OOB);
            depth = 0;
            going = false;
        }
        const bool childless = going && kid < 0;
        if (__any_sync(FULL, childless)) {
            // no child yet: one traversal may expand the joint action, the others back off
            int won = 0;
            if (childless && sub == 0)
                won = kid == CHILD_NONE && atomicCAS(&child_of[here * joints + joint], CHILD_NONE, CHILD_CLAIMED) == CHILD_NONE ? 1 : 0;
            won = __shfl_sync(FULL, won, base);
            if (childless) {
                if (won) {
                    result = pack(EXPAND, here, joint, R_OK_EXPAND);
                } else {
                    rollback(depth);
                    result = pack(BUSY, here, joint, R_BUSY_EXPAND_INFLIGHT);
                    depth = 0;
                }
                going = false;
            }
        }
        node = kid;
    }
    if (exists && sub == 0) {
        out_selected[out] = result;
        out_len[out] = depth;
    }
}

static unsigned select_blocks(int trees, int trees_per_warp, int warps) {
    const long long units = ((long long)trees + trees_per_warp - 1) / trees_per_warp * warps;
    return (unsigned)((units + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK);
}

// per path entry: both players' claims are returned, and with `values` the visit counts and value sums are updated
// (values are from player 0's point of view; player 1 receives the negative).  An EXPAND result either installs
// new_child (when given and >= 0) in the claimed slot or frees the slot again.
__global__ void backup_kernel(int virtual_loss, int *child, float *node_w, int *node_n, int *node_inflight, const int *out_selected,
                              const int *out_path, const int *out_len, const float *values, const int *new_child, int nodes, int A,
                              int traversals, int warps, int path_depth, int log2_lanes) {
    const BackupLane at_work(traversals, log2_lanes);
    const int out = at_work.traversal;
    if (out < 0) return;
    const int len = out_len[out];
    const int sel = at_work.lane == 0 ? out_selected[out] : 0;
    const int tree = out / warps;
    const int *path = out_path + (long long)out * path_depth;
    const long long stats_base = (long long)tree * nodes * 2 * A;
    for (int d = at_work.lane; d < len; d += 1 << log2_lanes) {
        const int enc = path[d];
        const float v = values ? values[(long long)out * path_depth + d] : 0.f;
        const int node = enc >> 8, joint = enc & 0xFF, a0 = joint / A;
        const long long s0 = stats_base + (long long)node * 2 * A + a0;
        const long long s1 = s0 + A - a0 + (joint - a0 * A);
        atomicSub(&node_inflight[s0], virtual_loss);
        atomicSub(&node_inflight[s1], virtual_loss);
        if (values) {
            atomicAdd(&node_n[s0], 1);
            atomicAdd(&node_n[s1], 1);
            atomicAdd(&node_w[s0], v);
            atomicAdd(&node_w[s1], -v);
        }
    }
    if (at_work.lane == 0 && ((sel >> KIND_SHIFT) & 7) == EXPAND) {
        const int node = sel & (NODE_LIMIT - 1), joint = (sel >> SLOT_SHIFT) & 0xFF;
        const int kid = new_child ? new_child[out] : CHILD_NONE;
        child[((long long)tree * nodes + node) * A * A + joint] = kid >= 0 ? kid : CHILD_NONE;
    }
}

}  // namespace duct

extern "C" int duct_select_launch(float cpuct, int virtual_loss, int *child, const float *node_prior, const float *node_w,
                                  const int *node_n, int *node_inflight, const int *node_terminal, const int *tree_nodes,
                                  int *out_selected, int *out_path, int *out_len, int trees, int nodes, int actions, int warps,
                                  int path_depth, void *stream) {
    if (trees <= 0 || nodes <= 0 || nodes > duct::NODE_LIMIT || actions <= 0 || actions > duct::MAX_ACTIONS || warps <= 0 ||
        warps > 32 || path_depth <= 0 || virtual_loss < 0)
        return (int)cudaErrorInvalidValue;
#define DUCT_LAUNCH(L)                                                                                                        \
    duct::select_kernel<L><<<duct::select_blocks(trees, 16 / L, warps), duct::WARPS_PER_BLOCK * 32, 0, (cudaStream_t)stream>>>( \
        cpuct, virtual_loss, child, node_prior, node_w, node_n, node_inflight, node_terminal, tree_nodes, out_selected,       \
        out_path, out_len, trees, nodes, actions, warps, path_depth)
    if (actions <= 4) DUCT_LAUNCH(4);
    else if (actions <= 8) DUCT_LAUNCH(8);
    else DUCT_LAUNCH(16);
#undef DUCT_LAUNCH
    return (int)cudaGetLastError();
}

extern "C" int duct_backup_launch(int virtual_loss, int *child, float *node_w, int *node_n, int *node_inflight,
                                  const int *out_selected, const int *out_path, const int *out_len, const float *values,
                                  const int *new_child, int trees, int nodes, int actions, int warps, int path_depth, void *stream) {
    if (trees <= 0 || nodes <= 0 || nodes > duct::NODE_LIMIT || actions <= 0 || actions > duct::MAX_ACTIONS || warps <= 0 ||
        warps > 32 || path_depth <= 0 || virtual_loss < 0)
        return (int)cudaErrorInvalidValue;
    if ((long long)trees * warps > 0x7FFFFFFF) return (int)cudaErrorInvalidValue;
    const select_math::BackupGrid g(trees * warps, path_depth);
    duct::backup_kernel<<<g.blocks, g.THREADS, 0, (cudaStream_t)stream>>>(virtual_loss, child, node_w, node_n, node_inflight, out_selected,
                                                                          out_path, out_len, values, new_child, nodes, actions,
                                                                          trees * warps, warps, path_depth, g.log2_lanes);
    return (int)cudaGetLastError();
}
