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
select_kernel(float cpuct, int virtual_loss, int *child_all, const float *node_prior, const float *node_w,
              const int *node_n, int *node_inflight_all, const int *node_terminal,
              const int *tree_nodes, int *out_selected, int *out_path, int *out_len, int trees, int nodes, int A, int warps,
              int path_depth) {
    constexpr int GROUP = 2 * LANES, PER_WARP = 32 / GROUP;
    constexpr int SLOTS = (LANES * LANES + GROUP - 1) / GROUP;   // child ids a lane may hold
    let_the_next_kernel_come();
    const unsigned block = block_after_the_kernel_before();
    const int lane = threadIdx.x & 31;
    const int sub = lane & (GROUP - 1), base = lane & ~(GROUP - 1);   // lane within the traversal, its first lane
    const int player = sub / LANES, action = sub & (LANES - 1);
    // the traversals of a warp belong to neighbouring trees (those of one tree would lose each other's claims in step)
    const int unit = (int)block * WARPS_PER_BLOCK + (int)(threadIdx.x >> 5);
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

// ---------------------------------------------------------------------------------------------------------------
// Two to eight traversals per tree: all traversals of a tree in one warp, four lanes each, APL actions of either player per lane.
// A turn of the warp is one choice of every traversal at the node it has come to: a traversal that gets its claims goes on to the
// child, one that loses a claim reads the counts in flight again and chooses again in the next turn, while the others move on.
// Who meets whom is known in registers: of the traversals of a tree that want the same action in the same turn the first has
// it, and their counts are from the same moment, so the others are those whose compare-and-swap would fail.  A claim
// is therefore an addition that nobody waits for.  A third choice, which needs no answer, follows the second at once, as it does in
// select_kernel while the winners still wait for theirs; with that nearly the same paths come out (counts that differ after a wave and
// its backup, between two runs of select_kernel / between it and this kernel: 4096 trees x 8 actions x 8 traversals 0.09 / 0.12 %, two
// waves one after the other 0.75 / 0.78 %; 2500 x 8 x 4 0.012 / 0.015 %; 4096 x 7 x 8 0.22 / 0.33 %).
// The claims of earlier turns are seen: __syncwarp orders them before the next loads, and no other warp is in the tree.
// The child of the joint action is loaded when it is known: a node's whole row of children, loaded ahead as in
// select_kernel, is as much as all its statistics, and with every traversal on the device at once memory's throughput counts.
// What bounds it: a chain of two round trips to memory and some 400 instructions a turn (1500 trees: 31 % of the issue slots, half of a
// warp's time waiting for memory); 4096 trees x 8 actions x 8 traversals x 16 levels 159 us with select_kernel, 95 so (111 with all choices of a level in one turn, which takes the whole
// warp along).
// VECTORS: rows of 4 * APL actions on addresses that take a lane's actions in one load.
constexpr int GROUP_LANES = 4, GROUPS = 8, GROUP_WARPS = 4;

template <int APL, bool VECTORS, typename T>
__device__ __forceinline__ void load_row(T (&v)[APL], const T *p, int actions, bool fresh) {
    static_assert(sizeof(T) == 4 && (APL == 1 || APL == 2 || APL == 4), "words");
    unsigned raw[APL];
    const unsigned *q = reinterpret_cast<const unsigned *>(p);
    if (VECTORS && APL == 2) {
        const uint2 x = fresh ? __ldcv(reinterpret_cast<const uint2 *>(q)) : *reinterpret_cast<const uint2 *>(q);
        raw[0] = x.x;
        raw[APL > 1 ? 1 : 0] = x.y;
    } else if (VECTORS && APL == 4) {
        const uint4 x = fresh ? __ldcv(reinterpret_cast<const uint4 *>(q)) : *reinterpret_cast<const uint4 *>(q);
        raw[0] = x.x;
        raw[APL > 1 ? 1 : 0] = x.y;
        raw[APL > 2 ? 2 : 0] = x.z;
        raw[APL > 3 ? 3 : 0] = x.w;
    } else {
#pragma unroll
        for (int k = 0; k < APL; k++) raw[k] = k < actions ? (fresh ? __ldcv(q + k) : q[k]) : 0u;
    }
#pragma unroll
    for (int k = 0; k < APL; k++) v[k] = *reinterpret_cast<T *>(&raw[k]);
}

// the scores of a lane's actions, as `score` has them; one look at all operands decides whether any quotient needs a division
template <int APL>
__device__ __forceinline__ void scores(float (&value)[2][APL], float cpuct, const float (&prior)[2][APL], const float (&w)[2][APL],
                                       const int (&n)[2][APL], const int (&inflight)[2][APL], int virtual_loss, const float (&sqrt_total)[2]) {
    bool plain = true;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
        for (int k = 0; k < APL; k++) {
            const int n_eff = n[p][k] + virtual_loss * inflight[p][k];
            const float w_eff = __fsub_rn(w[p][k], (float)(virtual_loss * inflight[p][k]));
            const float up = __fmul_rn(__fmul_rn(cpuct, prior[p][k]), sqrt_total[p]);
            plain = plain && (unsigned)n_eff < (1u << 22) && Count::plain(w_eff, up);
            const float q = Count(max(n_eff, 1)).divides(w_eff);
            value[p][k] = __fadd_rn(n_eff > 0 ? q : 0.f, Count(n_eff + 1).divides(up));
        }
    if (!plain) {
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int k = 0; k < APL; k++)
                value[p][k] = score(cpuct, prior[p][k], w[p][k], n[p][k], inflight[p][k], virtual_loss, sqrt_total[p]);
    }
}

template <int APL, bool VECTORS>
__global__ void __launch_bounds__(GROUP_WARPS * 32, 7)
group_select_kernel(float cpuct, int virtual_loss, int *child_all, const float *node_prior, const float *node_w,
                    const int *node_n, int *node_inflight_all, const int *node_terminal,
                    const int *tree_nodes, int *out_selected, int *out_path, int *out_len, int trees, int nodes, int A, int warps,
                    int path_depth) {
    let_the_next_kernel_come();
    const unsigned block = block_after_the_kernel_before();
    const int lane = threadIdx.x & 31;
    const int sub = lane & (GROUP_LANES - 1), base = lane & ~(GROUP_LANES - 1);   // lane within the traversal, its first lane
    const int trees_per_warp = GROUPS / warps;
    const int mine = (lane / GROUP_LANES) / warps, wid = (lane / GROUP_LANES) - mine * warps;   // tree of the warp, traversal of the tree
    const int unit = (int)block * GROUP_WARPS + (int)(threadIdx.x >> 5);
    const bool exists = mine < trees_per_warp && unit * trees_per_warp + mine < trees;
    const int tree = exists ? unit * trees_per_warp + mine : 0;
    const int out = tree * warps + wid;
    int *path = out_path + (long long)out * path_depth;
    const int node_cnt = tree_nodes[tree];
    const int first = sub * APL, own = A - first;   // the lane's actions are first .. first + min(own, APL) - 1
    const int joints = A * A;
    const long long tree_nodes_base = (long long)tree * nodes;
    const long long stats_base = tree_nodes_base * 2 * A;
    int *child_of = child_all + tree_nodes_base * joints;
    int *inflight_of = node_inflight_all + stats_base;
    const float *prior_of = node_prior + stats_base, *w_of = node_w + stats_base;
    const int *n_of = node_n + stats_base, *terminal_of = node_terminal + tree_nodes_base;

    float prior[2][APL], w[2][APL];
    int n[2][APL], inflight[2][APL], terminal = 0;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
        for (int k = 0; k < APL; k++) {
            prior[p][k] = w[p][k] = 0.f;
            n[p][k] = inflight[p][k] = 0;
        }
    auto request_claims = [&](int at_node) {
#pragma unroll
        for (int p = 0; p < 2; p++) load_row<APL, VECTORS>(inflight[p], inflight_of + at_node * 2 * A + p * A + first, own, true);
    };
    auto request = [&](int at_node) {
        terminal = terminal_of[at_node];
        request_claims(at_node);
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int s = at_node * 2 * A + p * A + first;
            load_row<APL, VECTORS>(prior[p], prior_of + s, own, false);
            load_row<APL, VECTORS>(w[p], w_of + s, own, false);
            load_row<APL, VECTORS>(n[p], n_of + s, own, false);
        }
    };
    // gives back the claims of the first `count` path entries of the traversal
    auto rollback = [&](int count) {
        for (int d = sub; d < count; d += GROUP_LANES) {
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
    if (going) request(0);
    int evaluation = 1, pick[2] = {0, 0};
    bool open[2] = {true, true};             // this player has no claim at the node yet
    while (__any_sync(FULL, going)) {
        if (going && evaluation == 1) {
            if (terminal) {
                result = pack(TERMINAL, node, 0, R_OK_TERMINAL);
                going = false;
            } else if (depth >= path_depth) {
                result = pack(DEPTH_LIMIT, node, 0, R_OK_DEPTH_LIMIT);
                going = false;
            }
        }
        bool choosing = going;
        for (;;) {
            float sqrt_total[2];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                int total = 0;
#pragma unroll
                for (int k = 0; k < APL; k++)
                    if (k < own) total += n[p][k] + virtual_loss * inflight[p][k];
                total += __shfl_xor_sync(FULL, total, 1);
                total += __shfl_xor_sync(FULL, total, 2);
                sqrt_total[p] = root_of_count(max(total, 1));
            }
            float value[2][APL];
            scores<APL>(value, cpuct, prior, w, n, inflight, virtual_loss, sqrt_total);
            unsigned key[2] = {0u, 0u}, best[2];
            int at[2] = {0, 0};
#pragma unroll
            for (int p = 0; p < 2; p++) {
#pragma unroll
                for (int k = 0; k < APL; k++) {
                    const unsigned v = ordered(value[p][k]);
                    if (k < own && (k == 0 || v > key[p])) {   // the lowest action on ties
                        key[p] = v;
                        at[p] = first + k;
                    }
                }
                best[p] = max(key[p], __shfl_xor_sync(FULL, key[p], 1));
                best[p] = max(best[p], __shfl_xor_sync(FULL, best[p], 2));
            }
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const unsigned tied = __ballot_sync(FULL, own > 0 && key[p] == best[p]) >> base;
                const int chosen = __shfl_sync(FULL, at[p], base + __ffs(tied & ((1u << GROUP_LANES) - 1u)) - 1);
                if (choosing && open[p]) pick[p] = chosen;
            }
            // lane 0 of a traversal claims for player 0, lane 1 for player 1
            const int action = sub == 0 ? pick[0] : pick[1];
            const bool claims = choosing && sub < 2 && (sub == 0 ? open[0] : open[1]);
            const unsigned same = __match_any_sync(FULL, claims ? (unsigned)(((mine << 14) | node) << 5 | sub << 4 | action) : 0x80000000u);
            const bool won = claims && (evaluation == MAX_EVALUATIONS || __ffs(same) - 1 == lane);
            if (won) atomicAdd(&inflight_of[node * 2 * A + sub * A + action], virtual_loss);
            const unsigned lost = __ballot_sync(FULL, claims && !won) >> base;
            if (choosing) {
                open[0] = lost & 1u;
                open[1] = lost & 2u;
            }
            choosing = choosing && (open[0] || open[1]) && evaluation == MAX_EVALUATIONS - 1;
            if (!__any_sync(FULL, choosing)) break;
            __syncwarp();   // the claims just made are seen
            if (choosing) {
                evaluation++;
                request_claims(node);
            }
        }
        const bool moves = going && !open[0] && !open[1];
        const int here = node, joint = pick[0] * A + pick[1];
        int kid = CHILD_NONE;
        if (moves) {
            kid = *(volatile const int *)&child_of[here * joints + joint];
            if (sub == 0) path[depth] = (here << 8) | joint;
            depth++;
        }
        __syncwarp();   // the rollbacks below read the entry, and the loads that follow see the claims made so far
        if (going && !moves) {
            evaluation++;
            request_claims(node);
        }
        if (moves && kid >= node_cnt) {
            rollback(depth);
            result = pack(INVALID, here, joint, R_INVALID_CHILD_OOB);
            depth = 0;
            going = false;
        }
        const bool childless = moves && kid < 0;
        if (__any_sync(FULL, childless)) {
            // no child yet: one traversal may expand the joint action, the others back off
            int expands = 0;
            if (childless && sub == 0)
                expands = kid == CHILD_NONE && atomicCAS(&child_of[here * joints + joint], CHILD_NONE, CHILD_CLAIMED) == CHILD_NONE ? 1 : 0;
            expands = __shfl_sync(FULL, expands, base);
            if (childless) {
                if (expands) {
                    result = pack(EXPAND, here, joint, R_OK_EXPAND);
                } else {
                    rollback(depth);
                    result = pack(BUSY, here, joint, R_BUSY_EXPAND_INFLIGHT);
                    depth = 0;
                }
                going = false;
            }
        }
        if (moves && going) {
            node = kid;
            evaluation = 1;
            open[0] = open[1] = true;
            request(kid);
        }
    }
    if (exists && sub == 0) {
        out_selected[out] = result;
        out_len[out] = depth;
    }
}

// Whether a launch goes to group_select_kernel: two to eight traversals a tree, and more warps of select_kernel than are on the
// device at once (32 an SM).  Below that its level is the shorter one: a lane has one action to score, not four or eight, and the child
// comes with the level.  Microseconds of the select, select_kernel / this (actions: trees x traversals a tree; 16 levels, of 7 actions 12, of
// 12 actions 4):
//   3: 2500 x 8 80 / 52, 4096 x 8 87 / 64   7: 2500 x 4 59 / 48, 4096 x 8 136 / 81   8: 2500 x 4 70 / 58, 1500 x 8 80 / 64, 4096 x 8 159 / 95
//   12: 4096 x 2 33 / 27, 2000 x 4 37 / 33, 4096 x 8 156 / 70;   not taken: 3: 4096 x 4 44 / 41   8: 4096 x 2 42 / 52, 1000 x 8 48 / 58
//   12: 1000 x 4 27 / 30
static bool traversals_in_step(int trees, int actions, int warps) {
    const int per_warp = actions <= 4 ? 4 : (actions <= 8 ? 2 : 1);
    return warps >= 2 && warps <= GROUPS && ((long long)trees + per_warp - 1) / per_warp * warps > 32 * sm_count();
}

// whether every row of A words starts where a load of A / 4 words may
static bool rows_take_vectors(int A, const void *a, const void *b, const void *c, const void *d) {
    const uintptr_t bits = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d;
    return (A == 8 || A == 16) && bits % (uintptr_t)A == 0;
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
    const BackupLane at_work(block_after_the_kernel_before(), traversals, log2_lanes);
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
    select_math::launch_behind(duct::select_kernel<L>, duct::select_blocks(trees, 16 / L, warps), duct::WARPS_PER_BLOCK * 32, (cudaStream_t)stream,  \
        cpuct, virtual_loss, child, node_prior, node_w, node_n, node_inflight, node_terminal, tree_nodes, out_selected,       \
        out_path, out_len, trees, nodes, actions, warps, path_depth)
    if (duct::traversals_in_step(trees, actions, warps)) {
        const int per_warp = duct::GROUPS / warps;
        const long long units = ((long long)trees + per_warp - 1) / per_warp;
        const unsigned blocks = (unsigned)((units + duct::GROUP_WARPS - 1) / duct::GROUP_WARPS);
        const bool vectors = duct::rows_take_vectors(actions, node_prior, node_w, node_n, node_inflight);
#define DUCT_GROUP_LAUNCH(APL, V)                                                                                             \
    select_math::launch_behind(duct::group_select_kernel<APL, V>, blocks, duct::GROUP_WARPS * 32, (cudaStream_t)stream,                           \
        cpuct, virtual_loss, child, node_prior, node_w, node_n, node_inflight, node_terminal, tree_nodes, out_selected,       \
        out_path, out_len, trees, nodes, actions, warps, path_depth)
        if (actions <= 4) DUCT_GROUP_LAUNCH(1, false);
        else if (actions <= 8 && vectors) DUCT_GROUP_LAUNCH(2, true);
        else if (actions <= 8) DUCT_GROUP_LAUNCH(2, false);
        else if (vectors) DUCT_GROUP_LAUNCH(4, true);
        else DUCT_GROUP_LAUNCH(4, false);
#undef DUCT_GROUP_LAUNCH
        return (int)cudaGetLastError();
    }
    if (actions <= 4) DUCT_LAUNCH(4);
    else if (actions <= 8) DUCT_LAUNCH(8);
    else DUCT_LAUNCH(16);
#undef DUCT_LAUNCH
    return (int)cudaGetLastError();
}

extern "C" const char *duct_select_kernel_name(int trees, int actions, int warps) {
    return duct::traversals_in_step(trees, actions, warps) ? "duct::group_select_kernel" : "duct::select_kernel";
}

extern "C" int duct_backup_launch(int virtual_loss, int *child, float *node_w, int *node_n, int *node_inflight,
                                  const int *out_selected, const int *out_path, const int *out_len, const float *values,
                                  const int *new_child, int trees, int nodes, int actions, int warps, int path_depth, void *stream) {
    if (trees <= 0 || nodes <= 0 || nodes > duct::NODE_LIMIT || actions <= 0 || actions > duct::MAX_ACTIONS || warps <= 0 ||
        warps > 32 || path_depth <= 0 || virtual_loss < 0)
        return (int)cudaErrorInvalidValue;
    if ((long long)trees * warps > 0x7FFFFFFF) return (int)cudaErrorInvalidValue;
    const select_math::BackupGrid g(trees * warps, path_depth);
    select_math::launch_behind(duct::backup_kernel, g.blocks, g.THREADS, (cudaStream_t)stream, virtual_loss, child, node_w, node_n, node_inflight, out_selected,
                                                                          out_path, out_len, values, new_child, nodes, actions,
                                                                          trees * warps, warps, path_depth, g.log2_lanes);
    return (int)cudaGetLastError();
}
