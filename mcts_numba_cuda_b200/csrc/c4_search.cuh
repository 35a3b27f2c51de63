// Connect-4 search kernel: the whole MCTS-NC loop of one tree in one thread block, all steps on the device.
//
// Replaces, per step, the reference kernels _select (src/mctsnc.py:1293-1365), _expand_1_* (:1368-1681),
// _expand_2_* (:1691-1821), _playout_ocp / _playout_acp_* (:1824-2081), _backup_ocp / _backup_1_acp_* /
// _backup_2_acp (:2084-2220), the _reset kernel (:1260-1290) and the Connect-4 device functions
// (src/mctsnc_game_mechanics.py:89-179).
//
// Work split inside a block: warp 0 walks the tree (select), creates the children (expand) and writes the statistics
// back (backup); all threads play the random games.  A thread keeps playing its own list of games back to back (one
// per expanded child and playout index, the reference's thread (tree, action, t)), so the lanes of a warp wait for
// each other once per step, not once per game.
//
// Position encoding: column c of the 6x7 board owns byte c + 1 of a 64-bit word: bits 8c + 8 .. 8c + 13 (bottom cell first) and
// two guard bits that stay 0; byte 0 holds no cell.  Four columns are exactly the high 32-bit word: a horizontal or diagonal
// four ends in one of them, so its test works on four words of four columns each (see fours_across), and the column of a
// stone is one byte permute away.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "rng.cuh"

namespace mctsnc {
namespace c4 {

constexpr int ROWS = 6, COLS = 7, A = 7;
__host__ __device__ constexpr int column_shift(int c) { return 8 * c + 8; }
// plies of a playout between two looks at whether the game is over
constexpr int PLIES_PER_CHECK = 4, STRAIGHT_PLIES = 4;
constexpr unsigned long long BOTTOM_ROW = 0x0101010101010100ULL;
constexpr unsigned long long FULL_BOARD = BOTTOM_ROW * 0x3FULL;
constexpr unsigned BOTTOM_LO = 0x01010100u, BOTTOM_HI = 0x01010101u;   // of the columns 0..2 and 3..6
constexpr unsigned TOP_LO = 0x20202000u, TOP_HI = 0x20202020u;

// Four in a row that end in the high word's columns (horizontal and both diagonals) of the stone set (lo, hi), added to `r`.
// x1, x2, x3: the columns one, two and three to the left of each, so the stones of a diagonal meet after shifts within the
// columns.  All of those go to the left (a shift to the left can be done by the multiply-add pipe, the logic pipe is the
// busy one): the falling diagonal is lifted by three rows.  Shifts by up to three rows leave a column across its two guard bits
// only where the word shifted by one or two rows holds a guard bit, so nothing is found there.  (Nine funnel shifts of
// the pair, one for every word and direction: a fifth of the headline batch 20.3 ms, 19.1 so.)
__host__ __device__ __forceinline__ unsigned fours_across(unsigned lo, unsigned hi, unsigned r = 0u) {
    const unsigned long long p = ((unsigned long long)hi << 32) | lo;
    const unsigned x1 = (unsigned)(p >> 24), x2 = (unsigned)(p >> 16), x3 = (unsigned)(p >> 8);
    r |= hi & x1 & x2 & x3;
    r |= hi & (x1 << 1) & (x2 << 2) & (x3 << 3);
    r |= (hi << 3) & (x1 << 2) & (x2 << 1) & x3;
    return r;
}

// four in a row anywhere in the stone set p
__host__ __device__ __forceinline__ bool has_four(unsigned long long p) {
    unsigned long long v = p & (p >> 1);
    v &= v >> 2;
    return (fours_across((unsigned)p, (unsigned)(p >> 32)) | (unsigned)v | (unsigned)(v >> 32)) != 0u;
}

// set of columns that still have room, from the occupancy bitboard
__host__ __device__ __forceinline__ unsigned legal_columns(unsigned long long all) {
    unsigned l = 0;
#pragma unroll
    for (int c = 0; c < COLS; c++) l |= ((all >> (column_shift(c) + 5)) & 1ULL) ? 0u : (1u << c);
    return l;
}

// index of the n-th set bit (n = 0 is the lowest)
__device__ __forceinline__ int nth_set(int mask, int n) {
    for (; n > 0; n--) mask &= mask - 1;
    return __ffs(mask) - 1;
}

// among tied maxima the reference's stride-halving reduction keeps the left operand (src/mctsnc.py:1343-1351), which
// over 8 slots ranks the actions 0,4,2,6,1,5,3 (smallest bit-reversed index wins)
__device__ __forceinline__ int pick_among_tied(unsigned m) {
    if (m & 1u) return 0;
    if (m & 16u) return 4;
    if (m & 4u) return 2;
    if (m & 64u) return 6;
    if (m & 2u) return 1;
    if (m & 32u) return 5;
    return 3;
}

// ---------------------------------------------------------------------------------------------------------------
// Byte-for-byte emulation of one playout of the reference (src/mctsnc.py:2049-2069 with the Connect-4 functions of
// src/mctsnc_game_mechanics.py:102-179) on int8 arrays.  Only entered when a uniform draw equals 1.0f, which makes
// the reference read legal_actions_with_count[count]: a value left by an earlier ply of the same playout, or a slot
// never written (read as 0 here).  numba wraps negative indices once; rows below 0 therefore address the board from
// the bottom.  The playout is replayed from its first ply so that the stale slots hold what they would hold.
struct EmuResult {
    int outcome;
    unsigned plies;
    unsigned ub;
    unsigned err;
    unsigned long long s0, s1;  // stream state after the game
};

__device__ __forceinline__ int emu_cell(const signed char *board, int i, int j, unsigned &err) {
    if (i < 0) i += ROWS;
    if (j < 0) j += COLS;
    if (i < 0 || i >= ROWS || j < 0 || j >= COLS) {
        err = 1;
        return 0;
    }
    return board[i * COLS + j];
}

__device__ __forceinline__ int emu_line(const signed char *board, int i, int j, int di, int dj, int token, unsigned &err) {
    int total = 0;
    for (int k = 1; k < 4; k++) {
        int ii = i + k * di, jj = j + k * dj;
        if ((di < 0 && ii < 0) || (di > 0 && ii >= ROWS) || (dj < 0 && jj < 0) || (dj > 0 && jj >= COLS)) break;
        if (emu_cell(board, ii, jj, err) != token) break;
        total++;
    }
    return total;
}

__device__ __noinline__ EmuResult playout_emulated(unsigned long long neg, unsigned long long pos, int turn,
                                                   unsigned long long s0, unsigned long long s1) {
    unsigned err = 0;
    signed char board[ROWS * COLS];
    signed char fills[COLS];
    short legal[COLS + 1];
    for (int j = 0; j < COLS; j++) {
        int f = 0;
        for (int h = 0; h < ROWS; h++) {
            int bit = column_shift(j) + h;
            int v = ((pos >> bit) & 1ULL) ? 1 : (((neg >> bit) & 1ULL) ? -1 : 0);
            board[(ROWS - 1 - h) * COLS + j] = (signed char)v;
            f += v != 0;
        }
        fills[j] = (signed char)f;
    }
    for (int j = 0; j <= COLS; j++) legal[j] = 0;
    EmuResult r = {2, 0u, 0u, 0u, 0ULL, 0ULL};
    for (;;) {
        int count = 0;
        for (int j = 0; j < COLS; j++)
            if (fills[j] < ROWS) legal[count++] = (short)j;
        float u = rng_uniform_f32(s0, s1);
        int ord = (int)(short)__float2int_rz(__fmul_rn(u, (float)count));
        if (u >= 1.0f) r.ub++;
        if (ord < 0 || ord > COLS) {
            err = 1;
            ord = 0;
        }
        int a = legal[ord];
        fills[a] += 1;
        int row = ROWS - fills[a];
        if (row < 0) row += ROWS;
        if (row < 0) {
            err = 1;
            row = 0;
        }
        board[row * COLS + a] = (signed char)turn;
        turn = -turn;
        r.plies++;
        // compute_outcome_c4(board, fills, turn, a)
        int token = -turn;
        int i = ROWS - fills[a];
        int out = 2;
        if (emu_line(board, i, a, -1, 0, token, err) + emu_line(board, i, a, 1, 0, token, err) >= 3) out = token;
        else if (emu_line(board, i, a, 0, 1, token, err) + emu_line(board, i, a, 0, -1, token, err) >= 3) out = token;
        else if (emu_line(board, i, a, -1, 1, token, err) + emu_line(board, i, a, 1, -1, token, err) >= 3) out = token;
        else if (emu_line(board, i, a, -1, -1, token, err) + emu_line(board, i, a, 1, 1, token, err) >= 3) out = token;
        else {
            bool draw = true;
            for (int j = 0; j < COLS; j++)
                if (fills[j] < ROWS) draw = false;
            if (draw) out = 0;
        }
        if (r.plies > 4096u) {  // cannot happen; keeps the loop bounded whatever the memory holds
            err = 1;
            out = 0;
        }
        if (out != 2) {
            r.outcome = out;
            r.err = err;
            r.s0 = s0;
            r.s1 = s1;
            return r;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------

// everything a thread needs to start a game from one child, fetched with two 16-byte shared-memory loads
struct __align__(16) GameSlot {
    unsigned long long cur;    // stones of the side to move
    unsigned long long other;  // stones of the other side
    float row;                 // move_row(set of columns with room)
    float count;               // number of columns with room times 2^-64 (the playout loop draws uniforms scaled by 2^64)
    int rng_base;              // index of the child's first stream in the block's stream array
    int stones;                // stones on the board
};

// move_lut[(set ^ 1) * 8 + ord]: the ord-th column (ascending) of the column set `set`, as the six cells of that column in
// the two words of a position.  The low bits of `lo`, where no cell is, hold the number of the column's byte.  The index is
// computed in float: the playout loop keeps row = 2^23 + 8 * (set ^ 1), and row + u * count added with rounding towards zero is
// 2^23 + the index, in the low bits of the mantissa.
// An ordinal the set does not have (only a uniform draw of exactly 1.0f gives one: ord == number of columns) is a move to
// MARK, a bit of byte 0, which stays in the position and tells the end of the game.  The empty set has no move at all.
struct __align__(8) MoveEntry {
    unsigned lo, hi;
};
constexpr float MOVE_LUT_BASE = 8388608.f;
constexpr unsigned MOVE_LUT_BASE_BITS = 0x4B000000u;
constexpr unsigned MARK = 0x10u;
__host__ __device__ constexpr float move_row(unsigned set) { return MOVE_LUT_BASE + (float)(8u * (set ^ 1u)); }
constexpr float NO_MOVES = MOVE_LUT_BASE + 8.f;   // move_row(0)

constexpr int MAX_PATH = 48;

// What the walker of a tree keeps between the stages of a step.
struct Walk {
    int4 path_rec[MAX_PATH]; // the records of the selected path as the select read them
    PathTerm term[MAX_PATH];
    int path[MAX_PATH];
    int child_outcome[A];    // per expanded child (expansion order): its outcome (2 = ongoing)
    int child_slot[A];       // and its slot (-1: no playouts: terminal, or not picked in OCP)
    int child_out[A][2];     // trees_playout_outcomes_children (persists over steps)
    short ae[A + 2];         // trees_actions_expanded row (persists over steps)
    int n_slots;
    int mode;
    int first_child;
    int exp_mask;
    int selected;
    int sel_meta;
    int path_len;
    int pick;                // OCP: index (among expanded children) of the child that is played out
    int root_turn;
    int size;
    int max_depth;           // of the nodes, and the sum of their depths
    long long depth_sum;
    int out_neg, out_pos;
    unsigned status;
    unsigned long long plies;
    unsigned long long ub;
    unsigned long long stage_cycles[4];  // cycles of this slice spent in select, expand, playouts, backup
    unsigned stage_mark;        // cycle counter when the playouts of the current step began
};

struct Shared : Walk {
    GameSlot slot[A];        // children that need real playouts, in expansion order
    MoveEntry move_lut[128 * 8];
    int tally[A][2];         // per slot: games won by -1, by +1 (of the games this block played)
    int gather[A][2];        // cluster of blocks per tree: the sums over the blocks, kept by the first block
    int job;                 // tree of the slice being run (-1: none left)
    int held, held_level;    // tree of the slice before if it has steps left (-1: it has none), and its ring
    int next_item;           // next game to hand out in the playout phase
};

// Node records through the copy the walker keeps of a tree's first `cache_n` records (cluster kernel: the walk down the tree
// is a chain of dependent loads, and the upper levels of a tree are its oldest nodes); cache_n = 0: global memory only.
// Every store goes to both.
__device__ __forceinline__ int4 rec_load(const int4 *rec, const int4 *cache, int cache_n, int i) {
    return i < cache_n ? cache[i] : rec[i];
}
__device__ __forceinline__ void rec_store(int4 *rec, int4 *cache, int cache_n, int i, int4 v) {
    rec[i] = v;
    if (i < cache_n) cache[i] = v;
}

// What the backup of the selected path needs and what does not depend on how the games end: the visit counts it will leave
// are known as soon as the leaf is, so every logarithm, division and square root of the UCBs can be done while the games
// are being played.  Eight lanes per level (lane = action), four levels at a time.
template <bool OCP>
__device__ __forceinline__ void prepare_backup(Walk &s, const int4 *rec, const int4 *cache, int cache_n, double c_ucb, int lane,
                                               int plen, int n_tot, int leaf_playouts) {
    const int a = lane & 7, shift = lane & 24;
    for (int base = 0; base < plen - 1; base += 4) {
        const int e = base + (lane >> 3);
        const bool level = e < plen - 1;
        const int4 pr = s.path_rec[level ? e : 0];
        const int n_path = s.path_rec[level ? e + 1 : 0].x + n_tot;
        const unsigned mask = pr.w & 0x7F;
        const bool has = level && ((mask >> a) & 1u);
        const int rank = __popc(mask & ((1u << a) - 1u));
        const bool on_path = rank == meta_best(pr.w);
        int n = n_path, w = 0;
        if (has && !on_path) {
            const int4 cr = rec_load(rec, cache, cache_n, pr.z + rank);
            n = cr.x;
            w = cr.y;
        }
        const double explore = sqrt(log((double)(pr.x + n_tot)) / (double)n);
        const double n_f = (double)__int2float_rn(n), reciprocal = 1.0 / n_f;
        unsigned key = 0;
        if (has && !on_path) key = ordered_key(n == 0 ? __int_as_float(0x7f800000) : ucb_value(c_ucb, explore, n_f, reciprocal, w));
        unsigned best = max(key, __shfl_xor_sync(0xFFFFFFFFu, key, 1));
        best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, 2));
        best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, 4));
        const unsigned tied = (__ballot_sync(0xFFFFFFFFu, key != 0u && key == best) >> shift) & 0x7Fu;
        if (has && on_path) {
            PathTerm t;
            t.explore = explore;
            t.n = n_f;
            t.reciprocal = reciprocal;
            t.other_key = best;
            const int o = pick_among_tied(tied);
            t.other = __popc(mask & ((1u << o) - 1u)) | (pick_among_tied((1u << o) | (1u << a)) == a ? 256 : 0);
            s.term[e] = t;
        }
    }
    if (leaf_playouts > 0) {
        PathTerm t;
        t.n = (double)leaf_playouts;   // at most 512: the same as a float32
        t.explore = sqrt(log((double)(s.path_rec[plen - 1].x + n_tot)) / t.n);
        t.reciprocal = 1.0 / t.n;
        t.other_key = 0u;
        t.other = 0;
        if (lane == 0) s.term[plen - 1] = t;
    }
}

// The state a tree has in global memory, or that of a tree of its root alone.  One thread.
__device__ __forceinline__ void load_tree(const SearchParams &p, Walk &s, int g, bool first, int4 *cache, int cache_n) {
    int4 *rec = p.rec + (long long)g * p.cap;
    TreeState *st = p.state + g;
    const int b = g / p.n_trees;
    if (first) {
        const int turn = p.root_turn[b];
        rec_store(rec, cache, cache_n, 0, make_int4(0, 0, -1, make_meta(0, false, 2, turn, 0)));
        p.board[(long long)g * p.cap] = p.root_board[b];
        p.parent[(long long)g * p.cap] = -1;
        s.size = 1;
        s.max_depth = 0;
        s.depth_sum = 0;
        s.root_turn = turn;
        s.status = 0;
        s.plies = 0;
        s.ub = 0;
        s.selected = 0;
        s.path_len = 1;
    } else {
        s.size = st->size;
        s.max_depth = st->max_depth;
        s.depth_sum = st->depth_sum;
        s.root_turn = meta_turn(rec[0].w);
        s.status = st->status;
        s.plies = st->plies;
        s.ub = st->ub_draws;
        s.selected = st->selected;
        s.path_len = st->path_len;
    }
    for (int k = 0; k < 4; k++) s.stage_cycles[k] = 0;
    // the "last step" arrays of the reference live as long as the instance: a new search starts from what the
    // previous one left in them (trees_actions_expanded keeps stale entries in the thrifty layout)
    s.out_neg = st->out_neg;
    s.out_pos = st->out_pos;
    for (int a = 0; a < A; a++) {
        s.child_out[a][0] = p.child_out[(g * A + a) * 2 + 0];
        s.child_out[a][1] = p.child_out[(g * A + a) * 2 + 1];
    }
    for (int a = 0; a < A + 2; a++) s.ae[a] = p.actions_expanded[g * (A + 2) + a];
}

// and back.  One thread.
__device__ __forceinline__ void store_tree(const SearchParams &p, const Walk &s, int g, bool first) {
    TreeState *st = p.state + g;
    st->size = s.size;
    st->max_depth = s.max_depth;
    st->depth_sum = s.depth_sum;
    st->selected = s.selected;
    st->path_len = s.path_len;
    st->out_neg = s.out_neg;
    st->out_pos = s.out_pos;
    st->status = s.status;
    st->plies = s.plies;
    st->ub_draws = s.ub;
    for (int k = 0; k < 4; k++) st->stage_ms[k] = (first ? 0.f : st->stage_ms[k]) + (float)s.stage_cycles[k] * p.ms_per_cycle;
    for (int a = 0; a < A; a++) {
        p.child_out[(g * A + a) * 2 + 0] = s.child_out[a][0];
        p.child_out[(g * A + a) * 2 + 1] = s.child_out[a][1];
    }
    for (int a = 0; a < A + 2; a++) p.actions_expanded[g * (A + 2) + a] = s.ae[a];
    for (int e = 0; e < s.path_len; e++) p.paths[g * PATH_CAP + e] = s.path[e];
}

// Backup of a step (_backup_* of the reference) by one warp, after prepare_backup; wins(j): games of slot j won by -1 and by +1.
template <bool OCP, class Wins>
__device__ __forceinline__ void backup(Walk &s, int4 *rec, int4 *cache, int cache_n, double c_ucb, int P, int lane, Wins wins) {
    __syncwarp();
    const unsigned c_backup = (unsigned)clock();
    const int mode = s.mode;
    const int exp_mask = s.exp_mask;
    const int sel_meta = s.sel_meta;
    const int child_turn = -meta_turn(sel_meta);
    const int plen = s.path_len;
    // Lanes 0..6: the children of the expanded node (lane = action).  The other lanes: the levels of the path.
    int neg_tot = 0, pos_tot = 0;
    int n_tot = P;
    int my_neg = 0, my_pos = 0;
    const int k = __popc(exp_mask & ((1 << lane) - 1));
    const bool child = mode == MODE_ALL_CHILDREN && lane < A && ((exp_mask >> lane) & 1);
    bool played = false;
    int outcome = 2;
    if (child) {
        outcome = s.child_outcome[k];
        const int j = s.child_slot[k];
        played = !OCP || k == s.pick;
        if (j >= 0) {
            const int2 won = wins(j);
            my_neg = won.x;
            my_pos = won.y;
        } else if (played) {
            // a terminal child: its stored outcome stands for all P playouts (src/mctsnc.py:2016-2021)
            my_neg = outcome == -1 ? P : 0;
            my_pos = outcome == 1 ? P : 0;
        }
        if (!OCP) {
            s.child_out[lane][0] = my_neg;
            s.child_out[lane][1] = my_pos;
        }
    }
    if (mode == MODE_ALL_CHILDREN) {
        // the sums of the children's games, both in one reduction (at most 7 * 512 games a side)
        const int both = __reduce_add_sync(0xFFFFFFFFu, my_neg | (my_pos << 16));
        neg_tot = both & 0xFFFF;
        pos_tot = both >> 16;
        if (!OCP) n_tot = P * __popc(exp_mask);
    } else if (mode == MODE_TERMINAL) {
        neg_tot = s.out_neg;
        pos_tot = s.out_pos;
    } else {
        const int2 won = wins(0);
        neg_tot = won.x;
        pos_tot = won.y;
        if (!OCP && lane == 0) {
            s.child_out[0][0] = neg_tot;
            s.child_out[0][1] = pos_tot;
        }
    }
    // The counts and wins of the path change the UCBs of its own nodes' children only, so this is where the child
    // that the next select goes on to is decided: on every level of the path the child on the path against the
    // best of the others, at its end the best of the new children.
    constexpr int LEVEL_LANES = 32 - 8;
    const int root_turn = s.root_turn;
    for (int base = 0; base < plen; base += LEVEL_LANES) {
        const int e = lane < 8 ? plen - 1 : base + lane - 8;
        const bool level = lane >= 8 && e < plen - 1;
        const int turn_e = (e & 1) ? -root_turn : root_turn;
        int wins_n = turn_e == 1 ? pos_tot : neg_tot;   // of the child on the path: the other side's
        if (level) wins_n += s.path_rec[e + 1].y;
        else wins_n = turn_e == 1 ? my_pos : my_neg;
        const PathTerm t = s.term[min(e, plen - 1)];
        const bool evaluate = level || (child && played);
        unsigned key = evaluate ? ordered_key(ucb_value(c_ucb, t.explore, t.n, t.reciprocal, wins_n)) : 0u;
        if (child && !played) key = ordered_key(__int_as_float(0x7f800000));
        int leaf_best = 0;
        if (base == 0 && mode == MODE_ALL_CHILDREN) {
            const unsigned leaf_key = lane < 8 ? key : 0u;
            const unsigned best = __reduce_max_sync(0xFFFFFFFFu, leaf_key);
            const int a = pick_among_tied(__ballot_sync(0xFFFFFFFFu, leaf_key != 0u && leaf_key == best));
            leaf_best = __popc(exp_mask & ((1 << a) - 1));
            // children start from ns = ns_wins = 0 (src/mctsnc.py:1819-1820), then _backup_1_acp_* / the
            // thread-0 part of _backup_ocp credit them (:2172-2177, :2104-2114)
            if (child)
                rec_store(rec, cache, cache_n, s.first_child + k,
                          make_int4(played ? P : 0, played ? wins_n : 0, -1,
                                    make_meta(0, outcome != 2, outcome, child_turn, meta_depth(sel_meta) + 1)));
        }
        if (level || (lane == 7 && base == 0)) {   // lane 7: the end of the path
            int4 r = s.path_rec[e];
            r.x += n_tot;
            r.y += turn_e == 1 ? neg_tot : pos_tot;
            if (level) {
                if (key < t.other_key || (key == t.other_key && !(t.other & 256)))
                    r.w = (r.w & ~META_BEST_MASK) | ((t.other & 7) << META_BEST_SHIFT);
            } else if (mode == MODE_ALL_CHILDREN) {
                r.z = s.first_child;
                r.w |= exp_mask | (leaf_best << META_BEST_SHIFT);
            }
            rec_store(rec, cache, cache_n, s.path[e], r);
        }
    }
    __syncwarp();
    if (lane == 0) {
        s.out_neg = neg_tot;
        s.out_pos = pos_tot;
        s.stage_cycles[2] += c_backup - s.stage_mark;
        s.stage_cycles[3] += (unsigned)clock() - c_backup;
    }
    __syncwarp();
}

struct Selected {
    int mode, n_slots, depth, meta;
};

// Select and expand of a step by one warp.  put(j, slot, mover) takes slot j (`mover`: the side to move there) and empties its
// tally.
template <bool OCP, class Put>
__device__ __forceinline__ Selected select_expand(const SearchParams &p, Walk &s, int4 *rec, ulonglong2 *board, int *parent, int4 *cache,
                                                  int cache_n, ulonglong2 &pick_stream, int lane, Put put) {
    const int P = p.n_playouts;
    const bool thrifty = (p.variant == 0 || p.variant == 2);
    // A node names the child that the arg-max over its children's UCBs picks (the backup of every path keeps that up to
    // date), so the walk is one dependent load per level.
    const unsigned c_step = (unsigned)clock();   // 32-bit cycle counts: differences are right modulo 2^32
    int node = 0;
    int4 r = rec_load(rec, cache, cache_n, 0);
    int depth = 0;
    if (lane == 0) {
        s.path[0] = 0;
        s.path_rec[0] = r;
    }
    while ((r.w & 0x7F) != 0 && depth < MAX_PATH - 2) {
        node = r.z + meta_best(r.w);
        r = rec_load(rec, cache, cache_n, node);
        depth++;
        if (lane == 0) {
            s.path[depth] = node;
            s.path_rec[depth] = r;
        }
    }
    // ------------------------------------------------------- expand (_expand_1_* and _expand_2_*)
    const unsigned c_expand = (unsigned)clock();
    const int sel_turn = meta_turn(r.w);
    int mode, n_exp = 0, exp_mask = 0, first_child = -1, pick = 0, n_slots = 0;
    if (r.w & META_TERMINAL) {
        mode = MODE_TERMINAL;
        if (lane == 0) {
            const int o = meta_outcome(r.w);
            s.out_neg = o == -1 ? P : 0;
            s.out_pos = o == 1 ? P : 0;
        }
    } else {
        const ulonglong2 bb = board[node];  // x: stones of -1, y: stones of +1
        const unsigned long long all = bb.x | bb.y;
        const unsigned legal = legal_columns(all);
        const int n_legal = __popc(legal);
        long long room = p.node_limit - (long long)s.size;
        if (room < 0) room = 0;
        n_exp = n_legal < room ? n_legal : (int)room;
        exp_mask = (int)legal;
        for (int drop = n_legal - n_exp; drop > 0; drop--)  // keep the n_exp lowest legal actions
            exp_mask &= ~(1 << (31 - __clz(exp_mask)));
        if (n_exp < n_legal && lane == 0) s.status |= STATUS_TREE_FULL;
        if (n_exp > 0) {
            mode = MODE_ALL_CHILDREN;
            first_child = s.size;
            if (OCP) {
                // src/mctsnc.py:1435 / :1511 -- float32 * int64 is a float64 product, truncated
                if (lane == 0) {
                    const float u = rng_uniform_f32(pick_stream.x, pick_stream.y);
                    pick = __double2int_rz((double)u * (double)n_exp);
                    if (pick >= n_exp) {  // u == 1.0f: undefined in the reference, clamped
                        pick = n_exp - 1;
                        s.ub++;
                        s.status |= STATUS_UB_DRAW;
                    }
                }
                pick = __shfl_sync(0xFFFFFFFFu, pick, 0);
            }
            const bool has_child = lane < A && ((exp_mask >> lane) & 1);
            const int k = __popc(exp_mask & ((1 << lane) - 1));
            unsigned long long cneg = bb.x, cpos = bb.y, call = all;
            int outcome = 2;
            if (has_child) {
                const unsigned long long move = (all + (1ULL << column_shift(lane))) & (0x3FULL << column_shift(lane));
                if (sel_turn > 0) cpos |= move;
                else cneg |= move;
                call = all | move;
                const bool win = has_four(sel_turn > 0 ? cpos : cneg);
                outcome = win ? sel_turn : (call == FULL_BOARD ? 0 : 2);
                board[first_child + k] = make_ulonglong2(cneg, cpos);
                parent[first_child + k] = node;
            }
            const bool plays = has_child && outcome == 2 && (!OCP || k == pick);
            const unsigned play_mask = __ballot_sync(0xFFFFFFFFu, plays);
            n_slots = __popc(play_mask);
            if (has_child) {
                const int j = plays ? __popc(play_mask & ((1u << lane) - 1u)) : -1;
                s.child_outcome[k] = outcome;
                s.child_slot[k] = j;
                if (plays) {
                    GameSlot gs;
                    const unsigned open = legal_columns(call);
                    gs.cur = sel_turn > 0 ? cneg : cpos;  // the child is to be moved in by the other side
                    gs.other = sel_turn > 0 ? cpos : cneg;
                    gs.row = move_row(open);
                    gs.count = (float)__popc(open) * RNG_2M64;
                    gs.rng_base = OCP ? 0 : lane * P;
                    gs.stones = __popcll(call);
                    put(j, gs, -sel_turn);
                }
            }
        } else {
            // no room for a single child: the selected node itself is played out
            mode = MODE_TREE_FULL;
            n_slots = 1;
            if (lane == 0) {
                GameSlot gs;
                gs.cur = sel_turn > 0 ? bb.y : bb.x;
                gs.other = sel_turn > 0 ? bb.x : bb.y;
                gs.row = move_row(legal);
                gs.count = (float)n_legal * RNG_2M64;
                gs.rng_base = 0;
                gs.stones = __popcll(all);
                put(0, gs, sel_turn);
            }
        }
    }
    // trees_actions_expanded in the layout of the variant (src/mctsnc.py:1430-1454, :1509-1531, :1583-1604,
    // :1656-1681)
    if (lane < A) {
        if (thrifty) {
            if (mode == MODE_ALL_CHILDREN && ((exp_mask >> lane) & 1))
                s.ae[__popc(exp_mask & ((1 << lane) - 1))] = (short)lane;
        } else {
            if (mode == MODE_ALL_CHILDREN) s.ae[lane] = ((exp_mask >> lane) & 1) ? (short)lane : (short)-1;
            else s.ae[lane] = -1;
        }
    }
    __syncwarp();
    if (lane == 0) {
        if (mode == MODE_ALL_CHILDREN) {
            s.size += n_exp;
            s.depth_sum += n_exp * (depth + 1);
            s.max_depth = max(s.max_depth, depth + 1);
        }
        s.ae[A + 1] = (short)(mode == MODE_ALL_CHILDREN ? n_exp : 1);
        int m2 = mode;
        if (OCP && mode == MODE_ALL_CHILDREN) m2 = thrifty ? pick : nth_set(exp_mask, pick);
        s.ae[A] = (short)m2;
        if (!OCP && mode != MODE_ALL_CHILDREN) s.ae[0] = 0;
        s.n_slots = n_slots;
        s.pick = pick;
        s.mode = mode;
        s.exp_mask = exp_mask;
        s.first_child = first_child;
        s.selected = node;
        s.sel_meta = r.w;
        s.path_len = depth + 1;
        const unsigned c_play = (unsigned)clock();
        s.stage_cycles[0] += c_expand - c_step;
        s.stage_cycles[1] += c_play - c_expand;
        s.stage_mark = c_play;
    }
    return {mode, n_slots, depth, r.w};
}

// Shared-memory address of the table less the offset of the float exponent: address of entry i = base + 8 * (bits of the
// float 2^23 + i), modulo 2^32
__device__ __forceinline__ unsigned move_lut_base(const MoveEntry *move_lut) {
    return (unsigned)__cvta_generic_to_shared(move_lut) - MOVE_LUT_BASE_BITS * (unsigned)sizeof(MoveEntry);
}
__device__ __forceinline__ MoveEntry load_move(unsigned base, unsigned float_bits) {
    MoveEntry m;
    asm("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(m.lo), "=r"(m.hi) : "r"(base + float_bits * (unsigned)sizeof(MoveEntry)));
    return m;
}

// A column that has just been filled (`filled` != 0) leaves the set of columns with room: `row` drops by 8 << column, a power of
// two whose exponent is the column's byte number in the entry's low bits (the shift's other bits fall out, but for the
// bottom cell of column 0, which flips the sign: that is why the set's bit 0 is kept inverted).  Two predicated additions:
// the branch the compiler makes of it cost the warp its resolving on every ply.
__device__ __forceinline__ void close_column(unsigned filled, float &row, float &count, unsigned entry_lo, unsigned times2p23) {
    const unsigned drop = entry_lo * times2p23 + (0x80000000u + (129u << 23));
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p add.rn.f32 %0, %0, %3;\n\t@p add.rn.f32 %1, %1, %4;\n\t}"
        : "+f"(row), "+f"(count) : "r"(filled), "f"(__uint_as_float(drop)), "f"(-RNG_2M64));
}

// fours of the side that has just put a stone into the column of entry `entry_lo`: a new vertical four can only be in that
// column, whose byte is tested alone
// (the permute takes the entry as it is: its other selectors name byte 0 or columns that hold no four)
// (shifts to the left: the multiply-add pipe can do those too, and the logic pipe is the busy one; 118.4 -> 115 ms on the headline
// batch, 23.1 -> 22.5 ms on the ocp batch)
__device__ __forceinline__ unsigned fours_with(unsigned lo, unsigned hi, unsigned entry_lo, unsigned before, unsigned two, unsigned four) {
    unsigned v = __byte_perm(lo, hi, entry_lo);
    v &= v * two;
    return fours_across(lo, hi, before) | (v & (v * four));
}

// A game in progress: three pairs of words -- the stones of the side that moves at the even plies of a block of PLIES plies (a
// game starts at ply 0 of a block, so that is the side to move in the game's first position), the stones of the other side, and
// `top`, one bit per column at its lowest empty cell (the guard bit once the column is full; top = all stones + bottom row).
// A move in a column with room is then top & (six cells of the column), and top + move puts the marker one cell up; columns
// are bytes, so the two words never carry.
//
// A block has no branch: a game that has been won plays on to its end, and what it does then is not looked at, but its generator
// must stop where the game did.
//   STRAIGHT (one game per thread, where a ply's latency counts): the generator does not wait for the four tests and goes back
//   when the game is closed, so that a ply's chain is only the one from the table to the next index.
//   Otherwise (several games per thread, where instructions count): its step is predicated on the tests of the plies before.  (With
//   a branch behind every ply, 65 instructions a ply: moves where the paths meet.)
__device__ __forceinline__ unsigned top_low(unsigned occupied_lo) { return occupied_lo + BOTTOM_LO + MARK; }
__device__ __forceinline__ unsigned top_high(unsigned occupied_hi) { return occupied_hi + BOTTOM_HI; }

//   AHEAD (STRAIGHT, where the threads that play idle while the walker makes the next step): the draws come out of a ring per stream
//   that those threads fill meanwhile, see Draws.
constexpr int AHEAD_DRAWS = 64;     // of a stream: no fewer than a game can use, 42 and the rest of its last block
constexpr int AHEAD_STRIDE = AHEAD_DRAWS + PLIES_PER_CHECK + 1;   // floats: the first ones again behind the last, and an odd number
static_assert(AHEAD_DRAWS >= ROWS * COLS + STRAIGHT_PLIES && STRAIGHT_PLIES <= PLIES_PER_CHECK, "a block of draws is read in one piece");

template <bool STRAIGHT, bool AHEAD = false>
struct Game {
    static_assert(STRAIGHT || !AHEAD, "draws made ahead: one game per thread");
    static constexpr int PLIES = STRAIGHT ? STRAIGHT_PLIES : PLIES_PER_CHECK;
    static_assert(PLIES % 2 == 0, "the two sides alternate by the parity of the ply within a block; the way back takes a power of two");
    unsigned even_lo = 0, even_hi = 0, odd_lo = 0, odd_hi = 0, top_lo = 0, top_hi = 0;
    unsigned long long s0 = 0, s1 = 0;
    float row = 0.f, count = 0.f;
    int stones = 0;
    int drawn = 0;        // draws of the game, those behind its end too where STRAIGHT
    unsigned ring = 0;    // AHEAD: shared-memory address of the stream's ring, and the ring's place of the game's first draw
    int place = 0;
    unsigned fours = 0;   // of the last block (STRAIGHT: bit k for ply k)

    __device__ __forceinline__ void start(const GameSlot &gs, unsigned first_top_lo, unsigned first_top_hi, const ulonglong2 &stream) {
        even_lo = (unsigned)gs.cur;
        even_hi = (unsigned)(gs.cur >> 32);
        odd_lo = (unsigned)gs.other;
        odd_hi = (unsigned)(gs.other >> 32);
        top_lo = first_top_lo;
        top_hi = first_top_hi;
        row = gs.row;
        count = gs.count;
        stones = gs.stones;
        s0 = stream.x;
        s1 = stream.y;
        drawn = -(stones & ~255);
    }
    __device__ __forceinline__ void play_block(unsigned lut_base, const SearchParams &p) {
        fours = 0u;
        float ahead[PLIES];
        if (AHEAD) {
            const unsigned at = ring + (unsigned)((place + drawn) & (AHEAD_DRAWS - 1)) * 4u;
#pragma unroll
            for (int k = 0; k < PLIES; k++) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(ahead[k]) : "r"(at + 4u * k));
        }
        if (STRAIGHT) drawn += PLIES;
        // (a warp that is alone on its scheduler has no pipe to spare and is better off with the shifts)
        const unsigned two = STRAIGHT ? 2u : p.times2, four = STRAIGHT ? 4u : p.times4, two23 = STRAIGHT ? 1u << 23 : p.times2p23;
#pragma unroll
        for (int k = 0; k < PLIES; k++) {
            // ---- one ply (src/mctsnc.py:2059-2064, :2069)
            // float32 u * int16 count -> float32 (:2061); here (u * 2^64) * (count * 2^-64): the same product
            float f;
            if (AHEAD) {
                f = ahead[k];
            } else if (STRAIGHT || k == 0) {
                f = rng_uniform_times_2p64(s0, s1);
                if (!STRAIGHT) drawn++;
            } else {
                f = rng_uniform_times_2p64_unless(fours, s0, s1, drawn);
            }
            const MoveEntry m = load_move(lut_base, __float_as_uint(__fadd_rz(__fmul_rn(f, count), row)));
            const unsigned move_lo = top_lo & m.lo, move_hi = top_hi & m.hi;
            top_lo += move_lo;
            top_hi += move_hi;
            // The sides take turns with the plies of the unrolled block: no swap of "mine" and "theirs".  The cell was empty, so the
            // stone is added (an addition can go to the multiply-add pipe, an OR cannot; 25.1 -> 24.4 ms on a fifth of the headline batch).
            const unsigned before = STRAIGHT ? 0u : fours;
            unsigned made;
            if (k & 1) {
                odd_lo += move_lo;
                odd_hi += move_hi;
                made = fours_with(odd_lo, odd_hi, m.lo, before, two, four);
            } else {
                even_lo += move_lo;
                even_hi += move_hi;
                made = fours_with(even_lo, even_hi, m.lo, before, two, four);
            }
            if (!STRAIGHT) fours = made;
            else if (made != 0u) fours |= 1u << k;
            close_column((move_lo & TOP_LO) | (move_hi & TOP_HI), row, count, m.lo, two23);
        }
    }
    __device__ __forceinline__ bool marked() const { return ((even_lo | odd_lo) & MARK) != 0u; }   // a draw of 1.0f, see MoveEntry
    __device__ __forceinline__ bool over() const { return fours != 0u || marked() || row == NO_MOVES; }
    // Plies of the game that has just ended (the last one was made by the first mover iff they are odd), less any multiple of 256
    // that was added to the `stones` of its slot; the generator goes back to where the game left it.
    __device__ __forceinline__ int finish() {
        int n = drawn;
        if (fours == 0u) n = __popc(even_lo | odd_lo) + __popc(even_hi | odd_hi) - stones;   // the board is full
        else if (STRAIGHT) n = drawn - PLIES + __ffs(fours);
        if (!AHEAD && (STRAIGHT || fours == 0u))
            for (int k = drawn - n; k > 0; k--) rng_back(s0, s1);
        return n;
    }
};

// The draws of a block's streams made ahead: of every stream the next AHEAD_DRAWS, scaled by 2^64, in a ring that starts at `place`.
// The stream's state in the block's array is the one behind them; `used`: draws of the step's game, made up by refill while the
// walker makes the next step and the threads that play would wait for it.  A ply has 14 of 58 instructions less then, and
// nothing is taken back when a game is closed; what the threads lose is a part of the walker's issue slots.  One search of 1000
// steps, without / with: 1 x 32 ocp 4.75 / 4.57 ms, 8 x 256 ocp 5.61 / 5.57, 4 x 32 acp 5.31 / 4.92; on clusters 4 x 64 acp 5.59 / 5.41, 4 x 256
// 5.81 / 5.72, 4 x 512 7.93 / 7.51.  With two to four warps that play the walker loses more than they gain: 4 x 128 ocp 4.69 / 4.96, 4 x 64
// ocp 4.72 / 4.82, on clusters 4 x 128 acp 5.67 / 5.70.
struct Draws {
    float *ring;       // [streams][AHEAD_STRIDE]
    int *place, *used; // [streams]
    static __host__ __device__ size_t bytes(int streams) { return (size_t)streams * (AHEAD_STRIDE * sizeof(float) + 2 * sizeof(int)); }
    __device__ __forceinline__ Draws(void *memory, int streams) {
        ring = reinterpret_cast<float *>(memory);
        place = reinterpret_cast<int *>(ring + (size_t)streams * AHEAD_STRIDE);
        used = place + streams;
    }
    // `count` more of stream i, over those that have been used
    __device__ __forceinline__ void make(ulonglong2 *s_rng, int i, int count) {
        ulonglong2 state = s_rng[i];
        float *mine = ring + i * AHEAD_STRIDE;
        int at = place[i];
        for (; count > 0; count--) {
            const float f = rng_uniform_times_2p64(state.x, state.y);
            mine[at] = f;
            if (at < PLIES_PER_CHECK) mine[AHEAD_DRAWS + at] = f;
            at = (at + 1) & (AHEAD_DRAWS - 1);
        }
        s_rng[i] = state;
        place[i] = at;
    }
    __device__ __forceinline__ void refill(ulonglong2 *s_rng, int i) {
        const int n = used[i];
        if (n == 0) return;
        used[i] = 0;
        make(s_rng, i, n);
    }
    // where the stream stands: before the draws of the ring
    __device__ __forceinline__ ulonglong2 state_of(const ulonglong2 *s_rng, int i) const {
        ulonglong2 state = s_rng[i];
        for (int k = 0; k < AHEAD_DRAWS; k++) rng_back(state.x, state.y);
        return state;
    }
};

// `n_steps` steps of tree g by the whole block, from the state the tree has in global memory and back to it.
// The random streams of the tree (ACP: 7*P, OCP: P states of 16 B) stay in dynamic shared memory meanwhile: they are
// read at the start of every game and written back at its end, by one thread each.
//
// CL > 1: a thread-block cluster of CL blocks grows the tree (launches with so few trees that a tree would otherwise be
// bound by what one SM can play per step).  The first block of the cluster walks, expands and backs up as before and
// hands the step's games (slots) to the shared memory of the others; every block plays the games of P / CL of the P
// playout indices of every child -- it keeps the streams of exactly those in its shared memory -- and adds its tallies
// to the first block's `gather`.  Two cluster barriers per step; all blocks run the same loop, so every block reaches
// every barrier.
//
// STRAIGHT: how a game is played, see the playouts.
// AHEAD: draws made ahead (by all warps but the walker's, of which there is at least one), in `ahead`.
template <bool OCP, int CL, bool STRAIGHT, bool AHEAD>
__device__ __forceinline__ void run_slice(const SearchParams &p, Shared &s, ulonglong2 *s_rng, int4 *cache, void *ahead, const int g,
                                          const int n_steps, const bool first) {
    namespace cg = cooperative_groups;
    const int cache_n = CL > 1 ? p.cache_nodes : 0;
    static_assert(CL == 1 || CL == 8 || CL == 16, "cluster sizes");
    constexpr int LOG_CL = CL == 16 ? 4 : (CL == 8 ? 3 : 0);
    const int tid = threadIdx.x;
    const int nt = blockDim.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int P = p.n_playouts;
    const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int log2_local = p.log2_playouts - LOG_CL;   // this block plays P_local = P / CL playout indices of every child
    const int P_local = P >> LOG_CL;
    int4 *rec = p.rec + (long long)g * p.cap;
    ulonglong2 *board = p.board + (long long)g * p.cap;
    int *parent = p.parent + (long long)g * p.cap;
    const bool walker = warp == 0 && rank == 0;   // the warp that selects, expands and backs up
    // threads whose first game of a step is fixed by their number: all, but for the walker where it is not the only warp
    const int first_free_item = rank == 0 && nt > 32 ? nt - 32 : nt;
    const unsigned lut_base = move_lut_base(s.move_lut);

    const int n_streams = OCP ? P : A * P;
    ulonglong2 *g_rng = p.rng_playout + (long long)g * n_streams;
    // stream (action, t) of the tree sits at local index action * P_local + (t - rank * P_local)
    for (int i = tid; i < (n_streams >> LOG_CL); i += nt)
        s_rng[i] = g_rng[((i >> log2_local) << p.log2_playouts) + rank * P_local + (i & (P_local - 1))];
    Draws draws(ahead, n_streams >> LOG_CL);
    if (AHEAD)
        for (int i = tid; i < (n_streams >> LOG_CL); i += nt) {
            draws.place[i] = draws.used[i] = 0;
            draws.make(s_rng, i, AHEAD_DRAWS);
        }
    if (CL > 1 && tid < 2 * A) s.tally[tid >> 1][tid & 1] = 0;
    if (tid == 0 && rank == 0) {
        load_tree(p, s, g, first, cache, cache_n);
    }
    if (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (CL > 1 && rank == 0 && !first) {   // a search that goes on: the records the tree has so far
        const int have = s.size < cache_n ? s.size : cache_n;
        for (int i = tid; i < have; i += nt) cache[i] = rec[i];
        __syncthreads();
    }

    const double c_ucb = (double)p.ucb_c;
    unsigned my_plies = 0, my_ub = 0, my_err = 0;
    ulonglong2 pick_stream = make_ulonglong2(0ULL, 0ULL);   // OCP: the stream of the child picks (lane 0 of the walker)
    if (OCP && walker && lane == 0) pick_stream = p.rng_expand[g];

    // The walker warp runs steps on its own for as long as they select a terminal node (nothing to play: the backup follows
    // at once) and meets the other threads only for a step with games, or when the steps are done (MODE_DONE).
    int step = 0;
    bool backup_due = false;   // the walker's: the step it selected last has not been backed up yet
    for (;;) {
        // =========================================================== backup of the step before, select + expand (warp 0)
        if (walker) for (;;) {
            if (backup_due) {
                const int (*tally)[2] = CL > 1 ? s.gather : s.tally;
                backup<OCP>(s, rec, cache, cache_n, c_ucb, P, lane, [&](int j) { return make_int2(tally[j][0], tally[j][1]); });
                backup_due = false;
            }
            if (step == n_steps) {
                if (lane == 0) s.mode = MODE_DONE;
                if (CL > 1 && lane > 0 && lane < CL) cg::this_cluster().map_shared_rank(&s, lane)->mode = MODE_DONE;
                break;
            }
            const Selected leaf = select_expand<OCP>(p, s, rec, board, parent, cache, cache_n, pick_stream, lane, [&](int j, const GameSlot &gs, int) {
                s.slot[j] = gs;
                s.tally[j][0] = 0;
                s.tally[j][1] = 0;
                s.gather[j][0] = 0;
                s.gather[j][1] = 0;
            });
            if (lane == 0) s.next_item = first_free_item;
            step++;
            backup_due = true;
            if (leaf.mode == MODE_TERMINAL) {
                __syncwarp();
                prepare_backup<OCP>(s, rec, cache, cache_n, c_ucb, lane, leaf.depth + 1, P, 0);
                continue;
            }
            if (CL > 1) {
                // the step's games for the other blocks of the cluster: stores into their shared memory, made visible by
                // the barrier below
                __syncwarp();
                // A lane for every block where one lane's stores would be many times those of another way round: sixteen blocks (one
                // search of 4 x 256, 1000 steps, 5.99 -> 5.71 ms) or a single slot (4 x 512 ocp 5.76 -> 5.61).  Eight blocks and seven
                // slots are as well off with a lane for every slot (4 x 64 5.31 against 5.36).
                auto tell = [&](Shared *rs) {
                    rs->n_slots = leaf.n_slots;
                    rs->mode = leaf.mode;
                    rs->sel_meta = leaf.meta;
                    rs->next_item = nt;
                };
                if (CL == 16 || OCP) {
                    if (lane > 0 && lane < CL) {
                        Shared *rs = cg::this_cluster().map_shared_rank(&s, lane);
                        for (int k = 0; k < leaf.n_slots; k++) rs->slot[k] = s.slot[k];
                        tell(rs);
                    }
                } else {
                    for (int other = 1; other < CL; other++) {
                        Shared *rs = cg::this_cluster().map_shared_rank(&s, other);
                        if (lane < leaf.n_slots) rs->slot[lane] = s.slot[lane];
                        if (lane == 0) tell(rs);
                    }
                }
            }
            break;
        }
        // the others make up the draws that the games have used (five warps: not the one that shares the walker's scheduler)
        if (AHEAD && CL == 16 && rank == 0) {
            if (warp & 3)
                for (int i = tid - 32; i < (n_streams >> LOG_CL); i += 3 * 32) draws.refill(s_rng, i);
        } else if (AHEAD && !walker) {
            for (int i = tid - (nt - first_free_item); i < (n_streams >> LOG_CL); i += first_free_item) draws.refill(s_rng, i);
        }
        if (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
        if (s.mode == MODE_DONE) break;

        // =========================================================== playouts (all threads)
        // Games are handed out one at a time from a counter in shared memory, so the threads of the block stay busy
        // until the step's games run out whatever their lengths.  Game `item` is playout t = item % P of slot
        // item / P; it draws from the stream the reference's thread (tree, action, t) owns (src/mctsnc.py:1938, :2028;
        // OCP: cuda.grid(1), :1849), so which thread plays it does not matter.
        //
        // The first game of every thread is its own number.  The walker has the counts and logarithms of the backup to work
        // out first and takes what games are left after that.
        {
            const int n_items = s.n_slots << log2_local;
            // the side to move in the played-out positions: the other side than at the selected node, unless the
            // selected node itself is played out
            const int first_mover = (s.mode == MODE_TREE_FULL) ? meta_turn(s.sel_meta) : -meta_turn(s.sel_meta);
            Game<STRAIGHT, AHEAD> game;
            int rng_idx = 0, j = 0;
            int item = tid - (nt - first_free_item);
            if (walker) {
                const int sel_n = s.mode == MODE_ALL_CHILDREN && !OCP ? P * __popc(s.exp_mask) : P;
                prepare_backup<OCP>(s, rec, cache, cache_n, c_ucb, lane, s.path_len, sel_n, s.mode == MODE_ALL_CHILDREN ? P : 0);
                if (item < 0) item = atomicAdd(&s.next_item, 1);
            }
            auto start_game = [&]() {
                j = item >> log2_local;
                const GameSlot gs = s.slot[j];
                rng_idx = (gs.rng_base >> LOG_CL) + (item & (P_local - 1));
                const unsigned long long occupied = gs.cur | gs.other;
                game.start(gs, top_low((unsigned)occupied), top_high((unsigned)(occupied >> 32)), AHEAD ? make_ulonglong2(0, 0) : s_rng[rng_idx]);
                if (AHEAD) {
                    game.ring = (unsigned)__cvta_generic_to_shared(draws.ring + rng_idx * AHEAD_STRIDE);
                    game.place = draws.place[rng_idx];
                }
            };
            auto close_game = [&]() {
                int n = game.finish();
                int winner = 0;
                if (game.fours != 0u) winner = (n & 1) ? first_mover : -first_mover;
                if (game.marked()) {
                    // u == 1.0f somewhere in this game: replay it through the byte-level emulation of the reference
                    const GameSlot gs = s.slot[j];
                    const ulonglong2 rs = AHEAD ? draws.state_of(s_rng, rng_idx) : s_rng[rng_idx];
                    const EmuResult er = playout_emulated(first_mover > 0 ? gs.other : gs.cur, first_mover > 0 ? gs.cur : gs.other,
                                                          first_mover, rs.x, rs.y);
                    game.s0 = er.s0;
                    game.s1 = er.s1;
                    winner = er.outcome == 2 ? 0 : er.outcome;
                    n = (int)er.plies;
                    my_ub += er.ub;
                    my_err |= er.err;
                }
                if (AHEAD) draws.used[rng_idx] = n;   // one draw a ply
                else s_rng[rng_idx] = make_ulonglong2(game.s0, game.s1);
                my_plies += n;
                if (winner != 0) atomicAdd(&s.tally[j][winner > 0 ? 1 : 0], 1);
                item = atomicAdd(&s.next_item, 1);
            };
            if (STRAIGHT) {
                // About one game per thread: a warp plays its games to the end together and closes them together.  Closed one by
                // one, every game that ends would hold up the ones still going on in its warp by the closing (a few hundred
                // cycles of shared-memory atomics and the generator's way back, nine times per 32 games).
                while (__any_sync(0xFFFFFFFFu, item < n_items)) {
                    if (item < n_items) {
                        start_game();
                        do game.play_block(lut_base, p);
                        while (!game.over());
                    }
                    __syncwarp();
                    if (item < n_items) close_game();
                }
            } else {
                // Several games per thread: a lane takes its next game at once.  A finished game is noticed only every PLIES
                // plies (its lane sits out the plies in between): the code that closes a game and starts the next one (about 40
                // instructions) runs for the few lanes whose games have just ended while the others wait, and with a look
                // after every ply it ran in nearly every iteration.
                if (item < n_items) start_game();
                while (item < n_items) {
                    game.play_block(lut_base, p);
                    if (game.over()) {
                        close_game();
                        if (item < n_items) start_game();
                    }
                }
            }
        }
        if (CL > 1) {
            // this block's tallies go to the first block's sums (atomic adds into its shared memory), then start from zero
            __syncthreads();
            if (tid < 2 * A) {
                const int v = s.tally[tid >> 1][tid & 1];
                if (v != 0) {
                    atomicAdd(&cg::this_cluster().map_shared_rank(&s, 0)->gather[tid >> 1][tid & 1], v);
                    s.tally[tid >> 1][tid & 1] = 0;
                }
            }
            cg::this_cluster().sync();
        } else {
            __syncthreads();
        }
    }

    // =============================================================== leave the per-tree state for the next launch
    {
        Shared *home = CL > 1 ? cg::this_cluster().map_shared_rank(&s, 0) : &s;   // the first block keeps the tree's counters
        if (my_plies) atomicAdd(&home->plies, (unsigned long long)my_plies);
        if (my_ub) {
            atomicAdd(&home->ub, (unsigned long long)my_ub);
            atomicOr(&home->status, STATUS_UB_DRAW);
        }
        if (my_err) atomicOr(&home->status, STATUS_INTERNAL);
    }
    if (OCP && walker && lane == 0) p.rng_expand[g] = pick_stream;
    if (CL > 1) cg::this_cluster().sync();   // also: no block leaves while another may still write to its shared memory
    else __syncthreads();
    for (int i = tid; i < (n_streams >> LOG_CL); i += nt)
        g_rng[((i >> log2_local) << p.log2_playouts) + rank * P_local + (i & (P_local - 1))] = AHEAD ? draws.state_of(s_rng, i) : s_rng[i];
    if (rank != 0) return;
    if (tid == 0) {
        store_tree(p, s, g, first);
    }
}

// One block grows one tree at a time.  Without a queue block b runs the whole launch of tree b.  With a queue (batched
// launches with more trees than blocks fit on the device) the grid is persistent and the blocks take slices of
// p.chunk steps of whichever tree is next in the ring.
__device__ __forceinline__ long long global_timer_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A slice of a queued launch is over (its writes precede, by a barrier): its record, and the ring in which the tree waits for its
// next one (-1: the tree has no steps left).  One thread.
__device__ __forceinline__ int finish_slice(const SearchParams &p, int g, int rem, int n_steps, long long t_start) {
    if (p.trace) {
        const int k = atomicAdd(p.trace_count, 1);
        if (k < p.trace_cap) {
            unsigned sm;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
            p.trace[4 * k] = g;
            p.trace[4 * k + 1] = t_start;
            p.trace[4 * k + 2] = global_timer_ns();
            p.trace[4 * k + 3] = ((long long)sm << 32) | (unsigned)n_steps;
        }
    }
    const int left = rem - n_steps;
    p.remaining[g] = left;
    __threadfence();
    if (left <= 0) return -1;
    // band of the time the tree still needs at the pace of this slice, counted down from the longest whole
    // search seen so far in this launch
    // the pace of a tree changes from slice to slice (its tree deepens, its neighbours on the SM change): half
    // the weight goes to the slices before (worth 1-2 % on the headline batch: 16.7-17.2 G playouts/s against
    // 16.6-16.8 with the last slice alone)
    float us_per_step = (float)(global_timer_ns() - t_start) * 1e-3f / (float)n_steps;
    if (rem != p.steps) us_per_step = 0.5f * us_per_step + 0.5f * p.state[g].us_per_step;
    p.state[g].us_per_step = us_per_step;
    const int whole = (int)fminf(us_per_step * (float)p.steps, 2e9f);
    const int longest = max(atomicMax(&p.queue->longest_us, whole), max(whole, 1));
    const float below = QUEUE_LEVELS_PER_OCTAVE * log2f((float)longest / fmaxf(us_per_step * (float)left, 1e-3f));
    return max(0, QUEUE_LEVELS - 1 - (int)fminf(fmaxf(below, 0.f), (float)QUEUE_LEVELS));
}

__device__ __forceinline__ void build_move_lut(MoveEntry *move_lut) {
    for (int i = threadIdx.x; i < 128 * 8; i += blockDim.x) {
        const int set = (i >> 3) ^ 1, ord = i & 7;
        MoveEntry m;
        m.lo = m.hi = 0u;
        if (ord < __popc(set)) {
            const int col = nth_set(set, ord);
            const unsigned long long cells = 0x3FULL << column_shift(col);
            m.lo = (unsigned)cells | (unsigned)(col + 1);
            m.hi = (unsigned)(cells >> 32);
        } else if (set != 0) {
            m.lo = MARK;
        }
        move_lut[i] = m;
    }
}

#ifndef MCTSNC_C4_MAXNREG
#define MCTSNC_C4_MAXNREG 64
#endif
template <bool OCP, bool STRAIGHT, bool AHEAD = false>
__global__ void __maxnreg__(MCTSNC_C4_MAXNREG) search_kernel(const SearchParams p) {
    __shared__ Shared s;
    extern __shared__ ulonglong2 s_rng[];
    const int tid = threadIdx.x;
    build_move_lut(s.move_lut);
    const bool queued = p.queue != nullptr;
    if (queued && tid == 0) s.held = -1;
    for (;;) {
        int g = blockIdx.x, rem = p.steps;
        if (queued) {
            if (tid == 0) {
                // Where a quarter more trees than blocks share the queue, the next tree is taken before the last one is put back, so that
                // trees go round the SMs: a tree with slow neighbours on its SM falls behind, has the most time left, and would be what
                // its own block takes next (with a block per tree for all of them: 256 x 4 x 256 acp, 300 steps, 20.7 instead of 22.4 ms;
                // 256 x 8 x 256 ocp, 500 steps, 16.9 instead of 18.2).  Where hardly any tree waits that order exchanges the trees with the most time left for those
                // with the least at every slice (600 x 4 x 128 ocp, 1000 steps, 2400 trees on 2368 blocks: 32.8 instead of 24.7 ms).
                int next = -1;
                const int held = s.held;
                if (held < 0 || 4 * p.ring_cap >= 5 * p.places) next = queue_pop(p.queue, p.ring, p.ring_cap);
                if (held >= 0) {
                    if (!queue_push(p.queue, p.ring, p.ring_cap, s.held_level, held)) atomicOr(&p.state[held].status, STATUS_INTERNAL);
                    if (next < 0) next = queue_pop(p.queue, p.ring, p.ring_cap);
                }
                s.job = next;
            }
            __syncthreads();
            g = s.job;
            if (g < 0) break;
            rem = p.remaining[g];
        }
        const int n_steps = (queued && rem > p.chunk) ? p.chunk : rem;
        long long t_start = 0;
        if (queued && tid == 0) t_start = global_timer_ns();
        run_slice<OCP, 1, STRAIGHT, AHEAD>(p, s, s_rng, nullptr, s_rng + (OCP ? 1 : A) * p.n_playouts, g, n_steps, p.first != 0 && rem == p.steps);
        if (!queued) break;
        __syncthreads();  // every thread's writes of the slice precede the fence of thread 0
        if (tid == 0) {
            s.held_level = finish_slice(p, g, rem, n_steps, t_start);
            s.held = s.held_level >= 0 ? g : -1;
        }
    }
}

// A cluster of CL blocks per tree: launches with few trees (one search), where a step of a tree is bound by what one SM can play.
// Launched with the cluster dimension as a launch attribute; cluster c grows tree c for the whole launch.  THREADS: of a block.
template <bool OCP, int CL, bool AHEAD>
__device__ __forceinline__ void run_cluster(const SearchParams &p) {
    __shared__ Shared s;
    extern __shared__ ulonglong2 s_rng[];
    build_move_lut(s.move_lut);
    const int n_local = ((OCP ? 1 : A) * p.n_playouts) / CL;   // streams this block keeps; the record cache follows
    int4 *cache = reinterpret_cast<int4 *>(s_rng + n_local);
    run_slice<OCP, CL, true, AHEAD>(p, s, s_rng, cache, cache + p.cache_nodes, (int)(blockIdx.x / CL), p.steps, p.first != 0);
}

template <bool OCP, int CL, int THREADS, bool AHEAD>
__global__ void __launch_bounds__(THREADS, 2) search_cluster_kernel(const SearchParams p) { run_cluster<OCP, CL, AHEAD>(p); }

// Clusters of 8 blocks of 256 threads, or -- from as many games a step as those blocks have threads beside the walking warp (1792) -- of
// 16 blocks of 128 and a warp for the walk: a scheduler has one warp of games then instead of two.  4 trees, ACP 64 /
// 128 / 256 / 512 playouts, us a step: 5.6 / 5.6 / 7.2 / 9.9 with 8 blocks, 6.0 / 6.0 / 6.8 / 8.4 with 16 (the barriers of the larger
// cluster cost more).
constexpr int CLUSTER_BLOCKS = 8, CLUSTER_THREADS = 256;
constexpr int WIDE_CLUSTER_BLOCKS = 16, WIDE_CLUSTER_THREADS = 160, WIDE_CLUSTER_MIN_GAMES = CLUSTER_BLOCKS * (CLUSTER_THREADS - 32);

// The same with the registers capped so that four blocks share an SM, for trees whose clusters do not fit otherwise (33 to 64 trees
// on 148 SMs, 64 registers instead of 128): 4 x 256 acp, 500 steps, 9 / 12 / 16 searches in one launch 4.97 / 5.58 / 6.99 ms against
// 11.14 with a block per tree.  Where both fit the cap costs: 1 / 8 searches of 4 x 64 acp 3.16 / 3.57 ms against 2.91 / 3.24.
template <bool OCP>
__global__ void __launch_bounds__(CLUSTER_THREADS, 4) search_packed_cluster_kernel(const SearchParams p) {
    run_cluster<OCP, CLUSTER_BLOCKS, false>(p);
}

}  // namespace c4
}  // namespace mctsnc
