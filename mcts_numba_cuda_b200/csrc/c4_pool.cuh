// Connect-4 search of many trees: one block per SM grows several trees side by side, and its threads play the games of all of them.
//
// A block per tree (c4_search.cuh) leaves its lanes idle from the moment a step has no game left to hand out until its longest
// game is over and the walker has made the next step.  Here the games of all trees of an SM go through one queue
// in shared memory: a lane whose game is over takes the next one, whichever tree it belongs to.
//
// Measured with the same plies in both: 256 roots of 4 x 256 acp, 400 steps, 22.7 ms with a block per tree, 19.1 with the pool; of 8 x 128
// ocp 8.65 and 6.2; a step's lanes 27 of 32 in play instead of 21.  What bounds it: issue slots (87 % busy) and the logic pipe
// (83 %) where games are many; where they are few (ocp: 22 to 23 lanes) the chain of a step, walk and longest game.
//
// The first `walkers` warps select, expand and back up, each for the trees w, w + walkers, ... of the block; the others play.
// Every game slot that a step needs played out becomes an entry of the queue, P games with one ticket each: ticket t is
// game t % P of entry t / P, so that a lane takes a game with one addition, as in the other kernel, and entries are played in the
// order in which they were made.  A lane keeps a ticket whose entry does not exist yet and looks for it again after its warp's next block
// of plies.  Which lane plays a game does not matter: it draws from the stream of the reference's thread (tree, action, t).
#pragma once
#include <stddef.h>

#include "c4_search.cuh"

namespace mctsnc {
namespace c4 {

constexpr int POOL_MAX_TREES = 31;            // of a block
constexpr int POOL_RING = 256;                // cells of the queue
static_assert(POOL_MAX_TREES * A <= POOL_RING, "entries that exist at once");
// A cell: the number modulo 2^14 of the entry that has it over the shared-memory address of that entry's slot, or, while it is free, the
// number of the entry that has it next over an address that no slot has.  So the cells change hands in the order of the entries,
// whichever walker is held up: the oldest entry that exists can always be written, and its tickets are the first to be taken.  The
// numbers of the entries that wait for a cell or for games lie within POOL_RING and the trees' slots, those of the
// tickets that idle lanes hold within 1024 more.
constexpr int POOL_ADDRESS_BITS = 18;
constexpr unsigned POOL_FREE = (1u << POOL_ADDRESS_BITS) - 1u;
constexpr unsigned POOL_MEMORY = 227 * 1024;        // of an SM; an address below it is a slot
__device__ __forceinline__ unsigned pool_cell(unsigned entry, unsigned address) { return (entry << POOL_ADDRESS_BITS) | address; }
// Looks of an idle warp for work before it takes its wait for endless; the pauses between them are nominally 0.08 s (walkers) and 0.4 s
// (players).  A walker waits for games that are played or handed out, some hundred microseconds at most, and gives the launch up.  A player
// may wait as long as the walkers have nothing to play: steps that select a terminal node play no game, and a tree with a won root
// has stretches of millions of them.  It gives up when no tree of the block has gone on since its last such wait.
constexpr int POOL_IDLE_LIMIT = 1 << 22;

enum PoolPhase { POOL_EMPTY, POOL_READY, POOL_PENDING, POOL_PLAYING };

struct PoolTree : Walk {
    ulonglong2 pick_stream;   // OCP: the stream of the child picks
    int tree;                 // -1: none
    int phase;
    int remaining;            // steps of the launch when the slice began, and of the slice: all, and made so far
    int n_steps, step;
    int backup_due;           // the step made last has not been backed up yet
    unsigned first_entry;     // of the step's slots
    long long t_start;
};

// A position that is played out P times and what has become of its games
struct __align__(16) PoolSlot {
    GameSlot start;           // (`rng_base` is the shared-memory address of the first stream, `stones` 256 more where +1 is to move)
    unsigned top_lo, top_hi;
    unsigned games;           // games that are over << 16 | their plies
    unsigned won;             // games won by -1 | games won by +1 << 16
};

struct Pool {
    MoveEntry move_lut[128 * 8];
    unsigned ring[POOL_RING];
    unsigned next_ticket, next_entry;
    int walkers_left;
    int given_up;
    unsigned seen[32];   // by a warp that plays, see pool_moves
};
static_assert(sizeof(Pool) % 16 == 0, "the trees follow");

__host__ __device__ __forceinline__ size_t pool_bytes(int trees, int streams) {
    return sizeof(Pool) + (size_t)trees * (sizeof(PoolTree) + A * sizeof(PoolSlot) + sizeof(ulonglong2) * (size_t)streams);
}

__device__ __forceinline__ unsigned shared_address(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(shared_address(p)) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(unsigned *p, unsigned v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(shared_address(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void add_release(unsigned *p, unsigned v) {
    asm volatile("red.release.cta.shared.add.u32 [%0], %1;" ::"r"(shared_address(p)), "r"(v) : "memory");
}

// Whether a tree of the block has made a step since this warp asked last, and the launch has not been given up: a slice's start and the
// steps made of it, which only grow, summed over the trees.  Neither in the players' loop nor with a vote, which make that loop slower
// (256 roots of 4 x 256 acp 2 %, 200 of 4 x 64 5 %); with a count kept by the walkers an ocp batch is 1 to 6 % slower.
__device__ __noinline__ bool pool_moves(Pool &pool, const PoolTree *trees, int n) {
    long long now = 0;
    for (int k = 0; k < n; k++) now += *(volatile const long long *)&trees[k].t_start + *(volatile const int *)&trees[k].step;
    volatile unsigned &seen = pool.seen[threadIdx.x >> 5];
    const bool moves = (unsigned)now != seen;
    __syncwarp();
    seen = (unsigned)now;
    return moves && !*(volatile int *)&pool.given_up;
}

template <bool OCP>
__device__ __forceinline__ void pool_walk(const SearchParams &p, Pool &pool, PoolTree *trees, PoolSlot *slots, ulonglong2 *s_rng, int warp, int lane) {
    const int P = p.n_playouts;
    const int n_streams = OCP ? P : A * P;
    const double c_ucb = (double)p.ucb_c;
    const bool queued = p.queue != nullptr;

    // the next tree of place k: from the queue, or tree blockIdx.x + k * gridDim.x, once
    auto take = [&](int k, int next) {
        PoolTree &t = trees[k];
        __syncwarp();   // the tree's state is read by all lanes, lane 0 has it from the queue
        if (next < 0) {
            if (lane == 0) {
                t.tree = -1;
                t.phase = POOL_EMPTY;
            }
            __syncwarp();
            return;
        }
        const int rem = queued ? p.remaining[next] : p.steps;
        if (lane == 0) {
            t.tree = next;
            t.remaining = rem;
            t.n_steps = queued && rem > p.chunk ? p.chunk : rem;
            t.step = 0;
            t.backup_due = 0;
            t.phase = POOL_READY;
            t.t_start = queued ? global_timer_ns() : 0;
            load_tree(p, t, next, p.first != 0 && rem == p.steps, nullptr, 0);
            if (OCP) t.pick_stream = p.rng_expand[next];
        }
        const ulonglong2 *g_rng = p.rng_playout + (long long)next * n_streams;
        for (int i = lane; i < n_streams; i += 32) s_rng[k * n_streams + i] = g_rng[i];
        __syncwarp();
    };
    auto leave = [&](int k) {
        PoolTree &t = trees[k];
        const int g = t.tree;
        ulonglong2 *g_rng = p.rng_playout + (long long)g * n_streams;
        for (int i = lane; i < n_streams; i += 32) g_rng[i] = s_rng[k * n_streams + i];
        if (lane == 0) {
            if (OCP) p.rng_expand[g] = t.pick_stream;
            store_tree(p, t, g, p.first != 0 && t.remaining == p.steps);
        }
        __syncwarp();
        int next = -1;
        if (queued && lane == 0) {
            const int level = finish_slice(p, g, t.remaining, t.n_steps, t.t_start);
            // see search_kernel for the order of the two
            if (level < 0 || 4 * p.ring_cap >= 5 * p.places) next = queue_pop(p.queue, p.ring, p.ring_cap);
            if (level >= 0) {
                if (!queue_push(p.queue, p.ring, p.ring_cap, level, g)) atomicOr(&p.state[g].status, STATUS_INTERNAL);
                if (next < 0) next = queue_pop(p.queue, p.ring, p.ring_cap);
            }
        }
        return __shfl_sync(0xFFFFFFFFu, next, 0);
    };
    // the step's slots become entries, unless a cell still belongs to the entry POOL_RING before (false: try again)
    auto publish = [&](PoolTree &t, int k) {
        const unsigned e = t.first_entry + lane;
        const bool mine = lane < t.n_slots;
        unsigned *cell = &pool.ring[e & (POOL_RING - 1)];
        const bool free = !mine || load_acquire(cell) == pool_cell(e, POOL_FREE);
        if (!__all_sync(0xFFFFFFFFu, free)) return false;
        if (mine) store_release(cell, pool_cell(e, shared_address(slots + k * A + lane)));
        return true;
    };

    for (int k = warp; k < p.pool_trees; k += p.pool_walkers) {
        int g = (int)blockIdx.x + k * (int)gridDim.x;
        if (queued) {
            g = lane == 0 ? queue_pop(p.queue, p.ring, p.ring_cap) : 0;
            g = __shfl_sync(0xFFFFFFFFu, g, 0);
        } else if (g >= p.n_trees_launched) {
            g = -1;
        }
        take(k, g);
    }
    int idle = 0;
    for (;;) {
        bool any = false, moved = false;
        for (int k = warp; k < p.pool_trees; k += p.pool_walkers) {
            PoolTree &t = trees[k];
            const int phase = t.phase;
            if (phase == POOL_EMPTY) continue;
            any = true;
            if (phase == POOL_PENDING) {
                if (publish(t, k)) {
                    __syncwarp();
                    if (lane == 0) t.phase = POOL_PLAYING;
                    __syncwarp();
                    moved = true;
                }
                continue;
            }
            if (phase == POOL_PLAYING) {
                const bool done = lane >= t.n_slots || (load_acquire(&slots[k * A + lane].games) >> 16) == (unsigned)P;
                if (!__all_sync(0xFFFFFFFFu, done)) continue;
            }
            moved = true;
            int g = t.tree;
            if (t.backup_due) {
                const int n_slots = t.n_slots;
                if (phase == POOL_PLAYING) {
                    int plies = lane < n_slots ? (int)(slots[k * A + lane].games & 0xFFFFu) : 0;
                    plies = __reduce_add_sync(0xFFFFFFFFu, plies);
                    const unsigned e = t.first_entry + lane;
                    if (lane < n_slots) store_release(&pool.ring[e & (POOL_RING - 1)], pool_cell(e + POOL_RING, POOL_FREE));
                    if (lane == 0) atomicAdd(&t.plies, (unsigned long long)plies);   // (a replayed game adds its own)
                }
                backup<OCP>(t, p.rec + (long long)g * p.cap, nullptr, 0, c_ucb, P, lane, [&](int j) {
                    const unsigned w = slots[k * A + j].won;
                    return make_int2((int)(w & 0xFFFFu), (int)(w >> 16));
                });
            }
            if (t.step == t.n_steps) {
                g = leave(k);
                take(k, g);
                continue;
            }
            ulonglong2 pick_stream = make_ulonglong2(0ULL, 0ULL);
            if (OCP && lane == 0) pick_stream = t.pick_stream;
            const Selected leaf = select_expand<OCP>(p, t, p.rec + (long long)g * p.cap, p.board + (long long)g * p.cap,
                                                     p.parent + (long long)g * p.cap, nullptr, 0, pick_stream, lane, [&](int j, GameSlot gs, int mover) {
                PoolSlot &slot = slots[k * A + j];
                const unsigned long long occupied = gs.cur | gs.other;
                slot.top_lo = top_low((unsigned)occupied);
                slot.top_hi = top_high((unsigned)(occupied >> 32));
                gs.rng_base = (int)shared_address(s_rng + k * n_streams + gs.rng_base);
                if (mover > 0) gs.stones += 256;
                slot.start = gs;
                slot.games = 0u;
                slot.won = 0u;
            });
            __syncwarp();
            if (OCP && lane == 0) t.pick_stream = pick_stream;
            const bool plays = leaf.n_slots > 0;
            bool published = true;
            if (plays) {
                if (lane == 0) t.first_entry = atomicAdd(&pool.next_entry, (unsigned)leaf.n_slots);
                __syncwarp();
                published = publish(t, k);
            }
            const int n_tot = leaf.mode == MODE_ALL_CHILDREN && !OCP ? P * __popc(t.exp_mask) : P;
            prepare_backup<OCP>(t, p.rec + (long long)g * p.cap, nullptr, 0, c_ucb, lane, leaf.depth + 1, n_tot,
                                leaf.mode == MODE_ALL_CHILDREN ? P : 0);
            if (lane == 0) {
                t.step++;
                t.backup_due = 1;
                t.phase = !plays ? POOL_READY : (published ? POOL_PLAYING : POOL_PENDING);
            }
            __syncwarp();
        }
        if (!any) break;
        if (moved) {
            idle = 0;
        } else {
            __nanosleep(20);
            if (++idle > POOL_IDLE_LIMIT || *(volatile int *)&pool.given_up) {
                // (cannot happen) the trees keep the steps they have; the launch reports it
                for (int k = warp; k < p.pool_trees; k += p.pool_walkers)
                    if (lane == 0 && trees[k].phase != POOL_EMPTY) atomicOr(&p.state[trees[k].tree].status, STATUS_INTERNAL);
                if (lane == 0) *(volatile int *)&pool.given_up = 1;
                break;
            }
        }
    }
    __syncwarp();
    if (lane == 0) atomicSub(&pool.walkers_left, 1);
}

__device__ __forceinline__ void pool_play(const SearchParams &p, Pool &pool, PoolTree *trees, const PoolSlot *first_slot) {
    const int log2_p = p.log2_playouts;
    const unsigned lut_base = move_lut_base(pool.move_lut), ring = shared_address(pool.ring), last = (unsigned)p.n_playouts - 1u;
    Game<false> game;
    bool playing = false;
    unsigned slot = 0u, stream = 0u;   // of the game, shared-memory addresses
    unsigned ticket = atomicAdd(&pool.next_ticket, 1u);
    int idle = 0;
    auto close_game = [&]() {
        // plies of the game, and 256 less where +1 was the first to move
        const int m = game.finish();
        int n = m & 255;
        unsigned winner = ((m ^ (m >> 8)) & 1) ? 1u : 0x10000u;   // odd: the first mover
        if (game.fours == 0u) winner = 0u;
        if (game.marked()) {
            // u == 1.0f somewhere in this game: replay it through the byte-level emulation of the reference
            const bool first_is_pos = m < 0;
            const GameSlot gs = reinterpret_cast<const PoolSlot *>(__cvta_shared_to_generic(slot))->start;
            const ulonglong2 rs = *reinterpret_cast<const ulonglong2 *>(__cvta_shared_to_generic(stream));
            const EmuResult er = playout_emulated(first_is_pos ? gs.other : gs.cur, first_is_pos ? gs.cur : gs.other, first_is_pos ? 1 : -1,
                                                  rs.x, rs.y);
            game.s0 = er.s0;
            game.s1 = er.s1;
            winner = er.outcome == 1 ? 0x10000u : (er.outcome == -1 ? 1u : 0u);
            n = 0;
            PoolTree &t = trees[(slot - shared_address(first_slot)) / (unsigned)(A * sizeof(PoolSlot))];
            atomicAdd(&t.plies, (unsigned long long)er.plies);
            atomicAdd(&t.ub, (unsigned long long)er.ub);
            atomicOr(&t.status, (er.ub ? STATUS_UB_DRAW : 0u) | (er.err ? STATUS_INTERNAL : 0u));
        }
        asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(stream), "l"(game.s0), "l"(game.s1) : "memory");
        asm volatile("red.shared.add.u32 [%0 + 44], %1;" ::"r"(slot), "r"(winner) : "memory");
        asm volatile("red.release.cta.shared.add.u32 [%0 + 40], %1;" ::"r"(slot), "r"(0x10000 + n) : "memory");
    };
    static_assert(offsetof(PoolSlot, games) == 40 && offsetof(PoolSlot, won) == 44, "");
    auto start_game = [&]() {
        GameSlot gs;
        unsigned top_lo, top_hi;
        int4 a, b;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w) : "r"(slot));
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4 + 16];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(slot));
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2 + 32];" : "=r"(top_lo), "=r"(top_hi) : "r"(slot));
        gs.cur = ((unsigned long long)(unsigned)a.y << 32) | (unsigned)a.x;
        gs.other = ((unsigned long long)(unsigned)a.w << 32) | (unsigned)a.z;
        gs.row = __int_as_float(b.x);
        gs.count = __int_as_float(b.y);
        gs.stones = b.w;
        stream = (unsigned)b.z + (ticket & last) * (unsigned)sizeof(ulonglong2);
        ulonglong2 rs;
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(rs.x), "=l"(rs.y) : "r"(stream) : "memory");
        game.start(gs, top_lo, top_hi, rs);
    };
    static_assert(offsetof(GameSlot, cur) == 0 && offsetof(GameSlot, other) == 8 && offsetof(GameSlot, row) == 16 && offsetof(GameSlot, count) == 20 &&
                      offsetof(GameSlot, rng_base) == 24 && offsetof(GameSlot, stones) == 28 && offsetof(PoolSlot, top_lo) == 32, "");
    for (;;) {
        if (playing) {
            game.play_block(lut_base, p);
            if (game.over()) {
                close_game();
                ticket = atomicAdd(&pool.next_ticket, 1u);
                playing = false;
            }
        }
        if (!playing) {
            const unsigned e = ticket >> log2_p;
            unsigned cell;
            asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(cell) : "r"(ring + (e & (POOL_RING - 1)) * 4u) : "memory");
            slot = cell - (e << POOL_ADDRESS_BITS);
            if (slot < POOL_MEMORY) {
                start_game();
                playing = true;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, playing)) {
            if (*(volatile int *)&pool.walkers_left == 0) break;
            __nanosleep(100);
            if (++idle > POOL_IDLE_LIMIT || *(volatile int *)&pool.given_up) {
                idle = 0;
                if (!pool_moves(pool, trees, p.pool_trees)) {
                    *(volatile int *)&pool.given_up = 1;
                    break;
                }
            }
        } else {
            idle = 0;
        }
    }
}

template <bool OCP>
__global__ void __launch_bounds__(1024, 1) pool_kernel(const SearchParams p) {
    extern __shared__ __align__(16) unsigned char pool_memory[];
    Pool &pool = *reinterpret_cast<Pool *>(pool_memory);
    PoolTree *trees = reinterpret_cast<PoolTree *>(pool_memory + sizeof(Pool));
    PoolSlot *slots = reinterpret_cast<PoolSlot *>(trees + p.pool_trees);
    ulonglong2 *s_rng = reinterpret_cast<ulonglong2 *>(slots + p.pool_trees * A);
    build_move_lut(pool.move_lut);
    for (int i = threadIdx.x; i < POOL_RING; i += blockDim.x) pool.ring[i] = pool_cell(i, POOL_FREE);
    if (threadIdx.x == 0) {
        pool.next_ticket = 0u;
        pool.next_entry = 0u;
        pool.walkers_left = p.pool_walkers;
        pool.given_up = 0;
        for (int i = 0; i < 32; i++) pool.seen[i] = 0u;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    if (warp < p.pool_walkers) pool_walk<OCP>(p, pool, trees, slots, s_rng, warp, threadIdx.x & 31);
    else pool_play(p, pool, trees, slots);
}

}  // namespace c4
}  // namespace mctsnc
