// Host side of libmctsnc_b200.so: the C ABI declared in include/mctsnc_b200.h, the handle that owns the device
// memory of a searcher, the random-stream set-up, the two reduction kernels and the export of trees in the
// reference's array formats.
#include "../../include/mctsnc_b200.h"

#include <cuda_runtime.h>

#include <chrono>
#include <cstdio>
#include <mutex>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "c4_pool.cuh"
#include "c4_search.cuh"
#include "common.cuh"
#include "gomoku_search.cuh"
#include "rng.cuh"

using namespace mctsnc;

namespace {

constexpr int GOMOKU_STREAMS = 8;     // tree groups of a Gomoku search launch that run out of step with each other
constexpr int MAX_TREE_DEPTH = 2048;  // src/mctsnc.py:197
#ifndef MCTSNC_C4_CLUSTER_MIN_GAMES
#define MCTSNC_C4_CLUSTER_MIN_GAMES 256    // Connect 4: clusters only for steps with more games than this
#endif
#ifndef MCTSNC_C4_CACHE_NODES
#define MCTSNC_C4_CACHE_NODES 6144      // Connect-4 cluster kernel, one block per SM: node records kept in shared memory
#endif
#ifndef MCTSNC_C4_CLUSTER_SM_SHARE
#define MCTSNC_C4_CLUSTER_SM_SHARE 4   // Connect 4: clusters of blocks per tree while they make at most this many blocks per SM
#endif
#define CUDA_TRY(expr)                        \
    do {                                      \
        cudaError_t _e = (expr);              \
        if (_e != cudaSuccess) return (int)_e; \
    } while (0)

int pow2ceil(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// device-side result block of one search, filled by the two reduction kernels
struct DevResult {
    int best_action;
    int best_win_flag;
    long long best_n;
    long long best_n_wins;
    long long playouts;
    long long plies;
    long long ub_draws;
    unsigned status;
    int n_root_actions;
    int max_depth;
    int max_size;
    long long total_nodes;
    long long depth_sum;
    float stage_ms[4];   // mean over the search's trees of TreeState::stage_ms
};

// the forms a cluster per tree comes in, in the order they are tried (WIDE_AHEAD and AHEAD: draws made ahead, a block on an SM)
enum ClusterForm { WIDE_AHEAD, WIDE, AHEAD, PLAIN, PACKED, CLUSTER_FORMS };
bool is_wide(int form) { return form == WIDE_AHEAD || form == WIDE; }
bool is_ahead(int form) { return form == WIDE_AHEAD || form == AHEAD; }

}  // namespace

struct mctsnc_handle {
    mctsnc_config cfg;
    int A = 0;
    int tpb_e1 = 0;
    int tpb_roa = 0;
    int sm_count = 0;
    bool cluster_ok = false;      // thread-block clusters can be launched (and MCTSNC_B200_NO_CLUSTER is not set)
    int cluster_fit[CLUSTER_FORMS][2] = {};   // clusters that fit on the device at once, [ClusterForm][small record cache] (0: not asked yet, -1: unknown)
    int threads = 0;
    int blocks_per_sm = 0;
    const char *kernel = "";     // of the last search launch
    long long bytes = 0;
    long long n_trees_total = 0;  // max_batch * n_trees
    long long rng_per_search = 0; // playout streams per search of this handle
    // device memory
    int4 *rec = nullptr;
    ulonglong2 *board = nullptr;
    int *parent = nullptr;
    TreeState *state = nullptr;
    int *paths = nullptr;
    short *actions_expanded = nullptr;
    int *child_out = nullptr;
    ulonglong2 *rng_playout = nullptr;
    ulonglong2 *rng_expand = nullptr;
    ulonglong2 *rng_playout_base = nullptr;
    ulonglong2 *rng_expand_base = nullptr;
    JumpColumn *jump_cols = nullptr;      // [JUMP_LEVELS][128] matrices of the 2^64-step jump, for seeding streams on the device
    ulonglong2 *root_board = nullptr;
    signed char *root_turn = nullptr;     // behind the boards of the staged roots
    WorkQueues *queue = nullptr;          // Connect 4: work queue of batched launches
    QueueCell *ring = nullptr;            // [QUEUE_LEVELS][n_trees_total]
    int *remaining = nullptr;             // [n_trees_total]
    long long *trace = nullptr;           // optional slice record of queued launches: [trace_cap][4]
    int *trace_count = nullptr;
    int trace_cap = 0;
    // Gomoku only
    unsigned *gboard = nullptr;           // [trees][cap][16]
    gomoku::StepInfo *gstep = nullptr;    // [trees]
    unsigned *gsheet = nullptr;           // [trees][gomoku::SHEET_WORDS]
    int4 *path_rec = nullptr;             // [trees][PATH_CAP]
    PathTerm *path_term = nullptr;        // [trees][PATH_CAP]
    signed char *child_outcome = nullptr;
    unsigned char *child_action = nullptr;
    gomoku::StepGames *gwork = nullptr;   // [trees]
    unsigned *root_gboard = nullptr;      // [max_batch][16]
    unsigned *h_root_gboard = nullptr;
    // [max_batch] results, [max_batch][3A] sums, [max_batch][2A] flags (win flags, expanded-at-root) in one piece of memory
    DevResult *dres = nullptr;
    long long *sums = nullptr;
    unsigned char *flags = nullptr;
    // pinned host staging
    ulonglong2 *h_root_board = nullptr;
    DevResult *h_dres = nullptr;          // the same three in one pinned piece
    long long *h_sums = nullptr;
    unsigned char *h_flags = nullptr;
    size_t result_bytes = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t ev_staged = nullptr;  // recorded behind the host-to-device copies of the staged roots
    bool staging_in_flight = false;
    float last_ms = 0.f;
    long long last_steps = 0;
    // Gomoku: streams of the tree groups of a search launch, with the events that fork them from and join them to the
    // caller's stream
    cudaStream_t g_stream[GOMOKU_STREAMS] = {};
    cudaEvent_t g_fork = nullptr, g_join[GOMOKU_STREAMS] = {};
    float ms_per_cycle = 0.f;  // 1 / nominal SM clock in kHz
    cudaEvent_t ev_r0 = nullptr, ev_r1 = nullptr;  // behind the two reduction kernels of mctsnc_run
    float reduce_ms[2] = {0.f, 0.f};
    int staged_roots = 0;  // roots resident on the device from the last staging
    size_t dyn_smem = 0;   // dynamic shared memory of the search kernel: the tree's random streams
};

namespace {

// ---------------------------------------------------------------------------------------------------------------
// kernels outside the search loop

// fills the work queue of a batched launch with every tree once (in the highest ring: nothing is known yet about the
// work a tree has), each with `steps` steps to do
__global__ void init_queue_kernel(WorkQueues *q, QueueCell *rings, int *remaining, int trees, int steps) {
    const int gsz = gridDim.x * blockDim.x;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = gid; i < trees * QUEUE_LEVELS; i += gsz) {
        const int level = i / trees, c = i - level * trees;
        const bool top = level == QUEUE_LEVELS - 1;
        rings[i].tree = top ? c : -1;
        rings[i].seq = top ? c + 1 : c;
    }
    for (int i = gid; i < trees; i += gsz) remaining[i] = steps;
    if (gid < QUEUE_LEVELS) {  // blocks have 256 threads
        q->level[gid].head = 0;
        q->level[gid].tail = q->level[gid].ready = gid == QUEUE_LEVELS - 1 ? trees : 0;
    }
    if (gid == 0) {
        q->nonempty = 1ULL << (QUEUE_LEVELS - 1);
        q->longest_us = 0;
    }
}

// after a queued launch: a tree that still has steps to do was lost by the queue; report it instead of returning a
// short search
__global__ void check_queue_kernel(const int *remaining, TreeState *state, int trees) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < trees; i += gridDim.x * blockDim.x)
        if (remaining[i] != 0) atomicOr(&state[i].status, STATUS_INTERNAL);
}

// copies the freshly seeded streams of one search into the slots of `batch` searches
__global__ void replicate_streams_kernel(ulonglong2 *dst, const ulonglong2 *base, long long per_search, int batch) {
    const long long n = per_search * batch;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = base[i % per_search];
}

// The part of the two reductions over trees that both games share.  Every load of a search's trees is independent of the others
// (roots first, then their children; a tree's counters by a lane of the last warp): read one tree after the other they were a
// chain of 16 to 32 memory latencies (86 us for 4 trees of 14000 nodes with the node scan for the depths, which the search
// now keeps itself; 390 us for Gomoku).
constexpr int REDUCE_THREADS = 256;
__device__ __forceinline__ void load_roots(int4 *s_root, const int4 *r0, long long cap, int n_trees) {
    for (int t = threadIdx.x; t < n_trees; t += REDUCE_THREADS) s_root[t] = r0[(long long)t * cap];
    __syncthreads();
}
__device__ __forceinline__ long long warp_sum(long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}
__device__ __forceinline__ void gather_statistics(const TreeState *state, const int4 *s_root, int n_trees, int n_root_actions, DevResult *out) {
    if (threadIdx.x < REDUCE_THREADS - 32) return;
    const int lane = threadIdx.x & 31;
    long long playouts = 0, plies = 0, ub = 0, nodes = 0, depths = 0;
    int max_size = 0, max_depth = 0;
    unsigned status = 0;
    float stage[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t = lane; t < n_trees; t += 32) {
        const TreeState ts = state[t];
        playouts += s_root[t].x;
        plies += (long long)ts.plies;
        ub += (long long)ts.ub_draws;
        nodes += ts.size;
        depths += ts.depth_sum;
        status |= ts.status;
        max_size = max(max_size, ts.size);
        max_depth = max(max_depth, ts.max_depth);
        for (int k = 0; k < 4; k++) stage[k] += ts.stage_ms[k];
    }
    DevResult d;
    d.playouts = warp_sum(playouts);
    d.plies = warp_sum(plies);
    d.ub_draws = warp_sum(ub);
    d.total_nodes = warp_sum(nodes);
    d.depth_sum = warp_sum(depths);
    d.status = __reduce_or_sync(0xFFFFFFFFu, status);
    d.max_size = __reduce_max_sync(0xFFFFFFFFu, max_size);
    d.max_depth = __reduce_max_sync(0xFFFFFFFFu, max_depth);
    for (int k = 0; k < 4; k++) {
        for (int o = 16; o > 0; o >>= 1) stage[k] += __shfl_down_sync(0xFFFFFFFFu, stage[k], o);
        d.stage_ms[k] = stage[k] / (float)n_trees;
    }
    d.best_action = -1;
    d.best_win_flag = 0;
    d.best_n = 0;
    d.best_n_wins = 0;
    d.n_root_actions = n_root_actions;
    if (lane == 0) *out = d;
}

// _reduce_over_trees_* (src/mctsnc.py:2223-2296): per root action the sums over the trees of a search of the root
// visit count, the child's visit count and the child's win count; win flag from tree 0.  One block per search.
// Also gathers the statistics behind performance_info (:448-494).
__global__ void reduce_over_trees_kernel(const int4 *rec, const TreeState *state, long long cap, int n_trees, int A,
                                         long long *sums, unsigned char *flags, DevResult *dres) {
    const int b = blockIdx.x;
    const int tid = threadIdx.x;
    const int4 *r0 = rec + (long long)b * n_trees * cap;
    __shared__ int4 s_root[512];
    load_roots(s_root, r0, cap, n_trees);
    const int root_meta0 = s_root[0].w;
    const int root_turn = meta_turn(root_meta0);
    const unsigned mask0 = root_meta0 & 0x7F;
    for (int a = tid; a < A; a += blockDim.x) {
        long long n_root = 0, s_n = 0, s_w = 0;
        unsigned char win = 0;
        const bool expanded = (mask0 >> a) & 1u;
        if (expanded) {
#pragma unroll 4
            for (int t = 0; t < n_trees; t++) {
                const int4 *rt = r0 + (long long)t * cap;
                const int4 root = s_root[t];
                n_root += root.x;
                const unsigned mk = root.w & 0x7F;
                if ((mk >> a) & 1u) {
                    const int4 c = rt[root.z + __popc(mk & ((1u << a) - 1u))];
                    s_n += c.x;
                    s_w += c.y;
                    if (t == 0) win = (c.w & META_TERMINAL) && meta_outcome(c.w) == root_turn;
                }
            }
        }
        sums[(long long)b * 3 * A + a] = n_root;
        sums[(long long)b * 3 * A + A + a] = s_n;
        sums[(long long)b * 3 * A + 2 * A + a] = s_w;
        flags[(long long)b * 2 * A + a] = win;
        flags[(long long)b * 2 * A + A + a] = expanded;
    }
    gather_statistics(state + b * n_trees, s_root, n_trees, __popc(mask0), dres + b);
}

// _reduce_over_actions_* (src/mctsnc.py:2299-2375): lexicographic max/argmax over (win_flag, n, n_wins) with the
// reference's stride-halving reduction, which keeps the left operand on ties.  The thrifty variants reduce over
// ordinals among the root's expanded actions, the prodigal ones over action indices.  One block of `width` threads
// per search (width = tpb_roa).
__global__ void reduce_over_actions_kernel(const long long *sums, const unsigned char *flags, int A, int width, int thrifty,
                                           DevResult *dres) {
    __shared__ short s_a[512];
    __shared__ unsigned char s_f[512];
    __shared__ long long s_n[512];
    __shared__ long long s_w[512];
    __shared__ short s_ord2act[512];
    __shared__ int s_expanded[16];   // expanded actions by warp
    const int b = blockIdx.x;
    const int t = threadIdx.x;
    const long long *sm = sums + (long long)b * 3 * A;
    const unsigned char *fl = flags + (long long)b * 2 * A;
    // the expanded actions in ascending order: ballot and prefix over the warps (width >= A; below 32 it is a part of a warp)
    const unsigned whole = width < 32 ? (1u << width) - 1u : 0xFFFFFFFFu;
    const bool expanded = t < A && fl[A + t];
    const unsigned set = __ballot_sync(whole, expanded);
    if ((t & 31) == 0) s_expanded[t >> 5] = __popc(set);
    __syncthreads();
    int n_expanded = 0, before = __popc(set & ((1u << (t & 31)) - 1u));
    for (int w = 0; w < (width + 31) / 32; w++) {
        if (w < (t >> 5)) before += s_expanded[w];
        n_expanded += s_expanded[w];
    }
    if (expanded) s_ord2act[before] = (short)t;
    __syncthreads();
    const int limit = thrifty ? n_expanded : A;
    const int src = thrifty ? (t < limit ? s_ord2act[t] : 0) : t;
    s_a[t] = (short)t;
    if (t < limit) {
        s_f[t] = fl[src];
        s_n[t] = sm[A + src];
        s_w[t] = sm[2 * A + src];
    } else {
        s_f[t] = 0;
        s_n[t] = 0;
        s_w[t] = 0;
    }
    __syncthreads();
    for (int stride = width >> 1; stride > 0; stride >>= 1) {
        if (t < stride) {
            const int o = t + stride;
            if ((s_f[t] < s_f[o]) || (s_f[t] == s_f[o] && s_n[t] < s_n[o]) ||
                (s_f[t] == s_f[o] && s_n[t] == s_n[o] && s_w[t] < s_w[o])) {
                s_a[t] = s_a[o];
                s_f[t] = s_f[o];
                s_n[t] = s_n[o];
                s_w[t] = s_w[o];
            }
        }
        __syncthreads();
    }
    if (t == 0) {
        int best = s_a[0];
        if (thrifty) best = best < n_expanded ? s_ord2act[best] : 0;
        dres[b].best_action = best;
        dres[b].best_win_flag = s_f[0];
        dres[b].best_n = s_n[0];
        dres[b].best_n_wins = s_w[0];
    }
}

// _reduce_over_trees_* for Gomoku nodes (first child + number of children; the child of action a is found through the
// empty cells of the root position)
__global__ void gomoku_reduce_over_trees_kernel(const int4 *rec, const unsigned *board, const TreeState *state, long long cap,
                                                int n_trees, long long *sums, unsigned char *flags, DevResult *dres) {
    constexpr int A = gomoku::A;
    const int b = blockIdx.x;
    const int tid = threadIdx.x;
    const int4 *r0 = rec + (long long)b * n_trees * cap;
    const unsigned *b0 = board + (long long)b * n_trees * cap * 16;   // root position (the same in every tree)
    __shared__ unsigned s_empty[8];
    __shared__ int s_prefix[9];
    __shared__ int4 s_root[512];
    if (tid < 8) s_empty[tid] = ~(b0[tid] | b0[8 + tid]) & (tid == 7 ? 0x1u : 0xFFFFFFFFu);
    load_roots(s_root, r0, cap, n_trees);
    if (tid == 0) {
        int acc = 0;
        for (int w = 0; w < 8; w++) {
            s_prefix[w] = acc;
            acc += __popc(s_empty[w]);
        }
        s_prefix[8] = acc;
    }
    __syncthreads();
    const int root_turn = gomoku::g_turn(s_root[0].w);
    const int n_children0 = s_root[0].w & gomoku::G_NCHILD_MASK;
    for (int a = tid; a < A; a += blockDim.x) {
        long long n_root = 0, s_n = 0, s_w = 0;
        unsigned char win = 0;
        const int w = a >> 5, bit = a & 31;
        const int rank = s_prefix[w] + __popc(s_empty[w] & ((1u << bit) - 1u));
        const bool expanded = ((s_empty[w] >> bit) & 1u) && rank < n_children0;
        if (expanded) {
#pragma unroll 4
            for (int t = 0; t < n_trees; t++) {
                const int4 *rt = r0 + (long long)t * cap;
                const int4 root = s_root[t];
                n_root += root.x;
                if (rank < (root.w & gomoku::G_NCHILD_MASK)) {
                    const int4 c = rt[root.z + rank];
                    s_n += c.x;
                    s_w += c.y;
                    if (t == 0) win = (c.w & gomoku::G_TERMINAL) && gomoku::g_outcome(c.w) == root_turn;
                }
            }
        }
        sums[(long long)b * 3 * A + a] = n_root;
        sums[(long long)b * 3 * A + A + a] = s_n;
        sums[(long long)b * 3 * A + 2 * A + a] = s_w;
        flags[(long long)b * 2 * A + a] = win;
        flags[(long long)b * 2 * A + A + a] = expanded;
    }
    gather_statistics(state + b * n_trees, s_root, n_trees, n_children0, dres + b);
}

// ---------------------------------------------------------------------------------------------------------------
// host helpers

// create_xoroshiro128p_states(n, seed) restricted to the streams [first, first + count) with stride `stride`
// between wanted streams (stream i is stream i-1 jumped 2^64 steps ahead)
void make_streams(uint64_t seed, long long first, long long count, long long stride, ulonglong2 *out) {
    RngState s;
    rng_seed(s, seed);
    long long idx = 0;
    for (long long k = 0; k < count; k++) {
        const long long want = first + k * stride;
        while (idx < want) {
            rng_jump(s);
            idx++;
        }
        out[k].x = s.s0;
        out[k].y = s.s1;
    }
}

// the jump matrices, computed once per process
const JumpColumn *jump_matrix_table() {
    static JumpColumn table[JUMP_LEVELS * 128];
    static std::once_flag once;
    std::call_once(once, [] { jump_matrices(table); });
    return table;
}

bool is_ocp(const mctsnc_config &c) { return c.variant == MCTSNC_OCP_THRIFTY || c.variant == MCTSNC_OCP_PRODIGAL; }
bool is_thrifty(const mctsnc_config &c) { return c.variant == MCTSNC_OCP_THRIFTY || c.variant == MCTSNC_ACP_THRIFTY; }

// int8 board + column fills -> bitboards; rejects positions the bitboard mechanics cannot represent
int c4_encode_root(const int8_t *board, const int8_t *fills, ulonglong2 *out) {
    unsigned long long neg = 0, pos = 0;
    for (int j = 0; j < c4::COLS; j++) {
        int f = 0;
        bool gap = false;
        for (int h = 0; h < c4::ROWS; h++) {
            const int v = board[(c4::ROWS - 1 - h) * c4::COLS + j];
            if (v == 0) {
                gap = true;
                continue;
            }
            if (gap || (v != 1 && v != -1)) return MCTSNC_E_BAD_ROOT;  // a disc above an empty cell
            if (v > 0) pos |= 1ULL << (c4::column_shift(j) + h);
            else neg |= 1ULL << (c4::column_shift(j) + h);
            f++;
        }
        if (fills && fills[j] != f) return MCTSNC_E_BAD_ROOT;
    }
    if (c4::has_four(neg) || c4::has_four(pos)) return MCTSNC_E_BAD_ROOT;  // the game is over already
    out->x = neg;
    out->y = pos;
    return 0;
}

// int8 board -> two 225-bit stone sets (cell (i, j) = bit i*15+j)
int gomoku_encode_root(const int8_t *board, unsigned *out) {
    for (int k = 0; k < 16; k++) out[k] = 0;
    for (int c = 0; c < gomoku::A; c++) {
        const int v = board[c];
        if (v == -1) out[c >> 5] |= 1u << (c & 31);
        else if (v == 1) out[8 + (c >> 5)] |= 1u << (c & 31);
        else if (v != 0) return MCTSNC_E_BAD_ROOT;
    }
    return 0;
}

bool is_gomoku(const mctsnc_config &c) { return c.game == MCTSNC_GAME_GOMOKU; }

template <typename T>
int dev_alloc(mctsnc_handle *h, T **p, long long n) {
    if (n <= 0) n = 1;
    cudaError_t e = cudaMalloc((void **)p, (size_t)n * sizeof(T));
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? MCTSNC_E_NO_MEMORY : (int)e;
    }
    h->bytes += n * (long long)sizeof(T);
    return 0;
}

void release(mctsnc_handle *h) {
    cudaFree(h->rec);
    cudaFree(h->board);
    cudaFree(h->parent);
    cudaFree(h->state);
    cudaFree(h->paths);
    cudaFree(h->actions_expanded);
    cudaFree(h->child_out);
    cudaFree(h->rng_playout);
    cudaFree(h->rng_expand);
    cudaFree(h->rng_playout_base);
    cudaFree(h->rng_expand_base);
    cudaFree(h->jump_cols);
    cudaFree(h->root_board);
    cudaFree(h->queue);
    cudaFree(h->ring);
    cudaFree(h->remaining);
    cudaFree(h->trace);
    cudaFree(h->trace_count);
    cudaFree(h->gboard);
    cudaFree(h->gstep);
    cudaFree(h->gsheet);
    cudaFree(h->path_rec);
    cudaFree(h->path_term);
    cudaFree(h->gwork);
    cudaFree(h->child_outcome);
    cudaFree(h->child_action);
    cudaFree(h->root_gboard);
    cudaFreeHost(h->h_root_gboard);
    cudaFree(h->dres);
    cudaFreeHost(h->h_root_board);
    cudaFreeHost(h->h_dres);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    if (h->ev_staged) cudaEventDestroy(h->ev_staged);
    if (h->ev_r0) cudaEventDestroy(h->ev_r0);
    if (h->ev_r1) cudaEventDestroy(h->ev_r1);
    if (h->g_fork) cudaEventDestroy(h->g_fork);
    for (int g = 0; g < GOMOKU_STREAMS; g++) {
        if (h->g_join[g]) cudaEventDestroy(h->g_join[g]);
        if (h->g_stream[g]) cudaStreamDestroy(h->g_stream[g]);
    }
}

#ifndef MCTSNC_SLICE_STEPS
#define MCTSNC_SLICE_STEPS 32
#endif
constexpr int SLICE_STEPS = MCTSNC_SLICE_STEPS;  // steps a block runs of one tree before it takes the next tree from the queue

// A step whose games all have a thread of their own is as long as its longest game: the playouts then go straight through
// blocks of plies (2.7 us a step against 4.6 for 32 games; with five games a thread 49 ms against 36 for a search of 2000 steps
// that takes a block of 1024 threads, so with more games than threads a lane takes its next game at once).
// mctsnc_search_c4_static does not ask: it has the kernel for more games than threads whatever the sizes.
bool play_straight(const mctsnc_config &c, int threads) { return threads >= c.n_playouts * (is_ocp(c) ? 1 : c4::A); }

const void *search_kernel_ptr(const mctsnc_config &c, bool straight) {
    if (straight) return is_ocp(c) ? (const void *)c4::search_kernel<true, true> : (const void *)c4::search_kernel<false, true>;
    return is_ocp(c) ? (const void *)c4::search_kernel<true, false> : (const void *)c4::search_kernel<false, false>;
}

// Threads that play the games of one tree in a block of its own, from the games a step plays (n_playouts, times the children of a node
// for the ACP variants) and from how many trees there are for the device.  Launches of more trees than SMs come here only where
// choose_pool leaves them: up to 32 games or 32 steps, and what it says of few steps; the figures below for such trees are of longer launches.
//   Many trees (at least two per SM): a quarter of the games, between 32 and 320; half of them when a step has at most 256
//   games.  Measured on 256 roots, G playouts/s: ACP 4 x 256 (1792 games a step), 500 steps, 18.2 / 20.3 / 20.2 / 18.7 / 19.0 / 19.0 at 256 /
//   288 / 320 / 352 / 384 / 512 threads (a thread of a smaller block plays more games per step, so less of a step is spent
//   waiting for its last games); OCP 8 trees x 1000 steps (small blocks put more trees on an SM, which hides the latency of
//   the select/expand/backup warp) with 128 playouts 9.4 / 10.7 / 8.4 at 32 / 64 / 128 threads, with 256 13.8 / 15.0 / 13.7 at 64 / 128 /
//   256, with 512 22.6 / 20.6 / 19.0 / 14.3 at 128 / 192 / 256 / 512.  The rule misses the best count where a step has 224 to 448 games
//   (ACP 4 x 32 8.5 against 9.4 and 4 x 64 11.0 against 13.3 at 224 threads), with 64 playouts of OCP (7.0 against 8.4 at 64) and with 512
//   of ACP (20.5 against 22.3 at 512).
//   Few trees (a tree has an SM to itself): one thread per game, at most 1024: 132 trees of ACP 4 x 256, 1000 steps, 27.6 / 23.1 / 21.1 / 20.5 /
//   21.7 ms at 256 / 384 / 512 / 768 / 1024 threads; of OCP 4 x 128 17.9 / 11.6 / 6.5 / 5.0 at 32 / 64 / 128 / 160.
//   In between: half the games, at most 512: 200 trees of ACP 4 x 256 29.8 / 26.0 / 27.0 / 21.9 / 23.4 ms at 256 / 384 / 512 / 768 / 1024
//   threads, of OCP 4 x 128 11.7 / 7.0 / 5.4 at 64 / 128 / 160: a block of more threads would pay there too.
int choose_threads(mctsnc_handle *h, long long trees) {
    const int games = h->cfg.n_playouts * (is_ocp(h->cfg) ? 1 : h->A);
    auto fit = [](int want, int most) {
        const int t = (want + 31) / 32 * 32;
        return t < 32 ? 32 : (t > most ? most : t);
    };
    int threads;
    if (trees >= 2LL * h->sm_count) threads = fit(games <= 256 ? games / 2 : games / 4, 320);
    else if (trees <= h->sm_count) threads = fit(games, 1024);
    else threads = fit(games / 2, 512);
    const void *fn = search_kernel_ptr(h->cfg, play_straight(h->cfg, threads));
    int per_sm = 0;
    while (threads > 32 &&
           (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, h->dyn_smem) != cudaSuccess || per_sm < 1))
        threads -= 32;
    return threads;
}

// The block per SM of c4_pool.cuh: the trees it grows side by side, its walking warps and its threads
struct PoolShape {
    int trees, walkers, threads;
};
constexpr int POOL_SMEM_LIMIT = 226 * 1024, AHEAD_SMEM_LIMIT = 200 * 1024;

const void *pool_kernel_ptr(bool ocp) { return ocp ? (const void *)c4::pool_kernel<true> : (const void *)c4::pool_kernel<false>; }

// Whether the trees of a launch grow in a block per SM that plays the games of all its trees together, and that block's shape.
// Everything is chosen by the games of a step (`games`) and the trees there are for an SM; 200 steps from random positions,
// ms with a block per tree / with the pool:
//   games a step                      56          128         224         256         448         512         896         1792
//   184 trees                     1.95/1.32   2.11/1.51   1.91/1.71   2.16/1.82   2.45/2.23   2.69/2.41   3.73/3.03   5.92/4.18
//   300 trees                     1.97/1.34   2.14/1.51   1.96/1.70   2.26/1.83   2.90/2.25   3.38/2.47   4.41/3.15   7.43/4.98
//   600 trees                     2.04/1.49   2.35/1.83   2.53/2.03   2.86/2.21   3.84/2.77   4.43/3.06   5.97/3.90   (120 steps) 5.89/4.20
//   1024 trees                    2.22/1.67   2.89/2.15   3.64/2.46   4.10/2.82   5.69/3.56   6.52/3.92   7.18/5.57   7.83/6.22
//   2048 trees                    2.76/2.05   4.34/3.16   4.69/3.67   5.37/4.25   7.45/5.81   (120 steps) 5.68/4.16   7.89/6.38   14.3/12.1
// Up to 32 games a step a block of one warp has a lane for every game and no queue to go through (1024 trees 1.53 against 1.90).  A tree
// for every SM or fewer: nothing to share; with 896 games or more a tree and an SM the block per tree is also faster while few SMs
// have two (160 trees of 1792 games 3.82 against 4.10).
// Trees at once: all of an SM's while their games are few, since a tree that waits for a place stands still; where the games
// of fewer trees fill the lanes, fewer, so that the work queue can even out the SMs.
// Walkers: one for two trees, more where the games are few and the walk is most of a step.  Players: enough lanes, but a lane
// of a smaller block plays its ply sooner.
// Launches of up to SLICE_STEPS steps keep the block per tree.  (The table is of six trees of 896 games and four of 1792 at most.)
bool choose_pool(const mctsnc_handle *h, long long trees, int steps, PoolShape *shape) {
    const int games = h->cfg.n_playouts * (is_ocp(h->cfg) ? 1 : h->A);
    const bool large = games >= 896;
    if (h->cfg.threads_per_tree > 0 || steps <= SLICE_STEPS || games <= 32 || trees <= (large ? h->sm_count + h->sm_count / 6 : h->sm_count)) return false;
    const long long need = (trees + h->sm_count - 1) / h->sm_count;
    // 4 trees of 1792 games, 10 of 256, 14 of 128.  One more of 896 games and more pays where the trees are many for the places, and the more
    // so the longer they take turns with them: ms with 4 / 5 trees of 1792 games, 200, 500, 1000 and 2000 steps, 908 trees (1.23 a place of
    // the 5) 9.03 / 10.07, 20.8 / 24.7, 39.6 / 45.0, 75.4 / 83.7; 980 (1.32) 9.72 / 10.15, 22.6 / 23.3, 43.2 / 44.0, 82.5 / 82.6; 1024 (1.38) 10.12 /
    // 10.38, 23.7 / 23.8, 45.2 / 44.8, 86.4 / 84.7; 1220 (1.65) 11.50 / 11.56, 27.1 / 26.9, 51.7 / 50.5, 99.1 / 95.3; with 6 / 7 of 896 games 1352
    // (1.30) 6.87 / 7.05, 16.1 / 16.5, 31.1 / 31.6, 60.5 / 60.8; 1420 (1.37) 7.25 / 7.36, 17.1 / 17.0, 33.0 / 32.2, 64.3 / 61.8; 1536 (1.48) 7.75 /
    // 7.74, 18.4 / 18.1, 35.4 / 34.7, 69.1 / 66.8; 40 and 100 steps of 2048 trees of 896 games 2.40 / 2.57 and 5.28 / 5.30, of 1536 of 1792 3.50 / 3.73
    // and 7.59 / 7.71.
    long long most = (long long)ceilf(150.f / sqrtf((float)games));
    if (large && steps >= 200 && (double)trees >= (1.31 + 45. / steps) * (double)((most + 1) * h->sm_count)) most++;
    long long k = need;
    if (large) k = (long long)(0.72f * (float)trees / (float)h->sm_count + 0.6f);
    else if (need > 3 && games > 128 && need * games > 2048) k = need * 18 / 25 < 3 ? 3 : need * 18 / 25;
    if (k > most) k = most;
    if (k < 1) k = 1;
    if (k > c4::POOL_MAX_TREES) k = c4::POOL_MAX_TREES;
    while (k > 1 && c4::pool_bytes((int)k, (int)(h->rng_per_search / h->cfg.n_trees)) > (size_t)POOL_SMEM_LIMIT) k--;
    // Trees that take turns with one place an SM, and not enough steps to make up for the first turns: us with a block per tree / with the
    // pool, 896 games, 33, 48, 64 and 100 steps, 210 trees 698 / 804, 1002 / 1011, 1319 / 1232, 2041 / 1790; 250 728 / 890, 1027 / 1107, 1366 / 1332, 2081 /
    // 1874; 286 727 / 960, 1040 / 1189, 1364 / 1420, 2083 / 2008; 1792 games, 33, 40 and 48 steps, 210 trees 1109 / 1101, 1346 / 1246, 1588 / 1404; 250
    // 1157 / 1248, 1387 / 1383, 1651 / 1539; 286 1151 / 1340, 1385 / 1484, 1643 / 1647; 3584 games, 250 trees 1993 / 2022, 2392 / 2235, 2837 / 2497.
    if (k == 1 && steps < (games < 1792 ? 60 : 40) && 20 * trees > 29 * h->sm_count) return false;
    shape->trees = (int)k;
    shape->walkers = (int)(k + 1) / 2;
    if (games <= 512 && shape->walkers < 5) shape->walkers = k < 5 ? (int)k : 5;
    const float side_by_side = (float)(k * games);
    float lanes = (k <= 3 && games >= 224 ? 10.f : 8.f) * sqrtf(side_by_side);
    if (side_by_side > 1024.f) lanes = fminf(lanes + 0.08f * (side_by_side - 1024.f), 12.f * sqrtf(side_by_side));
    int players = (int)lanes / 32;
    if (players < 1) players = 1;
    if (players > 32 - shape->walkers) players = 32 - shape->walkers;
    shape->threads = 32 * (shape->walkers + players);
    return true;
}

// the launch takes its trees from the work queue, SLICE_STEPS steps at a time
void use_queue(mctsnc_handle *h, SearchParams &p, long long trees, int steps, cudaStream_t stream) {
    init_queue_kernel<<<(unsigned)((trees + 255) / 256), 256, 0, stream>>>(h->queue, h->ring, h->remaining, (int)trees, steps);
    p.queue = h->queue;
    p.ring = h->ring;
    p.remaining = h->remaining;
    p.ring_cap = (int)trees;
    p.chunk = SLICE_STEPS;
    if (h->trace) {
        cudaMemsetAsync(h->trace_count, 0, sizeof(int), stream);
        p.trace = h->trace;
        p.trace_count = h->trace_count;
        p.trace_cap = h->trace_cap;
    }
}

int seed_streams(mctsnc_handle *h, int batch, cudaStream_t stream) {
    const int grid = 148 * 4;
    replicate_streams_kernel<<<grid, 256, 0, stream>>>(h->rng_playout, h->rng_playout_base, h->rng_per_search, batch);
    if (is_ocp(h->cfg))
        replicate_streams_kernel<<<grid, 256, 0, stream>>>(h->rng_expand, h->rng_expand_base, h->cfg.n_trees, batch);
    return (int)cudaGetLastError();
}

// the turns of the roots lie behind the `batch` boards, so that one copy takes both
int send_roots(mctsnc_handle *h, void *boards, const void *host_boards, size_t board_bytes, int batch, cudaStream_t stream) {
    h->root_turn = reinterpret_cast<signed char *>(boards) + board_bytes;
    CUDA_TRY(cudaMemcpyAsync(boards, host_boards, board_bytes + (size_t)batch, cudaMemcpyHostToDevice, stream));
    CUDA_TRY(cudaEventRecord(h->ev_staged, stream));
    h->staging_in_flight = true;
    return 0;
}

int stage_roots(mctsnc_handle *h, int batch, const int8_t *boards, const int8_t *extras, const int8_t *turns,
                cudaStream_t stream) {
    const int cells = h->cfg.board_rows * h->cfg.board_cols;
    const int extra = h->cfg.extra_info_memory;
    // the pinned staging buffers are about to be rewritten: the copies of the previous call (asynchronous entry points
    // return before they ran) must have read them
    if (h->staging_in_flight) {
        CUDA_TRY(cudaEventSynchronize(h->ev_staged));
        h->staging_in_flight = false;
    }
    signed char *host_turns = is_gomoku(h->cfg) ? reinterpret_cast<signed char *>(h->h_root_gboard + (long long)batch * 16)
                                                : reinterpret_cast<signed char *>(h->h_root_board + batch);
    if (is_gomoku(h->cfg)) {
        for (int b = 0; b < batch; b++) {
            if (turns[b] != 1 && turns[b] != -1) return MCTSNC_E_BAD_ARGUMENT;
            const int rc = gomoku_encode_root(boards + (long long)b * cells, h->h_root_gboard + (long long)b * 16);
            if (rc) return rc;
            host_turns[b] = turns[b];
        }
        return send_roots(h, h->root_gboard, h->h_root_gboard, sizeof(unsigned) * 16 * batch, batch, stream);
    }
    for (int b = 0; b < batch; b++) {
        if (turns[b] != 1 && turns[b] != -1) return MCTSNC_E_BAD_ARGUMENT;
        const int rc = c4_encode_root(boards + (long long)b * cells, extras ? extras + (long long)b * extra : nullptr,
                                      &h->h_root_board[b]);
        if (rc) return rc;
        host_turns[b] = turns[b];
    }
    return send_roots(h, h->root_board, h->h_root_board, sizeof(ulonglong2) * batch, batch, stream);
}

// one_tree: acp only (ocp searches of few trees run in gomoku_block_kernel)
const void *gomoku_playout_kernel(bool ocp, bool one_tree) {
    if (ocp) return (const void *)gomoku::playout_dynamic_kernel<true, false>;
    return one_tree ? (const void *)gomoku::playout_dynamic_kernel<false, true> : (const void *)gomoku::playout_dynamic_kernel<false, false>;
}

// The kernel that runs an OCP search of Gomoku with a block per tree, its threads and dynamic shared memory: a player for every
// game of a step up to 256
const void *gomoku_block_kernel(int playouts, int *threads, size_t *smem) {
    if (playouts <= 32) {
        *threads = 32 + 32;
        *smem = sizeof(gomoku::BlockMemory<32>);
        return (const void *)gomoku::search_block_kernel<32>;
    }
    if (playouts <= 64) {
        *threads = 64 + 32;
        *smem = sizeof(gomoku::BlockMemory<64>);
        return (const void *)gomoku::search_block_kernel<64>;
    }
    if (playouts <= 128) {
        *threads = 128 + 32;
        *smem = sizeof(gomoku::BlockMemory<128>);
        return (const void *)gomoku::search_block_kernel<128>;
    }
    *threads = 256 + 32;
    *smem = sizeof(gomoku::BlockMemory<256>);
    return (const void *)gomoku::search_block_kernel<256>;
}

int launch_search_gomoku(mctsnc_handle *h, int batch, int steps, int first, cudaStream_t stream) {
    gomoku::Params p;
    p.rec = h->rec;
    p.board = h->gboard;
    p.parent = h->parent;
    p.state = h->state;
    p.step = h->gstep;
    p.paths = h->paths;
    p.path_rec = h->path_rec;
    p.term = h->path_term;
    p.actions_expanded = h->actions_expanded;
    p.child_out = reinterpret_cast<int2 *>(h->child_out);
    p.child_outcome = h->child_outcome;
    p.child_action = h->child_action;
    p.sheet = h->gsheet;
    p.rng_playout = h->rng_playout;
    p.rng_expand = h->rng_expand;
    p.root_board = h->root_gboard;
    p.root_turn = h->root_turn;
    p.work = h->gwork;
    p.cap = h->cfg.node_capacity;
    p.node_limit = h->cfg.max_tree_size < h->cfg.node_capacity ? h->cfg.max_tree_size : h->cfg.node_capacity;
    p.n_trees = h->cfg.n_trees;
    p.n_playouts = h->cfg.n_playouts;
    p.variant = h->cfg.variant;
    p.first = first;
    p.steps = steps;
    p.ucb_c = h->cfg.ucb_c;
    p.ms_per_cycle = h->ms_per_cycle;
    const int trees = (int)((long long)batch * h->cfg.n_trees);
    p.tree_base = 0;
    p.backup_only = 0;
    const bool ocp = is_ocp(h->cfg);
    void *args[] = {&p};
    if (ocp) {
        // a block per tree while all of them are on the device at once
        int threads = 0, fit = 0;
        size_t smem = 0;
        const void *kernel = gomoku_block_kernel(p.n_playouts, &threads, &smem);
        CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, smem) == cudaSuccess &&
            trees <= (long long)fit * h->sm_count) {
            h->threads = threads;
            h->kernel = "gomoku::search_block_kernel";
            h->blocks_per_sm = fit;
            return (int)cudaLaunchKernel(kernel, dim3((unsigned)trees), dim3((unsigned)threads), args, smem, stream);
        }
    }
    // Else two launches per step (tree step, playouts) and a closing backup, or, where a group of an acp search is one tree, one launch
    // per step after the first tree step; all enqueued without waiting.
    //
    // The trees are split into groups, each with a stream of its own: a tree's next step only needs that tree's games to be
    // over, so the groups run out of step with each other and the lanes one tree leaves idle while its longest games finish
    // (up to ~170 plies against a mean of ~85) play the games of the others.  No kernel waits for another: the order inside a
    // group is stream order, the groups are forked from and joined to the caller's stream with events.
    int per_sm = 0;
    const int groups = trees < GOMOKU_STREAMS ? trees : GOMOKU_STREAMS;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gomoku_playout_kernel(ocp, trees == groups), gomoku::DYN_THREADS, h->dyn_smem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const long long resident = (long long)per_sm * h->sm_count;
    h->threads = gomoku::DYN_THREADS;
    h->kernel = "gomoku::playout_dynamic_kernel";
    h->blocks_per_sm = per_sm;
    CUDA_TRY(cudaEventRecord(h->g_fork, stream));
    for (int g = 0; g < groups; g++) CUDA_TRY(cudaStreamWaitEvent(h->g_stream[g], h->g_fork, 0));
    for (int s = 0; s <= steps; s++) {
        for (int g = 0; g < groups; g++) {
            const int t0 = (int)((long long)trees * g / groups), t1 = (int)((long long)trees * (g + 1) / groups);
            const int n = t1 - t0;
            const bool one_tree = !ocp && n == 1;
            p.tree_base = t0;
            cudaStream_t gs = h->g_stream[g];
            if (s == 0 || !one_tree) {   // the playouts of one tree make the tree's step that follows them
                p.first = (first && s == 0) ? 1 : 0;
                p.backup_only = s == steps ? 1 : 0;
                if (ocp) gomoku::tree_step_kernel<true><<<n, 32, 0, gs>>>(p);
                else gomoku::tree_step_kernel<false><<<n, 32, 0, gs>>>(p);
            }
            if (s == steps) continue;
            p.first = 0;
            p.backup_only = s + 1 == steps ? 1 : 0;
            // Blocks of the launch.  A lane for every game while that does not oversubscribe the device much (OCP: one child
            // per tree); otherwise 1.5 to 2 times the group's share of the blocks that fit on the device at once, so that a
            // lane plays several games one after the other and its warp stays full, and blocks are waiting to start
            // where another group's launch is running out of games.
            const long long games = (long long)n * h->cfg.n_playouts * (ocp ? 1 : h->A);
            const long long enough = (games + gomoku::DYN_THREADS - 1) / gomoku::DYN_THREADS;
            long long blocks = enough;
            const long long quarters = groups >= GOMOKU_STREAMS ? 8 : 6;
            if (enough * groups > (5 * resident) / 2) blocks = (quarters * resident + 4 * groups - 1) / (4 * groups);
            if (blocks > enough) blocks = enough;
            if (blocks > resident) blocks = resident;
            if (blocks < 1) blocks = 1;
            int count = n;
            void *play_args[] = {&p, &count};
            // Steps of one tree follow each other without a gap: the next launch's blocks come to the device while the last warp of this
            // one walks.  Not where all games of all trees have a lane at once, and the trees are several (2 x 128 13.0 -> 13.4 ms of 200
            // steps; 4 x 256 42.2 -> 41.3 of 300, 8 x 256 25.0 -> 24.0 of 100, 1 x 256 15.2 -> 14.7, 4 x 128 12.6 -> 12.4).
            cudaLaunchConfig_t lc = {};
            lc.gridDim = dim3((unsigned)blocks);
            lc.blockDim = dim3(gomoku::DYN_THREADS);
            lc.dynamicSmemBytes = h->dyn_smem;
            lc.stream = gs;
            cudaLaunchAttribute overlap;
            overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            overlap.val.programmaticStreamSerializationAllowed = 1;
            lc.attrs = &overlap;
            lc.numAttrs = one_tree && (groups == 1 || enough * groups > resident) ? 1 : 0;
            CUDA_TRY(cudaLaunchKernelExC(&lc, gomoku_playout_kernel(ocp, one_tree), play_args));
        }
    }
    for (int g = 0; g < groups; g++) {
        CUDA_TRY(cudaEventRecord(h->g_join[g], h->g_stream[g]));
        CUDA_TRY(cudaStreamWaitEvent(stream, h->g_join[g], 0));
    }
    return (int)cudaGetLastError();
}

const void *cluster_kernel_ptr(bool ocp, int form) {
    // acp only
    if (form == WIDE_AHEAD) return (const void *)c4::search_cluster_kernel<false, c4::WIDE_CLUSTER_BLOCKS, c4::WIDE_CLUSTER_THREADS, true>;
    if (form == WIDE) return (const void *)c4::search_cluster_kernel<false, c4::WIDE_CLUSTER_BLOCKS, c4::WIDE_CLUSTER_THREADS, false>;
    if (form == PACKED) return ocp ? (const void *)c4::search_packed_cluster_kernel<true> : (const void *)c4::search_packed_cluster_kernel<false>;
    if (form == AHEAD) return ocp ? (const void *)c4::search_cluster_kernel<true, c4::CLUSTER_BLOCKS, c4::CLUSTER_THREADS, true>
                                  : (const void *)c4::search_cluster_kernel<false, c4::CLUSTER_BLOCKS, c4::CLUSTER_THREADS, true>;
    return ocp ? (const void *)c4::search_cluster_kernel<true, c4::CLUSTER_BLOCKS, c4::CLUSTER_THREADS, false>
               : (const void *)c4::search_cluster_kernel<false, c4::CLUSTER_BLOCKS, c4::CLUSTER_THREADS, false>;
}

// Draws made ahead (c4::Draws) cost a launch 64 draws of every stream at its begin and the way back at its end, 3 us where a
// thread has one stream and 7 where it has two, and save a part of a step.  Launches of fewer steps than this play without: us with /
// without, 8 and 16 steps, 1 x 32 ocp 47.7 / 46.9 and 80.9 / 82.0, 8 x 256 ocp 67.5 / 65.4 and 110.5 / 110.5, 4 x 32 acp 61.3 / 61.3 and 101.3 /
// 104.5; clusters 4 x 64 acp 54.0 / 53.2 and 97.2 / 98.4, 4 x 512 ocp 56.0 / 55.2 and 100.2 / 102.3, 4 x 256 acp 57.4 / 56.1 and 101.2 / 101.4.
constexpr int AHEAD_MIN_STEPS = 16;

// And of clusters, by the streams of a block; us with / without, 32, 64, 200 and 1000 steps:
//   8 blocks, 64 streams (512 ocp) 189 / 195, 365 / 378, 1110 / 1159, 5697 / 5847; 56 (64 acp) 184 / 187, 354 / 363, 1078 / 1116, 5418 / 5608;
//   112 (128 acp), four warps that play beside the walker's: never, 193 / 188, 373 / 367, 1139 / 1129, 5739 / 5697; 224 (256 acp, 12
//   trees) 214 / 222, 414 / 430, 1274 / 1329, 6372 / 6564; 448 (512 acp), two a thread: no gain, 633 / 633, 1961 / 1962, 9415 / 9419 from 64 steps;
//   16 blocks, 112 streams (256 acp) 186 / 190, 358 / 372, 1094 / 1144, 5726 / 5824; 224 (512 acp) 275 / 270, 528 / 528, 1570 / 1618,
//   7539 / 7934.
bool cluster_draws_pay(int steps, int streams, bool wide) {
    if (wide) return steps >= (streams > c4::WIDE_CLUSTER_THREADS ? 4 * AHEAD_MIN_STEPS : AHEAD_MIN_STEPS);
    return steps >= AHEAD_MIN_STEPS && (streams <= 64 || (streams > 128 && streams <= c4::CLUSTER_THREADS));
}

const char *cluster_kernel_name(int form) {
    if (form == WIDE_AHEAD) return "c4::search_cluster_kernel, 16 blocks, draws ahead";
    if (form == WIDE) return "c4::search_cluster_kernel, 16 blocks";
    if (form == AHEAD) return "c4::search_cluster_kernel, 8 blocks, draws ahead";
    return form == PACKED ? "c4::search_packed_cluster_kernel" : "c4::search_cluster_kernel, 8 blocks";
}

int launch_search(mctsnc_handle *h, int batch, int steps, int first, cudaStream_t stream) {
    if (is_gomoku(h->cfg)) return launch_search_gomoku(h, batch, steps, first, stream);
    SearchParams p;
    p.rec = h->rec;
    p.board = h->board;
    p.parent = h->parent;
    p.state = h->state;
    p.paths = h->paths;
    p.actions_expanded = h->actions_expanded;
    p.child_out = h->child_out;
    p.rng_playout = h->rng_playout;
    p.rng_expand = h->rng_expand;
    p.root_board = h->root_board;
    p.root_turn = h->root_turn;
    p.cap = h->cfg.node_capacity;
    p.node_limit = h->cfg.max_tree_size < h->cfg.node_capacity ? h->cfg.max_tree_size : h->cfg.node_capacity;
    p.n_trees = h->cfg.n_trees;
    p.n_playouts = h->cfg.n_playouts;
    p.log2_playouts = 0;
    while ((1 << p.log2_playouts) < h->cfg.n_playouts) p.log2_playouts++;
    p.n_actions = h->A;
    p.variant = h->cfg.variant;
    p.steps = steps;
    p.first = first;
    p.ucb_c = h->cfg.ucb_c;
    p.ms_per_cycle = h->ms_per_cycle;
    p.cache_nodes = 0;
    const long long trees = (long long)batch * h->cfg.n_trees;
    p.queue = nullptr;
    p.ring = nullptr;
    p.remaining = nullptr;
    p.ring_cap = 0;
    p.chunk = 0;
    p.trace = nullptr;
    p.trace_count = nullptr;
    p.trace_cap = 0;
    p.n_trees_launched = (int)trees;
    p.places = (int)trees;
    p.pool_trees = p.pool_walkers = 0;
    p.times2 = 2u;
    p.times4 = 4u;
    p.times2p23 = 1u << 23;
    // Few trees (one search, a few searches): a cluster of blocks per tree, so that the games of a step are played on
    // several SMs at once.  Measured without draws made ahead, 4 x 256 acp_prodigal, 2000 steps, 1 / 4 / 8 searches in one launch: 13.7 /
    // 14.4 / 20.6 ms with clusters (one, with them, 12.6) against 42.2 with a block of 1024 threads per tree; 500 steps, 9 / 12 / 16 searches:
    // 5.0 / 5.6 / 7.0 against 11.1 -- up to four cluster blocks per SM pay, and more do not fit.
    // Only where a step has more than 256 games (ACP with 64 playouts or more, OCP with 512).  One search of 2000 steps, 4
    // trees, with a block / with clusters: ACP 8 / 16 / 32 / 64 / 128 / 256 / 512 playouts 9.1 / 9.3 / 11.7 / 16.6 / 25.4 / 42.2 / 64.5 ms
    // against 11.2 / 11.4 / 11.8 / 12.0 / 12.5 / 13.7 / 18.2; OCP 128 / 256 / 512 playouts 10.1 / 12.3 / 17.6 against 12.2 / 12.4 / 12.7: with few
    // games the two cluster barriers of a step cost more than the games take.
    if (h->cfg.threads_per_tree == 0 && h->cluster_ok && h->cfg.n_playouts >= c4::CLUSTER_BLOCKS &&
        (long long)(is_ocp(h->cfg) ? 1 : h->A) * h->cfg.n_playouts > MCTSNC_C4_CLUSTER_MIN_GAMES &&
        trees * c4::CLUSTER_BLOCKS <= (long long)MCTSNC_C4_CLUSTER_SM_SHARE * h->sm_count) {
        const bool ocp = is_ocp(h->cfg);
        // the wide cluster first where a step has games for it (an ocp step never has: 512 at most); then the first form that fits
        // on the device
        for (int form = !ocp && h->A * h->cfg.n_playouts >= c4::WIDE_CLUSTER_MIN_GAMES ? WIDE_AHEAD : AHEAD; form <= PACKED; form++) {
            const bool wide = is_wide(form), ahead = is_ahead(form);
            const int blocks = wide ? c4::WIDE_CLUSTER_BLOCKS : c4::CLUSTER_BLOCKS;
            const int streams = (int)(h->dyn_smem / sizeof(ulonglong2)) / blocks;   // of a block
            if (ahead && !cluster_draws_pay(steps, streams, wide)) continue;
            // 16 blocks without draws made ahead come before 8 with them only where those do not pay either (8 trees of 512: 64, 200 and
            // 1000 steps 590, 1879, 9093 us against 632, 1960, 9415; of 256, 9 trees, with 16 / with 8: 410 / 410, 1249 / 1271, 6368 / 6342)
            if (form == WIDE && cluster_draws_pay(steps, (int)(h->dyn_smem / sizeof(ulonglong2)) / c4::CLUSTER_BLOCKS, false)) continue;
            const void *kernel = cluster_kernel_ptr(ocp, form);
            if (wide && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            cudaLaunchConfig_t lc = {};
            lc.gridDim = dim3((unsigned)(trees * blocks));
            lc.blockDim = dim3(wide ? c4::WIDE_CLUSTER_THREADS : c4::CLUSTER_THREADS);
            lc.stream = stream;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = (unsigned)blocks;
            attr.val.clusterDim.y = 1;
            attr.val.clusterDim.z = 1;
            lc.attrs = &attr;
            lc.numAttrs = 1;
            CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            // The first records of a tree stay in the first block's shared memory: many if every block can have an SM to itself,
            // else few.  All clusters of the launch have to be on the device at once (clusters do not spread over GPCs, so fewer
            // fit than blocks / 8): a tree whose cluster waits for another to finish would take two searches' time.  A wide cluster
            // and one with draws made ahead are for blocks that have an SM each, a packed one for blocks that share it.
            bool fits = false;
            const bool own_sm = trees * blocks <= h->sm_count;
            for (int small = own_sm && form != PACKED ? 0 : 1; small < (wide || ahead ? 1 : 2) && !fits; small++) {
                p.cache_nodes = small ? 2048 : MCTSNC_C4_CACHE_NODES;
                lc.dynamicSmemBytes = h->dyn_smem / blocks + sizeof(int4) * (size_t)p.cache_nodes +
                                      (ahead ? c4::Draws::bytes(streams) : 0);
                int &fit = h->cluster_fit[form][small];
                if (fit == 0) {
                    int n = 0;
                    const cudaError_t q = cudaOccupancyMaxActiveClusters(&n, kernel, &lc);
                    if (q != cudaSuccess) cudaGetLastError();
                    fit = q == cudaSuccess && n > 0 ? n : -1;
                }
                fits = fit >= trees;
            }
            if (!fits) continue;
            h->threads = wide ? (c4::WIDE_CLUSTER_THREADS - 32) * blocks : c4::CLUSTER_THREADS * blocks;
            h->blocks_per_sm = 1;
            void *args[] = {&p};
            h->kernel = cluster_kernel_name(form);
            if (cudaLaunchKernelExC(&lc, kernel, args) == cudaSuccess) return 0;
            cudaGetLastError();      // the launch was refused (nothing ran): one block per tree from now on
            h->cluster_ok = false;
            break;
        }
        p.cache_nodes = 0;
    }
    PoolShape pool;
    if (choose_pool(h, trees, steps, &pool)) {
        const void *kernel = pool_kernel_ptr(is_ocp(h->cfg));
        CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, POOL_SMEM_LIMIT));
        const unsigned grid = (unsigned)(trees < h->sm_count ? trees : h->sm_count);
        p.pool_trees = pool.trees;
        p.pool_walkers = pool.walkers;
        p.places = pool.trees * (int)grid;
        if (trees > p.places) use_queue(h, p, trees, steps, stream);
        h->threads = pool.threads / pool.trees;
        h->kernel = "c4::pool_kernel";
        h->blocks_per_sm = pool.trees;
        void *args[] = {&p};
        CUDA_TRY(cudaLaunchKernel(kernel, dim3(grid), dim3((unsigned)pool.threads), args,
                                  c4::pool_bytes(pool.trees, (int)(h->rng_per_search / h->cfg.n_trees)), stream));
        if (p.queue) check_queue_kernel<<<(unsigned)((trees + 255) / 256), 256, 0, stream>>>(h->remaining, h->state, (int)trees);
        return (int)cudaGetLastError();
    }
    int threads = h->cfg.threads_per_tree > 0 ? h->cfg.threads_per_tree : choose_threads(h, trees);
    h->threads = threads;
    h->kernel = "c4::search_kernel";
    // A tree that has an SM to itself gets a warp more, for the walker: it works out the counts and logarithms of the backup
    // while the others play (one warp for 32 games and the walker: 5.9 us a step, two: 4.4).
    if (h->cfg.threads_per_tree == 0 && trees <= h->sm_count && threads + 32 <= 1024) threads += 32;
    int per_sm = 0;
    const void *kernel = search_kernel_ptr(h->cfg, play_straight(h->cfg, threads));
    size_t smem = h->dyn_smem;
    // The threads that play make their draws while that warp walks (see Draws), where shared memory has room for them; two to four
    // warps do not.
    const size_t with_draws = smem + c4::Draws::bytes((int)(smem / sizeof(ulonglong2)));
    const int playing_warps = h->threads / 32;
    if (steps >= AHEAD_MIN_STEPS && threads > h->threads && play_straight(h->cfg, h->threads) && (playing_warps == 1 || playing_warps > 4) &&
        with_draws <= (size_t)AHEAD_SMEM_LIMIT) {
        kernel = is_ocp(h->cfg) ? (const void *)c4::search_kernel<true, true, true> : (const void *)c4::search_kernel<false, true, true>;
        CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AHEAD_SMEM_LIMIT));
        smem = with_draws;
        h->kernel = "c4::search_kernel, draws ahead";
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
        return MCTSNC_E_BAD_ARGUMENT;
    h->blocks_per_sm = per_sm;
    // More trees than blocks fit on the device at once: a persistent grid takes slices of SLICE_STEPS steps from the
    // work queue, so that trees with long games do not keep a few SMs busy after the others have run out of work (a block per tree in
    // both, as with an explicit threads_per_tree: 1024 trees of 2000 steps, 4 x 256 acp_prodigal, 156 ms without the queue, 115 with it; 3200
    // trees of 4 x 128 ocp_prodigal, 1000 steps, 37.3 and 29.0).  Otherwise block b grows tree b for the whole launch.
    const long long resident = (long long)per_sm * h->sm_count;
    unsigned grid = (unsigned)trees;
    if (trees > resident && steps > SLICE_STEPS) {
        use_queue(h, p, trees, steps, stream);
        grid = (unsigned)resident;
        p.places = (int)resident;
    }
    void *args[] = {&p};
    CUDA_TRY(cudaLaunchKernel(kernel, dim3(grid), dim3((unsigned)threads), args, smem, stream));
    if (p.queue) check_queue_kernel<<<(unsigned)((trees + 255) / 256), 256, 0, stream>>>(h->remaining, h->state, (int)trees);
    return (int)cudaGetLastError();
}

int launch_reduce_trees(mctsnc_handle *h, int batch, long long *sums, cudaStream_t stream) {
    if (is_gomoku(h->cfg)) {
        gomoku_reduce_over_trees_kernel<<<batch, REDUCE_THREADS, 0, stream>>>(h->rec, h->gboard, h->state, h->cfg.node_capacity,
                                                                  h->cfg.n_trees, sums, h->flags, h->dres);
        return (int)cudaGetLastError();
    }
    reduce_over_trees_kernel<<<batch, REDUCE_THREADS, 0, stream>>>(h->rec, h->state, h->cfg.node_capacity, h->cfg.n_trees, h->A, sums,
                                                        h->flags, h->dres);
    return (int)cudaGetLastError();
}

int launch_reduce_actions(mctsnc_handle *h, int batch, const long long *sums, cudaStream_t stream) {
    reduce_over_actions_kernel<<<batch, h->tpb_roa, 0, stream>>>(sums, h->flags, h->A, h->tpb_roa, is_thrifty(h->cfg) ? 1 : 0,
                                                                 h->dres);
    return (int)cudaGetLastError();
}

// the results of `batch` searches on their way to the host: one copy where the whole handle is in use or little more is copied
// than is needed (a copy costs about as much as 100 KB), else one for each part
int copy_results(mctsnc_handle *h, int batch, const long long *sums_dev, cudaStream_t stream) {
    const int A = h->A;
    const size_t per_search = h->result_bytes / h->cfg.max_batch;
    if (sums_dev == h->sums && per_search * (size_t)(h->cfg.max_batch - batch) <= 100 * 1024)
        return (int)cudaMemcpyAsync(h->h_dres, h->dres, h->result_bytes, cudaMemcpyDeviceToHost, stream);
    CUDA_TRY(cudaMemcpyAsync(h->h_sums, sums_dev, sizeof(long long) * 3 * A * batch, cudaMemcpyDeviceToHost, stream));
    CUDA_TRY(cudaMemcpyAsync(h->h_flags, h->flags, (size_t)2 * A * batch, cudaMemcpyDeviceToHost, stream));
    CUDA_TRY(cudaMemcpyAsync(h->h_dres, h->dres, sizeof(DevResult) * batch, cudaMemcpyDeviceToHost, stream));
    return 0;
}

// what copy_results has brought, after a synchronisation, in the form of the ABI
void fill_results(mctsnc_handle *h, int batch, mctsnc_result *results) {
    const int A = h->A;
    for (int b = 0; b < batch; b++) {
        mctsnc_result &r = results[b];
        const DevResult &d = h->h_dres[b];
        memset(&r, 0, sizeof(r));
        r.best_action = d.best_action;
        r.best_win_flag = d.best_win_flag;
        r.best_n = d.best_n;
        r.best_n_wins = d.best_n_wins;
        r.steps = h->last_steps;
        r.playouts = d.playouts;
        r.plies = d.plies;
        r.ub_draws = d.ub_draws;
        r.status = d.status;
        r.n_root_actions = d.n_root_actions;
        r.device_ms = h->last_ms;
        r.max_depth = d.max_depth;
        r.total_nodes = d.total_nodes;
        r.depth_sum = d.depth_sum;
        r.max_size = d.max_size;
        for (int k = 0; k < 4; k++) r.stage_ms[k] = d.stage_ms[k];
        if (is_gomoku(h->cfg)) {
            // the playouts of a Gomoku step are not a tree's own (a kernel that all trees share), or run beside the walk (the block
            // kernel): their time is what is left of the loop after the per-tree stages
            const float rest = h->last_ms - (d.stage_ms[0] + d.stage_ms[1] + d.stage_ms[3]);
            r.stage_ms[2] = rest > 0.f ? rest : 0.f;
        }
        r.reduce_ms[0] = h->reduce_ms[0];
        r.reduce_ms[1] = h->reduce_ms[1];
        for (int a = 0; a < A; a++) {
            r.root_ns[a] = h->h_sums[(long long)b * 3 * A + a];
            r.actions_ns[a] = h->h_sums[(long long)b * 3 * A + A + a];
            r.actions_ns_wins[a] = h->h_sums[(long long)b * 3 * A + 2 * A + a];
            r.actions_win_flags[a] = h->h_flags[(long long)b * 2 * A + a];
            r.actions_expanded[a] = h->h_flags[(long long)b * 2 * A + A + a];
        }
    }
}

}  // namespace

// ===================================================================================================================
// C ABI

extern "C" int mctsnc_create(const mctsnc_config *cfg, mctsnc_handle **out) {
    if (!cfg || !out) return MCTSNC_E_BAD_ARGUMENT;
    *out = nullptr;
    const mctsnc_config &c = *cfg;
    if (c.variant < 0 || c.variant > 3 || c.n_trees < 1 || c.n_trees > 512 || c.n_playouts < 1 || c.n_playouts > 512 ||
        (c.n_playouts & (c.n_playouts - 1)) != 0 || c.max_batch < 1 || c.node_capacity < 2 || c.max_tree_size < 1 ||
        c.max_actions < 1 || c.max_actions > MCTSNC_MAX_ACTIONS || c.tree_offset < 0 ||
        c.n_trees_global < c.tree_offset + c.n_trees || !(c.ucb_c >= 0.f))
        return MCTSNC_E_BAD_ARGUMENT;
    if (c.threads_per_tree != 0 && (c.threads_per_tree < 32 || c.threads_per_tree > 1024 || c.threads_per_tree % 32))
        return MCTSNC_E_BAD_ARGUMENT;
    if (c.game == MCTSNC_GAME_C4) {
        if (c.board_rows != c4::ROWS || c.board_cols != c4::COLS || c.max_actions != c4::A || c.extra_info_memory != c4::COLS)
            return MCTSNC_E_UNSUPPORTED;
    } else if (c.game == MCTSNC_GAME_GOMOKU) {
        if (c.board_rows != gomoku::M || c.board_cols != gomoku::N || c.max_actions != gomoku::A || c.extra_info_memory > 1)
            return MCTSNC_E_UNSUPPORTED;
    } else {
        return MCTSNC_E_UNSUPPORTED;
    }
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev < 1) {
        cudaGetLastError();
        return MCTSNC_E_NO_DEVICE;
    }
    if (c.device < 0 || c.device >= n_dev) return MCTSNC_E_BAD_ARGUMENT;
    CUDA_TRY(cudaSetDevice(c.device));
    mctsnc_handle *h = new (std::nothrow) mctsnc_handle();
    if (!h) return MCTSNC_E_NO_MEMORY;
    h->cfg = c;
    if (h->cfg.node_capacity > h->cfg.max_tree_size) h->cfg.node_capacity = h->cfg.max_tree_size;
    if (h->cfg.node_capacity < 2) h->cfg.node_capacity = 2;
    h->A = c.max_actions;
    // tpb table of the reference, src/mctsnc.py:360-370 (only the entries that influence results)
    const int tpb_board = pow2ceil(c.board_rows * c.board_cols);
    const int tpb_extra = pow2ceil(c.extra_info_memory < 1 ? 1 : c.extra_info_memory);
    const int tpb_actions = pow2ceil(c.max_actions);
    int tpb_r = tpb_board > tpb_extra ? tpb_board : tpb_extra;
    if (tpb_r > 512) tpb_r = 512;
    h->tpb_e1 = tpb_r > tpb_actions ? tpb_r : tpb_actions;
    if (h->tpb_e1 > 512) h->tpb_e1 = 512;
    h->tpb_roa = tpb_actions;
    cudaDeviceProp prop;
    CUDA_TRY(cudaGetDeviceProperties(&prop, c.device));
    h->sm_count = prop.multiProcessorCount;
    {
        int can = 0;
        const char *off = getenv("MCTSNC_B200_NO_CLUSTER");
        h->cluster_ok = cudaDeviceGetAttribute(&can, cudaDevAttrClusterLaunch, c.device) == cudaSuccess && can != 0 &&
                        !(off && off[0] == '1');
    }
    int clock_khz = 0;
    if (cudaDeviceGetAttribute(&clock_khz, cudaDevAttrClockRate, c.device) != cudaSuccess || clock_khz <= 0) clock_khz = 1965000;
    h->ms_per_cycle = 1.0f / (float)clock_khz;
    h->n_trees_total = (long long)c.max_batch * c.n_trees;
    const long long nodes = h->n_trees_total * h->cfg.node_capacity;
    const bool ocp = is_ocp(c);
    h->rng_per_search = ocp ? (long long)c.n_trees * c.n_playouts : (long long)c.n_trees * h->A * c.n_playouts;
    h->dyn_smem = sizeof(ulonglong2) * (size_t)(h->rng_per_search / c.n_trees);
    if (is_gomoku(c))   // per-thread game state + per-warp sheets
        h->dyn_smem = gomoku::DYN_SMEM_BYTES;
    if (h->dyn_smem > 28 * 1024) {   // with the kernels' static part more than the 48 KB every launch may have
        const void *kernels[2] = {is_gomoku(c) ? gomoku_playout_kernel(ocp, false) : search_kernel_ptr(c, false),
                                  is_gomoku(c) ? gomoku_playout_kernel(ocp, true) : search_kernel_ptr(c, true)};
        for (const void *kernel : kernels) {
            // the limit belongs to the kernel, not to the handle: never lower what another handle (or a launch) has asked for
            cudaFuncAttributes now;
            cudaError_t e = cudaFuncGetAttributes(&now, kernel);
            if (e == cudaSuccess && (size_t)now.maxDynamicSharedSizeBytes < h->dyn_smem)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h->dyn_smem);
            if (e != cudaSuccess) {
                delete h;
                return (int)e;
            }
        }
    }
    int rc = 0;
    if (!rc) rc = dev_alloc(h, &h->rec, nodes);
    if (!rc && !is_gomoku(c)) rc = dev_alloc(h, &h->board, nodes);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->gboard, nodes * 16);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->gstep, h->n_trees_total);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->gsheet, h->n_trees_total * gomoku::SHEET_WORDS);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->path_rec, h->n_trees_total * PATH_CAP);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->path_term, h->n_trees_total * PATH_CAP);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->gwork, h->n_trees_total);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->child_outcome, h->n_trees_total * h->A);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->child_action, h->n_trees_total * h->A);
    if (!rc && is_gomoku(c)) rc = dev_alloc(h, &h->root_gboard, (long long)c.max_batch * 17);   // boards and turns
    if (!rc && is_gomoku(c) && cudaMallocHost((void **)&h->h_root_gboard, sizeof(unsigned) * 17 * c.max_batch) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && is_gomoku(c)) rc = (int)cudaMemset(h->gstep, 0, sizeof(gomoku::StepInfo) * h->n_trees_total);
    if (!rc) rc = dev_alloc(h, &h->parent, nodes);
    if (!rc) rc = dev_alloc(h, &h->state, h->n_trees_total);
    if (!rc) rc = dev_alloc(h, &h->paths, h->n_trees_total * PATH_CAP);
    if (!rc) rc = dev_alloc(h, &h->actions_expanded, h->n_trees_total * (h->A + 2));
    if (!rc) rc = dev_alloc(h, &h->child_out, h->n_trees_total * h->A * 2);
    if (!rc) rc = dev_alloc(h, &h->rng_playout, h->rng_per_search * c.max_batch);
    if (!rc) rc = dev_alloc(h, &h->rng_playout_base, h->rng_per_search);
    if (!rc) rc = dev_alloc(h, &h->rng_expand, h->n_trees_total);
    if (!rc) rc = dev_alloc(h, &h->rng_expand_base, (long long)c.n_trees);
    if (!rc) rc = dev_alloc(h, &h->jump_cols, (long long)JUMP_LEVELS * 128);
    if (!rc) rc = (int)cudaMemcpy(h->jump_cols, jump_matrix_table(), sizeof(JumpColumn) * JUMP_LEVELS * 128, cudaMemcpyHostToDevice);
    if (!rc) rc = dev_alloc(h, &h->root_board, (long long)c.max_batch * 2);   // boards and turns
    if (!rc && !is_gomoku(c)) rc = dev_alloc(h, &h->queue, 1);
    if (!rc && !is_gomoku(c)) rc = dev_alloc(h, &h->ring, h->n_trees_total * QUEUE_LEVELS);
    if (!rc && !is_gomoku(c)) rc = dev_alloc(h, &h->remaining, h->n_trees_total);
    {
        const size_t sums_at = sizeof(DevResult) * c.max_batch, flags_at = sums_at + sizeof(long long) * 3 * h->A * c.max_batch;
        h->result_bytes = flags_at + (size_t)2 * h->A * c.max_batch;
        unsigned char *dev = nullptr, *host = nullptr;
        if (!rc) rc = dev_alloc(h, &dev, (long long)h->result_bytes);
        if (!rc && cudaMallocHost((void **)&host, h->result_bytes) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
        h->dres = reinterpret_cast<DevResult *>(dev);
        h->h_dres = reinterpret_cast<DevResult *>(host);
        if (!rc) {
            h->sums = reinterpret_cast<long long *>(dev + sums_at);
            h->flags = dev + flags_at;
            h->h_sums = reinterpret_cast<long long *>(host + sums_at);
            h->h_flags = host + flags_at;
        }
    }
    if (!rc && cudaMallocHost((void **)&h->h_root_board, sizeof(ulonglong2) * 2 * c.max_batch) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && cudaEventCreate(&h->ev0) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && cudaEventCreate(&h->ev1) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && cudaEventCreateWithFlags(&h->ev_staged, cudaEventDisableTiming) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && cudaEventCreate(&h->ev_r0) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && cudaEventCreate(&h->ev_r1) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
    if (!rc && is_gomoku(c)) {
        if (cudaEventCreateWithFlags(&h->g_fork, cudaEventDisableTiming) != cudaSuccess) rc = MCTSNC_E_NO_MEMORY;
        for (int g = 0; g < GOMOKU_STREAMS && !rc; g++)
            if (cudaStreamCreateWithFlags(&h->g_stream[g], cudaStreamNonBlocking) != cudaSuccess ||
                cudaEventCreateWithFlags(&h->g_join[g], cudaEventDisableTiming) != cudaSuccess)
                rc = MCTSNC_E_NO_MEMORY;
    }
    if (!rc) rc = (int)cudaMemset(h->state, 0, sizeof(TreeState) * h->n_trees_total);
    if (!rc) rc = (int)cudaMemset(h->actions_expanded, 0, sizeof(short) * h->n_trees_total * (h->A + 2));
    if (!rc) rc = (int)cudaMemset(h->child_out, 0, sizeof(int) * h->n_trees_total * h->A * 2);
    if (rc) {
        release(h);
        delete h;
        cudaGetLastError();
        return rc;
    }
    *out = h;
    rc = mctsnc_reset_rng(h);
    if (rc) {
        mctsnc_destroy(h);
        *out = nullptr;
    }
    return rc;
}

extern "C" int mctsnc_destroy(mctsnc_handle *h) {
    if (!h) return MCTSNC_E_BAD_ARGUMENT;
    cudaSetDevice(h->cfg.device);
    cudaDeviceSynchronize();
    release(h);
    delete h;
    return 0;
}

extern "C" int mctsnc_reset_rng(mctsnc_handle *h) {
    if (!h) return MCTSNC_E_BAD_ARGUMENT;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    const mctsnc_config &c = h->cfg;
    const bool ocp = is_ocp(c);
    RngState seeded;
    rng_seed(seeded, c.seed);
    // playout streams: ACP stream (tree, action, t) = tree*A*P + action*P + t (src/mctsnc.py:1938, :2028),
    // OCP stream (tree, t) = tree*P + t (cuda.grid(1), :1849); `tree` counts over the whole (sharded) search.  Every
    // stream is computed on the device from its index (numba builds them one after the other on the host).
    const long long per_tree = ocp ? (long long)c.n_playouts : (long long)h->A * c.n_playouts;
    const unsigned grid = (unsigned)((h->rng_per_search + 127) / 128 < 4096 ? (h->rng_per_search + 127) / 128 : 4096);
    init_streams_kernel<<<grid, 128>>>(h->rng_playout_base, h->jump_cols, seeded.s0, seeded.s1, (long long)c.tree_offset * per_tree,
                                       1, h->rng_per_search);
    if (ocp)  // the child pick of tree `tree` uses stream tree * tpb_e1 of a second array with the same seed (:391, :1385)
        init_streams_kernel<<<1, 128>>>(h->rng_expand_base, h->jump_cols, seeded.s0, seeded.s1,
                                        (long long)c.tree_offset * h->tpb_e1, h->tpb_e1, c.n_trees);
    CUDA_TRY(cudaGetLastError());
    int rc = seed_streams(h, c.max_batch, 0);
    if (rc) return rc;
    CUDA_TRY(cudaDeviceSynchronize());
    return 0;
}

extern "C" int mctsnc_run(mctsnc_handle *h, const int8_t *board, const int8_t *extra_info, int32_t turn, int64_t steps_limit,
                          double time_limit_s, mctsnc_result *out) {
    if (!h || !board || !out) return MCTSNC_E_BAD_ARGUMENT;
    if (steps_limit < 0 && !(time_limit_s > 0)) return MCTSNC_E_BAD_ARGUMENT;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    const int8_t t8 = (int8_t)turn;
    h->staged_roots = 0;
    int rc = stage_roots(h, 1, board, extra_info, &t8, 0);
    if (rc) return rc;
    h->staged_roots = 1;
    // behind the last launch of the search: the reductions and the copy of the results, then one wait for everything
    auto finish = [&]() -> int {
        int e = launch_reduce_trees(h, 1, h->sums, 0);
        if (e) return e;
        CUDA_TRY(cudaEventRecord(h->ev_r0, 0));
        e = launch_reduce_actions(h, 1, h->sums, 0);
        if (e) return e;
        CUDA_TRY(cudaEventRecord(h->ev_r1, 0));
        e = copy_results(h, 1, h->sums, 0);
        if (e) return e;
        return (int)cudaStreamSynchronize(0);
    };
    const auto t0 = std::chrono::steady_clock::now();
    long long done = 0;
    float total_ms = 0.f;
    const bool timed = time_limit_s > 0;   // otherwise all steps in launches of at most a million
    int chunk = timed ? 16 : (int)(steps_limit > 1000000 ? 1000000 : steps_limit);
    int first = 1;
    bool finished = false;
    for (;;) {
        bool stop = steps_limit >= 0 && done >= steps_limit;
        if (!stop && timed) {
            const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
            stop = el >= time_limit_s;
        }
        if (stop && !first) break;
        long long n = stop ? 0 : chunk;  // a search without a single step still resets the trees to the root
        if (steps_limit >= 0 && done + n > steps_limit) n = steps_limit - done;
        CUDA_TRY(cudaEventRecord(h->ev0, 0));
        rc = launch_search(h, 1, (int)n, first, 0);
        if (rc) return rc;
        CUDA_TRY(cudaEventRecord(h->ev1, 0));
        finished = steps_limit >= 0 && done + n >= steps_limit;   // known to be the last launch
        if (finished) rc = finish();
        else rc = (int)cudaEventSynchronize(h->ev1);
        if (rc) return rc;
        float ms = 0.f;
        CUDA_TRY(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
        total_ms += ms;
        done += n;
        first = 0;
        if (stop || finished) break;
        if (timed && n > 0) {
            // aim at launches of about 2 ms so that the clock is read often enough
            const double per_step = ms / (double)n;
            int next = per_step > 0 ? (int)(2.0 / per_step) : chunk * 2;
            if (next < 1) next = 1;
            if (next > 4096) next = 4096;
            chunk = next;
        }
    }
    if (!finished) {
        rc = finish();
        if (rc) return rc;
    }
    h->last_ms = total_ms;
    h->last_steps = done;
    CUDA_TRY(cudaEventElapsedTime(&h->reduce_ms[0], h->ev1, h->ev_r0));
    CUDA_TRY(cudaEventElapsedTime(&h->reduce_ms[1], h->ev_r0, h->ev_r1));
    fill_results(h, 1, out);
    return 0;
}

extern "C" int mctsnc_launch_batch_device(mctsnc_handle *h, int32_t batch, const int8_t *boards, const int8_t *extras,
                                         const int8_t *turns, int64_t steps, int32_t reseed, void *stream) {
    if (!h || (boards && !turns) || batch < 1 || steps < 0 || steps > 0x7fffffff) return MCTSNC_E_BAD_ARGUMENT;
    if (batch > h->cfg.max_batch) return MCTSNC_E_CAPACITY;
    if (!boards && batch > h->staged_roots) return MCTSNC_E_BAD_ARGUMENT;  // nothing staged to search again
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    cudaStream_t s = (cudaStream_t)stream;
    int rc = 0;
    if (boards) {
        h->staged_roots = 0;
        rc = stage_roots(h, batch, boards, extras, turns, s);
        if (rc) return rc;
        h->staged_roots = batch;
    }
    if (reseed) {
        rc = seed_streams(h, batch, s);
        if (rc) return rc;
    }
    CUDA_TRY(cudaEventRecord(h->ev0, s));
    rc = launch_search(h, batch, (int)steps, 1, s);
    if (rc) return rc;
    CUDA_TRY(cudaEventRecord(h->ev1, s));
    h->last_steps = steps;
    h->reduce_ms[0] = h->reduce_ms[1] = 0.f;
    return 0;
}

extern "C" int mctsnc_reduce_trees_device(mctsnc_handle *h, int32_t batch, int64_t *partial_sums_device, void *stream) {
    if (!h || batch < 1) return MCTSNC_E_BAD_ARGUMENT;
    if (batch > h->cfg.max_batch) return MCTSNC_E_CAPACITY;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    return launch_reduce_trees(h, batch, partial_sums_device ? (long long *)partial_sums_device : h->sums, (cudaStream_t)stream);
}

extern "C" int mctsnc_search_batch_device(mctsnc_handle *h, int32_t batch, const int8_t *boards, const int8_t *extras,
                                          const int8_t *turns, int64_t steps, int32_t reseed, int64_t *partial_sums_device,
                                          void *stream) {
    int rc = mctsnc_launch_batch_device(h, batch, boards, extras, turns, steps, reseed, stream);
    if (rc) return rc;
    return mctsnc_reduce_trees_device(h, batch, partial_sums_device, stream);
}

extern "C" int mctsnc_finish_batch_device(mctsnc_handle *h, int32_t batch, const int64_t *summed_device, mctsnc_result *results,
                                          void *stream) {
    if (!h || batch < 1) return MCTSNC_E_BAD_ARGUMENT;
    if (batch > h->cfg.max_batch) return MCTSNC_E_CAPACITY;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    cudaStream_t s = (cudaStream_t)stream;
    const long long *sums = summed_device ? (const long long *)summed_device : h->sums;
    int rc = launch_reduce_actions(h, batch, sums, s);
    if (rc) return rc;
    if (!results) return 0;  // the caller keeps everything on the device
    rc = copy_results(h, batch, sums, s);
    if (rc) return rc;
    CUDA_TRY(cudaStreamSynchronize(s));
    CUDA_TRY(cudaEventSynchronize(h->ev1));   // recorded on another stream, perhaps
    CUDA_TRY(cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1));
    fill_results(h, batch, results);
    return 0;
}

extern "C" int mctsnc_run_batch(mctsnc_handle *h, int32_t batch, const int8_t *boards, const int8_t *extras, const int8_t *turns,
                                int64_t steps, int32_t reseed, mctsnc_result *results) {
    int rc = mctsnc_search_batch_device(h, batch, boards, extras, turns, steps, reseed, nullptr, nullptr);
    if (rc) return rc;
    return mctsnc_finish_batch_device(h, batch, nullptr, results, nullptr);
}

// per-node fields of Gomoku trees in the reference's formats (see mctsnc_export)
static int export_nodes_gomoku(mctsnc_handle *h, const std::vector<TreeState> &st, long long g0, int field, void *dst,
                               long long max_nodes) {
    constexpr int A = gomoku::A;
    const int T = h->cfg.n_trees;
    const long long cap = h->cfg.node_capacity;
    const int extra = h->cfg.extra_info_memory < 1 ? 1 : h->cfg.extra_info_memory;
    std::vector<int4> rec;
    std::vector<unsigned> brd;
    std::vector<int> par;
    for (int t = 0; t < T; t++) {
        long long n = st[t].size < max_nodes ? st[t].size : max_nodes;
        if (n > cap) n = cap;
        rec.resize((size_t)n);
        CUDA_TRY(cudaMemcpy(rec.data(), h->rec + (g0 + t) * cap, sizeof(int4) * n, cudaMemcpyDeviceToHost));
        if (field == MCTSNC_F_TREES) {
            par.resize((size_t)n);
            CUDA_TRY(cudaMemcpy(par.data(), h->parent + (g0 + t) * cap, sizeof(int) * n, cudaMemcpyDeviceToHost));
        }
        if (field == MCTSNC_F_TREES || field == MCTSNC_F_BOARDS) {
            brd.resize((size_t)n * 16);
            CUDA_TRY(cudaMemcpy(brd.data(), h->gboard + (g0 + t) * cap * 16, sizeof(unsigned) * 16 * n, cudaMemcpyDeviceToHost));
        }
        for (long long i = 0; i < max_nodes; i++) {
            const bool valid = i < n;
            const int4 r = valid ? rec[(size_t)i] : make_int4(0, 0, -1, 0);
            const long long o = (long long)t * max_nodes + i;
            const unsigned *b = valid && !brd.empty() ? &brd[(size_t)i * 16] : nullptr;
            switch (field) {
            case MCTSNC_F_TREES: {
                int32_t *row = (int32_t *)dst + o * (1 + A);
                row[0] = valid ? par[(size_t)i] : -1;
                const int n_children = r.w & gomoku::G_NCHILD_MASK;
                int rank = 0;
                for (int a = 0; a < A; a++) {
                    const bool empty = valid && !(((b[a >> 5] | b[8 + (a >> 5)]) >> (a & 31)) & 1u);
                    row[1 + a] = (empty && rank < n_children) ? r.z + rank : -1;
                    rank += empty;
                }
                break;
            }
            case MCTSNC_F_DEPTHS: ((int16_t *)dst)[o] = valid ? (int16_t)gomoku::g_depth(r.w) : 0; break;
            case MCTSNC_F_TURNS: ((int8_t *)dst)[o] = valid ? (int8_t)gomoku::g_turn(r.w) : 0; break;
            case MCTSNC_F_LEAVES: ((uint8_t *)dst)[o] = valid ? ((r.w & gomoku::G_NCHILD_MASK) == 0) : 0; break;
            case MCTSNC_F_TERMINALS: ((uint8_t *)dst)[o] = valid ? ((r.w & gomoku::G_TERMINAL) != 0) : 0; break;
            case MCTSNC_F_OUTCOMES: ((int8_t *)dst)[o] = valid ? (int8_t)gomoku::g_outcome(r.w) : 0; break;
            case MCTSNC_F_NS: ((int32_t *)dst)[o] = valid ? r.x : 0; break;
            case MCTSNC_F_NS_WINS: ((int32_t *)dst)[o] = valid ? r.y : 0; break;
            case MCTSNC_F_BOARDS: {
                int8_t *bo = (int8_t *)dst + o * A;
                for (int a = 0; a < A; a++)
                    bo[a] = !valid ? 0 : (((b[8 + (a >> 5)] >> (a & 31)) & 1u) ? 1 : (((b[a >> 5] >> (a & 31)) & 1u) ? -1 : 0));
                break;
            }
            case MCTSNC_F_EXTRA_INFOS: memset((int8_t *)dst + o * extra, 0, extra); break;
            }
        }
    }
    return 0;
}

extern "C" int mctsnc_export(mctsnc_handle *h, int32_t search, int32_t field, void *dst, int64_t max_nodes) {
    if (!h || !dst || search < 0 || search >= h->cfg.max_batch) return MCTSNC_E_BAD_ARGUMENT;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    CUDA_TRY(cudaDeviceSynchronize());
    const int T = h->cfg.n_trees, A = h->A;
    const long long cap = h->cfg.node_capacity;
    const long long g0 = (long long)search * T;
    std::vector<TreeState> st(T);
    CUDA_TRY(cudaMemcpy(st.data(), h->state + g0, sizeof(TreeState) * T, cudaMemcpyDeviceToHost));
    switch (field) {
    case MCTSNC_F_SIZES:
        for (int t = 0; t < T; t++) ((int32_t *)dst)[t] = st[t].size;
        return 0;
    case MCTSNC_F_NODES_SELECTED:
        for (int t = 0; t < T; t++) ((int32_t *)dst)[t] = st[t].selected;
        return 0;
    case MCTSNC_F_PLAYOUT_OUTCOMES:
        for (int t = 0; t < T; t++) {
            ((int32_t *)dst)[2 * t] = st[t].out_neg;
            ((int32_t *)dst)[2 * t + 1] = st[t].out_pos;
        }
        return 0;
    case MCTSNC_F_SELECTED_PATHS: {
        std::vector<int> paths((size_t)T * PATH_CAP);
        CUDA_TRY(cudaMemcpy(paths.data(), h->paths + g0 * PATH_CAP, sizeof(int) * paths.size(), cudaMemcpyDeviceToHost));
        int32_t *o = (int32_t *)dst;
        memset(o, 0, sizeof(int32_t) * T * (MAX_TREE_DEPTH + 2));
        for (int t = 0; t < T; t++) {
            for (int e = 0; e < st[t].path_len && e < PATH_CAP; e++) o[(long long)t * (MAX_TREE_DEPTH + 2) + e] = paths[(size_t)t * PATH_CAP + e];
            o[(long long)t * (MAX_TREE_DEPTH + 2) + MAX_TREE_DEPTH + 1] = st[t].path_len;
        }
        return 0;
    }
    case MCTSNC_F_ACTIONS_EXPANDED:
        CUDA_TRY(cudaMemcpy(dst, h->actions_expanded + g0 * (A + 2), sizeof(short) * T * (A + 2), cudaMemcpyDeviceToHost));
        return 0;
    case MCTSNC_F_PLAYOUT_OUTCOMES_CHILDREN:
        CUDA_TRY(cudaMemcpy(dst, h->child_out + g0 * A * 2, sizeof(int) * T * A * 2, cudaMemcpyDeviceToHost));
        return 0;
    default:
        break;
    }
    if (field < 0 || field > MCTSNC_F_EXTRA_INFOS || max_nodes < 1) return MCTSNC_E_BAD_ARGUMENT;
    if (is_gomoku(h->cfg)) return export_nodes_gomoku(h, st, g0, field, dst, max_nodes);
    const int cells = h->cfg.board_rows * h->cfg.board_cols;
    const int extra = h->cfg.extra_info_memory;
    std::vector<int4> rec;
    std::vector<ulonglong2> brd;
    std::vector<int> par;
    for (int t = 0; t < T; t++) {
        long long n = st[t].size < max_nodes ? st[t].size : max_nodes;
        if (n > cap) n = cap;
        rec.resize((size_t)n);
        CUDA_TRY(cudaMemcpy(rec.data(), h->rec + (g0 + t) * cap, sizeof(int4) * n, cudaMemcpyDeviceToHost));
        if (field == MCTSNC_F_TREES) {
            par.resize((size_t)n);
            CUDA_TRY(cudaMemcpy(par.data(), h->parent + (g0 + t) * cap, sizeof(int) * n, cudaMemcpyDeviceToHost));
        }
        if (field == MCTSNC_F_BOARDS || field == MCTSNC_F_EXTRA_INFOS) {
            brd.resize((size_t)n);
            CUDA_TRY(cudaMemcpy(brd.data(), h->board + (g0 + t) * cap, sizeof(ulonglong2) * n, cudaMemcpyDeviceToHost));
        }
        for (long long i = 0; i < max_nodes; i++) {
            const bool valid = i < n;
            const int4 r = valid ? rec[(size_t)i] : make_int4(0, 0, -1, 0);
            const long long o = (long long)t * max_nodes + i;
            switch (field) {
            case MCTSNC_F_TREES: {
                int32_t *row = (int32_t *)dst + o * (1 + A);
                row[0] = valid ? par[(size_t)i] : -1;
                const unsigned mask = r.w & 0x7F;
                int k = 0;
                for (int a = 0; a < A; a++) row[1 + a] = (valid && ((mask >> a) & 1u)) ? r.z + k++ : -1;
                break;
            }
            case MCTSNC_F_DEPTHS: ((int16_t *)dst)[o] = valid ? (int16_t)meta_depth(r.w) : 0; break;
            case MCTSNC_F_TURNS: ((int8_t *)dst)[o] = valid ? (int8_t)meta_turn(r.w) : 0; break;
            case MCTSNC_F_LEAVES: ((uint8_t *)dst)[o] = valid ? ((r.w & 0x7F) == 0) : 0; break;
            case MCTSNC_F_TERMINALS: ((uint8_t *)dst)[o] = valid ? ((r.w & META_TERMINAL) != 0) : 0; break;
            case MCTSNC_F_OUTCOMES: ((int8_t *)dst)[o] = valid ? (int8_t)meta_outcome(r.w) : 0; break;
            case MCTSNC_F_NS: ((int32_t *)dst)[o] = valid ? r.x : 0; break;
            case MCTSNC_F_NS_WINS: ((int32_t *)dst)[o] = valid ? r.y : 0; break;
            case MCTSNC_F_BOARDS: {
                int8_t *bo = (int8_t *)dst + o * cells;
                memset(bo, 0, cells);
                if (valid)
                    for (int j = 0; j < c4::COLS; j++)
                        for (int hgt = 0; hgt < c4::ROWS; hgt++) {
                            const int bit = c4::column_shift(j) + hgt;
                            const int v = ((brd[(size_t)i].y >> bit) & 1ULL) ? 1 : (((brd[(size_t)i].x >> bit) & 1ULL) ? -1 : 0);
                            bo[(c4::ROWS - 1 - hgt) * c4::COLS + j] = (int8_t)v;
                        }
                break;
            }
            case MCTSNC_F_EXTRA_INFOS: {
                int8_t *eo = (int8_t *)dst + o * extra;
                memset(eo, 0, extra);
                if (valid) {
                    const unsigned long long all = brd[(size_t)i].x | brd[(size_t)i].y;
                    for (int j = 0; j < c4::COLS; j++) eo[j] = (int8_t)__builtin_popcountll((all >> c4::column_shift(j)) & 0x3FULL);
                }
                break;
            }
            }
        }
    }
    return 0;
}

extern "C" int mctsnc_export_rng(mctsnc_handle *h, int32_t search, int32_t which, uint64_t *dst, int64_t n) {
    if (!h || !dst || search < 0 || search >= h->cfg.max_batch || n < 0) return MCTSNC_E_BAD_ARGUMENT;
    CUDA_TRY(cudaSetDevice(h->cfg.device));
    CUDA_TRY(cudaDeviceSynchronize());
    if (which == 0) {
        if (n > h->rng_per_search) return MCTSNC_E_BAD_ARGUMENT;
        CUDA_TRY(cudaMemcpy(dst, h->rng_playout + (long long)search * h->rng_per_search, sizeof(ulonglong2) * n, cudaMemcpyDeviceToHost));
    } else {
        if (!is_ocp(h->cfg) || n > h->cfg.n_trees) return MCTSNC_E_BAD_ARGUMENT;
        CUDA_TRY(cudaMemcpy(dst, h->rng_expand + (long long)search * h->cfg.n_trees, sizeof(ulonglong2) * n, cudaMemcpyDeviceToHost));
    }
    return 0;
}

extern "C" int mctsnc_query(mctsnc_handle *h, int32_t *threads_per_tree, int32_t *blocks_per_sm, int32_t *sm_count,
                            int64_t *bytes_allocated) {
    if (!h) return MCTSNC_E_BAD_ARGUMENT;
    if (threads_per_tree) *threads_per_tree = h->threads;
    if (blocks_per_sm) *blocks_per_sm = h->blocks_per_sm;
    if (sm_count) *sm_count = h->sm_count;
    if (bytes_allocated) *bytes_allocated = h->bytes;
    return 0;
}

extern "C" const char *mctsnc_search_kernel(mctsnc_handle *h) { return h ? h->kernel : ""; }

extern "C" int mctsnc_trace_slices(mctsnc_handle *h, int32_t max_records) {
    if (!h || max_records < 0) return MCTSNC_E_BAD_ARGUMENT;
    cudaFree(h->trace);
    cudaFree(h->trace_count);
    h->trace = nullptr;
    h->trace_count = nullptr;
    h->trace_cap = 0;
    if (max_records == 0) return 0;
    int rc = dev_alloc(h, &h->trace, 4LL * max_records);
    if (!rc) rc = dev_alloc(h, &h->trace_count, 1);
    if (rc) return rc;
    CUDA_TRY(cudaMemset(h->trace_count, 0, sizeof(int)));
    h->trace_cap = max_records;
    return 0;
}

extern "C" int mctsnc_read_slices(mctsnc_handle *h, int64_t *dst, int32_t max_records, int32_t *n_records) {
    if (!h || !n_records || (max_records > 0 && !dst)) return MCTSNC_E_BAD_ARGUMENT;
    *n_records = 0;
    if (!h->trace) return 0;
    int n = 0;
    CUDA_TRY(cudaMemcpy(&n, h->trace_count, sizeof(int), cudaMemcpyDeviceToHost));
    if (n > h->trace_cap) n = h->trace_cap;
    if (n > max_records) n = max_records;
    if (n > 0) CUDA_TRY(cudaMemcpy(dst, h->trace, sizeof(long long) * 4 * n, cudaMemcpyDeviceToHost));
    *n_records = n;
    return 0;
}

extern "C" const char *mctsnc_error_string(int code) {
    switch (code) {
    case 0: return "success";
    case MCTSNC_E_BAD_ARGUMENT: return "mctsnc: bad argument";
    case MCTSNC_E_UNSUPPORTED: return "mctsnc: game or shape not supported by this build";
    case MCTSNC_E_NO_MEMORY: return "mctsnc: out of memory";
    case MCTSNC_E_BAD_ROOT: return "mctsnc: root board and extra_info do not describe a reachable, unfinished position";
    case MCTSNC_E_CAPACITY: return "mctsnc: batch or step count beyond the capacity of the handle";
    case MCTSNC_E_NO_DEVICE: return "mctsnc: no CUDA device";
    default: break;
    }
    if (code > 0) return cudaGetErrorString((cudaError_t)code);
    return "mctsnc: unknown error";
}

// ===================================================================================================================
// mctsnc_search_c4_static: one Connect-4 search that allocates nothing.
//
// Every other entry point works on a handle whose pools come from cudaMalloc in mctsnc_create.  Some callers cannot do
// that: code that runs while a framework's caching allocator owns the whole device, services that forbid allocation
// after start-up so that a search can never fail for lack of memory, plug-ins that are handed a stream and two buffers
// and nothing else.  For them the tree pools, the random streams and the per-tree bookkeeping of this variant live in
// one file-scope device array of fixed size (every device that loads the library carries it until the process exits),
// so the limits below are modest.
//
// The array's name is only a host-side stand-in for the device object, not a device address: the first call on a device
// (with that device current) asks the runtime for the address with cudaGetSymbolAddress and every launch gets that
// pointer.  That first call also fills the cache of seeded streams; it synchronises, so it has to come before any
// stream capture.  All calls share the one array and it keeps what the last call left: what has to start from zero is
// cleared on the caller's stream at the start of every call, and two calls whose work overlaps on the GPU (different
// streams, different host threads) would race on it -- run them one after the other.  The host-side statics (address
// per device, stream cache, staging buffer) are guarded by a mutex.
namespace {
namespace fixed {

constexpr int MAX_TREES = MCTSNC_STATIC_MAX_TREES;
constexpr int MAX_PLAYOUTS = MCTSNC_STATIC_MAX_PLAYOUTS;
constexpr int MAX_STEPS = MCTSNC_STATIC_MAX_STEPS;
constexpr int A = c4::A;
constexpr long long CAP = (long long)MAX_STEPS * A + 1 + A;   // nodes per tree
constexpr int MAX_STREAMS = MAX_TREES * A * MAX_PLAYOUTS;
constexpr int MAX_DEVICES = 64;

struct Scratch {
    int4 rec[MAX_TREES * CAP];
    ulonglong2 board[MAX_TREES * CAP];
    ulonglong2 rng[MAX_STREAMS];
    ulonglong2 rng_base[MAX_STREAMS];
    ulonglong2 rng_expand[MAX_TREES];
    ulonglong2 rng_expand_base[MAX_TREES];
    ulonglong2 root_board[1];
    long long sums[3 * A];
    DevResult dres[1];
    TreeState state[MAX_TREES];
    int parent[MAX_TREES * CAP];
    int paths[MAX_TREES * PATH_CAP];
    int child_out[MAX_TREES * A * 2];
    short actions_expanded[MAX_TREES * (A + 2)];
    unsigned char flags[2 * A];
    signed char root_turn[16];
};

// the figure quoted in include/mctsnc_b200.h ("about 0.75 MB")
static_assert(sizeof(Scratch) > 700 * 1024 && sizeof(Scratch) < 800 * 1024, "update the size quoted in the header");

static __device__ __align__(256) unsigned char g_static_scratch[sizeof(Scratch)];

struct DeviceSetup {
    Scratch *ptr = nullptr;       // device address of g_static_scratch on this device
    bool streams_cached = false;  // rng_base / rng_expand_base hold the streams of the key below
    unsigned long long seed = 0;
    int n_trees = 0, n_playouts = 0, ocp = 0;
};
DeviceSetup g_setup[MAX_DEVICES];
ulonglong2 g_host_streams[MAX_STREAMS];   // staging for the seeded streams (static: no host allocation either)
std::mutex g_setup_mutex;                 // the two objects above are shared by all devices and all host threads

// the root arrives as kernel arguments (by value): no host memory is read after the call has returned
__global__ void set_root_kernel(ulonglong2 *root_board, signed char *root_turn, ulonglong2 root, int turn) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        root_board[0] = root;
        root_turn[0] = (signed char)turn;
    }
}

__global__ void copy_streams_kernel(ulonglong2 *dst, const ulonglong2 *src, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

// [root_ns | actions_ns | actions_ns_wins] are already in `out`; append best action, win flag, n, n_wins
__global__ void append_best_kernel(const DevResult *dres, long long *out, int A_) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        out[3 * A_ + 0] = dres->best_action;
        out[3 * A_ + 1] = dres->best_win_flag;
        out[3 * A_ + 2] = dres->best_n;
        out[3 * A_ + 3] = dres->best_n_wins;
    }
}

}  // namespace fixed
}  // namespace

extern "C" int mctsnc_search_c4_static(const int8_t *board, const int8_t *extra_info, int32_t turn, int32_t variant,
                                       int32_t n_trees, int32_t n_playouts, int64_t steps, float ucb_c, uint64_t seed,
                                       int64_t *out_device, void *stream) {
    using namespace fixed;
    if (!board || !out_device || (turn != 1 && turn != -1) || variant < 0 || variant > 3 || n_trees < 1 || n_playouts < 1 ||
        (n_playouts & (n_playouts - 1)) != 0 || steps < 0 || !(ucb_c >= 0.f))
        return MCTSNC_E_BAD_ARGUMENT;
    if (n_trees > MAX_TREES || n_playouts > MAX_PLAYOUTS || steps > MAX_STEPS) return MCTSNC_E_CAPACITY;
    int device = -1;
    CUDA_TRY(cudaGetDevice(&device));
    if (device < 0 || device >= MAX_DEVICES) return MCTSNC_E_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    ulonglong2 root;
    int rc = c4_encode_root(board, extra_info, &root);
    if (rc) return rc;
    // the set-up below touches host-side state shared by every device and thread: one caller at a time
    std::unique_lock<std::mutex> setup_lock(g_setup_mutex);
    DeviceSetup &su = g_setup[device];
    if (!su.ptr) {
        // once per device, with that device current: the device address behind the symbol
        void *p = nullptr;
        CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scratch));
        su.ptr = reinterpret_cast<Scratch *>(p);
        su.streams_cached = false;
    }
    Scratch *sc = su.ptr;
    const bool ocp = variant == MCTSNC_OCP_THRIFTY || variant == MCTSNC_OCP_PRODIGAL;
    const int per_tree = ocp ? n_playouts : A * n_playouts;
    const int n_streams = n_trees * per_tree;
    if (!su.streams_cached || su.seed != seed || su.n_trees != n_trees || su.n_playouts != n_playouts || su.ocp != (int)ocp) {
        // seeded streams of this configuration (numba's create_xoroshiro128p_states): computed on the host into a
        // static buffer and kept on the device for the calls to come
        su.streams_cached = false;
        CUDA_TRY(cudaStreamSynchronize(s));  // the staging buffer is reused: nothing may still be reading it
        make_streams(seed, 0, n_streams, 1, g_host_streams);
        CUDA_TRY(cudaMemcpyAsync(sc->rng_base, g_host_streams, sizeof(ulonglong2) * n_streams, cudaMemcpyHostToDevice, s));
        CUDA_TRY(cudaStreamSynchronize(s));
        if (ocp) {
            const int tpb_e1 = 64;  // Connect 4: min(max(pow2(42), pow2(7)), 512), src/mctsnc.py:360-365
            make_streams(seed, 0, n_trees, tpb_e1, g_host_streams);
            CUDA_TRY(cudaMemcpyAsync(sc->rng_expand_base, g_host_streams, sizeof(ulonglong2) * n_trees, cudaMemcpyHostToDevice, s));
            CUDA_TRY(cudaStreamSynchronize(s));
        }
        su.seed = seed;
        su.n_trees = n_trees;
        su.n_playouts = n_playouts;
        su.ocp = (int)ocp;
        su.streams_cached = true;
    }
    setup_lock.unlock();
    // what has to start from zero, and the root
    CUDA_TRY(cudaMemsetAsync(sc->state, 0, sizeof(sc->state), s));
    CUDA_TRY(cudaMemsetAsync(sc->child_out, 0, sizeof(sc->child_out), s));
    CUDA_TRY(cudaMemsetAsync(sc->actions_expanded, 0, sizeof(sc->actions_expanded), s));
    set_root_kernel<<<1, 32, 0, s>>>(sc->root_board, sc->root_turn, root, turn);
    copy_streams_kernel<<<32, 256, 0, s>>>(sc->rng, sc->rng_base, n_streams);
    if (ocp) copy_streams_kernel<<<1, 32, 0, s>>>(sc->rng_expand, sc->rng_expand_base, n_trees);
    SearchParams p;
    p.rec = sc->rec;
    p.board = sc->board;
    p.parent = sc->parent;
    p.state = sc->state;
    p.paths = sc->paths;
    p.actions_expanded = sc->actions_expanded;
    p.child_out = sc->child_out;
    p.rng_playout = sc->rng;
    p.rng_expand = sc->rng_expand;
    p.root_board = sc->root_board;
    p.root_turn = sc->root_turn;
    p.cap = CAP;
    p.node_limit = CAP;
    p.n_trees = n_trees;
    p.n_playouts = n_playouts;
    p.log2_playouts = 0;
    while ((1 << p.log2_playouts) < n_playouts) p.log2_playouts++;
    p.n_actions = A;
    p.variant = variant;
    p.steps = (int)steps;
    p.first = 1;
    p.ucb_c = ucb_c;
    p.queue = nullptr;
    p.ring = nullptr;
    p.remaining = nullptr;
    p.ring_cap = 0;
    p.chunk = 0;
    p.trace = nullptr;
    p.trace_count = nullptr;
    p.trace_cap = 0;
    p.ms_per_cycle = 0.f;
    p.cache_nodes = 0;
    p.n_trees_launched = p.places = n_trees;
    p.pool_trees = p.pool_walkers = 0;
    p.times2 = 2u;
    p.times4 = 4u;
    p.times2p23 = 1u << 23;
    const size_t dyn_smem = sizeof(ulonglong2) * (size_t)per_tree;   // <= 28 KB: below the 48 KB that need an opt-in
    // 256 threads and the kernel for more games than threads at every size
    if (ocp) c4::search_kernel<true, false><<<n_trees, 256, dyn_smem, s>>>(p);
    else c4::search_kernel<false, false><<<n_trees, 256, dyn_smem, s>>>(p);
    CUDA_TRY(cudaGetLastError());
    long long *out = reinterpret_cast<long long *>(out_device);
    reduce_over_trees_kernel<<<1, REDUCE_THREADS, 0, s>>>(sc->rec, sc->state, CAP, n_trees, A, out, sc->flags, sc->dres);
    const bool thrifty = variant == MCTSNC_OCP_THRIFTY || variant == MCTSNC_ACP_THRIFTY;
    reduce_over_actions_kernel<<<1, 8, 0, s>>>(out, sc->flags, A, 8, thrifty ? 1 : 0, sc->dres);
    append_best_kernel<<<1, 32, 0, s>>>(sc->dres, out, A);
    return (int)cudaGetLastError();
}
