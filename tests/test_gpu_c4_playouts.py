"""The ways the Connect-4 kernel can play a step's games -- a thread of its own for every game, several games per thread, a
cluster of blocks, with and without a warp kept for the walk -- against the oracle, where they can go wrong: games that fill
the board, steps without a game, one column left, block sizes that do not divide the games."""
import numpy as np
import pytest

from mcts_numba_cuda_b200 import MCTSNC
from oracle.oracle import OracleMCTSNC
from tests.test_gpu_parity_c4 import compare_trees

pytestmark = pytest.mark.gpu


def late_root(empty, seed):
    """A position without four in a row that has `empty` cells left, reached by legal play; (board, fills, turn)."""
    from mcts_numba_cuda_b200.roots import _c4_won
    rng = np.random.default_rng(seed)
    while True:
        board, fills, turn = np.zeros((6, 7), np.int8), np.zeros(7, np.int8), 1
        for _ in range(42 - empty):
            j = int(rng.choice(np.flatnonzero(fills < 6)))
            board[5 - fills[j], j] = turn
            fills[j] += 1
            if _c4_won(board, 6 - fills[j], j):
                break
            turn = -turn
        else:
            return board, fills, turn


@pytest.mark.parametrize("variant,n_playouts,threads,empty", [
    ("ocp_prodigal", 32, 0, 9), ("ocp_thrifty", 8, 32, 3), ("ocp_thrifty", 64, 64, 14), ("ocp_prodigal", 64, 32, 14),
    ("acp_prodigal", 8, 0, 5), ("acp_thrifty", 32, 224, 12), ("acp_prodigal", 32, 96, 12), ("acp_thrifty", 64, 0, 8),
    ("acp_prodigal", 256, 0, 20), ("acp_prodigal", 256, 320, 20), ("acp_thrifty", 1, 0, 30),
    ("acp_thrifty", 512, 0, 18), ("acp_prodigal", 256, 0, 2), ("acp_prodigal", 128, 0, 22)])
def test_late_positions_match_oracle_whatever_thread_plays_a_game(variant, n_playouts, threads, empty):
    steps, trees = 70, 2
    board, fills, turn = late_root(empty, seed=empty)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=trees, n_playouts=n_playouts, variant=variant,
                seed=5, verbose_info=False, threads_per_tree=threads)
    ai.init_device_side_arrays()
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=trees, n_playouts=n_playouts, variant=variant, seed=5, node_capacity=steps * 7 + 8)
    for _ in range(2):      # the streams run on: what a game left of its stream is what the next one starts from
        best = ai.run(board, fills, turn)
        orc.run(board, fills, turn, steps)
        compare_trees(ai, orc)
        assert int(best) == orc.best_action
        assert (ai._res["playouts"], ai._res["plies"]) == (orc.playouts, orc.plies)


@pytest.mark.parametrize("variant,n_trees,n_playouts,empty,steps", [
    ("ocp_thrifty", 1, 32, 20, 150), ("ocp_prodigal", 2, 256, 3, 60), ("ocp_prodigal", 1, 512, 30, 60), ("acp_prodigal", 2, 32, 12, 60),
    ("acp_thrifty", 1, 64, 42, 60), ("acp_prodigal", 3, 128, 9, 60), ("acp_prodigal", 9, 256, 16, 40), ("acp_thrifty", 1, 512, 42, 40)])
def test_draws_made_ahead_match_oracle(variant, n_trees, n_playouts, empty, steps):
    """A block or a cluster whose SMs are its own: the threads that play make the draws between the steps.  The streams have to stand
    where the games left them: the next search starts from there."""
    board, fills, turn = late_root(empty, seed=empty) if empty < 42 else (np.zeros((6, 7), np.int8), np.zeros(7, np.int8), 1)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=n_trees, n_playouts=n_playouts, variant=variant,
                seed=11, verbose_info=False)
    ai.init_device_side_arrays()
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=n_trees, n_playouts=n_playouts, variant=variant, seed=11, node_capacity=steps * 7 + 8)
    for _ in range(3):
        best = ai.run(board, fills, turn)
        orc.run(board, fills, turn, steps)
        compare_trees(ai, orc)
        assert int(best) == orc.best_action
        assert (ai._res["playouts"], ai._res["plies"]) == (orc.playouts, orc.plies)


@pytest.mark.parametrize("variant,n_trees,n_playouts,steps,kernel", [
    ("ocp_thrifty", 1, 32, 15, "search_kernel"), ("ocp_thrifty", 1, 32, 16, "search_kernel, draws ahead"),
    ("acp_prodigal", 4, 64, 15, "search_cluster_kernel, 8 blocks"), ("acp_prodigal", 4, 64, 16, "search_cluster_kernel, 8 blocks, draws ahead"),
    ("acp_thrifty", 2, 128, 40, "search_cluster_kernel, 8 blocks"), ("acp_prodigal", 12, 256, 16, "search_cluster_kernel, 8 blocks, draws ahead"),
    ("acp_prodigal", 2, 256, 15, "search_cluster_kernel, 16 blocks"), ("acp_thrifty", 2, 256, 16, "search_cluster_kernel, 16 blocks, draws ahead"),
    ("acp_prodigal", 1, 512, 63, "search_cluster_kernel, 16 blocks"), ("acp_prodigal", 1, 512, 64, "search_cluster_kernel, 16 blocks, draws ahead")])
def test_draws_are_made_ahead_only_where_they_pay(variant, n_trees, n_playouts, steps, kernel):
    """A launch of a few steps does not get back what the draws cost at its begin and end.  A long search, a short one and a long one on the
    streams that the one before has left."""
    board, fills, turn = late_root(30, seed=4)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=n_trees, n_playouts=n_playouts, variant=variant,
                seed=6, verbose_info=False)
    ai.init_device_side_arrays()
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=n_trees, n_playouts=n_playouts, variant=variant, seed=6, node_capacity=steps * 7 + 8)
    for count in (steps, 5, steps):
        best = ai.run(board, fills, turn, forced_search_steps_limit=count)
        assert ai.launch_geometry()["kernel"] == "c4::" + (kernel if count == steps else kernel.replace(", draws ahead", ""))
        orc.run(board, fills, turn, count)
        compare_trees(ai, orc)
        assert int(best) == orc.best_action and ai._res["plies"] == orc.plies
