"""The two ways a Gomoku search can run -- a block per tree (ocp, where all trees fit on the device) and two launches a step --
against the oracle, at the block sizes' edges, with more games than players, more trees than blocks, and from a position that
holds a line of five already (only lines through the last stone count, so the search goes on)."""
import numpy as np
import pytest

from mcts_numba_cuda_b200 import MCTSNC, _abi
from oracle.oracle import OracleMCTSNC
from tests.test_gpu_parity_gomoku import compare, make_pair

pytestmark = pytest.mark.gpu


def spread_root(seed, stones=20):
    rng = np.random.default_rng(seed)
    board = np.zeros(225, np.int8)
    board[rng.choice(225, size=stones, replace=False)] = np.where(np.arange(stones) % 2 == 0, 1, -1)
    return board.reshape(15, 15)


@pytest.mark.parametrize("variant,n_trees,n_playouts,steps", [
    ("ocp_thrifty", 1, 1, 40), ("ocp_prodigal", 2, 32, 40), ("ocp_thrifty", 2, 64, 30), ("ocp_prodigal", 3, 128, 30),
    ("ocp_thrifty", 1, 256, 20), ("ocp_prodigal", 1, 512, 20), ("acp_thrifty", 1, 1, 12), ("acp_prodigal", 9, 8, 5)])
def test_every_block_size_matches_oracle(variant, n_trees, n_playouts, steps):
    ai, orc = make_pair(variant, n_trees, n_playouts, steps, seed=3)
    board = spread_root(n_playouts)
    for _ in range(2):      # the streams run on
        best = ai.run(board, None, 1)
        orc.run(board, None, 1, steps)
        compare(ai, orc)
        assert int(best) == orc.best_action and ai._res["plies"] == orc.plies


def test_more_trees_than_blocks_fit():
    steps, roots = 4, 40    # 320 trees of 256 playouts: one block of 288 threads on an SM
    ai, _ = make_pair("ocp_prodigal", 8, 256, steps, seed=2, max_batch=roots)
    boards = np.stack([spread_root(100 + b) for b in range(roots)])
    out = ai.run_batch(boards, None, np.ones(roots, np.int8), steps=steps, reseed=True)
    assert (out["status"] & 4 == 0).all()
    for b in (0, 23, 39):
        orc = OracleMCTSNC((15, 15), 0, 225, n_trees=8, n_playouts=256, variant="ocp_prodigal", device_memory=16.0, seed=2,
                           node_capacity=steps * 225 + 230)
        orc.run(boards[b], None, 1, steps)
        compare(ai, orc, search=b)
        assert out["plies"][b] == orc.plies


@pytest.mark.parametrize("variant", ["ocp_prodigal", "acp_prodigal"])
def test_a_line_of_five_on_the_root_is_not_a_win_of_later_stones(variant):
    board = np.zeros((15, 15), np.int8)
    board[3, 4:9] = 1       # a row of five
    board[6:11, 12] = -1    # a column of five
    board[12, 1:6] = 1
    for turn in (1, -1):
        ai, orc = make_pair(variant, 1, 32, 6, seed=4)
        best = ai.run(board, None, turn)
        orc.run(board, None, turn, 6)
        compare(ai, orc)
        assert int(best) == orc.best_action and ai._res["plies"] == orc.plies


@pytest.mark.parametrize("seed,stones", [(10, 0), (7, 20), (12, 20)])
def test_a_draw_of_one_is_replayed_like_the_oracle(seed, stones):
    steps = 6
    ai, orc = make_pair("acp_prodigal", 1, 64, steps, seed=seed)
    board = spread_root(7, stones)
    best = ai.run(board, None, 1)
    orc.run(board, None, 1, steps)
    compare(ai, orc)
    assert orc.ub_draws > 0 and ai._res["ub_draws"] == orc.ub_draws
    assert int(best) == orc.best_action and ai._res["plies"] == orc.plies


@pytest.mark.parametrize("variant,n_trees,n_playouts", [("ocp_prodigal", 3, 32), ("acp_thrifty", 1, 8), ("acp_prodigal", 9, 2)])
def test_a_search_over_several_launches_equals_one_of_as_many_steps(variant, n_trees, n_playouts):
    """With a time limit a search is cut into launches, the first of 16 steps: a block per tree, one launch a step, and groups of one
    and of two trees."""
    steps = 40
    ai = MCTSNC((15, 15), 0, 225, search_time_limit=1000.0, search_steps_limit=steps, n_trees=n_trees, n_playouts=n_playouts,
                variant=variant, device_memory=16.0, seed=5, verbose_info=False)
    ai.init_device_side_arrays()
    orc = OracleMCTSNC((15, 15), 0, 225, n_trees=n_trees, n_playouts=n_playouts, variant=variant, device_memory=16.0, seed=5,
                       node_capacity=steps * 225 + 230)
    board = spread_root(8)
    for _ in range(2):
        best = ai.run(board, None, 1)
        orc.run(board, None, 1, steps)
        assert ai.steps == steps
        compare(ai, orc)
        assert int(best) == orc.best_action and ai._res["plies"] == orc.plies


@pytest.mark.parametrize("variant", MCTSNC.VARIANTS)
def test_a_full_tree_stops_growing_and_is_played_on(variant):
    """Trees of at most 300 nodes: the second expansion has room for a part of the children (as the oracle has it); from then on the
    selected leaf itself is played out."""
    T, P, limit = 2, 16, 300
    per_tree = 4 + 4 + 2 * 227 + 8 + 4 * 2050 + (4 * 225 * 2 if "acp" in variant else 0)    # src/mctsnc.py:350-358
    per_state = 225 + 1 + 4 * 226 + 14
    memory = T * (per_tree + limit * per_state) / 2 ** 30
    board = spread_root(9)                                                                   # 20 stones
    played = {}
    for steps in (2, 12):
        ai = MCTSNC((15, 15), 0, 225, search_time_limit=np.inf, search_steps_limit=steps, n_trees=T, n_playouts=P, variant=variant,
                    device_memory=memory, seed=6, verbose_info=False)
        ai.init_device_side_arrays()
        assert ai.max_tree_size == limit
        ai.run(board, None, 1)
        assert ai.status == _abi.STATUS_TREE_FULL and (ai.export("trees_sizes") == limit).all()
        if steps == 2:
            orc = OracleMCTSNC((15, 15), 0, 225, n_trees=T, n_playouts=P, variant=variant, device_memory=memory, seed=6, node_capacity=limit)
            orc.run(board, None, 1, steps)
            assert orc.tree_full_events > 0
            compare(ai, orc)
            assert ai._res["plies"] == orc.plies
        ns, wins = ai.export("trees_ns").astype(np.int64), ai.export("trees_ns_wins").astype(np.int64)
        children = ai.export("trees")[:, :, 1:]
        for t in range(T):
            for node in (0, ai.export("trees")[t, -1, 0]):         # the root and the node that was expanded in part
                c = children[t, node][children[t, node] >= 0]
                alone = 0 if node == 0 else (P if "acp" in variant else ns[t, node] - ns[t, c].sum())
                assert alone in (0, P) and ns[t, node] == alone + ns[t, c].sum()
            assert ((wins[t] >= 0) & (wins[t] <= ns[t])).all()
        played[steps] = ns[:, 0]
        assert ai._res["playouts"] == ns[:, 0].sum()
    assert (played[12] == played[2] + 10 * P).all()
