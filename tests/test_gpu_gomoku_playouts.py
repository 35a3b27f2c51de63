"""The two ways a Gomoku search can run -- a block per tree (ocp, where all trees fit on the device) and two launches a step --
against the oracle, at the block sizes' edges, with more games than players, more trees than blocks, and from a position that
holds a line of five already (only lines through the last stone count, so the search goes on)."""
import numpy as np
import pytest

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
