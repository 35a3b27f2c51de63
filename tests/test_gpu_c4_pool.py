"""Connect-4 batches in which a block grows several trees and plays the games of all of them from one queue, against the oracle,
where that can go wrong: few and many games a step, all trees at once and through the work queue, one tree a block, more
entries than the queue has cells, positions about to end, full trees."""
import numpy as np
import pytest

from mcts_numba_cuda_b200 import MCTSNC, _abi
from mcts_numba_cuda_b200.roots import c4_random_roots
from oracle.oracle import OracleMCTSNC
from tests.test_gpu_c4_playouts import late_root
from tests.test_gpu_parity_c4 import compare_trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,n_trees,n_playouts,roots,steps,at_once", [
    ("ocp_prodigal", 3, 64, 50, 40, 2),         # 150 trees: two places on an SM, some of them empty
    ("ocp_thrifty", 8, 128, 40, 70, 3),
    ("ocp_prodigal", 8, 512, 100, 40, 4),       # work queue
    ("acp_thrifty", 4, 8, 128, 100, 4),         # 56 games a step: entries of eight games
    ("acp_prodigal", 6, 8, 560, 70, 21),        # 3360 trees, work queue: the walkers run far apart
    ("acp_thrifty", 4, 64, 150, 50, 3),
    ("acp_prodigal", 4, 256, 46, 40, 1),        # 184 trees take turns with a place on an SM
    ("acp_prodigal", 1, 512, 300, 34, 2),
])
def test_pooled_trees_match_the_oracle(variant, n_trees, n_playouts, roots, steps, at_once):
    boards, fills, turns = c4_random_roots(roots, 20, seed=roots)
    for b, empty in ((0, 2), (1, 7), (2, 12)):        # full boards, one column left, steps without a game
        boards[b], fills[b], turns[b] = late_root(empty, seed=empty)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=n_trees, n_playouts=n_playouts, variant=variant,
                seed=3, verbose_info=False, max_batch=roots)
    ai.init_device_side_arrays()
    outs = [ai.run_batch(boards, fills, turns, steps=steps, reseed=first) for first in (True, False)]   # the streams run on
    assert ai.launch_geometry()["blocks_per_sm"] == at_once
    assert (outs[1]["status"] & _abi.STATUS_INTERNAL == 0).all()
    for b in (0, 1, 2, roots // 2, roots - 1):
        orc = OracleMCTSNC((6, 7), 7, 7, n_trees=n_trees, n_playouts=n_playouts, variant=variant, seed=3, node_capacity=steps * 7 + 8)
        for out in outs:
            orc.run(boards[b], fills[b], int(turns[b]), steps)
            assert (out["playouts"][b], out["plies"][b], out["best_action"][b]) == (orc.playouts, orc.plies, orc.best_action)
        compare_trees(ai, orc, search=b)


@pytest.mark.parametrize("variant", MCTSNC.VARIANTS)
def test_pooled_trees_that_fill_up_equal_a_block_per_tree(variant):
    """A memory budget for about 150 nodes a tree (src/mctsnc.py:350-358): the leaf itself is played out from then on."""
    roots, n_trees, steps = 60, 5, 60
    boards, fills, turns = c4_random_roots(roots, 20, seed=1)
    outs, handles = [], []
    for threads in (0, 160):
        ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=n_trees, n_playouts=64, variant=variant, seed=3,
                    verbose_info=False, max_batch=roots, device_memory=n_trees * (8300 + 150 * 95) / 2 ** 30, threads_per_tree=threads)
        ai.init_device_side_arrays()
        assert 100 < ai.max_tree_size < 200
        outs.append(ai.run_batch(boards, fills, turns, steps=steps))
        handles.append(ai)
    assert handles[0].launch_geometry()["blocks_per_sm"] == 3       # trees of a block
    assert (outs[0]["status"] & _abi.STATUS_TREE_FULL).any()
    for name in ("playouts", "plies", "best_action", "actions_ns", "actions_ns_wins", "status", "max_size", "depth_sum"):
        assert np.array_equal(outs[0][name], outs[1][name]), name
    for b in (0, roots - 1):
        for name in ("trees_ns", "trees_ns_wins", "trees_playout_outcomes", "trees_actions_expanded"):
            assert np.array_equal(*(ai.export(name, b) for ai in handles)), name


def test_a_search_over_several_launches_equals_one():
    """A search of many trees under a time limit: its launches go on from what the one before has left."""
    kw = dict(n_trees=200, n_playouts=16, variant="acp_prodigal", seed=4, verbose_info=False)
    board, fills = np.zeros((6, 7), np.int8), np.zeros(7, np.int8)
    timed = MCTSNC((6, 7), 7, 7, search_time_limit=0.03, search_steps_limit=np.inf, **kw)
    timed.init_device_side_arrays()
    best = timed.run(board, fills, 1)
    assert timed.steps > 70 and timed.launch_geometry()["blocks_per_sm"] == 2        # launches of 2 ms, trees of a block
    whole = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=float(timed.steps), **kw)
    whole.init_device_side_arrays()
    assert best == whole.run(board, fills, 1)
    for name in ("playouts", "plies", "total_nodes", "depth_sum"):
        assert timed._res[name] == whole._res[name], name
    sizes = timed.export("trees_sizes")
    assert np.array_equal(sizes, whole.export("trees_sizes"))
    for name in ("trees_ns", "trees_ns_wins"):
        assert np.array_equal(timed.export(name, max_nodes=int(sizes.max())), whole.export(name, max_nodes=int(sizes.max()))), name


@pytest.mark.parametrize("empty,seed", [(11, 84), (13, 37)])
def test_pooled_trees_outlast_a_million_steps_without_a_game(empty, seed):
    """The mover wins at once: from some step before 2000 to one after 1500000 every step selects the won child, and no game is played;
    then there are games again.  The players of a block wait that long, for seconds."""
    steps, roots = 1_700_000, 200
    board, fills, turn = late_root(empty, seed)
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=1, n_playouts=64, variant="ocp_prodigal", seed=3, node_capacity=20000)
    orc.run(board, fills, turn, 2000)
    early = orc.plies
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=1, n_playouts=64, variant="ocp_prodigal", seed=3, node_capacity=20000)
    orc.run(board, fills, turn, 1_500_000)
    assert orc.plies == early
    orc = OracleMCTSNC((6, 7), 7, 7, n_trees=1, n_playouts=64, variant="ocp_prodigal", seed=3, node_capacity=20000)
    orc.run(board, fills, turn, steps)
    assert orc.plies > early
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=1, n_playouts=64, variant="ocp_prodigal", seed=3,
                verbose_info=False, max_batch=roots, device_memory=2e6 / 2 ** 30)      # far more nodes than the tree comes to
    ai.init_device_side_arrays()
    out = ai.run_batch(np.stack([board] * roots), np.stack([fills] * roots), np.full(roots, turn), steps=steps)
    assert ai.launch_geometry()["blocks_per_sm"] == 2      # trees of a block
    assert (out["status"] == 0).all()
    assert (out["playouts"] == orc.playouts).all() and (out["plies"] == orc.plies).all()
    for b in (0, roots - 1):
        compare_trees(ai, orc, search=b)


@pytest.mark.parametrize("n_playouts,roots,steps,at_once", [(256, 227, 2000, 4), (256, 256, 600, 4), (256, 256, 700, 5), (256, 384, 100, 4),
                                                            (256, 384, 300, 5), (128, 338, 1000, 6), (128, 384, 500, 7), (128, 384, 200, 6), (512, 256, 500, 3)])
def test_a_tree_more_on_an_sm_only_where_many_wait_for_long(n_playouts, roots, steps, at_once):
    boards, fills, turns = c4_random_roots(roots, 20, seed=3)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=4, n_playouts=n_playouts, variant="acp_prodigal", seed=5,
                verbose_info=False, max_batch=roots)
    ai.init_device_side_arrays()
    out = ai.run_batch(boards, fills, turns, steps=steps)
    assert ai.launch_geometry()["blocks_per_sm"] == at_once
    assert (out["status"] & _abi.STATUS_INTERNAL == 0).all() and (out["steps"] == steps).all()
    assert (out["root_ns"][:, :7].sum(axis=1) > 0).all()


@pytest.mark.parametrize("n_playouts,roots,steps,kernel", [(128, 250, 36, "c4::search_kernel"), (128, 250, 60, "c4::pool_kernel"),
                                                           (128, 210, 33, "c4::pool_kernel"), (128, 290, 33, "c4::pool_kernel"),
                                                           (256, 250, 39, "c4::search_kernel"), (256, 250, 40, "c4::pool_kernel")])
def test_few_steps_of_trees_in_turns_have_a_block_per_tree(n_playouts, roots, steps, kernel):
    boards, fills, turns = c4_random_roots(roots, 20, seed=4)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, n_trees=1, n_playouts=n_playouts, variant="acp_prodigal", seed=5,
                verbose_info=False, max_batch=roots)
    ai.init_device_side_arrays()
    out = ai.run_batch(boards, fills, turns, steps=steps)
    assert ai.launch_geometry()["kernel"] == kernel and (out["status"] & _abi.STATUS_INTERNAL == 0).all()
    for b in (0, roots - 1):
        orc = OracleMCTSNC((6, 7), 7, 7, n_trees=1, n_playouts=n_playouts, variant="acp_prodigal", seed=5, node_capacity=steps * 7 + 8)
        orc.run(boards[b], fills[b], int(turns[b]), steps)
        assert (out["playouts"][b], out["plies"][b], out["best_action"][b]) == (orc.playouts, orc.plies, orc.best_action)
        compare_trees(ai, orc, search=b)


def test_draws_of_one_in_pooled_trees_are_replayed_like_the_oracle():
    """Games that meet a uniform draw of exactly 1.0f, with either side to move first, found in a block of several trees."""
    roots, steps, kw = 100, 40, dict(n_trees=4, n_playouts=256, variant="acp_prodigal", seed=7)
    boards, fills, turns = c4_random_roots(roots, 20, seed=1)
    ai = MCTSNC((6, 7), 7, 7, search_time_limit=np.inf, search_steps_limit=steps, verbose_info=False, max_batch=roots, **kw)
    ai.init_device_side_arrays()
    out = ai.run_batch(boards, fills, turns, steps=steps)
    assert ai.launch_geometry()["kernel"] == "c4::pool_kernel" and ai.launch_geometry()["blocks_per_sm"] == 2
    for b, ub in ((0, 1), (20, 1), (40, 1), (10, 0)):       # the first mover of the game is -1, +1, -1
        orc = OracleMCTSNC((6, 7), 7, 7, node_capacity=steps * 7 + 8, **kw)
        orc.run(boards[b], fills[b], int(turns[b]), steps)
        assert orc.ub_draws == ub == out["ub_draws"][b]
        assert bool(out["status"][b] & _abi.STATUS_UB_DRAW) == bool(ub) and out["status"][b] & _abi.STATUS_INTERNAL == 0
        assert (out["playouts"][b], out["plies"][b], out["best_action"][b]) == (orc.playouts, orc.plies, orc.best_action)
        compare_trees(ai, orc, search=b)
