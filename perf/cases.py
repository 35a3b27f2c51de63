"""Workloads of the framework as its users call it: one search per move, searches of many roots in one call, and the
select / backup waves of the PUCT and DUCT trees, over the range of sizes from the smallest calls to the benchmark's own.

A case is a dict of plain values with the key ``kind``:

* ``move``   ``MCTSNC.run``: a player searches one position (keys ``game, variant, trees, playouts, steps, plies``);
* ``batch``  ``MCTSNC.run_batch``: ``roots`` positions in one call, the form of self-play and of position analysis;
* ``puct``   ``puct.launch_select`` and ``puct.launch_backup`` (statistics per edge);
* ``puct_v2``  ``puct.launch_select_v2`` and ``puct.launch_backup_v2`` (virtual visits per node, ``variant`` 0 or 1);
* ``duct``   ``duct.launch_select`` and ``duct.launch_backup`` (two players, ``edges`` actions each).

A search gives a program its statistics at the root; its trees stay in the searcher, and their sizes, depths and the counts of
playouts and plies stand for them here (every one of them changes with any change of a tree).
"""
import math

import numpy as np
import torch

from mcts_numba_cuda_b200 import MCTSNC, duct, puct
from mcts_numba_cuda_b200.roots import c4_random_roots, gomoku_random_roots

# board shape, bytes of extra information, actions, device_memory (GiB) of the reference's configurations, mean plies of a
# random game, integer operations of one ply (generator step, choice and placement of the move, line test)
GAMES = {"c4": ((6, 7), 7, 7, 2.0, 15, 65), "gomoku": ((15, 15), 0, 225, 16.0, 82, 100)}
VARIANTS = ("ocp_thrifty", "ocp_prodigal", "acp_thrifty", "acp_prodigal")


def _search(kind, game, variant, trees, playouts, steps, plies, roots=1):
    return {"kind": kind, "game": game, "variant": variant, "trees": trees, "playouts": playouts, "steps": steps, "plies": plies,
            "roots": roots}


def _wave(kind, trees, edges, depth, warps, virtual_loss, variant=0):
    return {"kind": kind, "trees": trees, "edges": edges, "depth": depth, "warps": warps, "virtual_loss": virtual_loss,
            "variant": variant}


def _named(name, case):
    return dict(case, name=name)


def listed():
    return [
        # a quick move of a weak player: the smallest search of the benchmark's configurations, latency of the whole call counts
        _named("c4 move small", _search("move", "c4", "ocp_thrifty", 1, 32, 200, 4)),
        # a move of a full-strength player
        _named("c4 move", _search("move", "c4", "acp_prodigal", 4, 256, 2000, 4)),
        # a few dozen positions looked at briefly
        _named("c4 batch small", _search("batch", "c4", "ocp_thrifty", 1, 32, 200, 10, roots=64)),
        # the headline configuration: 256 positions searched in full
        _named("c4 batch acp", _search("batch", "c4", "acp_prodigal", 4, 256, 2000, 20, roots=256)),
        # the same number of positions with one child played out per step
        _named("c4 batch ocp", _search("batch", "c4", "ocp_prodigal", 8, 128, 1000, 20, roots=256)),
        # Gomoku moves: one child played out per step, and all of them (the benchmark's configuration)
        _named("gomoku move ocp", _search("move", "gomoku", "ocp_prodigal", 8, 128, 300, 30)),
        _named("gomoku move acp", _search("move", "gomoku", "acp_prodigal", 4, 256, 500, 30)),
        # eight Gomoku positions in one call
        _named("gomoku batch acp", _search("batch", "gomoku", "acp_prodigal", 4, 256, 200, 30, roots=8)),
        # a wave of selects over many trees, eight traversals a tree, and its backup: the benchmark's configuration
        _named("puct wave", _wave("puct", 4096, 64, 16, 8, 3)),
        # few trees with few, oddly many edges, one traversal each: a game server with some games in progress
        _named("puct small", _wave("puct", 100, 19, 12, 1, 1)),
        # the older layout with visits per node, preclaim variant, one traversal a tree
        _named("puct v2", _wave("puct_v2", 1000, 82, 9, 1, 1)),
        # simultaneous moves, two players of eight actions: the benchmark's configuration
        _named("duct wave", _wave("duct", 4096, 8, 16, 8, 3)),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


MOST_OPS = {"c4": 256 * 4 * 2000 * 7 * 256 * 15 * 65, "gomoku": 8 * 4 * 200 * 225 * 256 * 82 * 100}   # of the listed batches
MOST_WAVE_BYTES = 6 << 30


def draw(rng):
    while True:
        kind = rng.choice(("move", "move", "batch", "batch", "puct", "puct_v2", "duct"))
        if kind in ("move", "batch"):
            game = rng.choice(("c4", "c4", "gomoku"))
            roots = 1 if kind == "move" else _log_int(rng, 2, 256 if game == "c4" else 32)
            case = _search(kind, game, rng.choice(VARIANTS), rng.randint(1, 8), 2 ** rng.randint(5, 8),
                           _log_int(rng, 50, 2000 if game == "c4" else 500), rng.randint(0, 20 if game == "c4" else 30), roots)
            if work(case)["flops"] <= MOST_OPS[game]:
                return case
            continue
        if kind == "duct":
            case = _wave(kind, _log_int(rng, 16, 4096), rng.randint(2, 16), rng.randint(4, 16), rng.choice((1, 1, 2, 4, 8)),
                         rng.randint(1, 3))
        else:
            case = _wave(kind, _log_int(rng, 16, 4096), _log_int(rng, 4, 256), rng.randint(4, 16), rng.choice((1, 1, 2, 4, 8)), 1,
                         rng.randint(0, 1) if kind == "puct_v2" else 0)
            if kind == "puct":
                case["virtual_loss"] = rng.choice((1, 1, 3))
        if _wave_bytes(case) <= MOST_WAVE_BYTES:
            return case


def _nodes(case):
    width = case["edges"] ** 2 if case["kind"] == "duct" else case["edges"]
    return 1 + width * case["depth"]


def _node_bytes(case):
    a = case["edges"]
    return 4 * a * a + 2 * a * 16 + 4 if case["kind"] == "duct" else 20 * a + 8


def _wave_bytes(case):
    return case["trees"] * _nodes(case) * _node_bytes(case)


# ------------------------------------------------------------------------------------------------------ inputs and state
def _searcher(case, seed):
    shape, extra, actions, memory, _, _ = GAMES[case["game"]]
    ai = MCTSNC(shape, extra, actions, search_time_limit=np.inf, search_steps_limit=float(case["steps"]), n_trees=case["trees"],
                n_playouts=case["playouts"], variant=case["variant"], device_memory=memory, ucb_c=2.0, seed=seed, verbose_info=False,
                max_batch=case["roots"])
    ai.init_device_side_arrays()
    return ai


def _layers(width, depth, device):
    """Level and index within its level of every node of a layered tree: a root and `depth` levels of `width` nodes."""
    i = torch.arange(width * depth, device=device)
    level = torch.cat([torch.zeros(1, dtype=torch.long, device=device), i // width + 1])
    index = torch.cat([torch.zeros(1, dtype=torch.long, device=device), i % width])
    return level, index


def _dirichlet(shape, g, device):
    """Priors of a policy head at self-play noise: Dirichlet(0.3) over the last axis."""
    x = torch._standard_gamma(torch.full(shape, 0.3, device=device), generator=g)
    return x.div_(x.sum(dim=-1, keepdim=True).clamp_min(1e-30))


def _puct_trees(case, g, device):
    """Trees in mid-search: the nodes of a level share the nodes of the next as children, the last level is terminal; between
    half and all of a node's edges are expanded, with 0..49 visits each and values in [-1, 1]."""
    trees, edges, depth, warps, nodes = case["trees"], case["edges"], case["depth"], case["warps"], _nodes(case)
    level, index = _layers(edges, depth, device)
    child = 1 + edges * level[:, None] + (torch.arange(edges, device=device)[None, :] + index[:, None]) % edges
    child[level == depth] = -1
    expanded = torch.randint(max(1, edges // 2), edges + 1, (trees, nodes), device=device, generator=g, dtype=torch.int32)
    expanded[:, level == depth] = -1
    n = torch.randint(0, 50, (trees, nodes, edges), device=device, generator=g, dtype=torch.int32)
    w = torch.rand((trees, nodes, edges), device=device, generator=g).mul_(2).sub_(1).mul_(n)
    d = {"edge_child": child.to(torch.int32)[None].expand(trees, -1, -1).contiguous(),
         "edge_prior": _dirichlet((trees, nodes, edges), g, device), "edge_w": w, "edge_n": n,
         "node_expand_inflight": torch.zeros((trees, nodes), dtype=torch.int32, device=device), "node_expanded": expanded,
         "node_count": torch.full((trees,), nodes, dtype=torch.int32, device=device)}
    if case["kind"] == "puct":
        d["edge_inflight"] = torch.zeros((trees, nodes, edges), dtype=torch.int32, device=device)
    else:
        d["node_inflight"] = torch.zeros((trees, nodes), dtype=torch.int32, device=device)
    return d


def _duct_trees(case, g, device):
    """The same for two players of A actions: a child per joint action, the players' marginal statistics summed from joint
    counts 0..49 and values in [-1, 1] (player 1's are the negatives)."""
    trees, A, depth, nodes = case["trees"], case["edges"], case["depth"], _nodes(case)
    level, index = _layers(A * A, depth, device)
    child = 1 + A * A * level[:, None] + (torch.arange(A * A, device=device)[None, :] + index[:, None]) % (A * A)
    child[level == depth] = -1
    nj = torch.randint(0, 50, (trees, nodes, A, A), device=device, generator=g, dtype=torch.int32)
    wj = torch.rand((trees, nodes, A, A), device=device, generator=g).mul_(2).sub_(1).mul_(nj)
    return {"child": child.to(torch.int32)[None].expand(trees, -1, -1).contiguous(),
            "node_prior": _dirichlet((trees, nodes, 2, A), g, device),
            "node_w": torch.stack([wj.sum(dim=3), -wj.sum(dim=2)], dim=2),
            "node_n": torch.stack([nj.sum(dim=3), nj.sum(dim=2)], dim=2).to(torch.int32),
            "node_inflight": torch.zeros((trees, nodes, 2, A), dtype=torch.int32, device=device),
            "node_terminal": (level == depth).to(torch.int32)[None].expand(trees, -1).contiguous(),
            "node_count": torch.full((trees,), nodes, dtype=torch.int32, device=device)}


def prepare(case, seed):
    """Searches: an initialised searcher and seeded positions (host arrays, as a game program holds them).  Waves: the trees
    on the device and the values a network would have returned."""
    state = {"case": case}
    if case["kind"] in ("move", "batch"):
        if case["game"] == "c4":
            state["boards"], state["extras"], state["turns"] = c4_random_roots(case["roots"], case["plies"], seed)
        else:
            state["boards"], state["turns"] = gomoku_random_roots(case["roots"], case["plies"], seed)
            state["extras"] = None
        state["ai"] = _searcher(case, seed)
        return state
    device = "cuda"
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    trees, depth, warps = case["trees"], case["depth"], case["warps"]
    d = _duct_trees(case, g, device) if case["kind"] == "duct" else _puct_trees(case, g, device)
    d.update(trees=trees, warps=warps, out_selected=torch.zeros((trees, warps), dtype=torch.int32, device=device),
             out_path=torch.full((trees, warps, depth), -1, dtype=torch.int32, device=device),
             out_len=torch.zeros((trees, warps), dtype=torch.int32, device=device))
    state["d"] = d
    state["values"] = torch.rand((trees, warps, depth), device=device, generator=g).mul_(2).sub_(1)
    return state


# ------------------------------------------------------------------------------------------------------------ one pass
def _run_move(state):
    ai, extras = state["ai"], state["extras"]
    best = ai.run(state["boards"][0], None if extras is None else extras[0], int(state["turns"][0]))
    info, trees = ai.actions_info, ai.performance_info["trees"]
    rows = [info.get(a) for a in range(ai.state_max_actions)]   # by action; None: not expanded at the root
    return {"best": [int(best), int(ai.best_win_flag), int(ai.best_n), int(ai.best_n_wins), int(ai.steps)], "best_q": float(ai.best_q),
            "actions": np.array([[r["n_root"], r["win_flag"], r["n"], r["n_wins"]] if r else [-1] * 4 for r in rows]),
            "q": np.array([r["q"] if r else np.nan for r in rows]), "ucb": np.array([r["ucb"] if r else np.nan for r in rows]),
            "playouts": int(ai.performance_info["playouts"]), "trees": [trees["max_depth"], trees["max_size"]],
            "mean_depth": trees["mean_depth"], "mean_size": trees["mean_size"]}


def _run_batch(state):
    case = state["case"]
    r = state["ai"].run_batch(state["boards"], state["extras"], state["turns"], steps=case["steps"])
    out = {k: r[k] for k in ("best_action", "best_win_flag", "best_n", "best_n_wins", "steps", "playouts", "plies", "max_depth",
                             "total_nodes", "depth_sum", "max_size")}
    actions = GAMES[case["game"]][2]
    for k in ("root_ns", "actions_ns", "actions_ns_wins", "actions_win_flags", "actions_expanded"):
        out[k] = r[k][:, :actions]
    return out


def _run_wave(state):
    case, d, vl = state["case"], state["d"], state["case"]["virtual_loss"]
    if case["kind"] == "puct":
        puct.launch_select(d, cpuct=1.5, c_pw=0.0, virtual_loss=vl)
        puct.launch_backup(d, state["values"], virtual_loss=vl)
        updated = ("edge_n", "edge_w", "edge_inflight", "node_expand_inflight")
    elif case["kind"] == "puct_v2":
        puct.launch_select_v2(d, cpuct=1.5, c_pw=0.0, variant=case["variant"])
        puct.launch_backup_v2(d, state["values"], virtual_loss=vl)
        updated = ("edge_n", "edge_w", "node_inflight", "node_expand_inflight")
    else:
        duct.launch_select(d, cpuct=1.5, virtual_loss=vl)
        duct.launch_backup(d, state["values"], virtual_loss=vl)
        updated = ("node_n", "node_w", "node_inflight", "child")
    # With several traversals in a tree the winners of the claims depend on the schedule, and with them which traversal
    # holds which path: the statistics are what a program goes on with.
    if case["warps"] == 1:
        updated += ("out_selected", "out_path", "out_len")
    return {k: d[k] for k in updated}


def run(state):
    return {"move": _run_move, "batch": _run_batch}.get(state["case"]["kind"], _run_wave)(state)


# --------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Searches: the integer operations of the random games (estimated with the mean length of a game) and the nodes written
    once.  Waves: the edges of every node that one traversal of a tree meets, read once, and the statistics of its path."""
    if case["kind"] in ("move", "batch"):
        _, _, actions, _, plies, ops = GAMES[case["game"]]
        tree_steps = case["roots"] * case["trees"] * case["steps"]
        games = tree_steps * case["playouts"] * (actions if case["variant"].startswith("acp") else 1)
        node = 36 if case["game"] == "c4" else 84
        return {"bytes": tree_steps * actions * node, "flops": games * plies * ops}
    per_level = _node_bytes(case) - (20 if case["kind"] == "duct" else 4) + 24
    return {"bytes": case["trees"] * case["depth"] * per_level, "flops": case["trees"] * case["depth"] * case["edges"] * 10}


def tolerance(case):
    if case["kind"] in ("move", "batch"):
        return {"rel": 1e-12}   # whole numbers are exact; q and ucb are float64 of them
    if case["warps"] == 1:
        return "exact"          # one traversal a tree: nothing depends on the schedule
    # several: which of the traversals started together wins a claim does; their paths are all that may differ
    return {"rel": 0.01, "max": 0.5, "differ": 0.01}
