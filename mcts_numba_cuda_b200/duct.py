"""Host side of the decoupled-UCT (DUCT) select for simultaneous-move games (``csrc/duct_select.cu``,
``include/duct_b200.h``).  The reference has no such component; the interface follows the one of the PUCT select
(``puct.py``): a dict of device arrays and two launches.

``d`` holds ``child`` int32[trees, nodes, A*A], ``node_prior`` / ``node_w`` float32[trees, nodes, 2, A], ``node_n`` /
``node_inflight`` int32[trees, nodes, 2, A], ``node_terminal`` int32[trees, nodes], ``node_count`` int32[trees],
``out_selected`` / ``out_len`` int32[trees, warps], ``out_path`` int32[trees, warps, path_depth] and the ints ``trees``,
``warps`` — torch CUDA tensors or anything with ``__cuda_array_interface__``.
"""
from . import puct

KIND_INVALID, KIND_EXPAND, KIND_TERMINAL, KIND_DEPTH_LIMIT, KIND_BUSY = 0, 1, 2, 3, 4


def decode(selected):
    """(kind, node, joint action, reason) of packed results (array or int)."""
    return (selected >> 22) & 7, selected & 0x3FFF, (selected >> 14) & 0xFF, (selected >> 25) & 0x3F


def launch_select(d, cpuct=1.5, virtual_loss=1, stream=None):
    """One traversal per (tree, warp); results in ``d["out_selected"], d["out_path"], d["out_len"]``."""
    code = (puct._wave or puct._launcher()).duct_select(d, cpuct, int(virtual_loss), puct._stream(stream))
    puct._check(code, "select", "DUCT")


def launch_backup(d, values=None, new_child=None, virtual_loss=1, stream=None):
    """Returns the claims of the last select; with ``values`` (float32[trees, warps, path_depth], player 0's point of
    view) also updates counts and value sums; ``new_child`` (int32[trees, warps]) installs the expanded children."""
    code = (puct._wave or puct._launcher()).duct_backup(d, values, new_child, int(virtual_loss), puct._stream(stream))
    puct._check(code, "backup", "DUCT")
