"""Host side of the warp-level PUCT select: the same ``launch_select(d, cpuct, c_pw, alpha_pw, soft_winner)`` call on a
dict of device arrays that the reference's ``src/puct/puct_gpu_v3_cpp.py:118-156`` offers, bound to the sm_100a kernels
in ``libmctsnc_b200.so`` (``csrc/puct_select.cu``), plus the backup / release step.

``d`` maps the names the reference's tests use (``edge_child, edge_prior, edge_w, edge_n, edge_inflight,
node_expand_inflight, node_expanded, node_count, out_selected, out_path, out_len`` and the ints ``trees``, ``warps``) to
arrays that live on the device: torch CUDA tensors, or anything with ``__cuda_array_interface__`` (numba / cupy arrays).
"""
import ctypes

from . import _abi

_wave = None


def _launcher():
    """The extension that gathers a launch's arguments, bound to the library's launchers on first use."""
    global _wave
    if _wave is None:
        try:
            from . import _wave as module
        except ImportError as e:
            raise RuntimeError("the extension mcts_numba_cuda_b200/_wave is missing: build it with `python -m mcts_numba_cuda_b200.build`") from e
        L = _abi.lib()
        module.bind(*(ctypes.cast(getattr(L, name), ctypes.c_void_p).value for name in (
            "puct_select_winner_recalc_launch", "puct_select_virtual_loss_launch", "puct_backup_launch", "puct_v2_select_launch",
            "puct_v2_backup_launch", "duct_select_launch", "duct_backup_launch")))
        _wave = module
    return _wave


_raw_stream = _device_index = None


def _current_stream():
    """Handle of torch's current stream; 0 (the default stream) where torch or a device is missing."""
    global _raw_stream, _device_index
    try:
        if _raw_stream is not None:   # without building a Stream object (0.1 instead of 1.2 us)
            return _raw_stream(_device_index())
        import torch
        handle = torch.cuda.current_stream().cuda_stream
        _device_index = getattr(torch._C, "_cuda_getDevice", None)
        _raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) if _device_index else None
        return handle
    except Exception:
        return 0


def _stream(stream):
    return _current_stream() if stream is None else stream


def _check(code, what, name="PUCT"):
    if code != 0:
        text = _abi.lib().puct_cpp_cuda_error_string
        text.argtypes, text.restype = [ctypes.c_int], ctypes.c_char_p
        raise RuntimeError(f"{name} {what} launch failed: {text(code).decode('utf-8', 'replace')} ({code})")


def launch_select(d, cpuct=1.0, c_pw=1.0, alpha_pw=0.5, soft_winner=0, virtual_loss=1, stream=None):
    """One traversal per (tree, warp); results in ``d["out_selected"], d["out_path"], d["out_len"]``."""
    _check((_wave or _launcher()).puct_select(d, cpuct, c_pw, alpha_pw, int(soft_winner), int(virtual_loss), _stream(stream)), "select")


def launch_backup(d, values=None, virtual_loss=1, stream=None):
    """Turns the claims of the last select into statistics (``values``: float32[trees, warps, path_depth] on the device),
    or only releases them (``values=None``)."""
    _check((_wave or _launcher()).puct_backup(d, values, int(virtual_loss), _stream(stream)), "backup")


def launch_release(d, virtual_loss=1, stream=None):
    launch_backup(d, None, virtual_loss, stream)


V2_PRECLAIM, V2_COUNTER_CAS = 0, 1


def launch_select_v2(d, cpuct=1.0, c_pw=1.0, alpha_pw=0.5, variant=V2_PRECLAIM, stream=None):
    """The two older select kernels of the reference (``src/puct/puct_gpu_v2.py:573-840``), for trees that keep virtual
    visits per child node: ``d`` holds ``node_inflight`` (int32[trees, nodes]) in place of ``edge_inflight``.
    ``variant``: preclaim (every candidate is visited before it is scored, losers leave) or counter-CAS (the winner alone
    is claimed by compare-and-swap; a claim that met other visits is given back once)."""
    _check((_wave or _launcher()).puct_v2_select(d, int(variant), cpuct, c_pw, alpha_pw, _stream(stream)), "v2 select")


def launch_backup_v2(d, values=None, virtual_loss=1, stream=None):
    """``_backup_kernel_native`` of ``src/puct/puct_gpu_v2.py:847-927`` (``values=None``: release only)."""
    _check((_wave or _launcher()).puct_v2_backup(d, values, int(virtual_loss), _stream(stream)), "v2 backup")


def to_device(case, device="cuda"):
    """numpy case (as built by the tests) -> dict of torch CUDA tensors."""
    import torch
    return {k: (torch.from_numpy(v).to(device) if hasattr(v, "dtype") else v) for k, v in case.items()}


def to_host(d):
    return {k: (v.cpu().numpy() if hasattr(v, "cpu") else v) for k, v in d.items()}
