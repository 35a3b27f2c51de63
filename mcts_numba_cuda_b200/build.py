"""Builds ``libmctsnc_b200.so`` in-tree with nvcc for sm_100a (cross-compiles without a GPU), and ``_wave``, the Python
extension through which the tree selects are launched."""
import os
import shutil
import subprocess
import sysconfig
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB_PATH = os.path.join(HERE, "libmctsnc_b200.so")
# named with the interpreter's ABI tag: another Python on the same checkout does not load it but builds its own
WAVE_PATH = os.path.join(HERE, "_wave" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
WAVE_SOURCE = os.path.join(HERE, "csrc", "wave_module.cpp")
SOURCES = [os.path.join(HERE, "csrc", n) for n in ("mctsnc_abi.cu", "peer_exchange.cu", "puct_select.cu", "puct_select_v2.cu", "duct_select.cu")]
HEADERS = [os.path.join(HERE, "csrc", n) for n in ("c4_search.cuh", "c4_pool.cuh", "gomoku_search.cuh", "common.cuh", "rng.cuh", "select_math.cuh")]
WAVE_HEADERS = [os.path.join(ROOT, "include", n) for n in ("puct_b200.h", "duct_b200.h")]
HEADERS += WAVE_HEADERS + [os.path.join(ROOT, "include", "mctsnc_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-shared",
              "-Xcompiler", "-fPIC"]


def nvcc_path():
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found: libmctsnc_b200.so cannot be built")
    return path


def is_stale(path=LIB_PATH, sources=SOURCES + HEADERS):
    if not os.path.exists(path):
        return True
    built = os.path.getmtime(path)
    return any(os.path.exists(p) and os.path.getmtime(p) > built for p in sources)


def build_extension(force=False):
    """Compiles the extension if it is missing or older than its sources; returns its path."""
    if force or is_stale(WAVE_PATH, [WAVE_SOURCE] + WAVE_HEADERS):
        cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"], "-o", WAVE_PATH,
               WAVE_SOURCE]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
    return WAVE_PATH


def build(force=False, verbose=False):
    """Compiles the library and the extension if they are missing or older than their sources; returns the library's path.
    The searches need the library alone: an extension that cannot be built is a warning (a launch of a tree select says so
    again)."""
    if force or is_stale():
        cmd = [nvcc_path()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + SOURCES
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            print(res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    try:
        build_extension(force)
    except (OSError, RuntimeError) as e:
        warnings.warn(f"the extension that launches the tree selects could not be built: {e}", RuntimeWarning)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
