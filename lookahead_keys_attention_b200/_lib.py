"""Build and load the two native parts of the package, both built in-tree: the C-ABI CUDA library
(`libcastle_b200.so`) and the torch-facing host module (`_host.so`), which prepares its calls.

There is no fallback: if either is missing or fails to load, every operator of this package raises.
"""
from __future__ import annotations

import ctypes
import os
import re
import shutil
import subprocess
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libcastle_b200.so"
SOURCES = ["api.cu", "decode.cu", "selftest.cu", "convert.cu", "transform.cu", "token_linear.cu", "token_layer.cu", "linear.cu", "norm.cu", "fwd.cu", "bwd.cu", "bwd128.cu"]

BF16, F16, F32 = 0, 1, 2


class CastleTensor(ctypes.Structure):
    _fields_ = [("ptr", ctypes.c_void_p), ("stride_b", ctypes.c_int64), ("stride_h", ctypes.c_int64),
                ("stride_n", ctypes.c_int64)]


class CastleProblem(ctypes.Structure):
    _fields_ = [("batch", ctypes.c_int32), ("heads", ctypes.c_int32), ("seq_len", ctypes.c_int32),
                ("dim_head", ctypes.c_int32), ("dtype", ctypes.c_int32), ("scale", ctypes.c_float)]


class CastleRotary(ctypes.Structure):
    _fields_ = [("freqs", ctypes.c_void_p), ("dtype", ctypes.c_int32), ("inverse", ctypes.c_int32),
                ("position0", ctypes.c_int64)]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; cannot build libcastle_b200.so")


def _sources():
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()]


NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-shared",
              "-Xcompiler", "-fPIC"]
STAMP_PATH = PKG_DIR / "libcastle_b200.so.stamp"
HOST_PATH = PKG_DIR / "_host.so"
HOST_STAMP_PATH = PKG_DIR / "_host.so.stamp"
HOST_SOURCE = CSRC / "host.cpp"


def _deps():
    return sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list((PKG_DIR.parent / "include").glob("*.h")))


def _source_hash() -> str:
    """Digest of every source the library is built from plus the compiler flags.  Compared with
    the stamp written next to the library, so a stale build is noticed whatever the file times say
    (a copied tree does not keep them)."""
    import hashlib
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    for d in _deps():
        h.update(d.name.encode())
        h.update(d.read_bytes())
    return h.hexdigest()


def needs_build():
    if not LIB_PATH.exists() or not STAMP_PATH.exists():
        return True
    return STAMP_PATH.read_text().strip() != _source_hash()


def _host_command(out):
    import sysconfig
    import torch
    inc, lib = Path(torch.__file__).parent / "include", Path(torch.__file__).parent / "lib"
    nvcc = Path(_nvcc()).resolve()
    cxx = os.environ.get("CXX") or shutil.which("g++") or "g++"
    return [cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f"-I{inc}", f"-I{inc / 'torch' / 'csrc' / 'api' / 'include'}", f"-I{sysconfig.get_paths()['include']}",
            f"-I{nvcc.parent.parent / 'include'}", str(HOST_SOURCE), "-o", str(out), f"-L{lib}", "-ltorch_python", "-ltorch",
            "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]


def _host_hash() -> str:
    import hashlib
    import sys
    import torch
    h = hashlib.sha256(f"{torch.__version__} {sys.version}".encode())
    for d in (HOST_SOURCE, PKG_DIR.parent / "include" / "castle_b200.h"):
        h.update(d.read_bytes())
    return h.hexdigest()


def needs_host_build():
    if not HOST_PATH.exists() or not HOST_STAMP_PATH.exists():
        return True
    return HOST_STAMP_PATH.read_text().strip() != _host_hash()


def _locked(fn):
    """Run `fn` holding the build lock (one builder per tree; ranks that start together queue here)."""
    import fcntl
    with open(PKG_DIR / ".build.lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            return fn()
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def wrong_registers(text: str):
    """What ptxas -v says (`text`) against the registers that the kernel which shares its launch's registers out anew counts on
    (`check_launch_regs` refuses it at its launch): a message per instance that was compiled with another number."""
    wanted = int(re.search(r"kSplitLaunchRegs = (\d+)", (CSRC / "bwd_common.cuh").read_text()).group(1))
    used = re.findall(r"Compiling entry function '(\w*castle_bwd_kernel\w*)'(?:(?!Compiling entry).)*?Used (\d+) registers", text, re.S)
    return [f"{kernel} was compiled with {n} registers a thread instead of {wanted}" for kernel, n in used if int(n) != wanted]


def _compile(jobs, verbose: bool = False):
    """Run the compilers of `jobs` (target, stamp, digest, command for an output path) side by side; readers see
    each old file or the complete new one, never half of it."""
    running = []
    for target, stamp, digest, command in jobs:
        tmp = target.with_name(f".{target.stem}.{os.getpid()}.tmp.so")
        running.append((target, stamp, digest, tmp, subprocess.Popen(command(tmp), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = []
    for target, stamp, digest, tmp, proc in running:
        text = proc.communicate()[0]
        wrong = wrong_registers(text)
        if proc.returncode == 0 and not wrong:
            os.replace(tmp, target)
            stamp.write_text(digest + "\n")
        else:
            failed.append(f"building {target.name} failed:\n" + ("\n".join(wrong) if proc.returncode == 0 else text))
            if tmp.exists():
                tmp.unlink()
        if verbose:
            print(text)
    if failed:
        raise RuntimeError("\n".join(failed))


def _build_unlocked(force: bool = False, verbose: bool = False):
    def nvcc(out):
        return [_nvcc()] + NVCC_FLAGS + ["-t", "0", "-Xptxas", "-v", "-o", str(out)] + \
               [str(s) for s in _sources()]
    jobs = []
    if force or needs_build():
        jobs.append((LIB_PATH, STAMP_PATH, _source_hash(), nvcc))
    if force or needs_host_build():
        jobs.append((HOST_PATH, HOST_STAMP_PATH, _host_hash(), _host_command))
    _compile(jobs, verbose)


def build(force: bool = False, verbose: bool = False):
    """Compile every kernel for sm_100a into one shared library next to this file, and the host module."""
    _locked(lambda: _build_unlocked(force, verbose))
    return LIB_PATH


_lib = None

P = ctypes.POINTER
_T, _PR = P(CastleTensor), P(CastleProblem)
_vp, _i32, _sz = ctypes.c_void_p, ctypes.c_int32, ctypes.c_size_t

_SIGNATURES = {
    "castle_abi_version": (ctypes.c_int, []),
    "castle_last_error": (ctypes.c_char_p, []),
    "castle_fwd_workspace_bytes": (_sz, [_PR]),
    "castle_fwd": (ctypes.c_int, [_PR] + [_T] * 7 + [_vp, _T, _i32, _vp, _vp, _sz, _vp, _vp]),
    "castle_fwd_prefill": (ctypes.c_int, [_PR] + [_T] * 7 + [_vp] + [_T] * 4 + [_vp, _vp, _sz, _vp, _vp]),
    "castle_convert_16bit": (ctypes.c_int, [_i32, _vp, _vp, ctypes.c_int64, _vp, _vp]),
    "castle_transform": (ctypes.c_int, [_PR, _i32, _T, _T, _i32, _i32, _T, P(CastleRotary), ctypes.c_uint32, _vp, _vp]),
    "castle_amax_scale": (ctypes.c_int, [_i32, _vp, ctypes.c_int64, _vp, _vp, _vp]),
    "castle_rmsnorm_fwd": (ctypes.c_int, [_i32, ctypes.c_int64, _i32, _vp, _vp, ctypes.c_float, _vp, _vp, _vp]),
    "castle_rmsnorm_bwd_workspace_bytes": (_sz, [ctypes.c_int64, _i32]),
    "castle_rmsnorm_bwd": (ctypes.c_int, [_i32, ctypes.c_int64, _i32] + [_vp] * 7 + [_sz, _vp]),
    "castle_bwd_workspace_bytes": (_sz, [_PR]),
    "castle_bwd": (ctypes.c_int, [_PR] + [_T] * 8 + [_vp, _vp] + [_T] * 6 + [_vp, _sz, _vp, _vp]),
    "castle_decode_workspace_bytes": (_sz, [_PR, _i32]),
    "castle_decode_step": (ctypes.c_int, [_PR, _i32, _i32] + [_T] * 11 + [_vp, _sz, _vp, _vp]),
    "castle_decode_step_fused": (ctypes.c_int, [_PR, _i32, _i32] + [_T] * 11 + [P(CastleRotary), _vp, _i32, _vp, _sz, _vp, _vp]),
    "castle_token_linear_fits": (ctypes.c_int, [_i32] * 3),
    "castle_token_linear": (ctypes.c_int, [_i32] * 4 + [_vp, ctypes.c_int64, _vp, ctypes.c_float, _vp, _vp, _i32, _vp]),
    "castle_token_layer_fits": (ctypes.c_int, [_PR, _i32, _i32, _i32]),
    "castle_token_layer_workspace_bytes": (_sz, [_PR, _i32]),
    "castle_token_layer": (ctypes.c_int, [_PR] + [_i32] * 4 + [_vp, ctypes.c_int64, _vp, ctypes.c_float, _vp, _vp] + [_T] * 4 +
                           [P(CastleRotary), _vp, _vp, _i32, _vp, _sz, _vp, _vp]),
    "castle_linear": (ctypes.c_int, [_i32] * 5 + [_vp, ctypes.c_int64] * 3 + [_vp, _vp]),
    "castle_decode_step_static": (ctypes.c_int, [_PR, _i32, _i32] + [_T] * 11 + [_vp, _vp]),
    "castle_set_kernel_events": (ctypes.c_int, [_i32, _vp, _vp]),
    "castle_selftest_mma_rate": (ctypes.c_int, [_i32, _i32, _i32, _vp, _vp, _vp]),
    "castle_selftest_mma": (ctypes.c_int, [_i32, _vp, _vp, _vp, _vp, _vp]),
    "castle_selftest_wait_timeout": (ctypes.c_int, [_i32, _vp, _vp, _vp]),
    "castle_selftest_event_timeout": (ctypes.c_int, [_i32, _i32, _i32, _vp, _vp, _vp]),
    "castle_selftest_exp2": (ctypes.c_int, [_vp, _vp, _i32, _vp]),
}


def _ensure_built():
    """Compile on demand what is missing or was built from other sources; there is no other code path to fall back to."""
    def go():
        try:
            _build_unlocked()
        except Exception as e:
            raise RuntimeError(f"{LIB_PATH.name} or {HOST_PATH.name} is missing or stale and could not be rebuilt ({e}); run "
                               "`python -c 'import __graft_entry__ as g; g.build()'` where nvcc is "
                               "available - this package has no fallback path") from e
    _locked(go)


def load():
    """Return the ctypes handle of the library; raises if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    override = os.environ.get("CASTLE_B200_LIB")   # a developer's own build of the same sources (other -D flags)
    if override:
        return _bind(ctypes.CDLL(override))

    _ensure_built()
    return _bind(ctypes.CDLL(str(LIB_PATH)))


def _bind(lib):
    global _lib
    for name, (res, args) in _SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    if lib.castle_abi_version() != 1:
        raise RuntimeError("libcastle_b200.so ABI version mismatch")
    _lib = lib
    return lib


def last_error() -> str:
    return load().castle_last_error().decode()


def check(rc: int, what: str):
    if rc != 0:
        raise RuntimeError(f"{what} failed (rc={rc}): {last_error()}")


_host = None


def host():
    """The native host module, bound to the library; raises if either cannot be built or loaded."""
    global _host
    if _host is None:
        lib = load()
        if os.environ.get("CASTLE_B200_LIB"):
            _ensure_built()   # load() took the developer's library as it is
        from . import _host as native
        native.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _SIGNATURES})
        _host = native
    return _host
