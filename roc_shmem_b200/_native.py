"""ctypes bindings of the in-tree native libraries.

The libraries are plain ``extern "C"`` shared objects built by ``build.py`` into
``roc_shmem_b200/lib`` — no pybind/torch extension ABI, so they load in any
process (also C programs can link them).  Loading is lazy and fails loudly: a
GPU code path never falls back to eager PyTorch when its library is missing.
"""
from __future__ import annotations

import ctypes as C
import importlib.machinery
import importlib.util
import os
import threading
from pathlib import Path

from . import build as _build

_LIB_DIR = Path(__file__).resolve().parent / "lib"
_lock = threading.Lock()
_libs: dict[str, C.CDLL] = {}


class NativeLibraryMissing(ImportError):
    pass


def load(name: str, *, build_if_missing: bool = True) -> C.CDLL:
    """Load ``lib/<name>``.  An existing library is used as it is: a multi-rank job imports this module in every
    rank at once, and ranks that each decided to recompile a library whose sources look newer would spend minutes
    in the compiler, racing on the same object files, before the first collective.  A missing library is built
    (one process at a time, under a file lock); set ``B200SHMEM_AUTO_REBUILD=1`` to also rebuild a stale one at
    import, as a developer convenience on a single process.  ``python -m roc_shmem_b200.build`` is the build step."""
    with _lock:
        if name in _libs:
            return _libs[name]
        path = _LIB_DIR / name
        want_build = build_if_missing and (not path.exists() or os.environ.get("B200SHMEM_AUTO_REBUILD", "") == "1")
        if want_build:
            try:
                with _build_lock():
                    if name == "libbshmem_host.so":
                        _build.build_host()
                    elif name in _build.CUDA_TARGETS:
                        _build.build_cuda_target(name)
            except Exception as e:   # keep an existing binary usable if the rebuild fails
                if not path.exists():
                    raise NativeLibraryMissing(f"cannot build {name}: {e}") from e
        if not path.exists():
            raise NativeLibraryMissing(f"{path} is missing; run `python -m roc_shmem_b200.build`")
        lib = C.CDLL(str(path), mode=C.RTLD_GLOBAL if name == "libbshmem_cuda.so" else C.RTLD_LOCAL)
        _libs[name] = lib
        return lib


_pycall_mod = None


def _pycall():
    """The extension module of csrc/host/pycall.cc (built on first use like the other libraries)."""
    global _pycall_mod
    if _pycall_mod is None:
        with _lock:
            if _pycall_mod is None:
                path = _LIB_DIR / _build.PYCALL
                if not path.exists():
                    with _build_lock():
                        _build.build_pycall()
                loader = importlib.machinery.ExtensionFileLoader("bshmem_pycall", str(path))
                spec = importlib.util.spec_from_file_location("bshmem_pycall", str(path), loader=loader)
                mod = importlib.util.module_from_spec(spec)
                loader.exec_module(mod)
                _pycall_mod = mod
    return _pycall_mod


def fast(lib: C.CDLL, name: str):
    """The declared entry point `name` of `lib` as a callable that takes integers, and int or None for an address.

    For entry points on a path that runs once per message or per layer: a ctypes call of the same function costs 1.5 to
    3 us, this one 0.15 us.  A result declared as a pointer comes back as an integer (0 = null)."""
    fn = getattr(lib, name)
    if fn.argtypes is None:
        raise TypeError(f"{name}: declare argtypes first")
    kind = 0 if fn.restype is C.c_int else (2 if fn.restype is None else 1)
    pointers = sum(1 << i for i, t in enumerate(fn.argtypes) if t in (C.c_void_p, C.c_char_p) or issubclass(t, C._Pointer))
    return _pycall().Native(C.cast(fn, C.c_void_p).value, len(fn.argtypes), kind, pointers)


def mover(lib: C.CDLL, name: str, context, method: str, plain, local: int):
    """put or get of a context as a callable that reads the tensors' addresses and sizes itself (csrc/host/pycall.cc), for calls
    (dest, src, pe, nbi=True or False) of plain tensors whose `local`-th is on the runtime's device, while `method` of the context's
    type is `plain`; anything else goes to that method."""
    import torch
    table = getattr(torch.Tensor, "__dlpack_c_exchange_api__", None)
    if table is None:                             # a torch without it
        return getattr(context, method)
    rt = context.rt
    try:
        return _pycall().Mover(C.cast(getattr(lib, name), C.c_void_p).value, rt._hv, context.idx, rt._dev_index, local, torch.Tensor, table,
                               context, method, plain, rt._check)
    except ValueError:                            # a table of another version, or without what is used of it
        return getattr(context, method)


class _build_lock:
    """Inter-process lock around an import-time build (ranks of one job share the source tree)."""

    def __enter__(self):
        import fcntl
        _LIB_DIR.mkdir(exist_ok=True)
        self._f = open(_LIB_DIR / ".build.lock", "w")
        fcntl.flock(self._f, fcntl.LOCK_EX)
        return self

    def __exit__(self, *exc):
        import fcntl
        fcntl.flock(self._f, fcntl.LOCK_UN)
        self._f.close()
        return False


class ErrorRecord(C.Structure):
    _fields_ = [("code", C.c_uint32), ("pe", C.c_int32), ("where", C.c_uint32), ("count", C.c_uint32),
                ("addr", C.c_uint64), ("expected", C.c_uint64), ("seen", C.c_uint64)]

    def as_dict(self) -> dict:
        return {k: getattr(self, k) for k, _ in self._fields_}


class NativeConfig(C.Structure):
    _fields_ = [("heap_bytes", C.c_uint64), ("timeout_us", C.c_uint64), ("max_teams", C.c_int32),
                ("max_ctxs", C.c_int32), ("debug", C.c_int32), ("profile", C.c_int32),
                ("requested_thread_level", C.c_int32), ("reserved0", C.c_int32)]


_VP, _I, _U64, _SZ, _L = C.c_void_p, C.c_int, C.c_uint64, C.c_size_t, C.c_long


def declare_runtime_api(lib: C.CDLL) -> None:
    """Argument/return types of the bshmem.h entry points (present in both the
    host library and the CUDA runtime library)."""
    def f(name, res, *args):
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = list(args)
    f("bshmem_config_default", None, C.POINTER(NativeConfig))
    f("bshmem_cpu_world_create", _I, C.c_char_p, _I, _U64, C.POINTER(_VP))
    f("bshmem_cpu_world_open", _I, C.c_char_p, C.POINTER(_VP))
    f("bshmem_cpu_world_destroy", _I, _VP)
    f("bshmem_cpu_world_mark_dead", _I, _VP, _I)
    f("bshmem_cpu_init", _I, _VP, _I, C.POINTER(NativeConfig), C.POINTER(_VP))
    f("bshmem_finalize", _I, _VP)
    f("bshmem_query_thread", _I, _VP, C.POINTER(_I))
    f("bshmem_my_pe", _I, _VP)
    f("bshmem_n_pes", _I, _VP)
    f("bshmem_global_exit", _I, _VP, _I)
    f("bshmem_last_error", C.c_char_p, _VP)
    f("bshmem_get_error_record", _I, _VP, C.POINTER(ErrorRecord), _I)
    f("bshmem_status_string", C.c_char_p, _I)
    f("bshmem_set_timeout_us", _I, _VP, _U64)
    f("bshmem_get_timeout_us", _U64, _VP)
    f("bshmem_set_current", None, _VP)
    f("bshmem_get_current", _VP)
    f("bshmem_malloc", _VP, _VP, _SZ)
    f("bshmem_align", _VP, _VP, _SZ, _SZ)
    f("bshmem_calloc", _VP, _VP, _SZ, _SZ)
    f("bshmem_free", _I, _VP, _VP)
    f("bshmem_malloc_local", _VP, _VP, _SZ, _SZ)
    f("bshmem_free_local", _I, _VP, _VP)
    f("bshmem_ptr", _VP, _VP, _VP, _I)
    f("bshmem_heap_base", _VP, _VP)
    f("bshmem_heap_bytes", _U64, _VP)
    f("bshmem_heap_usage", _I, _VP, C.POINTER(_U64 * 9))
    f("bshmem_addr_accessible", _I, _VP, _VP, _I)
    f("bshmem_ctx_create", _I, _VP, _L, C.POINTER(C.c_int32))
    f("bshmem_team_create_ctx", _I, _VP, C.c_int32, _L, C.POINTER(C.c_int32))
    f("bshmem_ctx_destroy", _I, _VP, C.c_int32)
    f("bshmem_team_split_strided", _I, _VP, C.c_int32, _I, _I, _I, C.POINTER(C.c_int32))
    f("bshmem_team_destroy", _I, _VP, C.c_int32)
    f("bshmem_team_n_pes", _I, _VP, C.c_int32)
    f("bshmem_team_my_pe", _I, _VP, C.c_int32)
    f("bshmem_team_translate_pe", _I, _VP, C.c_int32, _I, C.c_int32)
    for nm in ("putmem", "getmem", "putmem_nbi", "getmem_nbi"):
        f("bshmem_ctx_" + nm, _I, _VP, C.c_int32, _VP, _VP, _SZ, _I)
    f("bshmem_ctx_p_word", _I, _VP, C.c_int32, _VP, _U64, _SZ, _I)
    f("bshmem_ctx_g_word", _I, _VP, C.c_int32, _VP, _SZ, _I, C.POINTER(_U64))
    for nm in ("putmem_signal", "putmem_signal_nbi"):
        f("bshmem_ctx_" + nm, _I, _VP, C.c_int32, _VP, _VP, _SZ, _VP, _U64, _I, _I)
    f("bshmem_signal_fetch", _U64, _VP, _VP)
    f("bshmem_ctx_amo", _I, _VP, C.c_int32, _I, _I, _VP, _U64, _U64, _I, C.POINTER(_U64))
    f("bshmem_ctx_fence", _I, _VP, C.c_int32)
    f("bshmem_ctx_quiet", _I, _VP, C.c_int32)
    f("bshmem_wait_until", _I, _VP, _I, _VP, _I, _U64)
    f("bshmem_test", _I, _VP, _I, _VP, _I, _U64, C.POINTER(_I))
    f("bshmem_barrier_all", _I, _VP)
    f("bshmem_sync_all", _I, _VP)
    f("bshmem_team_sync", _I, _VP, C.c_int32)
    f("bshmem_team_barrier", _I, _VP, C.c_int32)
    f("bshmem_team_broadcast", _I, _VP, C.c_int32, _VP, _VP, _SZ, _I)
    f("bshmem_team_reduce", _I, _VP, C.c_int32, _I, _I, _VP, _VP, _SZ)
    f("bshmem_team_reduce_scatter", _I, _VP, C.c_int32, _I, _I, _VP, _VP, _SZ)
    f("bshmem_team_reduce_root", _I, _VP, C.c_int32, _I, _I, _VP, _VP, _SZ, _I)
    f("bshmem_team_fcollect", _I, _VP, C.c_int32, _VP, _VP, _SZ)
    f("bshmem_team_alltoall", _I, _VP, C.c_int32, _VP, _VP, _SZ)
    f("bshmem_barrier", _I, _VP, _I, _I, _I, _VP)
    f("bshmem_sync", _I, _VP, _I, _I, _I, _VP)
    f("bshmem_broadcast", _I, _VP, _VP, _VP, _SZ, _I, _I, _I, _I, _VP)
    f("bshmem_to_all", _I, _VP, _I, _I, _VP, _VP, _SZ, _I, _I, _I, _VP, _VP)
    f("bshmem_stats_count", _I)
    f("bshmem_stats_name", C.c_char_p, _I)
    f("bshmem_get_stats", _I, _VP, C.POINTER(_U64), _I)
    f("bshmem_reset_stats", _I, _VP)
    f("bshmem_dump_stats", _I, _VP)


_host_declared = False


def host_lib() -> C.CDLL:
    global _host_declared
    lib = load("libbshmem_host.so")
    if not _host_declared:
        declare_runtime_api(lib)
        _host_declared = True
    return lib
