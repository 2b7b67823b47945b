"""ctypes loader of the in-tree sm_100a kernel library.

The library is plain ``extern "C"`` over raw device pointers and a stream handle, so loading
it needs neither the torch C++ headers nor a JIT cache.  ``load()`` builds it on demand when
the shared object is missing or older than its sources and nvcc is present.
"""
from __future__ import annotations

import ctypes
import functools
import warnings
from ctypes import c_char_p, c_double, c_float, c_int, c_longlong, c_uint, c_ulonglong, c_void_p

import torch

from ..utils import build as _build

P, I, LL, F, D, U, ULL = c_void_p, c_int, c_longlong, c_float, c_double, c_uint, c_ulonglong

_SIGNATURES = {
    "ob_wgrad_clip": [P, P, I, I, I, LL, LL, P, P, I, I, P, P, LL, P, LL, LL, LL, LL, I, I, I, P, D, I, P],
    "ob_ghost_norm_batch": [c_char_p, I, P, D, I, P],
    "ob_wgrad_clip_batch": [c_char_p, I, P, P, LL, I, P, D, I, P],
    "ob_wgrad_clip_pe_batch": [c_char_p, I, P, P, LL, P, D, I, P],
    "ob_gemm_tn": [P, P, P, P, P, P, LL, I, I, I, LL, LL, LL, LL, LL, I, I, F, P, I, I, P, D, I, P],
    "ob_lora_pack": [P, P, P, P, P, P, P, P, I, I, I, I, I, I, P],
    "ob_gemm_pair": [P, P, P, P, P, P, P, P, P, P, LL, I, I, I, LL, LL, LL, LL, LL, I, I, I, I, I, P, D, I, P],
    "ob_pair_init": [],
    "ob_pair_set_die_aware": [I],
    "ob_die_map": [P, I],
    "ob_layernorm_bwd_sums": [P, P, P, P, P, P, P, I, I, I, P, P, LL, P],
    "ob_rope_qkv_gather": [P, P, P, P, P, P, P, LL, I, I, I, I, I, I, P],
    "ob_gemm_tn_act": [P, P, P, P, P, LL, I, I, LL, LL, I, I, I, P, D, I, P],
    "ob_gemm_pair_glu_bwd": [P, P, P, P, P, P, LL, I, I, LL, LL, LL, LL, I, I, P, D, I, P],
    "ob_linear_ce_fwd": [P, P, P, P, P, P, P, LL, I, I, LL, LL, LL, F, F, LL, P, D, I, P],
    "ob_linear_ce_dlogits": [P, P, P, P, LL, I, LL, F, F, LL, P],
    "ob_moe_combine": [P, P, P, P, LL, I, I, I, P],
    "ob_moe_row_grad": [P, P, P, P, P, P, P, LL, I, I, P],
    "ob_moe_glu_bwd": [P, P, P, LL, I, I, P],
    "ob_clip_tree_chunks": [P, I],
    "ob_clip_tree": [P, P, P, I, I, D, D, D, D, I, F, P, P, P, P, P],
    "ob_layernorm_fwd": [P, P, P, P, P, P, LL, I, F, P],
    "ob_layernorm_bwd_dx": [P, P, P, P, P, P, LL, I, P],
    "ob_rows_group_sum": [P, P, P, P, I, I, I, LL, P, LL, I, P, LL, P],
    "ob_add_layernorm_fwd": [P, P, P, P, P, P, P, P, LL, I, F, P],
    "ob_add_layernorm_bwd_dx": [P, P, P, P, P, P, P, LL, I, P],
    "ob_rows_sum_batch": [c_char_p, I, I, I, P],
    "ob_merge_heads3": [P, P, P, P, P, LL, I, I, I, I, P],
    "ob_activation": [P, P, P, LL, I, I, P],
    "ob_ghost_set_wide": [I],
    "ob_push_grad": [P, LL, P, LL, P, I, P],
    "ob_rmsnorm_fwd": [P, P, P, P, P, P, LL, I, F, F, I, P],
    "ob_rmsnorm_bwd": [P, P, P, P, P, P, P, P, I, I, LL, I, F, P],
    "ob_glu_fwd": [P, P, P, LL, I, LL, I, I, P],
    "ob_glu_bwd": [P, P, P, P, P, LL, I, LL, LL, I, I, P],
    "ob_rope_qk": [P, P, P, P, P, LL, I, I, I, I, LL, LL, I, I, P],
    "ob_rope_qk_oop": [P, P, P, P, P, P, P, LL, I, I, I, I, LL, LL, LL, LL, LL, LL, I, I, P],
    "ob_cross_entropy": [P, I, P, P, P, P, LL, I, LL, F, F, F, LL, I, P],
    "ob_philox_normal_add": [P, I, LL, ULL, LL, F, U, I, P],
    "ob_rows_sumsq": [P, I, LL, LL, P, I, P],
    "ob_clip_weighted_sum": [P, P, I, LL, LL, P, P, LL, LL, I, P],
    "ob_embedding_wgrad": [P, P, P, LL, I, LL, P, P, LL, LL, I, P],
    "ob_shard_step": [P, P, P, P, P, P, P, P, P, LL, LL, I, ULL, F, F, I, I, I, P, I, F, F, F, F, F, F, F, F, I, I, I, I, P, I, P],
    "ob_peer_barrier": [P, P, I, I, I, P, D, P],
    "ob_ipc_alloc": [P, LL],
    "ob_ipc_free": [P],
    "ob_ipc_get_handle": [P, P],
    "ob_ipc_open_handle": [P, P],
    "ob_ipc_close_handle": [P],
    "ob_last_cuda_error": [c_char_p, I],
    "ob_last_detail": [c_char_p, I],
}


# entry points called with host arrays or handles (and once-only queries) stay with ctypes
_CTYPES_ONLY = {"ob_die_map", "ob_pair_init", "ob_pair_set_die_aware", "ob_ghost_set_wide", "ob_merge_heads3",
                "ob_clip_tree_chunks", "ob_clip_tree", "ob_shard_step", "ob_peer_barrier", "ob_ipc_alloc", "ob_ipc_free", "ob_ipc_get_handle",
                "ob_ipc_open_handle", "ob_ipc_close_handle", "ob_last_cuda_error", "ob_last_detail"}
_LETTER = {P: "P", c_char_p: "P", I: "I", LL: "L", F: "F", D: "D", U: "U", ULL: "Q"}


def launch_signatures() -> dict[str, str]:
    """Entry points that launch kernels, as ``{name: one letter per argument}`` (see ``utils.build.launcher_source``)."""
    return {n: "".join(_LETTER[a] for a in sig) for n, sig in _SIGNATURES.items() if n not in _CTYPES_ONLY}


class _Entries:
    """The library's entry points: launches through the compiled caller (0.3 us for 25 arguments, most of it their
    conversion), the rest through ctypes (2.6 us)."""

    def __init__(self, lib: ctypes.CDLL):
        self._cdll = lib
        for name in _SIGNATURES:
            setattr(self, name, getattr(lib, name))
        self.ob_debug_idesc_bf16 = lib.ob_debug_idesc_bf16

    def __getattr__(self, name: str):
        return getattr(self._cdll, name)


class KernelLibraryError(RuntimeError):
    pass


def _load_launcher(signatures: dict[str, str]):
    """The compiled caller, or ``None`` (with a warning: every call stays with ctypes) where it can neither be built nor loaded."""
    import importlib.util
    for force in (False, True):                 # an extension that does not load (another machine's, damaged) is built afresh
        try:
            path = _build.build_launcher(signatures, force)
            spec = importlib.util.spec_from_file_location("opaque_b200.ops._launch", path)
            launch = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(launch)
            return launch
        except (RuntimeError, OSError, ImportError) as exc:
            reason = exc
    warnings.warn(f"no compiled caller, launches go through ctypes at 2 us more each: {reason}", RuntimeWarning, stacklevel=3)
    return None


@functools.lru_cache(maxsize=None)
def load() -> _Entries:
    """The entry points of the kernel library (built on demand, loaded once)."""
    try:
        path = _build.build_kernels()
    except Exception as exc:
        if not _build.KERNEL_LIB.exists():
            raise KernelLibraryError(f"sm_100a kernel library is missing and could not be built: {exc}") from exc
        path = _build.KERNEL_LIB
    import os
    override = os.environ.get("OPAQUE_B200_KERNEL_LIB")          # a differently built library (kernel experiments)
    lib = ctypes.CDLL(override or str(path))
    for name, argtypes in _SIGNATURES.items():
        fn = getattr(lib, name)
        fn.argtypes = argtypes
        fn.restype = c_int
    lib.ob_clip_tree_chunks.restype = c_longlong
    lib.ob_debug_idesc_bf16.argtypes = [I, I, I, I]
    lib.ob_debug_idesc_bf16.restype = c_uint
    entries = _Entries(lib)
    signatures = launch_signatures()
    launch = _load_launcher(signatures)
    if launch is None:
        return entries
    for name in signatures:
        launch.bind(name, ctypes.cast(getattr(lib, name), c_void_p).value)
        setattr(entries, name, getattr(launch, name))
    return entries


def load_block_steps(plan, splits, budget: float):
    """The extension of ``csrc/block_steps.cpp`` with the library's entry points bound, or ``None`` (with a warning) where it can neither
    be built nor loaded: the callers then run their operations one by one."""
    import importlib.util
    entries = load()
    for force in (False, True):                 # as for the compiled caller
        try:
            path = _build.build_block_steps(force)
            spec = importlib.util.spec_from_file_location("opaque_b200.ops._blocks", path)
            steps = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(steps)
            for name in steps.entries().split():
                steps.bind(name, ctypes.cast(getattr(entries._cdll, name), c_void_p).value)
            steps.setup(check, plan, splits, sm_count(), budget)
            return steps
        except (RuntimeError, OSError, ImportError) as exc:
            reason = exc
    warnings.warn(f"no compiled launch sequences, decoder blocks run operation by operation: {reason}", RuntimeWarning, stacklevel=3)
    return None


def available() -> bool:
    """True when a CUDA device is present and the library loads."""
    if not torch.cuda.is_available():
        return False
    try:
        load()
        return True
    except Exception:
        return False


LAUNCHES = 0   # entry points called so far (each launches at least one kernel of this library)


def check(rc: int, what: str) -> None:
    global LAUNCHES
    LAUNCHES += 1
    if rc != 0:
        buf = ctypes.create_string_buffer(256)
        try:
            load().ob_last_cuda_error(buf, 256)
        except Exception:
            pass
        detail = ctypes.create_string_buffer(256)
        try:
            load().ob_last_detail(detail, 256)
        except Exception:
            pass
        raise KernelLibraryError(f"{what} failed with code {rc} ({buf.value.decode(errors='replace')}) "
                                 f"{detail.value.decode(errors='replace')}")


def ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


def stream() -> int:
    """Handle of the current stream of the current device (``torch.cuda.current_stream()`` builds a stream object through
    several Python layers: 3.2 us a call against 0.2, once per launch)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


@functools.lru_cache(maxsize=None)
def sm_count(device_index: int | None = None) -> int:
    idx = torch.cuda.current_device() if device_index is None else device_index
    return torch.cuda.get_device_properties(idx).multi_processor_count


_WAIT_ERRORS = {1: "a consumer timed out waiting for a TMA stage", 2: "the producer timed out waiting for a free stage",
                3: "the epilogue timed out waiting for an accumulator", 4: "the MMA issuer timed out waiting for TMEM",
                5: "the MMA issuer timed out waiting for the scaler warps", 6: "a peer's flag did not arrive in time",
                7: "draining in-flight copies timed out"}


class DeviceWaitTimeout(KernelLibraryError):
    """A bounded device-side wait expired; the context is still usable."""


class StatusWord:
    """A device int32 that kernels set when a bounded wait expires."""

    def __init__(self, device: torch.device | str | None = None):
        self.tensor = torch.zeros(1, dtype=torch.int32, device=device or "cuda")

    def ptr(self) -> int:
        return self.tensor.data_ptr()

    def read(self) -> int:
        return int(self.tensor.item())

    def raise_if_set(self, what: str = "kernel") -> None:
        code = self.read()
        if code:
            self.tensor.zero_()
            raise DeviceWaitTimeout(f"{what}: {_WAIT_ERRORS.get(code, 'unknown device status')} (code {code})")
