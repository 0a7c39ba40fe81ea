"""Loader for the ahead-of-time built kernel library ``nanonemo_b200/csrc/libnanonemo_b200.so``.

The kernels are plain ``extern "C"`` launchers taking device pointers, sizes and a stream, compiled
by ``nanonemo_b200/csrc/build.py`` with ``nvcc -gencode arch=compute_100a,code=sm_100a`` and loaded
here with ctypes; they are built before the run (never JIT-compiled per process, unlike the
reference's ``torch.utils.cpp_extension.load`` in nanonemo/kernels/cuda/__init__.py:15-18) and the
library sits in the source tree. Every launcher returns 0 on success or a negative error code
(bad argument, CUDA launch error) that ``check`` turns into an exception.
"""

import ctypes
import importlib
import operator
import os
import sys
import types
from functools import lru_cache
from pathlib import Path

import torch

LIB_PATH = Path(__file__).resolve().parents[1] / "csrc" / "libnanonemo_b200.so"


@lru_cache(maxsize=1)
def _load():
    if not LIB_PATH.exists():
        return None
    lib = ctypes.CDLL(str(LIB_PATH))
    lib.nnb_last_error.restype = ctypes.c_char_p
    return lib


def available() -> bool:
    """True when the built library exists and a CUDA device is present."""
    return torch.cuda.is_available() and _load() is not None and os.environ.get("NANONEMO_DISABLE_SM100") != "1"


def lib():
    handle = _load()
    if handle is None:
        raise RuntimeError(f"{LIB_PATH} is missing: build it with `python -m nanonemo_b200.csrc.build` "
                           "(the sm100 operators have no fallback)")
    return handle


@lru_cache(maxsize=1)
def native():
    """The C++ binding (csrc/binding.cpp): raw launches and operators that run without Python in between."""
    lib()  # (says how to build it when it is missing)
    try:
        binding = importlib.import_module("nanonemo_b200.ops._native")
    except ImportError as e:
        raise RuntimeError(f"nanonemo_b200/ops/_native.so is missing or was built against another torch ({e}): build it with "
                           "`python -m nanonemo_b200.csrc.build` (the sm100 operators have no fallback)") from e
    importlib.import_module("nanonemo_b200.ops.library")  # the operators that its backward nodes look up by name
    return binding


def operator_call(name: str, *args):
    """Operator `name` of the binding, or NotImplemented where the call is not a plain one (see csrc/binding.cpp)."""
    return NotImplemented if torch.compiler.is_compiling() else getattr(native(), name)(*args)


# Argument types of every launcher (p pointer, i int, q long long, f float, d double), in the order of its C declaration. With
# them a call passes plain Python numbers; wrapping each of a launcher's 10 to 45 arguments in a ctypes object first took longer
# than the launch itself.
_SIGNATURES = {
    "nnb_sumsq_blocks": "",
    "nnb_sumsq_f32": "pqppip",
    "nnb_adamw_flat": "ppppppqfffffipfiip",
    "nnb_sumsq_f32_noalloc": "pqpp",
    "nnb_ce_inplace": "pppqiqfip",
    "nnb_ce_grad_from_stats": "pppipqiqfip",
    "nnb_ce_loss_from_stats": "pipppqip",
    "nnb_ce_stats": "pppqiqqip",
    "nnb_ce_grad_vp": "ppppqiqqqifip",
    "nnb_comm_timeout_probe": "pppiip",
    "nnb_comm_flag_words": "i",
    "nnb_allreduce_f32": "ppppppiiqqfiidp",
    "nnb_sumsq_combine": "pqpp",
    "nnb_reduce_scatter_f32": "pppppppiiqqfiidp",
    "nnb_reduce_scatter_adamw": "ppppppppppiiqqfiidfffffiip",
    "nnb_allgather_bytes": "pppppiiqqidp",
    "nnb_peer_fetch": "pppippiiidp",
    "nnb_vp_embedding_fwd": "pppppqiqqippiiidp",
    "nnb_vp_embedding_bwd": "pppppqiqqippiiidp",
    "nnb_add_rmsnorm_fwd": "ppppppiifiiip",
    "nnb_rmsnorm_bwd_blocks": "",
    "nnb_add_rmsnorm_bwd": "pppppppppiiiiiip",
    "nnb_scale": "pppqiip",
    "nnb_rope_packed": "ppppqiiiiqqfip",
    "nnb_swiglu_fwd": "pppqiqqqip",
    "nnb_swiglu_bwd": "pppppqiqqqqqip",
    "nnb_embedding_fwd": "pppqiiip",
    "nnb_embedding_bwd": "pppqiiip",
    "nnb_warmup_add": "pppqp",
    "nnb_cast_from_f32": "ppqip",
    "nnb_build_arch": "",
    "nnb_flash_bwd_registers": "i",
    "nnb_flash_bwd_split": "iiqii",
    "nnb_flash_bwd": "pppppppppppiiiiiqqqqqqqqqqqqqqqqqqqqqqqqfippipp",
    "nnb_flash_fwd": "pppppiiiiiqqqqqqqqqqqqfipp",
    "nnb_gemm_bf16": "pppiiiqqqiiiiiiiipp",
    "nnb_gemm_rows": "pppiiiqqqiiipp",
    "nnb_gemm_rows_rope": "pppppiiiqqqiiiiiipp",
    "nnb_gemm_rows_f32w_serves": "iiii",
    "nnb_gemm_rows_f32w": "pppiiiqqqiipp",
    "nnb_gemm_rows_f32w_swiglu": "pppiiiqqqipp",
    "nnb_gemm_swiglu": "ppppiiiqqqqipp",
    "nnb_gemm_swiglu_act": "pppiiiqqqipp",
    "nnb_gemm_rope": "pppppiiiqqqiiiipp",
    "nnb_gemm_swiglu_bwd": "ppppiiiqqqqipp",
    "nnb_gemm_ce_stats": "ppppiiiqqqipp",
    "nnb_gemm_ce_loss": "pppppiiiqqipp",
    "nnb_gemm_rs_bf16": "ppppppiiiiiiqqqiiipp",
    "nnb_ag_gemm_bf16": "ppppppiiiiiiiqqiipp",
    "nnb_gather_b_gemm_bf16": "pppppppiiiiqqqiiiqqipp",
    "nnb_gemm_mxfp8": "pppppiiiqqqiiiipp",
    "nnb_mxfp8_quantize_sw": "pqpqppqpiip",
    "nnb_mxfp8_swiglu": "pqpqppqpiip",
    "nnb_mxfp8_swiglu_bwd": "pqpqpqppqpiip",
    "nnb_mxfp8_fake_quant": "ppqiqqp",
    "nnb_mxfp8_quantize": "pppqiqqp",
}
_TYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "q": ctypes.c_longlong, "f": ctypes.c_float, "d": ctypes.c_double}


@lru_cache(maxsize=None)
def _launcher(name: str):
    fn = getattr(lib(), name)
    fn.argtypes = [_TYPES[c] for c in _SIGNATURES[name]]
    return fn


_python_launches = 0  # launchers called through `call` since import; the binding counts its own


class _Module(types.ModuleType):
    @property
    def LAUNCHES(self) -> int:  # all launches since import (the benchmark reports the delta)
        return self._python_launches + (native().launches() if native.cache_info().currsize else 0)

    @LAUNCHES.setter
    def LAUNCHES(self, n: int):
        self._python_launches += n - self.LAUNCHES


sys.modules[__name__].__class__ = _Module


def stream_ptr() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())  # torch.cuda.current_stream() without its Python objects


def call(name: str, *args) -> None:
    """Call launcher `name`; raises with the library's message on a non-zero return."""
    global _python_launches
    rc = _launcher(name)(*args)
    _python_launches += 1
    if rc != 0:
        msg = lib().nnb_last_error()
        raise RuntimeError(f"{name} failed (code {rc}): {msg.decode() if msg else 'no message'}")


def call_rc(name: str, *args) -> int:
    """Like `call`, for launchers that answer 1 when they do not serve the problem (nothing was launched): returns 0 or 1."""
    global _python_launches
    rc = _launcher(name)(*args)
    if rc == 0:
        _python_launches += 1
    elif rc != 1:
        msg = lib().nnb_last_error()
        raise RuntimeError(f"{name} failed (code {rc}): {msg.decode() if msg else 'no message'}")
    return rc


def ptr(t: torch.Tensor | None) -> int:
    return 0 if t is None else t.data_ptr()


def reachable(*tensors: torch.Tensor) -> None:
    """A kernel that is given pageable host memory faults, and the context is lost."""
    for t in tensors:
        if not t.is_cuda and not (t.device.type == "cpu" and t.is_pinned()):
            raise AssertionError(f"the GPU cannot reach an operand on {t.device}")


i32 = i64 = operator.index  # an integer, as it is (anything else raises)
f32 = float


def vp(address: int | None) -> int | None:
    return address  # None is the null pointer
