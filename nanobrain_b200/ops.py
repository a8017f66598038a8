"""``torch.library`` custom ops over the C-ABI attention library.

Two public entry points:

``sdpa(query, key, value, attn_mask=None, dropout_p=0.0, is_causal=False, scale=None, enable_gqa=False)``
    Same signature as ``F.scaled_dot_product_attention`` and a drop-in for the call at
    ``src/nanobrain/modules.py:62`` of the reference (``F.scaled_dot_product_attention(q, k, v,
    is_causal=self.causal)`` with ``causal=False``): logical ``[B, H, L, 64]`` bf16 CUDA tensors,
    no mask, no dropout, non-causal. The result is logical ``[B, H, L, 64]`` backed by
    ``[B, L, H, 64]`` memory so the head merge at ``modules.py:63`` stays a view.

``sdpa_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale=None)``
    Packed variable-length form: ``[T, H, 64]`` tokens, sequence ``i`` owns rows
    ``[cu_seqlens[i], cu_seqlens[i+1])``. ``max_seqlen_*`` are host integers, so the call never
    synchronises with the device.

Anything outside that subset raises; there is no fallback and no backend dispatch. The four ops
(forward and backward of both) have their CUDA and autograd kernels in native code
(``csrc/torch_ops.cpp``) and their schemas and fake (meta) kernels here, so they trace under
``torch.compile`` and ``loss.backward()`` reaches the CUDA backward
(``src/nanobrain/misc.py:368-371``).
"""

from __future__ import annotations

import ctypes as C
import importlib.machinery
import importlib.util
import math
import warnings
from typing import Optional

import torch
from torch import Tensor
from torch.overrides import has_torch_function

from . import _lib

HEAD_DIM = 64
BINDING_PATH = _lib.LIB_PATH.with_name("_nb_torch.so")

_native = None  # the binding, once loaded


def _load_native():
    """Load the binding (which registers the ops' CUDA and autograd kernels)."""
    global _native
    if _native is None:
        _lib.load()
        if not BINDING_PATH.exists():
            raise RuntimeError(
                f"{BINDING_PATH} is missing: build it with `python -m nanobrain_b200.build` "
                "(there is no CPU or PyTorch fallback for this operator)"
            )
        loader = importlib.machinery.ExtensionFileLoader(BINDING_PATH.stem, str(BINDING_PATH))
        spec = importlib.util.spec_from_file_location(BINDING_PATH.stem, str(BINDING_PATH), loader=loader)
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
        _native = module
    return _native


def _status_word(device: torch.device) -> Tensor:
    """One int32 per device that kernels write to when something went wrong on the device.

    The word lives in pinned host memory, which the GPU addresses directly: a kernel's rare write
    goes over the bus, and the host can look at the word at any time without synchronising."""
    idx = device.index if device.index is not None else torch.cuda.current_device()
    return _load_native().status_word(idx)


def _raise_for_status(word: Tensor) -> None:
    code = int(word[0])
    if code != 0:
        word.zero_()
        text = _lib.STATUS_TEXT.get(code, "unknown code")
        raise RuntimeError(f"nanobrain_b200 attention kernel reported device status {code}: {text}")


def poll_status(device: Optional[torch.device] = None) -> None:
    """Raise if a kernel that has already finished reported a problem. Never synchronises: every
    op does this before it launches, so a failed step surfaces at the next attention call."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    _raise_for_status(_status_word(device))


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronise with ``device`` and raise if any kernel launched so far reported a problem.
    Call it where the training step synchronises anyway (for example where the loss is read)."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    torch.cuda.synchronize(device)
    _raise_for_status(_status_word(device))


def _require(cond: bool, msg: str) -> None:
    if not cond:
        raise RuntimeError("nanobrain_b200.sdpa: " + msg)


# ------------------------------------------------------------------------------------------
# The ops: schemas and fake kernels (same shapes and strides as the real results)
# ------------------------------------------------------------------------------------------
def _new_dense(like: Tensor) -> Tensor:
    b, h, l, d = like.shape
    return like.new_empty((b, l, h, d)).transpose(1, 2)


def _define_ops() -> torch.library.Library:
    library = torch.library.Library("nanobrain_b200", "DEF")
    for schema in (
        "sdpa_fwd(Tensor q, Tensor k, Tensor v, float scale) -> (Tensor, Tensor)",
        "sdpa_bwd(Tensor d_out, Tensor q, Tensor k, Tensor v, Tensor out, Tensor lse, float scale)"
        " -> (Tensor, Tensor, Tensor)",
        "sdpa_varlen_fwd(Tensor q, Tensor k, Tensor v, Tensor cu_seqlens_q, Tensor cu_seqlens_k, SymInt max_seqlen_q,"
        " SymInt max_seqlen_k, float scale) -> (Tensor, Tensor)",
        "sdpa_varlen_bwd(Tensor d_out, Tensor q, Tensor k, Tensor v, Tensor out, Tensor lse, Tensor cu_seqlens_q,"
        " Tensor cu_seqlens_k, SymInt max_seqlen_q, SymInt max_seqlen_k, float scale) -> (Tensor, Tensor, Tensor)",
    ):
        library.define(schema, tags=(torch.Tag.pt2_compliant_tag,))

    @torch.library.register_fake("nanobrain_b200::sdpa_fwd", lib=library)
    def _(q, k, v, scale):
        b, h, lq, d = q.shape
        return _new_dense(q), q.new_empty((b, h, lq), dtype=torch.float32)

    @torch.library.register_fake("nanobrain_b200::sdpa_bwd", lib=library)
    def _(d_out, q, k, v, out, lse, scale):
        return _new_dense(q), _new_dense(k), _new_dense(v)

    @torch.library.register_fake("nanobrain_b200::sdpa_varlen_fwd", lib=library)
    def _(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale):
        tq, h, d = q.shape
        return q.new_empty((tq, h, d)), q.new_empty((h, tq), dtype=torch.float32)

    @torch.library.register_fake("nanobrain_b200::sdpa_varlen_bwd", lib=library)
    def _(d_out, q, k, v, out, lse, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale):
        return q.new_empty(q.shape), k.new_empty(k.shape), k.new_empty(k.shape)

    return library


if "_library" not in globals():  # (a reload of this module keeps them)
    _library = _define_ops()

sdpa_fwd = torch.ops.nanobrain_b200.sdpa_fwd.default
sdpa_bwd = torch.ops.nanobrain_b200.sdpa_bwd.default
sdpa_varlen_fwd = torch.ops.nanobrain_b200.sdpa_varlen_fwd.default
sdpa_varlen_bwd = torch.ops.nanobrain_b200.sdpa_varlen_bwd.default

try:
    _load_native()
except (RuntimeError, OSError, ImportError, AttributeError) as error:
    # Not built yet, or older than these sources: import works all the same (to build it), the first use raises.
    if BINDING_PATH.exists():
        warnings.warn(f"nanobrain_b200: the native binding could not be loaded ({error}); its ops have no kernels. "
                      "`python -m nanobrain_b200.build` rebuilds it.")


# ------------------------------------------------------------------------------------------
# FLOP formulas: the reference measures TFLOP/s with ``FlopCounterMode`` over one forward +
# backward (``src/nanobrain/train.py:414-432``); a custom op is invisible to it unless a formula
# is registered. Same convention as torch's own SDPA formulas: 2 GEMMs forward, 5 backward.
# ------------------------------------------------------------------------------------------
def _pair_sum(cu_q: Tensor, cu_k: Tensor) -> int:
    lq = (cu_q[1:] - cu_q[:-1]).to(torch.int64)
    lk = (cu_k[1:] - cu_k[:-1]).to(torch.int64)
    return int((lq * lk).sum().item())


def _register_flop_formulas() -> None:
    from torch.utils.flop_counter import register_flop_formula

    @register_flop_formula(torch.ops.nanobrain_b200.sdpa_fwd)
    def _(q_shape, k_shape, v_shape, scale, *args, out_shape=None, **kwargs) -> int:
        b, h, lq, d = q_shape
        return 4 * b * h * lq * k_shape[2] * d

    @register_flop_formula(torch.ops.nanobrain_b200.sdpa_bwd)
    def _(d_out_shape, q_shape, k_shape, *args, out_shape=None, **kwargs) -> int:
        b, h, lq, d = q_shape
        return 10 * b * h * lq * k_shape[2] * d

    # The varlen formulas need the lengths, i.e. tensor values: get_raw=True hands over the tensors.
    @register_flop_formula(torch.ops.nanobrain_b200.sdpa_varlen_fwd, get_raw=True)
    def _(q, k, v, cu_q, cu_k, *args, out_val=None, **kwargs) -> int:
        return 4 * q.shape[1] * q.shape[2] * _pair_sum(cu_q, cu_k)

    @register_flop_formula(torch.ops.nanobrain_b200.sdpa_varlen_bwd, get_raw=True)
    def _(d_out, q, k, v, out, lse, cu_q, cu_k, *args, out_val=None, **kwargs) -> int:
        return 10 * q.shape[1] * q.shape[2] * _pair_sum(cu_q, cu_k)


if not globals().get("_flop_formulas"):
    _register_flop_formulas()
    _flop_formulas = True


# ------------------------------------------------------------------------------------------
# Public functions
# ------------------------------------------------------------------------------------------
def sdpa(
    query: Tensor,
    key: Tensor,
    value: Tensor,
    attn_mask: Optional[Tensor] = None,
    dropout_p: float = 0.0,
    is_causal: bool = False,
    scale: Optional[float] = None,
    enable_gqa: bool = False,
) -> Tensor:
    """Drop-in for ``F.scaled_dot_product_attention`` as called at ``src/nanobrain/modules.py:62``."""
    _require(attn_mask is None, "attn_mask is not supported (the reference passes none)")
    _require(dropout_p == 0.0, "dropout_p must be 0.0")
    _require(not is_causal, "is_causal=True is not supported (the reference's blocks are bidirectional)")
    _require(not enable_gqa, "enable_gqa is not supported")
    scale = 1.0 / math.sqrt(query.shape[-1]) if scale is None else float(scale)
    if torch.compiler.is_compiling() or has_torch_function((query, key, value)):
        return sdpa_fwd(query, key, value, scale)[0]  # tracing and overrides see the op itself
    return (_native or _load_native()).sdpa(query, key, value, scale)


def sdpa_varlen(
    q: Tensor,
    k: Tensor,
    v: Tensor,
    cu_seqlens_q: Tensor,
    cu_seqlens_k: Tensor,
    max_seqlen_q: int,
    max_seqlen_k: int,
    scale: Optional[float] = None,
) -> Tensor:
    """Bidirectional attention over packed ``[T, H, 64]`` tokens addressed by ``cu_seqlens``."""
    scale = 1.0 / math.sqrt(q.shape[-1]) if scale is None else float(scale)
    if torch.compiler.is_compiling() or has_torch_function((q, k, v, cu_seqlens_q, cu_seqlens_k)):
        return sdpa_varlen_fwd(q, k, v, cu_seqlens_q, cu_seqlens_k, int(max_seqlen_q), int(max_seqlen_k), scale)[0]
    return (_native or _load_native()).sdpa_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, int(max_seqlen_q),
                                                   int(max_seqlen_k), scale)


def selftest_mma(mode: int, a: Tensor, b: Tensor) -> Tensor:
    """Run one tensor-core operand form on a [128,128] bf16 pair; see ``nb_attn_selftest_mma``."""
    _require(a.is_cuda and b.is_cuda and a.dtype == b.dtype == torch.bfloat16, "a and b must be CUDA bfloat16")
    _require(a.shape == (128, 128) and b.shape == (128, 128), "a and b must be [128, 128]")
    a, b = a.contiguous(), b.contiguous()
    d = torch.empty((128, 128 if mode == 0 else 64), dtype=torch.float32, device=a.device)
    lib = _lib.load()
    with torch.cuda.device(a.device):
        _lib.check(
            lib.nb_attn_selftest_mma(mode, a.data_ptr(), b.data_ptr(), d.data_ptr(),
                                     _status_word(a.device).data_ptr(),
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream)),
            "nb_attn_selftest_mma",
        )
    return d
