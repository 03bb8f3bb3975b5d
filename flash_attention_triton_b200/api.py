"""Drop-in Python surface of the reference's causal FlashAttention-2 operator.

Mirrors ``src/flash_attention_triton/flash_attention_2.py`` of flash-attention-triton:

* :func:`flash_attention_v2` (reference lines 646-697) — same name, arguments and defaults;
* :func:`flash_attention_v2_custom` (700-790) — same signature; the tile/warp knobs of the
  config are ignored (there is no Triton here), only its ``SEQUENCE_PARALLEL`` flag survives
  as the deterministic switch;
* :class:`FlashAttentionV2Function` (280-384) — ``apply(q, k, v, softmax_scale, deterministic)``
  returning five gradients ``(dq, dk, dv, None, None)``;
* :class:`KernelsConfigV2`, :func:`init_to_zero_v2` (``_configurators_v2.py:9-93``).

Differences, all deliberate: fp16 and bf16 inputs run natively (the reference casts
everything to fp16, lines 316/379); other float dtypes are cast to fp16 exactly as the
reference does.  Multiples of 8 run natively as head dimension (the kernels run them
zero-padded to 32 / 64 / 128 / 256 through TMA out-of-bounds fill; other sizes are
zero-padded to a multiple of 8 on the host first); head dimensions up to 256 are supported.
``seqlen_q != seqlen_k`` follows the reference's top-left aligned causal mask: query row i sees keys ``0 .. min(i, seqlen_k - 1)``;
keys beyond ``seqlen_q`` are seen by nobody and get zero gradients.
Everything runs through the C library on the tensors' CUDA device; there is no fallback.
"""

from __future__ import annotations

import functools
import math
import os
from collections.abc import Callable
from dataclasses import dataclass
from typing import Any

import torch

from . import _lib

_MAX_HEAD_DIM = 256  # the reference's max_headdim on B200 (line 533)


# ------------------------------------------------------------------ host launch wrappers
_COMPUTE_DTYPES = (torch.float16, torch.bfloat16)


def _check_status_if_asked(fn: str, device: torch.device) -> None:
    """Kernels that give up on a bounded wait leave their outputs unwritten and only set the
    device status word; reading it synchronises the device, so it is not read by default.
    ``FA2_B200_CHECK_STATUS=1`` makes every forward / backward call read that of the tensors' device and
    raise ``Fa2Error`` (``FA2_ERR_DEVICE_STATUS``) when it is non-zero."""
    if os.environ.get("FA2_B200_CHECK_STATUS") == "1":
        with torch.cuda.device(device):  # the library reads the current device's word
            word = _lib.device_status()
        if word:
            raise _lib.Fa2Error(fn, -7, f"{_lib.lib().fa2_strerror(-7).decode()} (status {word:#x})")


def _as_kernel_input(t: torch.Tensor) -> torch.Tensor:
    """The tensor itself when the kernels can read it through its own strides (unit last stride,
    16-byte aligned base, batch / head / row strides that are positive multiples of 8 elements;
    e.g. a transposed ``[B, N, H, D]`` buffer), else a contiguous copy (what the reference always
    makes, line 316)."""
    return t if _lib.host().readable_in_place(t) else t.contiguous()


def _flash_attention_forward(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, softmax_scale: float | None, f32: bool = False
) -> tuple[torch.Tensor, torch.Tensor, float] | tuple[torch.Tensor, torch.Tensor, float, torch.Tensor]:
    """Validate, allocate O and LSE, launch ``fa2_fwd``; with ``f32`` also return O as fp32.

    Counterpart of ``_flash_attention_forward`` (reference lines 61-144): the same asserts on
    shapes / device / dtype, ``softmax_scale or 1/sqrt(d)`` (so 0.0 means "default"), but
    LSE is an unpadded ``[B, H, N]`` fp32 tensor and no scratch buffer exists.
    """
    batch, nheads, seqlen_q, headdim = q.shape
    seqlen_k = k.shape[2]
    assert k.shape == (batch, nheads, seqlen_k, headdim)
    assert v.shape == (batch, nheads, seqlen_k, headdim)
    assert q.is_cuda and k.is_cuda and v.is_cuda, "All tensors must reside on CUDA device"
    assert q.dtype == k.dtype == v.dtype, "All tensors must be the same type"
    if headdim > _MAX_HEAD_DIM or headdim % 8:
        raise ValueError(f"head dimension {headdim} is not supported (multiples of 8 up to {_MAX_HEAD_DIM})")
    if seqlen_k > seqlen_q:  # no query sees the keys beyond seqlen_q - 1 (top-left aligned mask)
        k, v, seqlen_k = k[:, :, :seqlen_q], v[:, :, :seqlen_q], seqlen_q
    softmax_scale = softmax_scale or 1.0 / math.sqrt(headdim)
    assert q.dtype in _COMPUTE_DTYPES, "Supports only fp16 and bf16 compute dtypes"
    # output and LSE are dense, like the reference's
    code, output, lse, output32 = _lib.host().forward(q, k, v, float(softmax_scale), f32)
    _lib.check("fa2_fwd_strided", code)
    _check_status_if_asked("fa2_fwd_strided", q.device)
    return (output, lse, softmax_scale, output32) if f32 else (output, lse, softmax_scale)


#: dQ strategies of the C library (the ``deterministic`` argument of ``fa2_bwd``)
_MODE_ATOMIC, _MODE_RECOMPUTE, _MODE_SPILL = 0, 1, 2
_MODE_NAMES = {"atomic": _MODE_ATOMIC, "recompute": _MODE_RECOMPUTE, "spill": _MODE_SPILL}


def _backward_mode(deterministic: bool, headdim: int, seqlen_q: int) -> int:
    """Which dQ strategy serves ``deterministic``.

    ``True`` must give the same bits whatever the batch / head partitioning, so the choice
    depends on the head dim and the sequence length only.  Head dims above 64: the spill mode
    (fastest there, 10-25 % ahead of the recompute mode) unless one head's scratch (32 KiB per tile
    pair) exceeds 2 GiB (N above ~45 k), then the recompute mode, which needs none.  Head dims up to
    64: the recompute mode, which is 4-14 % ahead of the spill mode there (the 32 KiB dS tile does not
    shrink with the head dim, the tensor work does) and needs no scratch, like the reference's O(N) backward.
    ``False`` (the reference's default, atomics there) means "fastest": the atomic kernel at
    head dims up to 64 (14-21 % ahead of the recompute mode from 4096 rows, the same at 2048), the
    deterministic choice above.  ``FA2_B200_BWD_MODE`` =
    ``atomic`` / ``recompute`` / ``spill`` overrides both (for experiments).  The rule itself is
    ``backward_mode`` of ``csrc/host.cpp``, which calls that do not come here follow as well.
    """
    forced = os.environ.get("FA2_B200_BWD_MODE")
    if forced and headdim <= 128:  # above, one (deterministic) backward exists: scores with dV + two consumers
        return _MODE_NAMES[forced]
    return _lib.backward_mode(bool(deterministic), headdim, seqlen_q)


def _allocate_workspace(lib, device, batch, nheads, seqlen_q, headdim, mode):
    """The workspace of a backward mode, and the mode that will run.

    The scratch of the spill mode is a convenience, not a need (the reference's backward is
    O(N) in memory, ``flash_attention_2.py:195-196``): when the recommended size cannot be had,
    an eighth of it is tried (more chunks, a few per cent slower), then one head's worth, and
    when even that fails the recompute backward, which needs no scratch and gives the same dK,
    dV and a dQ that differs in the last bit at most, runs instead.  Head dims above 128 have no
    scratch-free backward: there the out-of-memory error propagates.  The steps themselves are
    ``allocate_workspace`` of ``csrc/host.cpp``, which calls that do not come here take as well; ``lib``
    is not asked.
    """

    def allocate(nbytes):
        try:
            return torch.empty(nbytes, device=device, dtype=torch.uint8)
        except torch.cuda.OutOfMemoryError:
            return None

    workspace, nbytes, served = _lib.allocate_workspace(allocate, batch, nheads, seqlen_q, headdim, mode)
    if served < 0:
        raise torch.cuda.OutOfMemoryError(f"no memory for the backward workspace ({nbytes} bytes at least)")
    return workspace, nbytes, served


def _flash_attention_backward(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    output: torch.Tensor,
    lse: torch.Tensor,
    dq: torch.Tensor,
    dk: torch.Tensor,
    dv: torch.Tensor,
    d_output: torch.Tensor,
    softmax_scale: float,
    deterministic: bool,
) -> None:
    """Launch ``fa2_bwd_preprocess`` and ``fa2_bwd``.

    Counterpart of ``_flash_attention_backward`` (reference lines 147-277).  The workspace
    depends on the dQ strategy (:func:`_backward_mode`): an fp32 accumulator for the atomic
    kernel, the dS scratch for the spill mode, nothing for the recompute mode; the
    deterministic modes write dQ once.  dq, dk and dv have the dtype of q, rounded once, or are
    fp32, unrounded.
    """
    batch, nheads, seqlen_q, headdim = q.shape
    seqlen_k = k.shape[2]
    if seqlen_k > seqlen_q:  # keys nobody sees: zero gradients, and the kernels skip them
        dk[:, :, seqlen_q:].zero_()
        dv[:, :, seqlen_q:].zero_()
        k, v, dk, dv = (t[:, :, :seqlen_q] for t in (k, v, dk, dv))
        seqlen_k = seqlen_q
    # The reference requires everything contiguous here (lines 183-192) and copies dO when it
    # is not (170-171); the inputs may keep their strides, only our own buffers are dense.
    assert lse.shape == (batch, nheads, seqlen_q)
    assert output.is_contiguous() and dq.is_contiguous()
    assert q.dtype in _COMPUTE_DTYPES, "Supports only fp16 and bf16 compute dtypes"
    host = _lib.host()
    assert host.readable_in_place(dk) and host.readable_in_place(dv)
    code, rowstats, d_output = host.preprocess(output, d_output, lse)
    _lib.check("fa2_bwd_preprocess_strided", code)
    mode = _backward_mode(bool(deterministic), headdim, seqlen_q)
    workspace, _, mode = _allocate_workspace(
        _lib.lib(), q.device, batch, nheads, seqlen_q, headdim, mode)
    _lib.check("fa2_bwd_strided", host.backward(
        q, k, v, d_output, dq, dk, dv, rowstats, workspace, float(softmax_scale), mode))
    _check_status_if_asked("fa2_bwd_strided", q.device)


# ------------------------------------------------------------------ autograd integration
def _compute_dtype(dtype: torch.dtype) -> torch.dtype:
    # fp16 / bf16 run natively; everything else takes the reference's route (cast to fp16,
    # reference line 316).
    return dtype if dtype in _COMPUTE_DTYPES else torch.float16


class FlashAttentionV2Function(torch.autograd.Function):
    """Autograd function for causal FlashAttention-2 (reference lines 280-384)."""

    @staticmethod
    def forward(ctx: Any, q, k, v, softmax_scale, deterministic):  # noqa: ANN001
        initial_dtype = q.dtype
        cdtype = _compute_dtype(q.dtype)
        f32 = q.dtype == k.dtype == v.dtype == torch.float32
        headdim = q.shape[-1]
        if headdim > _MAX_HEAD_DIM:
            raise ValueError(f"head dimension {headdim} is not supported (at most {_MAX_HEAD_DIM})")
        softmax_scale = softmax_scale or 1.0 / math.sqrt(headdim)  # reference line 94: 0.0 -> default
        q, k, v = [_as_kernel_input(t if t.dtype == cdtype else t.to(cdtype)) for t in (q, k, v)]
        pad = -headdim % 8  # zero columns change neither the scores nor the real output columns
        if pad:
            q, k, v = [torch.nn.functional.pad(t, (0, pad)) for t in (q, k, v)]
        ctx.deterministic = bool(deterministic)
        ctx.headdim = headdim
        # fp32 callers get fp32 results from the kernels' accumulators, without a cast pass
        ctx.f32 = f32 and not pad
        if ctx.f32:
            output, lse, ctx.softmax_scale, output32 = _flash_attention_forward(q, k, v, softmax_scale, True)
            ctx.save_for_backward(q, k, v, output, lse)
            return output32
        output, lse, ctx.softmax_scale = _flash_attention_forward(q, k, v, softmax_scale)
        ctx.save_for_backward(q, k, v, output, lse)
        if pad:
            output = output[..., :headdim].contiguous()
        else:
            output = output.view(output.shape)  # the tensor that is saved is not the one handed out
        return output if initial_dtype == cdtype else output.to(initial_dtype)

    @staticmethod
    def backward(ctx: Any, d_output):  # noqa: ANN001
        q, k, v, output, lse = ctx.saved_tensors
        dq, dk, dv = _lib.host().gradients(q, k, v, ctx.f32)
        if d_output.dtype != q.dtype:
            d_output = d_output.to(q.dtype)
        pad = q.shape[-1] - ctx.headdim
        if pad:
            d_output = torch.nn.functional.pad(d_output, (0, pad))
        _flash_attention_backward(
            q, k, v, output, lse, dq, dk, dv, d_output, ctx.softmax_scale, ctx.deterministic,
        )
        if pad:
            dq, dk, dv = [t[..., : ctx.headdim].contiguous() for t in (dq, dk, dv)]
        return dq, dk, dv, None, None


# ------------------------------------------------------------------ configuration shim
@dataclass(frozen=True)
class KernelsConfigV2:
    """Name-compatible stand-in for the reference's kernel configuration container.

    Same fields as ``_configurators_v2.py:9-38``.  Tile sizes, warp counts and stages have
    no meaning for the hand-written sm_100a kernels and are ignored; the only information
    used is whether the first backward config asks for ``SEQUENCE_PARALLEL`` (atomic dQ,
    non-deterministic) or not (deterministic), as in the reference's tables (lines 570-589).
    """

    block_rows_size: int
    block_cols_size: int
    min_block_headdim: int
    max_headdim: int
    seqlen_cache_divisor: int
    min_warps: int
    max_warps: int
    num_stages: int
    backward_autotune_configs: list

    def is_deterministic(self) -> bool:
        if not self.backward_autotune_configs:
            return True
        first = self.backward_autotune_configs[0]
        kwargs = getattr(first, "kwargs", first if isinstance(first, dict) else {})
        return not bool(kwargs.get("SEQUENCE_PARALLEL", False))


def init_to_zero_v2(name: str) -> Callable[[dict[str, torch.Tensor]], torch.Tensor]:
    """Pre-hook factory kept for source compatibility (``_configurators_v2.py:81-93``)."""
    return lambda nargs: nargs[name].zero_()


# ------------------------------------------------------------------ public API
@functools.lru_cache(maxsize=None)
def _capability(index: int) -> tuple[int, int]:
    return torch.cuda.get_device_capability(index)


def _check_device(q: torch.Tensor) -> None:
    assert q.is_cuda, "All tensors must reside on CUDA device"
    cc = _capability(q.device.index)
    if cc[0] != 10:
        raise RuntimeError(
            f"compute capability {cc} is not supported: this library targets B200 (sm_100a) only"
        )


def _attention(q, k, v, softmax_scale, deterministic):  # noqa: ANN001
    """The call through the native autograd function where it serves it (plain fp16, bf16 or fp32 tensors, no
    transform, trace or mode active), through :class:`FlashAttentionV2Function` otherwise: same kernels, same
    results, same errors."""
    if not torch.compiler.is_compiling():
        output = _lib.host().attention(q, k, v, softmax_scale, deterministic)
        if output is not None:
            return output
    return FlashAttentionV2Function.apply(q, k, v, softmax_scale, deterministic)


def flash_attention_v2(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    softmax_scale: float | None = None,
    deterministic: bool = False,
) -> torch.Tensor:
    """Causal FlashAttention-2 on B200; same contract as the reference (lines 646-697).

    Args:
        q, k, v: ``(batch, nheads, seqlen, headdim)`` CUDA tensors of one float dtype.
        softmax_scale: scaling factor (default and 0.0: ``1/sqrt(headdim)``).
        deterministic: use the backward whose dQ has a fixed summation order (bit-identical
            across runs and across batch x head partitionings) instead of fp32 atomics.

    Returns:
        Attention output, same shape and dtype as ``q``.
    """
    _check_device(q)
    return _attention(q, k, v, softmax_scale, deterministic)


def flash_attention_v2_custom(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    softmax_scale: float | None,
    kernels_configs: dict[tuple[int, int], KernelsConfigV2],
) -> torch.Tensor:
    """Same signature as the reference (lines 700-790): config looked up by compute capability.

    Raises ``ValueError`` when the current device's capability has no entry, as the
    reference does (lines 775-779).
    """
    _check_device(q)
    cc = torch.cuda.get_device_capability(q.device)
    if cc not in kernels_configs:
        raise ValueError(
            f"Missing kernel configuration for compute capability {cc}. "
            "KernelsConfig must be provided for the current GPU architecture"
        )
    deterministic = kernels_configs[cc].is_deterministic()
    return _attention(q, k, v, softmax_scale, deterministic)
