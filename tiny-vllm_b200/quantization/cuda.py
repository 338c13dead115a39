"""Python entry points of the quantized-linear kernels.

Counterpart of ``nanovllm/quantization/cuda.py`` in the reference: the same
public functions (``apply_int8_weight_only_linear`` — reference lines 303-366,
``apply_w8a8_linear`` — lines 468-504) with the same argument meaning and the
same input checks (reference lines 21-33, 225-258, 369-432).  Differences, all
deliberate:

* one backend — the sm_100a library behind ``include/b200q.h``; the backend
  environment switches of the reference are gone;
* no Python/CPU fallback: an input the kernels cannot take raises
  ``RuntimeError`` where the reference would silently run dequantize + matmul;
* kernels run on ``torch.cuda.current_stream()`` so CUDA-graph capture records
  them (the reference launches on the legacy default stream).
"""
from __future__ import annotations

import torch

from .. import _lib

_DTYPE_IDS = {torch.float16: _lib.DTYPE_F16, torch.bfloat16: _lib.DTYPE_BF16}

# The calls themselves are native (csrc/torch_binding.cpp): it checks the arguments, allocates the
# results and launches on the current stream.  A native function answers ``None`` when it does
# not take its arguments as they are; the functions below then say what is wrong with them or
# make them contiguous and call it again.


def _native():
    return _lib._native or _lib.native()


def reserve_workspace(nbytes: int, device: torch.device | None = None) -> None:
    """Makes the per-device scratch buffer at least ``nbytes`` large (call before CUDA-graph
    capture when a model's shapes need more than the default 64 MiB; ``b200q_workspace_bytes``
    of the C ABI gives the need of a shape).  With a ``device`` the buffer is allocated now."""
    index = -1
    if device is not None:
        device = torch.device(device)
        index = torch.cuda.current_device() if device.index is None else device.index
    _native().reserve(int(nbytes), index)


def _refuse(what: str, entry: str, dims: dict[str, int], *tensors: torch.Tensor | None) -> None:
    """Raises for dense tensors of the right types that the native function did not take: they are on
    different GPUs, or have a shape that the C entry point refuses."""
    if len({t.device for t in tensors if t is not None}) > 1:
        raise RuntimeError(f"{what} does not support the provided tensors (all of them must be on one GPU)")
    too_large = any(d >= 1 << 31 for d in dims.values())
    _lib.check(_lib.ERR_BAD_SHAPE if too_large else _lib.ERR_UNSUPPORTED_SHAPE, entry,
               " ".join(f"{name}={d}" for name, d in dims.items()))


def _require_cuda(*tensors: torch.Tensor) -> None:
    if not all(t.is_cuda for t in tensors):
        raise RuntimeError(
            "b200q kernels need CUDA tensors on a B200; there is no CPU implementation of this path")


def _dense(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous and, for the kernels' vector loads, on a 16-byte boundary."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def select_path(op: int, M: int, N: int, K: int) -> str:
    """Kernel family the library picks for a problem (reference: ``select_path`` of the
    pybind modules, ``csrc/w8a8_gemm.cpp:51-54``)."""
    return _lib.lib().b200q_select_path(op, M, N, K).decode()


def quantize_activation_int8(x_2d: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """Per-token dynamic int8 quantisation on the GPU (one kernel).

    ``x_2d`` is ``[M, K]`` fp16/bf16 with unit inner stride.  Returns ``(x_q int8
    [M, K], a_scales fp32 [M])``, bit-identical to the reference's
    ``quantize_int8_per_row_dynamic`` (``nanovllm/quantization/utils.py:28-32``).
    """
    out = _native().quantize(x_2d)
    if out is not None:
        return out
    _require_cuda(x_2d)
    if x_2d.dim() != 2 or x_2d.dtype not in _DTYPE_IDS:
        raise RuntimeError("activation quantisation expects a 2-D float16/bfloat16 tensor")
    M, K = x_2d.shape
    if M == 0:
        return (torch.empty((0, K), dtype=torch.int8, device=x_2d.device),
                torch.empty((0,), dtype=torch.float32, device=x_2d.device))
    out = _native().quantize(_dense(x_2d))
    if out is None:
        _refuse("activation quantisation", "b200q_act_quant_i8", {"M": M, "K": K}, x_2d)
    return out


def add_rmsnorm_quantize_int8(x: torch.Tensor, weight: torch.Tensor, eps: float,
                              residual: torch.Tensor | None = None, return_normed: bool = False):
    """RMSNorm (optionally with the residual add in front) and the per-token int8 quantisation
    of its output in one kernel: what ``RMSNorm.forward`` (``nanovllm/layers/layernorm.py:16-50``)
    followed by ``quantize_int8_per_row_dynamic`` computes, without the 16-bit round trip.
    The new residual is bit-identical to the module's; the normalised value is within two units
    in the last place of it in at most 2 % of the elements (the mean of squares is summed in a
    different order); codes and scales are bit-identical to quantising the value formed here.

    ``x``: ``[..., K]`` fp16/bf16; ``weight``: ``[K]`` same dtype; ``residual``: like ``x`` or
    ``None``.  Returns ``(x_q [M, K] int8, a_scales [M] fp32, new_residual or None, normed or
    None)`` with ``M`` the flattened token count; ``new_residual`` has ``x``'s shape."""
    out = _native().rmsnorm_quant(x, weight, eps, residual, return_normed)
    if out is not None:
        return out
    _require_cuda(x, weight)
    if x.dtype not in _DTYPE_IDS or weight.dtype != x.dtype or weight.dim() != 1 \
            or weight.numel() != x.shape[-1]:
        raise RuntimeError("add_rmsnorm_quantize_int8 expects fp16/bf16 x and a weight of its width and dtype")
    if residual is not None and (residual.shape != x.shape or residual.dtype != x.dtype or not residual.is_cuda):
        raise RuntimeError("residual must match x in shape, dtype and device")
    if x.numel() == 0:
        _lib.check(_lib.ERR_BAD_SHAPE, "b200q_add_rmsnorm_quant_i8", f"M=0 K={x.shape[-1]}")
    out = _native().rmsnorm_quant(_dense(x), _dense(weight), eps,
                                  None if residual is None else _dense(residual), return_normed)
    if out is None:
        K = x.shape[-1]
        _refuse("add_rmsnorm_quantize_int8", "b200q_add_rmsnorm_quant_i8", {"M": x.numel() // K, "K": K},
                x, weight, residual)
    return out


def silu_mul_quantize_int8(gate_up: torch.Tensor, return_act: bool = False):
    """``SiluAndMul.forward`` (``nanovllm/layers/activation.py:11-14``) and the per-token int8
    quantisation of its output in one kernel.  ``gate_up``: ``[..., 2 I]`` fp16/bf16.  Returns
    ``(x_q [M, I] int8, a_scales [M] fp32, act [..., I] or None)``.

    Rounding: the activation is formed as ``T(silu(float(gate)) * float(up))`` — ONE rounding of
    the fp32 product, which is what the module's ``torch.compile`` decorator produces on a GPU.
    Run operation by operation (no compiler), the module rounds ``silu(gate)`` to 16 bits before
    the product; against that form the activation is never more than one unit in the last place
    off, in 26-27 % of the elements (measured on the reference module's outputs), and codes and
    scales can differ accordingly.  Against the single-rounding form fewer than 2 % of the
    elements differ by one unit (hardware ``exp``).  The int8 codes and scales are always
    bit-identical to quantising the activation this kernel formed."""
    out = _native().silu_mul_quant(gate_up, return_act)
    if out is not None:
        return out
    _require_cuda(gate_up)
    if gate_up.dtype not in _DTYPE_IDS or gate_up.shape[-1] % 2 != 0:
        raise RuntimeError("silu_mul_quantize_int8 expects an fp16/bf16 tensor with an even last dimension")
    if gate_up.numel() == 0:
        _lib.check(_lib.ERR_BAD_SHAPE, "b200q_silu_mul_quant_i8", f"M=0 I={gate_up.shape[-1] // 2}")
    out = _native().silu_mul_quant(_dense(gate_up), return_act)
    if out is None:
        two_i = gate_up.shape[-1]
        _refuse("silu_mul_quantize_int8", "b200q_silu_mul_quant_i8",
                {"M": gate_up.numel() // two_i, "I": two_i // 2}, gate_up)
    return out


def _check_w8a16(x, qweight, scales, bias) -> None:
    _require_cuda(x, qweight, scales)
    if x.dtype not in _DTYPE_IDS or qweight.dtype != torch.int8 or scales.dtype != torch.float32:
        raise RuntimeError("CUDA INT8 weight-only backend does not support the provided tensors")
    if x.numel() == 0 or qweight.numel() == 0 or scales.numel() == 0:
        raise RuntimeError("CUDA INT8 weight-only backend does not support the provided tensors")
    if qweight.dim() != 2 or x.shape[-1] != qweight.shape[-1]:
        raise RuntimeError(f"Incompatible shapes: x[-1]={x.shape[-1]} vs qweight[-1]={qweight.shape[-1]}")
    if scales.dim() != 1 or scales.numel() != qweight.shape[0]:
        raise RuntimeError("scales must be 1D with one value per output channel")
    if bias is not None:
        if bias.dim() != 1 or bias.numel() != qweight.shape[0]:
            raise RuntimeError("bias must be 1D with one value per output channel")
        if bias.dtype != x.dtype or not bias.is_cuda:
            raise RuntimeError("bias must be a CUDA tensor of the activation dtype")


def apply_int8_weight_only_linear(
    x: torch.Tensor,
    qweight: torch.Tensor,
    scales: torch.Tensor,
    bias: torch.Tensor | None = None,
) -> torch.Tensor:
    """W8A16 linear ``y = x @ dequant(qweight, scales).T + bias``.

    ``x``: ``[..., K]`` fp16/bf16; ``qweight``: int8 ``[N, K]``; ``scales``: fp32
    ``[N]``; returns ``[..., N]`` in ``x.dtype``.
    """
    y = _native().w8a16(x, qweight, scales, bias)
    if y is not None:
        return y
    _check_w8a16(x, qweight, scales, bias)
    y = _native().w8a16(_dense(x), _dense(qweight), _dense(scales), None if bias is None else _dense(bias))
    if y is None:
        N, K = qweight.shape
        _refuse("CUDA INT8 weight-only backend", "b200q_w8a16_gemm", {"M": x.numel() // K, "N": N, "K": K},
                x, qweight, scales, bias)
    return y


def w8a8_linear_dynamic(
    x: torch.Tensor,
    qweight: torch.Tensor,
    w_scales: torch.Tensor,
    bias: torch.Tensor | None = None,
) -> torch.Tensor | None:
    """``quantize_activation_int8`` and ``apply_w8a8_linear`` in one native call on contiguous
    16-bit activations ``[..., K]``; returns ``[..., N]`` in ``x.dtype``, or ``None`` for inputs
    that have to go through the two functions."""
    return _native().w8a8_dynamic(x, qweight, w_scales, bias)


def _check_w8a8(x_q, a_scales, qweight, w_scales, bias, out_dtype) -> None:
    _require_cuda(x_q, a_scales, qweight, w_scales)
    ok = (x_q.dtype == torch.int8 and qweight.dtype == torch.int8
          and a_scales.dtype == torch.float32 and w_scales.dtype == torch.float32
          and out_dtype in _DTYPE_IDS and x_q.dim() == 2 and qweight.dim() == 2
          and x_q.numel() > 0 and qweight.numel() > 0)
    if not ok:
        raise RuntimeError("CUDA W8A8 backend does not support the provided tensors")
    if x_q.shape[-1] != qweight.shape[-1]:
        raise RuntimeError(f"Incompatible shapes: x_q[-1]={x_q.shape[-1]} vs qweight[-1]={qweight.shape[-1]}")
    if a_scales.dim() != 1 or a_scales.numel() != x_q.shape[0]:
        raise RuntimeError("a_scales must be 1D with one value per input row")
    if w_scales.dim() != 1 or w_scales.numel() != qweight.shape[0]:
        raise RuntimeError("w_scales must be 1D with one value per output channel")
    if bias is not None:
        if bias.dim() != 1 or bias.numel() != qweight.shape[0]:
            raise RuntimeError("bias must be 1D with one value per output channel")
        if bias.dtype != out_dtype or not bias.is_cuda:
            raise RuntimeError("bias must be a CUDA tensor of the output dtype")


def apply_w8a8_linear(
    x_q: torch.Tensor,
    a_scales: torch.Tensor,
    qweight: torch.Tensor,
    w_scales: torch.Tensor,
    bias: torch.Tensor | None = None,
    out_dtype: torch.dtype = torch.float16,
    out_shape: tuple[int, ...] | None = None,
    out: torch.Tensor | None = None,
) -> torch.Tensor:
    """W8A8 linear: exact int32 ``x_q @ qweight.T``, then
    ``(acc * a_scales[:, None]) * w_scales[None, :] + bias`` cast to ``out_dtype``.
    ``out``: a contiguous ``[M, N]`` tensor of ``out_dtype`` to write into instead of a new one
    (e.g. a slot of the symmetric buffer that a tensor-parallel exchange reads)."""
    dtype_id = _DTYPE_IDS.get(out_dtype, -1)
    y = _native().w8a8(x_q, a_scales, qweight, w_scales, bias, dtype_id, out_shape, out)
    if y is not None:
        return y
    _check_w8a8(x_q, a_scales, qweight, w_scales, bias, out_dtype)
    M, N = x_q.shape[0], qweight.shape[0]
    if out is not None and (tuple(out.shape) != (M, N) or out.dtype != out_dtype
                            or not out.is_contiguous() or out.device != x_q.device):
        raise RuntimeError(f"out must be a contiguous [{M}, {N}] {out_dtype} tensor on {x_q.device}")
    y = _native().w8a8(_dense(x_q), _dense(a_scales), _dense(qweight), _dense(w_scales),
                       None if bias is None else _dense(bias), dtype_id, None, out)
    if y is None:
        _refuse("CUDA W8A8 backend", "b200q_w8a8_gemm", {"M": M, "N": N, "K": x_q.shape[1]},
                x_q, a_scales, qweight, w_scales, bias)
    return y if out_shape is None else y.view(out_shape)


def w8a8_int32_accumulators(x_q: torch.Tensor, qweight: torch.Tensor) -> torch.Tensor:
    """Raw int32 ``x_q @ qweight.T`` from the same kernels (parity/debug entry)."""
    acc = _native().w8a8_i32(x_q, qweight)
    if acc is not None:
        return acc
    _require_cuda(x_q, qweight)
    if x_q.dtype != torch.int8 or qweight.dtype != torch.int8 or x_q.dim() != 2 or qweight.dim() != 2:
        raise RuntimeError("w8a8_int32_accumulators expects 2-D int8 tensors")
    if x_q.shape[1] != qweight.shape[1]:
        raise RuntimeError("x_q and qweight shapes do not align")
    acc = _native().w8a8_i32(_dense(x_q), _dense(qweight))
    if acc is None:
        (M, K), N = x_q.shape, qweight.shape[0]
        _refuse("w8a8_int32_accumulators", "b200q_w8a8_gemm_i32", {"M": M, "N": N, "K": K}, x_q, qweight)
    return acc
