"""The body the reference's serving patch gives `fused_experts_impl` (extra/sglang.patch:25-40), on this
library's own kernels: knob look-up for the batch size, activation quantisation, clearing of the buffer the
layer accumulates into, block schedule, fused operator.  `hidden_states` holds the layer output on return,
as in the patch.  Checks, buffers and the C-ABI call are one torch operator; where only the C library has been built, the same
three steps are taken here."""
from __future__ import annotations

import contextlib
import os

import torch

from . import capi, load_torch_op
from .utils import get_best_config

def _check_layer_arguments(hidden_states, w1, w1_scale, w2, w2_scale, topk_weights, topk_ids) -> None:
    """The checks the torch operator makes on its tensors (csrc/torch_interface.cpp:58-76 of the reference, plus
    the dtype / device / shape checks this library's operator adds), for calls that do not get to the torch operator, which
    checks its CUDA tensors by the same rules and in the same words (csrc/torch_interface.cpp): the C ABI sees only addresses."""
    # (written out: messages are only put together for a call that fails)
    if hidden_states.dtype != torch.bfloat16 or hidden_states.dim() != 2 or not hidden_states.is_contiguous():
        raise RuntimeError("hidden_states must be a contiguous 2-D bfloat16 tensor")
    dev = hidden_states.device
    m, k = hidden_states.shape
    if m <= 0:
        raise RuntimeError("hidden_states must have at least one row")
    if k % 128 != 0:
        raise RuntimeError("K dimension must be a multiple of 128")
    if w1.dim() != 3 or w2.dim() != 3:
        raise RuntimeError("w1 must be [E, 2I, K] and w2 [E, K, I]")
    e, n, kw = w1.shape
    if kw != k:
        raise RuntimeError("w1.size(2) must equal hidden_states.size(1)")
    if n % 256 != 0:
        raise RuntimeError("N (2 x intermediate size) must be a multiple of 256")
    if w2.shape != (e, k, n // 2):
        raise RuntimeError("w2 must be [E, K, N/2]")
    if w1.dtype != torch.float8_e4m3fn or w2.dtype != torch.float8_e4m3fn:
        raise RuntimeError("w1 and w2 must be float8_e4m3fn")
    if w1_scale.shape != (e, n // 128, k // 128):
        raise RuntimeError("w1_scale must be [E, N/128, K/128]")
    if w2_scale.shape != (e, k // 128, n // 256):
        raise RuntimeError("w2_scale must be [E, K/128, N/256]")
    if w1_scale.dtype != torch.float32 or w2_scale.dtype != torch.float32:
        raise RuntimeError("weight scales must be float32")
    if topk_ids.dim() != 2 or topk_ids.shape[0] != m:
        raise RuntimeError("topk_ids must be [M, top_k]")
    if topk_weights.shape != topk_ids.shape:
        raise RuntimeError("topk_weights must have the shape of topk_ids")
    weights = (w1, w1_scale, w2, w2_scale)
    for i, t in enumerate(weights):
        if not t.is_contiguous():
            raise RuntimeError(f"{('w1', 'w1_scale', 'w2', 'w2_scale')[i]} must be contiguous")
    for i, t in enumerate((*weights, topk_weights, topk_ids)):
        if t.device != dev:
            raise RuntimeError(f"{('w1', 'w1_scale', 'w2', 'w2_scale', 'topk_weights', 'topk_ids')[i]} must be on {dev}")

def _up(n: int) -> int:
    return (n + 255) & ~255


def _through_c_abi(hidden, w1, w1_scale, w2, w2_scale, topk_weights, topk_ids, block_m, block_n, warp_n, stages, scaling) -> None:
    """What the torch operator does, on the C library alone."""
    _check_layer_arguments(hidden, w1, w1_scale, w2, w2_scale, topk_weights, topk_ids)
    m, k = hidden.shape
    e, n, _ = w1.shape
    ids, wts = topk_ids.to(torch.int32).contiguous(), topk_weights.to(torch.float32).contiguous()
    top_k, dev = ids.shape[1], hidden.device
    total = m * top_k + e * (block_m - 1)
    ws_bytes = capi.align_workspace_bytes(m * top_k, e)
    x_s = _up(m * k)                                        # one allocation, its pieces 256-byte aligned
    sorted_ids = x_s + _up(m * (k // 128) * 4)
    expert_ids = sorted_ids + _up(total * 4)
    num_post_pad = expert_ids + _up((total + block_m - 1) // block_m * 4)
    ws = num_post_pad + 256
    buf = torch.empty(ws + ws_bytes, dtype=torch.uint8, device=dev)
    base = buf.data_ptr()
    with torch.cuda.device(dev) if dev.index != torch.cuda.current_device() else contextlib.nullcontext():
        capi.fused_experts(hidden.data_ptr(), base, base + x_s, w1.data_ptr(), w1_scale.data_ptr(), w2.data_ptr(),
                           w2_scale.data_ptr(), ids.data_ptr(), wts.data_ptr(), top_k, m, k, n, e, base + sorted_ids,
                           base + expert_ids, base + num_post_pad, base + ws if ws_bytes else 0, block_m, block_n, warp_n, stages,
                           scaling, torch.cuda.current_stream(dev).cuda_stream)


def _operator():
    try:
        load_torch_op()
    except ImportError:
        return _through_c_abi
    return torch.ops.alpha_moe._fused_experts.default


_fused_experts = _operator()


@torch.compiler.disable
def _fused_experts_outside_graphs(*args) -> None:
    """For torch.compile: the call (in place) stays outside its graphs."""
    _fused_experts(*args)


def fused_experts_impl(hidden_states: torch.Tensor, w1: torch.Tensor, w1_scale: torch.Tensor, w2: torch.Tensor,
                       w2_scale: torch.Tensor, topk_weights: torch.Tensor, topk_ids: torch.Tensor,
                       routed_scaling_factor: float | None = None, block_shape=(128, 128),
                       config: dict | str | None = None) -> torch.Tensor:
    """hidden_states bf16 [M,K] (overwritten with the result); w1 fp8 [E,2I,K] gate/up interleaved by 8 with
    w1_scale [E,2I/128,K/128] interleaved by 1; w2 fp8 [E,K,I], w2_scale [E,K/128,I/128]; topk_ids int32 [M,top_k],
    topk_weights f32 [M,top_k].  `config`: a knob dict, a table path, or None for $ALPHA_MOE_CONFIG."""
    if tuple(block_shape) != (128, 128):
        raise ValueError("only 128 x 128 block scales are supported (the operator's scale layout)")
    if not hidden_states.is_cuda:
        _check_layer_arguments(hidden_states, w1, w1_scale, w2, w2_scale, topk_weights, topk_ids)
        raise RuntimeError("hidden_states must be a CUDA tensor (there is no CPU implementation)")
    args = (hidden_states, w1, w1_scale, w2, w2_scale, topk_weights, topk_ids)
    try:
        if isinstance(config, dict):
            conf = config
        else:
            path = config or os.getenv("ALPHA_MOE_CONFIG")
            if not path:
                raise RuntimeError("no knob table: pass config= or set ALPHA_MOE_CONFIG")
            conf = get_best_config(path, hidden_states.size(0))
        knobs = conf["block_m"], conf["block_n"], conf["warp_n"], conf["stages"]
    except Exception:
        _check_layer_arguments(*args)        # a tensor that is refused comes before a table that is not there
        raise
    call = _fused_experts_outside_graphs if torch.compiler.is_compiling() else _fused_experts
    try:
        call(*args, *knobs, float(routed_scaling_factor or 1.0))
    except RuntimeError as err:
        raise capi.error_of(err)
    return hidden_states
