"""The two layer operators on either side of ``chunk_kda`` in a Kimi-Linear block (fla/layers/kda.py:147-165, 191, 306):

* ``short_conv`` -- the short causal depthwise convolution (+ SiLU) applied to the q / k / v projections; call surface of
  flash-linear-attention's ``causal_conv1d`` (fla/modules/convolution.py) for the arguments a KDA layer uses;
* ``rms_norm_gated`` -- the gated RMS norm applied to the attention output, ``rmsnorm(x) * weight * act(g)``; call
  surface of ``rms_norm_gated`` (fla/modules/fused_norm_gate.py:846-869) without residual / bias.

Both are differentiable (one streaming sm_100a kernel each way, autograd and launches in the host extension,
csrc/host/host_layer_ops.cpp). No Triton, no fallback."""
from __future__ import annotations

import torch

from .. import _native
from ..utils import get_varlen_tables


@torch.compiler.disable
def short_conv(x, weight, bias=None, initial_state=None, output_final_state=False, activation="silu", cu_seqlens=None,
               cu_seqlens_cpu=None):
    """Causal depthwise convolution over time, then SiLU (``activation`` ``"silu"``/``"swish"``) or nothing (``None``).

    x: ``[B, T, D]`` bf16 (``B == 1`` with ``cu_seqlens``); weight: ``[D, W]``, ``W <= 4`` (a ``[D, 1, W]`` conv1d weight
    is accepted), tap ``W - 1`` multiplies the current token; bias: ``[D]`` or None; initial_state: ``[N, D, W]`` -- the
    last ``W`` inputs of a previous call, newest last -- or None; with ``output_final_state`` the same record for this
    call is returned. Returns ``(y, final_state)``. Gradients flow to x, weight and bias."""
    assert activation in (None, "silu", "swish"), "activation must be None, 'silu' or 'swish'."
    tab = None if cu_seqlens is None else get_varlen_tables(cu_seqlens, cu_seqlens_cpu).native
    return _native.host().short_conv(x, weight, bias, initial_state, output_final_state, activation is not None, tab)


@torch.compiler.disable
def rms_norm_gated(x, g, weight, activation="sigmoid", eps=1e-6):
    """``x * rsqrt(mean(x^2, -1) + eps) * weight * act(g)`` with ``act`` = ``"sigmoid"`` (what the KDA layer uses) or
    ``"swish"``/``"silu"`` (``g * sigmoid(g)``). x, g: ``[..., D]`` bf16, D in {128, 256, 512, 1024}; weight ``[D]``.
    Gradients flow to x, g and weight."""
    assert activation in ("sigmoid", "swish", "silu"), "activation must be 'sigmoid', 'swish' or 'silu'."
    return _native.host().rms_norm_gated(x, g, weight, activation != "sigmoid", eps)
