"""``fused_kda_gate`` and ``fused_beta_sigmoid``: the layer-side activations that sit next to ``chunk_kda`` in a
Kimi-Linear block, for callers that do not let ``chunk_kda`` activate the gate itself (``use_gate_in_kernel=False``).
Same call surface and autograd behaviour as flash-linear-attention's functions of the same names
(fla/ops/kda/gate.py:321-345 and :431), which callers of the reference use around ``cula.kda.chunk_kda``.
One streaming sm_100a kernel each way, autograd and launches in the host extension (csrc/host/host_layer_ops.cpp); no Triton,
no fallback."""
from __future__ import annotations

import torch

from .. import _native


@torch.compiler.disable
def fused_kda_gate(g, A_log, dt_bias=None, lower_bound=None, output_dtype=torch.float32):
    """``-exp(A_log)[:, None] * softplus(g + dt_bias)`` for ``g`` ``[..., H, K]``, or, with ``lower_bound``,
    ``lower_bound * sigmoid(exp(A_log)[:, None] * (g + dt_bias))``. Differentiable in g, A_log and dt_bias."""
    assert output_dtype in (torch.bfloat16, torch.float32), "output_dtype must be bfloat16 or float32."
    return _native.host().kda_gate(g, A_log, dt_bias, lower_bound, output_dtype == torch.float32)


def fused_beta_sigmoid(x):
    """``sigmoid(x)`` in fp32 with autograd (fla/ops/kda/gate.py:431)."""
    return _native.host().beta_sigmoid(x)
