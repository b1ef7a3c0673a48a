"""Single-token KDA decode against a pool of fp32 states: ``kda_decode`` and
``fused_sigmoid_gating_delta_rule_update`` with the reference's signatures
(cula/ops/kda_decode.py:1794-2096). Checks, output and the one launch of ``kda_decode_kernel`` are in the host
extension (csrc/host/host_attention.cpp); the state pool is updated in place. There is no fallback: without the CUDA library the call raises."""
from __future__ import annotations

from .. import _native


def _canonical_layout(state_layout):
    lay = "vk" if state_layout is None else str(state_layout).lower()
    if lay not in ("vk", "kv"):
        raise ValueError(f"state_layout must be 'vk' or 'kv', got {state_layout!r}")
    return lay


def kda_decode(A_log, dt_bias, q, k, v, a, b, initial_state_source, initial_state_indices, cu_seqlens=None, scale=None,
               use_qk_l2norm_in_kernel=True, softplus_beta=1.0, softplus_threshold=20.0, out=None, state_layout="vk"):
    """Dense decode: q/k ``(N, 1, H, 128)``, v ``(N, 1, HV, V)``, a ``(N, 1, HV, 128)``, b ``(N, 1, HV)``.
    Varlen decode: the same with the first two axes swapped (``(1, N, ...)``; a / b may drop the leading 1).
    ``initial_state_source``: ``(pool, HV, V, K)`` for ``state_layout="vk"`` (default) or ``(pool, HV, K, V)`` for
    ``"kv"``, fp32, updated in place; None means zero states that are not kept. ``initial_state_indices``: int32
    ``[N]`` pool slots (negative = skip the sequence) or None for slot = sequence. ``cu_seqlens`` is accepted for
    signature compatibility: with one token per sequence it carries no information. Returns ``o`` shaped like ``v``
    in q's dtype (cula/ops/kda_decode.py:1845-2096)."""
    kv = state_layout == "kv" or (state_layout != "vk" and _canonical_layout(state_layout) == "kv")
    return _native.host().decode(A_log, dt_bias, q, k, v, a, b, initial_state_source, initial_state_indices, scale,
                                 use_qk_l2norm_in_kernel, softplus_beta, softplus_threshold, out, kv)


def fused_sigmoid_gating_delta_rule_update(A_log, a, dt_bias, softplus_beta, softplus_threshold, q, k, v, b,
                                           initial_state_source, initial_state_indices, scale=None,
                                           use_qk_l2norm_in_kernel=False, cu_seqlens=None, is_kda=False, out=None,
                                           state_layout="vk"):
    """Argument order of the reference's public decode entry (cula/ops/kda_decode.py:1794-1842)."""
    if not is_kda:
        raise NotImplementedError("cuLA fused decode currently supports only is_kda=True mode")
    return kda_decode(A_log=A_log, dt_bias=dt_bias, q=q, k=k, v=v, a=a, b=b, initial_state_source=initial_state_source,
                      initial_state_indices=initial_state_indices, cu_seqlens=cu_seqlens, scale=scale,
                      use_qk_l2norm_in_kernel=use_qk_l2norm_in_kernel, softplus_beta=softplus_beta,
                      softplus_threshold=softplus_threshold, out=out, state_layout=state_layout)
