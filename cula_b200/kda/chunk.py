"""``chunk_kda``: chunkwise Kimi Delta Attention on B200, same call surface as the reference's
``cula.kda.chunk_kda`` (cula/kda/chunk.py:217-412).

Argument checks, output allocation, autograd and the C-ABI launches on the current torch stream are in the host extension
(csrc/host/host_attention.cpp): in Python they cost 70 us (forward) to 300 us (forward + backward) per call. All arithmetic
happens in the sm_100a kernels of libcula_kda.so; there is no Triton, no FLA dispatch and no CPU fallback.
"""
from __future__ import annotations

import torch

from .. import _native
from ..utils import CHUNK, get_varlen_tables

GATE_NONE, GATE_SOFTPLUS, GATE_LOWER_BOUND = 0, 1, 2


def __getattr__(name):
    if name == "FORWARD_CALLS":     # how many forward orchestrations have run in this process (tests count recomputations)
        return _native.host().forward_calls()
    raise AttributeError(name)


def check_status(device=None):
    """Synchronise and raise if any kernel on ``device`` reported a problem (a bounded wait that gave up, a bad
    state-pool index, an intermediate outside the fp16 range). Every operator call also looks, without waiting, at what
    kernels that have already finished reported: the status word lives in pinned host memory, which the kernels write
    directly when they have something to say."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    torch.cuda.synchronize(device)
    _native.host().poll_status(torch.cuda.current_device() if device.index is None else device.index)


def _status_ptr(device):
    """Address of the device's status word, as the C ABI takes it."""
    return _native.host().status_ptr(torch.cuda.current_device() if device.index is None else device.index)


def _ptr(t):
    return None if t is None else t.data_ptr()


def _f32(t):
    return None if t is None else t.float().contiguous()


def _gate_mode(use_gate_in_kernel, safe_gate, lower_bound):
    if not use_gate_in_kernel:
        return GATE_NONE
    # the lower-bound (sigmoid) form whenever a lower bound is given, as kda_gate_chunk_cumsum does
    # (fla/ops/kda/gate.py:509-548 keys on ``lower_bound is not None`` alone)
    return GATE_LOWER_BOUND if lower_bound is not None else GATE_SOFTPLUS


def _tables(cu_seqlens, cu_seqlens_cpu):
    return None if cu_seqlens is None else get_varlen_tables(cu_seqlens, cu_seqlens_cpu).native


def _segments(q):
    """One long sequence: few scan CTAs, many dependent steps -> the pieces its scan is cut into (see `cp.auto_segments`). Packed
    batches and batches of a few long sequences are not cut, nor are the scans of a backward pass: they run one chain per
    sequence and head, however few there are."""
    if q.dim() != 4 or q.shape[0] != 1 or q.shape[1] < 4096 or not q.is_cuda:      # cheap first look; `auto_segments` decides
        return None
    from .cp import auto_segments, segment_bounds, segment_tables
    num_chunks = (q.shape[1] + CHUNK - 1) // CHUNK
    P = auto_segments(num_chunks, q.shape[2], q.device)
    return segment_tables(segment_bounds(q.shape[1], num_chunks, P), q.device).segments if P > 1 else None


def chunk_kda_fwd(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens, cu_seqlens_cpu,
                  use_qk_l2norm_in_kernel, use_gate_in_kernel, safe_gate, lower_bound, A_log, dt_bias,
                  store_states=False, store_akk=False, store_for_backward=False, want_output=True, beta_logit=False):
    """Forward orchestration without autograd (the role of cula/kda/chunk_fwd.py:39-152), on contiguous tensors. Returns a
    dict with o, final_state and the intermediates kept for backward."""
    return _native.host().forward(
        q, k, v, g, beta, float(scale), initial_state, output_final_state, _tables(cu_seqlens, cu_seqlens_cpu),
        bool(use_qk_l2norm_in_kernel), _gate_mode(use_gate_in_kernel, safe_gate, lower_bound),
        float(lower_bound if lower_bound is not None else 0.0), _f32(A_log), _f32(dt_bias), store_states, store_akk,
        store_for_backward, want_output, beta_logit, None)


def chunk_kda_bwd(q, k, v, g, beta, scale, initial_state, do, dht, cu_seqlens, cu_seqlens_cpu,
                  use_qk_l2norm_in_kernel, use_gate_in_kernel, safe_gate, lower_bound, A_log, dt_bias, saved=None,
                  beta_logit=False):
    """Backward orchestration without autograd (the role of cula/kda/chunk_bwd.py:432-604). ``saved`` holds the forward
    intermediates (tiles, akk, mkk, h32, vnew) when they were kept; otherwise they are recomputed here, as the
    reference does by default (cula/kda/chunk_bwd.py:459-500)."""
    if saved is None:
        saved = chunk_kda_fwd(q, k, v, g, beta, scale, initial_state, False, cu_seqlens, cu_seqlens_cpu,
                              use_qk_l2norm_in_kernel, use_gate_in_kernel, safe_gate, lower_bound, A_log, dt_bias,
                              store_for_backward=True, want_output=False, beta_logit=beta_logit)
    return _native.host().backward(
        q, k, v, g, beta, float(scale), initial_state is not None, do, dht, _tables(cu_seqlens, cu_seqlens_cpu),
        bool(use_qk_l2norm_in_kernel), _gate_mode(use_gate_in_kernel, safe_gate, lower_bound),
        float(lower_bound if lower_bound is not None else 0.0), _f32(A_log), _f32(dt_bias), saved, beta_logit)


@torch.compiler.disable
def chunk_kda(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
              use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False, cu_seqlens=None, cu_seqlens_cpu=None,
              safe_gate=False, lower_bound=None, disable_recompute=False, return_intermediate_states=False,
              cp_context=None, use_beta_sigmoid_in_kernel=False, **kwargs):
    r"""Chunkwise KDA forward (+ autograd backward).

    Args mirror ``cula.kda.chunk_kda`` (cula/kda/chunk.py:218-346):
        q, k: ``[B, T, H, 128]`` bf16.  v: ``[B, T, H, 128]`` bf16.
        g: ``[B, T, H, 128]``; the natural-log decay (fp32 or bf16) when ``use_gate_in_kernel=False``,
            else the raw gate input, activated in-kernel with ``A_log`` ``[H]`` and optional ``dt_bias``
            ``[H*128]`` passed as keyword arguments.
        beta: ``[B, T, H]`` bf16 or fp32.
        scale: defaults to ``128 ** -0.5``.
        initial_state: ``[N, H, 128, 128]`` fp32 (N sequences) or None.
        output_final_state: also return the ``[N, H, 128, 128]`` fp32 final state.
        use_qk_l2norm_in_kernel: L2-normalise q and k rows in-kernel.
        safe_gate / lower_bound: with ``use_gate_in_kernel`` selects
            ``lower_bound * sigmoid(exp(A_log) * (g + dt_bias))``; lower_bound must lie in [-5, 0).
        cu_seqlens: int32 ``[N+1]`` for a packed batch (then B must be 1); cu_seqlens_cpu: optional host copy.
        disable_recompute: keep forward intermediates for backward instead of recomputing them.
        return_intermediate_states: inference only; also return h ``[B, NT, H, 128, 128]`` bf16.
        use_beta_sigmoid_in_kernel: (extension) ``beta`` holds raw logits; ``sigmoid`` is applied in-kernel and the
            backward pass returns the gradient w.r.t. the logits, so the activated beta never round-trips HBM (the
            fusion of ``fused_beta_sigmoid`` into the call).
        cp_context: a :class:`cula_b200.kda.cp.KDACPContext` (process group of the context-parallel ranks); the call
            is then this rank's shard of ONE sequence and runs through ``chunk_kda_cp`` (the reference takes
            flash-linear-attention's ``FLACPContext`` here, cula/kda/chunk.py:348-355).

    Numeric range: the chunk-local intermediates w, u, kg, qg, Aqk travel as fp16 (the reference uses bf16), so
    ``|v|``, ``|beta v|``, ``|scale q|`` and ``|scale q k|`` must stay below 65504; q and k are unrestricted when
    ``use_qk_l2norm_in_kernel`` is set, and otherwise rows of any length that this allows. Decays of more than about 5.4
    (natural log, per token) on 16 tokens in a row lose the contributions inside such a block. A value that leaves the range is reported through the device
    status word (``check_status``; also raised by the next ``chunk_kda`` call on the device).

    Returns ``(o, final_state)`` (``final_state`` is None unless requested).
    Raises ValueError / AssertionError on the same conditions as the reference (cula/kda/chunk.py:348-388).
    """
    if cp_context is not None:
        from .cp import chunk_kda_cp
        assert cu_seqlens is None, "context parallelism takes this rank's shard of one sequence, not a packed batch"
        assert not return_intermediate_states, "return_intermediate_states is not supported for context parallelism"
        return chunk_kda_cp(q, k, v, g, beta, scale=scale, initial_state=initial_state,
                            output_final_state=output_final_state, use_qk_l2norm_in_kernel=use_qk_l2norm_in_kernel,
                            use_gate_in_kernel=use_gate_in_kernel, safe_gate=safe_gate, lower_bound=lower_bound,
                            group=cp_context.group, segments=getattr(cp_context, "segments", None), **kwargs)
    A_log = dt_bias = None
    if use_gate_in_kernel:
        assert "A_log" in kwargs, "A_log must be provided when use_gate_in_kernel=True."
        A_log, dt_bias = kwargs["A_log"], kwargs.get("dt_bias")
    if cu_seqlens is None:
        tables, segments = None, _segments(q)
    else:
        if q.shape[0] != 1:
            raise ValueError(
                f"The batch size is expected to be 1 rather than {q.shape[0]} when using `cu_seqlens`."
                f"Please flatten variable-length inputs before processing.")
        if initial_state is not None and initial_state.shape[0] != len(cu_seqlens) - 1:
            raise ValueError(
                f"The number of initial states is expected to be equal to the number of input sequences, "
                f"i.e., {len(cu_seqlens) - 1} rather than {initial_state.shape[0]}.")
        tables, segments = get_varlen_tables(cu_seqlens, cu_seqlens_cpu).native, None
    return _native.host().attend(q, k, v, g, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel,
                                 use_gate_in_kernel, A_log, dt_bias, tables, safe_gate, lower_bound, disable_recompute,
                                 return_intermediate_states, use_beta_sigmoid_in_kernel, False, segments)
