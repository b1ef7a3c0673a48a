"""The work a user of this framework has it do, as timed cases: decode steps against a state pool, prefill of single,
batched, packed and very long sequences, training steps (forward and backward) with the gate activated in the kernel or
by the caller, the scalar-gate variant, and the operators that surround the attention call in a layer.

A case is a dict of plain values. ``kind`` names the entry point:

  decode   ``kda_decode``: one token of each of ``N`` sequences, ``H`` query/key heads, ``HV`` value heads
  prefill  ``chunk_kda`` without gradients: ``B`` sequences of ``T`` tokens, or ``N`` packed ones of ``T`` tokens in all
  train    ``chunk_kda``, forward and backward
  gdn      ``chunk_gated_delta_rule``, forward and backward
  layer    short convolutions of q, k, v, gate and beta activation, gated RMS norm: forward and backward

``gate`` is ``"safe"`` (raw bf16 gate input, lower-bound activation in the kernel, q/k normalised in the kernel),
``"softplus"`` (the same with the softplus activation) or ``"pre"`` (fp32 log decays and unit q/k rows made by the
caller). ``states``: initial states go in and final states come out.
"""
import math

import torch
import torch.nn.functional as F

from cula_b200.gdn import chunk_gated_delta_rule
from cula_b200.kda import chunk_kda, fused_beta_sigmoid, fused_kda_gate, kda_decode, rms_norm_gated, short_conv

D = 128
LOWER_BOUND = -5.0
MOST_TRAIN = 4 * 8192 * 32          # tokens x heads of the largest training step
MOST_PREFILL = 65536 * 32           # tokens x heads of the largest prefill


def listed():
    return [
        # interactive generation: one sequence, one token; nothing but latency
        dict(name="decode_one", kind="decode", N=1, H=32, HV=32, layout="vk", indexed=False, fp32_gate=False),
        # a serving step with an odd number of live sequences in a shuffled pool, grouped value heads, (K, V) states
        dict(name="decode_odd_kv", kind="decode", N=33, H=16, HV=32, layout="kv", indexed=True, fp32_gate=True),
        # a serving step at a full batch
        dict(name="decode_full", kind="decode", N=256, H=32, HV=32, layout="vk", indexed=True, fp32_gate=False),
        # the next turn of a chat: a short ragged prompt continued from a state
        dict(name="prefill_short", kind="prefill", B=1, T=500, N=0, H=32, gate="safe", beta="bf16", states=True),
        # the batch the benchmark times
        dict(name="prefill_batch", kind="prefill", B=2, T=2048, N=0, H=32, gate="safe", beta="bf16", states=True),
        # many prompts of uneven length packed into one call
        dict(name="prefill_packed", kind="prefill", B=1, T=65536, N=64, H=32, gate="safe", beta="logit", states=False),
        # one long document: a single chain of a thousand chunks
        dict(name="prefill_long", kind="prefill", B=1, T=65536, N=0, H=32, gate="safe", beta="bf16", states=True),
        # a small model or a debugging run: few heads, a ragged length, every gradient, gate made by the caller
        dict(name="train_small", kind="train", B=2, T=1000, N=0, H=3, gate="pre", beta="fp32", states=True, keep=False),
        # fine-tuning on packed documents, intermediates kept instead of recomputed
        dict(name="train_packed", kind="train", B=1, T=8192, N=17, H=32, gate="pre", beta="bf16", states=True, keep=True),
        # pre-training: the largest step of the benchmark
        dict(name="train_large", kind="train", B=4, T=8192, N=0, H=32, gate="safe", beta="bf16", states=False, keep=False),
        # the scalar-gate layer of the same size as the benchmark's batch
        dict(name="gdn_train", kind="gdn", B=2, T=2048, N=0, H=32, gate="softplus", beta="bf16", states=False, keep=False),
        # what surrounds the attention call in a layer, in training
        dict(name="layer_train", kind="layer", B=2, T=2048, H=32, W=4, activation="sigmoid"),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "prefill", "train", "train", "gdn", "layer"])
    if kind == "decode":
        H = rng.choice([4, 8, 16, 32])
        return dict(kind=kind, N=_spread(rng, 1, 256), H=H, HV=min(32, H * rng.choice([1, 1, 2])),
                    layout=rng.choice(["vk", "vk", "kv"]), indexed=rng.random() < 0.7, fp32_gate=rng.random() < 0.3)
    if kind == "layer":
        H = rng.choice([4, 8, 16, 32])
        B = _spread(rng, 1, 4)
        return dict(kind=kind, B=B, T=_spread(rng, 32, 16384 * 32 // (B * H)), H=H, W=rng.choice([4, 4, 3, 2]),
                    activation=rng.choice(["sigmoid", "sigmoid", "swish"]))
    H = rng.choice([2, 3, 4, 8, 16, 32, 32, 64])
    most = MOST_PREFILL if kind == "prefill" else MOST_TRAIN
    N = _spread(rng, 2, 64) if rng.random() < 0.4 else 0
    if N:
        B, T = 1, _spread(rng, max(64, 8 * N), min(65536, most // H))
    else:
        B = _spread(rng, 1, 8)
        T = _spread(rng, 17, min(65536, most // (B * H)))
    case = dict(kind=kind, B=B, T=T, N=N, H=H,
                gate=rng.choice(["safe", "safe", "pre", "softplus"]) if kind != "gdn" else rng.choice(["softplus", "pre"]),
                beta=rng.choice(["bf16", "fp32"] if kind == "gdn" else ["bf16", "fp32", "logit"]), states=rng.random() < 0.6)
    if kind != "prefill":
        case["keep"] = rng.random() < 0.3
    return case


def _lengths(total, n, gen):
    """n uneven lengths (each at least 1) that add up to total."""
    w = (0.8 * torch.randn(n, generator=gen, device=gen.device)).exp().double().cpu()
    cuts = (torch.cumsum(w, 0) / w.sum() * (total - n)).floor().long() + torch.arange(1, n + 1)
    cuts[-1] = total
    return torch.cat([torch.zeros(1, dtype=torch.int64), cuts]).to(torch.int32)


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))

    def rn(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32).to(dtype)

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=gen, device=dev)

    s = dict(case)
    if case["kind"] == "decode":
        N, H, HV = case["N"], case["H"], case["HV"]
        pool = N + N // 4 + 1 if case["indexed"] else N
        gdt = torch.float32 if case["fp32_gate"] else torch.bfloat16
        s.update(q=rn(N, 1, H, D, dtype=torch.bfloat16), k=rn(N, 1, H, D, dtype=torch.bfloat16),
                 v=rn(N, 1, HV, D, dtype=torch.bfloat16), a=rn(N, 1, HV, D, dtype=gdt), b=rn(N, 1, HV, dtype=gdt),
                 A_log=uni(1.0, 4.0, HV).log(), dt_bias=uni(-6.0, 0.0, HV * D), pool=0.1 * rn(pool, HV, D, D),
                 slots=torch.randperm(pool, generator=gen, device=dev)[:N].to(torch.int32) if case["indexed"] else None)
        return s
    B, T, H = case["B"], case["T"], case["H"]
    if case["kind"] == "layer":
        bf = torch.bfloat16
        leaf = lambda t: t.requires_grad_(True)  # noqa: E731
        s.update(x=[leaf(rn(B, T, H * D, dtype=bf)) for _ in range(3)],
                 w=[leaf(0.3 * rn(H * D, case["W"])) for _ in range(3)],
                 raw_g=leaf(rn(B, T, H, D, dtype=bf)), raw_b=leaf(rn(B, T, H, dtype=bf)),
                 A_log=leaf(uni(1.0, 4.0, H).log()), dt_bias=leaf(uni(-6.0, 0.0, H * D)),
                 o=leaf(rn(B, T, H, D, dtype=bf)), og=leaf(rn(B, T, H, D, dtype=bf)), nw=leaf(1.0 + 0.1 * rn(D)))
        s["up"] = [rn(B, T, H * D, dtype=bf) for _ in range(3)] + [rn(B, T, H, D), rn(B, T, H), rn(B, T, H, D, dtype=bf)]
        return s
    n_seqs = case["N"] or B
    per_head = case["kind"] == "gdn"
    gshape = (B, T, H) if per_head else (B, T, H, D)
    q, k, v = (rn(B, T, H, D, dtype=torch.bfloat16) for _ in range(3))
    A_log = dt_bias = None
    if case["gate"] == "pre":
        q, k = F.normalize(q, dim=-1), F.normalize(k, dim=-1)
        g = (F.logsigmoid(rn(*gshape) + 1.0) / 4.0).clamp(-5.0, 0.0)      # decays from a few tokens to dozens
    else:
        # a trained layer's channels forget at very different rates: the biases spread over weak and strong decays
        g = (0.5 * rn(*gshape)).to(torch.bfloat16)
        A_log = uni(1.0, 2.0, H).log()
        dt_bias = uni(-7.0, 0.0, H) if per_head else uni(-7.0, 0.0, H * D)
    beta = rn(B, T, H)
    if case["beta"] != "logit":
        beta = beta.sigmoid()
    beta = beta.to(torch.float32 if case["beta"] == "fp32" else torch.bfloat16)
    h0 = 0.5 * rn(n_seqs, H, D, D) if case["states"] else None
    s.update(q=q, k=k, v=v, g=g, beta=beta, A_log=A_log, dt_bias=dt_bias, h0=h0, cu=None, cu_cpu=None,
             beta_logit=case["beta"] == "logit")
    if case["N"]:
        s["cu_cpu"] = _lengths(T, case["N"], gen)
        s["cu"] = s["cu_cpu"].to(dev)
    if case["kind"] != "prefill":
        s["leaves"] = [t for t in (q, k, v, g, beta, A_log, dt_bias, h0) if t is not None]
        for t in s["leaves"]:
            t.requires_grad_(True)
        s["do"] = rn(B, T, H, D, dtype=torch.bfloat16)
        s["dht"] = rn(n_seqs, H, D, D) if case["states"] else None
    return s


def _attend(s):
    kw = dict(initial_state=s["h0"], output_final_state=s["states"], cu_seqlens=s["cu"], cu_seqlens_cpu=s["cu_cpu"],
              disable_recompute=bool(s.get("keep", False)), use_qk_l2norm_in_kernel=s["gate"] != "pre")
    if s["gate"] != "pre":
        kw.update(use_gate_in_kernel=True, A_log=s["A_log"], dt_bias=s["dt_bias"])
    if s["kind"] == "gdn":
        return chunk_gated_delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"], **kw)
    if s["gate"] == "safe":
        kw.update(safe_gate=True, lower_bound=LOWER_BOUND)
    return chunk_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], use_beta_sigmoid_in_kernel=s["beta_logit"], **kw)


def run(state):
    s = state
    if s["kind"] == "decode":
        o = kda_decode(A_log=s["A_log"], dt_bias=s["dt_bias"], q=s["q"], k=s["k"], v=s["v"], a=s["a"], b=s["b"],
                       initial_state_source=s["pool"], initial_state_indices=s["slots"], state_layout=s["layout"])
        return [o, s["pool"]]
    if s["kind"] == "layer":
        outs = [short_conv(x, w, activation="silu")[0] for x, w in zip(s["x"], s["w"])]
        outs.append(fused_kda_gate(s["raw_g"], s["A_log"], s["dt_bias"], lower_bound=LOWER_BOUND))
        outs.append(fused_beta_sigmoid(s["raw_b"]))
        outs.append(rms_norm_gated(s["o"], s["og"], s["nw"], activation=s["activation"]))
        leaves = [*s["x"], *s["w"], s["raw_g"], s["raw_b"], s["A_log"], s["dt_bias"], s["o"], s["og"], s["nw"]]
        grads = torch.autograd.grad(outs, leaves, s["up"])
        return [*(t.detach() for t in outs), *grads]
    if s["kind"] == "prefill":
        with torch.no_grad():
            return list(_attend(s))
    o, ht = _attend(s)
    outs, ups = ([o, ht], [s["do"], s["dht"]]) if s["states"] else ([o], [s["do"]])
    grads = torch.autograd.grad(outs, s["leaves"], ups)
    return [*(t.detach() for t in outs), *grads]


def work(case):
    H = case["H"]
    if case["kind"] == "decode":
        N, HV = case["N"], case["HV"]
        e = 4 if case["fp32_gate"] else 2
        per = 2 * 4 * D * D + e * (D + 1) + 2 * 2 * D            # the state both ways, gate and beta input, v and o
        return dict(bytes=N * (HV * per + H * 2 * 2 * D) + HV * 4 * (D + 1), flops=N * HV * 7 * D * D)
    th = case["B"] * case["T"] * H
    if case["kind"] == "layer":
        # forward: every input and output once; backward: inputs again, upstream gradients, gradients
        conv, gate, norm = 3 * 2 * D * (2 + 3), D * (2 + 4 + 2 + 4 + 2), 2 * D * (3 + 5)
        return dict(bytes=th * (conv + gate + norm + 4 * 5), flops=th * D * (3 * 60 + 40 + 50))
    bb = 4 if case["beta"] == "fp32" else 2
    gb = (4 if case["gate"] == "pre" else 2) * (1 if case["kind"] == "gdn" else D)
    st = 4 * D * D * H * (case["N"] or case["B"]) if case["states"] else 0
    fwd_bytes, fwd_flops = th * (3 * 2 * D + gb + bb + 2 * D) + 2 * st, th * 11 * D * D
    if case["kind"] == "prefill":
        return dict(bytes=fwd_bytes, flops=fwd_flops)
    # a training step reads the inputs twice, writes o, reads do and writes the gradients
    return dict(bytes=fwd_bytes + th * (3 * 2 * D + gb + bb) + th * (3 * 2 * D + gb + bb + 2 * D) + 3 * st, flops=3 * fwd_flops)


def tolerance(case):
    # bf16 results of fp32 sums whose operands went through fp16 or tf32 tensor-core products; the streaming operators
    # and the decode step differ by one rounding of their bf16 results
    if case["kind"] in ("decode", "layer"):
        return dict(rel=4e-3)
    return dict(rel=5e-3) if case["kind"] == "prefill" else dict(rel=1e-2)
