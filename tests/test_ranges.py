"""Inputs at the ends of what the operators accept: decays, magnitudes and forms that the other tests do not reach.
Forward, final state and gradients against the CPU oracle; tolerances as in test_kda_bwd.py unless stated."""
import pytest
import torch
import torch.nn.functional as F

from oracle.naive_kda import chunk_kda_oracle, err_ratio

NAMES = ("q", "k", "v", "g", "beta", "h0")


def make(T=200, H=2, seed=0, B=1):
    gen = torch.Generator().manual_seed(seed)

    def rn(*s):
        return torch.randn(*s, generator=gen)

    return dict(q=rn(B, T, H, 128), k=rn(B, T, H, 128), v=rn(B, T, H, 128), g=-0.02 * torch.rand(B, T, H, 128, generator=gen),
                beta=torch.rand(B, T, H, generator=gen), h0=0.3 * rn(B, H, 128, 128), do=rn(B, T, H, 128), dht=rn(B, H, 128, 128))


def unit(x):
    return F.normalize(x, dim=-1)


def forward_backward(c, scale=None, l2=True, reference=True, dtype=torch.float32):
    """(results of the kernels, results of the oracle in ``dtype``): o, ht and the gradients of NAMES, by name."""
    from cula_b200.kda import check_status, chunk_kda
    c = {n: t.to(torch.bfloat16) if n in ("q", "k", "v", "beta", "do") else t for n, t in c.items()}
    dev = {n: c[n].cuda().requires_grad_(True) for n in NAMES}
    o, ht = chunk_kda(*(dev[n] for n in NAMES[:5]), scale=scale, initial_state=dev["h0"], output_final_state=True, use_qk_l2norm_in_kernel=l2)
    grads = torch.autograd.grad([o, ht], list(dev.values()), [c["do"].cuda(), c["dht"].cuda()])
    torch.cuda.synchronize()
    check_status()
    got = dict(o=o, ht=ht, **{"d" + n: g for n, g in zip(NAMES, grads)})
    got = {n: t.detach().float().cpu() for n, t in got.items()}
    if not reference:
        return got, None
    ref = {n: c[n].to(dtype).requires_grad_(True) for n in NAMES}
    ro, rh = chunk_kda_oracle(*(ref[n] for n in NAMES[:5]), scale=scale, initial_state=ref["h0"], output_final_state=True,
                              use_qk_l2norm_in_kernel=l2, dtype=dtype)
    rg = torch.autograd.grad([ro, rh], list(ref.values()), [c["do"].to(dtype), c["dht"].to(dtype)])
    return got, dict(o=ro.detach(), ht=rh.detach(), **{"d" + n: g for n, g in zip(NAMES, rg)})


def assert_close(got, ref, **tol):
    bad = []
    for n, r in ref.items():
        e = err_ratio(r, got[n])
        if not e <= tol.get(n, {"o": 5e-3, "ht": 2e-3, "dg": 2e-2, "dbeta": 2e-2}.get(n, 8e-3)):
            bad.append(f"{n} {e:.2e}")
    assert not bad, "; ".join(bad)


@pytest.mark.gpu
@pytest.mark.parametrize("l2", [True, False])
@pytest.mark.parametrize("decay", [7.0, 9.0, 30.0, 1000.0])
def test_decays_beyond_the_safe_range_stay_finite(decay, l2):
    """More than about 5.5 nats per token is past what the 16-row anchors carry: contributions inside a block are then lost (the
    reference does not accept such gates at all), but no factor may meet its inverse as 0 * inf, with normalised rows or without.
    The final state only needs the factors towards the end of the chunk, which are <= 1: it stays exact."""
    c = make(seed=1)
    c["g"] = torch.full_like(c["g"], -decay)
    if not l2:
        c["q"], c["k"] = unit(c["q"]), unit(c["k"])
    got, ref = forward_backward(c, l2=l2)
    assert torch.isfinite(got["o"]).all()
    assert err_ratio(ref["ht"], got["ht"]) <= 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("decay,magnitude,per_head", [(5.0, 1.0, False), (5.0, 300.0, False), (5.0, 300.0, True), (9.0, 300.0, False), (30.0, 1.0, False)])
def test_gradients_at_the_strongest_decays(decay, magnitude, per_head):
    """-5 nats on every token and channel, the end of the safe range: the factor of a 16-row block with itself is 2^116, and with
    values of a few hundred the sums that it scales are above 2^12. Beyond the safe range the gradients are not claimed to be
    accurate, but finite."""
    from cula_b200.gdn import chunk_gated_delta_rule
    c = make(seed=2)
    c["g"], c["v"], c["h0"] = torch.full_like(c["g"], -decay), magnitude * c["v"], magnitude * c["h0"]
    if per_head:
        expanded = c["g"]
        dev = {n: (c[n][..., 0] if n == "g" else c[n]).to(torch.float32 if n in ("g", "h0") else torch.bfloat16).cuda().requires_grad_(True) for n in NAMES}
        o, ht = chunk_gated_delta_rule(*(dev[n] for n in NAMES[:5]), initial_state=dev["h0"], output_final_state=True, use_qk_l2norm_in_kernel=True)
        grads = torch.autograd.grad([o, ht], list(dev.values()), [c["do"].to(torch.bfloat16).cuda(), c["dht"].cuda()])
        got = {n: t.detach().float().cpu() for n, t in dict(o=o, ht=ht, **{"d" + n: g for n, g in zip(NAMES, grads)}).items()}
        c["g"] = expanded
        _, ref = forward_backward(c)
        ref["dg"] = ref["dg"].sum(-1)
    else:
        got, ref = forward_backward(c)
    assert all(torch.isfinite(t).all() for t in got.values()), [n for n, t in got.items() if not torch.isfinite(t).all()]
    if decay <= 5:
        assert_close(got, ref)


@pytest.mark.gpu
def test_empty_batch():
    """B = 0: empty results, as for any operator of torch, with gradients wanted, kept states and a long T included."""
    from cula_b200.gdn import chunk_gated_delta_rule
    from cula_b200.kda import chunk_kda
    for T in (100, 8192):
        q, k, v = (torch.empty(0, T, 3, 128, dtype=torch.bfloat16, device="cuda") for _ in range(3))
        g, beta = torch.empty(0, T, 3, 128, device="cuda"), torch.empty(0, T, 3, device="cuda")
        o, ht = chunk_kda(q, k, v, g, beta, output_final_state=True)
        assert o.shape == (0, T, 3, 128) and ht.shape == (0, 3, 128, 128)
        with torch.inference_mode():
            o, ht, h = chunk_kda(q, k, v, g, beta, output_final_state=True, return_intermediate_states=True)
        assert h.shape == (0, (T + 63) // 64, 3, 128, 128)
        o, _ = chunk_gated_delta_rule(q.clone().requires_grad_(True), k, v, g[..., 0], beta)
        assert o.shape == (0, T, 3, 128) and o.requires_grad


@pytest.mark.gpu
def test_forward_mode_differentiation_is_refused():
    """No operator has a forward derivative: a dual tensor raises instead of losing its tangent."""
    import torch.autograd.forward_ad as fw

    from cula_b200.gdn import chunk_gated_delta_rule
    from cula_b200.kda import chunk_kda, fused_beta_sigmoid, fused_kda_gate, rms_norm_gated, short_conv
    c = {n: t.cuda().to(torch.float32 if n in ("g", "h0") else torch.bfloat16) for n, t in make(T=64).items()}
    c["q"], c["k"] = unit(c["q"]), unit(c["k"])
    weight, x = torch.ones(128, device="cuda"), c["v"].reshape(1, 64, 256)
    with fw.dual_level():
        def dual(t):
            return fw.make_dual(t, torch.ones_like(t))

        calls = [lambda n=n: chunk_kda(*(dual(c[m]) if m == n else c[m] for m in NAMES[:5])) for n in NAMES[:5]]
        calls += [lambda: chunk_kda(*(c[m] for m in NAMES[:5]), initial_state=dual(c["h0"])),
                  lambda: chunk_gated_delta_rule(dual(c["q"]), c["k"], c["v"], c["g"][..., 0], c["beta"]),
                  lambda: fused_kda_gate(dual(c["g"]), torch.zeros(2, device="cuda")), lambda: fused_beta_sigmoid(dual(c["beta"])),
                  lambda: short_conv(x, dual(torch.ones(256, 4, device="cuda"))), lambda: rms_norm_gated(c["q"], dual(c["k"]), weight)]
        for call in calls:
            with pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
                call()
        with torch.no_grad(), pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
            calls[0]()


@pytest.mark.gpu
def test_reverse_scan_of_a_packed_batch_does_not_depend_on_T():
    """Through the C ABI: T is the length of fixed-length sequences and means nothing beside d_cu_seqlens. Zero, a longest length
    and the packed total give the same bits, with full and ragged last chunks, and nothing past the packed rows is read."""
    from cula_b200 import _native
    from cula_b200.kda import check_status
    from cula_b200.kda.chunk import _status_ptr
    from cula_b200.utils import VarlenTables
    lens, H = [64, 1, 130, 0, 128, 63, 200], 2
    total = sum(lens)
    c = make(T=total, H=H, seed=3)
    d = {n: c[n].cuda().to(torch.float32 if n == "g" else torch.bfloat16) for n in ("q", "k", "v", "g", "beta")}
    do = torch.full((total + 64, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    do[:total] = c["do"][0]
    tab = VarlenTables(torch.tensor([0, *torch.tensor(lens).cumsum(0)], dtype=torch.int32).cuda())
    lib, nt, N, f32 = _native.lib(), tab.num_chunks * H, len(lens), dict(dtype=torch.float32, device="cuda")
    stream, status = torch.cuda.current_stream().cuda_stream, _status_ptr(do.device)
    pack = torch.empty(nt * lib.cula_kda_tile_pack_bytes(), dtype=torch.uint8, device="cuda")
    cu, ci, co = (t.data_ptr() for t in (tab.cu_seqlens, tab.chunk_indices, tab.chunk_offsets))
    _native.check(lib.cula_kda_fwd_intra(*(d[n].data_ptr() for n in ("q", "k", "v", "g")), 1, d["beta"].data_ptr(), 0, None, None, cu, ci, tab.num_chunks,
                                         0, H, 128 ** -0.5, 1, 0, 0.0, pack.data_ptr(), None, None, status, stream), "intra")
    gscale = torch.tensor([2.0, 0.5, 0, 0], **f32)
    dht, h0 = torch.randn(N, H, 128, 128, **f32), torch.randn(N, H, 128, 128, **f32)
    results = []
    for T in (total, 0, 200, -1):
        for both in (False, True):
            out = [torch.zeros(nt, 64, 128, dtype=torch.float16, device="cuda"), torch.zeros(nt, 128, 128, **f32), torch.zeros(N, H, 128, 128, **f32)]
            p = [t.data_ptr() for t in out]
            if both:
                vnew, h32 = torch.empty_like(out[0]), torch.empty_like(out[1])
                code = lib.cula_kda_bwd_both_scans(pack.data_ptr(), h0.data_ptr(), vnew.data_ptr(), h32.data_ptr(), do.data_ptr(), dht.data_ptr(),
                                                   gscale.data_ptr(), *p, cu, co, None, N, T, H, status, stream)
            else:
                code = lib.cula_kda_bwd_scan(pack.data_ptr(), do.data_ptr(), dht.data_ptr(), gscale.data_ptr(), *p, cu, co, None, N, T, H, status, stream)
            _native.check(code, "reverse scan")
            results.append(out)
    torch.cuda.synchronize()
    check_status()
    assert all(torch.isfinite(t).all() for t in results[0])
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,value", [("scale", 900.0), ("aligned_keys", 100.0), ("spread_keys", 100.0), ("small_keys", 1e-3)])
def test_the_scans_take_any_scale_and_key_length(kind, value):
    """The fp16 copies of the carried states are scaled by a bound that includes the largest |kg|, |qg|, |w| and decay: a large
    softmax scale with queries the keys do not see, keys far from unit length that all write to one channel or each to its own."""
    c, scale, l2 = make(seed=4), None, False
    if kind == "scale":            # queries orthogonal to the keys and gradients of one sign: the state gradient adds up scale * dO
        scale, l2 = value, True
        c["k"][..., 0], c["q"], c["do"], c["dht"] = 0, 0.01 * c["q"], c["do"].abs(), 0 * c["dht"]
        c["q"][..., 0] = 3
    else:
        c["k"] = unit(c["k"])
        if kind == "aligned_keys":
            c["k"] = torch.zeros_like(c["k"])
            c["k"][..., 0] = 1
            c["v"], c["h0"], c["beta"] = c["v"][:, :1].expand_as(c["v"]), 0 * c["h0"], torch.full_like(c["beta"], 0.6)
        elif kind == "spread_keys":
            c["k"] = F.one_hot(torch.arange(200) % 128, 128).float().view(1, 200, 1, 128).expand(1, 200, 2, 128)
        c["q"], c["k"], c["beta"] = unit(c["q"]), value * c["k"], 1.5 * c["beta"] / max(1, value ** 2)
    got, ref = forward_backward(c, scale=scale, l2=l2, dtype=torch.float64)
    # one key and one value over and over: what a token adds to the state falls to the few percent by which the state decays per
    # token, a difference of fp16 terms (2^-11 each) some 50 times as large, and dk and dg are proportional to it
    assert_close(got, ref, **({"dk": 5e-2, "dg": 1e-1} if kind == "aligned_keys" else {}))


@pytest.mark.gpu
@pytest.mark.parametrize("scale,gate", [(511.0, True), (513.0, True), (2e4, True), (2e4, False), (1e-3, False)])
def test_softmax_scale_up_to_the_fp16_range(scale, gate):
    """scale q k and scale q are stored as fp16, whose range is the limit; the operands of the Gram product must not end earlier."""
    from cula_b200.kda import check_status, chunk_kda
    c = make(seed=5)
    raw = (c["g"] * 100 - 2).to(torch.bfloat16)
    kw = dict(use_gate_in_kernel=True, safe_gate=True, lower_bound=-5.0, A_log=torch.zeros(2)) if gate else {}
    x = {n: c[n].to(torch.bfloat16) for n in ("q", "k", "v", "beta")}
    x["q"][..., 0], x["k"][..., 0] = 30, -30           # a channel that holds most of both rows
    args = [x["q"], x["k"], x["v"], raw if gate else c["g"], x["beta"]]
    ref, ref_h = chunk_kda_oracle(*args, scale=scale, initial_state=c["h0"], output_final_state=True, use_qk_l2norm_in_kernel=True,
                                  dtype=torch.float64, **kw)
    kw = {n: t.cuda() if isinstance(t, torch.Tensor) else t for n, t in kw.items()}
    o, ht = chunk_kda(*(t.cuda() for t in args), scale=scale, initial_state=c["h0"].cuda(), output_final_state=True, use_qk_l2norm_in_kernel=True, **kw)
    torch.cuda.synchronize()
    check_status()
    assert err_ratio(ref, o.cpu()) <= 5e-3 and err_ratio(ref_h, ht.cpu()) <= 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("growth", [0.05, 0.07])
def test_growing_states(growth):
    """Positive log decays (a factor of 88 over a chunk at 0.07) with normalised rows, every token with a key of its own: the column
    factors of the Gram product exceed 1 and must not be shifted towards the end of the fp16 range on top of that."""
    from cula_b200.gdn import chunk_gated_delta_rule
    from cula_b200.kda import check_status, chunk_kda
    c = make(seed=6)
    c["g"], c["h0"] = torch.full_like(c["g"], growth), 1e-2 * c["h0"]
    c["k"] = F.one_hot(torch.arange(200) % 128, 128).float().view(1, 200, 1, 128).expand(1, 200, 2, 128)
    c = {n: t.to(torch.bfloat16) if n in ("q", "k", "v", "beta") else t for n, t in c.items()}
    ref, ref_h = chunk_kda_oracle(*(c[n] for n in NAMES[:5]), initial_state=c["h0"], output_final_state=True, use_qk_l2norm_in_kernel=True,
                                  dtype=torch.float64)
    for fn, g in ((chunk_kda, c["g"]), (chunk_gated_delta_rule, c["g"][..., 0])):
        o, ht = fn(*(t.cuda() for t in (c["q"], c["k"], c["v"], g, c["beta"])), initial_state=c["h0"].cuda(), output_final_state=True,
                   use_qk_l2norm_in_kernel=True)
        torch.cuda.synchronize()
        check_status()
        assert err_ratio(ref, o.cpu()) <= 5e-3 and err_ratio(ref_h, ht.cpu()) <= 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("length,beta", [(1.0, 1e-3), (1.0, 1e-4), (300.0, 1.0), (3000.0, 1.0)])
def test_small_betas(length, beta):
    """Step sizes of 1e-5 and less, as keys of length 300 need them: beta rides on the fp16 operand (I + L)^-1, times a power of two
    where the whole tile is small. (u = beta v itself is stored in fp16: with unit keys 1e-4 is the end.)"""
    c = make(seed=7)
    c["q"], c["k"], c["beta"] = unit(c["q"]), length * unit(c["k"]), beta * c["beta"] / length ** 2
    if length == 1:
        c["h0"] = 0 * c["h0"]
    got, ref = forward_backward(c, l2=False, dtype=torch.float64)
    tol = {"ht": 4e-3, "dk": 1e-2} if length > 1000 else {}      # kg and u near opposite ends of fp16
    assert_close(got, ref, **tol)
