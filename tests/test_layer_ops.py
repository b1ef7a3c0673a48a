"""The short causal convolution and the gated RMS norm around chunk_kda: the oracle against torch's own conv1d with
left padding (CPU), and the CUDA operators against the oracle (GPU), forward, carried cache and gradients. bf16 in and
out: tolerances 4e-3 relative RMS for outputs and input gradients, 1e-2 for the parameter gradients (sums over all
tokens of bf16-rounded upstream gradients)."""
import pytest
import torch
import torch.nn.functional as F

from oracle.layer_ops import rms_norm_gated_ref, short_conv_ref
from oracle.naive_kda import err_ratio


def test_conv_oracle_is_left_padded_conv1d():
    gen = torch.Generator().manual_seed(0)
    x, w, b = torch.randn(2, 37, 16, generator=gen), torch.randn(16, 4, generator=gen), torch.randn(16, generator=gen)
    y, final = short_conv_ref(x, w, b, activation=None)
    ref = F.conv1d(x.transpose(1, 2), w.unsqueeze(1), b, padding=3, groups=16)[..., :37].transpose(1, 2)
    assert err_ratio(ref, y) < 1e-6
    assert torch.equal(final, x[:, -4:].transpose(1, 2))
    # continuing from the cache equals running the whole sequence at once
    y1, c1 = short_conv_ref(x[:, :20], w, b)
    y2, _ = short_conv_ref(x[:, 20:], w, b, initial_state=c1)
    y_all, _ = short_conv_ref(x, w, b)
    assert err_ratio(y_all, torch.cat([y1, y2], 1)) < 1e-6
    # packed sequences are independent
    cu = torch.tensor([0, 5, 37])
    yp, _ = short_conv_ref(x[:1], w, b, cu_seqlens=cu)
    assert err_ratio(short_conv_ref(x[:1, 5:], w, b)[0], yp[:, 5:]) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("W,bias,act,varlen", [(4, False, "silu", False), (4, True, "silu", True), (3, True, None, False),
                                               (2, False, "silu", True)])
def test_short_conv_matches_oracle(W, bias, act, varlen):
    from cula_b200.kda import short_conv
    gen = torch.Generator().manual_seed(1)
    B, T, D = (1, 333, 256) if varlen else (2, 200, 128)
    cu = torch.tensor([0, 1, 70, 198, 333], dtype=torch.int32) if varlen else None
    N = 4 if varlen else B
    x = torch.randn(B, T, D, generator=gen).to(torch.bfloat16)
    w, b = 0.5 * torch.randn(D, W, generator=gen), (0.1 * torch.randn(D, generator=gen) if bias else None)
    cache = torch.randn(N, D, W, generator=gen)
    dy = torch.randn(B, T, D, generator=gen).to(torch.bfloat16)
    ref_in = [x.float().requires_grad_(True), w.clone().requires_grad_(True)] + ([b.clone().requires_grad_(True)] if bias else [])
    y_ref, f_ref = short_conv_ref(ref_in[0], ref_in[1], ref_in[2] if bias else None, cache, act, cu)
    (y_ref * dy.float()).sum().backward()
    dev = [x.cuda().requires_grad_(True), w.cuda().requires_grad_(True)] + ([b.cuda().requires_grad_(True)] if bias else [])
    y, final = short_conv(dev[0], dev[1], dev[2] if bias else None, initial_state=cache.cuda(), output_final_state=True,
                          activation=act, cu_seqlens=None if cu is None else cu.cuda())
    y.backward(dy.cuda())
    torch.cuda.synchronize()
    assert err_ratio(y_ref.detach(), y.detach().float().cpu()) < 4e-3
    assert err_ratio(f_ref.detach(), final.cpu()) < 1e-6
    assert err_ratio(ref_in[0].grad, dev[0].grad.float().cpu()) < 4e-3
    assert err_ratio(ref_in[1].grad, dev[1].grad.cpu()) < 1e-2
    if bias:
        assert err_ratio(ref_in[2].grad, dev[2].grad.cpu()) < 1e-2


@pytest.mark.gpu
def test_short_conv_prefill_then_continue():
    """The final cache of one call is the initial cache of the next: two halves equal the whole sequence, bit for bit."""
    from cula_b200.kda import short_conv
    gen = torch.Generator().manual_seed(2)
    x = torch.randn(2, 300, 128, generator=gen).to(torch.bfloat16).cuda()
    w = torch.randn(128, 4, generator=gen).cuda()
    y_all, c_all = short_conv(x, w, output_final_state=True)
    y1, c1 = short_conv(x[:, :130].contiguous(), w, output_final_state=True)
    y2, c2 = short_conv(x[:, 130:].contiguous(), w, initial_state=c1, output_final_state=True)
    torch.cuda.synchronize()
    assert torch.equal(y_all, torch.cat([y1, y2], 1)) and torch.equal(c_all, c2)


@pytest.mark.gpu
@pytest.mark.parametrize("D,act", [(128, "sigmoid"), (128, "swish"), (256, "sigmoid"), (1024, "swish")])
def test_rms_norm_gated_matches_oracle(D, act):
    from cula_b200.kda import rms_norm_gated
    gen = torch.Generator().manual_seed(3)
    shape = (2, 77, 3, D)
    x, g = (torch.randn(*shape, generator=gen).to(torch.bfloat16) for _ in range(2))
    w = 1.0 + 0.1 * torch.randn(D, generator=gen)
    dy = torch.randn(*shape, generator=gen).to(torch.bfloat16)
    ref_in = [x.float().requires_grad_(True), g.float().requires_grad_(True), w.clone().requires_grad_(True)]
    y_ref = rms_norm_gated_ref(*ref_in, activation=act, eps=1e-5)
    (y_ref * dy.float()).sum().backward()
    dev = [x.cuda().requires_grad_(True), g.cuda().requires_grad_(True), w.cuda().requires_grad_(True)]
    y = rms_norm_gated(*dev, activation=act, eps=1e-5)
    y.backward(dy.cuda())
    torch.cuda.synchronize()
    assert y.dtype == torch.bfloat16 and err_ratio(y_ref.detach(), y.detach().float().cpu()) < 4e-3
    assert err_ratio(ref_in[0].grad, dev[0].grad.float().cpu()) < 4e-3
    assert err_ratio(ref_in[1].grad, dev[1].grad.float().cpu()) < 4e-3
    assert err_ratio(ref_in[2].grad, dev[2].grad.cpu()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("D,W,tail", [(8, 1, 0), (72, 4, 5), (200, 3, 0), (64, 2, 1), (200, 4, 0)])
def test_short_conv_at_chunk_and_channel_edges(D, W, tail):
    """Channel counts that leave part of a warp idle, sequences that end on and around a batch of tokens, half a chunk (an empty second
    half, one shorter than the window) and a chunk, rows past the last packed token (zero, with zero gradient)."""
    from cula_b200.kda import short_conv
    lens = [1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 34, 35, 61, 63, 64, 65, 67, 95, 96, 97, 98, 99, 128]
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32)
    T, gen = int(cu[-1]), torch.Generator().manual_seed(4)
    x, dy = (torch.randn(1, T + tail, D, generator=gen).to(torch.bfloat16) for _ in range(2))
    w, b, cache = 0.5 * torch.randn(D, W, generator=gen), 0.1 * torch.randn(D, generator=gen), torch.randn(len(lens), D, W, generator=gen)
    ref = [x[:, :T].float().requires_grad_(True), w.clone().requires_grad_(True), b.clone().requires_grad_(True)]
    y_ref, f_ref = short_conv_ref(ref[0], ref[1], ref[2], cache, "silu", cu)
    (y_ref * dy[:, :T].float()).sum().backward()
    dev = [t.cuda().requires_grad_(True) for t in (x, w, b)]
    y, final = short_conv(dev[0], dev[1], dev[2], initial_state=cache.cuda(), output_final_state=True, cu_seqlens=cu.cuda())
    y.backward(dy.cuda())
    torch.cuda.synchronize()
    assert err_ratio(y_ref.detach(), y.detach()[:, :T].float().cpu()) < 4e-3 and not y[:, T:].any()
    assert err_ratio(f_ref.detach(), final.cpu()) < 1e-6
    assert err_ratio(ref[0].grad, dev[0].grad[:, :T].float().cpu()) < 4e-3 and not dev[0].grad[:, T:].any()
    for r, d in zip(ref[1:], dev[1:]):
        assert err_ratio(r.grad, d.grad.cpu()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("W", [1, 2, 3, 4])
def test_short_conv_does_not_depend_on_how_chunks_are_split(W):
    """Many chunks are taken whole, few in halves: the same rows come out to the bit."""
    from cula_b200.kda import short_conv
    gen = torch.Generator(device="cuda").manual_seed(W)
    x = torch.randn(1, 64 * 2400 + 37, 64, device="cuda", generator=gen).to(torch.bfloat16)
    w = torch.randn(64, W, device="cuda", generator=gen)
    whole, _ = short_conv(x, w)
    n = 64 * 5 + 33
    few, _ = short_conv(x[:, :n].contiguous(), w)
    assert torch.equal(whole[:, :n], few)
    tail, _ = short_conv(x[:, -n:].contiguous(), w)
    assert torch.equal(whole[:, W - 1 - n:], tail[:, W - 1:])


@pytest.mark.gpu
@pytest.mark.parametrize("words", [1, 2, 3, 4, 5, 1023, 1024, 1025, 1 << 20, (1 << 20) + 3])
def test_clear_writes_its_words_and_no_others(words):
    from cula_b200 import _native
    buf = torch.full((words + 8,), 7.0, device="cuda")
    assert _native.lib().cula_kda_clear(buf[4:].data_ptr(), 4 * words, torch.cuda.current_stream().cuda_stream) == 0
    assert not buf[4:-4].any() and bool((buf[:4] == 7).all() and (buf[-4:] == 7).all())


@pytest.mark.gpu
@pytest.mark.parametrize("D", [128, 256, 512, 1024])
@pytest.mark.parametrize("R", [1, 3, 8, 9, 4099])
def test_rms_norm_gated_row_remainders(R, D):
    from cula_b200.kda import rms_norm_gated
    gen = torch.Generator().manual_seed(6)
    x, g, dy = (torch.randn(R, D, generator=gen).to(torch.bfloat16) for _ in range(3))
    w = 1.0 + 0.1 * torch.randn(D, generator=gen)
    ref = [x.float().requires_grad_(True), g.float().requires_grad_(True), w.clone().requires_grad_(True)]
    y_ref = rms_norm_gated_ref(*ref, activation="swish")
    (y_ref * dy.float()).sum().backward()
    dev = [t.cuda().requires_grad_(True) for t in (x, g, w)]
    y = rms_norm_gated(*dev, activation="swish")
    y.backward(dy.cuda())
    torch.cuda.synchronize()
    assert err_ratio(y_ref.detach(), y.detach().float().cpu()) < 4e-3
    for r, d, tol in zip(ref, dev, (4e-3, 4e-3, 1e-2)):
        assert err_ratio(r.grad, d.grad.float().cpu()) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [None, 1])
def test_short_conv_over_more_chunks_than_a_grid_dimension_takes(lens):
    """270,000 chunks, of one long sequence or of as many sequences of one token, forward and backward (no activation: both are
    weighted sums of shifted rows, exact but for the rounding of the results)."""
    from cula_b200.kda import short_conv
    n, gen = 270_000, torch.Generator(device="cuda").manual_seed(0)
    T = 64 * n if lens is None else n
    x = torch.randn(1, T, 8, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_(True)
    w = torch.randn(8, 2, device="cuda", generator=gen).requires_grad_(True)
    dy = torch.randn(1, T, 8, device="cuda", generator=gen).to(torch.bfloat16)
    cu = None if lens is None else torch.arange(n + 1, dtype=torch.int32)
    y, _ = short_conv(x, w, activation=None, cu_seqlens=None if cu is None else cu.cuda(), cu_seqlens_cpu=cu)
    dx, dw = torch.autograd.grad(y, [x, w], dy)
    far = 0.0 if cu is not None else 1.0                      # a sequence of one token has no neighbours
    xf, dyf, w0, w1 = x.detach().float(), dy.float(), w.detach()[:, 0], w.detach()[:, 1]
    y_ref = w1 * xf + far * w0 * F.pad(xf, (0, 0, 1, 0))[:, :T]
    dx_ref = w1 * dyf + far * w0 * F.pad(dyf, (0, 0, 0, 1))[:, 1:]
    dw_ref = torch.stack([far * (F.pad(xf, (0, 0, 1, 0))[:, :T].double() * dyf).sum((0, 1)), (xf.double() * dyf).sum((0, 1))], -1)
    assert err_ratio(y_ref, y.detach()) < 4e-3 and err_ratio(dx_ref, dx) < 4e-3
    # sums of T products of size 1 in fp32, by one atomic per four half chunks or sequences: as many roundings of up to 2^-24 of a sum that
    # walks to a few sqrt(T), which add up like their square root (8: a few times that walk, and four sigma)
    adds = T / 128 if cu is None else T / 4
    assert float((dw_ref - dw).abs().max()) < 8 * T ** 0.5 * adds ** 0.5 * 2.0 ** -24


def layer_chain(T, H, seed):
    """Leaves on the device and a function of them: every layer operator, forward and backward, as (results, gradients) in launch order."""
    from cula_b200.kda import fused_beta_sigmoid, fused_kda_gate, rms_norm_gated, short_conv
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    bf = lambda *s: rn(*s).to(torch.bfloat16)  # noqa: E731
    leaves = [bf(1, T, H * 128), 0.3 * rn(H * 128, 4), 0.1 * rn(H * 128), bf(1, T, H, 128), bf(1, T, H), rn(H), rn(H * 128), bf(1, T, H, 128),
              bf(1, T, H, 128), 1 + 0.1 * rn(128)]
    leaves = [t.requires_grad_(True) for t in leaves]
    up = [bf(1, T, H * 128), rn(1, T, H, 128), rn(1, T, H), bf(1, T, H, 128)]

    def run():
        x, w, b, g, beta, A_log, dt_bias, o, og, nw = leaves
        outs = [short_conv(x, w, b)[0], fused_kda_gate(g, A_log, dt_bias, lower_bound=-5.0), fused_beta_sigmoid(beta), rms_norm_gated(o, og, nw)]
        return outs, torch.autograd.grad(outs, leaves, up)

    return leaves, up, run


SUMMED = (1, 2, 5, 6, 9)          # gradients that atomics add up: the order of the additions is not fixed


def same(a, b):
    outs = all(torch.equal(x, y) for x, y in zip(a[0], b[0]))
    return outs and all(err_ratio(x, y) < 1e-5 if i in SUMMED else torch.equal(x, y) for i, (x, y) in enumerate(zip(a[1], b[1])))


@pytest.mark.gpu
@pytest.mark.parametrize("T,H", [(1, 1), (100, 3), (2048, 8)])
def test_layer_operators_launched_behind_one_another_equal_ones_waited_for(T, H):
    """Each kernel is launched while the one before it drains: passes queued without a pause, in memory that the passes before have just
    given back (results dropped at once), have the results of passes that start on an idle device."""
    chains = [layer_chain(T, H, seed) for seed in range(3)]
    alone = []
    for _, _, run in chains:
        torch.cuda.synchronize()
        alone.append(run())
    torch.cuda.synchronize()
    for _ in range(3):
        for _, _, run in chains:
            run()
    queued = [run() for _ in range(3) for _, _, run in chains]
    torch.cuda.synchronize()
    for i, r in enumerate(queued):
        assert same(alone[i % 3], r), i


@pytest.mark.gpu
def test_layer_operators_are_capturable_in_a_cuda_graph():
    """A pass of all of them, with its cleared buffers and early launches, replays on other values: equal to calls outside a graph."""
    leaves, up, run = layer_chain(300, 3, 0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = run()
    for seed in (1, 2):
        other = layer_chain(300, 3, seed)
        with torch.no_grad():
            for dst, src in zip([*leaves, *up], [*other[0], *other[1]]):
                dst.copy_(src)
        for _ in range(2):               # twice: the sums start from zero each time
            graph.replay()
        torch.cuda.synchronize()
        assert same(other[2](), replayed), seed


@pytest.mark.gpu
def test_a_refused_launch_leaves_no_error_behind():
    """The legacy stream takes no launch while a blocking stream is being captured: the call returns that error, and whoever asks the
    runtime next (torch, after its own next kernel) does not find it a second time. Buffer and sizes are real: were it not refused, it
    would run."""
    import ctypes

    from cula_b200 import _native
    runtime, lib = ctypes.CDLL("libcudart.so.12"), _native.lib()          # the runtime that the library and torch share
    buf = torch.full((1024,), 7.0, device="cuda")
    torch.cuda.synchronize()
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert runtime.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert runtime.cudaStreamBeginCapture(stream, 2) == 0                  # (relaxed)
    rc = lib.cula_kda_clear(buf.data_ptr(), 4096, None)
    left = runtime.cudaPeekAtLastError()
    runtime.cudaStreamEndCapture(stream, ctypes.byref(graph))              # the refusal has ended the capture as well
    runtime.cudaGetLastError()
    assert runtime.cudaStreamDestroy(stream) == 0
    assert rc > 0 and left == 0
    assert bool((buf == 7).all())
    assert lib.cula_kda_clear(buf.data_ptr(), 4096, torch.cuda.current_stream().cuda_stream) == 0 and not buf.any()
