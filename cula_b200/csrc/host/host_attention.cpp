// chunk_kda / chunk_gated_delta_rule (forward and backward) and the decode step on the native host path.
#include "host_common.h"

#include <algorithm>
#include <cmath>

#include <torch/csrc/autograd/python_cpp_function.h>

namespace cula_host {

namespace {

std::atomic<int64_t> forward_calls{0};      // forward orchestrations run so far (recomputations included)

struct Options {        // everything that is not a tensor
    double scale = 1.0, lower_bound = 0.0;
    bool l2norm = false, beta_logit = false;
    int gate_mode = GATE_NONE;
};

// Side-by-side segments of one long sequence (fixed by the caller): their index tables
struct Segments {
    int64_t count = 1;
    Tables tab;
};

struct Forward {
    Tensor o, final_state, tiles, akk, mkk, h, h32, vnew;
    int64_t num_chunks = 0;
};

int g_flags(const Tensor& g) { return (is_f32(g) ? CULA_KDA_G_FP32 : 0) | (g.dim() == 3 ? CULA_KDA_G_PER_HEAD : 0); }
int beta_flags(const Tensor& beta, bool logit) { return (is_f32(beta) ? CULA_KDA_BETA_FP32 : 0) | (logit ? CULA_KDA_BETA_LOGIT : 0); }

// an output in the shape of `like`; rows past the packed tokens are zero
Tensor output_like(const Tensor& like, const Tables* tab) {
    Tensor t = device_empty(like.sizes(), like.options());
    if (tab && tab->total_tokens < like.size(1)) t.narrow(1, tab->total_tokens, like.size(1) - tab->total_tokens).zero_();
    return t;
}

// Scan + output of one sequence in `segs.count` side-by-side pieces: a transition scan over all but the last, a fold per
// boundary, then all pieces from their now known incoming states.
void segmented_scan(const Tensor& v, const OptTensor& h0, bool want_final, const Segments& segs, Forward& f, cudaStream_t stream, int* status) {
    const int64_t P = segs.count, H = v.size(2), T = v.size(1);
    const auto f32 = v.options().dtype(at::kFloat);
    Tensor C = device_empty({2, P, H, DIM, DIM}, f32);
    Tensor states = device_empty({P, H, DIM, DIM}, f32);
    const int64_t per = H * DIM * DIM;
    float *c = fptr(C), *m = c + P * per, *s = fptr(states);
    int *cu = iptr(segs.tab.cu_seqlens), *co = iptr(segs.tab.chunk_offsets);
    check(lib.cula_kda_cp_transition(ptr(f.tiles), c, m, cu, co, (int)(P - 1), (int)T, (int)H, status, stream), "cula_kda_cp_transition");
    if (h0.has_value()) states.select(0, 0).copy_(h0->reshape({H, DIM, DIM}));
    else states.select(0, 0).zero_();
    for (int64_t i = 1; i < P; ++i)
        check(lib.cula_kda_cp_fold(c + (i - 1) * per, m + (i - 1) * per, i == 1 && !h0.has_value() ? nullptr : s + (i - 1) * per, s + i * per, 1,
                                   (int)H, 0, stream), "cula_kda_cp_fold");
    f.o = device_empty(v.sizes(), v.options());
    Tensor ht = want_final ? device_empty({P, H, DIM, DIM}, f32) : Tensor();
    check(lib.cula_kda_fwd_scan(ptr(f.tiles), s, ptr(f.o), fptr(ht), nullptr, nullptr, nullptr, cu, co, iptr(segs.tab.seq_order), (int)P, (int)T,
                                (int)H, status, stream), "cula_kda_fwd_scan");
    if (want_final) f.final_state = ht.narrow(0, P - 1, 1);
}

// How to lay the two stages of a fixed-length batch over the GPU. The scan is a chain per (sequence, head) and needs one SM for each,
// the chunk-parallel stage takes whatever it is given; run after one another, the scan leaves the other SMs idle. So the chunks are
// cut into pieces, and a piece's chunk-parallel stage runs beside the scan of the piece before. Sizes for which the two just keep
// step form a geometric series; the first piece's chunk-parallel stage and the last one's scan are exposed. The times are measured,
// in us. Above half the SMs the scan leaves too little for this to gain (3 x 4096 x 32 heads: 456 -> 476 us).
// Both stages one after the other -> in these pieces, us, cold L2, with a bf16 gate / an fp32 gate / a gate per head:
//   1 x 4096 x 32 heads   230 -> 205     232 -> 209     206 -> 185        2 x 2048 x 32   177 -> 172     183 -> 178     155 -> 148
//   2 x 8192 x 32         644 -> 582     660 -> 599     558 -> 498        4 x 4096 x 16   331 -> 315     339 -> 332     290 -> 260
//   1 x 65536 x 32       3266 -> 2443   3335 -> 2525   2913 -> 2222       1 x 16384 x 48 1039 -> 896    1072 -> 929     908 -> 767
// The three kernels take 0.048, 0.050 and 0.038 us per tile (8192 tiles; 0.0535, 0.056 and 0.043 in launches of 2048). One rate serves all:
// planned with their rates at 8192 tiles, 2 x 2048 x 32 comes out 172 -> 180, others 1 % slower to 3 % faster, for other reasons than
// the plan can know.
// What keeps its intermediates (training that recomputes, B > 1 that does not) and packed batches have no pieces, and only B = 1
// without gradients or kept intermediates has segments: few long chains are left as they are there.
struct Plan {
    std::vector<int> pieces;      // chunks per piece
    double us = 0;
};
Plan plan_pieces(int64_t ctas, int64_t nc, int sms) {
    const double intra = ctas * 0.0535 * 148 / sms;                        // per chunk of every sequence, on the whole GPU
    const double scan = 1.6 + ctas / 128.0;                                // and its scan (more when many share the memory system)
    Plan best;
    best.pieces = {(int)nc};
    best.us = nc * (intra + scan);
    if (2 * ctas > sms) return best;
    const double ratio = std::min(1.5, scan / (intra * sms / (sms - ctas)));
    for (int n = 2; n <= 8; ++n) {
        double sum = 0, f = 1;
        for (int i = 0; i < n; ++i, f *= ratio) sum += f;
        Plan p;
        int64_t done = 0;
        f = 1;
        for (int i = 0; i < n; ++i, f *= ratio) {
            const int64_t c = i == n - 1 ? nc - done : std::llround(nc * f / sum);
            p.pieces.push_back((int)c);
            done += c;
        }
        if (*std::min_element(p.pieces.begin(), p.pieces.end()) < 4) break;
        p.us = p.pieces[0] * intra + nc * scan + 16 * (n - 1);      // 16: a tail and a ramp of the chunk-parallel stage, launches
        if (p.us < best.us) best = p;
    }
    return best;
}

// The upstream gradients and the power-of-two scale they are carried in.
struct Upstream {
    Tensor d_o, work;             // work: [0:2] = {s, 1/s}, [2] = running max (as bits)
    Tensor sums;                  // the atomically accumulated gradients of dt_bias (if any) and A_log, cleared
    OptTensor dht;
    int64_t n_dht() const { return dht.has_value() ? dht->numel() : 0; }
    unsigned int* amax() const { return reinterpret_cast<unsigned int*>(fptr(work) + 2); }
};
// (cleared in front of everything: between two kernels of the chain a launch would keep the second from being set up behind the first)
Upstream upstream(const Tensor& d_out, const OptTensor& d_final, const Tensor& q, const OptTensor& dt_bias, const Options& opt) {
    c10::cuda::CUDAGuard guard(q.device());
    const auto f32 = q.options().dtype(at::kFloat);
    const int64_t H = q.size(2);
    const bool bias = dt_bias.has_value() && dt_bias->defined();
    return {d_out.contiguous(), device_empty({4}, d_out.options().dtype(at::kFloat)),
            opt.gate_mode != GATE_NONE ? device_zeros({bias ? H + H * DIM : H}, f32, stream_of(q)) : Tensor(), contiguous_f32(d_final)};
}
void scale_gradients(const Upstream& u) {
    c10::cuda::CUDAGuard guard(u.d_o.device());
    check(lib.cula_kda_bwd_grad_scale(ptr(u.d_o), u.d_o.numel(), fptr(u.dht), u.n_dht(), u.amax(), fptr(u.work), stream_of(u.d_o)),
          "cula_kda_bwd_grad_scale");
}

// Forward orchestration (the role of cula/kda/chunk_fwd.py:39-152): the chunk-parallel stage writes one tile pack per
// (chunk, head); the scan consumes them, carries the fp32 state and writes o. All tensors contiguous; A_log, dt_bias fp32.
// recompute_for: in front of a backward pass. The scale of its upstream gradients is worked out beside the chunk-parallel stage, and of the
// scan only the buffers are made: backward_core launches it, beside the reverse scan.
Forward forward_core(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& h0,
                     const OptTensor& A_log, const OptTensor& dt_bias, const Options& opt, const Tables* tab, const Segments* segs, bool want_final,
                     bool store_states, bool store_akk, bool store_bwd, bool want_output, const Upstream* recompute_for = nullptr) {
    ++forward_calls;
    const bool leave_scan = recompute_for != nullptr;
    c10::cuda::CUDAGuard guard(q.device());
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2);
    cudaStream_t stream = stream_of(q);
    int* status = status_word(q.device().index());
    if (tab && tab->total_tokens > T)
        throw pybind11::value_error("cu_seqlens[-1]=" + std::to_string(tab->total_tokens) + " exceeds the " + std::to_string(T) + " packed tokens");
    Forward f;
    f.num_chunks = tab ? tab->num_chunks : B * ((T + CHUNK - 1) / CHUNK);
    const int64_t tiles = f.num_chunks * H, n_seqs = tab ? tab->n_seqs : B;
    int *cu = tab ? iptr(tab->cu_seqlens) : nullptr, *ci = tab ? iptr(tab->chunk_indices) : nullptr;
    int *co = tab ? iptr(tab->chunk_offsets) : nullptr, *so = tab ? iptr(tab->seq_order) : nullptr;
    const auto f32 = q.options().dtype(at::kFloat);
    f.tiles = device_empty({tiles * lib.cula_kda_tile_pack_bytes()}, q.options().dtype(at::kByte));
    if (store_akk || store_bwd) f.akk = device_empty({tiles, CHUNK, CHUNK}, f32);
    if (store_bwd) f.mkk = device_empty({tiles, CHUNK, CHUNK}, f32);
    // a batch of several sequences comes out piece by piece, which what is kept for later cannot
    if (!leave_scan && !tab && !store_states && !(store_akk && !store_bwd) && (B == 1 || !store_bwd)) {
        const Plan plan = plan_pieces(B * H, (T + CHUNK - 1) / CHUNK, at::cuda::getDeviceProperties(q.device().index())->multiProcessorCount);
        // side-by-side segments are the other way to fill the GPU, better with few heads (the two cross between 24 and 32)
        const double nc = (double)f.num_chunks, seg_us = segs ? nc * (H * 0.0535 + 2 * (1.6 + H / 128.0) / segs->count) + 10 * segs->count : 1e30;
        if (plan.pieces.size() > 1 && 1.06 * plan.us < seg_us) {
            if (want_output) f.o = device_empty(v.sizes(), v.options());
            if (want_final) f.final_state = device_empty({B, H, DIM, DIM}, f32);
            if (store_bwd) {
                f.h32 = device_empty({tiles, DIM, DIM}, f32);
                f.vnew = device_empty({tiles, CHUNK, DIM}, q.options().dtype(at::kHalf));
            }
            Tensor states = device_empty({2, B, H, DIM, DIM}, f32);
            check(lib.cula_kda_fwd_pieces(ptr(q), ptr(k), ptr(v), ptr(g), g_flags(g), ptr(beta), beta_flags(beta, opt.beta_logit), fptr(A_log),
                                          fptr(dt_bias), (int)B, (int)T, (int)H, (float)opt.scale, opt.l2norm, opt.gate_mode,
                                          (float)opt.lower_bound, ptr(f.tiles), fptr(f.akk), fptr(f.mkk), fptr(h0), ptr(f.o), fptr(f.final_state),
                                          ptr(f.vnew), fptr(f.h32), fptr(states), plan.pieces.data(), (int)plan.pieces.size(), status, stream),
                  "cula_kda_fwd_pieces");
            return f;
        }
    }
    if (recompute_for) {
        const Upstream& u = *recompute_for;
        check(lib.cula_kda_bwd_scale_and_intra(ptr(u.d_o), u.d_o.numel(), fptr(u.dht), u.n_dht(), u.amax(), fptr(u.work), ptr(q), ptr(k), ptr(v), ptr(g),
                                               g_flags(g), ptr(beta), beta_flags(beta, opt.beta_logit), fptr(A_log), fptr(dt_bias), cu, ci,
                                               (int)f.num_chunks, (int)T, (int)H, (float)opt.scale, opt.l2norm, opt.gate_mode, (float)opt.lower_bound,
                                               ptr(f.tiles), fptr(f.akk), fptr(f.mkk), status, stream), "cula_kda_bwd_scale_and_intra");
    } else {
        check(lib.cula_kda_fwd_intra(ptr(q), ptr(k), ptr(v), ptr(g), g_flags(g), ptr(beta), beta_flags(beta, opt.beta_logit), fptr(A_log),
                                     fptr(dt_bias), cu, ci, (int)f.num_chunks, (int)T, (int)H, (float)opt.scale, opt.l2norm, opt.gate_mode,
                                     (float)opt.lower_bound, ptr(f.tiles), fptr(f.akk), fptr(f.mkk), status, stream), "cula_kda_fwd_intra");
    }
    if (segs && segs->count > 1) {
        segmented_scan(v, h0, want_final, *segs, f, stream, status);
        return f;
    }
    if (want_output) f.o = output_like(v, tab);
    if (want_final) f.final_state = device_empty({n_seqs, H, DIM, DIM}, f32);
    if (store_states) f.h = device_empty({tiles, DIM, DIM}, q.options().dtype(at::kBFloat16));
    if (store_bwd) f.h32 = device_empty({tiles, DIM, DIM}, f32);
    if (store_states || store_bwd) f.vnew = device_empty({tiles, CHUNK, DIM}, q.options().dtype(at::kHalf));
    if (leave_scan) return f;
    check(lib.cula_kda_fwd_scan(ptr(f.tiles), fptr(h0), ptr(f.o), fptr(f.final_state), ptr(f.h), ptr(f.vnew), fptr(f.h32), cu, co, so, (int)n_seqs,
                                (int)T, (int)H, status, stream), "cula_kda_fwd_scan");
    return f;
}

struct Backward {
    Tensor dq, dk, dv, dg, dbeta, dA, dbias, dh0;
};

// Backward orchestration (the role of cula/kda/chunk_bwd.py:432-604) from the forward intermediates in `f`. With scan_left the
// forward scan of `f` (from h0) has not run yet: the reverse scan reads none of its results, so the two chains run side by side.
Backward backward_core(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& A_log,
                       const OptTensor& dt_bias, const Options& opt, const Tables* tab, const Forward& f, bool want_dh0, const Upstream& up,
                       bool scan_left = false, const OptTensor& h0 = {}) {
    c10::cuda::CUDAGuard guard(q.device());
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2);
    cudaStream_t stream = stream_of(q);
    int* status = status_word(q.device().index());
    const int64_t tiles = f.num_chunks * H, n_seqs = tab ? tab->n_seqs : B;
    int *cu = tab ? iptr(tab->cu_seqlens) : nullptr, *ci = tab ? iptr(tab->chunk_indices) : nullptr;
    int *co = tab ? iptr(tab->chunk_offsets) : nullptr, *so = tab ? iptr(tab->seq_order) : nullptr;
    const auto f32 = q.options().dtype(at::kFloat);
    const Tensor &d_o = up.d_o, &work = up.work;
    const OptTensor& dht = up.dht;
    Tensor dvn = device_empty({tiles, CHUNK, DIM}, q.options().dtype(at::kHalf)), ds = device_empty({tiles, DIM, DIM}, f32);
    Backward r;
    if (want_dh0) r.dh0 = device_empty({n_seqs, H, DIM, DIM}, f32);
    if (scan_left)
        check(lib.cula_kda_bwd_both_scans(ptr(f.tiles), fptr(h0), ptr(f.vnew), fptr(f.h32), ptr(d_o), fptr(dht), fptr(work), ptr(dvn), fptr(ds),
                                          fptr(r.dh0), cu, co, so, (int)n_seqs, (int)T, (int)H, status, stream), "cula_kda_bwd_both_scans");
    else
        check(lib.cula_kda_bwd_scan(ptr(f.tiles), ptr(d_o), fptr(dht), fptr(work), ptr(dvn), fptr(ds), fptr(r.dh0), cu, co, so, (int)n_seqs, (int)T,
                                    (int)H, status, stream), "cula_kda_bwd_scan");
    r.dv = output_like(v, tab);
    Tensor scratch = device_empty({tiles, lib.cula_kda_bwd_scratch_floats()}, f32);
    check(lib.cula_kda_bwd_dense(fptr(f.h32), fptr(ds), ptr(f.vnew), ptr(dvn), ptr(d_o), ptr(v), ptr(beta), beta_flags(beta, opt.beta_logit),
                                 fptr(f.akk), fptr(work), ptr(r.dv), fptr(scratch), cu, ci, (int)f.num_chunks, (int)T, (int)H, status, stream),
          "cula_kda_bwd_dense");
    r.dq = output_like(q, tab);
    r.dk = output_like(k, tab);
    r.dg = output_like(g, tab);
    r.dbeta = output_like(beta, tab);
    if (opt.gate_mode != GATE_NONE) {
        if (dt_bias.has_value() && dt_bias->defined()) r.dbias = part_of(up.sums, 0, {H * DIM});
        r.dA = part_of(up.sums, up.sums.numel() - H, {H});
    }
    check(lib.cula_kda_bwd_gated_checked(ptr(q), ptr(k), ptr(g), g_flags(g), ptr(beta), beta_flags(beta, opt.beta_logit), fptr(A_log), fptr(dt_bias),
                                         fptr(f.akk), fptr(f.mkk), fptr(scratch), fptr(work), ptr(r.dq), ptr(r.dk), ptr(r.dg), ptr(r.dbeta),
                                         fptr(r.dA), fptr(r.dbias), cu, ci, (int)f.num_chunks, (int)T, (int)H, (float)opt.scale, opt.l2norm,
                                         opt.gate_mode, (float)opt.lower_bound, status, stream), "cula_kda_bwd_gated");
    return r;
}

// ---------------------------------------------------------------------------------------------------------------------
// Autograd boundary (the role of cula/kda/chunk.py:28-214). Gradients flow to q, k, v, g, beta, A_log, dt_bias, h0.
// ---------------------------------------------------------------------------------------------------------------------
struct Call {
    Options opt;
    std::optional<Tables> tab;
    const Segments* segs = nullptr;
    bool want_final = false, keep = false;
};

class Attention : public torch::autograd::Function<Attention> {
public:
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                                                  const Tensor& g_in, const Tensor& beta_in, const OptTensor& A_log_in, const OptTensor& dt_bias_in,
                                                  const OptTensor& h0_in, const Call* call) {
        const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous(), g = g_in.contiguous(), beta = beta_in.contiguous();
        const OptTensor A_log = contiguous_f32(A_log_in), dt_bias = contiguous_f32(dt_bias_in);
        const OptTensor h0 = h0_in.has_value() ? OptTensor(h0_in->contiguous()) : OptTensor();
        const Options& o = call->opt;
        Forward f = forward_core(q, k, v, g, beta, h0, A_log, dt_bias, o, call->tab ? &*call->tab : nullptr, call->segs, call->want_final, false,
                                 false, call->keep, true);
        const Tensor none;
        ctx->save_for_backward({q, k, v, g, beta, A_log.value_or(none), dt_bias.value_or(none), h0.value_or(none)});
        ctx->saved_data["scale"] = o.scale;
        ctx->saved_data["flags"] = (int64_t)((o.l2norm ? 1 : 0) | (o.beta_logit ? 2 : 0) | (o.gate_mode << 2));
        ctx->saved_data["lower_bound"] = o.lower_bound;
        if (call->tab) {
            const Tables& t = *call->tab;
            ctx->saved_data["tab"] = std::vector<Tensor>{t.cu_seqlens, t.chunk_indices, t.chunk_offsets, t.seq_order};
            ctx->saved_data["tab_sizes"] = std::vector<int64_t>{t.n_seqs, t.num_chunks, t.total_tokens};
        }
        // kept intermediates are internal buffers nobody else can modify, so they ride on the node directly
        if (call->keep) ctx->saved_data["kept"] = std::vector<Tensor>{f.tiles, f.akk, f.mkk, f.h32, f.vnew};
        ctx->set_materialize_grads(false);
        if (f.final_state.defined()) return {f.o, f.final_state};
        return {f.o};
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        auto s = ctx->get_saved_variables();
        auto opt_of = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
        const Tensor &q = s[0], &k = s[1], &v = s[2], &g = s[3], &beta = s[4];
        const OptTensor A_log = opt_of(s[5]), dt_bias = opt_of(s[6]), h0 = opt_of(s[7]);
        Options o;
        const int64_t flags = ctx->saved_data["flags"].toInt();
        o.scale = ctx->saved_data["scale"].toDouble();
        o.lower_bound = ctx->saved_data["lower_bound"].toDouble();
        o.l2norm = flags & 1; o.beta_logit = flags & 2; o.gate_mode = (int)(flags >> 2);
        std::optional<Tables> tab;
        if (auto it = ctx->saved_data.find("tab"); it != ctx->saved_data.end()) {
            auto t = it->second.toTensorVector();
            auto n = ctx->saved_data["tab_sizes"].toIntVector();
            tab = Tables{t[0], t[1], t[2], t[3], n[0], n[1], n[2]};
        }
        const Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(v);
        const OptTensor dht = grads.size() > 1 && grads[1].defined() ? OptTensor(grads[1]) : OptTensor();
        const Upstream up = upstream(d_o, dht, q, dt_bias, o);
        Forward f;
        bool scan_left = false;
        if (auto it = ctx->saved_data.find("kept"); it != ctx->saved_data.end()) {
            auto t = it->second.toTensorVector();
            f.tiles = t[0]; f.akk = t[1]; f.mkk = t[2]; f.h32 = t[3]; f.vnew = t[4];
            f.num_chunks = tab ? tab->num_chunks : q.size(0) * ((q.size(1) + CHUNK - 1) / CHUNK);
            scale_gradients(up);
        } else {        // recomputed, as the reference does by default (cula/kda/chunk_bwd.py:459-500)
            f = forward_core(q, k, v, g, beta, h0, A_log, dt_bias, o, tab ? &*tab : nullptr, nullptr, false, false, false, true, false, &up);
            scan_left = true;
        }
        Backward b = backward_core(q, k, v, g, beta, A_log, dt_bias, o, tab ? &*tab : nullptr, f, h0.has_value(), up, scan_left, h0);
        if (b.dA.defined()) b.dA = shaped_like(b.dA, *A_log);
        if (b.dbias.defined()) b.dbias = shaped_like(b.dbias, *dt_bias);
        return {b.dq, b.dk, b.dv, b.dg, b.dbeta, b.dA, b.dbias, b.dh0, Tensor()};
    }
};

bool any_requires_grad(std::initializer_list<const Tensor*> ts, std::initializer_list<const OptTensor*> os) {
    for (const Tensor* t : ts) if (has_tangent(*t)) return true;
    for (const OptTensor* t : os) if (t->has_value() && has_tangent(**t)) return true;
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts) if (t->requires_grad()) return true;
    for (const OptTensor* t : os) if (t->has_value() && (*t)->requires_grad()) return true;
    return false;
}

void check_packed(const Tensor& q, const OptTensor& h0, int64_t n_seqs) {
    if (q.size(0) != 1)
        throw pybind11::value_error("The batch size is expected to be 1 rather than " + std::to_string(q.size(0)) +
                                    " when using `cu_seqlens`.Please flatten variable-length inputs before processing.");
    if (h0.has_value() && h0->size(0) != n_seqs)
        throw pybind11::value_error("The number of initial states is expected to be equal to the number of input sequences, i.e., " +
                                    std::to_string(n_seqs) + " rather than " + std::to_string(h0->size(0)) + ".");
}

// What chunk_kda checks before anything touches the device (cula/kda/chunk.py:348-388). n_seqs < 0: a fixed-length batch.
void check_kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& h0, int64_t n_seqs,
               bool gate_in_kernel, bool safe_gate, const std::optional<double>& lower_bound) {
    if (n_seqs >= 0) check_packed(q, h0, n_seqs);
    if (h0.has_value()) require(is_f32(*h0), "initial_state must be in float32.");
    if (safe_gate && gate_in_kernel) {
        if (!lower_bound.has_value())
            throw pybind11::value_error("`lower_bound` must be specified when `safe_gate=True` and `use_gate_in_kernel=True`.");
        if (!(-5 <= *lower_bound && *lower_bound < 0))
            throw pybind11::value_error("`lower_bound` must be in the safe range [-5, 0), got " + std::to_string(*lower_bound) + ".");
    }
    require(q.dim() == 4 && q.sizes() == k.sizes() && q.sizes() == g.sizes(), "q, k, g must have the same shape.");
    require(k.size(3) <= 256, "Currently we only support key headdim <=256 for KDA :-(");
    require(beta.sizes() == q.sizes().slice(0, 3), "beta must be of shape (batch size, seq len, num of head).");
    require(v.dim() == 4 && v.sizes().slice(0, 3) == q.sizes().slice(0, 3), "v must be of shape (batch size, seq len, num of head, head dim).");
    require(is_bf16(q) && is_bf16(k) && is_bf16(v), "q, k, v must be in bfloat16.");
    require(is_bf16(beta) || is_f32(beta), "beta must be in bfloat16 or float32.");
    require(q.size(3) == DIM && v.size(3) == DIM, "Currently we only support head dim of 128 for KDA");
    require(is_bf16(g) || is_f32(g), "g must be in bfloat16 or float32.");
    if (h0.has_value() && n_seqs < 0) require(h0->size(0) == q.size(0), "one initial state per batch entry is expected.");
}

void check_gdn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const OptTensor& h0, int64_t n_seqs) {
    if (n_seqs >= 0) check_packed(q, h0, n_seqs);
    require(is_bf16(q) && is_bf16(k) && is_bf16(v), "q, k, v must be in bfloat16.");
    require(q.dim() == 4 && v.dim() == 4 && q.sizes() == k.sizes() && q.size(3) == DIM && v.size(3) == DIM,
            "only head dim 128 is supported for keys and values");
    require(v.sizes().slice(0, 3) == q.sizes().slice(0, 3), "grouped value heads (HV > H) are not supported");
    require(g.sizes() == q.sizes().slice(0, 3) && beta.sizes() == q.sizes().slice(0, 3), "g and beta must be of shape (batch size, seq len, heads)");
    require((is_f32(g) || is_bf16(g)) && (is_f32(beta) || is_bf16(beta)), "g and beta must be in bfloat16 or float32.");
    if (h0.has_value()) require(is_f32(*h0), "initial_state must be in float32.");
}

// The whole call behind chunk_kda (`scalar_gate` false) and chunk_gated_delta_rule (true). Returns (o, final_state or None)
// or, with return_states, (o, final_state or None, h).
pybind11::tuple attend(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, std::optional<double> scale,
                       const OptTensor& h0, bool want_final, bool l2norm, bool gate_in_kernel, const OptTensor& A_log, const OptTensor& dt_bias,
                       const Tables* tab, bool safe_gate, std::optional<double> lower_bound, bool disable_recompute, bool return_states,
                       bool beta_logit, bool scalar_gate, const Segments* segs) {
    const int64_t n_seqs = tab ? tab->n_seqs : -1;
    if (scalar_gate) check_gdn(q, k, v, g, beta, h0, n_seqs);
    else check_kda(q, k, v, g, beta, h0, n_seqs, gate_in_kernel, safe_gate, lower_bound);
    assert_blackwell(q);
    poll_status(q.device().index());
    Call call;
    Options& o = call.opt;
    o.scale = scale.has_value() ? *scale : 1.0 / std::sqrt((double)DIM);
    // the lower-bound (sigmoid) form whenever a lower bound is given, as kda_gate_chunk_cumsum does
    // (fla/ops/kda/gate.py:509-548 keys on ``lower_bound is not None`` alone)
    o.gate_mode = !gate_in_kernel ? GATE_NONE : lower_bound.has_value() ? GATE_LOWER_BOUND : GATE_SOFTPLUS;
    o.lower_bound = lower_bound.value_or(0.0);
    o.l2norm = l2norm;
    o.beta_logit = beta_logit;
    if (tab) call.tab = *tab;
    call.want_final = want_final;
    const bool grad = any_requires_grad({&q, &k, &v, &g, &beta}, {&A_log, &dt_bias, &h0});
    call.keep = disable_recompute && grad;          // the intermediates are worth keeping only if a backward pass can follow
    call.segs = call.keep || return_states ? nullptr : segs;
    auto obj = [](const Tensor& t) -> pybind11::object { return t.defined() ? pybind11::cast(t) : pybind11::object(pybind11::none()); };
    if (grad && !return_states) {
        auto out = Attention::apply(q, k, v, g, beta, A_log, dt_bias, h0, (const Call*)&call);
        return pybind11::make_tuple(obj(out[0]), out.size() > 1 ? obj(out[1]) : pybind11::object(pybind11::none()));
    }
    at::NoGradGuard no_grad;
    Forward f = forward_core(q.contiguous(), k.contiguous(), v.contiguous(), g.contiguous(), beta.contiguous(),
                             h0.has_value() ? OptTensor(h0->contiguous()) : OptTensor(), contiguous_f32(A_log), contiguous_f32(dt_bias), o, tab,
                             call.segs, want_final, return_states, false, false, true);
    if (!return_states) return pybind11::make_tuple(obj(f.o), obj(f.final_state));
    require(c10::InferenceMode::is_enabled(), "return_intermediate_states is only allowed in inference mode");
    require(!disable_recompute, "return_intermediate_states must be used with disable_recompute=False");
    const int64_t B = q.size(0), H = q.size(2);
    Tensor h = f.h.view({tab ? 1 : B, tab ? f.num_chunks : (q.size(1) + CHUNK - 1) / CHUNK, H, DIM, DIM});
    return pybind11::make_tuple(obj(f.o), obj(f.final_state), obj(h));
}

// The forward and backward orchestrations on their own, for the context-parallel path.
pybind11::dict forward_dict(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale, const OptTensor& h0,
                            bool want_final, const Tables* tab, bool l2norm, int gate_mode, double lower_bound, const OptTensor& A_log,
                            const OptTensor& dt_bias, bool store_states, bool store_akk, bool store_bwd, bool want_output, bool beta_logit,
                            const Segments* segs) {
    at::NoGradGuard no_grad;
    Options o;
    o.scale = scale; o.lower_bound = lower_bound; o.l2norm = l2norm; o.beta_logit = beta_logit; o.gate_mode = gate_mode;
    Forward f = forward_core(q, k, v, g, beta, h0, A_log, dt_bias, o, tab, segs, want_final, store_states, store_akk, store_bwd, want_output);
    pybind11::dict d;
    auto put = [&](const char* n, const Tensor& t) { d[n] = t.defined() ? pybind11::cast(t) : pybind11::object(pybind11::none()); };
    put("o", f.o); put("final_state", f.final_state); put("tiles", f.tiles); put("akk", f.akk); put("mkk", f.mkk); put("h", f.h);
    put("h32", f.h32); put("vnew", f.vnew);
    d["num_chunks"] = f.num_chunks;
    return d;
}

pybind11::tuple backward_tuple(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale,
                               bool want_dh0, const Tensor& d_o, const OptTensor& dht, const Tables* tab, bool l2norm, int gate_mode,
                               double lower_bound, const OptTensor& A_log, const OptTensor& dt_bias, const pybind11::dict& saved, bool beta_logit) {
    at::NoGradGuard no_grad;
    Options o;
    o.scale = scale; o.lower_bound = lower_bound; o.l2norm = l2norm; o.beta_logit = beta_logit; o.gate_mode = gate_mode;
    Forward f;
    auto get = [&](const char* n) { return saved[n].cast<Tensor>(); };
    f.tiles = get("tiles"); f.akk = get("akk"); f.mkk = get("mkk"); f.h32 = get("h32"); f.vnew = get("vnew");
    f.num_chunks = saved["num_chunks"].cast<int64_t>();
    const Upstream up = upstream(d_o, dht, q, dt_bias, o);
    scale_gradients(up);
    Backward b = backward_core(q, k, v, g, beta, A_log, dt_bias, o, tab, f, want_dh0, up);
    auto obj = [](const Tensor& t) -> pybind11::object { return t.defined() ? pybind11::cast(t) : pybind11::object(pybind11::none()); };
    return pybind11::make_tuple(obj(b.dq), obj(b.dk), obj(b.dv), obj(b.dg), obj(b.dbeta), obj(b.dA), obj(b.dbias), obj(b.dh0));
}

std::string shape_text(const Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + ")";
}

// kda_decode (cula/ops/kda_decode.py:1845-2096): checks, output, one launch.
Tensor decode(const Tensor& A_log_in, const OptTensor& dt_bias_in, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& a_in,
              const Tensor& b_in, const OptTensor& state_in, const OptTensor& indices, std::optional<double> scale, bool l2norm,
              double softplus_beta, double softplus_threshold, const OptTensor& out_in, bool kv) {
    at::NoGradGuard no_grad;
    const int64_t Bq = q_in.size(0), Tq = q_in.size(1), H = q_in.size(2), K = q_in.size(3), HV = v_in.size(2), V = v_in.size(3);
    const int64_t N = indices.has_value() ? indices->size(0) : (Bq == 1 && Tq > 1 ? Tq : Bq);
    if (K != DIM) require(false, ("the decode kernel requires K=128, got " + std::to_string(K)).c_str());
    if (V % 32 != 0) require(false, ("the decode kernel requires V % 32 == 0, got V=" + std::to_string(V)).c_str());
    require(is_bf16(q_in) && is_bf16(k_in) && is_bf16(v_in), "q, k, v must be in bfloat16.");
    require(HV % H == 0, "the number of value heads must be a multiple of the number of q/k heads");
    require(Bq * Tq == N, "decode takes exactly one token per sequence");
    if (scale.has_value() && !(*scale > 0)) require(false, ("scale must be positive, got " + std::to_string(*scale)).c_str());
    assert_blackwell(q_in);
    c10::cuda::CUDAGuard guard(q_in.device());
    const int dev = q_in.device().index();
    const auto f32 = q_in.options().dtype(at::kFloat);
    Tensor state = state_in.has_value() ? *state_in : at::zeros({N, HV, kv ? K : V, kv ? V : K}, f32);
    if (state.dim() != 4 || state.size(1) != HV || state.size(2) != (kv ? K : V) || state.size(3) != (kv ? V : K)) {
        throw pybind11::value_error(std::string("State layout mismatch for state_layout='") + (kv ? "kv" : "vk") + "': got " + shape_text(state) +
                                    ", expected (..., " + std::to_string(HV) + ", " + std::to_string(kv ? K : V) + ", " + std::to_string(kv ? V : K) + ")");
    }
    require(is_f32(state) && state.is_contiguous(), "the state pool must be contiguous float32");
    const int64_t pool = state.size(0);
    OptTensor idx;
    if (indices.has_value()) {
        idx = indices->to(q_in.device(), at::kInt).contiguous();
        require(idx->numel() == N, "initial_state_indices must hold one slot per sequence");
    } else if (pool < N) {
        throw pybind11::value_error("the state pool holds " + std::to_string(pool) + " states for " + std::to_string(N) +
                                    " sequences and no indices were given");
    }
    const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous(), a = a_in.contiguous(), b = b_in.contiguous();
    require(a.numel() == N * HV * K && b.numel() == N * HV, "a must be (N, HV, K) and b (N, HV) up to singleton axes");
    require((is_bf16(a) || is_f32(a)) && (is_bf16(b) || is_f32(b)), "a and b must be in bfloat16 or float32");
    const Tensor A_log = contiguous_f32(A_log_in);
    const OptTensor dt_bias = contiguous_f32(dt_bias_in);
    require(A_log.numel() == HV, "A_log must have one entry per value head");
    if (dt_bias.has_value()) require(dt_bias->numel() == HV * K, "dt_bias must have HV * K entries");
    const bool varlen = Bq == 1 && Tq == N && N > 1;
    const int64_t s0 = varlen ? 1 : N, s1 = varlen ? N : 1;
    Tensor out;
    if (out_in.has_value()) {
        out = *out_in;
        if (out.dim() != 4 || out.size(0) != s0 || out.size(1) != s1 || out.size(2) != HV || out.size(3) != V || out.scalar_type() != q.scalar_type()) {
            throw pybind11::value_error("out must have shape (" + std::to_string(s0) + ", " + std::to_string(s1) + ", " + std::to_string(HV) + ", " +
                                        std::to_string(V) + ") and dtype torch.bfloat16");
        }
        if (!out.is_contiguous()) throw pybind11::value_error("out must be contiguous");
    } else {
        out = device_empty({s0, s1, HV, V}, q.options());
    }
    check(lib.cula_kda_decode(ptr(q), ptr(k), ptr(v), ptr(a), is_f32(a), ptr(b), is_f32(b), fptr(A_log), fptr(dt_bias), fptr(state), iptr(idx), ptr(out),
                              (int)N, (int)H, (int)HV, (int)V, (int)pool, (float)scale.value_or(1.0 / std::sqrt((double)K)), l2norm,
                              (float)softplus_beta, (float)softplus_threshold, kv, status_word(dev), stream_of(q)), "cula_kda_decode");
    return out;
}

// `o.grad_fn.kept`: the forward intermediates a node holds for its backward pass (disable_recompute), or None
PyObject* node_kept(PyObject* self, void*) {
    auto& node = static_cast<torch::autograd::CppNode<Attention>&>(*reinterpret_cast<torch::autograd::THPCppFunction*>(self)->cdata);
    auto it = node.ctx_.saved_data.find("kept");
    if (it == node.ctx_.saved_data.end()) Py_RETURN_NONE;
    static const char* const names[] = {"tiles", "akk", "mkk", "h32", "vnew"};
    pybind11::dict d;
    const auto t = it->second.toTensorVector();
    for (int i = 0; i < 5; ++i) d[names[i]] = t[i];
    return d.release().ptr();
}
void register_node_type() {
    using namespace torch::autograd;        // the property macro names its functions unqualified
    static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES, {(char*)"kept", node_kept, nullptr, nullptr, nullptr}, {nullptr}};
    static PyTypeObject type;
    torch::autograd::_initFunctionPyTypeObject(type, "ChunkKDABackward", properties, nullptr);
    Py_INCREF(&type);
    torch::autograd::registerCppFunction(typeid(torch::autograd::CppNode<Attention>), &type);
}

}  // namespace

void bind_attention(pybind11::module_& m) {
    namespace py = pybind11;
    py::class_<Tables>(m, "Tables")
        .def(py::init([](Tensor cu, Tensor ci, Tensor co, Tensor so, int64_t n_seqs, int64_t num_chunks, int64_t total) {
            return Tables{cu, ci, co, so, n_seqs, num_chunks, total};
        }));
    py::class_<Segments>(m, "Segments").def(py::init([](int64_t count, const Tables& t) { return Segments{count, t}; }));
    register_node_type();
    m.def("attend", &attend);
    m.def("forward", &forward_dict);
    m.def("backward", &backward_tuple);
    m.def("decode", &decode);
    m.def("forward_calls", [] { return forward_calls.load(); });
}

}  // namespace cula_host
