// The two layer operators on either side of chunk_kda in a Kimi-Linear block, as stand-alone streaming kernels:
//   short causal depthwise convolution + SiLU on the q / k / v projections (kernel width <= 4), forward and backward,
//   gated RMS norm on the attention output, y = rmsnorm(x) * w * act(g), forward and backward.
// They replace flash-linear-attention's ShortConvolution / causal_conv1d (fla/modules/convolution.py) and
// FusedRMSNormGated / rms_norm_gated (fla/modules/fused_norm_gate.py:35-120, 846-869), which the layer that calls the
// reference's chunk_kda uses (fla/layers/kda.py:147-165, 191, 306). Each element is read and written once (the convolution
// re-reads a halo of at most 3 tokens per chunk or half chunk, 6 per half in the backward pass); the norm waits on memory, the convolution on its own instructions.
#include "kda_common.cuh"
#include "kda_params.h"

namespace kda {

constexpr int LO_THREADS = 128;

__device__ __forceinline__ void lo_unpack8(const uint4& a, float2 (&v)[4]) {
    v[0] = unpack_bf16(a.x); v[1] = unpack_bf16(a.y); v[2] = unpack_bf16(a.z); v[3] = unpack_bf16(a.w);
}
__device__ __forceinline__ uint4 lo_pack8(const float2 (&v)[4]) {
    return make_uint4(pack_bf16(v[0].x, v[0].y), pack_bf16(v[1].x, v[1].y), pack_bf16(v[2].x, v[2].y), pack_bf16(v[3].x, v[3].y));
}
__device__ __forceinline__ float2 sigmoid2(float2 x) {
    return make_float2(fast_rcp(1.f + fast_exp2(-RCP_LN2 * x.x)), fast_rcp(1.f + fast_exp2(-RCP_LN2 * x.y)));
}

// ------------------------------------------------------------------------------------------------------------------
// Causal depthwise convolution: pre[t, d] = bias[d] + sum_i w[d, i] x[t - (W-1) + i, d],  y = silu(pre) (or pre).
// Tokens before the start of a sequence come from cache[n, d, :] (the last W inputs of the previous call, newest
// last) or are zero. A warp walks one 64-token chunk (chunks never straddle sequences: the same tables as the attention
// kernels) of 64 channels, two per lane, with the window in registers under compile-time slots (token t sits in slot
// (t - t0) mod 4, so nothing is shifted); the rows of NB tokens are requested before the first of them is used. The backward pass
// takes half a chunk and four channels per lane.
// Two or four channels per lane make a row access 128 or 256 contiguous bytes per warp, the arithmetic packed pairs, and enough warps
// to cover the memory latency: with eight channels per thread there were seven per SM at 4096 x 4096.
// The weight gradients of the CTA's four units are added in shared memory, then one 16-byte atomic per channel goes out.
// Measured at 4096 tokens x 4096 channels, W = 4: forward 27.7 -> 17.8 us (67 MB: 3.8 TB/s), backward 88 -> 36 -> 25 us (101 MB: 4 TB/s;
// the last step: four channels per lane instead of two, no checks inside a unit), 8192 x 512: 24 -> 6 us. Backward in quarters of a
// chunk: 32 us; five CTAs per SM by a register limit spill (70 us).
// What bounds the backward: its instructions (72 per token and warp for two channels, now 110 for four, or 55) and the fixed latencies
// between them at four warps per scheduler, a fifth of the time memory.
// ------------------------------------------------------------------------------------------------------------------
constexpr int CONV_WARPS = LO_THREADS / 32;

__device__ __forceinline__ float2 conv_row(const ConvArgs& a, int seq, int seq_start, int t, int ch) {
    // token t of the flattened axis, or (t < seq_start) the cached inputs of the previous call, or zero
    if (t >= seq_start) return unpack_bf16(*reinterpret_cast<const uint32_t*>(a.x + (size_t)t * a.D + ch));
    if (a.cache_in && seq_start - t <= a.W) {
        const float* c = a.cache_in + ((size_t)seq * a.D + ch) * a.W + (a.W - (seq_start - t));
        return make_float2(c[0], c[a.W]);
    }
    return make_float2(0.f, 0.f);
}
template <int V>
struct ConvRow {              // V pairs of channels of a token as they are
    uint32_t w[V];
};
template <int V>
__device__ __forceinline__ ConvRow<V> conv_load(const __nv_bfloat16* p) {
    ConvRow<V> r;
    if constexpr (V == 2) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        r.w[0] = x.x; r.w[1] = x.y;
    } else r.w[0] = *reinterpret_cast<const uint32_t*>(p);
    return r;
}
template <int V>
__device__ __forceinline__ void conv_store(__nv_bfloat16* p, const float2 (&v)[V]) {
    if constexpr (V == 2) *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v[0].x, v[0].y), pack_bf16(v[1].x, v[1].y));
    else *reinterpret_cast<uint32_t*>(p) = pack_bf16(v[0].x, v[0].y);
}
// V: pairs of channels per lane; UNIT: tokens that a warp walks, a chunk or half of one
template <int W, bool BWD, int V, int UNIT>
__global__ void __launch_bounds__(LO_THREADS) kda_short_conv_kernel(const ConvArgs a, const int num_chunks) {
    constexpr int CH = 2 * V, GROUP = 32 * CH;               // channels of a lane, of a warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ch = GROUP * blockIdx.x + CH * lane, unit = CONV_WARPS * (blockIdx.z * gridDim.y + blockIdx.y) + warp, c = unit / (BT / UNIT);
    bool live = ch < a.D && c < num_chunks;
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float s_dw[BWD ? CONV_WARPS : 1][GROUP][W + 1];       // weight and bias gradients per warp
    ChunkInfo ci{};
    int t0 = 0, t1 = 0;
    if (live) {
        ci = chunk_info(c, a.cu_seqlens, a.chunk_indices, a.T);
        t0 = ci.row0 + UNIT * (unit % (BT / UNIT));
        t1 = min(t0 + UNIT, ci.row0 + ci.valid);
        live = t0 < t1;
    }
    if (live) {
        const int seq_start = a.cu_seqlens ? a.cu_seqlens[ci.seq] : ci.seq * a.T;
        const int seq_end = a.cu_seqlens ? a.cu_seqlens[ci.seq + 1] : (ci.seq + 1) * a.T;
        float2 w[W][V], b[V], win[4][V];                            // tap i multiplies x[t - (W-1) + i]; x by slot: slots 1..3 start with tokens t0-3 .. t0-1
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int cv = ch + 2 * v;
#pragma unroll
            for (int i = 0; i < W; ++i) w[i][v] = make_float2(a.w[(size_t)cv * W + i], a.w[(size_t)(cv + 1) * W + i]);
            b[v] = a.bias ? make_float2(a.bias[cv], a.bias[cv + 1]) : make_float2(0.f, 0.f);
            win[0][v] = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 1; k < 4; ++k) win[k][v] = k >= 5 - W ? conv_row(a, ci.seq, seq_start, t0 - 4 + k, cv) : make_float2(0.f, 0.f);
        }
        const __nv_bfloat16* xp = a.x + ch;
        auto preact = [&](int i, int v) {                           // with token t in slot i
            float2 pre = b[v];
#pragma unroll
            for (int k = 0; k < W; ++k) pre = fma2(w[W - 1 - k][v], win[(i - k) & 3][v], pre);
            return pre;
        };
        if constexpr (!BWD) {
            constexpr int NB = 8;
            ConvRow<V> raw[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) raw[i] = conv_load<V>(xp + (size_t)min(t0 + i, t1 - 1) * a.D);
            for (int tb = t0; tb < t1; tb += NB) {
                ConvRow<V> cur[NB];
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    cur[i] = raw[i];                                // the next batch is on its way while this one is computed
                    raw[i] = conv_load<V>(xp + (size_t)min(tb + NB + i, t1 - 1) * a.D);
                }
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const int t = tb + i;
                    if (t >= t1) break;
                    float2 y[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        win[i & 3][v] = unpack_bf16(cur[i].w[v]);
                        y[v] = preact(i, v);
                        if (a.silu) y[v] = mul2(y[v], sigmoid2(y[v]));
                    }
                    conv_store<V>(a.y + (size_t)t * a.D + ch, y);
                }
            }
            if (a.cache_out && t1 == seq_end) {      // the last W inputs of the sequence, newest last, zero-padded on the left
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float* co = a.cache_out + ((size_t)ci.seq * a.D + ch + 2 * v) * W;
#pragma unroll
                    for (int i = 0; i < W; ++i) {
                        const float2 x = conv_row(a, ci.seq, seq_start, t1 - W + i, ch + 2 * v);
                        co[i] = x.x;
                        co[W + i] = x.y;
                    }
                }
            }
        } else {
            // walk W-1 tokens past the unit (inside the sequence): dx[u] = sum_i w[i] dpre[u + (W-1) - i] needs them
            float2 dwin[4][V], dw[W][V], db[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                db[v] = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) dwin[k][v] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < W; ++i) dw[i][v] = make_float2(0.f, 0.f);
            }
            const __nv_bfloat16* dyp = a.dy + ch;
            const int t_end = t1 + (W - 1), t_last = seq_end - 1;
            constexpr int NBB = 4;
            ConvRow<V> rx[NBB], ry[NBB];
            auto fetch = [&](int t) {                               // clamped: tokens past the sequence are not used
#pragma unroll
                for (int i = 0; i < NBB; ++i) {
                    const size_t off = (size_t)min(t + i, t_last) * a.D;
                    rx[i] = conv_load<V>(xp + off);
                    ry[i] = conv_load<V>(dyp + off);
                }
            };
            // token in slot i: dpre, and (own token of the unit) its part of the parameter gradients
            auto take = [&](int i, const ConvRow<V>& x, const ConvRow<V>& dy, bool own) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    win[i][v] = unpack_bf16(x.w[v]);
                    float2 dp = unpack_bf16(dy.w[v]);
                    if (a.silu) {
                        const float2 pre = preact(i, v), s = sigmoid2(pre);
                        // silu' = s (1 + pre (1 - s))
                        dp = mul2(dp, mul2(s, fma2(pre, fma2(s, splat2(-1.f), splat2(1.f)), splat2(1.f))));
                    }
                    dwin[i][v] = dp;
                    if (own) {
                        db[v] = add2(db[v], dp);
#pragma unroll
                        for (int k = 0; k < W; ++k) dw[W - 1 - k][v] = fma2(dp, win[(i - k) & 3][v], dw[W - 1 - k][v]);
                    }
                }
            };
            auto emit = [&](int i, int u) {                         // dx of token u, W-1 before the one in slot i
                float2 o[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    o[v] = mul2(w[0][v], dwin[i][v]);
#pragma unroll
                    for (int k = 1; k < W; ++k) o[v] = fma2(w[k][v], dwin[(i - k) & 3][v], o[v]);     // dpre[u + (W-1) - k] = dpre[t - k]
                }
                conv_store<V>(a.dx + (size_t)u * a.D + ch, o);
            };
            fetch(t0);
            for (int tb = t0; tb < t_end; tb += NBB) {
                ConvRow<V> cx[NBB], cy[NBB];
#pragma unroll
                for (int i = 0; i < NBB; ++i) { cx[i] = rx[i]; cy[i] = ry[i]; }
                fetch(tb + NBB);
                if (tb + NBB <= t1) {                               // four tokens of the unit
#pragma unroll
                    for (int i = 0; i < NBB; ++i) {
                        take(i, cx[i], cy[i], true);
                        if (i >= W - 1 || tb > t0) emit(i, tb + i - (W - 1));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < NBB; ++i) {
                        const int t = tb + i;
                        if (t >= t_end) break;
                        if (t < seq_end) take(i, cx[i], cy[i], t < t1);
                        else {
#pragma unroll
                            for (int v = 0; v < V; ++v) dwin[i][v] = make_float2(0.f, 0.f);
                        }
                        if (t - (W - 1) >= t0) emit(i, t - (W - 1));
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    s_dw[warp][CH * lane + 2 * v][i] = dw[i][v].x;
                    s_dw[warp][CH * lane + 2 * v + 1][i] = dw[i][v].y;
                }
                s_dw[warp][CH * lane + 2 * v][W] = db[v].x;
                s_dw[warp][CH * lane + 2 * v + 1][W] = db[v].y;
            }
        }
    } else if constexpr (BWD) {
#pragma unroll
        for (int e = 0; e < CH; ++e)
#pragma unroll
            for (int i = 0; i <= W; ++i) s_dw[warp][CH * lane + e][i] = 0.f;
    }
    if constexpr (BWD) {
        __syncthreads();
        const int cl = threadIdx.x, cg = GROUP * blockIdx.x + cl;
        if (cl < GROUP && cg < a.D) {
            float v[W + 1];
#pragma unroll
            for (int i = 0; i <= W; ++i) {
                v[i] = 0.f;
#pragma unroll
                for (int x = 0; x < CONV_WARPS; ++x) v[i] += s_dw[x][cl][i];
            }
            if (W == 4 && (reinterpret_cast<uintptr_t>(a.dw) & 15) == 0) atomicAdd(reinterpret_cast<float4*>(a.dw + (size_t)cg * 4), make_float4(v[0], v[1], v[2], v[3]));
            else {
#pragma unroll
                for (int i = 0; i < W; ++i) atomicAdd(&a.dw[(size_t)cg * W + i], v[i]);
            }
            if (a.dbias) atomicAdd(&a.dbias[cg], v[W]);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Gated RMS norm over rows of D elements (128, 256, 512 or 1024): LPR lanes share a row, 8 elements per lane and vector.
//   n = x * rstd, rstd = rsqrt(mean(x^2) + eps);  y = n * w * act(g), act = sigmoid or swish.
// A row of 128 takes a half warp, so that every access is 16 bytes per lane and no lane works on padding. Measured at
// 131,072 rows of 128: forward 29 -> 22.5 us (101 MB: 4.5 TB/s), backward 88 -> 31 us (168 MB: 5.4 TB/s).
// ------------------------------------------------------------------------------------------------------------------

template <int LPR, int VPL, bool BWD>       // D = 8 * LPR * VPL
__global__ void __launch_bounds__(LO_THREADS) kda_rms_norm_gated_kernel(const NormArgs a) {
    constexpr int D = 8 * LPR * VPL, GROUPS = LO_THREADS / LPR;      // rows a CTA works on side by side
    const int lane = threadIdx.x & (LPR - 1), grp = threadIdx.x / LPR;
    const long long row0 = (long long)blockIdx.x * GROUPS + grp, stride = (long long)gridDim.x * GROUPS;
    float2 wv[VPL][4], dw_acc[VPL][4];
    pdl_launch_dependents();
    pdl_wait();
#pragma unroll
    for (int v = 0; v < VPL; ++v)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            wv[v][e] = make_float2(a.w[8 * (LPR * v + lane) + 2 * e], a.w[8 * (LPR * v + lane) + 2 * e + 1]);
            dw_acc[v][e] = make_float2(0.f, 0.f);
        }
    // Rows are taken NB at a time and all their loads are issued before the first is used (a thread has dozens of rows
    // and one row per dependent step would pay a full memory latency each).
    constexpr int NB = VPL == 1 ? 4 : (VPL == 2 ? 2 : 1);
    for (long long rb = row0; rb - grp < a.R; rb += NB * stride) {     // rb - grp: the CTA's first row, the same for all
        uint4 rx[NB][VPL], rg[NB][VPL], rd[NB][VPL];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const size_t base = (size_t)min(rb + (long long)i * stride, a.R - 1) * D + 8 * lane;       // clamped: surplus rows are not used
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                rx[i][v] = *reinterpret_cast<const uint4*>(a.x + base + 8 * LPR * v);
                rg[i][v] = *reinterpret_cast<const uint4*>(a.g + base + 8 * LPR * v);
                if (BWD) rd[i][v] = *reinterpret_cast<const uint4*>(a.dy + base + 8 * LPR * v);
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const long long row = rb + (long long)i * stride;
            const bool live = row < a.R;
            const size_t base = (size_t)row * D + 8 * lane;
            float2 xv[VPL][4], gv[VPL][4];
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                lo_unpack8(rx[i][v], xv[v]);
                lo_unpack8(rg[i][v], gv[v]);
            }
            if constexpr (!BWD) {
                float2 ss2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int v = 0; v < VPL; ++v)
#pragma unroll
                    for (int e = 0; e < 4; ++e) ss2 = fma2(xv[v][e], xv[v][e], ss2);
                float ss = ss2.x + ss2.y;
#pragma unroll
                for (int o = LPR / 2; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float rstd = rsqrtf(ss * (1.f / D) + a.eps);
                if (live) {
                    if (lane == 0) a.rstd[row] = rstd;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        float2 out[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 s = sigmoid2(gv[v][e]);
                            out[e] = mul2(mul2(mul2(xv[v][e], splat2(rstd)), wv[v][e]), a.swish ? mul2(gv[v][e], s) : s);
                        }
                        *reinterpret_cast<uint4*>(a.y + base + 8 * LPR * v) = lo_pack8(out);
                    }
                }
            } else {
                const float rstd = a.rstd[min(row, a.R - 1)];
                float2 dn[VPL][4], dot2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    float2 dyv[4], dgo[4];
                    lo_unpack8(rd[i][v], dyv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 gg = gv[v][e], s = sigmoid2(gg), n = mul2(xv[v][e], splat2(rstd));
                        const float2 t = make_float2(1.f - s.x, 1.f - s.y);
                        const float2 act = a.swish ? mul2(gg, s) : s;
                        const float2 dact = a.swish ? mul2(s, fma2(gg, t, splat2(1.f))) : mul2(s, t);
                        const float2 dz = mul2(dyv[e], act);
                        dgo[e] = mul2(mul2(dyv[e], mul2(n, wv[v][e])), dact);
                        if (live) dw_acc[v][e] = fma2(dz, n, dw_acc[v][e]);
                        dn[v][e] = mul2(dz, wv[v][e]);
                        dot2 = fma2(dn[v][e], n, dot2);
                    }
                    if (live) *reinterpret_cast<uint4*>(a.dg + base + 8 * LPR * v) = lo_pack8(dgo);
                }
                float dot = dot2.x + dot2.y;
#pragma unroll
                for (int o = LPR / 2; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                const float2 m = splat2(-dot * (1.f / D) * rstd);           // dx = rstd (dn - x rstd mean(dn n))
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    float2 out[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) out[e] = mul2(splat2(rstd), fma2(xv[v][e], m, dn[v][e]));
                    if (live) *reinterpret_cast<uint4*>(a.dx + base + 8 * LPR * v) = lo_pack8(out);
                }
            }
        }
    }
    if constexpr (BWD) {
        // the weight gradient: the CTA's rows are summed in shared memory first, then one global atomic per column and CTA
        __shared__ float s_dw[D];
        for (int c = threadIdx.x; c < D; c += LO_THREADS) s_dw[c] = 0.f;
        __syncthreads();
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                atomicAdd(&s_dw[8 * (LPR * v + lane) + 2 * e], dw_acc[v][e].x);
                atomicAdd(&s_dw[8 * (LPR * v + lane) + 2 * e + 1], dw_acc[v][e].y);
            }
        __syncthreads();
        for (int c = threadIdx.x; c < D; c += LO_THREADS) atomicAdd(&a.dw[c], s_dw[c]);
    }
}

}  // namespace kda

extern "C" int kda_launch_short_conv(const kda::ConvArgs* a, int num_chunks, int backward, cudaStream_t stream) {
    using namespace kda;
    if (num_chunks <= 0) return 0;
    // Backward: two pairs of channels per lane halve the instructions that do not depend on the number of channels and double the work
    // between dependent ones (rows are 16-byte pieces). Forward: one pair (two: 17.5 -> 19.5 us at 4096 x 4096), and half chunks where
    // whole ones would leave fewer than 16 warps per SM (8192 x 512: 11.5 -> 8.5 us).
    const int groups = (a->D + (backward ? 127 : 63)) / (backward ? 128 : 64);
    const bool halves = backward || (long long)num_chunks * groups < 16LL * sm_count();
    // The second dimension takes 65535 blocks and there may be more units than that: what is above goes into the third. (Both in the first,
    // divided in the kernel: 268 -> 272 us for the six operators around a call at 2 x 2048 x 32 heads, forward and backward.)
    const long long units = num_chunks * (halves ? 2LL : 1LL), blocks = (units + CONV_WARPS - 1) / CONV_WARPS, layers = (blocks + 65534) / 65535;
    const dim3 grid(groups, (unsigned)((blocks + layers - 1) / layers), (unsigned)layers);
    void (*kernel)(const ConvArgs, const int) = nullptr;
#define KDA_CONV_KERNEL(W)                                                                                          \
    kernel = backward ? kda_short_conv_kernel<W, true, 2, 32> : halves ? kda_short_conv_kernel<W, false, 1, 32> : kda_short_conv_kernel<W, false, 1, 64>
    switch (a->W) {
        case 1: KDA_CONV_KERNEL(1); break;
        case 2: KDA_CONV_KERNEL(2); break;
        case 3: KDA_CONV_KERNEL(3); break;
        case 4: KDA_CONV_KERNEL(4); break;
        default: return -1;
    }
#undef KDA_CONV_KERNEL
    return (int)launch_early(kernel, grid, LO_THREADS, 0, stream, *a, num_chunks);
}

extern "C" int kda_launch_rms_norm_gated(const kda::NormArgs* a, int backward, cudaStream_t stream) {
    using namespace kda;
    if (a->R <= 0) return 0;
    const int groups = a->D == 128 ? LO_THREADS / 16 : LO_THREADS / 32;
    long long blocks = (a->R + groups - 1) / groups;
    const long long cap = (backward ? 4LL : 16LL) * sm_count();     // backward: fewer, longer-lived CTAs keep the dw atomics few
    if (blocks > cap) blocks = cap;
    void (*kernel)(const NormArgs) = nullptr;
#define KDA_NORM_KERNEL(L, V) kernel = backward ? kda_rms_norm_gated_kernel<L, V, true> : kda_rms_norm_gated_kernel<L, V, false>
    if (a->D == 128) KDA_NORM_KERNEL(16, 1);
    else if (a->D == 256) KDA_NORM_KERNEL(32, 1);
    else if (a->D == 512) KDA_NORM_KERNEL(32, 2);
    else if (a->D == 1024) KDA_NORM_KERNEL(32, 4);
    else return -1;
#undef KDA_NORM_KERNEL
    return (int)launch_early(kernel, dim3((unsigned)blocks), LO_THREADS, 0, stream, *a);
}
