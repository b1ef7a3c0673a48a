// Layer-side elementwise operators that sit next to chunk_kda in a Kimi-Linear block, as stand-alone kernels:
//   kda_gate fwd / bwd   : a = -exp(A_log[h]) softplus(g + dt_bias[h,:])           (softplus form)
//                          a = lower_bound sigmoid(exp(A_log[h]) (g + dt_bias[h,:]))  (lower-bound form)
//   beta_sigmoid fwd/bwd : y = sigmoid(x) in fp32
// They replace flash-linear-attention's fused_kda_gate / fused_beta_sigmoid (fla/ops/kda/gate.py:282-345, 348-432),
// which the reference's callers use when the gate is not computed inside chunk_kda. Pure streaming work: every element
// is read once and written once; the two parameter gradients are block-reduced and finished with atomics.
#include "kda_common.cuh"
#include "kda_params.h"

namespace kda {

constexpr int GATE_THREADS = 256;


__device__ __forceinline__ void load8(const void* p, int fp32, size_t idx, float (&v)[8]) {
    if (fp32) {
        const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + idx);
        const float4 b = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + idx + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
        const uint4 a = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p) + idx);
        float2 f;
        f = unpack_bf16(a.x); v[0] = f.x; v[1] = f.y;
        f = unpack_bf16(a.y); v[2] = f.x; v[3] = f.y;
        f = unpack_bf16(a.z); v[4] = f.x; v[5] = f.y;
        f = unpack_bf16(a.w); v[6] = f.x; v[7] = f.y;
    }
}
__device__ __forceinline__ void store8(void* p, int fp32, size_t idx, const float (&v)[8]) {
    if (fp32) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p) + idx) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p) + idx + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p) + idx) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    }
}
// A warp owns 256 channels (8 per lane, kept for the whole launch: the bias and the head's exp(A_log) are loaded once);
// the CTA's eight warps and grid.y stride over the tokens. HBM-bound; NB rows per warp are requested before the first is
// used. The parameter gradients of a CTA are added in shared memory, then one atomic per channel (16 bytes at a time where
// the buffer is aligned) and head goes out. Measured at 4096 tokens x 32 heads x 128: backward 47 -> 31 us (134 MB: 4.4 TB/s);
// shared-memory atomics instead of a slot per warp 38 us, two or six CTAs per SM instead of four 44 / 38 us.
template <bool BWD>
__global__ void __launch_bounds__(GATE_THREADS) kda_gate_kernel(const GateArgs a) {
    constexpr int WARPS = GATE_THREADS / 32;
    __shared__ __align__(16) float s_bias[BWD ? WARPS : 1][BWD ? 256 : 4];
    __shared__ float s_dA[BWD ? 10 : 1];     // at most 256 / 32 + 1 heads meet 256 channels (K >= 32)
    pdl_launch_dependents();
    const int HK = a.H * a.K, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ch0 = 256 * blockIdx.x, ch_raw = ch0 + 8 * lane;
    const bool active = ch_raw < HK;
    const int ch = active ? ch_raw : 0, h = ch / a.K, h_lo = ch0 / a.K;
    if (BWD) {
        if (threadIdx.x < 10) s_dA[threadIdx.x] = 0.f;
        __syncthreads();
    }
    pdl_wait();
    const float alpha = __expf(a.A_log[h]);
    float2 bias[4], dbias[4];
    float dA = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        bias[e] = a.dt_bias ? make_float2(a.dt_bias[ch + 2 * e], a.dt_bias[ch + 2 * e + 1]) : make_float2(0.f, 0.f);
        dbias[e] = make_float2(0.f, 0.f);
    }
    if (active) {
        constexpr int NB = BWD ? 2 : 4;
        const long long step = (long long)gridDim.y * WARPS;
        for (long long mb = (long long)blockIdx.y * WARPS + warp; mb < a.M; mb += NB * step) {
            float gv[NB][8], dy[NB][8];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const long long m = min(mb + i * step, a.M - 1);      // clamped: the surplus rows are not used
                const size_t idx = (size_t)m * HK + ch;
                load8(a.g, a.g_fp32, idx, gv[i]);
                if (BWD) load8(a.dy, a.dy_fp32, idx, dy[i]);
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const long long m = mb + i * step;
                if (m >= a.M) break;
                const size_t idx = (size_t)m * HK + ch;
                float o[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = add2(make_float2(gv[i][2 * e], gv[i][2 * e + 1]), bias[e]);
                    float2 v;
                    if (a.use_lower_bound) {
                        const float c = -alpha * RCP_LN2;
                        const float2 sg = make_float2(fast_rcp(1.f + fast_exp2(c * x.x)), fast_rcp(1.f + fast_exp2(c * x.y)));
                        if (!BWD) {
                            v = mul2(splat2(a.lower_bound), sg);
                        } else {                     // d/dx of lb sigmoid(alpha x); times x it is d/dA_log
                            const float2 q = mul2(sg, make_float2(1.f - sg.x, 1.f - sg.y));
                            v = mul2(mul2(make_float2(dy[i][2 * e], dy[i][2 * e + 1]), splat2(a.lower_bound * alpha)), q);
                            dA = fmaf(v.x, x.x, fmaf(v.y, x.y, dA));
                        }
                    } else {
                        const float2 sp = softplus2(x);
                        if (!BWD) {
                            v = mul2(splat2(-alpha), sp);
                        } else {
                            const float2 d = mul2(make_float2(dy[i][2 * e], dy[i][2 * e + 1]), splat2(-alpha));
                            v = mul2(d, make_float2(fast_rcp(1.f + fast_exp2(-RCP_LN2 * x.x)), fast_rcp(1.f + fast_exp2(-RCP_LN2 * x.y))));
                            dA = fmaf(d.x, sp.x, fmaf(d.y, sp.y, dA));
                        }
                    }
                    if (BWD) dbias[e] = add2(dbias[e], v);
                    o[2 * e] = v.x;
                    o[2 * e + 1] = v.y;
                }
                store8(a.out, BWD ? a.g_fp32 : a.out_fp32, idx, o);
            }
        }
    }
    if (BWD) {
        *reinterpret_cast<float4*>(&s_bias[warp][8 * lane]) = make_float4(dbias[0].x, dbias[0].y, dbias[1].x, dbias[1].y);
        *reinterpret_cast<float4*>(&s_bias[warp][8 * lane + 4]) = make_float4(dbias[2].x, dbias[2].y, dbias[3].x, dbias[3].y);
        if (a.dA_log) {
            // the 16 lanes of a 128-channel head are added by shuffles first
            if (a.K == 128) {
#pragma unroll
                for (int o = 8; o; o >>= 1) dA += __shfl_xor_sync(0xffffffffu, dA, o);
                if (active && (lane & 15) == 0) atomicAdd(&s_dA[h - h_lo], dA);
            } else if (active) {
                atomicAdd(&s_dA[h - h_lo], dA);
            }
        }
        __syncthreads();
        if (a.ddt_bias && threadIdx.x < 64 && ch0 + 4 * threadIdx.x < HK) {
            const int c4 = 4 * threadIdx.x;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const float4 x = *reinterpret_cast<const float4*>(&s_bias[w][c4]);
                v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
            }
            float* dst = a.ddt_bias + ch0 + c4;
            if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
                atomicAdd(reinterpret_cast<float4*>(dst), v);
            } else {
                atomicAdd(dst, v.x); atomicAdd(dst + 1, v.y); atomicAdd(dst + 2, v.z); atomicAdd(dst + 3, v.w);
            }
        }
        if (a.dA_log && threadIdx.x < 10 && h_lo + threadIdx.x < a.H && s_dA[threadIdx.x] != 0.f) atomicAdd(&a.dA_log[h_lo + threadIdx.x], s_dA[threadIdx.x]);
    }
}

template <bool BWD>
__global__ void __launch_bounds__(GATE_THREADS) kda_beta_sigmoid_kernel(const void* x, int x_fp32, const float* dy, void* out,
                                                                       long long n) {
    pdl_launch_dependents();
    pdl_wait();
    for (long long i = (long long)blockIdx.x * GATE_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * GATE_THREADS) {
        const float xv = x_fp32 ? reinterpret_cast<const float*>(x)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i]);
        const float y = __fdividef(1.f, 1.f + __expf(-xv));
        if (!BWD) {
            reinterpret_cast<float*>(out)[i] = y;
        } else {
            const float d = dy[i] * y * (1.f - y);
            if (x_fp32) reinterpret_cast<float*>(out)[i] = d;
            else reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(d);
        }
    }
}

// Zeros for buffers that atomics add to: unlike a memset, which ends and starts a chain of early launches, this is part of it.
__global__ void __launch_bounds__(GATE_THREADS) kda_clear_kernel(unsigned int* dst, long long words) {
    pdl_launch_dependents();
    pdl_wait();
    const long long i = (long long)blockIdx.x * GATE_THREADS + threadIdx.x, n = (long long)gridDim.x * GATE_THREADS, quads = words / 4;
    for (long long j = i; j < quads; j += n) reinterpret_cast<uint4*>(dst)[j] = make_uint4(0, 0, 0, 0);
    for (long long j = 4 * quads + i; j < words; j += n) dst[j] = 0;
}

}  // namespace kda

extern "C" int kda_launch_clear(unsigned int* dst, long long words, cudaStream_t stream) {
    using namespace kda;
    long long blocks = (words / 4 + GATE_THREADS - 1) / GATE_THREADS;
    const long long most = 4LL * sm_count();
    blocks = blocks < 1 ? 1 : blocks > most ? most : blocks;
    return (int)launch_early(kda_clear_kernel, dim3((unsigned)blocks), GATE_THREADS, 0, stream, dst, words);
}

extern "C" int kda_launch_gate(const kda::GateArgs* a, int backward, cudaStream_t stream) {
    using namespace kda;
    if (a->M <= 0) return 0;
    const int sms = sm_count();
    const int gx = (a->H * a->K + 255) / 256;
    // about eight CTAs per SM in flight; the backward pass ends in atomics, so it runs half as many, longer-lived CTAs
    long long gy = ((backward ? 4LL : 8LL) * sms + gx - 1) / gx;
    const long long most = (a->M + GATE_THREADS / 32 - 1) / (GATE_THREADS / 32);
    if (gy > most) gy = most;
    if (gy > 65535) gy = 65535;
    dim3 grid(gx, (unsigned)gy);
    return (int)launch_early(backward ? kda_gate_kernel<true> : kda_gate_kernel<false>, grid, GATE_THREADS, 0, stream, *a);
}

extern "C" int kda_launch_beta_sigmoid(const void* x, int x_fp32, const float* dy, void* out, long long n, int backward,
                                       cudaStream_t stream) {
    using namespace kda;
    if (n <= 0) return 0;
    const int sms = sm_count();
    long long blocks = (n + GATE_THREADS - 1) / GATE_THREADS;
    if (blocks > 8LL * sms) blocks = 8LL * sms;
    return (int)launch_early(backward ? kda_beta_sigmoid_kernel<true> : kda_beta_sigmoid_kernel<false>, dim3((unsigned)blocks), GATE_THREADS, 0, stream, x,
                             x_fp32, dy, out, n);
}
