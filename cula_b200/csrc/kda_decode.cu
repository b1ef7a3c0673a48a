// KDA decode: one token per sequence against a pool of fp32 states, updated in place.
//     gate  = exp(-exp(A_log[hv]) * softplus(a + dt_bias[hv, :]))            [K]
//     v_new = sigmoid(b) * (v - S^T (gate * k_hat))                           [V]
//     S    <- diag(gate) S + k_hat v_new^T                                    [K x V]
//     o     = S^T (scale * q_hat)                                             [V]
// per (sequence n, value head hv); q/k head = hv / (HV / H) (grouped heads). Semantics of kda_decode /
// fused_sigmoid_gating_delta_rule_update (cula/ops/kda_decode.py:1794-2096) and of the reference's torch
// restatement (tests/test_kda_decode.py:42-104); a negative state index skips the sequence: no state access, as in
// the reference kernel (cula/ops/kda_decode.py:11-13), and a zero output row (the reference leaves it unwritten).
//
// The step is pure HBM streaming: 64 KB of state read and 64 KB written per (n, hv) against a few hundred bytes
// of vectors, so the kernel is organised around coalesced 16-byte accesses with many rows in flight:
//   layout "vk" (pool, HV, V, K), the reference's default: a warp walks its value rows 8 at a time (8 x 128
//     floats in registers, lane = 4 consecutive k, the next 8 rows already in flight), both contractions are
//     4 FMAs + a warp reduction per row;
//   layout "kv" (pool, HV, K, V): a warp owns 16 value columns of all 128 keys (4 lanes x float4 per row, 16 rows in
//     registers, all 8 KB requested before the first is used) and works alone: the contractions are 16 FMAs per lane
//     and a reduction over the 8 lanes that share the columns; no barriers between the loads and the stores. (With the
//     keys spread over the four warps and three CTA barriers per 32 columns, 33 sequences x 32 heads took 34.8 us a call for
//     138 MB, now 29.7.)
// Work items = N * HV * slices (K = 128; V any multiple of 32; slices divides V / 32 and is chosen on the host: 1
// when there are enough states to fill the GPU, more for small batches); kv items are 16 columns each.
#include "kda_common.cuh"

namespace kda {

struct DecodeParams {
    const void* q;        // [N, H, 128] bf16
    const void* k;        // [N, H, 128] bf16
    const void* v;        // [N, HV, V] bf16 (V a multiple of 32)
    const void* a;        // [N, HV, 128] bf16 or fp32 (raw gate input)
    const void* b;        // [N, HV] bf16 or fp32 (raw beta input)
    const float* A_log;   // [HV]
    const float* dt_bias; // [HV, 128] or nullptr
    float* state;         // [pool, HV, V, 128] (vk) or [pool, HV, 128, V] (kv) fp32, updated in place
    const int* indices;   // [N] pool slot of every sequence, or nullptr (slot = n)
    void* o;              // [N, HV, V] bf16
    int N, H, HV, V, pool, slices;   // slices: CTAs per state, each owning V / slices value rows (vk only)
    int a_fp32, b_fp32, use_l2norm, state_kv;
    float scale, softplus_beta, softplus_threshold;
    int* status;
};

constexpr int DEC_THREADS = 128;

__device__ __forceinline__ float dec_softplus(float x, float beta, float threshold) {
    const float bx = beta * x;
    return bx > threshold ? x : log1pf(__expf(bx)) / beta;      // torch.nn.functional.softplus(beta, threshold)
}
__device__ __forceinline__ float dec_load(const void* p, int is_fp32, size_t i) {
    return is_fp32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

// The per-key vectors of one (n, hv) for the 4 keys k0..k0+3 of a lane that covers the key axis with 32 lanes:
// gate, k_hat, scale * q_hat. The L2 norms are warp reductions over the 128 keys.
__device__ __forceinline__ void dec_key_vectors(const DecodeParams& p, int n, int hv, int hq, int k0, float (&gate)[4], float (&kh)[4],
                                                float (&qs)[4]) {
    const __nv_bfloat16* qp = reinterpret_cast<const __nv_bfloat16*>(p.q) + ((size_t)n * p.H + hq) * DK + k0;
    const __nv_bfloat16* kp = reinterpret_cast<const __nv_bfloat16*>(p.k) + ((size_t)n * p.H + hq) * DK + k0;
    const uint2 qr = *reinterpret_cast<const uint2*>(qp), kr = *reinterpret_cast<const uint2*>(kp);
    float2 f;
    f = unpack_bf16(qr.x); qs[0] = f.x; qs[1] = f.y;
    f = unpack_bf16(qr.y); qs[2] = f.x; qs[3] = f.y;
    f = unpack_bf16(kr.x); kh[0] = f.x; kh[1] = f.y;
    f = unpack_bf16(kr.y); kh[2] = f.x; kh[3] = f.y;
    float rq = p.scale, rk = 1.f;
    if (p.use_l2norm) {
        float sq = qs[0] * qs[0] + qs[1] * qs[1] + qs[2] * qs[2] + qs[3] * qs[3];
        float sk = kh[0] * kh[0] + kh[1] * kh[1] + kh[2] * kh[2] + kh[3] * kh[3];
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
        }
        rq = p.scale * rsqrtf(sq + 1e-6f);
        rk = rsqrtf(sk + 1e-6f);
    }
    const float alpha = __expf(p.A_log[hv]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        qs[e] *= rq;
        kh[e] *= rk;
        const float x = dec_load(p.a, p.a_fp32, ((size_t)n * p.HV + hv) * DK + k0 + e) + (p.dt_bias ? p.dt_bias[hv * DK + k0 + e] : 0.f);
        gate[e] = __expf(-alpha * dec_softplus(x, p.softplus_beta, p.softplus_threshold));
    }
}

// One work item of the (V, K) layout = one slice of one (sequence, value head) state.
__device__ __forceinline__ void dec_item(const DecodeParams& p, const int item) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int slice = item % p.slices, nh = item / p.slices;
    const int per_cta = p.V / p.slices;                     // value rows of this CTA, a multiple of 32
    const int n = nh / p.HV, hv = nh - n * p.HV;
    const int hq = hv / (p.HV / p.H);
    const int slot = p.indices ? p.indices[n] : n;
    if (slot < 0) {                                         // padded sequence: no state access; its output row is zeroed
        __nv_bfloat16* oz = reinterpret_cast<__nv_bfloat16*>(p.o) + ((size_t)n * p.HV + hv) * p.V + slice * per_cta;
        for (int i = tid; i < per_cta; i += DEC_THREADS) oz[i] = __float2bfloat16_rn(0.f);
        return;
    }
    if (slot >= p.pool) {                                   // caller error: report, touch nothing
        if (tid == 0) report_status(p.status, STATUS_BAD_INDEX);
        return;
    }
    float* S = p.state + ((size_t)slot * p.HV + hv) * (size_t)DK * p.V;
    const float beta = 1.f / (1.f + __expf(-dec_load(p.b, p.b_fp32, (size_t)n * p.HV + hv)));
    const __nv_bfloat16* vp = reinterpret_cast<const __nv_bfloat16*>(p.v) + ((size_t)n * p.HV + hv) * p.V;
    __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.o) + ((size_t)n * p.HV + hv) * p.V;

    {
        // ---- (V, K) rows: the warp owns per_cta / 4 value rows and walks them 8 at a time, the next 8 already in
        //      flight while the current 8 are updated; the lane owns keys 4*lane .. 4*lane+3 ----
        const int rows_warp = per_cta >> 2, nb = rows_warp >> 3;
        const int vbase = slice * per_cta + warp * rows_warp, k0 = 4 * lane;
        float4 row[8], nxt[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) row[i] = __ldcs(reinterpret_cast<const float4*>(S + (size_t)(vbase + i) * DK + k0));
        float gate[4], kh[4], qs[4];
        dec_key_vectors(p, n, hv, hq, k0, gate, kh, qs);
        float gk[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) gk[e] = gate[e] * kh[e];
        for (int bi = 0; bi < nb; ++bi) {
            const int v0 = vbase + 8 * bi;
            if (bi + 1 < nb) {
#pragma unroll
                for (int i = 0; i < 8; ++i) nxt[i] = __ldcs(reinterpret_cast<const float4*>(S + (size_t)(v0 + 8 + i) * DK + k0));
            }
            float hk[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) hk[i] = row[i].x * gk[0] + row[i].y * gk[1] + row[i].z * gk[2] + row[i].w * gk[3];
#pragma unroll
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) hk[i] += __shfl_xor_sync(0xffffffffu, hk[i], o);
            float ov[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float vn = beta * (__bfloat162float(vp[v0 + i]) - hk[i]);
                row[i].x = fmaf(gate[0], row[i].x, vn * kh[0]);
                row[i].y = fmaf(gate[1], row[i].y, vn * kh[1]);
                row[i].z = fmaf(gate[2], row[i].z, vn * kh[2]);
                row[i].w = fmaf(gate[3], row[i].w, vn * kh[3]);
                __stcs(reinterpret_cast<float4*>(S + (size_t)(v0 + i) * DK + k0), row[i]);
                ov[i] = row[i].x * qs[0] + row[i].y * qs[1] + row[i].z * qs[2] + row[i].w * qs[3];
            }
#pragma unroll
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) ov[i] += __shfl_xor_sync(0xffffffffu, ov[i], o);
            if (lane < 8) {
                float mine = ov[0];
#pragma unroll
                for (int i = 1; i < 8; ++i) mine = (lane == i) ? ov[i] : mine;
                op[v0 + lane] = __float2bfloat16_rn(mine);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) row[i] = nxt[i];
        }
    }
}

// One work item of the (K, V) layout = 16 value columns of one (sequence, value head) state, for one warp. `vec` is the warp's own
// [3][128] floats: gate, k-hat and scale * q-hat, read key by key.
__device__ __forceinline__ void dec_item_kv(const DecodeParams& p, const int item, float (*vec)[DK]) {
    const int lane = threadIdx.x & 31, cols = p.V >> 4;
    const int cs = item % cols, nh = item / cols;
    const int n = nh / p.HV, hv = nh - n * p.HV, hq = hv / (p.HV / p.H);
    const int rg = lane >> 2, c = 16 * cs + 4 * (lane & 3);      // rows rg, rg + 8, ..., columns c .. c + 3
    const int slot = p.indices ? p.indices[n] : n;
    __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.o) + ((size_t)n * p.HV + hv) * p.V + c;
    if (slot < 0) {                                         // padded sequence: no state access; its output row is zeroed
        if (rg == 0)
#pragma unroll
            for (int e = 0; e < 4; ++e) op[e] = __float2bfloat16_rn(0.f);
        return;
    }
    if (slot >= p.pool) {                                   // caller error: report, touch nothing
        if (lane == 0) report_status(p.status, STATUS_BAD_INDEX);
        return;
    }
    float* S = p.state + ((size_t)slot * p.HV + hv) * (size_t)DK * p.V + (size_t)rg * p.V + c;
    float4 row[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) row[i] = __ldcs(reinterpret_cast<const float4*>(S + (size_t)(8 * i) * p.V));
    {
        float gate[4], kh[4], qs[4];
        dec_key_vectors(p, n, hv, hq, 4 * lane, gate, kh, qs);
        *reinterpret_cast<float4*>(&vec[0][4 * lane]) = make_float4(gate[0], gate[1], gate[2], gate[3]);
        *reinterpret_cast<float4*>(&vec[1][4 * lane]) = make_float4(kh[0], kh[1], kh[2], kh[3]);
        *reinterpret_cast<float4*>(&vec[2][4 * lane]) = make_float4(qs[0], qs[1], qs[2], qs[3]);
        __syncwarp();
    }
    const float beta = 1.f / (1.f + __expf(-dec_load(p.b, p.b_fp32, (size_t)n * p.HV + hv)));
    const __nv_bfloat16* vp = reinterpret_cast<const __nv_bfloat16*>(p.v) + ((size_t)n * p.HV + hv) * p.V + c;      // v and o may be unaligned
    const float2 v0 = make_float2(__bfloat162float(vp[0]), __bfloat162float(vp[1])), v1 = make_float2(__bfloat162float(vp[2]), __bfloat162float(vp[3]));
    auto over_rows = [&](float4 a) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            a.x += __shfl_xor_sync(0xffffffffu, a.x, o); a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
            a.z += __shfl_xor_sync(0xffffffffu, a.z, o); a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
        }
        return a;
    };
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float w = vec[0][8 * i + rg] * vec[1][8 * i + rg];
        acc.x = fmaf(row[i].x, w, acc.x); acc.y = fmaf(row[i].y, w, acc.y);
        acc.z = fmaf(row[i].z, w, acc.z); acc.w = fmaf(row[i].w, w, acc.w);
    }
    acc = over_rows(acc);
    const float4 vn = make_float4(beta * (v0.x - acc.x), beta * (v0.y - acc.y), beta * (v1.x - acc.z), beta * (v1.y - acc.w));
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float gt = vec[0][8 * i + rg], kh = vec[1][8 * i + rg], qv = vec[2][8 * i + rg];
        row[i].x = fmaf(gt, row[i].x, kh * vn.x); row[i].y = fmaf(gt, row[i].y, kh * vn.y);
        row[i].z = fmaf(gt, row[i].z, kh * vn.z); row[i].w = fmaf(gt, row[i].w, kh * vn.w);
        __stcs(reinterpret_cast<float4*>(S + (size_t)(8 * i) * p.V), row[i]);
        acc.x = fmaf(row[i].x, qv, acc.x); acc.y = fmaf(row[i].y, qv, acc.y);
        acc.z = fmaf(row[i].z, qv, acc.z); acc.w = fmaf(row[i].w, qv, acc.w);
    }
    acc = over_rows(acc);
    if (rg == 0) {
        op[0] = __float2bfloat16_rn(acc.x); op[1] = __float2bfloat16_rn(acc.y);
        op[2] = __float2bfloat16_rn(acc.z); op[3] = __float2bfloat16_rn(acc.w);
    }
}

// One item per CTA (vk) or per warp (kv): a CTA that ends makes room for one that starts with all its loads, so that the memory
// system always has requests. (As four resident CTAs per SM that walked the items, 256 sequences x 32 heads in vk took 185.6 us a call for
// 1.08 GB; now 182.5, and 181 to 171 with the same pool over and over. Five or six CTAs per SM spill: 186, 208.)
__global__ void __launch_bounds__(DEC_THREADS, 4) kda_decode_kernel(const DecodeParams p) { dec_item(p, blockIdx.x); }
__global__ void __launch_bounds__(DEC_THREADS, 4) kda_decode_kv_kernel(const DecodeParams p, const int items) {
    __shared__ float vec[DEC_THREADS / 32][3][DK];
    const int warp = threadIdx.x >> 5;
    const long long item = (long long)(DEC_THREADS / 32) * blockIdx.x + warp;
    if (item < items) dec_item_kv(p, (int)item, vec[warp]);
}

}  // namespace kda

extern "C" int kda_launch_decode(const void* q, const void* k, const void* v, const void* a, int a_fp32, const void* b, int b_fp32,
                                 const float* A_log, const float* dt_bias, float* state, const int* indices, void* o,
                                 int N, int H, int HV, int V, int pool, float scale, int use_l2norm, float softplus_beta,
                                 float softplus_threshold, int state_kv, int* status, cudaStream_t stream) {
    using namespace kda;
    if (N <= 0) return 0;
    DecodeParams p{};
    p.q = q; p.k = k; p.v = v; p.a = a; p.b = b; p.A_log = A_log; p.dt_bias = dt_bias; p.state = state; p.indices = indices;
    p.o = o; p.N = N; p.H = H; p.HV = HV; p.V = V; p.pool = pool; p.a_fp32 = a_fp32; p.b_fp32 = b_fp32; p.use_l2norm = use_l2norm;
    p.state_kv = state_kv; p.scale = scale; p.softplus_beta = softplus_beta; p.softplus_threshold = softplus_threshold;
    p.status = status;
    if (state_kv) {
        const long long items = (long long)N * HV * (V / 16), ctas = (items + DEC_THREADS / 32 - 1) / (DEC_THREADS / 32);
        if (items > 0x7fffffffLL) return -1;
        kda_decode_kv_kernel<<<(int)ctas, DEC_THREADS, 0, stream>>>(p, (int)items);
        return (int)cudaGetLastError();
    }
    // enough CTAs to fill the machine several times over, else as few (= as much work per CTA) as possible
    const int sms = sm_count();
    int slices = 1;
    while (slices < V / 32 && (long long)N * HV * slices < 8LL * sms && (V / 32) % (2 * slices) == 0) slices *= 2;
    p.slices = slices;
    const long long items = (long long)N * HV * slices;
    if (items > 0x7fffffffLL) return -1;
    kda_decode_kernel<<<(int)items, DEC_THREADS, 0, stream>>>(p);
    return (int)cudaGetLastError();
}
