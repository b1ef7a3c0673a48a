// Reverse state scan of the backward pass, on tcgen05 (the mirror of kda_fwd_scan.cu).
//
// One CTA per (sequence, head) walks the chunks from last to first and carries the fp32 gradient of the state TRANSPOSED in tensor
// memory (dS^T: lane = value column, column = key channel); per chunk
//     ADO    = dO^T Aqk                              dO as fp16 A operand in tensor memory; nothing of this is on the chain
//     ACC    = S16 KG^T                              S16: dS' as fp16 A operand, one power-of-two scale per lane
//     dVn^T  = ACC + ADO                             gradient of v_new -> fp16 A operand (negated) and HBM
//     dS^T   = dS'^T diag(decay) + dO^T QG - dVn^T W (gradient of the state entering the chunk)
// What bounds a few long sequences is the latency of that chain: two MMA groups and two register passes per chunk. What bounds a
// full GPU is HBM, 154 KB in and out per chunk. (The register-resident mma.sync version of this scan ran 224 dependent-issue
// MMAs per warp and chunk: 3.2 us per chunk, now 2.27 with 2 heads. 4 sequences of 128 chunks x 32 heads 661 -> 429 us, cold, of
// which the bytes are 385.) The warps are those of the forward scan:
//   warps 0-3     dVn: lane-per-column values become token rows in shared memory and leave as one bulk store;
//   warps 4-19    dS': out of tensor memory, fp16 copy back in (chain), then the decayed state, dS' per chunk to HBM, dht / dh0;
//   warps 20-27   dVn (chain), 32 tokens each, and between two chunks the next dO as operand;
//   warp 28       issues the MMAs;
//   warp 29       streams the tile packs and the dO rows (2 stages) by TMA.
//
// Replaces chunk_gated_delta_rule_bwd_dhu (flash-linear-attention, fla/ops/common/chunk_delta_h.py:316-718, called
// at cula/kda/chunk_bwd.py:541-555) and the dv half of chunk_kda_bwd_kernel_dAv (cula/kda/chunk_bwd.py:63-125).
//
// Range: every gradient-like operand (dO, dht, dS', dVn) is carried in units of a power-of-two scale s chosen
// from max|dO|, max|dht| (kda_grad_amax_kernel), so fp16 MMA operands neither overflow nor go subnormal.
#include "kda_common.cuh"
#include "kda_params.h"
#include "scan_common.cuh"

namespace kda {

constexpr int BS_STAGES = 2;
constexpr int BS_OUT_WARPS = 4, BS_STATE_WARPS = 16, BS_VALUE_WARPS = 8;
constexpr int BS_MMA_WARP = BS_OUT_WARPS + BS_STATE_WARPS + BS_VALUE_WARPS, BS_LOAD_WARP = BS_MMA_WARP + 1;
constexpr int BS_THREADS = 32 * (BS_LOAD_WARP + 1);
// shared-memory stage: W, QG, KG as [2 atoms of 64 channels][64 tokens][128 B], Aqk, the dO rows as they are, the decays
constexpr int BS_W = 0, BS_QG = 16384, BS_KG = 32768, BS_AQK = 49152, BS_DO = 57344, BS_DECAY = 73728, BS_STAGE_BYTES = 74752;
static_assert(BS_STAGE_BYTES % 1024 == 0, "operand atoms are 1024-byte aligned");
constexpr int BS_OST_BYTES = BT * DV * 2;                    // staged dVn rows
constexpr int BS_OST = BS_STAGES * BS_STAGE_BYTES, BS_MISC = BS_OST + 2 * BS_OST_BYTES;
constexpr int BS_SMEM = BS_MISC + 8512 + 1024;
// tensor-memory columns: dS, its fp16 copy, two S16 KG^T accumulators (by turn parity; -dVn replaces what was read), two dO
// operands (by turn parity), dO^T Aqk
constexpr uint32_t BM_S32 = 0, BM_S16 = 128, BM_ACC = 192, BM_DO = 320, BM_ADO = 384;

constexpr int AMAX_THREADS = 512;
// s = 2^k with max(|dO|, |dht|) * s in [4, 8); written as {s, 1/s}. amax_bits holds the running maximum, gscale[0] counts the blocks that
// are done until the last one writes the scale there (both start as zero). The recomputation of the chunk-parallel stage, which reads none
// of this, may start under this kernel, but under nothing before it: the trigger stands behind the wait.
__global__ void kda_grad_amax_kernel(const __nv_bfloat16* d_o, size_t n_do, const float* dht, size_t n_dht,
                                     unsigned int* amax_bits, float* gscale) {
    pdl_wait();
    pdl_launch_dependents();
    float m = 0.f;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nthr = (size_t)gridDim.x * blockDim.x;
    // 16-byte loads over the bulk (the tensors come 16-byte aligned from the C ABI), scalar loads over the tail
    const uint4* do4 = reinterpret_cast<const uint4*>(d_o);
    auto take = [&](const uint4& v) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_bf16(w[e]);
            m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
    };
    size_t i0 = tid;
    for (; i0 + 7 * nthr < n_do / 8; i0 += 8 * nthr) {          // eight loads in flight per thread
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = do4[i0 + j * nthr];
#pragma unroll
        for (int j = 0; j < 8; ++j) take(v[j]);
    }
    for (; i0 < n_do / 8; i0 += nthr) take(do4[i0]);
    for (size_t i = (n_do / 8) * 8 + tid; i < n_do; i += nthr) m = fmaxf(m, fabsf(__bfloat162float(d_o[i])));
    const float4* h4 = reinterpret_cast<const float4*>(dht);
    size_t i1 = tid;
    for (; i1 + 7 * nthr < n_dht / 4; i1 += 8 * nthr) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = h4[i1 + j * nthr];
#pragma unroll
        for (int j = 0; j < 8; ++j) m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
    }
    for (; i1 < n_dht / 4; i1 += nthr) {
        const float4 v = h4[i1];
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    for (size_t i = (n_dht / 4) * 4 + tid; i < n_dht; i += nthr) m = fmaxf(m, fabsf(dht[i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    // one atomic per block instead of one per warp (33 MB: 14.4 -> 12.3 us)
    __shared__ float wmax[AMAX_THREADS / 32];
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m < INFINITY ? m : 0.f;
    __syncthreads();
    if (threadIdx.x == 0) {
        m = 0.f;
#pragma unroll
        for (int w = 0; w < AMAX_THREADS / 32; ++w) m = fmaxf(m, wmax[w]);
        if (m > 0.f) atomicMax(amax_bits, __float_as_uint(m));
        __threadfence();
        if (atomicAdd(reinterpret_cast<unsigned int*>(gscale), 1u) == gridDim.x - 1) {
            __threadfence();
            m = __uint_as_float(atomicMax(amax_bits, 0u));
            const int e = ((__float_as_int(m) >> 23) & 0xff) - 127;      // floor(log2 m); m == 0 gives -127
            int shift = m > 0.f ? 2 - e : 0;
            shift = max(-120, min(120, shift));
            gscale[0] = __int_as_float((shift + 127) << 23);
            gscale[1] = __int_as_float((127 - shift) << 23);
        }
    }
}

__global__ void __launch_bounds__(BS_THREADS, 1) kda_bwd_scan_kernel(const BwdScanParams p, const __grid_constant__ CUtensorMap map,
                                                                     const __grid_constant__ CUtensorMap map_do) {
    extern __shared__ unsigned char bs_smem_raw[];
    unsigned char* sm = bs_smem_raw + ((1024u - (smem_u32(bs_smem_raw) & 1023u)) & 1023u);
    const uint32_t smb = smem_u32(sm);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + BS_MISC);
    uint64_t *full = bars, *empty = bars + 2, *b_s16 = bars + 4, *b_dec = bars + 5, *b_acc = bars + 6, *b_s32 = bars + 7, *b_do = bars + 8,
             *b_ado = bars + 9, *b_ost = bars + 10, *b_vsum = bars + 11, *b_max = bars + 12 /* [4] */;
    // pairs, because a wait by phase parity must not fall two completions behind (see kda_fwd_scan.cu): turn i uses barrier i & 1
    uint64_t *b_v16 = bars + 16 /* [2] */, *b_oread = bars + 18 /* [2] */;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + BS_MISC + 240);
    float* sDown = reinterpret_cast<float*>(sm + BS_MISC + 256);         // [4 turns][128 value columns] 1 / scale of S16
    float* sMax = reinterpret_cast<float*>(sm + BS_MISC + 2304);         // [2 turn parities][4 key quarters][128] largest |decayed dS'| of a column
    float* sVsum = reinterpret_cast<float*>(sm + BS_MISC + 6400);        // [2 turn parities][2 token halves][128] sum of |dVn| + |dO|
    uint32_t* sQW = reinterpret_cast<uint32_t*>(sm + BS_MISC + 8448);    // [4 turns] what |qg| and |w| can reach (see or_operands)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.x, n = p.seq_order ? p.seq_order[blockIdx.y] : blockIdx.y;
    int bos, len, chunk0;
    if (p.cu_seqlens) {
        bos = p.cu_seqlens[n];
        len = p.cu_seqlens[n + 1] - bos;
        chunk0 = p.chunk_offsets[n];
    } else {
        bos = n * p.T;
        len = p.T;
        chunk0 = n * ((p.T + BT - 1) / BT);
    }
    const int nchunks = (len + BT - 1) / BT;

    if (tid == 0) {
        for (int s = 0; s < BS_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1 + BS_STATE_WARPS + BS_VALUE_WARPS);
        }
        mbar_init(b_s16, BS_STATE_WARPS);
        mbar_init(b_dec, BS_STATE_WARPS);
        mbar_init(b_acc, 1);
        mbar_init(b_s32, 1);
        mbar_init(b_do, BS_VALUE_WARPS);
        mbar_init(b_ado, 1);
        mbar_init(b_ost, BS_OUT_WARPS);
        mbar_init(b_vsum, BS_VALUE_WARPS);
        for (int b = 0; b < 4; ++b) sQW[b] = 0;
        for (int q = 0; q < 4; ++q) mbar_init(&b_max[q], BS_STATE_WARPS / 4);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&b_v16[b], BS_VALUE_WARPS);
            mbar_init(&b_oread[b], BS_OUT_WARPS);
        }
        fence_mbar_init();
    }
    if (warp == BS_MMA_WARP) umma::tmem_alloc(tmem_slot, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    auto wait = [&](uint64_t* bar, int phase) -> bool {
        if (mbar_wait(bar, phase & 1)) return true;
        report_status(p.status, STATUS_WAIT_TIMEOUT);
        return false;
    };

    if (warp == BS_LOAD_WARP) {
        // ------------------------------- producer -------------------------------
        // The ragged last chunk of a sequence, which comes first, fetches its dO rows one by one in a packed batch: a box of 64 rows
        // would reach past the end of the tensor, and how many rows that has is not known here (T says nothing about it). The map
        // of a fixed-length batch ends where the tensor does, and the box takes 1.7 us less.
        const int ragged = len - (nchunks - 1) * BT;
        const bool by_rows = p.cu_seqlens && ragged < BT;
        if (nchunks > 0 && by_rows) {
            if (lane == 0) mbar_expect_tx(&full[0], ragged * DV * 2);
            __syncwarp();
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(p.d_o) + ((size_t)(bos + (nchunks - 1) * BT) * p.H + h) * DV;
            for (int row = lane; row < ragged; row += 32) bulk_g2s(sm + BS_DO + row * DV * 2, src + (size_t)row * p.H * DV, DV * 2, &full[0]);
        }
        if (lane == 0) {
            int issued = 0;
            bool ok = true;
            for (int it = 0; it < nchunks; ++it) {
                const int c = nchunks - 1 - it, s = it % BS_STAGES, use = it / BS_STAGES;
                if (use > 0 && !(ok = wait(&empty[s], use - 1))) break;
                const int t_id = (chunk0 + c) * p.H + h;
                const unsigned char* tile = p.tiles + (size_t)t_id * TP_BYTES;
                unsigned char* dst = sm + s * BS_STAGE_BYTES;
                const uint32_t d = smb + s * BS_STAGE_BYTES;
                const bool box = it > 0 || !by_rows;
                mbar_arrive_expect_tx(&full[s], 3 * 16384 + 8192 + 512 + (box ? 16384 : 0));
                if (box) tma_load_3d(d + BS_DO, &map_do, 0, h, bos + c * BT, &full[s]);     // first: the value warps work on it ahead of the chain
                bulk_g2s(dst + BS_AQK, tile + TP_AQK, 8192, &full[s]);
#pragma unroll
                for (int m = 2; m >= 0; --m)       // KG, QG, W
#pragma unroll
                    for (int a = 0; a < 2; ++a) tma_load_4d(d + m * 16384 + a * 8192, &map, 0, a, 64 * m, t_id, &full[s]);
                bulk_g2s(dst + BS_DECAY, tile + TP_DECAY, 512, &full[s]);
                issued = it + 1;
            }
            // do not leave with copies to this CTA's shared memory in flight
            if (!ok)
                for (int it = max(0, issued - BS_STAGES); it < issued; ++it) mbar_wait(&full[it % BS_STAGES], (it / BS_STAGES) & 1);
        }
    } else if (warp == BS_MMA_WARP) {
        // ------------------------------- MMA issue (the whole warp in step, one elected lane issues) -------------------------------
        const uint32_t id_kg = umma::make_idesc(umma::FMT_F16, 128, 64, false, false);
        const uint32_t id_qw = umma::make_idesc(umma::FMT_F16, 128, 128, false, true);
        const uint32_t id_a = umma::make_idesc(umma::FMT_F16, 128, 64, false, true);
        for (int it = 0; it < nchunks; ++it) {
            const int s = it % BS_STAGES;
            const uint32_t st = smb + s * BS_STAGE_BYTES;
            const uint64_t d_kg = sc_sdesc(st + BS_KG, 16, 1024), d_qg = sc_sdesc(st + BS_QG, 8192, 1024), d_w = sc_sdesc(st + BS_W, 8192, 1024),
                           d_a = sc_sdesc(st + BS_AQK, 8192, 1024);
            const uint32_t acc = tmem + BM_ACC + 64 * (it & 1), t_do = tmem + BM_DO + 32 * (it & 1);
            if (!wait(&full[s], it / BS_STAGES) || !wait(b_do, it)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) umma::mma_f16_ta(tmem + BM_ADO, t_do + 8 * ks, d_a + ((ks * 2048) >> 4), id_a, ks != 0);
                umma::commit(b_ado);
            }
            __syncwarp();
            if (!wait(b_s16, it)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma::mma_f16_ta(acc, tmem + BM_S16 + 8 * ks, d_kg + (((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), id_kg, ks != 0);
                umma::commit(b_acc);
            }
            __syncwarp();
            if (!wait(b_dec, it)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) umma::mma_f16_ta(tmem + BM_S32, t_do + 8 * ks, d_qg + ((ks * 2048) >> 4), id_qw, 1);
            }
            __syncwarp();
            if (!wait(&b_v16[it & 1], it >> 1)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)       // -dVn^T: tokens 0..31 in columns 0..15, tokens 32..63 in columns 32..47 of the accumulator
                    umma::mma_f16_ta(tmem + BM_S32, acc + 32 * (ks >> 1) + 8 * (ks & 1), d_w + ((ks * 2048) >> 4), id_qw, 1);
                umma::commit(b_s32);
                umma::commit(&empty[s]);
            }
            __syncwarp();
            // the dVn of the turn before has been read: its accumulator is free for the next turn
            if (p.dvn_out && it > 0 && !wait(&b_oread[(it - 1) & 1], (it - 1) >> 1)) break;
        }
    } else if (warp >= BS_OUT_WARPS && warp < BS_OUT_WARPS + BS_STATE_WARPS) {
        // ------------------------------- dS: lane = value column v, 32 key channels per warp -------------------------------
        const int q = warp & 3, kq = (warp - BS_OUT_WARPS) >> 2, v = 32 * q + lane, k0 = 32 * kq;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        float s[32];
        if (p.dht) {
            const float gs = p.gscale[0];
            const float* d0 = p.dht + ((size_t)n * p.H + h) * DK * DV + (size_t)k0 * DV + v;
#pragma unroll
            for (int k = 0; k < 32; ++k) s[k] = gs * d0[(size_t)k * DV];
        } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) s[k] = 0.f;
        }
        auto load_state = [&]() {
            umma::ld_32x32b_x32(tl + BM_S32 + k0, reinterpret_cast<uint32_t(&)[32]>(s));
            umma::wait_ld();
        };
        // Largest |entry| of the value column in what turn `it` starts from, the decayed dS' of the turn before (see kda_fwd_scan.cu).
        auto publish_max = [&](int it, float decay) {
            sMax[(it & 1) * 512 + kq * 128 + v] = abs_max(s) * decay;
            warp_arrive(&b_max[q], lane);
        };
        bool ok = true;
        if (nchunks > 0) publish_max(0, 1.f);
        for (int it = 0; it < nchunks; ++it) {
            const int c = nchunks - 1 - it;
            // The scale of the fp16 copy comes from a bound that is known before the state is (see kda_fwd_scan.cu):
            // |dS| <= max |decayed dS'| + max(|qg|, |w|) (sum |dO| + sum |dVn|).
            if (!(ok = wait(&b_max[q], it))) break;
            const float* mx = sMax + (it & 1) * 512 + v;
            float bound = fmaxf(fmaxf(mx[0], mx[128]), fmaxf(mx[256], mx[384]));
            if (it > 0) {
                const int pt = (it - 1) & 1;
                if (!(ok = wait(b_vsum, it - 1))) break;
                bound = fmaf(or_bound(sQW[(it - 1) & 3]), sVsum[pt * 256 + v] + sVsum[pt * 256 + 128 + v], bound);
            }
            float up, down;
            fp16_scale(bound, up, down);
            if (kq == 0) sDown[(it & 3) * 128 + v] = down;
            if (it > 0) {
                if (!(ok = wait(b_s32, it - 1))) break;
                umma::fence_after_sync();
                load_state();
            }
            store_f16(tl + BM_S16 + 16 * kq, s, up);
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(b_s16, lane);
            // ---- beside the MMAs: the decayed state, then dS' (gradient of the state leaving this chunk) to HBM ----
            const int st = it % BS_STAGES;
            if (!(ok = wait(&full[st], it / BS_STAGES))) break;
            const float* dec = reinterpret_cast<const float*>(sm + st * BS_STAGE_BYTES + BS_DECAY) + k0;
            const float dec_lane = dec[lane];
            store_decayed(tl + BM_S32 + k0, s, dec);
            warp_arrive(&empty[st], lane);
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(b_dec, lane);
            publish_max(it + 1, warp_max_decay(dec_lane));
            if (p.ds_out) {
                float* dsg = p.ds_out + ((size_t)(chunk0 + c) * p.H + h) * (size_t)(DK * DV) + (size_t)k0 * DV + v;
#pragma unroll
                for (int k = 0; k < 32; ++k) dsg[(size_t)k * DV] = s[k];
            }
        }
        if (ok && nchunks > 0 && (ok = wait(b_s32, nchunks - 1))) {
            umma::fence_after_sync();
            load_state();
        }
        if (ok && p.dh0) {
            const float gs_inv = p.gscale[1];
            float* d0 = p.dh0 + ((size_t)n * p.H + h) * DK * DV + (size_t)k0 * DV + v;
#pragma unroll
            for (int k = 0; k < 32; ++k) d0[(size_t)k * DV] = gs_inv * s[k];
        }
    } else if (warp >= BS_OUT_WARPS + BS_STATE_WARPS) {
        // ------------------------------- dVn: lane = value column v, 32 tokens per warp -------------------------------
        const int q = warp & 3, th = (warp - BS_OUT_WARPS - BS_STATE_WARPS) >> 2, v = 32 * q + lane, t0 = 32 * th;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        const float gs = p.gscale[0];
        float dosum = 0.f;
        // dO^T of a turn as fp16 A operand, in units of gs; rows past the end of the sequence belong to others and count as zero
        auto convert = [&](int it) -> bool {
            const int st = it % BS_STAGES, rows = min(BT, len - (nchunks - 1 - it) * BT) - t0;
            if (!wait(&full[st], it / BS_STAGES)) return false;
            const unsigned char* src = sm + st * BS_STAGE_BYTES + BS_DO + t0 * 256 + v * 2;
            uint32_t pk[16];
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const uint32_t a = *reinterpret_cast<const uint16_t*>(src + (2 * e) * 256), b = *reinterpret_cast<const uint16_t*>(src + (2 * e + 1) * 256);
                const float2 f = make_float2(2 * e < rows ? gs * __uint_as_float(a << 16) : 0.f, 2 * e + 1 < rows ? gs * __uint_as_float(b << 16) : 0.f);
                sum.x += fabsf(f.x);
                sum.y += fabsf(f.y);
                pk[e] = pack_f16(f.x, f.y);
            }
            dosum = sum.x + sum.y;
            umma::st_32x32b_x16(tl + BM_DO + 32 * (it & 1) + 16 * th, pk);
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(b_do, lane);
            static_assert(BS_W == 0 && BS_QG == 16384, "one range");
            or_operands<32768 / BS_VALUE_WARPS>(sm + st * BS_STAGE_BYTES + (4 * th + q) * (32768 / BS_VALUE_WARPS), lane, &sQW[it & 3]);
            warp_arrive(&empty[st], lane);
            return true;
        };
        bool ok = nchunks == 0 || convert(0);
        for (int it = 0; ok && it < nchunks; ++it) {
            uint32_t ado[32];
            if (!wait(b_ado, it)) break;
            umma::fence_after_sync();
            umma::ld_32x32b_x32(tl + BM_ADO + t0, ado);
            umma::wait_ld();
            if (!wait(b_s16, it) || !wait(b_acc, it)) break;
            if (q == 0 && th == 0 && lane == 0) sQW[(it + 2) & 3] = 0;      // see kda_fwd_scan.cu
            umma::fence_after_sync();
            const uint32_t acc = tl + BM_ACC + 64 * (it & 1) + t0;
            const float2 down = splat2(sDown[(it & 3) * 128 + v]);
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[16], pk[8];
                umma::ld_32x32b_x16(acc + 16 * b, r);
                umma::wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 x = fma2(make_float2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), down,
                                          make_float2(__uint_as_float(ado[16 * b + 2 * e]), __uint_as_float(ado[16 * b + 2 * e + 1])));
                    pk[e] = pack_f16(x.x, x.y) ^ 0x80008000u;
                    sum.x += fabsf(x.x);
                    sum.y += fabsf(x.y);
                }
                umma::st_32x32b_x8(acc + 8 * b, pk);      // columns this warp has already read
            }
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(&b_v16[it & 1], lane);
            sVsum[(it & 1) * 256 + th * 128 + v] = sum.x + sum.y + dosum;
            warp_arrive(b_vsum, lane);
            // the operand buffer and the product of two turns ago are free: b_acc of this turn came after their last MMA
            if (it + 1 < nchunks) ok = convert(it + 1);
        }
    } else if (p.dvn_out) {
        // ------------------------------- dVn rows: lane = value column v, all tokens -------------------------------
        const int q = warp, v = 32 * q + lane;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        for (int it = 0; it < nchunks; ++it) {
            if (it + 1 == nchunks) pdl_launch_dependents();      // the last chunk: the dense stage may be set up
            const uint32_t acc = tl + BM_ACC + 64 * (it & 1);
            if (!wait(&b_v16[it & 1], it >> 1)) break;
            umma::fence_after_sync();
            unsigned char* buf = sm + BS_OST + (it & 1) * BS_OST_BYTES;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                uint32_t w[8];
                umma::ld_32x32b_x8(acc + 32 * (b >> 1) + 8 * (b & 1), w);
                umma::wait_ld();
                if (b == 3) {
                    umma::fence_before_sync();
                    warp_arrive(&b_oread[it & 1], lane);
                }
                stage_rows(buf, 16 * b, v, w, 0x80008000u);
            }
            arrive_staged(b_ost, tid);
            if (!wait(b_ost, it)) break;
            if (tid == 0) {
                bulk_s2g(reinterpret_cast<unsigned char*>(p.dvn_out) + ((size_t)(chunk0 + nchunks - 1 - it) * p.H + h) * (size_t)(BT * DV * 2), buf,
                         BS_OST_BYTES);
                bulk_commit();
            }
        }
        if (tid == 0) bulk_wait_all();
    }
    __syncthreads();
    if (warp == BS_MMA_WARP) umma::tmem_dealloc(tmem, 512);
    // Beside the forward scan: it reads nothing of that scan, and was launched when the tile packs were complete (the trigger
    // stands behind the forward scan's own wait). What follows in the stream counts on both, so this grid ends after it.
    // Forward + backward against the two one after the other: 2 x 1000 x 3 heads 198 -> 157 us, 2 x 2048 x 32 (scalar gate) 909 -> 858,
    // 4 x 8192 x 32, where the forward scan leaves 20 SMs, 6386 -> 6351.
    pdl_wait();
}

}  // namespace kda

extern "C" int kda_launch_clear(unsigned int* dst, long long words, cudaStream_t stream);

extern "C" int kda_launch_grad_scale(const void* d_o, size_t n_do, const float* dht, size_t n_dht, unsigned int* amax_bits,
                                     float* gscale, cudaStream_t stream) {
    using namespace kda;
    const bool one_piece = reinterpret_cast<float*>(amax_bits) == gscale + 2;
    int rc = kda_launch_clear(reinterpret_cast<unsigned int*>(gscale), one_piece ? 3 : 1, stream);
    if (rc == 0 && !one_piece) rc = kda_launch_clear(amax_bits, 1, stream);
    if (rc != 0) return rc;
    // a block per 512 16-byte pieces, up to four of 512 threads per SM
    if (!dht) n_dht = 0;
    const size_t pieces = (n_do / 8 > n_dht / 4 ? n_do / 8 : n_dht / 4) / AMAX_THREADS + 1, most = (size_t)4 * sm_count();
    return (int)launch_early(kda_grad_amax_kernel, dim3((unsigned)(pieces < most ? pieces : most)), AMAX_THREADS, 0, stream,
                             reinterpret_cast<const __nv_bfloat16*>(d_o), n_do, dht, n_dht, amax_bits, gscale);
}

extern "C" int kda_launch_bwd_scan(const kda::BwdScanParams* p, cudaStream_t stream) {
    using namespace kda;
    if (p->N <= 0) return 0;
    static std::atomic<unsigned long long> done;
    cudaError_t e = allow_smem(kda_bwd_scan_kernel, BS_SMEM, done);
    if (e != cudaSuccess) return (int)e;
    // the numbers of tiles and (of a packed batch) tokens are not known here; the kernel's coordinates stay inside the caller's tensors
    CUtensorMap map, map_do;
    if (!make_pack_map(&map, p->tiles, 1ll << 24) || !make_rows_map(&map_do, const_cast<void*>(p->d_o), p->H, p->cu_seqlens ? 1ll << 30 : (long long)p->N * p->T))
        return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p->H, p->N);
    cfg.blockDim = dim3(BS_THREADS);
    cfg.dynamicSmemBytes = BS_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p->beside_forward ? 1 : 0;
    const cudaError_t launch = launched(cudaLaunchKernelEx(&cfg, kda_bwd_scan_kernel, *p, map, map_do));
    return (int)(launch != cudaSuccess ? launch : cudaGetLastError());
}
