// Sequential state scan fused with the output stage, on tcgen05.
//
// One CTA per (sequence, head) carries the fp32 state TRANSPOSED in tensor memory (S^T: lane = value column, column = key
// channel) over the chunks; per chunk
//     ACC  = S16 [W | QG]^T             S16: the state as fp16 A operand in tensor memory, one power-of-two scale per lane
//     v_new^T = u^T - ACC_W             -> fp16 A operand in tensor memory (over the columns it was computed from)
//     S^T  = S^T diag(decay) + v_new^T KG
//     o^T  = ACC_QG + v_new^T Aqk^T
// What bounds it is the latency of that chain, not the tensor pipe: two MMA groups and two register passes per chunk, each
// handed over by an mbarrier. So everything that is not on the chain runs beside it, in warps of its own. (Measured, 2 heads: 1.62
// us per chunk + 10 us, cold; 2.0 per chunk with the state in mma.sync registers. 0.1 of it is the bound on |kg|.)
//   warps 0-3     output rows and, when asked for, v_new: lane-per-column values are turned into token rows in shared memory
//                 and leave as one bulk (tensor) store;
//   warps 4-19    state: S out of tensor memory, fp16 copy back in (chain), then the decayed state (beside the MMAs),
//                 per-chunk states to HBM when asked for, initial / final state; four warps share a lane quadrant, 32 key
//                 channels each;
//   warps 20-27   v_new (chain), 32 tokens each;
//   warp 28       issues the MMAs;
//   warp 29       streams the tile packs (2 stages): TMA tensor boxes lay W, QG, KG out as 128-byte-swizzled operand atoms
//                 (the pack keeps 256-byte rows; its XOR swizzle is that of the atoms), untiled bulk copies bring the rest.
//
// The same kernel computes shard transitions S_out = M S_in + C for context parallelism (grid.z: 0 carries C from a zero
// state, 1 carries the K x K matrix M from the identity with u = 0; no output rows).
//
// Replaces chunk_gated_delta_rule_fwd_h (cula/ops/chunk_delta_h.py:1991-2168) and chunk_gla_fwd_o
// (cula/ops/fwd_o.py:1755-1852); the per-chunk states h and v_new only go to HBM when the caller
// asks for them (backward recomputation, return_intermediate_states). Every wait is bounded: on expiry the status word is
// set, all roles unwind to the end of the kernel, and the tensor memory is freed.
#include "kda_common.cuh"
#include "kda_params.h"
#include "scan_common.cuh"

namespace kda {

constexpr int SC_STAGES = 2;
constexpr int SC_OUT_WARPS = 4, SC_STATE_WARPS = 16, SC_VALUE_WARPS = 8;
constexpr int SC_MMA_WARP = SC_OUT_WARPS + SC_STATE_WARPS + SC_VALUE_WARPS, SC_LOAD_WARP = SC_MMA_WARP + 1;
constexpr int SC_THREADS = 32 * (SC_LOAD_WARP + 1);
// shared-memory stage: B operands as [2 k-atoms of 64 channels][W 64 rows | QG 64 rows][128 B], KG as [2 mn-atoms][64 tokens]
// [128 B], then the rest of the pack as it is
constexpr int ST_WQ = 0, ST_KG = 32768, ST_AQK = 49152, ST_U = 57344, ST_DECAY = 73728, SC_STAGE_BYTES = 74752;
static_assert(SC_STAGE_BYTES % 1024 == 0, "operand atoms are 1024-byte aligned");
constexpr int OST_BYTES = 64 * 256;                          // staged token rows
constexpr int SC_OST = SC_STAGES * SC_STAGE_BYTES, SC_MISC = SC_OST + 2 * OST_BYTES;
constexpr int SC_SMEM = SC_MISC + 8512 + 1024;
// tensor-memory columns: the state, its fp16 copy, two [W | QG] accumulators (by chunk parity, so that the next chunk's product
// does not wait until this one's outputs have been read), the Aqk product
constexpr uint32_t TM_S32 = 0, TM_S16 = 128, TM_ACC = 192, TM_QG = 64 /* inside an accumulator */, TM_O2 = 448;

__device__ __forceinline__ void tma_store_rows(const CUtensorMap* map, uint32_t smem_src, int h, int row) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 :: "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_src), "r"(0), "r"(h), "r"(row) : "memory");
}
__global__ void __launch_bounds__(SC_THREADS, 1) kda_fwd_scan_kernel(const ScanParams p, const __grid_constant__ CUtensorMap map,
                                                                     const __grid_constant__ CUtensorMap map_o) {
    extern __shared__ unsigned char sc_smem_raw[];
    unsigned char* sm = sc_smem_raw + ((1024u - (smem_u32(sc_smem_raw) & 1023u)) & 1023u);
    const uint32_t smb = smem_u32(sm);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + SC_MISC);
    uint64_t *full = bars, *empty = bars + 2, *b_s16 = bars + 4, *b_dec = bars + 6, *b_acc = bars + 7, *b_s32 = bars + 9, *b_o = bars + 10,
             *b_ost = bars + 12, *b_vsum = bars + 13, *b_max = bars + 14 /* [4] */;
    // A wait by phase parity must not fall two completions behind. v_new can be ready, and have been read, for a chunk while the
    // other side still waits for the chunk before it, so these two are pairs: chunk c uses barrier c & 1 in its phase c / 2.
    uint64_t *b_v16 = bars + 18 /* [2] */, *b_oread = bars + 20 /* [2] */;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + SC_MISC + 240);
    float* sDown = reinterpret_cast<float*>(sm + SC_MISC + 256);         // [4 chunks][128 value columns] 1 / scale of S16: the output warps may be a chunk behind
    float* sMax = reinterpret_cast<float*>(sm + SC_MISC + 2304);         // [2 chunk parities][4 key quarters][128] largest |decayed S| of a column
    float* sVsum = reinterpret_cast<float*>(sm + SC_MISC + 6400);        // [2 chunk parities][2 token halves][128] sum of |v_new|
    uint32_t* sKg = reinterpret_cast<uint32_t*>(sm + SC_MISC + 8448);    // [4 chunks] what |kg| can reach (see or_operands)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.x, n = p.seq_order ? p.seq_order[blockIdx.y] : blockIdx.y;
    const bool is_m = blockIdx.z == 1, want_o = p.o != nullptr, want_out = want_o || p.vnew_out;
    int bos, len, chunk0;
    if (p.cu_seqlens) {
        bos = p.cu_seqlens[n];
        len = p.cu_seqlens[n + 1] - bos;
        chunk0 = p.chunk_offsets[n];
    } else {
        bos = n * (p.stride ? p.stride : p.T);
        len = p.T;
        chunk0 = n * ((p.T + BT - 1) / BT);
    }
    const int nchunks = (len + BT - 1) / BT;

    if (tid == 0) {
        for (int s = 0; s < SC_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1 + SC_STATE_WARPS + SC_VALUE_WARPS);
        }
        mbar_init(b_s16, SC_STATE_WARPS);
        mbar_init(b_dec, SC_STATE_WARPS);
        mbar_init(b_acc, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&b_v16[b], SC_VALUE_WARPS);
            mbar_init(&b_oread[b], SC_OUT_WARPS);
        }
        mbar_init(b_vsum, SC_VALUE_WARPS);
        for (int b = 0; b < 4; ++b) sKg[b] = 0;
        mbar_init(b_s32, 1);
        mbar_init(b_o, 1);
        mbar_init(b_ost, SC_OUT_WARPS);
        for (int q = 0; q < 4; ++q) mbar_init(&b_max[q], SC_STATE_WARPS / 4);
        fence_mbar_init();
    }
    if (warp == SC_MMA_WARP) umma::tmem_alloc(tmem_slot, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    // Everything this kernel reads (tile packs, initial states) may come from the kernels before it in the stream; with
    // programmatic stream serialization the CTA can be resident before they have finished, so wait here (a no-op when
    // the launch does not carry the attribute). Only scheduling, the index arithmetic and the set-up above overlap.
    // A chunk-parallel stage of later tokens that follows may start once every CTA of this grid has its SM; the reverse scan of
    // the same tiles only once the tiles are complete, i.e. behind the wait.
    if (!p.reverse_follows) pdl_launch_dependents();
    pdl_wait();
    if (p.reverse_follows) pdl_launch_dependents();

    auto wait = [&](uint64_t* bar, int phase) -> bool {
        if (mbar_wait(bar, phase & 1)) return true;
        report_status(p.status, STATUS_WAIT_TIMEOUT);
        return false;
    };

    if (warp == SC_LOAD_WARP) {
        // ------------------------------- producer -------------------------------
        if (lane == 0) {
            int issued = 0;
            bool ok = true;
            for (int c = 0; c < nchunks; ++c) {
                const int s = c % SC_STAGES, use = c / SC_STAGES;
                if (use > 0 && !(ok = wait(&empty[s], use - 1))) break;
                const int t_id = (chunk0 + c) * p.H + h;
                const unsigned char* tile = p.tiles + (size_t)t_id * TP_BYTES;
                unsigned char* dst = sm + s * SC_STAGE_BYTES;
                const uint32_t d = smb + s * SC_STAGE_BYTES;
                mbar_arrive_expect_tx(&full[s], 16384 + 16384 + 512 + (is_m ? 0 : 16384) + (want_o ? 16384 + 8192 : 0));
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    tma_load_4d(d + ST_WQ + a * 16384, &map, 0, a, 0, t_id, &full[s]);
                    if (want_o) tma_load_4d(d + ST_WQ + a * 16384 + 8192, &map, 0, a, 64, t_id, &full[s]);
                }
                bulk_g2s(dst + ST_DECAY, tile + TP_DECAY, 512, &full[s]);
                if (!is_m) bulk_g2s(dst + ST_U, tile + TP_U, 16384, &full[s]);
#pragma unroll
                for (int a = 0; a < 2; ++a) tma_load_4d(d + ST_KG + a * 8192, &map, 0, a, 128, t_id, &full[s]);
                if (want_o) bulk_g2s(dst + ST_AQK, tile + TP_AQK, 8192, &full[s]);
                issued = c + 1;
            }
            // do not leave with copies to this CTA's shared memory in flight
            if (!ok)
                for (int c = max(0, issued - SC_STAGES); c < issued; ++c) mbar_wait(&full[c % SC_STAGES], (c / SC_STAGES) & 1);
        }
    } else if (warp == SC_MMA_WARP) {
        // ------------------------------- MMA issue (the whole warp in step, one elected lane issues) -------------------------------
        const uint32_t id_wq = umma::make_idesc(umma::FMT_F16, 128, want_o ? 128 : 64, false, false);
        const uint32_t id_kg = umma::make_idesc(umma::FMT_F16, 128, 128, false, true);
        const uint32_t id_o2 = umma::make_idesc(umma::FMT_F16, 128, 64, false, false);
        for (int c = 0; c < nchunks; ++c) {
            const int s = c % SC_STAGES;
            // descriptors differ in their address field (16-byte units) only
            const uint64_t d_wq = sc_sdesc(smb + s * SC_STAGE_BYTES + ST_WQ, 16, 1024), d_kg = sc_sdesc(smb + s * SC_STAGE_BYTES + ST_KG, 8192, 1024),
                           d_aqk = sc_sdesc(smb + s * SC_STAGE_BYTES + ST_AQK, 16, 1024);
            const uint32_t acc = tmem + TM_ACC + 128 * (c & 1);
            if (!wait(&full[s], c / SC_STAGES)) break;
            if (!wait(b_s16, c)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma::mma_f16_ta(acc, tmem + TM_S16 + 8 * ks, d_wq + (((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), id_wq, ks != 0);
                umma::commit(b_acc);
            }
            __syncwarp();
            if (!wait(b_dec, c) || !wait(&b_v16[c & 1], c >> 1)) break;
            umma::fence_after_sync();
            if (umma::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)       // v_new^T: tokens 0..31 in columns 0..15, tokens 32..63 in columns 32..47 of the W accumulator
                    umma::mma_f16_ta(tmem + TM_S32, acc + 32 * (ks >> 1) + 8 * (ks & 1), d_kg + ((ks * 2048) >> 4), id_kg, 1);
                umma::commit(b_s32);
            }
            __syncwarp();
            // the previous chunk's outputs and v_new have been read: TM_O2 is free, and so is the next product's accumulator
            if (want_out && c > 0 && !wait(&b_oread[(c - 1) & 1], (c - 1) >> 1)) break;
            if (umma::elect_one()) {
                if (want_o) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        umma::mma_f16_ta(tmem + TM_O2, acc + 32 * (ks >> 1) + 8 * (ks & 1), d_aqk + ((ks * 32) >> 4), id_o2, ks != 0);
                    umma::commit(b_o);
                }
                umma::commit(&empty[s]);
            }
            __syncwarp();
        }
    }
    else if (warp >= SC_OUT_WARPS && warp < SC_OUT_WARPS + SC_STATE_WARPS) {
        // ------------------------------- state: lane = value column v, 32 key channels per warp -------------------------------
        const int q = warp & 3, kq = (warp - SC_OUT_WARPS) >> 2, v = 32 * q + lane, k0 = 32 * kq;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        float s[32];
        if (is_m) {
#pragma unroll
            for (int k = 0; k < 32; ++k) s[k] = k0 + k == v ? 1.f : 0.f;
        } else if (p.h0) {
            const float* h0 = p.h0 + ((size_t)n * p.H + h) * DK * DV + (size_t)k0 * DV + v;
#pragma unroll
            for (int k = 0; k < 32; ++k) s[k] = h0[(size_t)k * DV];
        } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) s[k] = 0.f;
        }
        auto load_state = [&]() {
            umma::ld_32x32b_x32(tl + TM_S32 + k0, reinterpret_cast<uint32_t(&)[32]>(s));
            umma::wait_ld();
        };
        // Largest |entry| of the value column in what chunk c starts from, the decayed state of chunk c - 1 (before chunk 0 the state
        // itself): this warp's quarter of the keys here, the others from the partner warps. `decay`: largest of the quarter.
        auto publish_max = [&](int c, float decay) {
            sMax[(c & 1) * 512 + kq * 128 + v] = abs_max(s) * decay;
            warp_arrive(&b_max[q], lane);
        };
        bool ok = true;
        if (nchunks > 0) publish_max(0, 1.f);
        for (int c = 0; c < nchunks; ++c) {
            // The scale of the fp16 copy has to be known when the state arrives, not a reduction over it later. A bound is
            // enough, fp16 being a floating-point format: |S_c| <= max |decayed S_{c-1}| + max |kg| sum |v_new|, whose terms are
            // ready before the MMA that makes S_c is. It holds for any keys and decays, so the copy stays below 2^14; where the
            // terms of the sum cancel it is some binades smaller, of which fp16 has 28 before it loses bits of the largest entries.
            if (!(ok = wait(&b_max[q], c))) break;
            const float* mx = sMax + (c & 1) * 512 + v;
            float bound = fmaxf(fmaxf(mx[0], mx[128]), fmaxf(mx[256], mx[384]));
            if (c > 0) {
                const int pc = (c - 1) & 1;
                if (!(ok = wait(b_vsum, c - 1))) break;
                bound = fmaf(or_bound(sKg[(c - 1) & 3]), sVsum[pc * 256 + v] + sVsum[pc * 256 + 128 + v], bound);
            }
            float up, down;
            fp16_scale(bound, up, down);
            if (kq == 0) sDown[(c & 3) * 128 + v] = down;
            if (c > 0) {
                if (!(ok = wait(b_s32, c - 1))) break;
                umma::fence_after_sync();
                load_state();
            }
            store_f16(tl + TM_S16 + 16 * kq, s, up);
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(b_s16, lane);
            // ---- beside the MMAs: the decayed state, then the state entering this chunk to HBM if asked for ----
            const int st = c % SC_STAGES;
            if (!(ok = wait(&full[st], c / SC_STAGES))) break;
            const float* dec = reinterpret_cast<const float*>(sm + st * SC_STAGE_BYTES + ST_DECAY) + k0;
            const float dec_lane = dec[lane];
            store_decayed(tl + TM_S32 + k0, s, dec);
            warp_arrive(&empty[st], lane);
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(b_dec, lane);
            publish_max(c + 1, warp_max_decay(dec_lane));
            const size_t tile_idx = (size_t)(chunk0 + c) * p.H + h;
            if (p.h32_out) {
                float* hg = p.h32_out + tile_idx * (size_t)(DK * DV) + (size_t)k0 * DV + v;
#pragma unroll
                for (int k = 0; k < 32; ++k) hg[(size_t)k * DV] = s[k];
            }
            if (p.h_out) {
                __nv_bfloat16* hg = reinterpret_cast<__nv_bfloat16*>(p.h_out) + tile_idx * (size_t)(DK * DV) + (size_t)k0 * DV + v;
#pragma unroll
                for (int k = 0; k < 32; ++k) hg[(size_t)k * DV] = __float2bfloat16_rn(s[k]);
            }
        }
        float* final_dst = is_m ? p.m_out : p.ht;
        if (ok && nchunks > 0 && (ok = wait(b_s32, nchunks - 1))) {
            umma::fence_after_sync();
            load_state();
        }
        if (ok && final_dst) {
            float* ht = final_dst + ((size_t)n * p.H + h) * DK * DV + (size_t)k0 * DV + v;
#pragma unroll
            for (int k = 0; k < 32; ++k) ht[(size_t)k * DV] = s[k];
        }
    } else if (warp >= SC_OUT_WARPS + SC_STATE_WARPS) {
        // ------------------------------- v_new: lane = value column v, 32 tokens per warp -------------------------------
        const int q = warp & 3, th = (warp - SC_OUT_WARPS - SC_STATE_WARPS) >> 2, v = 32 * q + lane, t0 = 32 * th;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        // u[token][v] of the pack: value halves of 128-byte token rows, 16-byte groups XOR-swizzled by the token
        const int ub = ST_U + (v >> 6) * 8192 + (v & 7) * 2, uc = (v & 63) >> 3;
        for (int c = 0; c < nchunks; ++c) {
            const int st = c % SC_STAGES;
            uint32_t u2[16];                          // this lane's u of 32 tokens, two per register
            if (!wait(&full[st], c / SC_STAGES)) break;
            or_operands<16384 / SC_VALUE_WARPS>(sm + st * SC_STAGE_BYTES + ST_KG + (4 * th + q) * (16384 / SC_VALUE_WARPS), lane, &sKg[c & 3]);
            if (!is_m) {
                const unsigned char* us = sm + st * SC_STAGE_BYTES + ub;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const uint32_t a = *reinterpret_cast<const uint16_t*>(us + (t0 + 2 * e) * 128 + ((uc ^ ((2 * e) & 7)) << 4));
                    const uint32_t b = *reinterpret_cast<const uint16_t*>(us + (t0 + 2 * e + 1) * 128 + ((uc ^ ((2 * e + 1) & 7)) << 4));
                    u2[e] = __byte_perm(a, b, 0x5410);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) u2[e] = 0;
            }
            warp_arrive(&empty[st], lane);
            if (!wait(b_s16, c) || !wait(b_acc, c)) break;
            if (q == 0 && th == 0 && lane == 0) sKg[(c + 2) & 3] = 0;      // chunk c - 2 is behind the state warps, c + 2 ahead of every value warp
            umma::fence_after_sync();
            const uint32_t acc = tl + TM_ACC + 128 * (c & 1) + t0;
            const float2 down = splat2(-sDown[(c & 3) * 128 + v]);
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[16], pk[8];
                umma::ld_32x32b_x16(acc + 16 * b, r);
                umma::wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 x = fma2(make_float2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), down, unpack_f16(u2[8 * b + e]));
                    pk[e] = pack_f16(x.x, x.y);
                    sum.x += fabsf(x.x);
                    sum.y += fabsf(x.y);
                }
                umma::st_32x32b_x8(acc + 8 * b, pk);      // columns this warp has already read
            }
            umma::wait_st();
            umma::fence_before_sync();
            warp_arrive(&b_v16[c & 1], lane);
            sVsum[(c & 1) * 256 + th * 128 + v] = sum.x + sum.y;
            warp_arrive(b_vsum, lane);
        }
    } else {
        // ------------------------------- output rows (and v_new): lane = value column v, all tokens -------------------------------
        const int q = warp, v = 32 * q + lane;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
        int turns = 0;                               // staged matrices so far: the two buffers alternate
        // All rows staged: thread 0 sends a whole matrix with one bulk copy (v_new, or a full chunk of o); a ragged last chunk
        // goes out row by row. Passing the barrier of turn t also means that the copy of turn t - 1 has been read out.
        auto turn_over = [&]() -> bool {
            arrive_staged(b_ost, tid);
            return wait(b_ost, turns++);
        };
        for (int c = 0; want_out && c < nchunks; ++c) {
            const uint32_t acc = tl + TM_ACC + 128 * (c & 1);
            if (p.vnew_out) {
                if (!wait(&b_v16[c & 1], c >> 1)) break;
                umma::fence_after_sync();
                unsigned char* buf = sm + SC_OST + (turns & 1) * OST_BYTES;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t w[8];
                    umma::ld_32x32b_x8(acc + 32 * (b >> 1) + 8 * (b & 1), w);
                    umma::wait_ld();
                    stage_rows(buf, 16 * b, v, w);
                }
                if (!want_o) {
                    umma::fence_before_sync();
                    warp_arrive(&b_oread[c & 1], lane);
                }
                if (!turn_over()) break;
                if (tid == 0) {
                    bulk_s2g(reinterpret_cast<unsigned char*>(p.vnew_out) + ((size_t)(chunk0 + c) * p.H + h) * (size_t)(BT * DV * 2), buf, OST_BYTES);
                    bulk_commit();
                }
            }
            if (want_o) {
                if (!wait(b_o, c)) break;
                umma::fence_after_sync();
                const float2 down = splat2(sDown[(c & 3) * 128 + v]);
                unsigned char* buf = sm + SC_OST + (turns & 1) * OST_BYTES;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t r[16], r2[16], w[8];
                    umma::ld_32x32b_x16(acc + TM_QG + 16 * b, r);
                    umma::ld_32x32b_x16(tl + TM_O2 + 16 * b, r2);
                    umma::wait_ld();
                    if (b == 3) {
                        umma::fence_before_sync();
                        warp_arrive(&b_oread[c & 1], lane);
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float2 o = fma2(make_float2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), down,
                                              make_float2(__uint_as_float(r2[2 * e]), __uint_as_float(r2[2 * e + 1])));
                        w[e] = pack_bf16(o.x, o.y);
                    }
                    stage_rows(buf, 16 * b, v, w);
                }
                if (!turn_over()) break;
                const int rows = min(BT, len - c * BT);
                if (rows == BT) {
                    if (tid == 0) {
                        tma_store_rows(&map_o, smem_u32(buf), h, bos + c * BT);
                        bulk_commit();
                    }
                } else {
                    for (int row = tid >> 4; row < rows; row += 8)
                        *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(p.o) + ((size_t)(bos + c * BT + row) * p.H + h) * (DV * 2) + (tid & 15) * 16) =
                            *reinterpret_cast<const uint4*>(buf + row * 256 + (tid & 15) * 16);
                }
            }
        }
        if (tid == 0) bulk_wait_all();
    }
    __syncthreads();
    if (warp == SC_MMA_WARP) umma::tmem_dealloc(tmem, 512);
}

}  // namespace kda

extern "C" int kda_fwd_scan_smem_bytes() { return kda::SC_SMEM; }

namespace {
int launch_scan(const kda::ScanParams* p, int groups, cudaStream_t stream) {
    using namespace kda;
    if (p->N <= 0) return 0;
    static std::atomic<unsigned long long> done;
    cudaError_t e = allow_smem(kda_fwd_scan_kernel, SC_SMEM, done);
    if (e != cudaSuccess) return (int)e;
    CUtensorMap map, map_o = {};
    // the numbers of tiles and tokens are not known here for a packed batch; the kernel's coordinates stay inside the caller's tensors
    if (!make_pack_map(&map, p->tiles, 1ll << 24) || (p->o && !make_rows_map(&map_o, p->o, p->H, 1ll << 30))) return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p->H, p->N, groups);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = SC_SMEM;
    cfg.stream = stream;
    // Programmatic stream serialization: the grid may be scheduled while the previous kernel of the stream (the
    // chunk-parallel stage) is still draining; every thread calls pdl_wait() before it reads anything.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t launch = launched(cudaLaunchKernelEx(&cfg, kda_fwd_scan_kernel, *p, map, map_o));
    return (int)(launch != cudaSuccess ? launch : cudaGetLastError());
}
}  // namespace

extern "C" int kda_launch_fwd_scan(const kda::ScanParams* p, cudaStream_t stream) { return launch_scan(p, 1, stream); }

// Affine shard transitions of every (sequence, head): p->ht receives C, p->m_out receives M; p->o / p->h0 unused.
extern "C" int kda_launch_fwd_transition(const kda::ScanParams* p, cudaStream_t stream) { return launch_scan(p, 2, stream); }
