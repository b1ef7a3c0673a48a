// Chunk-parallel backward, gated part: per (chunk, head), from the scratch record of the dense stage,
//   dA  = dAu + stril(dW X^T),  dL = -stril(A^T dA A^T),  Zw = A^T dW  (gradient w.r.t. X = beta k 2^g)
//   VJPs of the two gated Gram matrices (Aqk and L), chain rule to q-hat, k-hat and the cumulative gate,
//   reverse cumulative sum, gate activation VJP (dg, dA_log, d dt_bias), L2-norm VJP; dq, dk, dg, dbeta to HBM.
//
// Covers the gate-dependent half of chunk_kda_bwd_kernel_wy_dqkg_fused (cula/kda/chunk_bwd.py:145-313),
// chunk_kda_bwd_kernel_intra (cula/kda/chunk_intra.py:367-627), the reverse chunk_local_cumsum and
// kda_gate_bwd (cula/kda/chunk_bwd.py:594-602) and l2norm_bwd (cula/kda/chunk.py:190-192).
//
// All contractions are tcgen05 kind::tf32 products. The Gram-matrix VJPs
//     dq_i += sum_{j<=i} cP_ij k_j 2^(g_i-g_j)        dk+_i += sum_{j<i} cR_ij k_j 2^(g_i-g_j)          (row side)
//     dk-_j += sum_{i>=j} (cP_ij q_i + cR_ij k_i) 2^(g_i-g_j)                                            (column side)
// never form 2^(g_i-g_j) pairwise: with r_I the cumulative gate at the first row of 16-row block I, row i of block I carries
// e_i = 2^(g_i-r_I), column j of block J carries f_j = 2^(r_{J+1}-g_j), and a pair of blocks the per-channel constant
// 2^(r_I-r_{J+1}) (inside a block e and f meet through its inverse). Every factor is either <= 1 or bounded by 2^116 under the
// safe gate, and the large ones only meet zero coefficients.
//
// Everything is held TRANSPOSED: a thread owns one channel (its tensor-memory lane) of the 16 tokens of one block. Cumulative sums
// are then serial in a thread, the block constants are one register, the operands k f, q e, k e go to tensor memory (A operand:
// lane = channel, column = token) without touching shared memory, the 64x64 coefficient matrices are the B operands, and every
// result comes back to the thread that owns its channel and token. The constant of a pair of blocks belongs to the channel, i.e.
// the lane, so it scales the 16 result columns of that pair on the way back.
// k f, q e and k e are held as tf32 high and low parts: every pair (i, j) adds +x to the gate gradient of row i and -x to that of
// row j through two different products, and the reverse cumulative sum relies on those two cancelling to about 2^-22.
//
// Per tile, products on the left, what the 16 warps do meanwhile on the right; 512 columns of tensor memory are used three times over:
//   dA                                 q e, dW^T -> tensor memory
//   Zw, q side of the columns          dA + dAu -> shared memory (the warps of lanes 0-63)
//   T1^T = A dA^T                      Zw and its part of dbeta; T1 -> shared memory
//   dL = -A^T T1                       k f, k e -> tensor memory; the q side read back
//   P part of the rows                 read back; dL -> dbeta, cR = beta dL -> shared memory
//   R part of the rows, k side         read back; then norms, gate VJP and rows out from registers
// The inputs of a tile come by TMA while the tile before is worked on (dAu and M at its own start, into the buffer of the rows to come).
//
// What bounds it: latency. 42.7 k warp instructions a tile take 37 % of the issue slots of 28 k cycles, tensor pipes 9 %, and one CTA of
// 16 warps (all registers, all of shared and tensor memory) walks through eight CTA barriers a tile. Measured at 4 x 8192 x 32 heads:
// 2.38 -> 1.60 ms (5.2 GB in and out, 0.8 ms at the copy peak) against mma.sync products in transposed fragments with 68.6 k warp
// instructions a tile, 2 x 2048 x 32: 317 -> 218 us, one tile 28.7 -> 22.5 us.
#include "kda_common.cuh"
#include "kda_params.h"
#include "scan_common.cuh"
#include "umma.cuh"

// Optional per-phase cycle counters (compile with -DKDA_PHASE_TIMERS): thread 0 (a warp of the dA / T1 / dL chain) of every CTA adds
// the clock64() spent between consecutive marks to a device array that kda_bwd_gated_read_timers() copies out (profiling builds only).
#ifdef KDA_PHASE_TIMERS
__device__ unsigned long long kda_bwd_gated_timers[16];
#define BG_MARK(i)                                                                            \
    do {                                                                                      \
        if (threadIdx.x == 0) {                                                               \
            const long long now_ = clock64();                                                 \
            atomicAdd(&kda_bwd_gated_timers[i], (unsigned long long)(now_ - bg_t0_));         \
            bg_t0_ = now_;                                                                    \
        }                                                                                     \
    } while (0)
#else
#define BG_MARK(i) do {} while (0)
#endif

namespace kda {

constexpr int BG_THREADS = 512;
constexpr int BG_NT = 16;         // tokens per thread: one block. (8 tokens and 1024 threads: 1.8 -> 2.2 ms, 64 registers are too few)
constexpr int BG_ISSUER = 3;      // the warp that issues the MMAs: no part of the dA / T1 / dL chain, few row-side results
// How the gate tensor is laid out: [B,T,H,128] in bf16 or fp32, or one value per (token, head).
enum BgGate : int { BG_BF16 = 0, BG_FP32 = 1, BG_PER_HEAD = 2 };
// shared-memory map (bytes from a 1024-aligned base). Operand matrices are fp32 in boxes of 32 columns, [64 rows][128 B], 16-byte
// groups XOR-swizzled by the row: K-major operands with the 128-byte swizzle. An M = 128 operand of 64 rows runs on into what
// follows: those lanes of the result are never read.
constexpr int BG_RAW = 0;                       // [2 tiles] raw q, k rows, [64][256 B] each; in the end dq, dk in their place, then dAu and M of the next tile
constexpr int BG_G = 65536;                     // raw gate rows (bf16: [2 tiles][64][256 B], fp32: [64][512 B])
constexpr int BG_A = 98304, BG_AT = 114688;     // A, A^T
constexpr int BG_CP = 131072, BG_CPT = 147456;  // dPs, dPs^T
constexpr int BG_DW = 163840;                   // dW [64][128]; later T1^T, and cR^T in its upper half
constexpr int BG_X = 196608;                    // X [64][128]; later dA, and cR in its upper half; in the end exchange between warps
constexpr int BG_T1 = BG_DW, BG_CRT = BG_DW + 16384, BG_DA = BG_X, BG_CR = BG_X + 16384;
// Corners of dPs (rows 0-31, columns 32-63) and of dPs^T (the mirrored one) that are no part of any operand: block edges of the
// cumulative gate, partial sums of dbeta
constexpr int BG_FIRST = BG_CP + 8192;          // [4][128] log2 decay of the first row of each block
constexpr int BG_SUM = BG_CPT + 4096;           // [4][128] sums over the other rows
constexpr int BG_DBZ = BG_CP + 8192 + 2048;     // [4][64] dbeta through Zw
constexpr int BG_DBL = BG_SUM;                  // [4][64] dbeta through dL
constexpr int BG_XCH = BG_X;                    // floats: [4 blocks][128] gate gradients, likewise dKg Kg, [4 quarters][128] norms, [16 warps][32] their totals, 2 x [4][128] bias, A, [4][64] per-head gates
constexpr int BG_MISC = 229376;                 // rstd [2 tiles][q, k][64], beta [64], 11 barriers, TMEM slot, abort flag, its copy, next tile
constexpr int BG_SMEM = BG_MISC + 1024 + 256 + 144 + 1024;
// tensor-memory columns
constexpr uint32_t BT_A0 = 0, BT_A1 = 128;      // A operands of 64 tokens, high then low parts: q e, then k f | dW^T and Zw, then k e
constexpr uint32_t BT_DW = 128, BT_ZW = 192;
constexpr uint32_t BT_D = 256;                  // results per pair of blocks: q side, P part, R part (160 columns each), block 3 of the k side (64)
constexpr uint32_t BT_C = 416;                  // dA, T1^T, dL (64 columns each); blocks 0-2 of the k side (96)

// The sums of the two Gram phases, and dq, dk+, dk- until they leave, are held times 2^-16. The factor of a block with itself,
// 2^(r_I - r_{I+1}), reaches 2^116 under the safe gate (2^126, where it is clamped, beyond it) and meets the row's or column's own
// factor, which takes it back, only after the sum: unscaled, a sum of more than 2^12 would be inf by then, and inf * 0 = NaN where
// that other factor has underflowed. A power of two changes no bit of what stays in range.
constexpr float BG_DOWN = 1.f / 65536.f, BG_UP = 65536.f;

// Round to tf32 (nearest, ties away from zero -- what cvt.rna.tf32.f32 does for finite values) with two integer
// instructions: add half an ulp of the 10-bit mantissa, clear the 13 low bits.
__device__ __forceinline__ float bg_tf32(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}
// byte offset of element (row, col) of an fp32 matrix in boxes of 32 columns
__device__ __forceinline__ uint32_t bg_off(int row, int col) {
    return (uint32_t)((col >> 5) * 8192 + row * 128 + ((((col >> 2) & 7) ^ (row & 7)) << 4) + (col & 3) * 4);
}
// column of the results of block pair (I, J) among the 160 (96 of the first three blocks): row side grouped by J, column side by I
__device__ __forceinline__ constexpr uint32_t bg_row_col(int J) { return J == 0 ? 0 : J == 1 ? 64 : J == 2 ? 112 : 144; }
__device__ __forceinline__ constexpr uint32_t bg_col_col(int I) { return 8 * I * (I + 1); }

__device__ __forceinline__ float bg_get(const float2 (&v)[BG_NT / 2], int t) { return t & 1 ? v[t / 2].y : v[t / 2].x; }
__device__ __forceinline__ void bg_ld(uint32_t taddr, float2 (&v)[BG_NT / 2]) {
    uint32_t r[BG_NT];
    umma::ld_32x32b_x16(taddr, r);
    umma::wait_ld();
#pragma unroll
    for (int t = 0; t < BG_NT / 2; ++t) v[t] = make_float2(__uint_as_float(r[2 * t]), __uint_as_float(r[2 * t + 1]));
}
__device__ __forceinline__ void bg_st(uint32_t taddr, const float2 (&v)[BG_NT / 2]) {
    uint32_t r[BG_NT];
#pragma unroll
    for (int t = 0; t < BG_NT; ++t) r[t] = __float_as_uint(bg_get(v, t));
    umma::st_32x32b_x16(taddr, r);
}
// tf32 parts of a thread's values: high = the value itself (the tensor core reads the upper 19 bits, i.e. truncates), low = what
// that leaves (exact), rounded
__device__ __forceinline__ void bg_store_split(uint32_t taddr, const float2 (&v)[BG_NT / 2]) {
    bg_st(taddr, v);
    float2 lo[BG_NT / 2];
#pragma unroll
    for (int t = 0; t < BG_NT / 2; ++t) {
        const float2 hi = make_float2(__uint_as_float(__float_as_uint(v[t].x) & 0xffffe000u), __uint_as_float(__float_as_uint(v[t].y) & 0xffffe000u));
        const float2 d = fma2(hi, splat2(-1.f), v[t]);
        lo[t] = make_float2(__uint_as_float(__float_as_uint(d.x) + 0x1000u), __uint_as_float(__float_as_uint(d.y) + 0x1000u));
    }
    bg_st(taddr + 64, lo);
}
// Sum 16 values over the 16 lanes of a half warp, halving the number of values with the lanes: the lane's place in its half is then the
// index of the value that is left in v[0].
__device__ __forceinline__ void bg_reduce(float (&v)[16], int lane) {
#pragma unroll
    for (int s = 8; s; s >>= 1) {
        const bool up = lane & s;
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const float send = up ? v[i] : v[i + s], keep = up ? v[i + s] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
}

struct BgMaps {
    CUtensorMap q, k, g, dq, dk, dg;      // token rows, 64 of a head at a time; g, dg: bf16 or fp32 (not for per-head gates)
    CUtensorMap a, m, dw, ps;             // Akk, M [tiles][64][64], dW [tiles][64][128], dPs and dAu [tiles][2 x 64][64]: 32 x 32 of fp32 at a time, 128-byte swizzle
};

// A wait gave up. `leave`: 2 + parity of the tile that the CTA left at its top, 0 if its last one ended. Products and copies in flight
// end before the shared and tensor memory go away (bounded again): those of the last tile worked on, and the inputs that had been asked
// for of the one left at. What the CTA has not computed, or has computed from what had not arrived, must not pass for a gradient, with or
// without a status word: all its tiles get NaN. (All of it in a function of its own, which needs nothing that the tile loop holds, and the
// parameters by address: with the tile and its parity from the loop the stage takes 1626 us at 4 x 8192 x 32, inlined 1669, like this 1598.)
template <int GK>
__device__ __noinline__ void bg_unwind(const BwdGatedParams& p, int num_tiles, uint64_t* bars, int leave) {
    const int tid = threadIdx.x;
    if (tid == 0) {
        const uint32_t last = leave ? (leave & 1u) ^ 1u : ((num_tiles - 1 - blockIdx.x) / gridDim.x) & 1u;
        for (int i = 0; i < 11; ++i) mbar_wait(&bars[i], leave && (i == 8 || i == 10) ? last ^ 1u : last, 1 << 13);
    }
    const float nan = __int_as_float(0x7fffffff);
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        const int c = t / p.H, h = t - c * p.H;
        const ChunkInfo ci = chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T);
        for (int i = tid; i < ci.valid * DK; i += BG_THREADS) {
            const size_t at = ((size_t)(ci.row0 + i / DK) * p.H + h) * DK + i % DK;
            reinterpret_cast<__nv_bfloat16*>(p.dq)[at] = __float2bfloat16_rn(nan);
            reinterpret_cast<__nv_bfloat16*>(p.dk)[at] = __float2bfloat16_rn(nan);
            if (GK == BG_FP32) reinterpret_cast<float*>(p.dg)[at] = nan;
            if (GK == BG_BF16) reinterpret_cast<__nv_bfloat16*>(p.dg)[at] = __float2bfloat16_rn(nan);
        }
        if (tid < ci.valid) {
            const size_t at = (size_t)(ci.row0 + tid) * p.H + h;
            if (p.beta_fp32) reinterpret_cast<float*>(p.dbeta)[at] = nan;
            else reinterpret_cast<__nv_bfloat16*>(p.dbeta)[at] = __float2bfloat16_rn(nan);
            if (GK == BG_PER_HEAD) {
                if (p.g_fp32) reinterpret_cast<float*>(p.dg)[at] = nan;
                else reinterpret_cast<__nv_bfloat16*>(p.dg)[at] = __float2bfloat16_rn(nan);
            }
        }
        if (p.gate_mode != GATE_NONE && tid < DK) {
            if (p.ddt_bias) atomicAdd(&p.ddt_bias[h * DK + tid], nan);
            if (p.dA_log && tid == 0) atomicAdd(&p.dA_log[h], nan);
        }
    }
}

// GIVES_UP: every wait gives up at once, to test what follows
template <int GK, bool GIVES_UP>
__global__ void __launch_bounds__(BG_THREADS, 1) kda_bwd_gated_kernel(const __grid_constant__ BwdGatedParams p, const int num_tiles, const __grid_constant__ BgMaps maps) {
    constexpr int NT = BG_NT, N2 = NT / 2;
    extern __shared__ unsigned char bg_smem_raw[];
    unsigned char* sm = bg_smem_raw + ((1024u - (smem_u32(bg_smem_raw) & 1023u)) & 1023u);
    const uint32_t smb = smem_u32(sm);
    float* sBeta = reinterpret_cast<float*>(sm + BG_MISC + 1024);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + BG_MISC + 1280);        // [0-7] commit groups of the products, [8] token rows, [9] dAu and M, [10] A, dPs, dW
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + BG_MISC + 1376);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sm + BG_MISC + 1380);
    volatile int* sLeave = reinterpret_cast<volatile int*>(sm + BG_MISC + 1384);
    int4* sNext = reinterpret_cast<int4*>(sm + BG_MISC + 1392);               // {first token row, valid rows, head, tile} of the next tile
    float* first = reinterpret_cast<float*>(sm + BG_FIRST);
    float* sums = reinterpret_cast<float*>(sm + BG_SUM);
    float* xch = reinterpret_cast<float*>(sm + BG_XCH);
    constexpr int X_CS = 512, X_NORM = 1024, X_TOT = 1536, X_BIAS = 2048, X_A = 2560, X_DG = 3072;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int qd = warp & 3, blk = warp >> 2, t0 = NT * blk;      // tensor-memory lanes 32 qd .., tokens t0 ..
    const int ch = 32 * qd + lane;
    const bool chain = qd < 2;                        // lanes 0-63: these warps also carry dA, T1, dL (row = ch, columns t0 ..)
    const size_t tok_stride = (size_t)p.H * DK;

    if (tid == 0) {
        for (int i = 0; i < 11; ++i) mbar_init(&bars[i], 1);
        *sAbort = 0;
        fence_mbar_init();
    }
    if (warp == 0) umma::tmem_alloc(tmem_slot, 512);
    auto geometry = [&](int t) {
        const int c = t / p.H;
        const ChunkInfo ci = chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T);
        return make_int4(ci.row0, ci.valid, t - c * p.H, t);
    };
    // launched while the dense stage drains: whoever reads device memory waits for that first. (One wait of everybody up here, or letting the
    // next kernel in with the last tile, moved spills into the tile loop: 1608 -> 1617, 1634 us at 4 x 8192 x 32)
    if (tid == 32) pdl_wait();
    if (tid == 32) *sNext = (int)blockIdx.x < num_tiles ? geometry(blockIdx.x) : make_int4(0, 0, 0, num_tiles);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tl = tmem + ((uint32_t)(32 * qd) << 16);

    uint32_t par = 0;
    // bounded wait; on expiry the CTA leaves at the next tile, in any case before a barrier whose phase did not end is used again
    auto wait_bar = [&](int which) {
        bool ok = !GIVES_UP && mbar_test(&bars[which], par);
        for (int i = 0; !GIVES_UP && !ok && i < (1 << 16) && !*sAbort; ++i) ok = mbar_test(&bars[which], par);
        if (!ok) {
            if (p.status) report_status(p.status, STATUS_WAIT_TIMEOUT);
            *sAbort = 1;
        }
    };
    auto wait_mma = [&](int which) {      // products up to and including commit group `which` of this tile have completed
        wait_bar(which);
        umma::fence_after_sync();
    };
    auto sync_tmem = [&]() {              // CTA barrier that orders tensor-memory and operand accesses on both sides
        umma::fence_before_sync();
        __syncthreads();
        umma::fence_after_sync();
    };
    // token rows of a tile: three boxes, or one bulk copy per row where the chunk is ragged (a box would reach past rows that may not
    // exist); rows past the end re-read the last real row: they are zeroed through their norm, gate and beta factors
    auto load_rows = [&](const int4 nf, uint32_t buf) {
        constexpr uint32_t G_ROW = GK == BG_BF16 ? 256 : GK == BG_FP32 ? 512 : 0;
        const uint32_t qk = BG_RAW + buf * 32768, gb = BG_G + (GK == BG_BF16 ? buf * 16384 : 0);
        if (nf.y == BT) {
            if (tid == 64) {
                mbar_arrive_expect_tx(&bars[8], BT * (512 + G_ROW));
                tma_load_3d(smb + qk, &maps.q, 0, nf.z, nf.x, &bars[8]);
                tma_load_3d(smb + qk + 16384, &maps.k, 0, nf.z, nf.x, &bars[8]);
                if (G_ROW) tma_load_3d(smb + gb, &maps.g, 0, nf.z, nf.x, &bars[8]);
            }
            return;
        }
        if (tid == 64) mbar_arrive_expect_tx(&bars[8], BT * (512 + G_ROW));
        constexpr int PER = 4;                                  // rows per warp
        if (lane < 3 * PER) {
            const int row = PER * warp + lane % PER, which = lane / PER;
            const size_t off = (size_t)(nf.x + min(row, nf.y - 1)) * tok_stride + (size_t)nf.z * DK;
            if (which < 2)
                bulk_g2s(sm + qk + which * 16384 + row * 256, reinterpret_cast<const __nv_bfloat16*>(which ? p.k : p.q) + off, 256, &bars[8]);
            else if (GK == BG_BF16)
                bulk_g2s(sm + gb + row * 256, reinterpret_cast<const __nv_bfloat16*>(p.g) + off, 256, &bars[8]);
            else if (GK == BG_FP32)
                bulk_g2s(sm + gb + row * 512, reinterpret_cast<const float*>(p.g) + off, 512, &bars[8]);
        }
    };

    pdl_wait();
    int4 info = *sNext;
    int tile = info.w;
    // one thread: an fp32 matrix of 64 rows and 32 `boxes` columns into the layout of an operand
    auto load_matrix = [&](const CUtensorMap* map, int t, int first_row, int boxes, int dst, uint64_t* bar) {
        for (int b = 0; b < boxes; ++b)
            for (int r = 0; r < 64; r += 32) tma_load_3d(smb + dst + b * 8192 + r * 128, map, 32 * b, first_row + r, t, bar);
    };
    auto load_operands = [&](int t) {         // one thread: A, dPs (the corner that holds the block edges stays as it is) and dW
        mbar_arrive_expect_tx(&bars[10], 16384 + 12288 + 32768);
        load_matrix(&maps.a, t, 0, 2, BG_A, &bars[10]);
        load_matrix(&maps.ps, t, 0, 1, BG_CP, &bars[10]);
        tma_load_3d(smb + BG_CP + 8192 + 4096, &maps.ps, 32, 32, t, &bars[10]);
        load_matrix(&maps.dw, t, 0, 4, BG_DW, &bars[10]);
    };
    // A and dPs in registers: a warp takes 8 rows x 4 16-byte groups (no bank conflicts in the operand, two-way ones in the transposed one)
    auto coef_row = [](int idx) { return 8 * (idx >> 7) + 4 * ((idx >> 2) & 1) + ((idx >> 3) & 3); };
    auto coef_group = [](int idx) { return 4 * ((idx >> 5) & 3) + (idx & 3); };
    float alpha_log = 0.f, bias_next = 0.f;   // A_log, dt_bias of the next tile's head (this channel)
    uint32_t beta_bits = 0;
    auto fetch_head = [&](const int4 nf) {
        if (tid < 64) {
            const size_t bi = (size_t)(nf.x + min(tid, nf.y - 1)) * p.H + nf.z;
            beta_bits = p.beta_fp32 ? reinterpret_cast<const uint32_t*>(p.beta)[bi] : (uint32_t)reinterpret_cast<const uint16_t*>(p.beta)[bi] << 16;
        }
        if (p.gate_mode != GATE_NONE) {
            alpha_log = p.A_log[nf.z];
            if (p.dt_bias) bias_next = p.dt_bias[nf.z * DK + ch];
        }
    };
    if (tile < num_tiles) {
        load_rows(info, 0);
        if (tid == 64) load_operands(tile);
        fetch_head(info);
    }
    const float gs_inv = p.gscale[1], gs_up = gs_inv * BG_UP;
    // descriptors are made where they are used: hoisted out of the tile loop they would take the registers of everybody
    auto sd = [&](uint32_t offset) {
        uint32_t base = smb;
        asm volatile("" : "+r"(base));
        return sc_sdesc(base + offset, 16, 1024);
    };
    const uint32_t id64 = umma::make_idesc(umma::FMT_TF32, 128, 64, false, false);
#ifdef KDA_PHASE_TIMERS
    long long bg_t0_ = clock64();
#endif
    for (; tile < num_tiles; par ^= 1u) {
    const float* scr = p.scratch + (size_t)tile * (size_t)BWD_SCRATCH_FLOATS;
    const int valid = info.y, h = info.z;
    const unsigned char* rawq = sm + BG_RAW + par * 32768 + t0 * 256 + ch * 2;       // + 256 t; k 16384 further on
    float* rstd = reinterpret_cast<float*>(sm + BG_MISC) + 128 * par;                 // q [64], k [64]
    auto bf16_at = [](const unsigned char* a) { return __uint_as_float((uint32_t)*reinterpret_cast<const unsigned short*>(a) << 16); };
    auto two = [&](const unsigned char* a, int x) { return make_float2(bf16_at(a + 512 * x), bf16_at(a + 512 * x + 256)); };   // tokens 2 x, 2 x + 1
    auto raw2 = [&](const unsigned char* a, int x) {
        return (uint32_t)*reinterpret_cast<const unsigned short*>(a + 512 * x) | (uint32_t)*reinterpret_cast<const unsigned short*>(a + 512 * x + 256) << 16;
    };
    auto four_at = [&](const float* a, int x, float2 (&v)[2]) {                       // tokens 2 x .. 2 x + 3 of a per-token array
        const float4 w = *reinterpret_cast<const float4*>(a + t0 + 2 * x);
        v[0] = make_float2(w.x, w.y);
        v[1] = make_float2(w.z, w.w);
    };

    const float alpha = p.gate_mode != GATE_NONE ? __expf(alpha_log) : 0.f, bias = bias_next;
    wait_bar(8);              // the token rows have landed
    wait_bar(10);             // A, dPs, dW
    if (tid == 0) *sLeave = *sAbort ? 2 | par : 0;
    BG_MARK(0);
    // ---- 1. norms, gates and their sums inside a block, coefficient matrices in both orientations ----
    {
        constexpr int TPR = 8;                              // threads per row
        const int row = tid / TPR, p8 = tid % TPR;
        float s[2] = {1.f, 1.f};
        if (p.use_l2norm) {
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int e = 0; e < 16 / TPR; ++e) {
                    const uint4 v = *reinterpret_cast<const uint4*>(sm + BG_RAW + par * 32768 + which * 16384 + row * 256 + (p8 + TPR * e) * 16);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpack_bf16(w[i]);
                        acc = fma2(f, f, acc);
                    }
                }
                s[which] = acc.x + acc.y;
            }
#pragma unroll
            for (int o = 1; o < TPR; o <<= 1) {
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
                s[1] += __shfl_xor_sync(0xffffffffu, s[1], o);
            }
            s[0] = rsqrtf(s[0] + 1e-6f);
            s[1] = rsqrtf(s[1] + 1e-6f);
        }
        if (p8 < 2) rstd[64 * p8 + row] = row < valid ? (p8 ? s[1] : s[0]) : 0.f;
    }
    float2 e[N2], f[N2];       // first the log2 decays summed over the thread's tokens (without the first row of the block)
    {
        // one branch on the activation, not one per element
        const float c1 = p.gate_mode == GATE_LOWER_BOUND ? p.lower_bound * RCP_LN2 : p.gate_mode == GATE_SOFTPLUS ? -alpha * RCP_LN2 : RCP_LN2;
        if constexpr (GK == BG_PER_HEAD) {      // a lane activates one token's value
            const int tok = t0 + (lane & (NT - 1));
            const size_t gi = (size_t)(info.x + min(tok, valid - 1)) * p.H + h;
            float x = p.g_fp32 ? reinterpret_cast<const float*>(p.g)[gi] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.g)[gi]);
            const float b0 = p.gate_mode != GATE_NONE && p.dt_bias ? p.dt_bias[h * DK] : 0.f;
            if (p.gate_mode == GATE_LOWER_BOUND) x = fast_rcp(1.f + fast_exp2(-alpha * RCP_LN2 * (x + b0)));
            else if (p.gate_mode == GATE_SOFTPLUS) x = softplus2(splat2(x + b0)).x;
            x *= tok < valid ? c1 : 0.f;
#pragma unroll
            for (int t = 0; t < N2; ++t) e[t] = make_float2(__shfl_sync(0xffffffffu, x, 2 * t), __shfl_sync(0xffffffffu, x, 2 * t + 1));
        } else {
#pragma unroll
            for (int x = 0; x < N2; ++x) {
                if constexpr (GK == BG_FP32) {
                    const float* a = reinterpret_cast<const float*>(sm + BG_G) + (t0 + 2 * x) * DK + ch;
                    e[x] = make_float2(a[0], a[DK]);
                } else e[x] = two(sm + BG_G + par * 16384 + t0 * 256 + ch * 2, x);
            }
            if (p.gate_mode == GATE_LOWER_BOUND) {
                const float c0 = -alpha * RCP_LN2, cb = c0 * bias;
#pragma unroll
                for (int x = 0; x < N2; ++x) {
                    const float2 a = fma2(e[x], splat2(c0), splat2(cb)), b = add2(ex2_2(a), splat2(1.f));
                    e[x] = make_float2(fast_rcp(b.x), fast_rcp(b.y));
                }
            } else if (p.gate_mode == GATE_SOFTPLUS) {
#pragma unroll
                for (int x = 0; x < N2; ++x) e[x] = softplus2(add2(e[x], splat2(bias)));
            }
            if (t0 + NT <= valid) {
#pragma unroll
                for (int x = 0; x < N2; ++x) e[x] = mul2(e[x], splat2(c1));
            } else {                            // padding rows contribute 0
#pragma unroll
                for (int x = 0; x < N2; ++x) {
                    e[x].x *= t0 + 2 * x < valid ? c1 : 0.f;
                    e[x].y *= t0 + 2 * x + 1 < valid ? c1 : 0.f;
                }
            }
        }
        first[blk * DK + ch] = e[0].x;
        e[0].x = 0.f;
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (x) e[x].x += e[x - 1].y;
            e[x].y += e[x].x;
        }
        sums[blk * DK + ch] = e[N2 - 1].y;
    }
    // the coefficient matrices, rounded in place and transposed
#pragma unroll
    for (int n = 0; n < 2048 / BG_THREADS; ++n) {
        const int idx = (tid + n * BG_THREADS) & 1023, row = coef_row(idx), c4 = coef_group(idx);
        const bool dps = n >= 1024 / BG_THREADS;
        if (!dps || row >= 32 || c4 < 8) {
            float4* at = reinterpret_cast<float4*>(sm + (dps ? BG_CP : BG_A) + bg_off(row, 4 * c4));
            const float4 u = *at;
            const float v[4] = {bg_tf32(u.x), bg_tf32(u.y), bg_tf32(u.z), bg_tf32(u.w)};
            *at = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float*>(sm + (dps ? BG_CPT : BG_AT) + bg_off(4 * c4 + i, row)) = v[i];
        }
    }
    if (tid < 64) {
        float b = 0.f;
        if (tid < valid) {
            b = __uint_as_float(beta_bits);
            if (p.beta_logit) b = __fdividef(1.f, 1.f + __expf(-b));
        }
        sBeta[tid] = b;
    }
    bulk_wait_read_all();     // the tile before: rows on their way out have been read (by the threads that sent them)
    __syncthreads();          // block edges, norms, beta
    if (*sLeave) break;
    if (tid == 64) {          // dAu and M where they were, until the next tile's rows come
        mbar_arrive_expect_tx(&bars[9], 32768);
        load_matrix(&maps.ps, tile, 64, 2, BG_RAW + (par ^ 1u) * 32768, &bars[9]);
        load_matrix(&maps.m, tile, 0, 2, BG_RAW + (par ^ 1u) * 32768 + 16384, &bars[9]);
    }
    BG_MARK(1);
    // ---- 2. block anchors, the factors e and f; X and dW as operands over the channels, dW^T and q e as operands over the tokens ----
    // r_b: cumulative gate (log2) at the first row of block b, r_4 at the last row of the chunk. Block pairs (I, J) get
    // 2^(r_I - r_{J+1}): inside a block (clamped), 1 next to each other, two apart, three apart; all times BG_DOWN
    float eI, gl, e_last, c_diag, c_two, c_three;
    float2 k[N2], dw[N2];     // k-hat; dW
    {
        float d[4], r[5];     // d_b = r_{b+1} - r_b
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            d[b] = sums[b * DK + ch];
            if (b < 3) d[b] += first[(b + 1) * DK + ch];
        }
        r[0] = first[ch];
#pragma unroll
        for (int b = 0; b < 4; ++b) r[b + 1] = r[b] + d[b];
        const float dl = blk == 0 ? d[0] : blk == 1 ? d[1] : blk == 2 ? d[2] : d[3];
        const float rI = blk == 0 ? r[0] : blk == 1 ? r[1] : blk == 2 ? r[2] : r[3], rN = blk == 0 ? r[1] : blk == 1 ? r[2] : blk == 2 ? r[3] : r[4];
        eI = fast_exp2(rI);
        gl = BG_DOWN * fast_exp2(r[4] - rN);
        e_last = BG_DOWN * fast_exp2(r[4]);
        c_diag = BG_DOWN * fast_exp2(fminf(-dl, 126.f));
        c_two = BG_DOWN * fast_exp2(blk == 0 || blk == 2 ? r[2] - r[1] : r[3] - r[2]);
        c_three = BG_DOWN * fast_exp2(r[3] - r[1]);
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            const float2 G = e[x];
            e[x] = ex2_2(G);
            f[x] = ex2_2(sub2(splat2(dl), G));
        }
        const uint32_t lc = (uint32_t)(qd * 8192 + t0 * 128 + (lane & 3) * 4);
        unsigned char *xs = sm + BG_X + lc, *ws = sm + BG_DW + lc;
        const uint32_t sw = (uint32_t)(lane >> 2) << 4;
        float2 rk[2], be[2];
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (!(x & 1)) {
                four_at(rstd + 64, x, rk);
                four_at(sBeta, x, be);
            }
            k[x] = mul2(two(rawq + 16384, x), rk[x & 1]);
            const float2 X = mul2(mul2(k[x], e[x]), mul2(be[x & 1], splat2(eI)));
            const uint32_t o0 = 256 * x + (sw ^ (((2 * x) & 7) << 4)), o1 = 256 * x + 128 + (sw ^ (((2 * x + 1) & 7) << 4));
            *reinterpret_cast<float*>(xs + o0) = bg_tf32(X.x);
            *reinterpret_cast<float*>(xs + o1) = bg_tf32(X.y);
            float *w0 = reinterpret_cast<float*>(ws + o0), *w1 = reinterpret_cast<float*>(ws + o1);
            dw[x] = make_float2(bg_tf32(*w0), bg_tf32(*w1));
            *w0 = dw[x].x;
            *w1 = dw[x].y;
        }
    }
    fence_proxy_async();
    sync_tmem();
    if (warp == BG_ISSUER) {
        if (umma::elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 16; ++ks) {          // dA[i][j] = sum over the channels of dW X
                const uint32_t o = (ks >> 2) * 8192 + (ks & 3) * 32;
                umma::mma_tf32(tmem + BT_C, sd(BG_DW + o), sd(BG_X + o), id64, ks != 0);
            }
            umma::commit(&bars[0]);
        }
        __syncwarp();
    }
    {
        float2 q[N2], rq[2];
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (!(x & 1)) four_at(rstd, x, rq);
            q[x] = mul2(mul2(two(rawq, x), mul2(rq[x & 1], splat2(p.scale))), e[x]);
        }
        bg_st(tl + BT_DW + t0, dw);
        bg_store_split(tl + BT_A0 + t0, q);
        umma::wait_st();
    }
    sync_tmem();
    BG_MARK(2);
    if (warp == BG_ISSUER) {
        if (umma::elect_one()) {
#pragma unroll
            for (int ks = 7; ks >= 0; --ks)            // Zw^T = dW^T A; A[i][j] = 0 for i < j: tokens i of this step reach columns up to 16 (ks / 2 + 1)
                umma::mma_tf32_ta(tmem + BT_ZW, tmem + BT_DW + 8 * ks, sd(BG_AT + (ks >> 2) * 8192 + (ks & 3) * 32),
                                  umma::make_idesc(umma::FMT_TF32, 128, 16 * (ks / 2 + 1), false, false), ks != 7);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {           // column side, q: block I = ks / 2 against the columns of blocks J <= I
                const uint32_t d = tmem + BT_D + bg_col_col(ks / 2), id = umma::make_idesc(umma::FMT_TF32, 128, 16 * (ks / 2 + 1), false, false);
                const uint64_t b = sd(BG_CPT + (ks >> 2) * 8192 + (ks & 3) * 32);
                umma::mma_tf32_ta(d, tmem + BT_A0 + 64 + 8 * ks, b, id, ks & 1);
                umma::mma_tf32_ta(d, tmem + BT_A0 + 8 * ks, b, id, 1);
            }
            umma::commit(&bars[1]);
        }
        __syncwarp();
    }
    // ---- 3. under these products: dKg; where the next tile lies, and what the dense stage and the forward left for it, towards L2 ----
    float2 col[N2];           // column side: dKg, then the sums over the rows
    auto fetch = [&](float2 (&v)[N2], int from) {
#pragma unroll
        for (int x = 0; x < N2; ++x) v[x] = make_float2(scr[from + (t0 + 2 * x) * DK + ch], scr[from + (t0 + 2 * x + 1) * DK + ch]);
    };
    const int next = tile + gridDim.x;
    if (warp == 2) {          // (not part of the chain)
        if (next < num_tiles) {
            if (lane == 0) {
                bulk_prefetch_l2(p.scratch + (size_t)next * (size_t)BWD_SCRATCH_FLOATS, BWD_SCRATCH_FLOATS * 4);
                bulk_prefetch_l2(p.akk + (size_t)next * 4096, 4096 * 4);
                bulk_prefetch_l2(p.mkk + (size_t)next * 4096, 4096 * 4);
                *sNext = geometry(next);
            }
        } else if (lane == 0) *sNext = make_int4(0, 0, 0, next);
        __syncwarp();
    }
    // ---- 4. dA = dAu + stril(dW X^T) ----
    const unsigned char* late = sm + BG_RAW + (par ^ 1u) * 32768;                     // dAu; M 16384 further on
    auto late4 = [&](int which, int c) { return *reinterpret_cast<const float4*>(late + which * 16384 + bg_off(ch, t0 + 4 * c)); };
    if (chain) {
        float2 a[N2];
        wait_bar(9);
        wait_mma(0);
        bg_ld(tl + BT_C + t0, a);
#pragma unroll
        for (int i = 0; i < NT / 4; ++i) {
            const int c = t0 + 4 * i;
            const float4 u = late4(0, i);
            *reinterpret_cast<float4*>(sm + BG_DA + bg_off(ch, c)) =
                make_float4(c < ch ? bg_tf32(a[2 * i].x + u.x) : 0.f, c + 1 < ch ? bg_tf32(a[2 * i].y + u.y) : 0.f,
                            c + 2 < ch ? bg_tf32(a[2 * i + 1].x + u.z) : 0.f, c + 3 < ch ? bg_tf32(a[2 * i + 1].y + u.w) : 0.f);
        }
        fence_proxy_async();
        umma::fence_before_sync();
        asm volatile("bar.arrive 1, 288;" ::: "memory");
    } else if (warp == BG_ISSUER) {
        asm volatile("bar.sync 1, 288;" ::: "memory");
        umma::fence_after_sync();
        if (umma::elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {       // T1^T = A dA^T
                const uint32_t o = (ks >> 2) * 8192 + (ks & 3) * 32;
                umma::mma_tf32(tmem + BT_C, sd(BG_A + o), sd(BG_DA + o), id64, ks != 0);
            }
            umma::commit(&bars[2]);
        }
        __syncwarp();
    }
    fetch(col, SCR_DKG);
    BG_MARK(3);
    // ---- 5. Zw: its part of dbeta; then it is the initial value of the dk+ sums, which get e_i at the end. dKg likewise for dk- ----
    float2 zw[N2], cs2 = make_float2(0.f, 0.f);   // cs: sum over the tokens of dKg * Kg (times BG_DOWN), the gradient that reaches g_last through kg
    {
        wait_mma(1);
        bg_ld(tl + BT_ZW + t0, zw);
        float s[NT];
        float2 be[2];
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (!(x & 1)) four_at(sBeta, x, be);
            const float2 v = mul2(mul2(zw[x], k[x]), mul2(e[x], splat2(eI)));
            s[2 * x] = v.x;
            s[2 * x + 1] = v.y;
            zw[x] = mul2(zw[x], mul2(be[x & 1], splat2(BG_DOWN * eI)));
        }
        bg_reduce(s, lane);
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 16);
        if (lane < NT) reinterpret_cast<float*>(sm + BG_DBZ)[qd * 64 + t0 + lane] = s[0];
    }
    // ---- 6. (between the halves of 5, so that dL is there when it is asked for) T1^T, rounded; then dL = -A^T T1 ----
    if (chain) {
        wait_mma(2);
        float2 a[N2];
        bg_ld(tl + BT_C + t0, a);
#pragma unroll
        for (int i = 0; i < NT / 4; ++i)
            *reinterpret_cast<float4*>(sm + BG_T1 + bg_off(ch, t0 + 4 * i)) =
                make_float4(bg_tf32(a[2 * i].x), bg_tf32(a[2 * i].y), bg_tf32(a[2 * i + 1].x), bg_tf32(a[2 * i + 1].y));
        fence_proxy_async();
        umma::fence_before_sync();
        asm volatile("bar.arrive 1, 288;" ::: "memory");
    } else if (warp == BG_ISSUER) {
        asm volatile("bar.sync 1, 288;" ::: "memory");
        umma::fence_after_sync();
        if (umma::elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const uint32_t o = (ks >> 2) * 8192 + (ks & 3) * 32;
                umma::mma_tf32(tmem + BT_C, sd(BG_AT + o), sd(BG_T1 + o), id64, ks != 0);
            }
            umma::commit(&bars[4]);
        }
        __syncwarp();
    }
    auto add_pair = [&](float2 (&acc)[N2], uint32_t column, float c) {
        float2 x[N2];
        bg_ld(tl + column, x);
#pragma unroll
        for (int t = 0; t < N2; ++t) acc[t] = fma2(splat2(c), x[t], acc[t]);
    };
    auto factor = [&](int apart) { return apart == 0 ? c_diag : apart == 1 ? BG_DOWN : apart == 2 ? c_two : c_three; };
    auto add_rows = [&](float2 (&acc)[N2]) {         // pairs (blk, J)
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J <= blk) add_pair(acc, BT_D + bg_row_col(J) + t0 - 16 * J, factor(blk - J));
    };
    {
        float2 v[N2];
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            v[x] = mul2(k[x], f[x]);
            col[x] = mul2(col[x], splat2(gl));
            cs2 = fma2(v[x], col[x], cs2);
        }
        bg_store_split(tl + BT_A0 + t0, v);
#pragma unroll
        for (int x = 0; x < N2; ++x) v[x] = mul2(k[x], e[x]);
        bg_store_split(tl + BT_A1 + t0, v);
#pragma unroll
        for (int I = 0; I < 4; ++I)                  // pairs (I, blk)
            if (I >= blk) add_pair(col, BT_D + bg_col_col(I) + t0, factor(I - blk));
        umma::wait_st();
    }
    sync_tmem();
    BG_MARK(4);
    auto issue_rows = [&](uint32_t coef) {           // columns of block J = ks / 2 against the rows of blocks I >= J
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const int J = ks / 2;
            const uint32_t d = tmem + BT_D + bg_row_col(J), id = umma::make_idesc(umma::FMT_TF32, 128, 64 - 16 * J, false, false);
            const uint64_t b = sd(coef + (ks >> 2) * 8192 + (ks & 3) * 32 + J * 2048);
            umma::mma_tf32_ta(d, tmem + BT_A0 + 64 + 8 * ks, b, id, ks & 1);
            umma::mma_tf32_ta(d, tmem + BT_A0 + 8 * ks, b, id, 1);
        }
    };
    if (warp == BG_ISSUER) {
        if (umma::elect_one()) {
            issue_rows(BG_CP);
            umma::commit(&bars[3]);
        }
        __syncwarp();
    }
    BG_MARK(5);
    // ---- 7. the P part of the rows, and dQg ----
    float2 row[N2];
    {
        float2 dqg[N2];
        fetch(dqg, SCR_DQG);
#pragma unroll
        for (int x = 0; x < N2; ++x) row[x] = make_float2(0.f, 0.f);
        wait_mma(3);
        add_rows(row);
#pragma unroll
        for (int x = 0; x < N2; ++x) row[x] = fma2(dqg[x], splat2(BG_DOWN * eI), row[x]);
    }
    BG_MARK(6);
    // ---- 8. dL: its part of dbeta (rowsum(dL * M)), cR = beta_i dL in both orientations ----
    if (chain) {
        const float be = sBeta[ch];
        wait_mma(4);
        float2 a[N2];
        bg_ld(tl + BT_C + t0, a);
        float db = 0.f;
#pragma unroll
        for (int i = 0; i < NT / 4; ++i) {
            const float4 m4 = late4(1, i);
            const float m[4] = {m4.x, m4.y, m4.z, m4.w}, v4[4] = {a[2 * i].x, a[2 * i].y, a[2 * i + 1].x, a[2 * i + 1].y};
            float c[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = t0 + 4 * i + j;
                const float v = t < ch ? -v4[j] : 0.f;
                db = fmaf(v, t < ch ? m[j] : 0.f, db);               // (M is not written above its diagonal blocks)
                c[j] = bg_tf32(be * v);
                *reinterpret_cast<float*>(sm + BG_CRT + bg_off(t, ch)) = c[j];
            }
            *reinterpret_cast<float4*>(sm + BG_CR + bg_off(ch, t0 + 4 * i)) = make_float4(c[0], c[1], c[2], c[3]);
        }
        reinterpret_cast<float*>(sm + BG_DBL)[blk * 64 + ch] = db;
    }
    fence_proxy_async();
    sync_tmem();
    BG_MARK(7);
    auto issue_k = [&](uint32_t d, int I) {          // column side, k: block I against the columns of blocks J <= I
        const uint32_t id = umma::make_idesc(umma::FMT_TF32, 128, 16 * (I + 1), false, false);
#pragma unroll
        for (int ks = 2 * I; ks < 2 * I + 2; ++ks) {
            const uint64_t b = sd(BG_CRT + (ks >> 2) * 8192 + (ks & 3) * 32);
            umma::mma_tf32_ta(d, tmem + BT_A1 + 64 + 8 * ks, b, id, ks & 1);
            umma::mma_tf32_ta(d, tmem + BT_A1 + 8 * ks, b, id, 1);
        }
    };
    if (warp == BG_ISSUER) {
        if (umma::elect_one()) {
            issue_rows(BG_CR);
            umma::commit(&bars[5]);
#pragma unroll
            for (int I = 0; I < 3; ++I) issue_k(tmem + BT_C + bg_col_col(I), I);
            umma::commit(&bars[6]);
        }
        __syncwarp();
    }
    const int4 ninfo = *sNext;
    if (next < num_tiles) load_rows(ninfo, par ^ 1u);
    if (tid < 64) {           // dbeta is complete
        float v = scr[SCR_DBU + tid];
#pragma unroll
        for (int w = 0; w < 4; ++w) v += reinterpret_cast<const float*>(sm + BG_DBL)[w * 64 + tid];
#pragma unroll
        for (int w = 0; w < 4; ++w) v += reinterpret_cast<const float*>(sm + BG_DBZ)[w * 64 + tid];
        if (tid < valid) {
            const size_t bi = (size_t)(info.x + tid) * p.H + h;
            v *= gs_inv;
            if (p.beta_logit) v *= sBeta[tid] * (1.f - sBeta[tid]);       // chain rule through the in-kernel sigmoid
            if (p.beta_fp32) reinterpret_cast<float*>(p.dbeta)[bi] = v;
            else reinterpret_cast<__nv_bfloat16*>(p.dbeta)[bi] = __float2bfloat16_rn(v);
        }
    }
    // ---- 9. the R part of the rows; then block 3 of the k side may take its columns ----
    wait_mma(5);
    add_rows(zw);
    sync_tmem();
    BG_MARK(8);
    if (warp == BG_ISSUER) {
        if (umma::elect_one()) {
            issue_k(tmem + BT_D, 3);
            umma::commit(&bars[7]);
        }
        __syncwarp();
    }
    const float dD = scr[SCR_DD + ch];
    if (next < num_tiles) fetch_head(ninfo);
#pragma unroll
    for (int x = 0; x < N2; ++x) {
        row[x] = mul2(row[x], mul2(e[x], splat2(p.scale)));        // dq
        zw[x] = mul2(zw[x], e[x]);                                  // dk+
    }
    wait_mma(6);
#pragma unroll
    for (int I = 0; I < 3; ++I)
        if (I >= blk) add_pair(col, BT_C + bg_col_col(I) + t0, factor(I - blk));
    wait_mma(7);
    if (tid == 64 && next < num_tiles) load_operands(next);         // no product reads an operand any more
    add_pair(col, BT_D + t0, factor(3 - blk));
    BG_MARK(9);
    // ---- 10. dk, dG; the sums that cross threads: over the channels q . dq and k . dk, over the blocks the gate gradient ----
    uint32_t qraw[N2], kraw[N2];       // the raw rows, two tokens each
    {
        float s[NT];
        float2 tot = make_float2(0.f, 0.f), rq[2], rk[2];
        const bool up = lane & NT;       // this lane bit: k . dk, else q . dq
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (!(x & 1)) {
                four_at(rstd, x, rq);
                four_at(rstd + 64, x, rk);
            }
            qraw[x] = raw2(rawq, x);
            kraw[x] = raw2(rawq + 16384, x);
            const float2 qh = mul2(unpack_bf16(qraw[x]), rq[x & 1]), kh = mul2(unpack_bf16(kraw[x]), rk[x & 1]);
            const float2 dm = mul2(f[x], col[x]), sq = mul2(qh, row[x]);
            col[x] = fma2(kh, fma2(dm, splat2(-1.f), zw[x]), sq);            // dG
            tot = add2(tot, col[x]);
            zw[x] = add2(zw[x], dm);                                         // dk
            const float2 sk = mul2(kh, zw[x]);
            s[2 * x] = (up ? sk.x : sq.x) + __shfl_xor_sync(0xffffffffu, up ? sq.x : sk.x, NT);
            s[2 * x + 1] = (up ? sk.y : sq.y) + __shfl_xor_sync(0xffffffffu, up ? sq.y : sk.y, NT);
        }
        xch[blk * DK + ch] = tot.x + tot.y;
        xch[X_CS + blk * DK + ch] = cs2.x + cs2.y;
        if (p.use_l2norm) {
            bg_reduce(s, lane);
            xch[X_NORM + qd * 128 + (lane / NT) * 64 + t0 + lane % NT] = s[0];
        }
    }
    __syncthreads();
    BG_MARK(10);
    // ---- 11. dq and dk through the norms, as rows on their way out ----
    {
        float* mine = xch + X_TOT + warp * 2 * NT;
        if (p.use_l2norm) {
            const float* x = xch + X_NORM + (lane / NT) * 64 + t0 + lane % NT;
            mine[lane] = -((x[0] + x[128]) + (x[256] + x[384])) * rstd[(lane / NT) * 64 + t0 + lane % NT];     // q-hat (q-hat . dq) = q rstd (q-hat . dq)
            __syncwarp();
        }
        unsigned char* out = const_cast<unsigned char*>(rawq);      // over the raw rows
        if (p.use_l2norm) {
#pragma unroll
            for (int x = 0; x < N2; x += 2) {
                const float4 tq = *reinterpret_cast<const float4*>(mine + 2 * x), tk = *reinterpret_cast<const float4*>(mine + NT + 2 * x);
                row[x] = fma2(unpack_bf16(qraw[x]), make_float2(tq.x, tq.y), row[x]);
                row[x + 1] = fma2(unpack_bf16(qraw[x + 1]), make_float2(tq.z, tq.w), row[x + 1]);
                zw[x] = fma2(unpack_bf16(kraw[x]), make_float2(tk.x, tk.y), zw[x]);
                zw[x + 1] = fma2(unpack_bf16(kraw[x + 1]), make_float2(tk.z, tk.w), zw[x + 1]);
            }
        }
        float2 rq[2], rk[2];
#pragma unroll
        for (int x = 0; x < N2; ++x) {
            if (!(x & 1)) {
                four_at(rstd, x, rq);
                four_at(rstd + 64, x, rk);
            }
            const float2 dq = mul2(row[x], mul2(rq[x & 1], splat2(gs_up))), dk = mul2(zw[x], mul2(rk[x & 1], splat2(gs_up)));
            *reinterpret_cast<__nv_bfloat16*>(out + 512 * x) = __float2bfloat16_rn(dq.x);
            *reinterpret_cast<__nv_bfloat16*>(out + 512 * x + 256) = __float2bfloat16_rn(dq.y);
            *reinterpret_cast<__nv_bfloat16*>(out + 16384 + 512 * x) = __float2bfloat16_rn(dk.x);
            *reinterpret_cast<__nv_bfloat16*>(out + 16384 + 512 * x + 256) = __float2bfloat16_rn(dk.y);
        }
    }
    // ---- 12. reverse cumulative sum of dG, gate VJP ----
    {
        // g_last sits in token 63 (padding rows repeat the last real value): its gradient starts the sum
        float run = e_last * dD;
#pragma unroll
        for (int b = 3; b >= 0; --b) {
            run += xch[X_CS + b * DK + ch];
            if (b > blk) run += xch[b * DK + ch];
        }
        if (p.gate_mode != GATE_NONE) {         // raw gates again: e is free
            if constexpr (GK == BG_PER_HEAD) {
                const size_t gi = (size_t)(info.x + min(t0 + (lane & (NT - 1)), valid - 1)) * p.H + h;
                const float x = p.g_fp32 ? reinterpret_cast<const float*>(p.g)[gi] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.g)[gi]);
#pragma unroll
                for (int t = 0; t < N2; ++t) e[t] = make_float2(__shfl_sync(0xffffffffu, x, 2 * t), __shfl_sync(0xffffffffu, x, 2 * t + 1));
            } else if constexpr (GK == BG_FP32) {
                const float* a = reinterpret_cast<const float*>(p.g) + (size_t)info.x * tok_stride + h * DK + ch;
#pragma unroll
                for (int x = 0; x < N2; ++x)
                    e[x] = make_float2(a[(size_t)min(t0 + 2 * x, valid - 1) * tok_stride], a[(size_t)min(t0 + 2 * x + 1, valid - 1) * tok_stride]);
            } else {
#pragma unroll
                for (int x = 0; x < N2; ++x) e[x] = two(sm + BG_G + par * 16384 + t0 * 256 + ch * 2, x);
            }
#pragma unroll
            for (int x = 0; x < N2; ++x) e[x] = add2(e[x], splat2(bias));
        }
#pragma unroll
        for (int x = N2 - 1; x >= 0; --x) {     // gradient w.r.t. the natural-log decays
            run += col[x].y;
            const float b = run;
            run += col[x].x;
            col[x] = mul2(make_float2(run, b), splat2(gs_up));
        }
        if (t0 + NT > valid) {
#pragma unroll
            for (int x = 0; x < N2; ++x) {
                if (t0 + 2 * x >= valid) col[x].x = 0.f;
                if (t0 + 2 * x + 1 >= valid) col[x].y = 0.f;
            }
        }
        if (p.gate_mode != GATE_NONE) {
            float2 dA = make_float2(0.f, 0.f), sum = dA;
            if (p.gate_mode == GATE_LOWER_BOUND) {
                const float c0 = -alpha * RCP_LN2, c1 = p.lower_bound * alpha;
#pragma unroll
                for (int x = 0; x < N2; ++x) {
                    const float2 a = add2(ex2_2(mul2(e[x], splat2(c0))), splat2(1.f)), sg = make_float2(fast_rcp(a.x), fast_rcp(a.y));
                    col[x] = mul2(mul2(col[x], splat2(c1)), mul2(sg, fma2(sg, splat2(-1.f), splat2(1.f))));
                    dA = fma2(col[x], e[x], dA);
                    sum = add2(sum, col[x]);
                }
            } else {
#pragma unroll
                for (int x = 0; x < N2; ++x) {
                    col[x] = mul2(col[x], splat2(-alpha));
                    dA = fma2(col[x], softplus2(e[x]), dA);
                    const float2 a = add2(ex2_2(mul2(e[x], splat2(-RCP_LN2))), splat2(1.f));
                    col[x] = mul2(col[x], make_float2(fast_rcp(a.x), fast_rcp(a.y)));
                    sum = add2(sum, col[x]);
                }
            }
            xch[X_BIAS + blk * DK + ch] = sum.x + sum.y;
            xch[X_A + blk * DK + ch] = dA.x + dA.y;
        }
        if constexpr (GK == BG_PER_HEAD) {        // the gate is shared by the 128 channels: its gradient is their sum
            float v[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) v[t] = bg_get(col, t);
            bg_reduce(v, lane);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
            if (lane < NT) xch[X_DG + qd * 64 + t0 + lane] = v[0];
        } else if constexpr (GK == BG_FP32) {
            float* dg = reinterpret_cast<float*>(p.dg) + (size_t)(info.x + t0) * tok_stride + h * DK + ch;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t0 + t < valid) *dg = bg_get(col, t);
                dg += tok_stride;
            }
        } else {
            unsigned char* out = sm + BG_G + par * 16384 + t0 * 256 + ch * 2;      // over the raw gates
#pragma unroll
            for (int x = 0; x < N2; ++x) {
                *reinterpret_cast<__nv_bfloat16*>(out + 512 * x) = __float2bfloat16_rn(col[x].x);
                *reinterpret_cast<__nv_bfloat16*>(out + 512 * x + 256) = __float2bfloat16_rn(col[x].y);
            }
        }
    }
    fence_proxy_async();
    __syncthreads();
    // ---- 13. rows out, the sums over the tokens and over the channel quarters ----
    {
        constexpr int PER = 4;
        const int r = PER * warp + lane % PER, which = lane / PER;
        if (valid == BT) {
            if (tid == 64) {
                tma_store_3d(&maps.dq, smb + BG_RAW + par * 32768, 0, h, info.x);
                tma_store_3d(&maps.dk, smb + BG_RAW + par * 32768 + 16384, 0, h, info.x);
                if (GK == BG_BF16) tma_store_3d(&maps.dg, smb + BG_G + par * 16384, 0, h, info.x);
            }
        } else if (which < (GK == BG_BF16 ? 3 : 2) && r < valid) {
            void* dst = which == 0 ? p.dq : which == 1 ? p.dk : p.dg;
            bulk_s2g(reinterpret_cast<__nv_bfloat16*>(dst) + (size_t)(info.x + r) * tok_stride + h * DK,
                     sm + (which < 2 ? BG_RAW + par * 32768 + which * 16384 : BG_G + par * 16384) + r * 256, 256);
        }
        bulk_commit();
        if (GK == BG_PER_HEAD && tid < valid) {
            const float v = (xch[X_DG + tid] + xch[X_DG + 64 + tid]) + (xch[X_DG + 128 + tid] + xch[X_DG + 192 + tid]);
            const size_t gi = (size_t)(info.x + tid) * p.H + h;
            if (p.g_fp32) reinterpret_cast<float*>(p.dg)[gi] = v;
            else reinterpret_cast<__nv_bfloat16*>(p.dg)[gi] = __float2bfloat16_rn(v);
        }
        if (p.gate_mode != GATE_NONE && tid < DK) {
            if (p.ddt_bias) {
                float v = 0.f;
#pragma unroll
                for (int b = 0; b < 4; ++b) v += xch[X_BIAS + b * DK + tid];
                atomicAdd(&p.ddt_bias[h * DK + tid], v);
            }
            if (p.dA_log) {
                float v = 0.f;
#pragma unroll
                for (int b = 0; b < 4; ++b) v += xch[X_A + b * DK + tid];
#pragma unroll
                for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) atomicAdd(&p.dA_log[h], v);
            }
        }
    }
    BG_MARK(11);
    tile = next;
    info = ninfo;
    }  // tile loop: what the next tile writes before its first barrier is read by nobody any more
    bulk_wait_all();
    __syncthreads();
    if (*sAbort) bg_unwind<GK>(p, num_tiles, bars, *sLeave);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

}  // namespace kda

#ifdef KDA_PHASE_TIMERS
extern "C" int kda_bwd_gated_read_timers(unsigned long long* out, int reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, kda_bwd_gated_timers, sizeof(kda_bwd_gated_timers));
    if (e == cudaSuccess && reset) {
        unsigned long long z[16] = {};
        e = cudaMemcpyToSymbol(kda_bwd_gated_timers, z, sizeof(z));
    }
    return (int)e;
}
#endif

// fp32 matrices [tiles][rows][cols], `stride` bytes from one tile to the next, fetched as 32 x 32 with the 128-byte swizzle
static bool make_matrix_map(CUtensorMap* map, const float* base, int cols, int rows, long long stride, int tiles) {
    kda::EncodeTiledFn fn = kda::encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)tiles}, strides[2] = {(cuuint64_t)cols * 4, (cuuint64_t)stride};
    const cuuint32_t box[3] = {32, 32, 1}, elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

extern "C" int kda_launch_bwd_gated(const kda::BwdGatedParams* p, int num_chunks, int gives_up, cudaStream_t stream) {
    using namespace kda;
    static_assert(BG_SMEM <= 227 * 1024, "shared memory budget");
    if (num_chunks <= 0) return 0;
    const int kind = p->g_per_head ? BG_PER_HEAD : p->g_fp32 ? BG_FP32 : BG_BF16;
    void (*const kernels[2][3])(BwdGatedParams, int, BgMaps) = {
        {kda_bwd_gated_kernel<BG_BF16, false>, kda_bwd_gated_kernel<BG_FP32, false>, kda_bwd_gated_kernel<BG_PER_HEAD, false>},
        {kda_bwd_gated_kernel<BG_BF16, true>, kda_bwd_gated_kernel<BG_FP32, true>, kda_bwd_gated_kernel<BG_PER_HEAD, true>}};
    const auto kernel = kernels[gives_up != 0][kind];
    static std::atomic<unsigned long long> done[2][3];
    cudaError_t e = allow_smem(kernel, BG_SMEM, done[gives_up != 0][kind]);
    if (e != cudaSuccess) return (int)e;
    const int sms = sm_count();
    const int tiles = num_chunks * p->H;
    // whole chunks lie inside the tensors. Their length is not known for a packed batch, whose chunks may also be those of some sequences
    // only, anywhere in it; for a fixed-length one num_chunks 64 is an upper bound
    const long long rows = p->cu_seqlens ? 1ll << 30 : (long long)num_chunks * BT;
    BgMaps maps{};
    const bool g_rows = kind != BG_PER_HEAD, g32 = kind == BG_FP32;
    if (!make_rows_map(&maps.q, const_cast<void*>(p->q), p->H, rows) || !make_rows_map(&maps.k, const_cast<void*>(p->k), p->H, rows) ||
        !make_rows_map(&maps.dq, p->dq, p->H, rows) || !make_rows_map(&maps.dk, p->dk, p->H, rows) ||
        (g_rows && (!make_rows_map(&maps.g, const_cast<void*>(p->g), p->H, rows, g32) || !make_rows_map(&maps.dg, p->dg, p->H, rows, g32))))
        return (int)cudaErrorInvalidValue;
    static_assert(SCR_DAU == SCR_DPS + 64 * 64, "one map addresses dPs and dAu as stacked matrices");
    const long long rec = BWD_SCRATCH_FLOATS * sizeof(float);
    if (!make_matrix_map(&maps.a, p->akk, 64, 64, 16384, tiles) || !make_matrix_map(&maps.m, p->mkk, 64, 64, 16384, tiles) ||
        !make_matrix_map(&maps.dw, p->scratch + SCR_DW, 128, 64, rec, tiles) || !make_matrix_map(&maps.ps, p->scratch + SCR_DPS, 64, 128, rec, tiles))
        return (int)cudaErrorInvalidValue;
    return (int)launch_early(kernel, dim3(tiles < sms ? tiles : sms), BG_THREADS, BG_SMEM, stream, *p, tiles, maps);
}
