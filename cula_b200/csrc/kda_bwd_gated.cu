// Chunk-parallel backward, gated part: per (chunk, head), from the scratch record of the dense stage,
//   dA  = dAu + stril(dW X^T),  dL = -stril(A^T dA A^T),  Zw = A^T dW  (gradient w.r.t. X = beta k 2^g)
//   VJPs of the two gated Gram matrices (Aqk and L), chain rule to q-hat, k-hat and the cumulative gate,
//   reverse cumulative sum, gate activation VJP (dg, dA_log, d dt_bias), L2-norm VJP; dq, dk, dg, dbeta to HBM.
//
// Covers the gate-dependent half of chunk_kda_bwd_kernel_wy_dqkg_fused (cula/kda/chunk_bwd.py:145-313),
// chunk_kda_bwd_kernel_intra (cula/kda/chunk_intra.py:367-627), the reverse chunk_local_cumsum and
// kda_gate_bwd (cula/kda/chunk_bwd.py:594-602) and l2norm_bwd (cula/kda/chunk.py:190-192).
//
// All contractions run as TF32 mma.sync (m16n8k8). The Gram-matrix VJPs
//     dq_i += sum_{j<=i} cP_ij k_j 2^(g_i-g_j)        dk+_i += sum_{j<i} cR_ij k_j 2^(g_i-g_j)          (row side)
//     dk-_j += sum_{i>=j} (cP_ij q_i + cR_ij k_i) 2^(g_i-g_j)                                            (column side)
// never form 2^(g_i-g_j) pairwise: with r_I the cumulative gate at the first row of 16-row block I, row i of block I carries
// 2^(g_i-r_I), column j of block J carries 2^(r_{J+1}-g_j), and a pair of blocks the per-channel constant 2^(r_I-r_{J+1})
// (inside a block the first two are merged). Every factor is either <= 1 or bounded by 2^116 under the safe gate, and the
// large ones only meet zero coefficients.
//
// The operands are made where they are used: a warp owns 16 channels of all 64 tokens in TRANSPOSED fragments (row = channel,
// column = token), in which the accumulator layout of m16n8k8 is also its A layout if the contraction index is taken in the
// order 0 2 4 6 1 3 5 7 of every eight tokens. So gates, q, k and the gradients live in registers under one layout, products
// chain without shared memory, the cumulative sums run over the four lanes of a quad, and the 64x64 coefficient matrices (in
// shared memory with their columns in that order, once per orientation) are read as B fragments by ldmatrix.
// The 16 warps are two groups over the same channels: the row group (Zw, row side, dq, dk) and the column group (dL, column
// side, dg) work at the same time and meet at four CTA barriers; each warp only ever waits for its own group in between.
//
// What bounds it: the legacy TF32 pipe is busy for about 10 k of a tile's 44 k cycles, all of them in the two Gram phases (14 to
// 16 k); the rest is a chain of short dependent phases with 16 warps per SM (41 % of the issue slots) and the 245 KB of the next
// tile. Measured at 4 x 8192 x 32 heads: 3.48 -> 2.30 ms against one group with token rows in shared memory.
#include "kda_common.cuh"
#include "kda_params.h"

// Optional per-phase cycle counters (compile with -DKDA_PHASE_TIMERS): the first thread of each group of every CTA adds the
// clock64() spent between consecutive marks to a device array that kda_bwd_gated_read_timers() copies out (profiling builds
// only): slots 0-7 row group, 8-15 column group.
#ifdef KDA_PHASE_TIMERS
__device__ unsigned long long kda_bwd_gated_timers[16];
#define BG_MARK(i)                                                                            \
    do {                                                                                      \
        if ((threadIdx.x & 255) == 0) {                                                       \
            const long long now_ = clock64();                                                 \
            atomicAdd(&kda_bwd_gated_timers[(i) + 8 * (threadIdx.x >> 8)], (unsigned long long)(now_ - bg_t0_)); \
            bg_t0_ = now_;                                                                    \
        }                                                                                     \
    } while (0)
#else
#define BG_MARK(i) do {} while (0)
#endif

namespace kda {

constexpr int BG_THREADS = 512;
// How the gate tensor is laid out: [B,T,H,128] in bf16 or fp32, or one value per (token, head).
enum BgGate : int { BG_BF16 = 0, BG_FP32 = 1, BG_PER_HEAD = 2 };
// shared-memory map (bytes). bf16 [64 tokens][128] arrays: 256-byte rows, 16-byte groups XOR-swizzled by the row; fp32 arrays:
// boxes of 32 columns, [64 rows][128 B], swizzled the same way: every access below that is not said to conflict does not
constexpr int BG_Q = 0, BG_K = 16384;           // raw q, k rows
constexpr int BG_G = 32768;                     // raw gate rows (bf16: 16 KB, fp32: 32 KB); later the cumulative gates (slots like dq)
constexpr int BG_DW = 65536;                    // dW [64][128]; later the row group's dq, a float4 per thread and 8 tokens
constexpr int BG_X = 98304;                     // X [64][128]; later cR^T (lower half) and ...
constexpr int BG_X2 = BG_X + 16384;             // ... partial sums, then the second half of Zw / dk+ (slots like dq)
constexpr int BG_AN = 131072, BG_AT = 147456;   // A, A^T [64][64]; later the column group's dk- (slots like dq)
constexpr int BG_PN = 163840, BG_PT = 180224;   // dPs, dPs^T; later dq and dk rows on their way out
constexpr int BG_R = BG_PN + 8192;              // [5][128] cumulative gate at the first row of each block, and at the last row:
                                                // in the part of dPs above the diagonal that nothing reads
constexpr int BG_C1 = 196608;                   // T1^T; later the first half of Zw / dk+
constexpr int BG_C2 = 212992;                   // dA, then cR; later partial sums
constexpr int BG_MISC = 229376;                 // rstd_q[64], rstd_k[64], beta[64]
constexpr int BG_SMEM = BG_MISC + 1024;

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
__device__ __forceinline__ void bg_mma(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                   "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
// the same with a zero accumulator input
__device__ __forceinline__ void bg_mma0(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                   "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)), "f"(0.f));
}
__device__ __forceinline__ void bg_cp16(uint32_t smem_dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_dst), "l"(src) : "memory");
}
__device__ __forceinline__ void bg_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void bg_bar(int id) { asm volatile("bar.sync %0, 256;" :: "r"(id) : "memory"); }

// byte offset of element (row, col) of an fp32 matrix in boxes of 32 columns
__device__ __forceinline__ uint32_t bg_off(int row, int col) {
    return (uint32_t)((col >> 5) * 8192 + row * 128 + ((((col >> 2) & 7) ^ (row & 7)) << 4) + (col & 3) * 4);
}
// position of token column c inside a coefficient matrix: 0 2 4 6 1 3 5 7 of every eight
__device__ __forceinline__ int bg_pos(int c) { return (c & ~7) | ((c & 7) >> 1) | ((c & 1) << 2); }

// Sum N values over the eight lanes that share a quad position, halving the number of values with the lanes: N + N/2 + N/4
// shuffles instead of 3 N. Lane (g, t) ends with the sums of values i * 8 + bg_owner(g), i < N / 8, in v[0 .. N/8).
template <int N>
__device__ __forceinline__ void bg_reduce8(float (&v)[N], int g) {
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const int half = N >> (s + 1), bit = 4 >> s;
        const bool up = g & bit;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit * 4);
        }
    }
}

template <int GK>
struct BgLoads {              // copies of one tile's inputs, spread over the CTA
    const BwdGatedParams& p;
    uint32_t smu;
    int tid;
    // rows past the end re-read the last real row; they are zeroed through their norm, gate and beta factors
    __device__ __forceinline__ void qk(const ChunkInfo& ci, int h, int lane256) const {
        const size_t stride = (size_t)p.H * DK, base = (size_t)ci.row0 * stride + (size_t)h * DK;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int idx = lane256 + 256 * n, row = idx >> 4, ch = idx & 15;
            const size_t off = base + (size_t)min(row, ci.valid - 1) * stride + 8 * ch;
            const uint32_t d = (uint32_t)(row * 256 + ((ch ^ (row & 7)) << 4));
            bg_cp16(smu + BG_Q + d, reinterpret_cast<const __nv_bfloat16*>(p.q) + off);
            bg_cp16(smu + BG_K + d, reinterpret_cast<const __nv_bfloat16*>(p.k) + off);
        }
    }
    __device__ __forceinline__ void g(const ChunkInfo& ci, int h, int lane256) const {
        if (GK == BG_PER_HEAD) return;
        const size_t stride = (size_t)p.H * DK, base = (size_t)ci.row0 * stride + (size_t)h * DK;
        if (GK == BG_FP32) {
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int idx = lane256 + 256 * n, row = idx >> 5, c4 = (idx & 31) * 4;
                bg_cp16(smu + BG_G + bg_off(row, c4), reinterpret_cast<const float*>(p.g) + base + (size_t)min(row, ci.valid - 1) * stride + c4);
            }
        } else {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int idx = lane256 + 256 * n, row = idx >> 4, ch = idx & 15;
                bg_cp16(smu + BG_G + (uint32_t)(row * 256 + ((ch ^ (row & 7)) << 4)),
                        reinterpret_cast<const __nv_bfloat16*>(p.g) + base + (size_t)min(row, ci.valid - 1) * stride + 8 * ch);
            }
        }
    }
    __device__ __forceinline__ void dw(int tile, int lane256) const {
        const float* src = p.scratch + (size_t)tile * BWD_SCRATCH_FLOATS + SCR_DW;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int idx = lane256 + 256 * n, row = idx >> 5, c4 = (idx & 31) * 4;
            bg_cp16(smu + BG_DW + bg_off(row, c4), src + row * DK + c4);
        }
    }
};

template <int GK>
__global__ void __launch_bounds__(BG_THREADS, 1) kda_bwd_gated_kernel(const BwdGatedParams p, const int num_tiles) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t smu = smem_u32(sm);
    float* rstd_q = reinterpret_cast<float*>(sm + BG_MISC);
    float* rstd_k = rstd_q + 64;
    float* sBeta = rstd_q + 128;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool col_group = warp >= 8;
    const int gt = tid & 255, cw = warp & 7;          // thread of the group, 16-channel slice
    const int g8 = lane >> 2, t4 = lane & 3, lr = lane & 7, lm = lane >> 3;
    const int ch0 = 16 * cw + g8;                     // this thread's channels: ch0, ch0 + 8
    // register matrices [8][4]: entry n holds tokens a = 8 n + 2 t4, b = a + 1 as {(ch0, a), (ch0, b), (ch0 + 8, a), (ch0 + 8, b)}
    const BgLoads<GK> loads{p, smu, tid};

    // ldmatrix of coefficient / operand matrices. A: 16 rows x 8 columns; B: two 8-row n-tiles x 8 columns
    auto ldsm_a = [&](int base, int row0, int ks, float (&f)[4]) {
        const int row = row0 + lr + 8 * (lm & 1), ch = 2 * ks + (lm >> 1);
        ldsm_x4(smu + base + (ch >> 3) * 8192 + row * 128 + (((ch & 7) ^ (row & 7)) << 4), reinterpret_cast<uint32_t&>(f[0]),
                reinterpret_cast<uint32_t&>(f[1]), reinterpret_cast<uint32_t&>(f[2]), reinterpret_cast<uint32_t&>(f[3]));
    };
    auto ldsm_b = [&](int base, int row0, int ks, float (&f)[4]) {      // f[0..1]: rows row0.., f[2..3]: rows row0 + 8..
        const int row = row0 + lr + 8 * (lm >> 1), ch = 2 * ks + (lm & 1);
        ldsm_x4(smu + base + (ch >> 3) * 8192 + row * 128 + (((ch & 7) ^ (row & 7)) << 4), reinterpret_cast<uint32_t&>(f[0]),
                reinterpret_cast<uint32_t&>(f[1]), reinterpret_cast<uint32_t&>(f[2]), reinterpret_cast<uint32_t&>(f[3]));
    };
    // the same B fragments by address: lane part, 16-row block and 8-column group (the XOR with the group touches two bits only)
    const uint32_t lane_b = (uint32_t)((lr + 8 * (lm >> 1)) * 128 + (((lm & 1) ^ lr) << 4));
    auto ldsm_blk = [&](int base, int blk, int n, float (&f)[4]) {
        ldsm_x4(smu + base + blk * 2048 + (n >> 2) * 8192 + (lane_b ^ (uint32_t)((n & 3) << 5)), reinterpret_cast<uint32_t&>(f[0]),
                reinterpret_cast<uint32_t&>(f[1]), reinterpret_cast<uint32_t&>(f[2]), reinterpret_cast<uint32_t&>(f[3]));
    };
    // 16 tokens (block b) of a bf16 array: r[h][x] = the pair of tokens a, b of 8-token group 2 b + h, channel ch0 + 8 x
    const uint32_t raw_row = (uint32_t)(8 * (lm >> 1) + lr);
    auto load_raw = [&](int base, int b, uint32_t (&r)[2][2]) {
        const uint32_t row = 16 * b + raw_row;
        ldsm_x4_t(smu + base + row * 256 + ((((uint32_t)(2 * cw + (lm & 1))) ^ (row & 7)) << 4), r[0][0], r[0][1], r[1][0], r[1][1]);
    };

    float* rt = reinterpret_cast<float*>(sm + BG_R);
    float* pZ = reinterpret_cast<float*>(sm + BG_X2);            // [8 slices][64] partial sums over channels
    float* pL = reinterpret_cast<float*>(sm + BG_X2 + 2048);     // [2 column halves][64]
    auto slot = [&](int base_lo, int base_hi, int n) -> float4* {     // one float4 per thread of a group and 8 tokens
        return reinterpret_cast<float4*>(sm + (n < 4 ? base_lo : base_hi) + ((n & 3) * 256 + gt) * 16);
    };
    // split an A fragment {(ch0, a), (ch0, b), (ch0 + 8, a), (ch0 + 8, b)} into tf32 high and low parts, in fragment order. Every
    // pair (i, j) adds +x to the gate gradient of row i and -x to that of row j through two different products; the reverse
    // cumulative sum relies on those two cancelling, so they must agree far better than tf32
    // (the tensor core reads the upper 19 bits: high part = the value, truncated; low part = what that leaves, exact, then rounded)
    auto split = [&](const float (&v)[4], float (&hi)[4], float (&lo)[4]) {
        const float o[4] = {v[0], v[2], v[1], v[3]};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            hi[e] = o[e];
            lo[e] = __uint_as_float(__float_as_uint(o[e] - __uint_as_float(__float_as_uint(o[e]) & 0xffffe000u)) + 0x1000u);
        }
    };
    auto sync_all = [&]() { asm volatile("bar.sync 0, 512;" ::: "memory"); };
    // dA = dAu + stril(dW X^T) -> C2: a 16x16 tile per warp of the CTA, tiles on and below the diagonal
    auto dA_tile = [&](const float* scr) {
        const int mt = warp & 3, nh = warp >> 2;
        if (nh <= mt) {
            const int r0 = 16 * mt + g8;
            float2 u[2][2];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int rr = 0; rr < 2; ++rr)
                    u[nt][rr] = *reinterpret_cast<const float2*>(scr + SCR_DAU + (r0 + 8 * rr) * BT + 16 * nh + 8 * nt + 2 * t4);
            float acc[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll 4
            for (int ks = 0; ks < 16; ++ks) {
                float fa[4], fb[4];
                ldsm_a(BG_DW, 16 * mt, ks, fa);
                ldsm_b(BG_X, 16 * nh, ks, fb);
#pragma unroll
                for (int e = 0; e < 4; ++e) fa[e] = bg_tf32(fa[e]);
                bg_mma(acc[0], fa, fb[0], fb[1]);
                bg_mma(acc[1], fa, fb[2], fb[3]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int rr = 0; rr < 2; ++rr) {
                    const int row = r0 + 8 * rr, col = 16 * nh + 8 * nt + 2 * t4, p0 = bg_pos(col);
                    *reinterpret_cast<float*>(sm + BG_C2 + bg_off(row, p0)) = col < row ? bg_tf32(acc[nt][2 * rr] + u[nt][rr].x) : 0.f;
                    *reinterpret_cast<float*>(sm + BG_C2 + bg_off(row, p0 + 4)) = col + 1 < row ? bg_tf32(acc[nt][2 * rr + 1] + u[nt][rr].y) : 0.f;
                }
        }
    };
#ifdef KDA_PHASE_TIMERS
    long long bg_t0_ = clock64();
#endif
    // The two groups run separate tile loops, so that neither holds the other's registers (one loop with branches spilled 850
    // bytes a thread); the six CTA barriers per tile match up.
    if (!col_group) {
    if ((int)blockIdx.x < num_tiles) {
        const int c = blockIdx.x / p.H, h = blockIdx.x - c * p.H;
        loads.qk(chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T), h, gt);
    }
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    const int c = tile / p.H, h = tile - c * p.H;
    const ChunkInfo ci = chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T);
    const size_t tok_stride = (size_t)p.H * DK;
    const size_t base = (size_t)ci.row0 * tok_stride + (size_t)h * DK;
    const float* scr = p.scratch + (size_t)tile * (size_t)BWD_SCRATCH_FLOATS;
    const float gs_inv = p.gscale[1];
    const float alpha = p.gate_mode != GATE_NONE ? __expf(p.A_log[h]) : 0.f;
    float bias[2] = {0.f, 0.f};
    if (p.gate_mode != GATE_NONE && p.dt_bias) {
        bias[0] = p.dt_bias[h * DK + ch0];
        bias[1] = p.dt_bias[h * DK + ch0 + 8];
    }
    uint32_t beta_bits = 0;
    if (tid < 64) {
        const size_t bi = (size_t)(ci.row0 + min(tid, ci.valid - 1)) * p.H + h;
        beta_bits = p.beta_fp32 ? reinterpret_cast<const uint32_t*>(p.beta)[bi] : (uint32_t)reinterpret_cast<const uint16_t*>(p.beta)[bi] << 16;
    }
    bg_cp_wait();
    sync_all();
    BG_MARK(0);       // inputs landed
    if (tid < 64) {
        float b = 0.f;
        if (tid < ci.valid) {
            b = __uint_as_float(beta_bits);
            if (p.beta_logit) b = __fdividef(1.f, 1.f + __expf(-b));
        }
        sBeta[tid] = b;
    }
    // ---- 1. cumulative gate (log2 domain), kept relative to the first row of each 16-row block ----
    float G[8][4], r[2][5];
    auto raw_gates = [&](int n2, float (&v)[2][4]) {      // raw gate values of 8-token groups 2 n2, 2 n2 + 1
        if constexpr (GK == BG_PER_HEAD) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const size_t gi = (size_t)(ci.row0 + min(16 * n2 + 8 * hh + 2 * t4 + e, ci.valid - 1)) * p.H + h;
                    v[hh][e] = v[hh][2 + e] = p.g_fp32 ? reinterpret_cast<const float*>(p.g)[gi] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.g)[gi]);
                }
        } else if constexpr (GK == BG_FP32) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[hh][e] = *reinterpret_cast<const float*>(sm + BG_G + bg_off(16 * n2 + 8 * hh + 2 * t4 + (e & 1), ch0 + 8 * (e >> 1)));
        } else {
            uint32_t w[2][2];
            load_raw(BG_G, n2, w);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 f = unpack_bf16(w[hh][x]);
                    v[hh][2 * x] = f.x;
                    v[hh][2 * x + 1] = f.y;
                }
        }
    };
    {
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) raw_gates(n2, reinterpret_cast<float(&)[2][4]>(G[2 * n2]));
        // one branch on the activation, not one per element: this kernel's code is long and runs once per tile
        const float c1 = p.gate_mode == GATE_LOWER_BOUND ? p.lower_bound * RCP_LN2 : p.gate_mode == GATE_SOFTPLUS ? -alpha * RCP_LN2 : RCP_LN2;
        if (p.gate_mode == GATE_LOWER_BOUND) {
            const float c0 = -alpha * RCP_LN2, cb[2] = {c0 * bias[0], c0 * bias[1]};
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) G[n][i] = fast_rcp(1.f + fast_exp2(fmaf(G[n][i], c0, cb[i >> 1])));
        } else if (p.gate_mode == GATE_SOFTPLUS) {
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 v = softplus2(make_float2(G[n][2 * x] + bias[x], G[n][2 * x + 1] + bias[x]));
                    G[n][2 * x] = v.x;
                    G[n][2 * x + 1] = v.y;
                }
        }
        float run[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int tok = 8 * n + 2 * t4;
            const float ca = tok < ci.valid ? c1 : 0.f, cb = tok + 1 < ci.valid ? c1 : 0.f;      // padding rows contribute 0
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float a = ca * G[n][2 * x], b = cb * G[n][2 * x + 1];
                float inc = a + b, y;
                y = __shfl_up_sync(0xffffffffu, inc, 1, 4); if (t4 >= 1) inc += y;
                y = __shfl_up_sync(0xffffffffu, inc, 2, 4); if (t4 >= 2) inc += y;
                G[n][2 * x + 1] = run[x] + inc;
                G[n][2 * x] = run[x] + (inc - b);
                run[x] += __shfl_sync(0xffffffffu, inc, 3, 4);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
#pragma unroll
            for (int b = 0; b < 4; ++b) r[x][b] = __shfl_sync(0xffffffffu, G[2 * b][2 * x], 0, 4);
            r[x][4] = run[x];
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                G[n][2 * x] -= r[x][n >> 1];
                G[n][2 * x + 1] -= r[x][n >> 1];
            }
        }
    }
    if (t4 == 0) {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int b = 0; b < 5; ++b) rt[b * DK + ch0 + 8 * x] = r[x][b];
    }
    sync_all();       // norms, beta, coefficient matrices, block anchors; the raw gates have been read
    BG_MARK(1);
    // ---- 2. X = beta k-hat 2^G, rounded to tf32; the gates into their slots ----
    {
#pragma unroll
        for (int b2 = 0; b2 < 4; ++b2) {
            uint32_t kr[2][2];
            load_raw(BG_K, b2, kr);
            const float gr[2] = {fast_exp2(r[0][b2]), fast_exp2(r[1][b2])};
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int n = 2 * b2 + hh, tok = 8 * n + 2 * t4;
                *slot(BG_G, BG_G + 16384, n) = make_float4(G[n][0], G[n][1], G[n][2], G[n][3]);
                const float2 rk = *reinterpret_cast<const float2*>(rstd_k + tok), be = *reinterpret_cast<const float2*>(sBeta + tok);
                const float2 f = mul2(rk, be);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 kk = mul2(mul2(unpack_bf16(kr[hh][x]), f), splat2(gr[x]));
                    *reinterpret_cast<float*>(sm + BG_X + bg_off(tok, ch0 + 8 * x)) = bg_tf32(kk.x * fast_exp2(G[n][2 * x]));
                    *reinterpret_cast<float*>(sm + BG_X + bg_off(tok + 1, ch0 + 8 * x)) = bg_tf32(kk.y * fast_exp2(G[n][2 * x + 1]));
                }
            }
        }
    }
    sync_all();
    BG_MARK(2);       // X
    dA_tile(scr);
    sync_all();
    BG_MARK(3);       // dA
    // ---- 4c. Zw = A^T dW (gradient w.r.t. X) in transposed fragments; its part of dbeta; then it becomes the initial value
    //          of the dk+ accumulators, which carry 2^(g_i - r_I) at the end ----
    float zw[8][4];
    {
#pragma unroll
        for (int n = 0; n < 8; ++n) zw[n][0] = zw[n][1] = zw[n][2] = zw[n][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const int tok = 8 * ks + 2 * t4;
            const float fa[4] = {bg_tf32(*reinterpret_cast<const float*>(sm + BG_DW + bg_off(tok, ch0))),
                                 bg_tf32(*reinterpret_cast<const float*>(sm + BG_DW + bg_off(tok, ch0 + 8))),
                                 bg_tf32(*reinterpret_cast<const float*>(sm + BG_DW + bg_off(tok + 1, ch0))),
                                 bg_tf32(*reinterpret_cast<const float*>(sm + BG_DW + bg_off(tok + 1, ch0 + 8)))};
#pragma unroll
            for (int I = 0; I <= ks / 2; ++I) {
                float fb[4];
                ldsm_b(BG_AT, 16 * I, ks, fb);
                bg_mma(zw[2 * I], fa, fb[0], fb[1]);
                bg_mma(zw[2 * I + 1], fa, fb[2], fb[3]);
            }
        }
        float s[16];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            uint32_t kr[2][2];
            load_raw(BG_K, b, kr);
            const float gr[2] = {fast_exp2(r[0][b]), fast_exp2(r[1][b])};
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int n = 2 * b + hh, tok = 8 * n + 2 * t4;
                const float2 rk = *reinterpret_cast<const float2*>(rstd_k + tok), be = *reinterpret_cast<const float2*>(sBeta + tok);
                float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 kk = unpack_bf16(kr[hh][x]);
                    sum.x = fmaf(zw[n][2 * x], kk.x * gr[x] * fast_exp2(G[n][2 * x]), sum.x);
                    sum.y = fmaf(zw[n][2 * x + 1], kk.y * gr[x] * fast_exp2(G[n][2 * x + 1]), sum.y);
                    zw[n][2 * x] *= be.x * (gr[x] * BG_DOWN);
                    zw[n][2 * x + 1] *= be.y * (gr[x] * BG_DOWN);
                }
                s[2 * n] = sum.x * rk.x;
                s[2 * n + 1] = sum.y * rk.y;
            }
        }
        bg_reduce8<16>(s, g8);
        *reinterpret_cast<float2*>(pZ + cw * 64 + 8 * g8 + 2 * t4) = make_float2(s[0], s[1]);
    }
    BG_MARK(4);       // Zw
    sync_all();
    BG_MARK(5);       // wait for the other group
    if (tid < 64) {   // dbeta is complete
        float v = scr[SCR_DBU + tid] + (pL[tid] + pL[64 + tid]);
#pragma unroll
        for (int w = 0; w < 8; ++w) v += pZ[w * 64 + tid];
        if (tid < ci.valid) {
            const size_t bi = (size_t)(ci.row0 + tid) * p.H + h;
            v *= gs_inv;
            if (p.beta_logit) v *= sBeta[tid] * (1.f - sBeta[tid]);       // chain rule through the in-kernel sigmoid
            if (p.beta_fp32) reinterpret_cast<float*>(p.dbeta)[bi] = v;
            else reinterpret_cast<__nv_bfloat16*>(p.dbeta)[bi] = __float2bfloat16_rn(v);
        }
    }
    // The factor 2^(r_I - r_{J+1}) of a pair of blocks belongs to the channel, which is the row of these products: it scales the
    // 16x16 result of the pair, so that the operands of a block are made once and used against every other block.
    {
        // ---- 5a. row side: columns of block J against rows of the blocks I >= J ----
        float accP[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float gr[2] = {BG_DOWN * fast_exp2(rt[(n >> 1) * DK + ch0]), BG_DOWN * fast_exp2(rt[(n >> 1) * DK + ch0 + 8])};
#pragma unroll
            for (int e = 0; e < 4; ++e) accP[n][e] = gr[e >> 1] * scr[SCR_DQG + (8 * n + 2 * t4 + (e & 1)) * DK + ch0 + 8 * (e >> 1)];
        }
#pragma unroll
        for (int J = 0; J < 4; ++J) {
            uint32_t kr[2][2];
            load_raw(BG_K, J, kr);
            const float rN[2] = {rt[(J + 1) * DK + ch0], rt[(J + 1) * DK + ch0 + 8]};
            const float d[2] = {rN[0] - rt[J * DK + ch0], rN[1] - rt[J * DK + ch0 + 8]};
            float hi[2][4], lo[2][4];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const float4 g4 = *slot(BG_G, BG_G + 16384, 2 * J + hh);
                const float2 rk = *reinterpret_cast<const float2*>(rstd_k + 16 * J + 8 * hh + 2 * t4);
                const float2 k0 = mul2(unpack_bf16(kr[hh][0]), rk), k1 = mul2(unpack_bf16(kr[hh][1]), rk);
                const float v[4] = {k0.x * fast_exp2(d[0] - g4.x), k0.y * fast_exp2(d[0] - g4.y), k1.x * fast_exp2(d[1] - g4.z), k1.y * fast_exp2(d[1] - g4.w)};
                split(v, hi[hh], lo[hh]);
            }
#pragma unroll
            for (int I = J; I < 4; ++I) {
                float bP[2][4], bR[2][4], f[4];
                ldsm_blk(BG_PN, I, 2 * J, f);
                bg_mma0(bP[0], lo[0], f[0], f[1]);
                bg_mma0(bP[1], lo[0], f[2], f[3]);
                bg_mma(bP[0], hi[0], f[0], f[1]);
                bg_mma(bP[1], hi[0], f[2], f[3]);
                ldsm_blk(BG_C2, I, 2 * J, f);
                bg_mma0(bR[0], lo[0], f[0], f[1]);
                bg_mma0(bR[1], lo[0], f[2], f[3]);
                bg_mma(bR[0], hi[0], f[0], f[1]);
                bg_mma(bR[1], hi[0], f[2], f[3]);
                ldsm_blk(BG_PN, I, 2 * J + 1, f);
                bg_mma(bP[0], lo[1], f[0], f[1]);
                bg_mma(bP[1], lo[1], f[2], f[3]);
                bg_mma(bP[0], hi[1], f[0], f[1]);
                bg_mma(bP[1], hi[1], f[2], f[3]);
                ldsm_blk(BG_C2, I, 2 * J + 1, f);
                bg_mma(bR[0], lo[1], f[0], f[1]);
                bg_mma(bR[1], lo[1], f[2], f[3]);
                bg_mma(bR[0], hi[1], f[0], f[1]);
                bg_mma(bR[1], hi[1], f[2], f[3]);
                float cji[2] = {BG_DOWN, BG_DOWN};
                if (I != J + 1) {
#pragma unroll
                    for (int x = 0; x < 2; ++x) cji[x] = BG_DOWN * fast_exp2(fminf(rt[I * DK + ch0 + 8 * x] - rN[x], 126.f));
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        accP[2 * I + hh][e] = fmaf(cji[e >> 1], bP[hh][e], accP[2 * I + hh][e]);
                        zw[2 * I + hh][e] = fmaf(cji[e >> 1], bR[hh][e], zw[2 * I + hh][e]);
                    }
            }
        }
        bg_bar(1);         // the partial sums have been read: their space takes a half of the results
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float4 g4 = *slot(BG_G, BG_G + 16384, n);
            const float f[4] = {fast_exp2(g4.x), fast_exp2(g4.y), fast_exp2(g4.z), fast_exp2(g4.w)};
            *slot(BG_DW, BG_DW + 16384, n) = make_float4(p.scale * f[0] * accP[n][0], p.scale * f[1] * accP[n][1], p.scale * f[2] * accP[n][2],
                                                         p.scale * f[3] * accP[n][3]);
            *slot(BG_C1, BG_X2, n) = make_float4(f[0] * zw[n][0], f[1] * zw[n][1], f[2] * zw[n][2], f[3] * zw[n][3]);
        }
    }
    BG_MARK(6);       // row side
    sync_all();       // dk- is ready for the row group, dq and dk+ for the column group
    BG_MARK(7);
    {
        // ---- 6a. dk, the L2-norm VJP, dq and dk out ----
        float* part = reinterpret_cast<float*>(sm + BG_C2);      // [2][8 slices][64], then totals [2][64]
        if (p.use_l2norm) {
#pragma unroll 1
            for (int b = 0; b < 4; ++b) {
                uint32_t qr[2][2], kr[2][2];
                load_raw(BG_Q, b, qr);
                load_raw(BG_K, b, kr);
                float s[8];                  // q . dq of the four tokens, then k . dk
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int n = 2 * b + hh;
                    const float4 dq = *slot(BG_DW, BG_DW + 16384, n), dp = *slot(BG_C1, BG_X2, n), dm = *slot(BG_AN, BG_AT, n);
                    const float2 q0 = unpack_bf16(qr[hh][0]), q1 = unpack_bf16(qr[hh][1]), k0 = unpack_bf16(kr[hh][0]), k1 = unpack_bf16(kr[hh][1]);
                    s[2 * hh] = dq.x * q0.x + dq.z * q1.x;
                    s[2 * hh + 1] = dq.y * q0.y + dq.w * q1.y;
                    s[4 + 2 * hh] = (dp.x + dm.x) * k0.x + (dp.z + dm.z) * k1.x;
                    s[4 + 2 * hh + 1] = (dp.y + dm.y) * k0.y + (dp.w + dm.w) * k1.y;
                }
                bg_reduce8<8>(s, g8);        // lane (g, t) holds value g
                part[512 * (g8 >> 2) + cw * 64 + 16 * b + 8 * ((g8 >> 1) & 1) + 2 * t4 + (g8 & 1)] = s[0];
            }
            bg_bar(1);
            if (gt < 128) {
                const int which = gt >> 6, row = gt & 63;
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) v += part[512 * which + 64 * w + row];
                const float rs = which ? rstd_k[row] : rstd_q[row];
                part[1024 + gt] = v * rs * rs;                  // q-hat (q-hat . dq) = q rstd^2 (q . dq)
            }
            bg_bar(1);
        }
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
            uint32_t qr[2][2], kr[2][2];
            load_raw(BG_Q, b, qr);
            load_raw(BG_K, b, kr);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int n = 2 * b + hh, tok = 8 * n + 2 * t4;
                const float4 dq = *slot(BG_DW, BG_DW + 16384, n), dp = *slot(BG_C1, BG_X2, n), dm = *slot(BG_AN, BG_AT, n);
                const float2 fq = mul2(*reinterpret_cast<const float2*>(rstd_q + tok), splat2(gs_inv * BG_UP)),
                             fk = mul2(*reinterpret_cast<const float2*>(rstd_k + tok), splat2(gs_inv * BG_UP));
                float2 tq = make_float2(0.f, 0.f), tk = tq;
                if (p.use_l2norm) {
                    tq = *reinterpret_cast<const float2*>(part + 1024 + tok);
                    tk = *reinterpret_cast<const float2*>(part + 1088 + tok);
                }
                const float dqv[4] = {dq.x, dq.y, dq.z, dq.w}, dkv[4] = {dp.x + dm.x, dp.y + dm.y, dp.z + dm.z, dp.w + dm.w};
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 q2 = unpack_bf16(qr[hh][x]), k2 = unpack_bf16(kr[hh][x]);
                    qr[hh][x] = pack_bf16(fq.x * (dqv[2 * x] - q2.x * tq.x), fq.y * (dqv[2 * x + 1] - q2.y * tq.y));
                    kr[hh][x] = pack_bf16(fk.x * (dkv[2 * x] - k2.x * tk.x), fk.y * (dkv[2 * x + 1] - k2.y * tk.y));
                }
            }
            const uint32_t row = 16 * b + raw_row, off = row * 256 + ((((uint32_t)(2 * cw + (lm & 1))) ^ (row & 7)) << 4);
            stsm_x4_t(smu + BG_PN + off, qr[0][0], qr[0][1], qr[1][0], qr[1][1]);
            stsm_x4_t(smu + BG_PT + off, kr[0][0], kr[0][1], kr[1][0], kr[1][1]);
        }
        // both groups are done with the raw q and k rows, this one with its slots: the next tile's rows may come
        asm volatile("bar.sync 3, 512;" ::: "memory");
        if (next < num_tiles) {
            const int cn = next / p.H, hn = next - cn * p.H;
            loads.qk(chunk_info(cn, p.cu_seqlens, p.chunk_indices, p.T), hn, gt);
            loads.dw(next, gt);
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int idx = gt + 256 * n, row = idx >> 4, chn = idx & 15;
            if (row < ci.valid) {
                const size_t off = base + (size_t)row * tok_stride + 8 * chn;
                const uint32_t so = (uint32_t)(row * 256 + ((chn ^ (row & 7)) << 4));
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dq) + off) = *reinterpret_cast<const uint4*>(sm + BG_PN + so);
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dk) + off) = *reinterpret_cast<const uint4*>(sm + BG_PT + so);
            }
        }
    }
    }  // tile loop: the first barrier of the next tile orders the reuse of everything written after the last one
    } else {
    if ((int)blockIdx.x < num_tiles) {
        const int c = blockIdx.x / p.H, h = blockIdx.x - c * p.H;
        loads.g(chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T), h, gt);
        loads.dw(blockIdx.x, gt);
    }
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    const int c = tile / p.H, h = tile - c * p.H;
    const ChunkInfo ci = chunk_info(c, p.cu_seqlens, p.chunk_indices, p.T);
    const size_t tok_stride = (size_t)p.H * DK;
    const size_t base = (size_t)ci.row0 * tok_stride + (size_t)h * DK;
    const float* scr = p.scratch + (size_t)tile * (size_t)BWD_SCRATCH_FLOATS;
    const float gs_up = p.gscale[1] * BG_UP;
    const float alpha = p.gate_mode != GATE_NONE ? __expf(p.A_log[h]) : 0.f;
    float bias[2] = {0.f, 0.f};
    if (p.gate_mode != GATE_NONE && p.dt_bias) {
        bias[0] = p.dt_bias[h * DK + ch0];
        bias[1] = p.dt_bias[h * DK + ch0 + 8];
    }
    // ---- 0. norms and the coefficient matrices A and dPs (a lane per row, so that both orientations are stored without bank
    //         conflicts), while the row group works out the gates ----
    uint32_t graw[8][2];      // bf16 gates: the raw values, for the gate VJP
    {
        float4 cm[2][4];
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int n = 0; n < 4; ++n)
                cm[w][n] = *reinterpret_cast<const float4*>((w ? scr + SCR_DPS : p.akk + (size_t)tile * 4096) + (gt & 63) * 64 + 4 * ((gt >> 6) + 4 * n));
        bg_cp_wait();
        sync_all();
        BG_MARK(0);   // inputs landed
        {   // norms: 4 threads per row, 32 channels each
            const int row = gt >> 2, part = gt & 3;
            float s[2];
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint4 v = *reinterpret_cast<const uint4*>(sm + (which ? BG_K : BG_Q) + row * 256 + (((part + 4 * e) ^ (row & 7)) << 4));
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
            for (int o = 1; o < 4; o <<= 1) {
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
                s[1] += __shfl_xor_sync(0xffffffffu, s[1], o);
            }
            if (part == 0) {
                const bool live = row < ci.valid;
                rstd_q[row] = live ? (p.use_l2norm ? rsqrtf(s[0] + 1e-6f) : 1.f) : 0.f;
                rstd_k[row] = live ? (p.use_l2norm ? rsqrtf(s[1] + 1e-6f) : 1.f) : 0.f;
            }
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            unsigned char* nat = sm + (w ? BG_PN : BG_AN);
            unsigned char* tr = sm + (w ? BG_PT : BG_AT);
            const int row = gt & 63, prow = bg_pos(row);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int c4 = 4 * ((gt >> 6) + 4 * n);
                const float v[4] = {bg_tf32(cm[w][n].x), bg_tf32(cm[w][n].y), bg_tf32(cm[w][n].z), bg_tf32(cm[w][n].w)};
                const int p0 = bg_pos(c4);                 // tokens c4, c4 + 2 sit at p0, p0 + 1 and c4 + 1, c4 + 3 at p0 + 4, p0 + 5
                if (row >= 32 || c4 < 32) {
                    *reinterpret_cast<float2*>(nat + bg_off(row, p0)) = make_float2(v[0], v[2]);
                    *reinterpret_cast<float2*>(nat + bg_off(row, p0 + 4)) = make_float2(v[1], v[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) *reinterpret_cast<float*>(tr + bg_off(c4 + e, prow)) = v[e];
            }
        }
        if (GK == BG_BF16) {
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) load_raw(BG_G, n2, reinterpret_cast<uint32_t(&)[2][2]>(graw[2 * n2]));
        }
    }
    sync_all();
    BG_MARK(1);
    const float glast[2] = {rt[4 * DK + ch0], rt[4 * DK + ch0 + 8]};
    sync_all();
    BG_MARK(2);       // X
    dA_tile(scr);
    sync_all();
    BG_MARK(3);       // dA
    {
        const int rb = cw & 3, half = cw >> 2;
        // ---- 4a. T1^T = A dA^T -> C1 (the tiles on and above the diagonal are all that dL needs) ----
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int cb = 2 * half + t;
            if (cb < rb) continue;
            float acc[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            for (int ks = 0; ks < 2 * rb + 2; ++ks) {
                float fa[4], fb[4];
                ldsm_a(BG_AN, 16 * rb, ks, fa);
                ldsm_b(BG_C2, 16 * cb, ks, fb);
                bg_mma(acc[0], fa, fb[0], fb[1]);
                bg_mma(acc[1], fa, fb[2], fb[3]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int rr = 0; rr < 2; ++rr) {
                    const int row = 16 * rb + g8 + 8 * rr, p0 = bg_pos(16 * cb + 8 * nt + 2 * t4);
                    *reinterpret_cast<float*>(sm + BG_C1 + bg_off(row, p0)) = bg_tf32(acc[nt][2 * rr]);
                    *reinterpret_cast<float*>(sm + BG_C1 + bg_off(row, p0 + 4)) = bg_tf32(acc[nt][2 * rr + 1]);
                }
        }
        bg_bar(2);
        // ---- 4b. dL = -stril(A^T T1); dbeta += rowsum(dL * M); cR = beta_i dL -> C2 and, transposed, the lower half of X ----
        float db[2] = {0.f, 0.f};
        const float* mk = p.mkk + (size_t)tile * 4096;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int nb = 2 * half + t;
            if (nb > rb) continue;
            float2 m[2][2];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int rr = 0; rr < 2; ++rr)
                    m[nt][rr] = *reinterpret_cast<const float2*>(mk + (16 * rb + g8 + 8 * rr) * BT + 16 * nb + 8 * nt + 2 * t4);
            float acc[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            for (int ks = 2 * rb; ks < 8; ++ks) {              // A[m][i] = 0 for m < i
                float fa[4], fb[4];
                ldsm_a(BG_AT, 16 * rb, ks, fa);
                ldsm_b(BG_C1, 16 * nb, ks, fb);
                bg_mma(acc[0], fa, fb[0], fb[1]);
                bg_mma(acc[1], fa, fb[2], fb[3]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int rr = 0; rr < 2; ++rr) {
                    const int row = 16 * rb + g8 + 8 * rr, col = 16 * nb + 8 * nt + 2 * t4, p0 = bg_pos(col), pr = bg_pos(row);
                    const float be = sBeta[row];
                    const float v0 = col < row ? -acc[nt][2 * rr] : 0.f, v1 = col + 1 < row ? -acc[nt][2 * rr + 1] : 0.f;
                    db[rr] += v0 * m[nt][rr].x + v1 * m[nt][rr].y;
                    const float c0 = bg_tf32(be * v0), c1 = bg_tf32(be * v1);
                    *reinterpret_cast<float*>(sm + BG_C2 + bg_off(row, p0)) = c0;
                    *reinterpret_cast<float*>(sm + BG_C2 + bg_off(row, p0 + 4)) = c1;
                    *reinterpret_cast<float*>(sm + BG_X + bg_off(col, pr)) = c0;
                    *reinterpret_cast<float*>(sm + BG_X + bg_off(col + 1, pr)) = c1;
                }
        }
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            db[rr] += __shfl_xor_sync(0xffffffffu, db[rr], 1);
            db[rr] += __shfl_xor_sync(0xffffffffu, db[rr], 2);
            if (t4 == 0) pL[half * 64 + 16 * rb + g8 + 8 * rr] = db[rr];
        }
    }
    BG_MARK(4);       // T1, dL
    sync_all();
    BG_MARK(5);       // wait for the other group
    if (gt == 0 && next < num_tiles) {      // the next tile's contiguous inputs on their way to L2
        bulk_prefetch_l2(p.scratch + (size_t)next * (size_t)BWD_SCRATCH_FLOATS, BWD_SCRATCH_FLOATS * 4);
        bulk_prefetch_l2(p.akk + (size_t)next * 4096, 4096 * 4);
        bulk_prefetch_l2(p.mkk + (size_t)next * 4096, 4096 * 4);
    }
    if (next < num_tiles) {      // and its token rows, a 128-byte line at a time
        const int cn = next / p.H, hn = next - cn * p.H;
        const ChunkInfo cin = chunk_info(cn, p.cu_seqlens, p.chunk_indices, p.T);
        const int row = gt >> 2, part = gt & 3;
        if (row < cin.valid) {
            const size_t o = (size_t)(cin.row0 + row) * tok_stride + (size_t)hn * DK;
            prefetch_l2(reinterpret_cast<const __nv_bfloat16*>(part < 2 ? p.q : p.k) + o + 64 * (part & 1));
            if (GK == BG_FP32) prefetch_l2(reinterpret_cast<const float*>(p.g) + o + 32 * part);
            if (GK == BG_BF16 && part < 2) prefetch_l2(reinterpret_cast<const __nv_bfloat16*>(p.g) + o + 64 * part);
        }
    }
    float cs[2] = {0.f, 0.f};      // sum over the tokens of dKg * Kg (times BG_DOWN), the gradient that reaches g_last through kg
    {
        // ---- 5b. column side: rows of block I against columns of the blocks J <= I ----
        float acc[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = scr[SCR_DKG + (8 * n + 2 * t4 + (e & 1)) * DK + ch0 + 8 * (e >> 1)];
#pragma unroll
        for (int J = 0; J < 4; ++J) {
            uint32_t kr[2][2];
            load_raw(BG_K, J, kr);
            const float rN[2] = {rt[(J + 1) * DK + ch0], rt[(J + 1) * DK + ch0 + 8]};
            const float d[2] = {rN[0] - rt[J * DK + ch0], rN[1] - rt[J * DK + ch0 + 8]};
            const float gl[2] = {BG_DOWN * fast_exp2(glast[0] - rN[0]), BG_DOWN * fast_exp2(glast[1] - rN[1])};
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int n = 2 * J + hh;
                const float4 g4 = *slot(BG_G, BG_G + 16384, n);
                const float2 rk = *reinterpret_cast<const float2*>(rstd_k + 8 * n + 2 * t4);
                const float2 k0 = mul2(unpack_bf16(kr[hh][0]), rk), k1 = mul2(unpack_bf16(kr[hh][1]), rk);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] *= gl[e >> 1];
                cs[0] = fmaf(k0.x * fast_exp2(d[0] - g4.x), acc[n][0], fmaf(k0.y * fast_exp2(d[0] - g4.y), acc[n][1], cs[0]));
                cs[1] = fmaf(k1.x * fast_exp2(d[1] - g4.z), acc[n][2], fmaf(k1.y * fast_exp2(d[1] - g4.w), acc[n][3], cs[1]));
            }
        }
#pragma unroll
        for (int I = 0; I < 4; ++I) {
            uint32_t qr[2][2], kr[2][2];
            load_raw(BG_Q, I, qr);
            load_raw(BG_K, I, kr);
            float qhi[2][4], qlo[2][4], khi[2][4], klo[2][4];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int n = 2 * I + hh, tok = 8 * n + 2 * t4;
                const float4 g4 = *slot(BG_G, BG_G + 16384, n);
                const float2 rq = mul2(*reinterpret_cast<const float2*>(rstd_q + tok), splat2(p.scale)), rk = *reinterpret_cast<const float2*>(rstd_k + tok);
                const float2 e0 = make_float2(fast_exp2(g4.x), fast_exp2(g4.y)), e1 = make_float2(fast_exp2(g4.z), fast_exp2(g4.w));
                const float2 q0 = mul2(mul2(unpack_bf16(qr[hh][0]), rq), e0), q1 = mul2(mul2(unpack_bf16(qr[hh][1]), rq), e1);
                const float2 k0 = mul2(mul2(unpack_bf16(kr[hh][0]), rk), e0), k1 = mul2(mul2(unpack_bf16(kr[hh][1]), rk), e1);
                const float vq[4] = {q0.x, q0.y, q1.x, q1.y}, vk[4] = {k0.x, k0.y, k1.x, k1.y};
                split(vq, qhi[hh], qlo[hh]);
                split(vk, khi[hh], klo[hh]);
            }
#pragma unroll
            for (int J = 0; J <= I; ++J) {
                float bl[2][4], f[4];
                ldsm_blk(BG_PT, J, 2 * I, f);
                bg_mma0(bl[0], qlo[0], f[0], f[1]);
                bg_mma0(bl[1], qlo[0], f[2], f[3]);
                bg_mma(bl[0], qhi[0], f[0], f[1]);
                bg_mma(bl[1], qhi[0], f[2], f[3]);
                ldsm_blk(BG_PT, J, 2 * I + 1, f);
                bg_mma(bl[0], qlo[1], f[0], f[1]);
                bg_mma(bl[1], qlo[1], f[2], f[3]);
                bg_mma(bl[0], qhi[1], f[0], f[1]);
                bg_mma(bl[1], qhi[1], f[2], f[3]);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    ldsm_blk(BG_X, J, 2 * I + hh, f);
                    bg_mma(bl[0], klo[hh], f[0], f[1]);
                    bg_mma(bl[1], klo[hh], f[2], f[3]);
                    bg_mma(bl[0], khi[hh], f[0], f[1]);
                    bg_mma(bl[1], khi[hh], f[2], f[3]);
                }
                float cji[2] = {BG_DOWN, BG_DOWN};
                if (I != J + 1) {
#pragma unroll
                    for (int x = 0; x < 2; ++x)
                        cji[x] = BG_DOWN * fast_exp2(fminf(rt[I * DK + ch0 + 8 * x] - rt[(J + 1) * DK + ch0 + 8 * x], 126.f));
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[2 * J + hh][e] = fmaf(cji[e >> 1], bl[hh][e], acc[2 * J + hh][e]);
            }
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float4 g4 = *slot(BG_G, BG_G + 16384, n);
            const float d[2] = {rt[(n / 2 + 1) * DK + ch0] - rt[(n / 2) * DK + ch0], rt[(n / 2 + 1) * DK + ch0 + 8] - rt[(n / 2) * DK + ch0 + 8]};
            *slot(BG_AN, BG_AT, n) = make_float4(fast_exp2(d[0] - g4.x) * acc[n][0], fast_exp2(d[0] - g4.y) * acc[n][1],
                                                 fast_exp2(d[1] - g4.z) * acc[n][2], fast_exp2(d[1] - g4.w) * acc[n][3]);
        }
    }
    BG_MARK(6);       // column side
    sync_all();
    BG_MARK(7);
    {
        // ---- 6b. dG, its reverse cumulative sum down the tokens, the gate VJP ----
        float run[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {     // g_last sits in token 63 (padding rows repeat the last real value): its gradient starts the sum
            cs[x] += __shfl_xor_sync(0xffffffffu, cs[x], 1);
            cs[x] += __shfl_xor_sync(0xffffffffu, cs[x], 2);
            run[x] = cs[x] + BG_DOWN * fast_exp2(glast[x]) * scr[SCR_DD + ch0 + 8 * x];
        }
        float dA_part = 0.f, colsum[2] = {0.f, 0.f};
        float* hpart = reinterpret_cast<float*>(sm + BG_X);      // per-head gates: [8 slices][64] sums over channels
        bg_bar(2);                          // cR^T is no longer read: its space takes the rows of dg
        const float c0 = -alpha * RCP_LN2;
#pragma unroll 1
        for (int b = 3; b >= 0; --b) {
            uint32_t qr[2][2], kr[2][2], gw[2][2];
            load_raw(BG_Q, b, qr);
            load_raw(BG_K, b, kr);
            if constexpr (GK == BG_BF16) {          // a rolled loop may not index registers
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int hh = i >> 1, x = i & 1;
                    gw[hh][x] = b < 2 ? (b ? graw[2 + hh][x] : graw[hh][x]) : (b == 3 ? graw[6 + hh][x] : graw[4 + hh][x]);
                }
            }
            float D[2][4];
#pragma unroll
            for (int hh = 1; hh >= 0; --hh) {
                const int n = 2 * b + hh, tok = 8 * n + 2 * t4;
                const float4 dq = *slot(BG_DW, BG_DW + 16384, n), dp = *slot(BG_C1, BG_X2, n), dm = *slot(BG_AN, BG_AT, n);
                const float2 rq = *reinterpret_cast<const float2*>(rstd_q + tok), rk = *reinterpret_cast<const float2*>(rstd_k + tok);
                const float dqv[4] = {dq.x, dq.y, dq.z, dq.w}, dkv[4] = {dp.x - dm.x, dp.y - dm.y, dp.z - dm.z, dp.w - dm.w};
                const float sa = tok < ci.valid ? gs_up : 0.f, sb = tok + 1 < ci.valid ? gs_up : 0.f;
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 qh = mul2(unpack_bf16(qr[hh][x]), rq), kh = mul2(unpack_bf16(kr[hh][x]), rk);
                    const float ga = qh.x * dqv[2 * x] + kh.x * dkv[2 * x], gb = qh.y * dqv[2 * x + 1] + kh.y * dkv[2 * x + 1];
                    float inc = ga + gb, y;
                    y = __shfl_down_sync(0xffffffffu, inc, 1, 4); if (t4 < 3) inc += y;
                    y = __shfl_down_sync(0xffffffffu, inc, 2, 4); if (t4 < 2) inc += y;
                    float2 da = make_float2(sa * (run[x] + inc), sb * (run[x] + (inc - ga)));     // gradient w.r.t. the natural-log decays
                    run[x] += __shfl_sync(0xffffffffu, inc, 0, 4);
                    if (p.gate_mode != GATE_NONE) {
                        float2 z;
                        if constexpr (GK == BG_BF16) z = unpack_bf16(gw[hh][x]);
                        else {
                            const int ta = min(tok, ci.valid - 1), tb = min(tok + 1, ci.valid - 1);
                            if constexpr (GK == BG_FP32) {
                                const float* gp = reinterpret_cast<const float*>(p.g) + base + ch0 + 8 * x;
                                z = make_float2(gp[(size_t)ta * tok_stride], gp[(size_t)tb * tok_stride]);
                            } else {
                                const size_t ia = (size_t)(ci.row0 + ta) * p.H + h, ib = (size_t)(ci.row0 + tb) * p.H + h;
                                z = p.g_fp32 ? make_float2(reinterpret_cast<const float*>(p.g)[ia], reinterpret_cast<const float*>(p.g)[ib])
                                             : make_float2(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.g)[ia]),
                                                           __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.g)[ib]));
                            }
                        }
                        z = add2(z, splat2(bias[x]));
                        if (p.gate_mode == GATE_LOWER_BOUND) {
                            const float2 sg = make_float2(fast_rcp(1.f + fast_exp2(c0 * z.x)), fast_rcp(1.f + fast_exp2(c0 * z.y)));
                            da = mul2(mul2(da, splat2(p.lower_bound * alpha)), make_float2(sg.x * (1.f - sg.x), sg.y * (1.f - sg.y)));
                            dA_part = fmaf(da.x, z.x, fmaf(da.y, z.y, dA_part));
                        } else {
                            const float2 sp = softplus2(z);
                            da = mul2(da, splat2(-alpha));
                            dA_part = fmaf(da.x, sp.x, fmaf(da.y, sp.y, dA_part));
                            da = mul2(da, make_float2(fast_rcp(1.f + fast_exp2(-RCP_LN2 * z.x)), fast_rcp(1.f + fast_exp2(-RCP_LN2 * z.y))));
                        }
                        colsum[x] += da.x + da.y;
                    }
                    D[hh][2 * x] = da.x;
                    D[hh][2 * x + 1] = da.y;
                    if constexpr (GK == BG_FP32) {        // whole 32-byte sectors: eight channels of a token per store
                        float* dst = reinterpret_cast<float*>(p.dg) + base + (size_t)tok * tok_stride + ch0 + 8 * x;
                        if (tok < ci.valid) dst[0] = da.x;
                        if (tok + 1 < ci.valid) dst[tok_stride] = da.y;
                    }
                }
            }
            if constexpr (GK == BG_BF16) {
                const uint32_t row = 16 * b + raw_row, off = row * 256 + ((((uint32_t)(2 * cw + (lm & 1))) ^ (row & 7)) << 4);
                stsm_x4_t(smu + BG_X + off, pack_bf16(D[0][0], D[0][1]), pack_bf16(D[0][2], D[0][3]), pack_bf16(D[1][0], D[1][1]),
                          pack_bf16(D[1][2], D[1][3]));
            }
            if constexpr (GK == BG_PER_HEAD) {            // the gate is shared by the 128 channels: its gradient is their sum
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float v = D[hh][e] + D[hh][2 + e];
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        if (g8 == 0) hpart[cw * 64 + 16 * b + 8 * hh + 2 * t4 + e] = v;
                    }
            }
        }
        asm volatile("bar.arrive 3, 512;" ::: "memory");     // done with the raw q and k rows and with the row group's slots
        bg_bar(2);            // rows of dg are staged; the gates are no longer read
        if (next < num_tiles) {
            const int cn = next / p.H, hn = next - cn * p.H;
            loads.g(chunk_info(cn, p.cu_seqlens, p.chunk_indices, p.T), hn, gt);
        }
        if constexpr (GK == BG_PER_HEAD) {
            if (gt < ci.valid) {
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) v += hpart[w * 64 + gt];
                const size_t gi = (size_t)(ci.row0 + gt) * p.H + h;
                if (p.g_fp32) reinterpret_cast<float*>(p.dg)[gi] = v;
                else reinterpret_cast<__nv_bfloat16*>(p.dg)[gi] = __float2bfloat16_rn(v);
            }
        } else if constexpr (GK == BG_BF16) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int idx = gt + 256 * n, row = idx >> 4, chn = idx & 15;
                if (row < ci.valid)
                    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dg) + base + (size_t)row * tok_stride + 8 * chn) =
                        *reinterpret_cast<const uint4*>(sm + BG_X + (uint32_t)(row * 256 + ((chn ^ (row & 7)) << 4)));
            }
        }
        if (p.gate_mode != GATE_NONE) {
            if (p.ddt_bias) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    colsum[x] += __shfl_xor_sync(0xffffffffu, colsum[x], 1);
                    colsum[x] += __shfl_xor_sync(0xffffffffu, colsum[x], 2);
                    if (t4 == 0) atomicAdd(&p.ddt_bias[h * DK + ch0 + 8 * x], colsum[x]);
                }
            }
            if (p.dA_log) {
#pragma unroll
                for (int o = 16; o; o >>= 1) dA_part += __shfl_xor_sync(0xffffffffu, dA_part, o);
                if (lane == 0) atomicAdd(&p.dA_log[h], dA_part);
            }
        }
    }
    }
    }
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

extern "C" int kda_launch_bwd_gated(const kda::BwdGatedParams* p, int num_chunks, cudaStream_t stream) {
    using namespace kda;
    static_assert(BG_SMEM <= 227 * 1024, "shared memory budget");
    if (num_chunks <= 0) return 0;
    const int kind = p->g_per_head ? BG_PER_HEAD : p->g_fp32 ? BG_FP32 : BG_BF16;
    auto kernel = kind == BG_PER_HEAD ? kda_bwd_gated_kernel<BG_PER_HEAD> : kind == BG_FP32 ? kda_bwd_gated_kernel<BG_FP32> : kda_bwd_gated_kernel<BG_BF16>;
    static std::atomic<unsigned long long> done[3];
    cudaError_t e = allow_smem(kernel, BG_SMEM, done[kind]);
    if (e != cudaSuccess) return (int)e;
    const int sms = sm_count();
    const int tiles = num_chunks * p->H;
    kernel<<<tiles < sms ? tiles : sms, BG_THREADS, BG_SMEM, stream>>>(*p, tiles);
    return (int)cudaGetLastError();
}
