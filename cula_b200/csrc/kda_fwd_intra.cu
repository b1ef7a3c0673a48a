// Chunk-parallel forward stage: one CTA per (chunk, head) tile fuses
//   gate activation + per-chunk cumulative sum (log2 domain), q/k L2 normalisation,
//   the gated 64x64 Gram matrices Aqk / L (diagonal 16x16 blocks: tf32 mma.sync on register operands; everything below
//   the diagonal: one M=128 x N=96 x K=128 fp16 tcgen05 chain, accumulators in TMEM),
//   Akk = (I + L)^-1 (blocked 16 -> 32 -> 64 inverse in fp32),
//   [w | u] = Akk diag(beta) [k 2^g | v] (two M=128 x N=128 FP16 tcgen05 chains),
//   kg = k 2^(g_last - g), qg = scale q 2^g,
// and writes the tile pack the state scan consumes (layout in kda_common.cuh).
//
// It replaces, in one launch, what the reference does with l2norm_fwd x2 (cula/kda/chunk.py:58-60),
// kda_gate_chunk_cumsum (cula/kda/chunk_fwd.py:69-78), chunk_kda_fwd_intra_cuda and
// recompute_w_u_cuda (csrc/api/kda_sm100.cu:22-120), so the fp32 gate, q-hat and k-hat never
// travel through HBM.
//
// Exponent handling ("safe gate"): 2^(g_i - g_j) is never formed pairwise. Row i of 16-row block I is scaled by
// eA = 2^(g_i - r_I) (r_I = g at the first row of the block), column j of block J by f = 2^(r_{J+1} - g_j); both are <= 1,
// and a column is carried on to a later anchor r_I, I > J + 1, by a per-channel constant <= 1. So every operand of the
// blocks below the diagonal is at most as large as q-hat / k-hat and fits fp16 (11 significant bits, the same as tf32;
// with normalised rows both sides are scaled by 2^6 so that small factors stay clear of fp16's subnormals).
// Inside a diagonal block the column factor 2^(r_I - g_j) reaches 2^(16*5*log2 e) ~ 2^116, which needs the exponent range
// of tf32: those 16x16 blocks are computed by mma.sync, whose fragments are exactly the registers in which the operand
// generation leaves the values (thread (g, t) of a warp owns two rows and 16 channels, and both the A and the B fragment
// of m16n8k8 want rows by g and contraction columns by t), so they cost no shared-memory traffic at all.
//
// What bounds it: instruction latency of the CUDA-core phases (44 % of the issue slots taken with four warps per scheduler;
// the tensor pipes and HBM are far from busy). Warp w owns 16-row block w & 3 and channel half w >> 2 of all first phases; its
// 16-byte row segments make every global access and every operand store a full vector. Two CTAs are resident per SM, so one
// CTA's operand generation overlaps the other's MMAs, inverse and epilogues.
// Measured at B=2, T=2048, H=32 (2048 tiles, cold L2): 143.6 -> 119 us, 31.7 k -> 24 k warp instructions per tile against the
// version that formed all of the Gram product as tf32 operands in shared memory, two channel halves one after the other; with the
// q and k rows of whole chunks by TMA where their operands will stand, instead of in registers from tile to tile: 119 -> 112 us, 844 ->
// 774 us at 4 x 8192 x 32 (requested right at the start of a tile, where the thread that asks waits for the copies out: 789 us); with the
// Gram epilogue as a loop 109 us, 762 us: a tenth of the stalls are for instructions. Rolling the gates and cumulative sums too: no gain.
#include "kda_common.cuh"
#include "kda_params.h"
#include "scan_common.cuh"
#include "umma.cuh"

// Optional per-phase cycle counters (compile with -DKDA_PHASE_TIMERS): thread 0 of every CTA adds the clock64() spent
// between consecutive marks to a device array that kda_fwd_intra_read_timers() copies out (profiling builds only).
#ifdef KDA_PHASE_TIMERS
__device__ unsigned long long kda_fwd_intra_timers[16];
#define PHASE_MARK(i)                                                                     \
    do {                                                                                  \
        if (tid == 0) {                                                                   \
            const long long now_ = clock64();                                             \
            atomicAdd(&kda_fwd_intra_timers[i], (unsigned long long)(now_ - phase_t0_));  \
            phase_t0_ = now_;                                                             \
        }                                                                                 \
    } while (0)
#else
#define PHASE_MARK(i) do {} while (0)
#endif

namespace kda {

constexpr int INTRA_THREADS = 256;
constexpr int INFO_THREAD = 224;                 // the thread that works out the next tile's geometry
constexpr int MMA_THREAD = 128;                  // the thread that issues the tcgen05 MMAs, waits for them and sends the bulk copies

// How the gate tensor is laid out: [B,T,H,128] in bf16 or fp32, or one value per (token, head).
enum GateKind : int { GK_BF16 = 0, GK_FP32 = 1, GK_PER_HEAD = 2 };

// shared-memory map (bytes from a 1024-aligned base)
constexpr int SM_OPA = 0;                 // A operand [q-hat; k-hat] eA, fp16: [2 k-atoms][128 rows][128 B], SW128
constexpr int SM_OPB = 32768;             // B operand, fp16: k-hat anchored at blocks 1, 2, 3 (16 + 32 + 48 rows): [2 k-atoms][96 rows][128 B]
constexpr int SM_XS = 57344;              // X = k 2^g, fp16 [2 mn-atoms][64 tokens][128 B], SW128 (MN-major B operand)
constexpr int SM_AINV = 73728;            // fp32 [64][68]: L below the diagonal blocks, turned into (I+L)^-1 in place
constexpr int SM_TAB = 91136;             // [8 warps][6][64] fp32: per-channel constants of the warp's (block, channel half)
constexpr int SM_EDGE = 103424;           // [4][128] log2 decay of the first row of each block, [4][128] sum over its other rows
constexpr int SM_NORM = 107520;           // [2 halves][64 rows] float2: sums of squares of q and k
constexpr int SM_MISC = 108544;           // beta[2][64], barriers, TMEM base, abort flag, alpha[2], tile info[2]
constexpr int SM_BIAS = SM_MISC + 1024;   // [2][128] fp32
constexpr int SM_TOTAL = SM_BIAS + 1024;
constexpr int KATOM_A = 16384, KATOM_B = 12288;
// regions reused once their first use is over
constexpr int SM_YS = SM_OPA;             // Y = v, same layout as X (after the Gram MMAs)
constexpr int SM_STG_AQK = SM_OPA + 16384;   // outputs are staged in the exact tile-pack image and leave as bulk copies:
constexpr int SM_STG_U = SM_OPA;             // Aqk [64][128 B]; U0 | U1 [2][64][128 B] over Y, W [64][256 B] over X, both
constexpr int SM_STG_W = SM_XS;              // dead once the W/U MMAs have completed
constexpr int SM_AKK16 = SM_OPB;          // Akk fp16, stacked twice: [128][128 B], SW128 (K-major A operand)
constexpr int SM_TM = SM_OPB + 16384;     // scratch of the last block product, [32][36] fp32
constexpr int SM_LDIAG = SM_TAB;          // the four diagonal blocks of L, [4][16][20] fp32 (the tables are dead by then)
constexpr int LROW = 68;                  // padded fp32 row of the 64x64 matrix
constexpr int LDROW = 20;
constexpr int TROW = 36;
static_assert(SM_TM + 32 * TROW * 4 <= SM_XS, "block-product scratch must fit the B operand region");

__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return umma::make_sdesc(addr, lbo, sbo) | (2ull << 61);
}

// D(16x8) += A(16 x 8) * B(8 x 8) on the hi/lo split of both operands: three TF32 MMAs recover fp32-level accuracy.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = __float_as_uint(x);                                           // the tensor core reads the upper 19 bits only
    lo = __float_as_uint(x - __uint_as_float(hi & 0xffffe000u));       // what it does not see (exact), again truncated by it
}
__device__ __forceinline__ void mma_tf32_16x8x8(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_3xtf32(float (&d)[4], float (&c)[4], const float (&af)[4], const float (&bf)[2]) {
    uint32_t ah[4], al[4], bh[2], bl[2];
#pragma unroll
    for (int e = 0; e < 4; ++e) split_tf32(af[e], ah[e], al[e]);
#pragma unroll
    for (int e = 0; e < 2; ++e) split_tf32(bf[e], bh[e], bl[e]);
    mma_tf32_16x8x8(c, al, bh);
    mma_tf32_16x8x8(d, ah, bh);
    mma_tf32_16x8x8(c, ah, bl);
}
// 16x8 tile of A * B, k-steps [0, KT); A, B fp32 in shared memory, row-major with strides lda / ldb
template <int KT>
__device__ __forceinline__ void mma_tile_3xtf32(const float* A, int lda, const float* B, int ldb, float (&acc)[4], int g, int t) {
    float corr[4] = {0.f, 0.f, 0.f, 0.f};  // the two small products in a chain of their own
#pragma unroll
    for (int ks = 0; ks < KT; ++ks) {      // unrolled: the loads of all k-steps are in flight together (a latency chain otherwise)
        const float af[4] = {A[g * lda + 8 * ks + t], A[(g + 8) * lda + 8 * ks + t], A[g * lda + 8 * ks + t + 4],
                             A[(g + 8) * lda + 8 * ks + t + 4]};
        const float bf[2] = {B[(8 * ks + t) * ldb + g], B[(8 * ks + t + 4) * ldb + g]};
        mma_3xtf32(acc, corr, af, bf);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] += corr[e];
}

// mma.sync reads only the upper 19 bits of a tf32 operand, i.e. it truncates. Instead of rounding every operand of the
// diagonal blocks (one more instruction per element), the mean relative error of truncation, -2^-11 / ln 2 = -3.52e-4 per
// operand for log-uniform mantissas, is taken out by one factor in the per-channel constant of the column operand.
constexpr float TF32_DEBIAS2_LOG2 = 2.f * 5.0775e-4f;     // log2 of (1 + 3.52e-4)^2: both operands

// q, k, v rows [tokens][heads][128], 64 channels x 64 tokens of a head at a time, 128-byte swizzle
struct IntraMaps {
    CUtensorMap q, k, v;
};

template <int GK>
__global__ void __launch_bounds__(INTRA_THREADS, 2) kda_fwd_intra_kernel(const IntraParams p, const __grid_constant__ IntraMaps maps) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sm_u32 = smem_u32(sm);
    float* sBetaBuf = reinterpret_cast<float*>(sm + SM_MISC);            // [2][64]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + SM_MISC + 512);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + SM_MISC + 544);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sm + SM_MISC + 552);
    float* sAlpha = reinterpret_cast<float*>(sm + SM_MISC + 560);        // [2] exp(A_log[h])
    int4* sInfo = reinterpret_cast<int4*>(sm + SM_MISC + 576);           // [2] {first token row, valid rows, head, tile slot}
    float* sBetaMax = reinterpret_cast<float*>(sm + SM_MISC + 608);      // [2][2 warps] largest |beta| of the tile
    float* sBiasBuf = reinterpret_cast<float*>(sm + SM_BIAS);            // [2][128]
    float* sEdgeA = reinterpret_cast<float*>(sm + SM_EDGE);              // [4][128]
    float* sEdgeT = sEdgeA + 4 * DK;                                     // [4][128]
    float2* sNorm = reinterpret_cast<float2*>(sm + SM_NORM);
    float* sAi = reinterpret_cast<float*>(sm + SM_AINV);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t tok_stride = (size_t)p.H * DK;
    // First phases: warp = (16-row block I, 64-channel half hf). Lane (g, t) owns rows 16 I + 2 pr and 16 I + 2 pr + 1 and the
    // channels 64 hf + 32 c + 8 t + e, c = 0, 1, e = 0..7. pr is g with its two low bits swapped and the two four-channel
    // halves of a segment are handled in the order h ^ (t >> 1): together that makes every 8-byte operand store of a half
    // warp hit 32 distinct banks of the swizzled layout.
    const int I = warp & 3, hf = warp >> 2;
    const int g = lane >> 2, t = lane & 3, pr = ((g & 1) << 1) | ((g >> 1) & 1) | (g & 4), sx = t >> 1;
    const int rowA = 16 * I + 2 * pr;

    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init(&bars[2], 1);          // q and k rows
        *sAbort = 0;
        fence_mbar_init();
    }
    if (warp == 0) umma::tmem_alloc(tmem_slot, 256);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    // the state scan that follows in the stream may be scheduled as soon as SMs free up, so that its launch and set-up
    // run under the tail of this kernel; it waits for this whole grid before it reads anything
    pdl_launch_dependents();
#ifdef KDA_PHASE_TIMERS
    long long phase_t0_ = clock64();
#endif

    // One thread waits (bounded) for the tensor-core completion barrier; everybody else parks on the CTA barrier.
    // On a time-out the status word is set and the whole CTA leaves the tile loop together (TMEM is freed below).
    auto wait_mma = [&](int which, uint32_t parity) -> bool {
        if (tid == MMA_THREAD) {
            if (!mbar_spin(&bars[which], parity)) {
                report_status(p.status, STATUS_WAIT_TIMEOUT);
                *sAbort = 1;
            }
            umma::fence_before_sync();
        }
        __syncthreads();
        umma::fence_after_sync();
        return *sAbort == 0;
    };

    // The geometry of a tile (integer divisions, table look-ups for a packed batch) is worked out by ONE thread, one
    // tile ahead, and handed to the others through shared memory.
    auto publish_info = [&](int t_id, int buf) {
        if (tid == INFO_THREAD) {
            int4 v = make_int4(0, 0, 0, 0);
            if (t_id < p.num_tiles) {
                const int c2 = t_id / p.H;
                const ChunkInfo ci2 = chunk_info(c2, p.cu_seqlens, p.chunk_indices, p.T, p.stride);
                v = make_int4(ci2.row0, ci2.valid, t_id - c2 * p.H, t_id);
            }
            sInfo[buf] = v;
        }
    };
    // Register prefetch: the raw gate rows are fetched one tile ahead, at the point of the tile from which their registers are free.
    // Loads are unconditional (nothing may depend on a loaded value before it is used): a padding row reads the last
    // real row of the chunk instead, and is zeroed where it is used (through its gate, norm and beta factors).
    constexpr int NGR = GK == GK_FP32 ? 8 : (GK == GK_BF16 ? 4 : 1);
    uint4 graw[NGR];                              // [row][c] segments of 8 bf16, [row][c][h] of 4 fp32, or the two rows' scalars
    auto fetch_g = [&](const int4 nf) {
        if constexpr (GK == GK_PER_HEAD) {
            const size_t i0 = (size_t)(nf.x + min(rowA, nf.y - 1)) * p.H + nf.z, i1 = (size_t)(nf.x + min(rowA + 1, nf.y - 1)) * p.H + nf.z;
            if (p.g_fp32) {
                graw[0].x = reinterpret_cast<const uint32_t*>(p.g)[i0];
                graw[0].y = reinterpret_cast<const uint32_t*>(p.g)[i1];
            } else {
                graw[0].x = reinterpret_cast<const uint16_t*>(p.g)[i0];
                graw[0].y = reinterpret_cast<const uint16_t*>(p.g)[i1];
            }
        } else {
            const size_t base2 = (size_t)nf.x * tok_stride + (size_t)nf.z * DK + 64 * hf + 8 * t;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const size_t roff = base2 + (size_t)min(rowA + j, nf.y - 1) * tok_stride;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if constexpr (GK == GK_BF16) {
                        graw[2 * j + c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.g) + roff + 32 * c);
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            graw[4 * j + 2 * c + h] = *reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(p.g) + roff + 32 * c + 4 * (h ^ sx));
                    }
                }
            }
        }
    };
    // The q and k rows of a whole chunk come by TMA into the buffer of the A operand, in its layout: each thread finds its values where it
    // will put the operand. Rows of a ragged chunk (a box would reach past them) are loaded one by one; padding rows read the last real
    // row and are zeroed through their norms.
    uint32_t qk_parity = 0;
    auto request_qk = [&](const int4 nf) {        // one thread
        if (nf.y < BT) return;
        mbar_arrive_expect_tx(&bars[2], 32768);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            tma_load_3d(sm_u32 + SM_OPA + half * KATOM_A, &maps.q, 64 * half, nf.z, nf.x, &bars[2]);
            tma_load_3d(sm_u32 + SM_OPA + half * KATOM_A + 8192, &maps.k, 64 * half, nf.z, nf.x, &bars[2]);
        }
    };
    // a tile's token rows towards L2: boxes of a whole chunk, the real rows of a ragged one
    auto prefetch_rows = [&](const int4 nf) {
        if (nf.y < BT) {
            const int row = tid >> 2, part = tid & 3;
            if (row < nf.y) {
                const size_t off = (size_t)(nf.x + row) * tok_stride + (size_t)nf.z * DK + 64 * (part & 1);
                prefetch_l2(reinterpret_cast<const __nv_bfloat16*>(part < 2 ? p.q : p.k) + off);
                if (part < 2) prefetch_l2(reinterpret_cast<const __nv_bfloat16*>(p.v) + off);
            }
        } else if (tid == INFO_THREAD) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                tma_prefetch_3d(&maps.q, 64 * half, nf.z, nf.x);
                tma_prefetch_3d(&maps.k, 64 * half, nf.z, nf.x);
                tma_prefetch_3d(&maps.v, 64 * half, nf.z, nf.x);
            }
        }
    };
    // Per-tile scalars (beta of the 64 rows, dt_bias and exp(A_log) of the head) are fetched one tile ahead by the
    // first 193 threads into a register each and parked in shared memory before the tile ends, so that no phase of
    // the next tile starts with a dependent global load.
    uint32_t sc_next = 0;        // raw bits: nothing may depend on the load before it is parked
    auto load_scalars = [&](const int4 nf) {
        const int h2 = nf.z;
        sc_next = 0;
        if (tid < BT) {
            if (tid < nf.y) {
                const size_t bi = (size_t)(nf.x + tid) * p.H + h2;
                sc_next = p.beta_fp32 ? reinterpret_cast<const uint32_t*>(p.beta)[bi]
                                      : (uint32_t)reinterpret_cast<const uint16_t*>(p.beta)[bi];
            }
        } else if (tid < BT + DK) {
            if (p.gate_mode != GATE_NONE && p.dt_bias) sc_next = __float_as_uint(p.dt_bias[h2 * DK + tid - BT]);
        } else if (tid == BT + DK) {
            if (p.gate_mode != GATE_NONE) sc_next = __float_as_uint(p.A_log[h2]);
        }
    };
    auto park_scalars = [&](int buf, int valid_rows) {
        if (tid < BT) {
            float b = p.beta_fp32 ? __uint_as_float(sc_next) : __uint_as_float(sc_next << 16);
            if (p.beta_logit) b = (tid < valid_rows) ? __fdividef(1.f, 1.f + __expf(-b)) : 0.f;    // padding rows stay 0
            sBetaBuf[buf * BT + tid] = b;
            const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(b) & 0x7fffffffu);
            if (lane == 0) sBetaMax[2 * buf + warp] = __uint_as_float(most);
        }
        else if (tid < BT + DK) sBiasBuf[buf * DK + tid - BT] = __uint_as_float(sc_next);
        else if (tid == BT + DK) sAlpha[buf] = p.gate_mode != GATE_NONE ? __expf(__uint_as_float(sc_next)) : 0.f;
    };
    publish_info(blockIdx.x, 0);
    __syncthreads();
    if ((int)blockIdx.x < p.num_tiles) {
        fetch_g(sInfo[0]);
        load_scalars(sInfo[0]);
        park_scalars(0, sInfo[0].y);
    }
    __syncthreads();

    // fp16 operands of the Gram product: 2^SH on either side keeps small gate factors of unit rows out of the subnormals. Where an
    // operand may be large, they are taken as they are: rows of unknown length (no normalisation in the kernel), decays that can
    // be positive (not activated in the kernel), a softmax scale, which rides on q, that 2^6 could carry past 65504
    const float SH = p.use_l2norm && p.gate_mode != GATE_NONE && fabsf(p.scale) <= 512.f ? 6.f : 0.f;
    const float unshift = fast_exp2(-SH), unshift2 = fast_exp2(-2.f * SH);
    // byte offset of this lane's segment of row A / B inside an atom (c and h toggle bits 6 and 3)
    const uint32_t segA = (uint32_t)(rowA * 128 + ((t ^ (rowA & 7)) << 4) + 8 * sx);
    const uint32_t segB = (uint32_t)((rowA + 1) * 128 + ((t ^ ((rowA + 1) & 7)) << 4) + 8 * sx);

    // persistent over (chunk, head) tiles; the completion barriers flip phase once per tile
    for (int tile_id = blockIdx.x, iter = 0; tile_id < p.num_tiles; tile_id += gridDim.x, ++iter) {
    const uint32_t par = iter & 1;
    const float* sBeta = sBetaBuf + par * BT;
    const int4 info = sInfo[par];
    const int valid = info.y;
    const size_t base = (size_t)info.x * tok_stride + (size_t)info.z * DK;
    unsigned char* tile = p.tiles + (size_t)tile_id * TP_BYTES;       // tile slot = chunk * H + head = tile_id
    const bool liveA = rowA < valid, liveB = rowA + 1 < valid;
    publish_info(tile_id + gridDim.x, par ^ 1);      // visible to everybody after the next barrier

    PHASE_MARK(15);

    // ---- 1. gate activation (log2 domain) and the cumulative sum over the block's 16 rows: in the thread over its two
    //         rows, then over the eight lanes that share its channels. The first row of the block is kept apart: G holds
    //         g_i - r_I (+ SH). Padding rows contribute 0 ----
    constexpr int NX = GK == GK_PER_HEAD ? 1 : 8;            // channel pairs with values of their own
    float2 GA[NX], GB[NX];
    {
        if constexpr (GK == GK_PER_HEAD) {
            GA[0] = splat2(__uint_as_float(p.g_fp32 ? graw[0].x : graw[0].x << 16));
            GB[0] = splat2(__uint_as_float(p.g_fp32 ? graw[0].y : graw[0].y << 16));
        } else {
#pragma unroll
            for (int x = 0; x < 8; ++x) {      // x = 4 c + 2 h + pair
                if constexpr (GK == GK_BF16) {
                    const uint4 a = graw[x >> 2], b = graw[2 + (x >> 2)];
                    const bool up = ((x >> 1) & 1) != sx;
                    GA[x] = unpack_bf16(x & 1 ? (up ? a.w : a.y) : (up ? a.z : a.x));
                    GB[x] = unpack_bf16(x & 1 ? (up ? b.w : b.y) : (up ? b.z : b.x));
                } else {
                    const uint4 a = graw[x >> 1], b = graw[4 + (x >> 1)];
                    GA[x] = x & 1 ? make_float2(__uint_as_float(a.z), __uint_as_float(a.w)) : make_float2(__uint_as_float(a.x), __uint_as_float(a.y));
                    GB[x] = x & 1 ? make_float2(__uint_as_float(b.z), __uint_as_float(b.w)) : make_float2(__uint_as_float(b.x), __uint_as_float(b.y));
                }
            }
        }
        auto bias2 = [&](int x) {
            return GK == GK_PER_HEAD ? splat2(sBiasBuf[par * DK])
                                     : *reinterpret_cast<const float2*>(sBiasBuf + par * DK + 64 * hf + 8 * t + 32 * (x >> 2) + 4 * (((x >> 1) & 1) ^ sx) + 2 * (x & 1));
        };
        const float alpha = sAlpha[par];
        if (p.gate_mode == GATE_LOWER_BOUND) {
            // lower_bound * sigmoid(alpha x) / ln2 with one ex2 and one rcp per element (flush-to-zero approximations)
            const float c0 = -alpha * RCP_LN2, lb = p.lower_bound * RCP_LN2, cA = liveA ? lb : 0.f, cB = liveB ? lb : 0.f;
            auto act = [&](float2 v, float2 bc, float c1) {
                const float2 e = make_float2(1.f + fast_exp2(fmaf(v.x, c0, bc.x)), 1.f + fast_exp2(fmaf(v.y, c0, bc.y)));
                return make_float2(c1 * fast_rcp(e.x), c1 * fast_rcp(e.y));
            };
#pragma unroll
            for (int x = 0; x < NX; ++x) {
                const float2 b = bias2(x), bc = make_float2(b.x * c0, b.y * c0);
                GA[x] = act(GA[x], bc, cA);
                GB[x] = act(GB[x], bc, cB);
            }
        } else if (p.gate_mode == GATE_SOFTPLUS) {
            const float c1 = -alpha * RCP_LN2;
            const float2 cA = splat2(liveA ? c1 : 0.f), cB = splat2(liveB ? c1 : 0.f);
#pragma unroll
            for (int x = 0; x < NX; ++x) {
                const float2 b = bias2(x);
                GA[x] = mul2(softplus2(add2(GA[x], b)), cA);
                GB[x] = mul2(softplus2(add2(GB[x], b)), cB);
            }
        } else {
            const float2 cA = splat2(liveA ? RCP_LN2 : 0.f), cB = splat2(liveB ? RCP_LN2 : 0.f);
#pragma unroll
            for (int x = 0; x < NX; ++x) {
                GA[x] = mul2(GA[x], cA);
                GB[x] = mul2(GB[x], cB);
            }
        }
    }
    if (tid == MMA_THREAD) {       // the previous tile's staged outputs have left the operand buffers
        bulk_wait_read_all();
        request_qk(info);
    }
    PHASE_MARK(0); // gate activation
    {
        if (pr == 0) {       // the block's first row
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                const float2 lo = GA[NX == 1 ? 0 : 2 * q4], hi = GA[NX == 1 ? 0 : 2 * q4 + 1];
                *reinterpret_cast<float4*>(sEdgeA + I * DK + 64 * hf + 8 * t + 32 * (q4 >> 1) + 4 * ((q4 & 1) ^ sx)) =
                    make_float4(lo.x, lo.y, hi.x, hi.y);
            }
#pragma unroll
            for (int x = 0; x < NX; ++x) GA[x] = splat2(SH);
        }
        // lanes of the row pairs 1, 2 and 4 before this one
        const auto lane_of = [&](int q) { return (((((q & 1) << 1) | ((q >> 1) & 1) | (q & 4)) << 2) | t); };
        const int src1 = lane_of(max(pr - 1, 0)), src2 = lane_of(max(pr - 2, 0)), src4 = lane_of(max(pr - 4, 0));
        const float2 m1 = splat2(pr >= 1 ? 1.f : 0.f), m2 = splat2(pr >= 2 ? 1.f : 0.f), m4 = splat2(pr >= 4 ? 1.f : 0.f);
#pragma unroll
        for (int x = 0; x < NX; ++x) {
            float2 inc = add2(GA[x], GB[x]);
            float2 y;
            y.x = __shfl_sync(0xffffffffu, inc.x, src1); y.y = NX == 1 ? y.x : __shfl_sync(0xffffffffu, inc.y, src1);
            inc = fma2(y, m1, inc);
            y.x = __shfl_sync(0xffffffffu, inc.x, src2); y.y = NX == 1 ? y.x : __shfl_sync(0xffffffffu, inc.y, src2);
            inc = fma2(y, m2, inc);
            y.x = __shfl_sync(0xffffffffu, inc.x, src4); y.y = NX == 1 ? y.x : __shfl_sync(0xffffffffu, inc.y, src4);
            inc = fma2(y, m4, inc);
            GA[x] = make_float2(inc.x - GB[x].x, inc.y - GB[x].y);
            GB[x] = inc;
        }
        if (pr == 7) {       // sum over rows 1..15 of the block (+ SH)
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                const float2 lo = GB[NX == 1 ? 0 : 2 * q4], hi = GB[NX == 1 ? 0 : 2 * q4 + 1];
                *reinterpret_cast<float4*>(sEdgeT + I * DK + 64 * hf + 8 * t + 32 * (q4 >> 1) + 4 * ((q4 & 1) ^ sx)) =
                    make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
    }
    PHASE_MARK(2);      // in-warp cumulative sum
    uint4 qraw[4], kraw[4];         // [row j][c]: 8 bf16 each
    if (valid == BT) {
        if (!mbar_wait(&bars[2], qk_parity)) {
            report_status(p.status, STATUS_WAIT_TIMEOUT);
            *sAbort = 1;
        }
        qk_parity ^= 1;
        const unsigned char* raw = sm + SM_OPA + hf * KATOM_A;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t so = ((j ? segB : segA) & ~15u) ^ (uint32_t)(64 * c);
                qraw[2 * j + c] = *reinterpret_cast<const uint4*>(raw + so);
                kraw[2 * j + c] = *reinterpret_cast<const uint4*>(raw + 8192 + so);
            }
    } else {
        const size_t at = base + 64 * hf + 8 * t;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const size_t roff = at + (size_t)min(rowA + j, valid - 1) * tok_stride;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                qraw[2 * j + c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.q) + roff + 32 * c);
                kraw[2 * j + c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.k) + roff + 32 * c);
            }
        }
    }
    // ---- 2. sums of squares of the thread's two q and k rows over this warp's 64 channels ----
    if (p.use_l2norm) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float2 sq = make_float2(0.f, 0.f), sk = sq;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t qw[4] = {qraw[2 * j + c].x, qraw[2 * j + c].y, qraw[2 * j + c].z, qraw[2 * j + c].w};
                const uint32_t kw[4] = {kraw[2 * j + c].x, kraw[2 * j + c].y, kraw[2 * j + c].z, kraw[2 * j + c].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 a = unpack_bf16(qw[e]), b = unpack_bf16(kw[e]);
                    sq = fma2(a, a, sq);
                    sk = fma2(b, b, sk);
                }
            }
            float s1 = sq.x + sq.y, s2 = sk.x + sk.y;
            s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s2 += __shfl_xor_sync(0xffffffffu, s2, 1);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 2); s2 += __shfl_xor_sync(0xffffffffu, s2, 2);
            if (t == 0) sNorm[hf * BT + rowA + j] = make_float2(s1, s2);
        }
    }
    PHASE_MARK(14);     // norms
    __syncthreads();          // block edges and sums of squares are visible
    PHASE_MARK(1);      // barrier
    // ---- 3. per-channel constants of this warp's block and channel half, two channels per lane ----
    float* tab = reinterpret_cast<float*>(sm + SM_TAB) + warp * 384;
    {
        const int ch = 64 * hf + 2 * lane;
        float2 a4[4], t4[4], r[5];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            a4[b] = *reinterpret_cast<const float2*>(sEdgeA + b * DK + ch);
            t4[b] = add2(*reinterpret_cast<const float2*>(sEdgeT + b * DK + ch), splat2(-SH));
        }
        r[0] = a4[0];             // r_b: cumulative log2 decay at the first row of block b; r_4 = g_last
#pragma unroll
        for (int b = 0; b < 4; ++b) r[b + 1] = b < 3 ? add2(r[b], add2(t4[b], a4[b + 1])) : add2(r[b], t4[b]);
        float2 rI = r[0], rN = r[1], dl = add2(t4[0], a4[1]);           // dl = r_{I+1} - r_I
        if (I == 1) { rI = r[1]; rN = r[2]; dl = add2(t4[1], a4[2]); }
        if (I == 2) { rI = r[2]; rN = r[3]; dl = add2(t4[2], a4[3]); }
        if (I == 3) { rI = r[3]; rN = r[4]; dl = t4[3]; }
        auto put = [&](int which, float2 v) { *reinterpret_cast<float2*>(tab + which * 64 + 2 * lane) = v; };
        put(0, add2(dl, splat2(2.f * SH)));                                             // f = 2^(this - G)
        put(1, mul2(ex2_2(rI), splat2(unshift)));                                       // q 2^g = qa * this
        // 2^(r_I - r_{I+1}) >= 1, <= 2^116 under the safe gate; the clamp keeps an unbounded gate from making inf * 0, also for
        // the last row of the chunk, whose f is 2^SH
        const float2 cb = sub2(splat2(TF32_DEBIAS2_LOG2 - 2.f * SH), dl);
        put(2, ex2_2(make_float2(fminf(cb.x, 126.f - SH), fminf(cb.y, 126.f - SH))));
        put(3, mul2(ex2_2(sub2(r[4], rN)), splat2(unshift)));                           // kg = kf * 2^(g_last - r_{I+1})
        if (I == 0) put(4, ex2_2(sub2(r[2], r[1])));                                    // copy anchored at block 2
        if (I < 2) put(5, ex2_2(sub2(r[3], rN)));                                       // copy anchored at block 3
        if (I == 3)                                                                     // 2^(g_last): the decay of the whole chunk
            *reinterpret_cast<float2*>(tile + TP_DECAY + 4 * ch) = ex2_2(r[4]);
    }
    float rq[2], rk[2];
    {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float a = 1.f, b = 1.f;
            if (p.use_l2norm) {
                const float2 n0 = sNorm[rowA + j], n1 = sNorm[BT + rowA + j];
                a = rsqrtf(n0.x + n1.x + 1e-6f);
                b = rsqrtf(n0.y + n1.y + 1e-6f);
            }
            const bool live = j ? liveB : liveA;
            rq[j] = live ? a * p.scale : 0.f;           // the softmax scale rides on q; padding rows: q = k = 0
            rk[j] = live ? b : 0.f;
        }
    }
    if (valid < BT) {             // the rows of a ragged chunk go where the box puts those of a whole one
        unsigned char* raw = sm + SM_OPA + hf * KATOM_A;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t so = ((j ? segB : segA) & ~15u) ^ (uint32_t)(64 * c);
                *reinterpret_cast<uint4*>(raw + so) = qraw[2 * j + c];
                *reinterpret_cast<uint4*>(raw + 8192 + so) = kraw[2 * j + c];
            }
    }
    __syncwarp();
    PHASE_MARK(3);      // tables
    // ---- 4. operand generation. Per element only two exponentials: eA = 2^(g_i - r_I) and f = 2^(r_{I+1} - g_i).
    //         Every other factor is one of them times a per-(block, channel) constant:
    //           2^(g_i)        = eA 2^(r_I)                   -> qg, x
    //           2^(r_I - g_i)  = f 2^(r_I - r_{I+1})          -> own-block columns (diagonal block, tf32 mma.sync)
    //           2^(g_last-g_i) = f 2^(g_last - r_{I+1})       -> kg
    //           2^(r_J - g_i)  = f 2^(r_J - r_{I+1}), J > I   -> columns of the later blocks J ----
    float dq[2][4], dk[2][4];             // diagonal block of q k^T and of k k^T: n-tile = parity of the column row, see below
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) dq[nt][e] = dk[nt][e] = 0.f;
    {
        unsigned char* opa = sm + SM_OPA + hf * KATOM_A;
        unsigned char* opb = sm + SM_OPB + hf * KATOM_B;
        unsigned char* xs = sm + SM_XS + hf * 8192;
        const int own = (8 * I * (I + 1)) * 128;      // first row of the copy anchored at block I + 1
        float eP[2], fP[2];
        if constexpr (GK == GK_PER_HEAD) {
            eP[0] = fast_exp2(GA[0].x); eP[1] = fast_exp2(GB[0].x);
            fP[0] = fast_exp2(tab[0] - GA[0].x); fP[1] = fast_exp2(tab[0] - GB[0].x);
        }
        const float2 rq2[2] = {splat2(rq[0]), splat2(rq[1])}, rk2[2] = {splat2(rk[0]), splat2(rk[1])};
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {                   // rolled: half the code, and the registers of one segment only
            uint2 kgp[2], qgp[2];                       // the first four channels of the segment, packed
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                asm volatile("" ::: "memory");          // one step at a time: the registers of four in flight would not fit
                const float* tp = tab + 32 * c + 8 * t + 4 * (h ^ sx);
                float2 kf[2][2];                                             // [row][pair]
                uint2 qr[2], kr[2];                                          // this thread's values, where their operands will go
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t so = (j ? segB : segA) ^ (uint32_t)(64 * c + 8 * h);
                    qr[j] = *reinterpret_cast<const uint2*>(opa + so);
                    kr[j] = *reinterpret_cast<const uint2*>(opa + 8192 + so);
                }
                uint32_t pa[2][2], pk[2][2], px[2][2], pg[2][2], pq[2][2];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float2 cG = *reinterpret_cast<const float2*>(tp + 64 + 2 * x), cB = *reinterpret_cast<const float2*>(tp + 128 + 2 * x),
                                 cK = *reinterpret_cast<const float2*>(tp + 192 + 2 * x);
                    float qa[2][2], ka[2][2];                                // [row][channel]; scalar products: they are MMA fragments
                    float2 ko[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t qw = x ? qr[j].y : qr[j].x, kw = x ? kr[j].y : kr[j].x;
                        float2 eA, f;
                        if constexpr (GK == GK_PER_HEAD) {
                            eA = splat2(eP[j]); f = splat2(fP[j]);
                        } else {
                            const float2 G = j ? GB[2 * h + x] : GA[2 * h + x], dl = *reinterpret_cast<const float2*>(tp + 2 * x);
                            eA = ex2_2(G);                                               // <= 2^SH
                            f = make_float2(fast_exp2(dl.x - G.x), fast_exp2(dl.y - G.y));   // <= 2^SH
                        }
                        const float2 kh = mul2(unpack_bf16(kw), rk2[j]), qh = mul2(unpack_bf16(qw), rq2[j]);
                        qa[j][0] = qh.x * eA.x; qa[j][1] = qh.y * eA.y;
                        ka[j][0] = kh.x * eA.x; ka[j][1] = kh.y * eA.y;
                        kf[j][x] = mul2(kh, f);
                        ko[j] = mul2(kf[j][x], cB);
                        const float2 kg = mul2(kf[j][x], cK);
                        pa[j][x] = pack_f16(qa[j][0], qa[j][1]);
                        pk[j][x] = pack_f16(ka[j][0], ka[j][1]);
                        pq[j][x] = pack_f16(qa[j][0] * cG.x, qa[j][1] * cG.y);
                        px[j][x] = pack_f16(ka[j][0] * cG.x, ka[j][1] * cG.y);
                        pg[j][x] = pack_f16(kg.x, kg.y);
                    }
                    const uint32_t aq[4] = {__float_as_uint(qa[0][0]), __float_as_uint(qa[1][0]), __float_as_uint(qa[0][1]), __float_as_uint(qa[1][1])};
                    const uint32_t ak[4] = {__float_as_uint(ka[0][0]), __float_as_uint(ka[1][0]), __float_as_uint(ka[0][1]), __float_as_uint(ka[1][1])};
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        const uint32_t b[2] = {__float_as_uint(ko[nt].x), __float_as_uint(ko[nt].y)};
                        mma_tf32_16x8x8(dq[nt], aq, b);
                        mma_tf32_16x8x8(dk[nt], ak, b);
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t so = (j ? segB : segA) ^ (uint32_t)(64 * c + 8 * h);
                    *reinterpret_cast<uint2*>(opa + so) = make_uint2(pa[j][0], pa[j][1]);
                    *reinterpret_cast<uint2*>(opa + 8192 + so) = make_uint2(pk[j][0], pk[j][1]);
                    *reinterpret_cast<uint2*>(xs + so) = make_uint2(px[j][0], px[j][1]);
                    if (h == 0) {
                        kgp[j] = make_uint2(pg[j][0], pg[j][1]);
                        qgp[j] = make_uint2(pq[j][0], pq[j][1]);
                    } else {
                        const int goff = swz256(rowA + j, 64 * hf + 32 * c + 8 * t);
                        const uint4 kv = sx ? make_uint4(pg[j][0], pg[j][1], kgp[j].x, kgp[j].y) : make_uint4(kgp[j].x, kgp[j].y, pg[j][0], pg[j][1]);
                        const uint4 qv = sx ? make_uint4(pq[j][0], pq[j][1], qgp[j].x, qgp[j].y) : make_uint4(qgp[j].x, qgp[j].y, pq[j][0], pq[j][1]);
                        *reinterpret_cast<uint4*>(tile + TP_KG + goff) = kv;
                        *reinterpret_cast<uint4*>(tile + TP_QG + goff) = qv;
                    }
                }
                // the columns of the later blocks; 8 I (I + 1) is a multiple of 16 rows: the swizzle is that of the row
                if (I < 3) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        *reinterpret_cast<uint2*>(opb + (uint32_t)own + ((j ? segB : segA) ^ (uint32_t)(64 * c + 8 * h))) =
                            make_uint2(pack_f16(kf[j][0].x, kf[j][0].y), pack_f16(kf[j][1].x, kf[j][1].y));
                }
                auto later = [&](int first_row, int which) {
                    const float4 cJ = *reinterpret_cast<const float4*>(tp + 64 * which);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 a = mul2(kf[j][0], make_float2(cJ.x, cJ.y)), b = mul2(kf[j][1], make_float2(cJ.z, cJ.w));
                        *reinterpret_cast<uint2*>(opb + first_row * 128 + ((j ? segB : segA) ^ (uint32_t)(64 * c + 8 * h))) =
                            make_uint2(pack_f16(a.x, a.y), pack_f16(b.x, b.y));
                    }
                };
                if (I < 2) later(48, 5);
                if (I < 1) later(16, 4);
            }
            if constexpr (NX == 8) {                    // the second segment moves into place
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    GA[x] = GA[x + 4];
                    GB[x] = GB[x + 4];
                }
            }
        }
    }
    // the two channel halves of a diagonal block are added through shared memory (rows 16 I .. of the inverse's buffer)
    float4* part = reinterpret_cast<float4*>(sAi + 16 * I * LROW);
    if (hf == 1) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            part[(2 * nt) * 32 + lane] = make_float4(dq[nt][0], dq[nt][1], dq[nt][2], dq[nt][3]);
            part[(2 * nt + 1) * 32 + lane] = make_float4(dk[nt][0], dk[nt][1], dk[nt][2], dk[nt][3]);
        }
    }
    fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    PHASE_MARK(5);      // operand generation
    if (tid == MMA_THREAD) {
        umma::fence_after_sync();
        const uint32_t idesc = umma::make_idesc(umma::FMT_F16, 128, 96, false, false);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const uint64_t ad = sdesc_sw128(sm_u32 + SM_OPA + (ks >> 2) * KATOM_A + (ks & 3) * 32, 16, 1024);
            const uint64_t bd = sdesc_sw128(sm_u32 + SM_OPB + (ks >> 2) * KATOM_B + (ks & 3) * 32, 16, 1024);
            umma::mma_f16(tmem, ad, bd, idesc, ks != 0);
        }
        umma::commit(&bars[0]);
    }
    // ---- 5. while the MMAs run: the loads whose results are needed later (this tile's v rows, the next tile's gate rows
    //         and scalars), L2 prefetches of the next tile's q, k, v rows ----
    uint4 vraw[8];
    if (hf == 1) {
        const __nv_bfloat16* vp = reinterpret_cast<const __nv_bfloat16*>(p.v) + base + 8 * (tid & 15);
#pragma unroll
        for (int n = 0; n < 8; ++n)     // rows (tid - 128) / 16 + 8 n; a padding row reads the last real row (its column of Akk is zeroed by beta)
            vraw[n] = *reinterpret_cast<const uint4*>(vp + (size_t)min(((tid - 128) >> 4) + 8 * n, valid - 1) * tok_stride);
    }
    {
        const int4 nf = sInfo[par ^ 1];
        if (nf.y > 0) {
            // (the order that spills least: a gate per head 609 -> 598 us at 4 x 8192 x 32 with the rows first, the others with them last)
            if constexpr (GK == GK_PER_HEAD) prefetch_rows(nf);
            fetch_g(nf);
            load_scalars(nf);
            if constexpr (GK != GK_PER_HEAD) prefetch_rows(nf);
        }
    }
    // ---- 6. diagonal blocks (warps 0-3, one each): add the channel halves, L = beta_i strictly lower; inverse of I + L by
    //         substitution, one column per lane ----
    uint32_t aqd[4];
    if (hf == 0) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const float4 a = part[(2 * nt) * 32 + lane], b = part[(2 * nt + 1) * 32 + lane];
            dq[nt][0] += a.x; dq[nt][1] += a.y; dq[nt][2] += a.z; dq[nt][3] += a.w;
            dk[nt][0] += b.x; dk[nt][1] += b.y; dk[nt][2] += b.z; dk[nt][3] += b.w;
        }
        // accumulator slot (row g / g + 8, column 2 t + e of n-tile nt) is row 2 pr / 2 pr + 1, column 2 perm(2 t + e) + nt
        const int cc0 = 2 * ((((2 * t) >> 1) & 1) | ((2 * t) & 4)), cc1 = cc0 + 4;    // perm(2t), perm(2t + 1) = perm(2t) + 2
        float* ld = reinterpret_cast<float*>(sm + SM_LDIAG) + I * 16 * LDROW;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = 2 * pr + j;
            const float bi = sBeta[rowA + j];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = e ? cc1 : cc0;
                const float q0 = dq[0][2 * j + e], q1 = dq[1][2 * j + e], k0 = dk[0][2 * j + e], k1 = dk[1][2 * j + e];
                aqd[2 * j + e] = pack_f16(col <= i ? q0 : 0.f, col + 1 <= i ? q1 : 0.f);
                const float m0 = col < i ? k0 : 0.f, m1 = col + 1 < i ? k1 : 0.f;
                *reinterpret_cast<float2*>(ld + i * LDROW + col) = make_float2(bi * m0, bi * m1);
                if (p.mkk_out)       // the same Gram entries without beta, for the backward pass
                    *reinterpret_cast<float2*>(p.mkk_out + (size_t)tile_id * BT * BT + (16 * I + i) * BT + 16 * I + col) = make_float2(m0, m1);
            }
        }
        __syncwarp();
        const int cc = lane & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float acc = (i == cc) ? 1.f : 0.f;
#pragma unroll
            for (int j4 = 0; j4 < i; j4 += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(ld + i * LDROW + j4);
                acc = fmaf(-l4.x, x[j4], acc);
                if (j4 + 1 < i) acc = fmaf(-l4.y, x[j4 + 1], acc);
                if (j4 + 2 < i) acc = fmaf(-l4.z, x[j4 + 2], acc);
                if (j4 + 3 < i) acc = fmaf(-l4.w, x[j4 + 3], acc);
            }
            x[i] = acc;
        }
        // lanes 16-31 clear the block right of the diagonal block inside its 32x32 pair (it is read as part of the pair)
        if (lane < 16 || !(I & 1)) {
            float* xd = sAi + 16 * I * LROW + 16 * I + lane;
#pragma unroll
            for (int i = 0; i < 16; ++i) xd[i * LROW] = lane < 16 ? x[i] : 0.f;
        }
    }
    PHASE_MARK(12);     // loads issued, diagonal blocks inverted
    if (!wait_mma(0, par)) break;
    PHASE_MARK(6);      // wait for the Gram MMAs
    // ---- 7. blocks below the diagonal out of TMEM (warps 4-7; lanes 0..63 hold the q rows -> Aqk, lanes 64..127 the k rows
    //         -> L, not yet inverted, in place); diagonal and upper blocks of Aqk (warps 0-3) ----
    if (hf == 1) {
        const int qd = warp & 3, row = 32 * (qd & 1) + lane, blk = row >> 4;
        const bool is_q = qd < 2;
        const float f = is_q ? unshift2 : unshift2 * sBeta[row];
        const uint32_t taddr = tmem + ((uint32_t)(qd * 32) << 16);
        auto emit = [&](const uint32_t (&r)[16], int b, int gcol) {
            if (blk == b) {
                if (is_q) {
#pragma unroll
                    for (int hc = 0; hc < 2; ++hc) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            o[e] = pack_f16(f * __uint_as_float(r[8 * hc + 2 * e]), f * __uint_as_float(r[8 * hc + 2 * e + 1]));
                        *reinterpret_cast<uint4*>(sm + SM_STG_AQK + swz128(row, 16 * gcol + 8 * hc)) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                } else {
                    float* mo = p.mkk_out ? p.mkk_out + (size_t)tile_id * BT * BT + row * BT + 16 * gcol : nullptr;
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        const float4 v = make_float4(__uint_as_float(r[4 * q4]), __uint_as_float(r[4 * q4 + 1]), __uint_as_float(r[4 * q4 + 2]),
                                                     __uint_as_float(r[4 * q4 + 3]));
                        *reinterpret_cast<float4*>(sAi + row * LROW + 16 * gcol + 4 * q4) = make_float4(f * v.x, f * v.y, f * v.z, f * v.w);
                        if (mo)
                            *reinterpret_cast<float4*>(mo + 4 * q4) = make_float4(unshift2 * v.x, unshift2 * v.y, unshift2 * v.z, unshift2 * v.w);
                    }
                }
            }
        };
        // rows 32..63: block 2 against blocks 0, 1, block 3 against 0, 1, 2; rows 0..31: block 1 against block 0. Not unrolled: the kernel
        // runs its code once a tile, the instruction cache does not hold it, and these are 8 KB of 95 (774 -> 762 us at 4 x 8192 x 32).
#pragma unroll 1
        for (int pair = qd & 1; pair <= 5 * (qd & 1); ++pair) {
            uint32_t r[16];
            umma::ld_32x32b_x16(taddr + 16 * pair, r);
            umma::wait_ld();
            emit(r, pair == 0 ? 1 : pair < 3 ? 2 : 3, pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3);
        }
    } else {
        const int cc0 = 2 * ((t & 1) | ((2 * t) & 4));
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                *reinterpret_cast<uint32_t*>(sm + SM_STG_AQK + swz128(rowA + j, 16 * I + cc0 + 4 * e)) = aqd[2 * j + e];
        for (int idx = lane; idx < 32 * (3 - I); idx += 32) {
            const int row = 16 * I + (idx & 15), ch = 2 * I + 2 + (idx >> 4);
            *reinterpret_cast<uint4*>(sm + SM_STG_AQK + swz128(row, 8 * ch)) = make_uint4(0, 0, 0, 0);
        }
    }
    PHASE_MARK(13);     // Gram epilogue
    park_scalars(par ^ 1, sInfo[par ^ 1].y);
    umma::fence_before_sync();
    __syncthreads();

    // ---- 8. Akk = (I + L)^-1: 16->32->64 block merges X = -D2inv C D1inv as split-TF32 mma.sync products (three MMAs per
    //         step recover fp32-level accuracy). First level: one warp per pair, the intermediate product D2inv C stays in
    //         its accumulators, which are the A fragments of the second product under a permutation of the contraction
    //         index; the other six warps stage Y = v meanwhile ----
    if (warp < 2) {
        float* blk = sAi + 32 * warp * LROW + 32 * warp;
        const float *D1 = blk, *C = blk + 16 * LROW, *D2 = C + 16;
        float P[2][4], X[2][4], Pc[2][4], Xc[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) P[nt][e] = X[nt][e] = Pc[nt][e] = Xc[nt][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const float af[4] = {D2[g * LROW + 8 * ks + t], D2[(g + 8) * LROW + 8 * ks + t], D2[g * LROW + 8 * ks + t + 4],
                                 D2[(g + 8) * LROW + 8 * ks + t + 4]};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float bf[2] = {C[(8 * ks + t) * LROW + 8 * nt + g], C[(8 * ks + t + 4) * LROW + 8 * nt + g]};
                mma_3xtf32(P[nt], Pc[nt], af, bf);
            }
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {          // k slot t is column 8 ks + 2 t, slot t + 4 column 8 ks + 2 t + 1
            const float af[4] = {P[ks][0] + Pc[ks][0], P[ks][2] + Pc[ks][2], P[ks][1] + Pc[ks][1], P[ks][3] + Pc[ks][3]};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float bf[2] = {D1[(8 * ks + 2 * t) * LROW + 8 * nt + g], D1[(8 * ks + 2 * t + 1) * LROW + 8 * nt + g]};
                mma_3xtf32(X[nt], Xc[nt], af, bf);
            }
        }
        __syncwarp();                             // every lane has read C
        float* xd = blk + 16 * LROW;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            *reinterpret_cast<float2*>(xd + g * LROW + 8 * nt + 2 * t) = make_float2(-X[nt][0] - Xc[nt][0], -X[nt][1] - Xc[nt][1]);
            *reinterpret_cast<float2*>(xd + (g + 8) * LROW + 8 * nt + 2 * t) = make_float2(-X[nt][2] - Xc[nt][2], -X[nt][3] - Xc[nt][3]);
        }
    } else if (hf == 1) {
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int j = ((tid - 128) >> 4) + 8 * n, ch = tid & 15;
            const uint32_t w4[4] = {vraw[n].x, vraw[n].y, vraw[n].z, vraw[n].w};
            uint32_t o4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16(w4[e]);
                o4[e] = pack_f16(f.x, f.y);
            }
            *reinterpret_cast<uint4*>(sm + SM_YS + (ch >> 3) * 8192 + j * 128 + (((ch & 7) ^ (j & 7)) << 4)) =
                make_uint4(o4[0], o4[1], o4[2], o4[3]);
        }
    }
    __syncthreads();
    // A tile whose betas are all small takes them times a power of two (largest in [1/2, 1)) into the fp16 operand, and that out of w
    // and u again; 1, and no work, from 2^-6 up
    float beta_up = 1.f;
    {
        const float most = fmaxf(sBetaMax[2 * par], sBetaMax[2 * par + 1]);
        if (most < 0.015625f && most > 0.f) beta_up = __int_as_float(min(253 - (__float_as_int(most) >> 23), 127 + 60) << 23);
    }
    {
        // second level: block rows 32..63 x columns 0..31. One 16x8 tile per warp (2 m-tiles x 4 n-tiles)
        const int mt = warp >> 2, nt = warp & 3;
        float* sT = reinterpret_cast<float*>(sm + SM_TM);
        {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            mma_tile_3xtf32<4>(sAi + (32 + 16 * mt) * LROW, LROW, sAi + 8 * nt, LROW, acc, g, t);
            float* td = sT + (16 * mt) * TROW + 8 * nt + 2 * t;
            *reinterpret_cast<float2*>(td + g * TROW) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(td + (g + 8) * TROW) = make_float2(acc[2], acc[3]);
        }
        __syncthreads();
        // Akk diag(beta) -> fp16 K-major operand, rows 64..127 repeating rows 0..63 (and fp32 Akk to HBM when the backward pass
        // wants it): the block just computed from its registers, the finished diagonal 32x32 blocks from shared memory
        {
            const int half = tid >> 7, row = 32 * half + ((tid >> 2) & 31), ch = 4 * half + (tid & 3);
            const float4 lo = *reinterpret_cast<const float4*>(sAi + row * LROW + 8 * ch), hi = *reinterpret_cast<const float4*>(sAi + row * LROW + 8 * ch + 4);
            float4 b0 = *reinterpret_cast<const float4*>(sBeta + 8 * ch), b1 = *reinterpret_cast<const float4*>(sBeta + 8 * ch + 4);
            if (beta_up != 1.f) {
                b0.x *= beta_up; b0.y *= beta_up; b0.z *= beta_up; b0.w *= beta_up;
                b1.x *= beta_up; b1.y *= beta_up; b1.z *= beta_up; b1.w *= beta_up;
            }
            const uint4 pk = make_uint4(pack_f16(b0.x * lo.x, b0.y * lo.y), pack_f16(b0.z * lo.z, b0.w * lo.w), pack_f16(b1.x * hi.x, b1.y * hi.y),
                                        pack_f16(b1.z * hi.z, b1.w * hi.w));
            unsigned char* dst = sm + SM_AKK16 + row * 128 + ((ch ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(dst) = pk;
            *reinterpret_cast<uint4*>(dst + 8192) = pk;
            if (half == 0) {                       // the 32x32 block right of the diagonal
                unsigned char* zd = sm + SM_AKK16 + row * 128 + (((4 + ch) ^ (row & 7)) << 4);
                *reinterpret_cast<uint4*>(zd) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(zd + 8192) = make_uint4(0, 0, 0, 0);
            }
            if (p.akk_out) {
                float* ao = p.akk_out + (size_t)tile_id * BT * BT + row * BT + 8 * ch;
                *reinterpret_cast<float4*>(ao) = lo;
                *reinterpret_cast<float4*>(ao + 4) = hi;
                if (half == 0) {
                    *reinterpret_cast<float4*>(ao + 32) = make_float4(0.f, 0.f, 0.f, 0.f);
                    *reinterpret_cast<float4*>(ao + 36) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            const float2 bc = mul2(*reinterpret_cast<const float2*>(sBeta + 8 * nt + 2 * t), splat2(beta_up));
            if (mt == 0) mma_tile_3xtf32<2>(sAi + 32 * LROW + 32, LROW, sT + 8 * nt, TROW, acc, g, t);     // D2inv is lower triangular
            else mma_tile_3xtf32<4>(sAi + 48 * LROW + 32, LROW, sT + 8 * nt, TROW, acc, g, t);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int row = 32 + 16 * mt + g + 8 * j;
                const float x0 = -acc[2 * j], x1 = -acc[2 * j + 1];
                const uint32_t pk = pack_f16(bc.x * x0, bc.y * x1);
                unsigned char* dst = sm + SM_AKK16 + swz128(row, 8 * nt + 2 * t);
                *reinterpret_cast<uint32_t*>(dst) = pk;
                *reinterpret_cast<uint32_t*>(dst + 8192) = pk;
                if (p.akk_out)
                    *reinterpret_cast<float2*>(p.akk_out + (size_t)tile_id * BT * BT + row * BT + 8 * nt + 2 * t) = make_float2(x0, x1);
            }
        }
    }
    fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    PHASE_MARK(8);      // triangular inverse, Y staging, Akk pack

    // ---- 9. [w | u] = Akk diag(beta * beta_up) [X | Y]: two M=128 x N=128 x K=64 products into TMEM columns 0..127 (w) and 128..255 (u).
    //         A = Akk diag(beta) stacked twice (K-major), so TMEM lanes 0..63 and 64..127 both hold the 64 token rows;
    //         B = X, then Y, each as two MN-major 64-channel atoms ----
    if (tid == MMA_THREAD) {
        umma::fence_after_sync();
        const uint32_t idesc = umma::make_idesc(umma::FMT_F16, 128, 128, false, true);
#pragma unroll
        for (int part2 = 0; part2 < 2; ++part2) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const uint64_t ad = sdesc_sw128(sm_u32 + SM_AKK16 + ks * 32, 16, 1024);
                const uint64_t bd = sdesc_sw128(sm_u32 + (part2 ? SM_YS : SM_XS) + ks * 2048, 8192, 1024);
                umma::mma_f16(tmem + 128 * part2, ad, bd, idesc, ks != 0);
            }
        }
        umma::commit(&bars[1]);
    }
    PHASE_MARK(9);      // W/U MMA issue
    if (!wait_mma(1, par)) break;
    PHASE_MARK(10);     // W/U MMA wait

    // ---- 10. epilogue: lane = token, columns = channels; lanes 0..63 write w, the duplicate lanes 64..127 write u;
    //          each thread converts 64 channels to fp16 and stores 16 bytes at a time ----
    {
        const int qd = warp & 3, is_u = qd >> 1, tok = 32 * (qd & 1) + lane;
        const int ch0 = (warp >> 2) * 64;                      // first channel (0..127) of this warp
        const uint32_t taddr = tmem + ((uint32_t)(32 * qd) << 16) + 128 * is_u + ch0;
        unsigned char* dst = is_u ? sm + SM_STG_U + (warp >> 2) * 8192 + tok * 128 : sm + SM_STG_W + tok * 256 + (warp >> 2) * 128;
        __half2 big = __floats2half2_rn(0.f, 0.f);             // running maximum of |.|; NaN propagates
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) {
            uint32_t r[2][16];
            umma::ld_32x32b_x16(taddr + 32 * cp, r[0]);
            umma::ld_32x32b_x16(taddr + 32 * cp + 16, r[1]);
            umma::wait_ld();
            if (beta_up != 1.f) {
                const float down = __int_as_float(0x7f000000 - __float_as_int(beta_up));      // 1 / beta_up
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    r[0][e] = __float_as_uint(down * __uint_as_float(r[0][e]));
                    r[1][e] = __float_as_uint(down * __uint_as_float(r[1][e]));
                }
            }
#pragma unroll
            for (int hc = 0; hc < 4; ++hc) {
                const uint32_t* rr = r[hc >> 1] + 8 * (hc & 1);
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __half2 v = __floats2half2_rn(__uint_as_float(rr[2 * e]), __uint_as_float(rr[2 * e + 1]));
                    big = __hmax2_nan(big, __habs2(v));
                    o[e] = *reinterpret_cast<const uint32_t*>(&v);
                }
                // 16-byte group of the row inside its 128-byte half, swizzled as the tile pack wants it
                *reinterpret_cast<uint4*>(dst + (((4 * cp + hc) ^ (tok & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
        // w and u inherit the range of v and of (I + L)^-1: fp16 has no room beyond 65504, so say so instead of
        // handing inf to the scan
        const bool out_of_range = f16x2_not_finite(*reinterpret_cast<const uint32_t*>(&big));
        if (__any_sync(0xffffffffu, out_of_range) && lane == 0) report_status(p.status, STATUS_RANGE);
    }
    fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();      // TMEM columns are free for the next tile; the staged outputs are complete
    umma::fence_after_sync();
    if (tid == MMA_THREAD) {       // w, u and Aqk leave as three bulk copies; their buffers are next written by the operand generation
        bulk_s2g(tile + TP_W, sm + SM_STG_W, 16384);
        bulk_s2g(tile + TP_U, sm + SM_STG_U, 16384);
        bulk_s2g(tile + TP_AQK, sm + SM_STG_AQK, 8192);
        bulk_commit();
    }
    PHASE_MARK(11);     // W/U epilogue
    }  // tile loop
    if (tid == MMA_THREAD) {
        if (*sAbort) mbar_wait(&bars[2], qk_parity ^ 1);      // q and k rows in flight (bounded again)
        bulk_wait_all();                           // staged outputs must be on their way before the shared memory goes away
    }
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 256);
    pdl_wait();      // an overlapping launch: what follows in the stream counts on the kernel before this one as well
}

}  // namespace kda

extern "C" int kda_fwd_intra_smem_bytes() { return kda::SM_TOTAL + 1024; }

#ifdef KDA_PHASE_TIMERS
extern "C" int kda_fwd_intra_read_timers(unsigned long long* out, int reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, kda_fwd_intra_timers, sizeof(kda_fwd_intra_timers));
    if (e == cudaSuccess && reset) {
        unsigned long long z[16] = {};
        e = cudaMemcpyToSymbol(kda_fwd_intra_timers, z, sizeof(z));
    }
    return (int)e;
}
#endif

extern "C" int kda_launch_fwd_intra(const kda::IntraParams* p, int num_chunks, cudaStream_t stream) {
    using namespace kda;
    if (num_chunks <= 0) return 0;
    const int smem = SM_TOTAL + 1024;
    const int kind = p->g_per_head ? GK_PER_HEAD : p->g_fp32 ? GK_FP32 : GK_BF16;
    auto kernel = kind == GK_PER_HEAD ? kda_fwd_intra_kernel<GK_PER_HEAD> : kind == GK_FP32 ? kda_fwd_intra_kernel<GK_FP32> : kda_fwd_intra_kernel<GK_BF16>;
    static std::atomic<unsigned long long> done[3];
    cudaError_t e = allow_smem(kernel, smem, done[kind]);
    if (e != cudaSuccess) return (int)e;
    const int sms = sm_count();
    IntraParams q = *p;
    q.num_tiles = num_chunks * p->H;
    const int most = q.max_ctas > 0 && q.max_ctas < 2 * sms ? q.max_ctas : 2 * sms;     // two resident CTAs per SM
    const int grid = q.num_tiles < most ? q.num_tiles : most;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(INTRA_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = q.overlap ? 1 : 0;
    // (whole chunks lie inside the tensors, whose length a packed batch does not tell)
    IntraMaps maps;
    if (!make_half_rows_map(&maps.q, p->q, p->H) || !make_half_rows_map(&maps.k, p->k, p->H) || !make_half_rows_map(&maps.v, p->v, p->H))
        return (int)cudaErrorInvalidValue;
    const cudaError_t launch = launched(cudaLaunchKernelEx(&cfg, kernel, q, maps));
    return (int)(launch != cudaSuccess ? launch : cudaGetLastError());
}
