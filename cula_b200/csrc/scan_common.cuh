// What the forward and the reverse state scan share: shared-memory operand descriptors, TMA moves of the tile packs and token
// rows, and the maps for them.
#pragma once
#include "kda_common.cuh"
#include "kda_params.h"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace kda {

__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 :: "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t smem_src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 :: "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int x, int y, int z) {      // towards L2
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
                 :: "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ uint64_t sc_sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return umma::make_sdesc(addr, lbo, sbo) | (2ull << 61);     // 128-byte swizzle
}
// arrival of a whole warp (its tensor-memory and shared-memory accesses before this point are ordered first)
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// ---- the carried state, 32 key channels of one value column per lane ----
__device__ __forceinline__ float abs_max(const float (&s)[32]) {
    float m0 = 0.f, m1 = 0.f;
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
        m0 = fmaxf(m0, fabsf(s[k]));
        m1 = fmaxf(m1, fabsf(s[k + 1]));
    }
    return fmaxf(m0, m1);
}
// Power of two that takes values of at most `bound` below 2^14, and its inverse
__device__ __forceinline__ void fp16_scale(float bound, float& up, float& down) {
    int shift = 13 - (((__float_as_int(bound) >> 23) & 0xff) - 127);
    shift = max(-100, min(100, shift));
    up = __int_as_float((shift + 127) << 23);
    down = __int_as_float((127 - shift) << 23);
}
// fp16 copy of the state in tensor memory, as A operand
__device__ __forceinline__ void store_f16(uint32_t taddr, const float (&s)[32], float up) {
    uint32_t pk[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const float2 x = mul2(make_float2(s[2 * e], s[2 * e + 1]), splat2(up));
        pk[e] = pack_f16(x.x, x.y);
    }
    umma::st_32x32b_x16(taddr, pk);
}
// The state times the decays of its 32 channels, as the accumulator that the chunk's products are added to
__device__ __forceinline__ void store_decayed(uint32_t taddr, const float (&s)[32], const float* dec) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        uint32_t r[8];
#pragma unroll
        for (int e = 0; e < 8; e += 4) {
            const float4 d = *reinterpret_cast<const float4*>(dec + 8 * b + e);
            const float2 x = mul2(make_float2(s[8 * b + e], s[8 * b + e + 1]), make_float2(d.x, d.y));
            const float2 y = mul2(make_float2(s[8 * b + e + 2], s[8 * b + e + 3]), make_float2(d.z, d.w));
            r[e] = __float_as_uint(x.x); r[e + 1] = __float_as_uint(x.y); r[e + 2] = __float_as_uint(y.x); r[e + 3] = __float_as_uint(y.y);
        }
        umma::st_32x32b_x8(taddr + 8 * b, r);
    }
}
// Largest of 32 decays, one per lane (they are not negative: as integers they order the same)
__device__ __forceinline__ float warp_max_decay(float d) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(d))); }

// ---- token rows in shared memory from lane-per-column registers ----
// A register holds the 16-bit values of tokens t0 + 2e and t0 + 2e + 1 of value column v; neighbouring lanes trade halves, so that
// the even lane stores the first token of both columns and the odd lane the second. `flip`: bits to toggle (signs).
__device__ __forceinline__ void stage_rows(unsigned char* buf, int t0, int v, const uint32_t (&w)[8], uint32_t flip = 0) {
    const int odd = v & 1;
    const uint32_t sel = odd ? 0x3276u : 0x5410u;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const uint32_t x = __shfl_xor_sync(0xffffffffu, w[e], 1);
        *reinterpret_cast<uint32_t*>(buf + (t0 + 2 * e + odd) * 256 + (v & ~1) * 2) = __byte_perm(w[e], x, sel) ^ flip;
    }
}
// Everything this thread staged may leave by a bulk copy once all warps have arrived on `bar`; thread 0 also waits until the copy of
// the turn before has been read out, so that passing the barrier frees that buffer.
__device__ __forceinline__ void arrive_staged(uint64_t* bar, int tid) {
    fence_proxy_async();
    if (tid == 0) bulk_wait_read_all();
    warp_arrive(bar, tid & 31);
}

// How large fp16 operands in shared memory can be: the bitwise OR of their words. This warp's BYTES of them are added to `acc`.
// (A maximum takes eight times the instructions, and the warps that have a stage's operands in hand wait for it on the chain.)
template <int BYTES>
__device__ __forceinline__ void or_operands(const unsigned char* part, int lane, uint32_t* acc) {
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < BYTES / 512; ++i) {
        const uint4 v = *reinterpret_cast<const uint4*>(part + i * 512 + lane * 16);
        x |= v.x | v.y | v.z | v.w;
    }
    x = __reduce_or_sync(0xffffffffu, x);
    if (lane == 0) atomicOr(acc, x);
}
// A power of two above every entry: twice that of the ORed exponents, which are at least the largest one. Entries on both sides of 1
// can make it overshoot by up to 2^16; in the bound behind an fp16 scale that costs none of the 11 bits of the largest entries.
__device__ __forceinline__ float or_bound(uint32_t x) { return __uint_as_float((((x | x >> 16) & 0x7c00u) << 13) + (113u << 23)); }

// W, QG and KG of the tile packs as a rank-4 tensor of fp16: 64 channels, 2 channel halves, 192 rows (64 of each matrix),
// tiles; fetched as boxes of 64 channels x 64 rows.
inline bool make_pack_map(CUtensorMap* map, const unsigned char* tiles, long long num_tiles) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    static_assert(TP_W == 0 && TP_QG == 16384 && TP_KG == 32768 && TP_BYTES % 16 == 0, "three stacked matrices of 256-byte rows");
    const cuuint64_t dims[4] = {64, 2, 192, (cuuint64_t)num_tiles};
    const cuuint64_t strides[3] = {128, 256, TP_BYTES};
    const cuuint32_t box[4] = {64, 1, 64, 1}, elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<unsigned char*>(tiles), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Token rows [tokens][heads][128] of bf16 (or fp32), moved as boxes of 64 tokens of one head; rows past `tokens` are read as zeros. It may be
// an upper bound where only whole chunks, which lie inside the tensor, are moved.
inline bool make_rows_map(CUtensorMap* map, void* rows, int H, long long tokens, bool fp32 = false) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {128, (cuuint64_t)H, (cuuint64_t)tokens};
    const cuuint64_t row = fp32 ? 512 : 256, strides[2] = {row, (cuuint64_t)H * row};
    const cuuint32_t box[3] = {128, 1, 64}, elem[3] = {1, 1, 1};
    return fn(map, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, rows, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The same in boxes of 64 channels, as 128-byte-swizzled atoms; only whole chunks, which lie inside the tensor, are moved.
inline bool make_half_rows_map(CUtensorMap* map, const void* rows, int H) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {128, (cuuint64_t)H, 1ull << 30}, strides[2] = {256, (cuuint64_t)H * 256};
    const cuuint32_t box[3] = {64, 1, 64}, elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(rows), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace kda
