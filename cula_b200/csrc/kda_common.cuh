// Shared definitions for the sm_100a KDA kernels: tile-pack layout, swizzles, PTX wrappers.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace kda {

constexpr int BT = 64;    // chunk length (tokens); fixed at 64 as in cula/kda/chunk.py:54
constexpr int DK = 128;   // key head dim
constexpr int DV = 128;   // value head dim
constexpr float RCP_LN2 = 1.4426950408889634f;

// ---------------------------------------------------------------------------------------------
// Forward tile pack: everything the state scans need for one (chunk, head), contiguous in HBM. The
// matrices are row-major with the 16-byte column groups XOR-swizzled by (row & 7), which is the 128-byte
// swizzle of tensor-core operand atoms: the scans fetch W, QG and KG as boxes of 64 channels that land as
// such atoms, and the rest (an atom column already, or no operand) with untiled bulk copies.
//   W    [64][128] fp16   w  = Akk (beta k 2^g)
//   QG   [64][128] fp16   qg = scale * q 2^g
//   KG   [64][128] fp16   kg = k 2^(g_last - g)
//   AQK  [64][64]  fp16   scale * tril(q k^T gated)
//   DECAY[128]     fp32   2^(g_last)
//   U   [2][64][64] fp16  u = Akk (beta v), value columns 0..63, then 64..127
// ---------------------------------------------------------------------------------------------
constexpr int TP_W = 0;
constexpr int TP_QG = 16384;
constexpr int TP_KG = 32768;
constexpr int TP_AQK = 49152;
constexpr int TP_DECAY = 57344;
constexpr int TP_U = 57856;
constexpr int TP_BYTES = 74240;

// byte offset of element (row, col) of a 2-byte matrix with 128 columns (256-byte rows)
__host__ __device__ __forceinline__ int swz256(int row, int col) {
    return row * 256 + ((((col >> 3) ^ (row & 7))) << 4) + ((col & 7) << 1);
}
// same for 64 columns (128-byte rows)
__host__ __device__ __forceinline__ int swz128(int row, int col) {
    return row * 128 + ((((col >> 3) ^ (row & 7))) << 4) + ((col & 7) << 1);
}

// Status word values written by kernels whose bounded waits give up.
constexpr int STATUS_OK = 0;
constexpr int STATUS_WAIT_TIMEOUT = 1;
constexpr int STATUS_BAD_INDEX = 2;        // a state-pool index past the end of the pool (decode)
constexpr int STATUS_RANGE = 3;            // a forward intermediate left the fp16 range (or is not finite)

// A plain store: the word may live in device memory or in pinned host memory (where the host polls it without a copy).
__device__ __forceinline__ void report_status(int* status, int code) { *reinterpret_cast<volatile int*>(status) = code; }

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
}
// one instruction asks for a whole contiguous range (16-byte aligned, a multiple of 16 bytes) to be brought into L2
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// true if either fp16 half of x is +-inf or NaN (exponent bits all ones)
__device__ __forceinline__ bool f16x2_not_finite(uint32_t x) {
    return __vcmpeq2(x & 0x7c007c00u, 0x7c007c00u) != 0u;
}
__device__ __forceinline__ float2 unpack_f16(uint32_t x) {
    return __half22float2(*reinterpret_cast<__half2*>(&x));
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t x) {
    // a bf16 is the upper half of an fp32: one shift and one mask (the library conversion takes a permute more per element)
    return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
}

// ---- packed fp32 pairs (one instruction per two lanes of arithmetic on sm_100) ----
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{.reg .b64 ra, rb, rc; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mul.rn.f32x2 rc, ra, rb; mov.b64 {%0, %1}, rc;}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{.reg .b64 ra, rb, rc; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; add.rn.f32x2 rc, ra, rb; mov.b64 {%0, %1}, rc;}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{.reg .b64 ra, rb, rc, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mov.b64 rc, {%6, %7}; "
        "fma.rn.f32x2 rd, ra, rb, rc; mov.b64 {%0, %1}, rd;}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 splat2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 ex2_2(float2 a) { return make_float2(fast_exp2(a.x), fast_exp2(a.y)); }
// softplus(x) = max(x, 0) + log1p(e), e = exp(-|x|) <= 1, with log1p(e) = 2 atanh(s), s = e / (2 + e) <= 1/3, by its series in
// s^2 <= 1/9 up to s^12 (next term 1.4e-8 relative): as accurate for strongly negative x (weak decays) as anywhere else.
__device__ __forceinline__ float2 softplus2(float2 x) {
    const float2 e = ex2_2(make_float2(-RCP_LN2 * fabsf(x.x), -RCP_LN2 * fabsf(x.y)));
    const float2 d = add2(e, splat2(2.f));
    const float2 s = mul2(e, make_float2(fast_rcp(d.x), fast_rcp(d.y))), z = mul2(s, s);
    float2 q = fma2(z, splat2(2.f / 13.f), splat2(2.f / 11.f));
    q = fma2(z, q, splat2(2.f / 9.f));
    q = fma2(z, q, splat2(2.f / 7.f));
    q = fma2(z, q, splat2(2.f / 5.f));
    q = fma2(z, q, splat2(2.f / 3.f));
    q = fma2(z, q, splat2(2.f));
    return fma2(s, q, make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}

// ---- programmatic dependent launch: a kernel launched with the programmatic-stream-serialization attribute may start
//      while its predecessor in the stream is still running; it must call pdl_wait() before it touches anything the
//      predecessor writes. pdl_launch_dependents() in the predecessor lets the dependent grid be scheduled early. ----
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- mbarrier + bulk copy (TMA engine, untiled form) ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// more bytes for the phase that is open, without an arrival
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// One bounded poll: the hardware suspends the warp until the phase completes or the hint (in nanoseconds) runs out, so that
// waiting warps do not take issue slots from the working ones of their scheduler.
constexpr uint32_t MBAR_SUSPEND_NS = 16384;
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(MBAR_SUSPEND_NS) : "memory");
    return ok != 0;
}
// Bounded wait: gives up after about a second (by default; at least `limit` short polls) and reports false (the caller
// records a status and unwinds).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit = (1 << 16)) {
    for (int i = 0; i < limit; ++i)
        if (mbar_test(bar, parity)) return true;
    return false;
}
// The same without the suspend hint: wakes up a little sooner, for the one waiting warp of a CTA whose others are parked on a barrier.
__device__ __forceinline__ bool mbar_spin(uint64_t* bar, uint32_t parity, int limit = (1 << 22)) {
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (i > 64) __nanosleep(64);
    }
    return false;
}
// global -> shared bulk copy; bytes multiple of 16, both addresses 16-byte aligned.
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// shared -> global bulk copy (same alignment rules), tracked by the issuing thread's bulk-async groups
__device__ __forceinline__ void bulk_s2g(void* gmem_dst, const void* smem_src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 :: "l"(gmem_dst), "r"(smem_u32(smem_src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all committed groups have finished READING shared memory (the buffers may be overwritten)
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// all committed groups have completed
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// Chunk geometry. A "chunk" never straddles two sequences. For a packed batch the host supplies
// cu_seqlens [N+1] and chunk_indices [NT][2] = (sequence, chunk inside the sequence), the same
// tables the reference builds with prepare_chunk_indices; a fixed-length batch passes null tables.
// ---------------------------------------------------------------------------------------------
struct ChunkInfo {
    int seq;     // sequence index
    int row0;    // first token row in the flattened [B*T] token axis
    int valid;   // number of real tokens in this chunk (1..64)
};
// stride: tokens from the start of one sequence of a fixed-length batch to the next (0: T)
__device__ __forceinline__ ChunkInfo chunk_info(int c, const int* cu_seqlens, const int* chunk_indices, int T, int stride = 0) {
    ChunkInfo ci;
    if (cu_seqlens) {
        ci.seq = chunk_indices[2 * c];
        int lc = chunk_indices[2 * c + 1];
        int bos = cu_seqlens[ci.seq], eos = cu_seqlens[ci.seq + 1];
        ci.row0 = bos + lc * BT;
        ci.valid = min(BT, eos - ci.row0);
    } else {
        int cps = (T + BT - 1) / BT;
        ci.seq = c / cps;
        int lc = c - ci.seq * cps;
        ci.row0 = ci.seq * (stride ? stride : T) + lc * BT;
        ci.valid = min(BT, T - lc * BT);
    }
    return ci;
}

// ---------------------------------------------------------------------------------------------
// Launch-side helpers: attributes that never change are asked for once per device, not on every launch
// ---------------------------------------------------------------------------------------------
constexpr int MAX_DEVICES = 64;
inline int current_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}
inline int sm_count() {
    static std::atomic<int> counts[MAX_DEVICES];
    const int dev = current_device();
    if (dev < 0 || dev >= MAX_DEVICES) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return sms;
    }
    int sms = counts[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        counts[dev].store(sms, std::memory_order_relaxed);
    }
    return sms;
}
// The result of a launch. One that was refused also leaves its error for whoever asks next (torch after its own next kernel): it is
// taken along here, since the caller gets it as the return value.
inline cudaError_t launched(cudaError_t e) {
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}
// A launch that may be scheduled while the kernel before it in the stream drains; the kernel calls pdl_launch_dependents() and, before it
// touches memory, pdl_wait().
template <typename... P, typename... A>
inline cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t stream, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return launched(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}
// raise the dynamic shared memory limit of one kernel (a function-local static `done` per kernel holds the devices it was
// raised on)
template <typename Kernel>
inline cudaError_t allow_smem(Kernel kernel, int bytes, std::atomic<unsigned long long>& done) {
    const int dev = current_device();
    const unsigned long long bit = dev >= 0 && dev < MAX_DEVICES ? 1ull << dev : 0;
    if (bit && (done.load(std::memory_order_relaxed) & bit)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

}  // namespace kda
