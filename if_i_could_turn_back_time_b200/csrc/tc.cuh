// Building blocks of the TMA-fed tensor-core kernels (sm_100a): mbarriers with bounded waits, TMA and bulk copies,
// tcgen05 instructions with the A operand in tensor memory, and the look-up of the tensor-map encoder.
#pragma once
#include "common.cuh"
#include <cuda.h>
#include <mutex>

namespace jqta {

constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{ .reg .b64 t; mbarrier.arrive.shared::cta.b64 t, [%0]; }" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 t; mbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// The same, suspended by the hardware for up to about a microsecond: a waiting warp that polls takes issue slots (some
// ten instructions every 50 clocks) from the decode warps beside it.
__device__ __forceinline__ bool mbar_try_suspended(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
    return ok != 0;
}
// Bounded wait: false (and the CTA-wide error flag raised) when it gives up, after kSpinLimit polls or
// about 0.25 s of SM clock, whichever comes first; also false as soon as another thread has raised the flag.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *err) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_suspended(bar, parity)) return true;
        if (*err) return false;
        if ((i & 63) == 63 && clock64() - t0 > 500000000LL) break;
    }
    *err = JQ_ERR_TIMEOUT;
    return false;
}
// global -> shared bulk copy (16-byte aligned, a multiple of 16 bytes); its bytes are counted on the mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// 2-D tiled TMA load: box at (x bytes, y rows) of the tensor map -> shared memory; x must be a multiple of 16
__device__ __forceinline__ void tma_2d_g2s(uint32_t dst, const void *tmap, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar) : "memory");
}
// a hint: memory that will be read soon, into the L2 (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void l2_prefetch(const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// K-major operand in shared memory without swizzle: 8 rows x 16 bytes are contiguous; lbo = bytes between
// the two 16-byte K chunks of one MMA, sbo = bytes between 8-row groups (bits 46-47 = 1: sm_100 descriptor).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3fffu);
    d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}
// kind::f16 instruction descriptor: D = fp32, A = B = fp16, both K-major
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// One lane of a converged warp.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(p));
    return p;
}
// D[128 x N] (+)= A[128 x 16] (tensor memory) . B[N x 16]^T (shared memory), issued by the elected lane.  The whole warp
// runs the issuing loop and only the instruction itself is predicated: its operands have to be in uniform registers, and
// in a loop that one lane runs alone every one of them is moved there for every MMA (150 clocks per MMA).
__device__ __forceinline__ void mma_f16_ts(uint32_t elected, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile("{ .reg .pred p, q; setp.ne.b32 p, %4, 0; setp.ne.b32 q, %5, 0;\n"
                 "  @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t elected, uint32_t bar) {
    asm volatile("{ .reg .pred q; setp.ne.b32 q, %1, 0;\n"
                 "  @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0]; }" ::"r"(bar), "r"(elected) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t dp4a_u(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) { return __byte_perm(a, b, s); }
__device__ __forceinline__ uint32_t prmt_raw(uint32_t a, uint32_t b, uint32_t s) {   // selector nibbles with the sign-replicate bit
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}

// a row's 16 fp16 codebook entries as two 16-byte tables: low bytes, high bytes
struct Codebook {
    uint32_t lo[4], hi[4];
    __device__ __forceinline__ void set(const uint4 &a, const uint4 &b) {
        lo[0] = prmt(a.x, a.y, 0x6420); hi[0] = prmt(a.x, a.y, 0x7531);
        lo[1] = prmt(a.z, a.w, 0x6420); hi[1] = prmt(a.z, a.w, 0x7531);
        lo[2] = prmt(b.x, b.y, 0x6420); hi[2] = prmt(b.x, b.y, 0x7531);
        lo[3] = prmt(b.z, b.w, 0x6420); hi[3] = prmt(b.z, b.w, 0x7531);
    }
    // eight codes -> four fp16 pairs.  A permute looks four codes up in eight bytes, so each byte plane takes two
    // (entries 0-7 and 8-15) and a select by the codes' top bits.
    __device__ __forceinline__ void look_up8(uint32_t w, uint32_t (&v)[4]) const {
        const uint32_t low3 = w & 0x77777777u, wl = w << 4;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint32_t sel = half ? low3 >> 16 : low3;
            const uint32_t top = prmt_raw(w, wl, half ? 0xBFAEu : 0x9D8Cu);   // 0xff where the code is 8 or more
            const uint32_t l = (prmt_raw(lo[0], lo[1], sel) & ~top) | (prmt_raw(lo[2], lo[3], sel) & top);
            const uint32_t h = (prmt_raw(hi[0], hi[1], sel) & ~top) | (prmt_raw(hi[2], hi[3], sel) & top);
            v[2 * half] = prmt(l, h, 0x5140);
            v[2 * half + 1] = prmt(l, h, 0x7362);
        }
    }
};

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}
// (acc0, acc1) += (d0, d1) * s, both in fp32
__device__ __forceinline__ void fma2(float &acc0, float &acc1, uint32_t d0, uint32_t d1, float s) {
    asm("{ .reg .b64 a, d, s; mov.b64 a, {%0, %1}; mov.b64 d, {%2, %3}; mov.b64 s, {%4, %4};\n"
        "  fma.rn.f32x2 a, d, s, a; mov.b64 {%0, %1}, a; }"
        : "+f"(acc0), "+f"(acc1) : "r"(d0), "r"(d1), "f"(s));
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, uint32_t rank) {
    float v;
    asm volatile("{ .reg .b32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a]; }"
                 : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}

// Programmatic dependent launch: the main kernels are launched while the activation preparation in front of them
// is still running; everything they do before pdl_wait() (barrier set-up, problem look-ups, the first weight boxes)
// overlaps it, everything that reads the prepared activation comes after.  Without the launch attribute both are
// no-ops.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// e with amax * 2^-e below 2^15 after the rotation's worst-case growth (the rule of the GEMV kernels)
__device__ __forceinline__ int act_exponent(float amax, bool had) {
    uint32_t bits = __float_as_uint(amax);
    int field = (bits >> 23) & 0xff;
    if (field == 0xff || (bits & 0x7fffffffu) == 0) return 0;
    int e = field - 127 - (had ? 10 : 14);
    return max(-100, min(100, e));
}

}  // namespace jqta

// The driver's tensor-map encoder, looked up once (no link-time dependency on the driver library).
typedef CUresult (*ta_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static inline ta_encode_fn ta_encoder() {
    static ta_encode_fn fn = nullptr;
    static bool tried = false;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<ta_encode_fn>(p);
    }
    return fn;
}
