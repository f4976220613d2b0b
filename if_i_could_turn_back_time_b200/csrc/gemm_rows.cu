// Packed 4-bit weights x many activation rows (prompts, evaluation batches, convolutions) on the 5th-generation
// tensor cores (sm_100a): every weight is decoded once per 256 activation rows.
//
// A CTA computes a tile of 128 weight rows x NT <= 256 activation rows ("tokens"), D = W . X^T:
//   * warps 0-3 decode: thread = weight row = tensor-memory lane.  The packed codes of a warp's 32 rows arrive by TMA
//     (32-row x 128-byte boxes, 128-byte swizzle).  GF4 looks its codes up in the row's 16-entry codebook held in eight
//     registers (byte permutes), E2M1 converts with cvt.rn.f16x2.e2m1x2; the fp16 weights go to tensor memory
//     (tcgen05.st) as the A operand, one 128-code group per slot;
//   * warp 12 issues tcgen05.mma kind::f16 with the prepared activation in shared memory as the B operand, warp 13
//     streams that activation in 64-code stages (one bulk copy each; the preparation kernel lays it out per stage);
//   * warps 4-11 fold: the accumulator of every scale group (at most 128 codes) is read back with tcgen05.ld and added,
//     times the row's fp16 group scale, to fp32 sums in registers, so weights and scales stay exact (MODE 2, E2M1 in
//     32-code groups, multiplies the scale into the fp16 weight instead, as gemm_ta.cu does for the same shapes).
// Tensor memory: three accumulators of 128 columns in rotation + two operand slots of 64.
//
// What bounds it: at NT = 256 a 128-code group is 1024 clocks of tensor pipe; decoding it takes about 670 clocks of the
// ALU pipe (GF4, 21 operations per 8 codes) and the folding 256 issue slots per scheduler, both beside the MMAs.  Measured,
// the one decode warp of a scheduler is bound by the latency of its own chain, not by a pipe:
//   11008 x 4096 GF4, 2048 rows:  247 us, 749 TFLOP/s (passes of 16 rows took 2868); ALU 38 %, tensor 46 %, issue 40 % busy
//   8192 x 8192 E2M1, 777 rows:   149 us, 701 TFLOP/s (passes of 64 rows took 646);  ALU 14 %, tensor 51 %, issue 31 %
// Two decode warps per scheduler with tiles of 192 rows, which is what the registers allow, took 277 and 185 us.  A pair
// table in shared memory (as in gemm_ta.cu) would save ALU work, but its lookups, the 64 KB of activations per group that
// land in shared memory and the MMA's own reads together exceed the shared-memory bandwidth.
//
// A call with few tiles splits K over the CTAs of a cluster (up to 8); the partial sums meet through distributed
// shared memory and are added in rank order.
//
// Every mbarrier wait is bounded (see tc.cuh); the status word works as in gemm_ta.cu.
#include "tc.cuh"

namespace jqrows {

using namespace jqta;

constexpr int kTileM = 128;
constexpr int kThreads = 512;                       // warpgroups: decode, fold, fold, issue / load / allocate
constexpr int kWStage = 32 * 128;                   // bytes: 32 rows x 256 codes
constexpr int kSW = 3;                              // weight stages per decode warp
constexpr int kXRingBytes = 160 * 1024;
constexpr int kXMaxStages = 8;
constexpr int kMaxNT = 256;
constexpr int kD = 128, kDBufs = 3;                 // tensor-memory columns of an accumulator, accumulators
constexpr int kA0 = kD * kDBufs;                    // first column of the operand slots
constexpr int kBars = 4 * kSW + 2 + 2 + kDBufs * 2 + kXMaxStages * 2;
constexpr int kSmemBytes = kXRingBytes + 4 * kSW * kWStage + kBars * 8 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");
static_assert(kMaxNT * kTileM * 4 <= kXRingBytes, "the K-split exchange reuses the activation ring");

enum { kGf4 = 0, kE2m1 = 1, kE2m1Folded = 2 };

struct Args {
    const __half *scales;      // [N][lds] or null
    const __half *codebook;    // GF4: [N][16]
    const float *bias;         // or null
    void *y;
    const __half *xp;          // prepared activation [token tile][64-code stage][8 pieces][NT tokens][8 halves]
    const float *xscale;       // [tokens] 2^e
    int *status;
    int N, K, T;               // weight rows, codes, tokens
    int G;                     // 128-code groups, the last one zero-padded
    int g, lds, unit;          // codes per scale (0: none), scales per row, codes folded at once (128, 64 or 32)
    int NT, halves, HN;        // tokens per tile; MMAs per K slice (1: NT columns, 2: NT / 2 columns); columns per fold thread
    int rt, tiles, split;      // weight-row tiles, all tiles, CTAs that share a tile's K range
    int y_dtype;
};

template <class T> __device__ __forceinline__ T out_cast(float v);
template <> __device__ __forceinline__ float out_cast<float>(float v) { return v; }
template <> __device__ __forceinline__ __half out_cast<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 out_cast<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <class T>
__device__ __forceinline__ void store_tile(const Args &p, const float (&acc)[128], const float (&xs)[4], float bias, int n, int t0,
                                           int cols) {
    T *y = reinterpret_cast<T *>(p.y) + (size_t)t0 * p.N + n;
#pragma unroll
    for (int c = 0; c < 128; ++c) {
        const float x = __shfl_sync(0xffffffffu, xs[c >> 5], c & 31);
        if (c < cols && n < p.N) y[(size_t)c * p.N] = out_cast<T>(fmaf(acc[c], x, bias));
    }
}

template <int N> struct Slices { static constexpr int n = N; };

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1) gemm_rows_kernel(const __grid_constant__ Args p,
                                                                const __grid_constant__ CUtensorMap wmap) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), wg = warp >> 2;   // (uniform for the compiler)
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t xring = sbase, wring0 = sbase + kXRingBytes, bars = wring0 + 4 * kSW * kWStage;
    auto wbar = [&](int w, int s) { return bars + 8u * (w * kSW + s); };                      // weight box landed
    auto afull = [&](int s) { return bars + 8u * (4 * kSW + s); };                            // operand slot written
    auto afree = [&](int s) { return bars + 8u * (4 * kSW + 2 + s); };                        // its MMAs are done
    auto dfull = [&](int b) { return bars + 8u * (4 * kSW + 4 + b); };                        // accumulator complete
    auto dfree = [&](int b) { return bars + 8u * (4 * kSW + 4 + kDBufs + b); };               // accumulator folded
    auto xfull = [&](int s) { return bars + 8u * (4 * kSW + 4 + 2 * kDBufs + s); };           // activation stage landed
    auto xfree = [&](int s) { return bars + 8u * (4 * kSW + 4 + 2 * kDBufs + kXMaxStages + s); };
    volatile int *err = &s_err;
    const uint32_t xstage = (uint32_t)p.NT * 128;                                             // 64 codes x NT tokens
    const int nxs = min(kXMaxStages, kXRingBytes / (int)xstage);

    if (tid == 0) {
        s_err = 0;
        for (int w = 0; w < 4; ++w)
            for (int s = 0; s < kSW; ++s) mbar_init(wbar(w, s), 1);
        for (int s = 0; s < 2; ++s) { mbar_init(afull(s), 128); mbar_init(afree(s), 1); }
        for (int b = 0; b < kDBufs; ++b) { mbar_init(dfull(b), 1); mbar_init(dfree(b), p.halves == 2 ? 128 : 256); }
        for (int s = 0; s < kXMaxStages; ++s) { mbar_init(xfull(s), 1); mbar_init(xfree(s), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 14) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    // this CTA's tiles and its part of every tile's K range, in 256-code steps
    const int rank = p.split > 1 ? (int)(blockIdx.x % p.split) : 0;
    const int tile_lo = blockIdx.x / p.split, tile_stride = p.split > 1 ? p.tiles : (int)gridDim.x;
    const int steps = (p.G + 1) >> 1;
    const int s_lo = steps * rank / p.split, s_hi = steps * (rank + 1) / p.split;
    const int g_lo = 2 * s_lo, g_hi = min(2 * s_hi, p.G);

    if (wg == 0) {
        // =============================== decode ===============================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        const int q = warp;
        const uint32_t lane_t = tmem + ((uint32_t)(q * 32) << 16) + kA0;
        const uint32_t wring = wring0 + warp * (kSW * kWStage);
        const uint32_t lrow = lane * 128, lkey = (lane & 7) << 4;
        int i_tile = tile_lo, i_step = s_lo, i_stage = 0;
        auto issue = [&]() {
            if (i_tile < p.tiles) {
                if (lane == 0) {
                    const uint32_t bar = wbar(warp, i_stage);
                    mbar_expect_tx(bar, kWStage);
                    tma_2d_g2s(wring + i_stage * kWStage, &wmap, i_step * 128, (i_tile % p.rt) * kTileM + q * 32, bar);
                }
                if (++i_step == s_hi) { i_step = s_lo; i_tile += tile_stride; }
            }
            i_stage = (i_stage + 1 == kSW) ? 0 : i_stage + 1;
        };
#pragma unroll
        for (int s = 0; s < kSW; ++s) issue();

        uint4 cb0 = make_uint4(0, 0, 0, 0), cb1 = cb0;
        auto fetch_codebook = [&](int tile) {
            if (MODE == kGf4 && tile < p.tiles) {
                const int row = min((tile % p.rt) * kTileM + q * 32 + lane, p.N - 1);
                const uint4 *src = reinterpret_cast<const uint4 *>(p.codebook + (size_t)row * 16);
                cb0 = __ldg(src);
                cb1 = __ldg(src + 1);
            }
        };
        fetch_codebook(tile_lo);
        Codebook cb;
        int w_stage = 0;
        uint32_t w_par = 0, a_par = 0;
        int a_slot = 0, pend = -1;
        uint32_t handed = 0;
        auto hand_over = [&]() {
            if (pend >= 0) {
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(afull(pend));
                pend = -1;
            }
        };
        const int tail = p.K & 127;
        bool ok = true;
        for (int tile = tile_lo; tile < p.tiles && ok; tile += tile_stride) {
            if (MODE == kGf4) cb.set(cb0, cb1);
            fetch_codebook(tile + tile_stride);
            const int row = min((tile % p.rt) * kTileM + q * 32 + lane, p.N - 1);
            const uint4 *srow = reinterpret_cast<const uint4 *>(p.scales + (size_t)row * p.lds);   // folded: 8 scales per step
            uint4 sc_nxt = make_uint4(0, 0, 0, 0);
            if (MODE == kE2m1Folded) sc_nxt = __ldg(srow + s_lo);
            for (int step = s_lo; step < s_hi && ok; ++step) {
                ok = __all_sync(0xffffffffu, mbar_wait(wbar(warp, w_stage), w_par, err));
                if (!ok) break;
                const uint32_t slot = wring + w_stage * kWStage + lrow;
                if (++w_stage == kSW) { w_stage = 0; w_par ^= 1; }
                const uint4 sc = sc_nxt;
                if (MODE == kE2m1Folded && step + 1 < s_hi) sc_nxt = __ldg(srow + step + 1);
#pragma unroll
                for (int gi = 0; gi < 2; ++gi) {
                    const int g = 2 * step + gi;
                    if (g >= p.G) break;
                    uint4 w4[4];
#pragma unroll
                    for (int part = 0; part < 4; ++part) w4[part] = lds128(slot + (((gi * 4 + part) << 4) ^ lkey));
                    const uint32_t a_t = lane_t + a_slot * 64;
                    const int left = (tail && g == p.G - 1) ? tail : 128;
                    auto decode16 = [&](int part, uint32_t (&v)[16]) {
#pragma unroll
                        for (int wi = 0; wi < 4; ++wi) {
                            const uint32_t w = wi == 0 ? w4[part].x : (wi == 1 ? w4[part].y : (wi == 2 ? w4[part].z : w4[part].w));
                            uint32_t hh[4];
                            if constexpr (MODE == kGf4) {
                                cb.look_up8(w, hh);
                            } else {
                                asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4;\n"
                                    "  cvt.rn.f16x2.e2m1x2 %0, b0; cvt.rn.f16x2.e2m1x2 %1, b1;\n"
                                    "  cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
                                    : "=r"(hh[0]), "=r"(hh[1]), "=r"(hh[2]), "=r"(hh[3]) : "r"(w));
                            }
                            if constexpr (MODE == kE2m1Folded) {
                                const uint32_t pr = gi ? (part < 2 ? sc.z : sc.w) : (part < 2 ? sc.x : sc.y);
                                const uint32_t s2 = (part & 1) ? prmt(pr, pr, 0x3232) : prmt(pr, pr, 0x1010);
#pragma unroll
                                for (int bj = 0; bj < 4; ++bj)
                                    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(v[wi * 4 + bj]) : "r"(hh[bj]), "r"(s2));
                            } else {
#pragma unroll
                                for (int bj = 0; bj < 4; ++bj) v[wi * 4 + bj] = hh[bj];
                            }
                        }
                        if (MODE == kGf4 && left < 128) {   // codes past the row's end decode to zero, not to codebook[0]
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                const int k = part * 32 + 2 * i;
                                v[i] = k + 1 < left ? v[i] : (k < left ? v[i] & 0xffffu : 0u);
                            }
                        }
                    };
                    // the decode of the next 32 codes is issued before the previous 16 pairs are stored; a group is
                    // handed to the issuer only once the next group's first lookups are under way, but before the wait
                    // for that group's slot (with the wait in front, decoding and multiplying took turns)
                    uint32_t va[16], vb[16];
                    decode16(0, va);
                    decode16(1, vb);
                    hand_over();
                    if (handed >= 2) {      // the slot's previous group has been multiplied
                        ok = __all_sync(0xffffffffu, mbar_wait(afree(a_slot), a_par ^ 1, err));
                        if (!ok) break;
                        tc_fence_after();
                    }
                    tmem_st16(a_t, va);
                    decode16(2, va);
                    tmem_st16(a_t + 16, vb);
                    decode16(3, vb);
                    tmem_st16(a_t + 32, va);
                    tmem_st16(a_t + 48, vb);
                    pend = a_slot;
                    ++handed;
                    if (++a_slot == 2) { a_slot = 0; a_par ^= 1; }
                }
                if (!ok) break;
                __syncwarp();
                fence_async_smem();
                issue();
            }
            hand_over();
        }
        if (p.split > 1) { __syncwarp(); cluster_sync(); cluster_sync(); }
    } else if (wg < 3) {
        // =============================== fold ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
        const int h = wg - 1, r = tid & 127;
        const uint32_t lane_t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (p.halves == 2 ? 0 : h * p.HN);
        int buf = p.halves == 2 ? h : 0;
        uint32_t par = 0;
        float acc[128];
        // The prepared activation's row factors are read below: with plain loads, as the preparation kernel may still be
        // writing them while this one starts, and a read-only load (__ldg) need not stay behind the wait.
        pdl_wait();
        bool ok = true;
        for (int tile = tile_lo; tile < p.tiles; tile += tile_stride) {
            const int n = (tile % p.rt) * kTileM + r, tt = tile / p.rt;
            const int t0 = tt * p.NT + h * p.HN;
            const unsigned short *srow = reinterpret_cast<const unsigned short *>(p.scales) + (size_t)min(n, p.N - 1) * p.lds;
            const int k_lo = g_lo * 128, k_hi = g_hi * 128;
            auto scale_at = [&](int k) -> float {
                if (MODE == kE2m1Folded || p.g == 0) return 1.f;
                return k < p.K ? __half2float(__ushort_as_half(__ldg(srow + k / p.g))) : 0.f;
            };
#pragma unroll
            for (int c = 0; c < 128; ++c) acc[c] = 0.f;
            float s_nxt = scale_at(k_lo);
            for (int k = k_lo; k < k_hi && ok; k += p.unit) {
                const float s = s_nxt;
                if (k + p.unit < k_hi) s_nxt = scale_at(k + p.unit);
                ok = __all_sync(0xffffffffu, mbar_wait(dfull(buf), par, err));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 128; c += 32) {
                    if (c < p.HN) {
                        uint32_t d[32];
                        tmem_ld32(lane_t + buf * kD + c, d);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i += 2) fma2(acc[c + i], acc[c + i + 1], d[i], d[i + 1], s);
                    }
                }
                tc_fence_before();
                mbar_arrive(dfree(buf));
                buf += p.halves;
                if (buf >= kDBufs) { buf -= kDBufs; par ^= 1; }
            }
            const int cols = max(0, min(p.HN, p.T - t0));
            const float bias = (p.bias && n < p.N) ? __ldg(p.bias + n) : 0.f;
            if (p.split > 1) {
                // both fold warpgroups have seen their last accumulator: no MMA reads the activation ring any more
                asm volatile("bar.sync 1, 256;" ::: "memory");
                const uint32_t ex = xring + (uint32_t)(h * p.HN) * (kTileM * 4) + r * 4;
#pragma unroll
                for (int c = 0; c < 128; ++c)
                    if (c < p.HN) asm volatile("st.shared.f32 [%0], %1;" ::"r"(ex + c * (kTileM * 4)), "f"(acc[c]) : "memory");
                cluster_sync();
                const int c_lo = p.NT * rank / p.split, c_hi = p.NT * (rank + 1) / p.split;
                for (int c = c_lo + h; c < c_hi; c += 2) {
                    const int t = tt * p.NT + c;
                    if (t >= p.T) break;
                    float v = 0.f;
                    for (int k = 0; k < p.split; ++k) v += ld_cluster_f32(xring + (uint32_t)c * (kTileM * 4) + r * 4, k);
                    if (ok && n < p.N) jq::store_out(p.y, (size_t)t * p.N + n, fmaf(v, p.xscale[t], bias), p.y_dtype);
                }
                cluster_sync();
            } else if (ok) {
                float xs[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) xs[i] = (t0 + i * 32 + lane < p.T) ? p.xscale[t0 + i * 32 + lane] : 0.f;
                if (p.y_dtype == JQ_F32) store_tile<float>(p, acc, xs, bias, n, t0, cols);
                else if (p.y_dtype == JQ_F16) store_tile<__half>(p, acc, xs, bias, n, t0, cols);
                else store_tile<__nv_bfloat16>(p, acc, xs, bias, n, t0, cols);
            } else {
                break;
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == 12) {
            // =============================== MMA issuer ===============================
            // (the warp runs converged, see mma_f16_ts)
            const uint32_t elected = elect_one();
            auto wait = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)); };
            const int cols = p.halves == 2 ? p.HN : p.NT;
            const uint32_t idesc = idesc_f16(kTileM, cols);
            const uint32_t lbo = (uint32_t)p.NT * 16;
            const uint32_t kstep = (2 * lbo) >> 4;             // descriptor address units per K = 16 slice
            // Only the address field of a descriptor changes, by constants, and the slices of a fold are unrolled (forming
            // a descriptor per MMA in a loop took 340 clocks per MMA; 2048 rows: 583 us).
            const uint64_t desc0 = smem_desc(xring, lbo, 128);
            const uint32_t stage_units = xstage >> 4, half_units = (uint32_t)p.HN;
            int a_slot = 0, buf = 0, xs = 0;
            uint32_t a_par = 0, d_par = 1, x_par = 0;          // (the first wait on a free accumulator passes at once)
            bool ok = true;
            for (int tile = tile_lo; tile < p.tiles && ok; tile += tile_stride)
                for (int g = g_lo; g < g_hi && ok; ++g) {
                    if (!(ok = wait(afull(a_slot), a_par))) break;
                    const int xs0 = xs;
                    const uint32_t par0 = x_par;
                    if (++xs == nxs) { xs = 0; x_par ^= 1; }
                    const int xs1 = xs;
                    const uint32_t par1 = x_par;
                    if (++xs == nxs) { xs = 0; x_par ^= 1; }
                    if (!(ok = wait(xfull(xs0), par0))) break;
                    tc_fence_after();
                    const uint32_t a_t = tmem + kA0 + a_slot * 64;
                    const uint64_t lo = desc0 + xs0 * stage_units, hi = desc0 + xs1 * stage_units;
                    auto fold_unit = [&](auto slices, int i0, uint64_t d0, uint64_t d1) -> bool {   // d0, d1: slices 0-3, 4-7 of the group
                        if (!wait(dfree(buf), d_par)) return false;
                        tc_fence_after();
                        const uint32_t d_t = tmem + buf * kD;
#pragma unroll
                        for (int i = 0; i < decltype(slices)::n; ++i)
                            mma_f16_ts(elected, d_t, a_t + 8 * (i0 + i), (i < 4 ? d0 : d1) + (uint64_t)((i & 3) * kstep), idesc, i > 0);
                        mma_commit(elected, dfull(buf));
                        if (++buf == kDBufs) { buf = 0; d_par ^= 1; }
                        return true;
                    };
                    if (p.unit == 128) {
                        if (!(ok = wait(xfull(xs1), par1))) break;
                        for (int h = 0; h < p.halves && ok; ++h) ok = fold_unit(Slices<8>{}, 0, lo + h * half_units, hi + h * half_units);
                    } else if (p.unit == 64) {
                        for (int h = 0; h < p.halves && ok; ++h) ok = fold_unit(Slices<4>{}, 0, lo + h * half_units, 0);
                        if (!ok || !(ok = wait(xfull(xs1), par1))) break;
                        for (int h = 0; h < p.halves && ok; ++h) ok = fold_unit(Slices<4>{}, 4, hi + h * half_units, 0);
                    } else {
                        if (!(ok = wait(xfull(xs1), par1))) break;
                        for (int i0 = 0; i0 < 8 && ok; i0 += 2)
                            for (int h = 0; h < p.halves && ok; ++h)
                                ok = fold_unit(Slices<2>{}, i0, (i0 < 4 ? lo : hi) + h * half_units + (uint64_t)((i0 & 3) * kstep), 0);
                    }
                    if (!ok) break;
                    mma_commit(elected, xfree(xs0));
                    mma_commit(elected, xfree(xs1));
                    mma_commit(elected, afree(a_slot));
                    if (++a_slot == 2) { a_slot = 0; a_par ^= 1; }
                }
        } else if (warp == 13 && lane == 0) {
            // =============================== activation loader ===============================
            pdl_wait();
            int s = 0;
            uint32_t par = 1;                                  // (the first round finds every stage free)
            bool ok = true;
            for (int tile = tile_lo; tile < p.tiles && ok; tile += tile_stride) {
                const unsigned char *src = reinterpret_cast<const unsigned char *>(p.xp) +
                                           ((size_t)(tile / p.rt) * (2 * p.G) + 2 * g_lo) * xstage;
                for (int i = 2 * g_lo; i < 2 * g_hi; ++i, src += xstage) {
                    if (!(ok = mbar_wait(xfree(s), par, err))) break;
                    mbar_expect_tx(xfull(s), xstage);
                    bulk_g2s(xring + s * xstage, src, xstage, xfull(s));
                    if (++s == nxs) { s = 0; par ^= 1; }
                }
            }
        }
        if (p.split > 1) { __syncwarp(); cluster_sync(); cluster_sync(); }
    }

    // ---- teardown
    if (*err) {   // a wait gave up: let the copies still in flight land before the CTA's shared memory goes away
        for (int i = 0; i < 400; ++i) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_err) atomicExch(p.status, s_err);
    if (warp == 14) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---- activation preparation ---------------------------------------------------------
struct PrepArgs {
    const void *x;
    __half *xp;
    float *xscale;
    int T, K, G, NT, had, x_dtype;
    int vec;                   // rows and base allow loads of four elements
};

__device__ __forceinline__ size_t xp_offset(int t, int piece, int G, int NT) {   // in halves
    const int tt = t / NT, r = t - tt * NT;
    return (((size_t)tt * 2 * G + (piece >> 3)) * 8 + (piece & 7)) * NT * 8 + (size_t)r * 8;
}
__device__ __forceinline__ float4 load4(const PrepArgs &p, size_t row, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.vec && k + 4 <= p.K) {
        const size_t i = row * p.K + k;
        if (p.x_dtype == JQ_F32) return *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.x) + i);
        const uint2 u = *reinterpret_cast<const uint2 *>(reinterpret_cast<const unsigned short *>(p.x) + i);
        if (p.x_dtype == JQ_F16) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
            return make_float4(a.x, a.y, b.x, b.y);
        }
        return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                           __uint_as_float(u.y & 0xffff0000u));
    }
    float *e = &v.x;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (k + j < p.K) e[j] = jq::load_act(p.x, row * p.K + k + j, p.x_dtype);
    return v;
}

// One block per two tokens: max|x| -> power of two -> x 2^-e -> block Hadamard -> fp16, in the layout that the main
// kernel copies stage by stage.  A lane holds four codes of both tokens; neighbours swap halves so that every lane
// stores one 16-byte piece and a pair of lanes a full 32-byte sector.
__global__ void __launch_bounds__(256) rows_prepare_kernel(const __grid_constant__ PrepArgs p) {
    __shared__ float red[2][8];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * 2;
    const bool two = t0 + 1 < p.T;
    float m[2] = {0.f, 0.f};
    for (int k = threadIdx.x * 4; k < p.K; k += 1024) {
        const float4 a = load4(p, t0, k);
        m[0] = fmaxf(fmaxf(m[0], fmaxf(fabsf(a.x), fabsf(a.y))), fmaxf(fabsf(a.z), fabsf(a.w)));
        if (two) {
            const float4 b = load4(p, t0 + 1, k);
            m[1] = fmaxf(fmaxf(m[1], fmaxf(fabsf(b.x), fabsf(b.y))), fmaxf(fabsf(b.z), fabsf(b.w)));
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
        if (lane == 0) red[j][warp] = m[j];
    }
    __syncthreads();
    float down[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float mm = red[j][0];
#pragma unroll
        for (int w = 1; w < 8; ++w) mm = fmaxf(mm, red[j][w]);
        const int e = act_exponent(mm, p.had != 0);
        down[j] = __uint_as_float((uint32_t)(127 - e) << 23);
        if (threadIdx.x == j && t0 + j < p.T) p.xscale[t0 + j] = __uint_as_float((uint32_t)(127 + e) << 23);
    }
    for (int blk = warp; blk < p.G; blk += 8) {
        const int k0 = blk * 128 + lane * 4;
        uint32_t u[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (j == 0 || two) {
                const float4 a = load4(p, t0 + j, k0);
                v[0] = a.x * down[j]; v[1] = a.y * down[j]; v[2] = a.z * down[j]; v[3] = a.w * down[j];
            }
            if (p.had) jq::fwht128_warp(v, lane);
            const __half2 h01 = __floats2half2_rn(v[0], v[1]), h23 = __floats2half2_rn(v[2], v[3]);
            u[j][0] = *reinterpret_cast<const uint32_t *>(&h01);
            u[j][1] = *reinterpret_cast<const uint32_t *>(&h23);
        }
        const bool odd = lane & 1;
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, odd ? u[0][0] : u[1][0], 1);
        const uint32_t r1 = __shfl_xor_sync(0xffffffffu, odd ? u[0][1] : u[1][1], 1);
        const uint4 out = odd ? make_uint4(r0, r1, u[1][0], u[1][1]) : make_uint4(u[0][0], u[0][1], r0, r1);
        if (!odd || two) *reinterpret_cast<uint4 *>(p.xp + xp_offset(t0 + odd, blk * 16 + (lane >> 1), p.G, p.NT)) = out;
    }
}

// Convolution: the receptive fields are gathered straight from the image into the same layout (no unfolded copy).
// lane = output position, so loads of one tap and stores of one 8-code piece are consecutive over the warp.  Bound by the
// instructions between the loads, so a block that can keep its 32 fields in shared memory (96 KB: K up to 768) gathers once;
// longer ones gather again for the second pass.  64 -> 128 channels, 3x3, 16 images of 32 x 32, the whole call: 56 us gathering
// twice, 40 us gathering once, 30 us with addresses formed by additions; loading from a valid place under every condition, so
// that the loads need not wait for one another, was slower (44 us).  Time grows with K, not with the positions, until the
// blocks fill the chip, so few blocks have more warps: 128 -> 128 channels, 3x3, 8 images of 14 x 14 (49 blocks): 49 us before,
// 32 with 8 warps a block, 26 with 32.
constexpr int kFieldBytes = 96 * 1024;
struct ConvArgs {
    const void *x;             // element (b, c, h, w) at b sb + c sc + h sr + w sx
    __half *xp;
    float *xscale;
    int T, K, G, NT, x_dtype;
    int C, H, W, kh, kw, sh, sw, ph, pw, dh, dw, wo, L;
    long long sb, sc, sr, sx;
    int keep;                  // the block's fields fit in shared memory
};

template <class T, int kWarps>
__global__ void __launch_bounds__(kWarps * 32) conv_prepare_kernel(const __grid_constant__ ConvArgs p) {
    __shared__ float red[kWarps][32];
    extern __shared__ __align__(16) float fields[];    // [pieces * 8][32], or empty
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // (uniform for the compiler: so is the walk over the taps)
    const int t = blockIdx.x * 32 + lane;
    const bool live = t < p.T;
    const int b = live ? t / p.L : 0, l = live ? t - b * p.L : 0;
    const int y0 = (l / p.wo) * p.sh - p.ph, x0 = (l % p.wo) * p.sw - p.pw;
    const T *const at0 = reinterpret_cast<const T *>(p.x) + (b * p.sb + y0 * p.sr + x0 * p.sx);   // (not read from there where out of range)
    const int taps = p.kh * p.kw;
    const int pieces = p.G * 16;
    // Walk of one piece's eight codes: k -> (channel, tap row, tap column).  Position and address go along by additions (three
    // products of 64 bits per code were most of this kernel's time).
    const long long to_x = p.dw * p.sx, to_y = p.dh * p.sr - p.kw * to_x, to_c = p.sc - p.kh * (p.dh * p.sr);
    const int back_x = p.kw * p.dw, back_y = p.kh * p.dh;
    auto gather = [&](int piece, float (&v)[8]) {
        const int k = piece * 8, c = k / taps, r = k - c * taps;
        int ky = r / p.kw, kx = r - ky * p.kw;
        int yy = y0 + ky * p.dh, xx = x0 + kx * p.dw;
        const T *at = at0 + (c * p.sc + (long long)(ky * p.dh) * p.sr + (long long)(kx * p.dw) * p.sx);
        const int left = live ? p.K - k : 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = (e < left && (unsigned)yy < (unsigned)p.H && (unsigned)xx < (unsigned)p.W) ? (float)*at : 0.f;
            at += to_x;
            xx += p.dw;
            if (++kx == p.kw) {
                kx = 0;
                xx -= back_x;
                yy += p.dh;
                at += to_y;
                if (++ky == p.kh) { ky = 0; yy -= back_y; at += to_c; }
            }
        }
    };
    float m = 0.f;
    for (int piece = warp; piece * 8 < p.K; piece += kWarps) {
        float v[8];
        gather(piece, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            m = fmaxf(m, fabsf(v[e]));
            if (p.keep) fields[(piece * 8 + e) * 32 + lane] = v[e];     // read back by the same thread
        }
    }
    red[warp][lane] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, red[w][lane]);
    const int ex = act_exponent(m, false);
    const float down = __uint_as_float((uint32_t)(127 - ex) << 23);
    if (warp == 0 && live) p.xscale[t] = __uint_as_float((uint32_t)(127 + ex) << 23);
    for (int piece = warp; piece < pieces; piece += kWarps) {
        float v[8];
        if (p.keep) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = piece * 8 < p.K ? fields[(piece * 8 + e) * 32 + lane] : 0.f;
        } else {
            gather(piece, v);
        }
        uint32_t u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __half2 h = __floats2half2_rn(v[2 * e] * down, v[2 * e + 1] * down);
            u[e] = *reinterpret_cast<const uint32_t *>(&h);
        }
        if (live) *reinterpret_cast<uint4 *>(p.xp + xp_offset(t, piece, p.G, p.NT)) = make_uint4(u[0], u[1], u[2], u[3]);
    }
}

// ---- host side -------------------------------------------------------------------------
struct Shape { int NT, halves, HN, ntt, split; };

// Tokens per tile and CTAs per tile, by a cost in SM clocks: a wave of tiles costs its 128-code groups (the slowest of
// multiplying, decoding and folding) plus a fixed part (first stage's latency, outputs; with a K split also the exchange).
static Shape search_shape(int mode, int N, int T, int G, int unit, int sms) {
    const int rt = (N + kTileM - 1) / kTileM, steps = (G + 1) / 2;
    const double decode = mode == kGf4 ? 700 : 450;
    Shape best{};
    double best_cost = 0;
    const int ntt0 = (T + kMaxNT - 1) / kMaxNT;
    for (int ntt = ntt0; ntt <= ntt0 * 2 + 6; ++ntt) {
        const int need = (T + ntt - 1) / ntt;
        const int NT = (need + 31) / 32 * 32;
        if (ntt > ntt0 && NT * (ntt - 1) >= T) continue;      // the last tile would be empty
        const int halves = NT > 128 ? 2 : 1, HN = NT / 2;
        const double mma = 8.0 * halves * (NT / halves / 2 > 50 ? NT / halves / 2 : 50);
        const double fold = (128.0 / unit) * (200 + 1.5 * HN);
        double group = mma > decode ? mma : decode;
        if (fold > group) group = fold;
        for (int s = 1; s <= 8; s *= 2) {
            if (s > steps) break;
            const long long ctas = (long long)rt * ntt * s;
            const int cap = s == 8 ? sms / 9 / 2 * 16 : (s == 4 ? sms / 18 * 16 : sms);
            const double waves = (double)((ctas + cap - 1) / (cap > 0 ? cap : 1));
            const double cost = waves * (((steps + s - 1) / s) * 2 * group + 3000 + 4.0 * HN + (s > 1 ? 2500 + 8.0 * NT : 0));
            if (best.NT == 0 || cost < best_cost) {
                best = Shape{NT, halves, HN, ntt, s};
                best_cost = cost;
            }
        }
    }
    return best;
}

// The search takes some microseconds, three times per call (the scratch of both forms, and the launch): a thread keeps its
// last answers.
static Shape choose_shape(int mode, int N, int T, int G, int unit, int sms) {
    struct Entry { int mode, N, T, G, unit, sms; Shape shape; };
    constexpr unsigned kEntries = 64;
    static thread_local Entry kept[kEntries] = {};
    unsigned h = (unsigned)N * 0x9E3779B1u ^ (unsigned)T * 0x85EBCA77u ^ (unsigned)G * 0xC2B2AE3Du ^ (unsigned)(mode * 1024 + unit) * 0x27D4EB2Fu;
    Entry &e = kept[(h >> 16) % kEntries];
    if (e.N != N || e.T != T || e.G != G || e.mode != mode || e.unit != unit || e.sms != sms)
        e = Entry{mode, N, T, G, unit, sms, search_shape(mode, N, T, G, unit, sms)};
    return e.shape;
}

static int fold_unit(int g) { return (g == 0 || g % 128 == 0) ? 128 : (g % 64 == 0 ? 64 : 32); }

// E2M1 in 32-code groups whose scales can be read in 16-byte pieces: the shapes for which gemm_ta.cu folds scales too
static int pick_mode(int fmt, int K, int g, const void *scales) {
    if (fmt == JQ_FMT_GF4) return kGf4;
    return (g == 32 && K % 256 == 0 && K >= 512 && jq_aligned16(scales)) ? kE2m1Folded : kE2m1;
}

static size_t scale_bytes(int tokens) { return ((size_t)tokens * 4 + 255) / 256 * 256; }

static size_t scratch_bytes(const Shape &s, int G) {
    return scale_bytes(s.ntt * s.NT) + (size_t)s.ntt * s.NT * G * 256;
}

static int launch(int fmt, const void *qw, const void *scales, const void *codebook, const float *bias, void *y, int N, int K,
                  int T, int g, int y_dtype, void *scratch, size_t scratch_size, int *status, cudaStream_t st,
                  PrepArgs *lin, ConvArgs *conv) {
    if (!qw || !y || !scratch || !status) return JQ_ERR_NULL_PTR;
    if (fmt != JQ_FMT_GF4 && fmt != JQ_FMT_E2M1) return JQ_ERR_UNSUPPORTED;
    if (fmt == JQ_FMT_GF4 && !codebook) return JQ_ERR_NULL_PTR;
    if (N <= 0 || K <= 0 || T <= 0 || g < 0 || (g && (g % 32 || K % g)) || (fmt == JQ_FMT_E2M1 && g == 0)) return JQ_ERR_BAD_SHAPE;
    if (g && !scales) return JQ_ERR_NULL_PTR;
    if (y_dtype < 0 || y_dtype > 2) return JQ_ERR_BAD_DTYPE;
    if (!jq_aligned16(qw) || (fmt == JQ_FMT_GF4 && !jq_aligned16(codebook)) || (g && (reinterpret_cast<uintptr_t>(scales) & 1u)) ||
        (reinterpret_cast<uintptr_t>(scratch) & 255u))
        return JQ_ERR_BAD_ALIGN;
    const int G = (K + 127) / 128, sms = jq_sm_count();
    const int mode = pick_mode(fmt, K, g, scales);
    const int unit = mode == kE2m1Folded ? 128 : fold_unit(g);
    const Shape s = choose_shape(mode, N, T, G, unit, sms);
    if (scratch_size < scratch_bytes(s, G)) return JQ_ERR_WORKSPACE;
    Args a{};
    a.scales = reinterpret_cast<const __half *>(scales);
    a.codebook = reinterpret_cast<const __half *>(codebook);
    a.bias = bias;
    a.y = y;
    float *xscale = reinterpret_cast<float *>(scratch);
    __half *xp = reinterpret_cast<__half *>(reinterpret_cast<unsigned char *>(scratch) + scale_bytes(s.ntt * s.NT));
    a.xp = xp;
    a.xscale = xscale;
    a.status = status;
    a.N = N; a.K = K; a.T = T; a.G = G; a.g = g; a.lds = g ? K / g : 0; a.unit = unit;
    a.NT = s.NT; a.halves = s.halves; a.HN = s.HN; a.rt = (N + kTileM - 1) / kTileM;
    a.tiles = a.rt * s.ntt; a.split = s.split; a.y_dtype = y_dtype;

    // tensor map over the packed rows: boxes of 32 rows x 128 bytes, 128-byte swizzle; outside reads as zeros
    ta_encode_fn enc = ta_encoder();
    if (!enc) return JQ_ERR_UNSUPPORTED;
    CUtensorMap map;
    const cuuint64_t ldw = (cuuint64_t)(jq_row_stride_codes(K) >> 1);
    const cuuint64_t dims[2] = {ldw, (cuuint64_t)N};
    const cuuint64_t strides[1] = {ldw};
    const cuuint32_t box[2] = {128, 32}, estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(qw), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return JQ_ERR_CUDA_BASE - (int)cudaErrorInvalidValue;

    auto kern = mode == kGf4 ? gemm_rows_kernel<kGf4> : (mode == kE2m1 ? gemm_rows_kernel<kE2m1> : gemm_rows_kernel<kE2m1Folded>);
    static jq_contexts done[3], conv_done[9];
    JQ_CUDA_TRY(jq_allow_smem(reinterpret_cast<const void *>(kern), kSmemBytes, done[mode]));
    if (lin) {
        lin->xp = xp; lin->xscale = xscale; lin->G = G; lin->NT = s.NT;
        rows_prepare_kernel<<<(T + 1) / 2, 256, 0, st>>>(*lin);
    } else {
        conv->xp = xp; conv->xscale = xscale; conv->G = G; conv->NT = s.NT;
        const int bytes = (K + 7) / 8 * 8 * 32 * (int)sizeof(float);
        conv->keep = K <= kFieldBytes / 128 && bytes <= kFieldBytes;
        // A block's time is its warps' walks along 32 fields: with few blocks, more warps share them
        const int blocks = (T + 31) / 32, more = blocks <= sms ? 2 : (blocks <= 2 * sms ? 1 : 0);
        void (*const kernels[3][3])(const ConvArgs) = {
            {conv_prepare_kernel<float, 8>, conv_prepare_kernel<float, 16>, conv_prepare_kernel<float, 32>},
            {conv_prepare_kernel<__half, 8>, conv_prepare_kernel<__half, 16>, conv_prepare_kernel<__half, 32>},
            {conv_prepare_kernel<__nv_bfloat16, 8>, conv_prepare_kernel<__nv_bfloat16, 16>, conv_prepare_kernel<__nv_bfloat16, 32>}};
        auto gather = kernels[conv->x_dtype][more];
        if (conv->keep) JQ_CUDA_TRY(jq_allow_smem(reinterpret_cast<const void *>(gather), kFieldBytes, conv_done[conv->x_dtype * 3 + more]));
        gather<<<blocks, 256 << more, conv->keep ? bytes : 0, st>>>(*conv);
    }
    int rc = jq_launch_status();
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)s.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3(s.split > 1 ? a.tiles * s.split : (a.tiles < sms ? a.tiles : sms));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = s.split > 1 ? 2 : 1;
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a, map));
    return jq_launch_status();
}

}  // namespace jqrows

using namespace jqrows;

extern "C" size_t jq_gemm_rows_scratch_bytes(int fmt, int N, int K, int B, int g) {
    if (N <= 0 || K <= 0 || B <= 0 || g < 0) return 0;
    const int G = (K + 127) / 128;
    // the shape depends on whether the scales allow the folded kernel: room for either
    size_t most = 0;
    for (int folded = 0; folded < 2; ++folded) {
        const int mode = fmt == JQ_FMT_GF4 ? kGf4 : (folded ? kE2m1Folded : kE2m1);
        const size_t b = scratch_bytes(choose_shape(mode, N, B, G, mode == kE2m1Folded ? 128 : fold_unit(g), jq_sm_count()), G);
        if (b > most) most = b;
    }
    return most;
}

extern "C" int jq_gemm_rows(int fmt, const void *qweight, const void *scales, const void *codebook, const void *x,
                            const float *bias, void *y, int N, int K, int B, int g, int had_block, int x_dtype, int y_dtype,
                            void *scratch, size_t scratch_size, int *status, jq_stream_t stream) {
    if (!x) return JQ_ERR_NULL_PTR;
    if (x_dtype < 0 || x_dtype > 2) return JQ_ERR_BAD_DTYPE;
    if (had_block != 0 && (had_block != 128 || K % 128)) return JQ_ERR_BAD_SHAPE;
    PrepArgs prep{};
    prep.x = x; prep.T = B; prep.K = K; prep.had = had_block; prep.x_dtype = x_dtype;
    const int esz = x_dtype == JQ_F32 ? 4 : 2;
    prep.vec = K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & (4 * esz - 1)) == 0;
    return launch(fmt, qweight, scales, codebook, bias, y, N, K, B, g, y_dtype, scratch, scratch_size, status,
                  reinterpret_cast<cudaStream_t>(stream), &prep, nullptr);
}

extern "C" int jq_conv_rows(int fmt, const void *qweight, const void *scales, const void *codebook, const void *x,
                            const float *bias, void *y, const jq_conv *c, int O, int K, int rows, int g, int x_dtype, int y_dtype,
                            void *scratch, size_t scratch_size, int *status, jq_stream_t stream) {
    if (!x || !c) return JQ_ERR_NULL_PTR;
    if (x_dtype < 0 || x_dtype > 2) return JQ_ERR_BAD_DTYPE;
    if (c->batch <= 0 || c->channels <= 0 || c->height <= 0 || c->width <= 0 || c->kernel_h <= 0 || c->kernel_w <= 0 ||
        c->stride_h <= 0 || c->stride_w <= 0 || c->pad_h < 0 || c->pad_w < 0 || c->dilation_h <= 0 || c->dilation_w <= 0)
        return JQ_ERR_BAD_SHAPE;
    const long long ho = ((long long)c->height + 2 * c->pad_h - (long long)c->dilation_h * (c->kernel_h - 1) - 1) / c->stride_h + 1;
    const long long wo = ((long long)c->width + 2 * c->pad_w - (long long)c->dilation_w * (c->kernel_w - 1) - 1) / c->stride_w + 1;
    const long long most = 0x3fffffff, taps = (long long)c->kernel_h * c->kernel_w;
    if (ho <= 0 || wo <= 0 || ho > most || wo > most || ho * wo > most || taps > most || rows > most) return JQ_ERR_BAD_SHAPE;
    // the weights' row stride and scales per row follow from K, the extent of y from rows
    if (ho * wo * c->batch != rows || taps * c->channels != K) return JQ_ERR_BAD_SHAPE;
    ConvArgs a{};
    a.x = x; a.T = rows; a.K = K; a.x_dtype = x_dtype;
    a.C = c->channels; a.H = c->height; a.W = c->width; a.kh = c->kernel_h; a.kw = c->kernel_w;
    a.sh = c->stride_h; a.sw = c->stride_w; a.ph = c->pad_h; a.pw = c->pad_w; a.dh = c->dilation_h; a.dw = c->dilation_w;
    a.wo = (int)wo; a.L = (int)(ho * wo);
    a.sb = c->stride_x[0]; a.sc = c->stride_x[1]; a.sr = c->stride_x[2]; a.sx = c->stride_x[3];
    return launch(fmt, qweight, scales, codebook, bias, y, O, K, rows, g, y_dtype, scratch, scratch_size, status,
                  reinterpret_cast<cudaStream_t>(stream), nullptr, &a);
}
