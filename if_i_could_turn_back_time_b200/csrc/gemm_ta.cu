// Packed 4-bit weights x activations on the 5th-generation tensor cores with
// the decoded weights handed over in tensor memory (tcgen05, sm_100a).
//
// Three kernels, by the rows of the activation: gf4_lut2_kernel (GF4, one row, on
// the CUDA cores: further below), gemm_ta_kernel (up to 16 rows) and
// wide::gemm_ta_wide_kernel (17 to 64 rows).  What the last two share:
//
// One persistent CTA per SM works through 128-row tiles of the weight matrices.
// A decode thread owns one weight row of the tile (= one tensor-memory lane)
// and every fourth 128-code group of that row (from 17 rows on: every other
// 256-code step):
//   * the packed codes of the tile arrive by TMA (cp.async.bulk.tensor, one
//     128-row x 128-byte box per 256 codes, from 17 rows on a 32-row box per
//     warp, with the 128-byte swizzle, completion counted on an mbarrier), so
//     that every lane reads its own row without bank conflicts;
//   * GF4: a byte (two codes) indexes the row's 256-entry table of fp16 pairs,
//     built once per tile in a shared-memory column that only this lane's bank
//     serves (one conflict-free 32-bit lookup per two codes, the address formed
//     by one dp4a); above 16 rows the row's codebook in registers, through byte
//     permutes; E2M1: cvt.rn.f16x2.e2m1x2 per byte, times the group's fp16
//     scale in fp16x2;
//   * the fp16 values go to tensor memory with tcgen05.st as the A operand
//     (M = 128 rows, K = 16 per instruction) of tcgen05.mma kind::f16; the B
//     operand is the prepared activation (rotated, normalised by a power of
//     two, fp16, in the K-major core-matrix layout), streamed from global
//     memory, one 128-code chunk per bulk copy;
//   * every 128-code group has an fp32 accumulator in tensor memory; fold
//     threads read it back with tcgen05.ld and, for GF4, apply the group's fp16
//     scale in fp32, so every product and every scale stays exact (the results
//     differ from the FMA kernels only in summation order).  E2M1 folds its
//     scales into the fp16 weights (one rounding per weight).
// The multiply-accumulate work thus costs the CUDA cores nothing, whatever the
// batch (up to 64 columns per pass), and up to 16 rows the lookups are halved.
//
// Every wait on an mbarrier is bounded: on expiry the CTA raises a status word
// in the workspace, all roles leave their loops, tensor memory is freed and
// the kernel returns.  Nothing traps or spins without a limit.
#include "tc.cuh"
#include <string.h>

namespace jqta {

constexpr int kTileM = 128;
constexpr int kWStage = kTileM * 128;        // bytes of a weight stage: 128 rows x 128 bytes (256 codes), swizzled by TMA
constexpr int kTabBytes = 4 * 256 * 128;     // GF4, up to 16 rows: 256 entries x 32 lanes x 4 bytes per 32-row quarter
constexpr int kHeaderBytes = 1024;           // workspace: int status

struct TaProblem {
    const uint8_t *qw;
    const __half *scales;
    const __half *codebook;
    const void *x;          // activations [B, K] as the caller gave them
    const float *bias;
    void *y;
    __half *xprep;          // prepared activation: [K / 8][B rows][8 halves]
    float *xscale;          // [B] 2^e of each batch row (the power of two taken out before rounding to fp16)
    int N, K, g, had;
    int ldw;                // bytes between packed rows
    int lds;                // scales between rows
    int ldy;                // outputs between batch rows
    int tile0;              // first tile of this problem in the launch's tile sequence
};

struct PeerInfo {
    int n;
    long long delta[8];
};

// ---- activation preparation -----------------------------------------------------
// One block per (problem, batch row): x -> (x 2^-e) -> block Hadamard -> fp16, written as
// [8-code piece][batch row][8 halves].  Copied to shared memory as it is, this is the K-major operand
// layout of the MMA with a piece stride of 16 B bytes: row n of piece c sits at (c B + n) 16 bytes.  The MMA
// reads 16, 32 or 64 rows; rows >= B are whatever follows (the next pieces), and their accumulator columns
// are never read.
// A thread has the same four elements of every 128 kWarps in both passes (maximum; rotation) and keeps what it has loaded, up
// to kKeep times four.  The pass is a chain of load -> rotate -> store per warp, and its latency is what a call waits for before
// the main kernel can start: few blocks (a single call, a decode step of one row) have 32 warps each; with many, 8 warps per
// block keep more rows resident per SM.
template <class T> __device__ __forceinline__ float4 load_four(const T *x, bool vec);
template <> __device__ __forceinline__ float4 load_four<float>(const float *x, bool vec) {
    return vec ? *reinterpret_cast<const float4 *>(x) : make_float4(x[0], x[1], x[2], x[3]);
}
template <> __device__ __forceinline__ float4 load_four<__half>(const __half *x, bool vec) {
    if (!vec) return make_float4(__half2float(x[0]), __half2float(x[1]), __half2float(x[2]), __half2float(x[3]));
    const uint2 u = *reinterpret_cast<const uint2 *>(x);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
template <> __device__ __forceinline__ float4 load_four<__nv_bfloat16>(const __nv_bfloat16 *x, bool vec) {
    if (!vec) return make_float4(__bfloat162float(x[0]), __bfloat162float(x[1]), __bfloat162float(x[2]), __bfloat162float(x[3]));
    const uint2 u = *reinterpret_cast<const uint2 *>(x);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}
template <int kPrepThreads, class T>
__global__ void __launch_bounds__(kPrepThreads) ta_prepare_kernel(const TaProblem *probs, TaProblem single, int B) {
    constexpr int kWarps = kPrepThreads / 32, kKeep = 4;
    __shared__ float sred[kWarps];
    __shared__ int sexp;
    pdl_launch_dependents();
    const int pi = blockIdx.x / B, b = blockIdx.x % B;
    const TaProblem p = probs ? probs[pi] : single;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const T *const x = reinterpret_cast<const T *>(p.x) + (size_t)b * p.K;       // (K is a multiple of 256)
    const bool vec = ((size_t)p.x & (4 * sizeof(T) - 1)) == 0;
    float4 kept[kKeep];
    float m = 0.f;
    auto largest = [&](const float4 &q) { m = fmaxf(m, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w)))); };
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
        const int k = (tid + i * kPrepThreads) * 4;
        kept[i] = k < p.K ? load_four(x + k, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < kKeep; ++i) largest(kept[i]);
    for (int k = (tid + kKeep * kPrepThreads) * 4; k < p.K; k += kPrepThreads * 4) largest(load_four(x + k, vec));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) sred[warp] = m;
    __syncthreads();
    if (warp == 0) {
        float mm = lane < kWarps ? sred[lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
        if (lane == 0) {
            sexp = act_exponent(mm, p.had != 0);
            p.xscale[b] = __uint_as_float((uint32_t)(127 + sexp) << 23);
        }
    }
    __syncthreads();
    const float down = __uint_as_float((uint32_t)(127 - sexp) << 23);
    auto finish = [&](int blk, const float4 &q) {
        float v[4] = {q.x * down, q.y * down, q.z * down, q.w * down};
        if (p.had) jq::fwht128_warp(v, lane);
        __half2 h01 = __floats2half2_rn(v[0], v[1]), h23 = __floats2half2_rn(v[2], v[3]);
        const size_t off = (((size_t)blk * 16 + (lane >> 1)) * B + b) * 8 + (lane & 1) * 4;
        *reinterpret_cast<uint2 *>(p.xprep + off) =
            make_uint2(*reinterpret_cast<uint32_t *>(&h01), *reinterpret_cast<uint32_t *>(&h23));
    };
#pragma unroll
    for (int i = 0; i < kKeep; ++i)
        if ((warp + i * kWarps) * 128 < p.K) finish(warp + i * kWarps, kept[i]);
    for (int blk = warp + kKeep * kWarps; blk * 128 < p.K; blk += kWarps) finish(blk, load_four(x + blk * 128 + lane * 4, vec));
}

// ---- main kernel --------------------------------------------------------------------
// Roles of a CTA (24 warps): warps 0-15 decode (warp = 32-row quarter q of the tile x phase ph: the CTA's 128-code groups are
// numbered through, phase ph takes groups t = ph, ph + 4, ...); warps 16-19 fold (thread = row): they read every group's
// accumulator back, add it, times the group's scale, to the row's fp32 sums, and write the outputs; warps 20 and 21 issue
// the MMAs of the even and the odd groups (two issuers reach 14 clocks per MMA of 16 columns, one 27); warp 22 streams the
// prepared activation, warp 23 the packed rows, and owns the tensor memory.
//
// Tensor-memory columns: kSlots operand slots of 64 columns (one 128-code group each, group t in slot t mod kSlots) and
// kAccs accumulators of NB columns (group t in t mod kAccs).  An activation stage belongs to the operand slot of its group.
//
// What bounds it: neither a pipe nor the decode warps alone.  7B-shaped GF4 step, 8 rows (70B-shaped E2M1, 7 layers, 16 rows),
// with 8 decode warps before: 1033 us (879); with this kernel: 949 (861).  Of its time, measured before the partition's costs
// were set: the lookups 17 % (11), seven MMAs of eight 12 % (7), folding nothing; with nothing but the barriers, the loads and a
// quarter of the stores it still takes 74 % (83).  Barrier operations are a large part of what is left (a ready wait with its
// vote takes 105 clocks, an elected arrival 50 to 70): operand slots of half a group, which are busy for a shorter time, were
// 2.7 % slower, one issuer and one slot per phase 1.2 %.
// GF4 looks every byte up in the pair table.  Up to 16 rows; more are for the kernel below.
//
// A row's sum is formed in four parts of K (one, for short rows and for 33 rows and more), each in group order, added in
// part order.  A single call with few tiles lets the CTAs of a cluster take the parts; the partial sums meet in
// distributed shared memory and are added in the same order, so the result does not depend on the split.
constexpr int kTaThreads = 24 * 32;
constexpr int kSlots = 6;
constexpr int kPartMinSteps = 8;                                    // 256-code steps from which a row is summed in parts
constexpr int NB = 16;                                              // columns of an MMA
constexpr int kAcc = kSlots * 64;                                   // first column of the accumulators
constexpr int kAccs = 128 / NB, kAccBars = kAccs / 2;               // the two of a step are handed over together
constexpr int kParts = 4;
// registers of a fold thread; the decode threads have 72 and the others 80: 61440 in all, what 768 threads start with at 80
constexpr int kFoldRegs = 112;
static_assert(512 * 72 + 128 * (kFoldRegs + 80) <= 80 * kTaThreads, "registers");
static_assert(kAcc + kAccs * NB <= 512, "tensor memory");

template <bool TABLE>
struct Smem {
    static constexpr int kTab = 0;
    static constexpr int kWRing = TABLE ? kTabBytes : 0;
    static constexpr int kWs = TABLE ? 4 : 8;                       // weight stages (even: a decode warp takes every other one)
    static constexpr int kXRing = kWRing + kWs * kWStage;
    static constexpr int kXStage = 256 * NB;                        // one group of up to NB rows
    static constexpr int kBars = kXRing + kSlots * kXStage;
    static constexpr int kNumBars = 2 * 8 + 3 * kSlots + 2 * 8 + 4;
    static constexpr int kBytes = kBars + kNumBars * 8 + 1024;      // + slack for the 1 KB alignment of the base (TMA swizzle)
    static constexpr int kExch = TABLE ? kTab : kXRing;             // K split: partial sums, once nothing else uses the region
    static_assert(kBytes <= 227 * 1024, "shared memory");
    static_assert(TABLE || 2 * NB * 512 <= kSlots * kXStage, "exchange");
};

// first step of part i of a row of nsteps 256-code steps
__host__ __device__ inline int part_step(int nsteps, int parts, int i) { return nsteps * i / parts; }

template <int FMT>
__global__ void __launch_bounds__(kTaThreads, 1) gemm_ta_kernel(const TaProblem *probs, const CUtensorMap *maps,
                                                                const __grid_constant__ TaProblem single,
                                                                const __grid_constant__ CUtensorMap single_map, int nprob,
                                                                const int *tile_start, const int *cta_first,
                                                                int B, int y_dtype, PeerInfo peers, int split, int *status) {
    constexpr bool kGf4 = FMT == JQ_FMT_GF4;                        // with pair tables in shared memory
    using S = Smem<kGf4>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (uniform for the compiler)
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = sbase + S::kBars;
    auto wfull = [&](int s) { return bars + 8u * s; };                                  // packed rows of a step landed
    auto wempty = [&](int s) { return bars + 8u * (8 + s); };                           // and read by the eight warps
    auto afull = [&](int s) { return bars + 8u * (16 + s); };                           // operand slot written
    auto sfree = [&](int s) { return bars + 8u * (16 + kSlots + s); };                  // its MMAs are done (activation stage too)
    auto xfull = [&](int s) { return bars + 8u * (16 + 2 * kSlots + s); };              // activation stage landed
    auto dfull = [&](int a) { return bars + 8u * (16 + 3 * kSlots + a); };              // accumulators complete
    auto dfree = [&](int a) { return bars + 8u * (24 + 3 * kSlots + a); };              // accumulators read
    auto qbar = [&](int q) { return bars + 8u * (32 + 3 * kSlots + q); };
    volatile int *err = &s_err;

    if (tid == 0) {
        s_err = 0;
        for (int s = 0; s < S::kWs; ++s) { mbar_init(wfull(s), 1); mbar_init(wempty(s), 8); }
        for (int s = 0; s < kSlots; ++s) { mbar_init(afull(s), 4); mbar_init(sfree(s), 1); mbar_init(xfull(s), 1); }
        for (int a = 0; a < kAccBars; ++a) { mbar_init(dfull(a), 2); mbar_init(dfree(a), 4); }
        for (int q = 0; q < 4; ++q) mbar_init(qbar(q), 4);             // the warps that share a quarter of the rows
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 23) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    // this CTA's tiles
    int tile_lo, tile_hi, rank = 0;
    if (nprob == 0) {   // one problem, passed by value: an even split of its tiles; with a K split one tile per cluster
        const int nt = (single.N + kTileM - 1) / kTileM, n_cl = gridDim.x / split, cl = blockIdx.x / split;
        rank = blockIdx.x - cl * split;
        tile_lo = (int)((long long)nt * cl / n_cl);
        tile_hi = (int)((long long)nt * (cl + 1) / n_cl);
    } else {
        tile_lo = cta_first[blockIdx.x];
        tile_hi = cta_first[blockIdx.x + 1];
    }
    // parts of a row's sum, and the steps [lo, hi) of a row that this CTA works on
    auto parts_of = [&](int nsteps) { return nsteps >= kPartMinSteps ? kParts : 1; };
    auto step_lo = [&](int nsteps) { return split > 1 ? part_step(nsteps, kParts, kParts / split * rank) : 0; };
    auto step_hi = [&](int nsteps) { return split > 1 ? part_step(nsteps, kParts, kParts / split * (rank + 1)) : nsteps; };
    // Problems change rarely along a CTA's tile sequence: every walker keeps what it needs of its current
    // problem in registers and goes back to global memory only for a tile beyond that problem's last one.
    auto problem_at = [&](int &pi, int &t_end, int tile, TaProblem &p) {
        if (nprob == 0) { p = single; t_end = 0x7fffffff; return; }
        if (t_end < 0) {
            // first look-up of a walker: bisect (a step's list can hold hundreds of problems, and a scan from the
            // first one is a chain of dependent global loads, 0.2 us each, in front of the last CTAs' first tile)
            int lo = 0, hi = nprob - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (tile_start[mid] <= tile) lo = mid; else hi = mid - 1;
            }
            pi = lo;
        } else {
            while (pi + 1 < nprob && tile_start[pi + 1] <= tile) ++pi;
        }
        p = probs[pi];
        t_end = tile_start[pi + 1];
    };
    auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)); };
    auto warp_arrive = [&](uint32_t bar) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };

    if (warp < 16) {
        // =============================== decode warps ===============================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const int q = warp & 3, ph = warp >> 2, gi = ph & 1;
        const int r = q * 32 + lane;                       // row of the tile = tensor-memory lane
        const uint32_t lane_t = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t tcol = sbase + S::kTab + q * (256 * 128) + lane * 4;   // pair table: entry e of this row at tcol + 128 e
        // this row's 64 bytes of the group: 16-byte piece c of a row sits at piece c ^ (row & 7) (128-byte swizzle)
        const uint32_t wrow = sbase + S::kWRing + r * 128, wkey = (lane & 7) << 4;

        // ---- per-row side data one tile ahead: GF4 codebook row
        int f_pi = 0, f_tend = -1, f_tile0 = 0, f_N = 1;
        const __half *f_cb = nullptr;
        uint4 cb0 = make_uint4(0, 0, 0, 0), cb1 = cb0;
        auto fetch_codebook = [&](int tile) {
            if (kGf4 && tile < tile_hi) {
                if (tile >= f_tend) {
                    TaProblem p;
                    problem_at(f_pi, f_tend, tile, p);
                    f_tile0 = p.tile0; f_N = p.N; f_cb = p.codebook;
                }
                const int row = min((tile - f_tile0) * kTileM + r, f_N - 1);
                const uint4 *src = reinterpret_cast<const uint4 *>(f_cb + (size_t)row * 16);
                cb0 = __ldg(src);
                cb1 = __ldg(src + 1);
            }
        };

        // The CTA's steps are numbered through: step c is in weight stage c mod kWs, its groups are t = 2 c and 2 c + 1.
        // This warp takes the steps of its parity.
        int skip = ph >> 1;                          // steps of other warps before this warp's next one (0 or 1)
        int w_stage = ph >> 1, slot = ph;            // slot of group ph: ph < kSlots
        uint32_t w_par = 0, s_par = 1;               // (the first use of a slot finds it free)
        uint32_t q_par = 0;
        auto quarter_sync = [&]() -> bool {
            warp_arrive(qbar(q));
            const bool ok = warp_wait(qbar(q), q_par);
            q_par ^= 1;
            return ok;
        };

        int c_pi = 0, c_tend = -1;
        int K = single.K, N = single.N, lds = single.lds, tile0 = 0;
        const __half *scales = single.scales;
        fetch_codebook(tile_lo);
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            if (tile >= c_tend) {
                TaProblem p;
                problem_at(c_pi, c_tend, tile, p);
                K = p.K; N = p.N; lds = p.lds; tile0 = p.tile0; scales = p.scales;
            }
            const int s_lo = step_lo(K >> 8), s_hi = step_hi(K >> 8);
            const int s_first = s_lo + skip;
            skip = (skip + s_hi - s_lo) & 1;         // (s_hi > s_lo)
            // E2M1: four fp16 scales (8 bytes) per group, one group of this warp ahead
            const int row = min((tile - tile0) * kTileM + r, N - 1);
            const uint2 *srow = reinterpret_cast<const uint2 *>(scales + (size_t)row * lds) + gi;
            uint2 sc_nxt = make_uint2(0, 0);
            if (!kGf4 && s_first < s_hi) sc_nxt = __ldg(srow + 2 * s_first);
            if constexpr (kGf4) {
                // ---- the pair table of this row (this thread fills the entries whose second code is 4 ph .. 4 ph + 3)
                if (!(ok = quarter_sync())) break;      // the four warps are done with the previous tile's lookups
                const uint32_t c[8] = {cb0.x, cb0.y, cb0.z, cb0.w, cb1.x, cb1.y, cb1.z, cb1.w};
                uint32_t ch[2] = {c[0], c[1]};
#pragma unroll
                for (int i = 1; i < 4; ++i) { ch[0] = ph == i ? c[2 * i] : ch[0]; ch[1] = ph == i ? c[2 * i + 1] : ch[1]; }
                const uint32_t tb = tcol + ph * (64 * 128);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int lo = 0; lo < 16; ++lo) {
                        const uint32_t e = __byte_perm(c[lo >> 1], ch[i >> 1],
                                                       ((lo & 1) ? 0x32u : 0x10u) | (((i & 1) ? 0x76u : 0x54u) << 8));
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(tb + (i * 16 + lo) * 128), "r"(e) : "memory");
                    }
            }
            fetch_codebook(tile + 1);
            if constexpr (kGf4) { if (!(ok = quarter_sync())) break; }
            for (int sg = s_first; sg < s_hi; sg += 2) {
                if (!(ok = warp_wait(wfull(w_stage), w_par))) break;
                const uint32_t src = wrow + w_stage * kWStage;
                const uint2 sc4 = sc_nxt;
                if (!kGf4 && sg + 2 < s_hi) sc_nxt = __ldg(srow + 2 * (sg + 2));
                const uint32_t a_t = lane_t + slot * 64;
                uint4 w4[4];
#pragma unroll
                for (int part = 0; part < 4; ++part) w4[part] = lds128(src + ((uint32_t)((gi * 4 + part) << 4) ^ wkey));
                // 32 codes (four words) -> 16 fp16 pairs
                auto decode16 = [&](int part, uint32_t (&v)[16]) {
#pragma unroll
                    for (int wi = 0; wi < 4; ++wi) {
                        const uint32_t w = wi == 0 ? w4[part].x : (wi == 1 ? w4[part].y : (wi == 2 ? w4[part].z : w4[part].w));
                        if constexpr (kGf4) {
#pragma unroll
                            for (int bj = 0; bj < 4; ++bj) v[wi * 4 + bj] = lds32(dp4a_u(w, 0x80u << (8 * bj), tcol));
                        } else {
                            // E2M1: the group scale folded into the fp16 weight (one rounding per weight)
                            const uint32_t pr = part < 2 ? sc4.x : sc4.y;
                            const uint32_t s2 = prmt(pr, pr, (part & 1) ? 0x3232 : 0x1010);
                            uint32_t hh[4];
                            asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4;\n"
                                "  cvt.rn.f16x2.e2m1x2 %0, b0; cvt.rn.f16x2.e2m1x2 %1, b1;\n"
                                "  cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
                                : "=r"(hh[0]), "=r"(hh[1]), "=r"(hh[2]), "=r"(hh[3]) : "r"(w));
#pragma unroll
                            for (int bj = 0; bj < 4; ++bj)
                                asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(v[wi * 4 + bj]) : "r"(hh[bj]), "r"(s2));
                        }
                    }
                };
                // half of the group is decoded before the wait for its slot, the rest while the first pairs are being stored;
                // handed over at once (kept until the next group's first lookups are under way, which spares a wait for the
                // stores, a slot is held for longer: 7 % slower on the 7B-shaped GF4 step with 8 rows)
                uint32_t va[16], vb[16];
                decode16(0, va);
                decode16(1, vb);
                if (!(ok = warp_wait(sfree(slot), s_par))) break;
                tc_fence_after();
                tmem_st16(a_t, va);
                decode16(2, va);
                tmem_st16(a_t + 16, vb);
                decode16(3, vb);
                tmem_st16(a_t + 32, va);
                tmem_st16(a_t + 48, vb);
                warp_arrive(wempty(w_stage));
                tmem_wait_st();
                tc_fence_before();
                warp_arrive(afull(slot));
                if ((slot += 4) >= kSlots) { slot -= kSlots; s_par ^= 1; }
                if ((w_stage += 2) >= S::kWs) { w_stage -= S::kWs; w_par ^= 1; }
            }
        }
        if (split > 1) { __syncwarp(); cluster_sync(); cluster_sync(); }
    } else if (warp < 20) {
        // =============================== fold threads ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFoldRegs));
        const int r = tid & 127;
        const uint32_t lane_t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kAcc;
        uint32_t buf = 0, par = 0;                  // accumulators of the next step (or group) and their phase
        int c_pi = 0, c_tend = -1;
        TaProblem p = single;
        pdl_wait();                                 // the row factors of the prepared activation are read below
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            if (tile >= c_tend) problem_at(c_pi, c_tend, tile, p);
            const int row_raw = (tile - p.tile0) * kTileM + r, row = min(row_raw, p.N - 1);
            const int nsteps = p.K >> 8, parts = parts_of(nsteps), s_lo = step_lo(nsteps), s_hi = step_hi(nsteps);
            const unsigned short *srow = reinterpret_cast<const unsigned short *>(p.scales) + (size_t)row * p.lds;
            const int gshift = kGf4 ? 31 - __clz(p.g >> 7) : 0;   // GF4: log2 of the 128-code groups per scale
            const bool word = gshift == 0 && ((size_t)p.scales & 3) == 0;
            const float xs = lane < B ? p.xscale[lane] : 0.f;
            const float bias = (p.bias && row_raw < p.N) ? p.bias[row_raw] : 0.f;
            float acc[NB], total[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) acc[b] = 0.f;
            const uint32_t exch = sbase + S::kExch + r * 4;
            int part = split > 1 ? kParts / split * rank : 0, part_end = part_step(nsteps, parts, part + 1);
            bool first = true;
            // the two scales of a step, a step ahead; in 128-code groups they are one aligned word (K is a multiple of 256)
            uint32_t raw = 0;
            auto load_scales = [&](int sg) {
                if (kGf4) {
                    if (word) raw = __ldg(reinterpret_cast<const unsigned int *>(srow + 2 * sg));
                    else raw = __ldg(srow + ((2 * sg) >> gshift)) | (uint32_t)__ldg(srow + ((2 * sg + 1) >> gshift)) << 16;
                }
            };
            load_scales(s_lo);
            for (int sg = s_lo; sg < s_hi && ok; ++sg) {
                const float sc[2] = {__half2float(__ushort_as_half((unsigned short)raw)),
                                     __half2float(__ushort_as_half((unsigned short)(raw >> 16)))};
                if (sg + 1 < s_hi) load_scales(sg + 1);
                // both groups of the step at once: the way from the barrier through tensor memory to the release is a
                // chain of latencies
                if (!(ok = warp_wait(dfull(buf), par))) break;
                tc_fence_after();
                uint32_t d0[16], d1[16];
                tmem_ld16(lane_t + buf * 2 * NB, d0);
                tmem_ld16(lane_t + buf * 2 * NB + NB, d1);
                tmem_wait_ld();
                tc_fence_before();
                warp_arrive(dfree(buf));
#pragma unroll
                for (int i = 0; i < 16; i += 2) fma2(acc[i], acc[i + 1], d0[i], d0[i + 1], kGf4 ? sc[0] : 1.f);
#pragma unroll
                for (int i = 0; i < 16; i += 2) fma2(acc[i], acc[i + 1], d1[i], d1[i + 1], kGf4 ? sc[1] : 1.f);
                if (++buf == (uint32_t)kAccBars) { buf = 0; par ^= 1; }
                if (!ok) break;
                if (sg + 1 == part_end) {      // a part of the row's sum is complete
                    if (split > 1) {        // at most two per CTA: the first waits in `total`, the second stays in `acc`
                        if (first) {
#pragma unroll
                            for (int b = 0; b < NB; ++b) { total[b] = acc[b]; acc[b] = 0.f; }
                        }
                    } else {
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            total[b] = first ? acc[b] : total[b] + acc[b];
                            acc[b] = 0.f;
                        }
                    }
                    first = false;
                    ++part;
                    part_end = part_step(nsteps, parts, part + 1);
                }
            }
            if (split > 1) {
                // every group of this CTA has been folded: nothing reads the tables or the activation stages any more.
                // Each CTA leaves its parts in its shared memory; rank k writes columns k, k + split, ...
                const int per = kParts / split;
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(exch + b * 512), "f"(total[b]) : "memory");
                    if (per == 2) asm volatile("st.shared.f32 [%0], %1;" ::"r"(exch + (NB + b) * 512), "f"(acc[b]) : "memory");
                }
                cluster_sync();
                for (int b = rank; b < B; b += split) {
                    float v = ld_cluster_f32(exch + b * 512, 0);
                    for (int i = 1; i < kParts; ++i) v += ld_cluster_f32(exch + ((i % per) * NB + b) * 512, i / per);
                    if (ok && row_raw < p.N) jq::store_out(p.y, (size_t)b * p.ldy + row_raw, fmaf(v, p.xscale[b], bias), y_dtype);
                }
                cluster_sync();
                break;
            }
            if (!ok) break;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const float xs_b = __shfl_sync(0xffffffffu, xs, b);
                acc[b] = fmaf(total[b], xs_b, bias);
            }
            if (row_raw < p.N) {
                for (int cpy = 0; cpy < peers.n; ++cpy) {
                    char *yb = reinterpret_cast<char *>(p.y) + jq::peer_offset(peers.delta, cpy);
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        if (b < B) jq::store_out(yb, (size_t)b * p.ldy + row_raw, acc[b], y_dtype);
                }
            }
        }
    } else {
        // walk of this CTA's tiles: (tile, its problem, the range of its steps)
        int pi = 0, t_end = -1, lo = 0, hi = 0;
        TaProblem p = single;
        auto open = [&](int tile) {
            if (tile >= t_end) {
                problem_at(pi, t_end, tile, p);
                lo = step_lo(p.K >> 8);
                hi = step_hi(p.K >> 8);
            }
        };
        bool ok = true;
        if (warp < 22) {
            // =============================== MMA issuers ===============================
            // (the warps run converged, see mma_f16_ts; slots, accumulators and parities are carried along instead of being
            // divided out of counters, and the operand descriptor is formed once per group)
            const uint32_t elected = elect_one();
            constexpr uint32_t idesc = idesc_f16(kTileM, NB);
            const uint32_t lbo = (uint32_t)B * 16;
            const uint32_t desc_step = (2 * lbo) >> 4;  // descriptor address field per K = 16 slice
            uint32_t slot = warp - 20, s_par = 0, acc = 0, d_par = 1;   // (the first use of an accumulator finds it free)
            for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
                open(tile);
                for (int sg = lo; sg < hi; ++sg) {
                    if (!(ok = warp_wait(dfree(acc), d_par) && warp_wait(xfull(slot), s_par) && warp_wait(afull(slot), s_par))) break;
                    tc_fence_after();
                    const uint32_t a_t = tmem + slot * 64;
                    const uint32_t d_t = tmem + kAcc + (2 * acc + warp - 20) * NB;
                    const uint64_t desc0 = smem_desc(sbase + S::kXRing + slot * S::kXStage, lbo, 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        mma_f16_ts(elected, d_t, a_t + 8 * i, desc0 + (uint64_t)(i * desc_step), idesc, i > 0);
                    mma_commit(elected, sfree(slot));
                    mma_commit(elected, dfull(acc));
                    if ((slot += 2) >= (uint32_t)kSlots) { slot -= kSlots; s_par ^= 1; }
                    if (++acc == (uint32_t)kAccBars) { acc = 0; d_par ^= 1; }
                }
            }
        } else if (warp == 22 && lane == 0) {
            // =============================== activation loader ===============================
            const uint32_t chunk = 256 * B;
            uint32_t slot = 0, par = 1;                 // (the first use of a stage finds it free)
            pdl_wait();
            for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
                open(tile);
                const unsigned char *src = reinterpret_cast<const unsigned char *>(p.xprep) + (size_t)(2 * lo) * chunk;
                for (int g = 2 * lo; g < 2 * hi; ++g, src += chunk) {
                    if (!(ok = mbar_wait(sfree(slot), par, err))) break;
                    mbar_expect_tx(xfull(slot), chunk);
                    bulk_g2s(sbase + S::kXRing + slot * S::kXStage, src, chunk, xfull(slot));
                    if (++slot == (uint32_t)kSlots) { slot = 0; par ^= 1; }
                }
            }
        } else if (warp == 23 && lane == 0) {
            // =============================== weight loader ===============================
            uint32_t stage = 0, par = 1;
            for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
                open(tile);
                const void *map = nprob ? &maps[pi] : &single_map;
                const int row0 = (tile - p.tile0) * kTileM;     // rows past N read as zeros
                if (split == 1) {
                    // the tile's scales are read in small pieces a step or two ahead, which hides the L2's latency but not
                    // the memory's: they are one piece of memory (rows of lds scales), fetched into the L2 by one instruction
                    const size_t a = (size_t)(p.scales + (size_t)row0 * p.lds) & ~(size_t)15;
                    const uint32_t bytes = (uint32_t)min(kTileM, p.N - row0) * (uint32_t)p.lds * 2u & ~15u;
                    if (bytes) l2_prefetch(reinterpret_cast<const void *>(a), bytes);
                }
                for (int sg = lo; sg < hi; ++sg) {
                    if (!(ok = mbar_wait(wempty(stage), par, err))) break;
                    mbar_expect_tx(wfull(stage), kWStage);
                    tma_2d_g2s(sbase + S::kWRing + stage * kWStage, map, sg * 128, row0, wfull(stage));
                    if (++stage == (uint32_t)S::kWs) { stage = 0; par ^= 1; }
                }
            }
        }
        __syncwarp();
        if (split > 1) { cluster_sync(); cluster_sync(); }
    }

    // ---- teardown
    if (*err) {   // a wait gave up: let the copies still in flight land before the CTA's shared memory goes away
        for (int i = 0; i < 400; ++i) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_err) atomicExch(status, s_err);
    if (warp == 23) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---- 17 to 64 rows --------------------------------------------------------------------
// With 32 or 64 columns the folding of the accumulators weighs as much as the decoding, and a kernel of fewer warps is ahead:
// the kernel above took 83 us for 28672 x 8192 E2M1 with 64 rows, this one 54; 17.0 and 14.8 for 11008 x 4096 with 24; 316 and
// 285 for a step of eight 8B-shaped layers with 24 rows.
// Roles of a CTA (16 warps): warps 0-7 decode (warp = 32-row quarter q of the tile x half h of the 256-code
// steps of a row: step sg belongs to half sg & 1); warps 8-11 fold (thread = row); warps 12-15 issue MMAs (two issuers per half)
// and stream the prepared activation of their own groups; warp 15 also owns the tensor-memory allocation.
//
// Tensor-memory columns: two slots per half of 64 columns each for the A operand (one 128-code group) and kAccBufs
// accumulators of NB columns per issuer.  GF4 words go through byte permutes: there is no shared memory for tables beside the
// activation rings.
namespace wide {

constexpr int kDecodeWarps = 8;              // warps 0-3: first half of the steps, warps 4-7: second half
constexpr int kWStage = 32 * 128;            // bytes of a weight stage: 32 rows x 128 bytes (256 codes), swizzled by TMA
constexpr int kXMaxStages = 8;               // stages of an MMA issuer's activation ring, at most
constexpr int kTaThreads = 16 * 32;
template <int FMT, int NB>
struct Cols {
    static constexpr int kRing = 2;                                 // groups a half may have in flight
    static constexpr int kAccBufs = NB == 64 ? 1 : 2;               // accumulators of an issuer
    static constexpr int kAcc = 2 * kRing * 64;                     // accumulator b of issuer i at kAcc + (i * kAccBufs + b) * NB
    static constexpr int kParts = NB == 64 ? 1 : 4;
    static_assert(kAcc + 4 * kAccBufs * NB <= 512, "tensor memory");
    // one barrier per accumulator says that a group's MMAs are done, to the fold threads and to the decode threads that
    // wait for the group's slot; before a slot's next group is written, no later group can have used the accumulator
    static_assert(2 * kAccBufs >= kRing, "the barrier would be a phase ahead");
};

struct Smem {
    static constexpr int kWRing = 0;
    static constexpr int kSW = 2;       // stages of a decode warp's weight ring (four did not change anything: the ring is not what the decode threads wait for)
    static constexpr int kXRing = kWRing + kDecodeWarps * kSW * kWStage;
    static constexpr int kXBytes = 152 * 1024;                      // two stages of 64 batch rows per issuer
    static constexpr int kBars = kXRing + kXBytes + 512;            // + what the MMA reads past the last chunk (rows >= B)
    static constexpr int kNumBars = kDecodeWarps * kSW + 6 + 2 * 8 + 4 * kXMaxStages;   // weights, A full, accumulator full/free, x full per issuer
    static constexpr int kBytes = kBars + kNumBars * 8 + 1024;      // + slack for the 1 KB alignment of the base (TMA swizzle)
    static constexpr int kExch = kXRing;                            // K split: partial sums, once nothing else uses the region
    static_assert(kBytes <= 227 * 1024, "shared memory");
};

// geometry of an issuer's activation ring for a batch of B rows: a stage is one group (128 codes), 256 B bytes
struct XGeom {
    int chunk, ring, nstages;
    __host__ __device__ XGeom(int B, int ring_bytes) {
        chunk = 256 * B;
        ring = ring_bytes;
        nstages = ring_bytes / chunk < kXMaxStages ? ring_bytes / chunk : kXMaxStages;
    }
};

template <int FMT, int NB>
__global__ void __launch_bounds__(kTaThreads, 1) gemm_ta_wide_kernel(const TaProblem *probs, const CUtensorMap *maps,
                                                                const __grid_constant__ TaProblem single,
                                                                const __grid_constant__ CUtensorMap single_map, int nprob,
                                                                const int *tile_start, const int *cta_first,
                                                                int B, int y_dtype, PeerInfo peers, int split, int *status) {
    using C = Cols<FMT, NB>;
    using S = Smem;
    constexpr bool kGf4 = FMT == JQ_FMT_GF4;
    constexpr int kRing = C::kRing;
    constexpr int kSW = S::kSW;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (uniform for the compiler)
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = sbase + S::kBars;
    constexpr int kB0 = kDecodeWarps * kSW;
    auto wbar = [&](int w, int s) { return bars + 8u * (w * kSW + s); };
    auto abar = [&](int h, int s) { return bars + 8u * (kB0 + h * 3 + s); };                  // operand slot written
    auto dbar = [&](int iss, int b) { return bars + 8u * (kB0 + 6 + iss * 2 + b); };          // accumulator complete: a group's MMAs are done
    auto ebar = [&](int iss, int b) { return bars + 8u * (kB0 + 14 + iss * 2 + b); };         // accumulator folded
    auto xbar = [&](int iss, int s) { return bars + 8u * (kB0 + 22 + iss * kXMaxStages + s); };   // issuer's stage filled
    volatile int *err = &s_err;
    const XGeom xg(B, S::kXBytes / 4);

    if (tid == 0) {
        s_err = 0;
        for (int w = 0; w < kDecodeWarps; ++w)
            for (int s = 0; s < kSW; ++s) mbar_init(wbar(w, s), 1);     // one arrive.expect_tx per fill
        for (int h = 0; h < 2; ++h)
            for (int s = 0; s < 3; ++s) mbar_init(abar(h, s), 128);     // the 128 decode threads of the half
        for (int i = 0; i < 4; ++i)
            for (int b = 0; b < 2; ++b) { mbar_init(dbar(i, b), 1); mbar_init(ebar(i, b), 128); }
        for (int i = 0; i < 4; ++i)
            for (int s = 0; s < kXMaxStages; ++s) mbar_init(xbar(i, s), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 15) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    // this CTA's tiles
    int tile_lo, tile_hi, rank = 0;
    if (nprob == 0) {   // one problem, passed by value: an even split of its tiles; with a K split one tile per cluster
        const int nt = (single.N + kTileM - 1) / kTileM, n_cl = gridDim.x / split, cl = blockIdx.x / split;
        rank = blockIdx.x - cl * split;
        tile_lo = (int)((long long)nt * cl / n_cl);
        tile_hi = (int)((long long)nt * (cl + 1) / n_cl);
    } else {
        tile_lo = cta_first[blockIdx.x];
        tile_hi = cta_first[blockIdx.x + 1];
    }
    // parts of a row's sum, and the steps [lo, hi) of a row that this CTA works on
    auto parts_of = [&](int nsteps) { return nsteps >= kPartMinSteps ? C::kParts : 1; };
    auto step_lo = [&](int nsteps) { return split > 1 ? part_step(nsteps, C::kParts, C::kParts / split * rank) : 0; };
    auto step_hi = [&](int nsteps) { return split > 1 ? part_step(nsteps, C::kParts, C::kParts / split * (rank + 1)) : nsteps; };
    // Problems change rarely along a CTA's tile sequence: every walker keeps what it needs of its current
    // problem in registers and goes back to global memory only for a tile beyond that problem's last one.
    auto problem_at = [&](int &pi, int &t_end, int tile, TaProblem &p) {
        if (nprob == 0) { p = single; t_end = 0x7fffffff; return; }
        if (t_end < 0) {
            // first look-up of a walker: bisect (a step's list can hold hundreds of problems, and a scan from the
            // first one is a chain of dependent global loads, 0.2 us each, in front of the last CTAs' first tile)
            int lo = 0, hi = nprob - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (tile_start[mid] <= tile) lo = mid; else hi = mid - 1;
            }
            pi = lo;
        } else {
            while (pi + 1 < nprob && tile_start[pi + 1] <= tile) ++pi;
        }
        p = probs[pi];
        t_end = tile_start[pi + 1];
    };

    if (warp < kDecodeWarps) {
        // =============================== decode threads ===============================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 112;");     // 256 x 112 + 128 x 184 + 128 x 96 of 65536 registers
        const int q = warp & 3, h = warp >> 2;
        const int r = q * 32 + lane;                       // row of the tile = tensor-memory lane
        const uint32_t lane_t = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t wring = sbase + S::kWRing + warp * (kSW * kWStage);     // + stage * kWStage; 1 KB aligned
        // 16-byte piece c of this lane's row sits at piece c ^ (lane & 7) of the row (128-byte swizzle)
        const uint32_t lrow = lane * 128, lkey = (lane & 7) << 4;

        // ---- producer side of the weight ring: the (tile, step) whose box is requested next
        int i_tile = tile_lo, i_pi = 0, i_tend = -1, i_j = 0, i_n = 0, i_x = 0, i_x0 = 0, i_y = 0, i_tile0 = 0, i_steps = 0, i_stage = 0;
        const void *i_map = nullptr;
        auto i_open = [&]() {
            while (i_tile < tile_hi) {
                if (i_tile >= i_tend) {
                    TaProblem p;
                    problem_at(i_pi, i_tend, i_tile, p);
                    const int ns = p.K >> 8, lo = step_lo(ns);
                    i_steps = (step_hi(ns) - lo - h + 1) >> 1;
                    i_x0 = (lo + h) * 128;
                    i_tile0 = p.tile0;
                    i_map = nprob ? &maps[i_pi] : &single_map;
                }
                i_n = i_steps;
                i_x = i_x0;
                i_y = (i_tile - i_tile0) * kTileM + q * 32;     // rows past N read as zeros
                i_j = 0;
                if (i_n > 0) return;
                ++i_tile;
            }
        };
        auto issue = [&]() {
            if (i_tile < tile_hi) {
                if (lane == 0) {
                    const uint32_t bar = wbar(warp, i_stage);
                    mbar_expect_tx(bar, kWStage);
                    tma_2d_g2s(wring + i_stage * kWStage, i_map, i_x, i_y, bar);
                }
                i_x += 256;
                if (++i_j == i_n) { ++i_tile; i_open(); }
            }
            i_stage = (i_stage + 1 == kSW) ? 0 : i_stage + 1;
        };
        i_open();
#pragma unroll
        for (int s = 0; s < kSW; ++s) issue();

        // ---- per-row side data one tile ahead: GF4 codebook row
        int f_pi = 0, f_tend = -1, f_tile0 = 0, f_N = 1;
        const __half *f_cb = nullptr;
        uint4 cb0 = make_uint4(0, 0, 0, 0), cb1 = cb0;
        auto fetch_codebook = [&](int tile) {
            if (kGf4 && tile < tile_hi) {
                if (tile >= f_tend) {
                    TaProblem p;
                    problem_at(f_pi, f_tend, tile, p);
                    f_tile0 = p.tile0; f_N = p.N; f_cb = p.codebook;
                }
                const int row = min((tile - f_tile0) * kTileM + r, f_N - 1);
                const uint4 *src = reinterpret_cast<const uint4 *>(f_cb + (size_t)row * 16);
                cb0 = __ldg(src);
                cb1 = __ldg(src + 1);
            }
        };

        // ---- consumer state
        int w_stage = 0, slot = 0, pend_slot = -1;   // pend_slot: its tensor-memory stores are issued but not yet handed over
        uint32_t w_par = 0;
        uint32_t t_next = 0;                         // groups this half has decoded so far
        Codebook book;
        auto hand_over = [&]() {
            if (pend_slot >= 0) {
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(abar(h, pend_slot));
                pend_slot = -1;
            }
        };
        int c_pi = 0, c_tend = -1;
        TaProblem p = single;
        fetch_codebook(tile_lo);
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            if (tile >= c_tend) problem_at(c_pi, c_tend, tile, p);
            const int s_lo = step_lo(p.K >> 8), s_hi = step_hi(p.K >> 8);
            // E2M1: eight fp16 scales (16 bytes) per 256-code step of the row, a step ahead
            const int row = min((tile - p.tile0) * kTileM + r, p.N - 1);
            const uint4 *srow = reinterpret_cast<const uint4 *>(p.scales + (size_t)row * p.lds);
            uint4 sc_nxt = make_uint4(0, 0, 0, 0);
            if (!kGf4 && s_lo + h < s_hi) sc_nxt = __ldg(srow + s_lo + h);
            if constexpr (kGf4) book.set(cb0, cb1);
            fetch_codebook(tile + 1);
            for (int sg = s_lo + h; sg < s_hi; sg += 2) {
                ok = __all_sync(0xffffffffu, mbar_wait(wbar(warp, w_stage), w_par, err));
                if (!ok) break;
                const uint32_t src = wring + w_stage * kWStage + lrow;
                if (++w_stage == kSW) { w_stage = 0; w_par ^= 1; }
                const uint4 sc_cur = sc_nxt;
                if (!kGf4 && sg + 2 < s_hi) sc_nxt = __ldg(srow + sg + 2);
#pragma unroll
                for (int gi = 0; gi < 2; ++gi) {
                    const uint2 sc4 = gi ? make_uint2(sc_cur.z, sc_cur.w) : make_uint2(sc_cur.x, sc_cur.y);
                    const uint32_t a_t = lane_t + (h * kRing + slot) * 64;
                    uint4 w4[4];
#pragma unroll
                    for (int part = 0; part < 4; ++part) w4[part] = lds128(src + (((gi * 4 + part) << 4) ^ lkey));
                    // 32 codes (four words) -> 16 fp16 pairs
                    auto decode16 = [&](int part, uint32_t (&v)[16]) {
#pragma unroll
                        for (int wi = 0; wi < 4; ++wi) {
                            const uint32_t w = wi == 0 ? w4[part].x : (wi == 1 ? w4[part].y : (wi == 2 ? w4[part].z : w4[part].w));
                            if constexpr (kGf4) {
                                uint32_t hh[4];
                                book.look_up8(w, hh);
#pragma unroll
                                for (int bj = 0; bj < 4; ++bj) v[wi * 4 + bj] = hh[bj];
                            } else {
                                // E2M1: the group scale folded into the fp16 weight (one rounding per weight)
                                const uint32_t pr = part < 2 ? sc4.x : sc4.y;
                                const uint32_t s2 = prmt(pr, pr, (part & 1) ? 0x3232 : 0x1010);
                                uint32_t hh[4];
                                asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4;\n"
                                    "  cvt.rn.f16x2.e2m1x2 %0, b0; cvt.rn.f16x2.e2m1x2 %1, b1;\n"
                                    "  cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
                                    : "=r"(hh[0]), "=r"(hh[1]), "=r"(hh[2]), "=r"(hh[3]) : "r"(w));
#pragma unroll
                                for (int bj = 0; bj < 4; ++bj)
                                    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(v[wi * 4 + bj]) : "r"(hh[bj]), "r"(s2));
                            }
                        }
                    };
                    // the decode of the next 32 codes is issued before the previous 16 pairs are stored, and the
                    // previous group is handed to the MMA issuer only once this group's first lookups are under way
                    // (its tensor-memory stores have had that long to land), and before the wait for this group's slot
                    uint32_t va[16], vb[16];
                    decode16(0, va);
                    decode16(1, vb);
                    hand_over();
                    // the slot is free once the MMAs of the group that used it last are done
                    if (t_next >= (uint32_t)kRing) {
                        const uint32_t t = t_next - kRing, n = t >> 1;     // group t was its issuer's n-th
                        ok = __all_sync(0xffffffffu, mbar_wait(dbar(h + 2 * (t & 1), n % C::kAccBufs), (n / C::kAccBufs) & 1, err));
                        if (!ok) break;
                        tc_fence_after();
                    }
                    ++t_next;
                    tmem_st16(a_t, va);
                    decode16(2, va);
                    tmem_st16(a_t + 16, vb);
                    decode16(3, vb);
                    tmem_st16(a_t + 32, va);
                    tmem_st16(a_t + 48, vb);
                    pend_slot = slot;
                    if (++slot == kRing) slot = 0;
                }
                if (!ok) break;
                __syncwarp();                           // every lane has read its row of the stage
                fence_async_smem();
                issue();                                // refill the stage just read
            }
            hand_over();
        }
        if (split > 1) { __syncwarp(); cluster_sync(); cluster_sync(); }
    } else if (warp < 12) {
        // =============================== fold threads ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
        const int r = tid & 127;
        const uint32_t lane_t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::kAcc;
        uint32_t counts = 0;                        // steps of each half so far, modulo 4 (two bits each)
        int c_pi = 0, c_tend = -1;
        TaProblem p = single;
        pdl_wait();                                 // the row factors of the prepared activation are read below
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            if (tile >= c_tend) problem_at(c_pi, c_tend, tile, p);
            const int row_raw = (tile - p.tile0) * kTileM + r, row = min(row_raw, p.N - 1);
            const int nsteps = p.K >> 8, parts = parts_of(nsteps), s_lo = step_lo(nsteps), s_hi = step_hi(nsteps);
            const unsigned short *srow = reinterpret_cast<const unsigned short *>(p.scales) + (size_t)row * p.lds;
            const int gshift = kGf4 ? 31 - __clz(p.g >> 7) : 0;   // GF4: log2 of the 128-code groups per scale
            float xs[(NB + 31) / 32];
#pragma unroll
            for (int i = 0; i < (NB + 31) / 32; ++i) xs[i] = (lane + 32 * i < B) ? p.xscale[lane + 32 * i] : 0.f;
            const float bias = (p.bias && row_raw < p.N) ? p.bias[row_raw] : 0.f;
            float acc[NB], total[C::kParts > 1 ? NB : 1];
#pragma unroll
            for (int b = 0; b < NB; ++b) acc[b] = 0.f;
            const uint32_t exch = sbase + S::kExch + r * 4;
            int part = split > 1 ? C::kParts / split * rank : 0, part_end = part_step(nsteps, parts, part + 1);
            bool first = true;
            unsigned short raw0 = 0, raw1 = 0;
            auto load_scales = [&](int sg) {
                if (kGf4) { raw0 = __ldg(srow + ((2 * sg) >> gshift)); raw1 = __ldg(srow + ((2 * sg + 1) >> gshift)); }
            };
            load_scales(s_lo);
            for (int sg = s_lo; sg < s_hi && ok; ++sg) {
                const int h = (sg - s_lo) & 1;
                const uint32_t cnt = (counts >> (2 * h)) & 3;
                const uint32_t buf = C::kAccBufs == 2 ? cnt & 1 : 0, par = C::kAccBufs == 2 ? cnt >> 1 : cnt & 1;
                const float sc[2] = {__half2float(__ushort_as_half(raw0)), __half2float(__ushort_as_half(raw1))};
                if (sg + 1 < s_hi) load_scales(sg + 1);
#pragma unroll
                for (int gi = 0; gi < 2; ++gi) {
                    const int iss = h + 2 * gi;
                    ok = __all_sync(0xffffffffu, mbar_wait(dbar(iss, buf), par, err));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d_t = lane_t + (iss * C::kAccBufs + buf) * NB;
#pragma unroll
                    for (int c = 0; c < NB; c += 32) {
                        uint32_t d[32];
                        tmem_ld32(d_t + c, d);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i += 2) fma2(acc[c + i], acc[c + i + 1], d[i], d[i + 1], kGf4 ? sc[gi] : 1.f);
                    }
                    tc_fence_before();
                    mbar_arrive(ebar(iss, buf));
                }
                if (!ok) break;
                counts = (counts & ~(3u << (2 * h))) | (((cnt + 1) & 3) << (2 * h));
                if (C::kParts > 1 && sg + 1 == part_end) {      // a part of the row's sum is complete
                    if (split > 1) {        // at most two per CTA: the first waits in `total`, the second stays in `acc`
                        if (first) {
#pragma unroll
                            for (int b = 0; b < NB; ++b) { total[b] = acc[b]; acc[b] = 0.f; }
                        }
                    } else {
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            total[b] = first ? acc[b] : total[b] + acc[b];
                            acc[b] = 0.f;
                        }
                    }
                    first = false;
                    ++part;
                    part_end = part_step(nsteps, parts, part + 1);
                }
            }
            if constexpr (C::kParts > 1) {
                if (split > 1) {
                    // every group of this CTA has been folded: nothing reads the activation rings any more.
                    // Each CTA leaves its parts in its shared memory; rank k writes columns k, k + split, ...
                    const int per = C::kParts / split;
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(exch + b * 512), "f"(total[b]) : "memory");
                        if (per == 2) asm volatile("st.shared.f32 [%0], %1;" ::"r"(exch + (NB + b) * 512), "f"(acc[b]) : "memory");
                    }
                    cluster_sync();
                    for (int b = rank; b < B; b += split) {
                        float v = ld_cluster_f32(exch + b * 512, 0);
                        for (int i = 1; i < C::kParts; ++i) v += ld_cluster_f32(exch + ((i % per) * NB + b) * 512, i / per);
                        if (ok && row_raw < p.N) jq::store_out(p.y, (size_t)b * p.ldy + row_raw, fmaf(v, p.xscale[b], bias), y_dtype);
                    }
                    cluster_sync();
                    break;
                }
            }
            if (!ok) break;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const float xs_b = __shfl_sync(0xffffffffu, xs[b >> 5], b & 31);
                const float v = C::kParts > 1 ? total[C::kParts > 1 ? b : 0] : acc[b];
                acc[b] = fmaf(v, xs_b, bias);
            }
            if (row_raw < p.N) {
                for (int cpy = 0; cpy < peers.n; ++cpy) {
                    char *yb = reinterpret_cast<char *>(p.y) + jq::peer_offset(peers.delta, cpy);
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        if (b < B) jq::store_out(yb, (size_t)b * p.ldy + row_raw, acc[b], y_dtype);
                }
            }
        }
    } else {
        // =============================== MMA issuers ===============================
        // Warps 12, 13: half 0, 1; warps 14, 15: the second issuer per half.  A half's groups alternate between its
        // issuers (the first group of every 256-code step to one, the second to the other).
        // Every issuer owns a ring of activation stages (one 128-code group each) that it fills itself, so the
        // only things it ever waits for are the decode and fold threads and its own earlier work.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        const int h = (warp - 12) & 1, sub = (warp - 12) >> 1, iss = warp - 12;
        // (the warps run converged, see mma_f16_ts)
        {
            const uint32_t elected = elect_one();
            auto wait = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)); };
            constexpr uint32_t idesc = idesc_f16(kTileM, NB);
            const uint32_t lbo = (uint32_t)B * 16;
            const uint32_t ring = sbase + S::kXRing + iss * xg.ring;
            // two walks over the same sequence of groups: the loads run ahead of the MMAs
            struct Walk { int tile, pi, t_end, lo, hi, sg; const unsigned char *xp; };
            auto open_tile = [&](Walk &w) {
                while (w.tile < tile_hi) {
                    if (w.tile >= w.t_end) {
                        TaProblem p;
                        problem_at(w.pi, w.t_end, w.tile, p);
                        w.lo = step_lo(p.K >> 8);
                        w.hi = step_hi(p.K >> 8);
                        w.xp = reinterpret_cast<const unsigned char *>(p.xprep);
                    }
                    w.sg = w.lo + h;
                    if (w.sg < w.hi) return;
                    ++w.tile;
                }
            };
            auto advance = [&](Walk &w) {
                w.sg += 2;
                if (w.sg >= w.hi) { ++w.tile; open_tile(w); }
            };
            Walk ld = {tile_lo, 0, -1, 0, 0, 0, nullptr};
            open_tile(ld);
            Walk mm = ld;
            // An issuer shares its scheduler with two decode warps, so every instruction of this loop costs several clocks:
            // ring positions and parities are carried along instead of being divided out of counters, and the operand
            // descriptor is formed once per group.
            uint32_t ld_s = 0;                          // stage the next load goes to
            auto load_next = [&]() {
                if (ld.tile < tile_hi) {
                    const int G = 2 * ld.sg + sub;
                    if (elected) {
                        mbar_expect_tx(xbar(iss, ld_s), xg.chunk);
                        bulk_g2s(ring + ld_s * xg.chunk, ld.xp + (size_t)G * xg.chunk, xg.chunk, xbar(iss, ld_s));
                    }
                    __syncwarp();
                    advance(ld);
                }
                ld_s = (ld_s + 1 == (uint32_t)xg.nstages) ? 0 : ld_s + 1;
            };
            pdl_wait();
            for (int i = 0; i < xg.nstages; ++i) load_next();
            bool ok = true;
            uint32_t cs = 0, cpar = 0;                  // stage and phase parity of the group being multiplied
            uint32_t slot = (uint32_t)sub % kRing, spar = 0;   // A slot of this issuer's next group (the half's group count t = 2 n + sub)
            uint32_t db = 0, dpar = 1;                  // accumulator (the first round finds it free)
            const bool tight = xg.nstages <= C::kAccBufs;
            const uint32_t desc_step = (2 * lbo) >> 4;  // descriptor address field per K = 16 slice
            for (uint32_t n = 0; mm.tile < tile_hi && ok; ++n) {
                // a ring with no more stages than accumulators refills the previous group's stage once its MMAs are done
                if (tight && n > 0) {
                    if (!(ok = wait(dbar(iss, (n - 1) % C::kAccBufs), ((n - 1) / C::kAccBufs) & 1))) break;
                    load_next();
                }
                // the accumulator's last group has been folded, so its MMAs have read their activation stage: refill that
                if (!(ok = wait(ebar(iss, db), dpar))) break;
                if (!tight && n >= (uint32_t)C::kAccBufs) load_next();
                if (!(ok = wait(xbar(iss, cs), cpar))) break;
                if (!(ok = wait(abar(h, slot), spar))) break;
                tc_fence_after();
                const uint32_t a_t = tmem + (h * kRing + slot) * 64;
                const uint32_t d_t = tmem + C::kAcc + (iss * C::kAccBufs + db) * NB;
                const uint64_t desc0 = smem_desc(ring + cs * xg.chunk, lbo, 128);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    mma_f16_ts(elected, d_t, a_t + 8 * i, desc0 + (uint64_t)(i * desc_step), idesc, i > 0);
                mma_commit(elected, dbar(iss, db));
                if (++cs == (uint32_t)xg.nstages) { cs = 0; cpar ^= 1; }
                if (++db == (uint32_t)C::kAccBufs) { db = 0; dpar ^= 1; }
                slot += 2;
                if (slot >= (uint32_t)kRing) { slot -= kRing; spar ^= 1; }
                advance(mm);
            }
        }
        if (split > 1) { __syncwarp(); cluster_sync(); cluster_sync(); }
    }

    // ---- teardown
    if (*err) {   // a wait gave up: let the copies still in flight land before the CTA's shared memory goes away
        for (int i = 0; i < 400; ++i) __nanosleep(256);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_err) atomicExch(status, s_err);
    if (warp == 15) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace wide

// ---- GF4, batch 1 on the CUDA cores (B is 1; sums and partial sums are laid out for two rows) ----
// Per-row pair tables as in the tensor-memory kernel for up to 16 rows, but tiles of 64 rows, a weight ring per warp, and the
// multiply-accumulate stays in the decode threads: lane = weight row, so all lanes of a warp need the same
// activation values, which they read as broadcast 16-byte shared-memory loads (one wavefront per eight
// codes) from the prepared activation of the whole problem, and a looked-up pair feeds two
// fma.rn.f32.f16 (fp16 x fp16 exact, fp32 accumulation).  Per 128-code group the partial sum is scaled by
// the group's fp16 scale in fp32.  At batch 1 the loop costs about 2.2 instructions and 0.75 shared-memory
// wavefronts per code of a warp, where one 16-bit lookup per code costs 1.2 wavefronts; a whole launch 1.17
// (tables, partial sums and syncs 0.25, global loads 0.17, most of them the scales' 2-byte loads), with the
// LSU data pipe 74 % busy (11008 x 4096, 122 us for 16); the tensor pipe, whose K = 16 instructions have a
// floor of about 45 clocks whatever the batch, is not involved.
// Per code a lane receives 2 bytes of looked-up pairs, 0.5 of packed weights and 2 of activations through
// the shared-memory pipe (128 bytes per clock and SM).  A variant whose lanes carry two rows each and read
// the activations once for both (8 warps instead of 16, same tables and ring) was slower: 950 against 1022
// tokens/s on the 7B-shaped stack.
constexpr int kLutQuarters = 2;                      // 32-row sets of a tile (each has its own pair table)
constexpr int kLutTileM = 32 * kLutQuarters;
constexpr int kLutSplit = 8;                         // warps that share a row set, each taking every 8th 256-code step
constexpr int kLutWarps = kLutQuarters * kLutSplit;
constexpr int kLutThreads = kLutWarps * 32;
constexpr int kLutStage = 32 * 128;                   // a weight stage: 32 rows x 128 bytes (two 128-code groups), 128-byte swizzle
constexpr int kLutSW = 2;                            // stages per warp (16 warps x 2 x 4 KB: this TMA pattern streams at 6.5 TB/s when
                                                     // nothing else limits it; 64-byte boxes four deep reached only 4.3 TB/s)
struct LutSmem {
    static constexpr int kTab = 0;
    static constexpr int kWRing = kTab + kLutQuarters * 256 * 128;
    static constexpr int kX = kWRing + kLutWarps * kLutSW * kLutStage;   // prepared activation of the current problem
    static constexpr int kXBytes = 24 * 1024;
    static constexpr int kPart = kX + kXBytes;                           // partial sums of the other warps of a row set, two tiles
    static constexpr int kBars = kPart + 2 * (kLutSplit - 1) * kLutTileM * 2 * 4;
    static constexpr int kNumBars = kLutWarps * kLutSW + kLutQuarters + 2;   // weights, row-set sync, x free / x full
    static constexpr int kBytes = kBars + kNumBars * 8 + 1024;
};

// acc0 += lo(w) * lo(x), acc1 += hi(w) * hi(x): fp16 operands, exact products, fp32 accumulation
__device__ __forceinline__ void fma_pair(float &acc0, float &acc1, uint32_t w, uint32_t x) {
    asm("{ .reg .b16 wl, wh, xl, xh; mov.b32 {wl, wh}, %2; mov.b32 {xl, xh}, %3;\n"
        "  fma.rn.f32.f16 %0, wl, xl, %0; fma.rn.f32.f16 %1, wh, xh, %1; }"
        : "+f"(acc0), "+f"(acc1) : "r"(w), "r"(x));
}

// kOwn: a single call, which prepares its activation itself (a kernel of its own, as the grouped one gets 0.7 % slower with that
// code in it)
template <int B, bool kOwn>
__global__ void __launch_bounds__(kLutThreads, 1) gf4_lut2_kernel(const TaProblem *probs, const CUtensorMap *maps,
                                                                  const __grid_constant__ TaProblem single,
                                                                  const __grid_constant__ CUtensorMap single_map,
                                                                  int nprob, const int *tile_start, const int *cta_first,
                                                                  int x_dtype, int y_dtype, PeerInfo peers, int *status) {
    using S = LutSmem;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float s_max[kLutWarps];
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *sgen = smem_raw + (sbase - smem_u32(smem_raw));
    const uint32_t bars = sbase + S::kBars;
    auto wbar = [&](int w, int s) { return bars + 8u * (w * kLutSW + s); };
    auto qbar = [&](int q) { return bars + 8u * (kLutWarps * kLutSW + q); };
    const uint32_t xfree = bars + 8u * (kLutWarps * kLutSW + kLutQuarters), xfull = xfree + 8;
    volatile int *err = &s_err;
    if (tid == 0) {
        s_err = 0;
        for (int w = 0; w < kLutWarps; ++w)
            for (int s = 0; s < kLutSW; ++s) mbar_init(wbar(w, s), 1);
        for (int q = 0; q < kLutQuarters; ++q) mbar_init(qbar(q), 32 * kLutSplit);
        mbar_init(xfree, kLutThreads);
        mbar_init(xfull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    int tile_lo, tile_hi;
    if (nprob == 0) {
        const int nt = (single.N + kLutTileM - 1) / kLutTileM;
        tile_lo = (int)((long long)nt * blockIdx.x / gridDim.x);
        tile_hi = (int)((long long)nt * (blockIdx.x + 1) / gridDim.x);
    } else {
        tile_lo = cta_first[blockIdx.x];
        tile_hi = cta_first[blockIdx.x + 1];
    }
    // Problems change rarely along a CTA's tile sequence, so every walker keeps its current problem's fields
    // in registers and goes back to global memory only when a tile lies beyond that problem's last tile.
    auto problem_at = [&](int &pi, int &t_end, int tile, TaProblem &p) {
        if (nprob == 0) { p = single; t_end = 0x7fffffff; return; }
        if (t_end < 0) {
            // first look-up of a walker: bisect (a step's list can hold hundreds of problems, and a scan from the
            // first one is a chain of dependent global loads, 0.2 us each, in front of the last CTAs' first tile)
            int lo = 0, hi = nprob - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (tile_start[mid] <= tile) lo = mid; else hi = mid - 1;
            }
            pi = lo;
        } else {
            while (pi + 1 < nprob && tile_start[pi + 1] <= tile) ++pi;
        }
        p = probs[pi];
        t_end = tile_start[pi + 1];
    };

    const int q = warp % kLutQuarters, h = warp / kLutQuarters;   // row set of the tile, which groups (g % kLutSplit == h)
    const int r = q * 32 + lane;
    const uint32_t tcol = sbase + S::kTab + q * (256 * 128) + lane * 4;
    const uint32_t wring = sbase + S::kWRing + warp * (kLutSW * kLutStage);
    // 16-byte piece c of this lane's row sits at piece c ^ (lane & 7) of the row (128-byte swizzle)
    const uint32_t lrow = lane * 128, lkey = (lane & 7) << 4;
    const uint32_t xs_u = sbase + S::kX;

    // ---- producer side of the weight ring: steps of this warp are 256 codes each (steps h, h + 8, ... of a row)
    int i_tile = tile_lo, i_pi = 0, i_tend = -1, i_j = 0, i_n = 0, i_x = 0, i_y = 0, i_tile0 = 0, i_steps = 0, i_stage = 0;
    const void *i_map = nullptr;
    auto i_open = [&]() {   // position on step 0 of tile i_tile
        while (i_tile < tile_hi) {
            if (i_tile >= i_tend) {
                TaProblem p;
                problem_at(i_pi, i_tend, i_tile, p);
                i_steps = ((p.K >> 8) - h + kLutSplit - 1) / kLutSplit;
                i_tile0 = p.tile0;
                i_map = nprob ? &maps[i_pi] : &single_map;
            }
            i_n = i_steps;
            i_x = h * 128;
            i_y = (i_tile - i_tile0) * kLutTileM + q * 32;     // rows past N read as zeros
            i_j = 0;
            if (i_n > 0) return;
            ++i_tile;
        }
    };
    auto issue = [&]() {
        if (i_tile < tile_hi) {
            if (lane == 0) {
                const uint32_t bar = wbar(warp, i_stage);
                mbar_expect_tx(bar, kLutStage);
                tma_2d_g2s(wring + i_stage * kLutStage, i_map, i_x, i_y, bar);
            }
            i_x += 128 * kLutSplit;
            if (++i_j == i_n) { ++i_tile; i_open(); }
        }
        i_stage = (i_stage + 1 == kLutSW) ? 0 : i_stage + 1;
    };
    i_open();
#pragma unroll
    for (int s = 0; s < kLutSW; ++s) issue();

    uint32_t wcount = 0, qcount = 0, xcount = 0;
    // ---- the codebook of this lane's row, one tile ahead
    int f_pi = 0, f_tend = -1, f_tile0 = 0, f_N = 1;
    const __half *f_cb = nullptr;
    uint4 cb0 = make_uint4(0, 0, 0, 0), cb1 = cb0;
    auto fetch_codebook = [&](int tile) {
        if (tile < tile_hi) {
            if (tile >= f_tend) {
                TaProblem p;
                problem_at(f_pi, f_tend, tile, p);
                f_tile0 = p.tile0; f_N = p.N; f_cb = p.codebook;
            }
            const int row = min((tile - f_tile0) * kLutTileM + r, f_N - 1);
            const uint4 *src = reinterpret_cast<const uint4 *>(f_cb + (size_t)row * 16);
            cb0 = __ldg(src);
            cb1 = __ldg(src + 1);
        }
    };
    auto quarter_sync = [&]() -> bool {
        mbar_arrive(qbar(q));
        const bool ok = mbar_wait(qbar(q), qcount & 1, err);
        ++qcount;
        return ok;
    };

    // ---- a finished tile whose outputs are written after the next row-set sync (first warp of the row set)
    float *part_s = reinterpret_cast<float *>(sgen + S::kPart);      // [2 parities][kLutSplit - 1][kLutTileM][2]
    constexpr int kPartStride = (kLutSplit - 1) * kLutTileM * 2;
    bool have_prev = false;
    float prev_acc[B], prev_xsc[B], prev_bias = 0.f;
    int prev_row = 0, prev_N = 0, prev_ldy = 0;
    void *prev_y = nullptr;
    auto write_prev = [&](int parity) {
        if (have_prev && h == 0 && prev_row < prev_N) {
            const float *ps = part_s + parity * kPartStride;
#pragma unroll
            for (int b = 0; b < B; ++b) {
                float v = prev_acc[b];
#pragma unroll
                for (int hh = 1; hh < kLutSplit; ++hh) v += ps[((hh - 1) * kLutTileM + r) * 2 + b];
                const float o = fmaf(v, prev_xsc[b], prev_bias);
                jq::store_out_copies(prev_y, peers.delta, peers.n, (size_t)b * prev_ldy + prev_row, o, y_dtype);
            }
        }
        have_prev = false;
    };

    int c_pi = 0, c_tend = -1, x_pi = -1;
    TaProblem p = single;
    fetch_codebook(tile_lo);
    float own_scale = 0.f;
    if constexpr (kOwn) {
        // in every CTA, as ta_prepare_kernel does (same operations, same bits): a launch in front of this one and the way
        // through memory cost more than the few hundred elements per warp (4096 x 4096: 15.9 -> 13.5 us per call)
        static_assert(B == 1, "one row");
        constexpr int kMost = (S::kXBytes / 2 / 128 + kLutWarps - 1) / kLutWarps;     // blocks of 128 elements per warp
        float v[kMost][4], m = 0.f;
#pragma unroll
        for (int i = 0; i < kMost; ++i) {
            const int k0 = (warp + i * kLutWarps) * 128 + lane * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[i][j] = k0 < p.K ? jq::load_act(p.x, (size_t)k0 + j, x_dtype) : 0.f;
                m = fmaxf(m, fabsf(v[i][j]));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) s_max[warp] = m;
        __syncthreads();
        m = s_max[0];
#pragma unroll
        for (int w = 1; w < kLutWarps; ++w) m = fmaxf(m, s_max[w]);
        const int ex = act_exponent(m, p.had != 0);
        own_scale = __uint_as_float((uint32_t)(127 + ex) << 23);
        const float down = __uint_as_float((uint32_t)(127 - ex) << 23);
#pragma unroll
        for (int i = 0; i < kMost; ++i) {
            const int blk = warp + i * kLutWarps;
            if (blk * 128 < p.K) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] *= down;
                if (p.had) jq::fwht128_warp(v[i], lane);
                const __half2 h01 = __floats2half2_rn(v[i][0], v[i][1]), h23 = __floats2half2_rn(v[i][2], v[i][3]);
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(xs_u + (blk * 128 + lane * 4) * 2),
                             "r"(*reinterpret_cast<const uint32_t *>(&h01)), "r"(*reinterpret_cast<const uint32_t *>(&h23)) : "memory");
            }
        }
        __syncthreads();
        x_pi = 0;
    }
    if (!kOwn) pdl_wait();          // from here on the prepared activation and its row factors are read
    bool ok = true;
    int tparity = 0;
    for (int tile = tile_lo; tile < tile_hi && ok; ++tile, tparity ^= 1) {
        if (tile >= c_tend) problem_at(c_pi, c_tend, tile, p);
        const int row_raw = (tile - p.tile0) * kLutTileM + r;
        const int row = min(row_raw, p.N - 1);
        // ---- a new problem: its prepared activation replaces the previous one in shared memory
        if (c_pi != x_pi) {
            mbar_arrive(xfree);                                      // this thread no longer reads the old activation
            if (tid == 0) {
                if ((ok = mbar_wait(xfree, xcount & 1, err))) {
                    const uint32_t bytes = (uint32_t)p.K * B * 2;
                    fence_async_smem();
                    mbar_expect_tx(xfull, bytes);
                    bulk_g2s(xs_u, p.xprep, bytes, xfull);
                }
            }
            ok = mbar_wait(xfull, xcount & 1, err);
            ++xcount;
            x_pi = c_pi;
            if (!ok) break;
        }
        // ---- row-set sync: the previous tile's lookups are over (its table may go) and its partial sums are visible
        if (!(ok = quarter_sync())) break;
        write_prev(tparity ^ 1);
        // ---- the pair table of this row: this thread fills the entries whose second code is 2 h or 2 h + 1
        {
            const uint32_t c[8] = {cb0.x, cb0.y, cb0.z, cb0.w, cb1.x, cb1.y, cb1.z, cb1.w};
            uint32_t ch = c[0];                                      // the pair register holding entries 2 h, 2 h + 1
#pragma unroll
            for (int hh = 1; hh < kLutSplit; ++hh) ch = (h == hh) ? c[hh] : ch;
            const uint32_t tb = tcol + h * (32 * 128);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int lo = 0; lo < 16; ++lo) {
                    const uint32_t e = __byte_perm(c[lo >> 1], ch,
                                                   ((lo & 1) ? 0x32u : 0x10u) | (((i & 1) ? 0x76u : 0x54u) << 8));
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(tb + (i * 16 + lo) * 128), "r"(e) : "memory");
                }
        }
        fetch_codebook(tile + 1);
        float acc[B], xsc[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            acc[b] = 0.f;
            xsc[b] = kOwn ? own_scale : p.xscale[b];                // in flight during the tile, needed at its end
        }
        const float bias = (p.bias && row_raw < p.N) ? p.bias[row_raw] : 0.f;
        const int nsteps = ((p.K >> 8) - h + kLutSplit - 1) / kLutSplit;
        const unsigned short *srow = reinterpret_cast<const unsigned short *>(p.scales) + (size_t)row * p.lds;
        const int gshift = 31 - __clz(p.g >> 7);
        if (!(ok = quarter_sync())) break;                           // the table is complete
        for (int j = 0; j < nsteps && ok; ++j) {
            const int stage = wcount % kLutSW;
            ok = __all_sync(0xffffffffu, mbar_wait(wbar(warp, stage), (wcount / kLutSW) & 1, err));
            if (!ok) break;
            ++wcount;
            const uint32_t slot = wring + stage * kLutStage + lrow;
#pragma unroll
            for (int gi = 0; gi < 2; ++gi) {
            const int grp = 2 * (kLutSplit * j + h) + gi;
            const unsigned short scale_raw = __ldg(srow + (grp >> gshift));
            const uint32_t xg0 = xs_u + (uint32_t)grp * (256 * B);   // the group's activations: [16 pieces][B][16 bytes]
            float part[B][4];
#pragma unroll
            for (int b = 0; b < B; ++b) part[b][0] = part[b][1] = part[b][2] = part[b][3] = 0.f;
#pragma unroll
            for (int pc = 0; pc < 4; ++pc) {                         // 32 codes
                const uint4 w4 = lds128(slot + (((gi * 4 + pc) << 4) ^ lkey));
#pragma unroll
                for (int wi = 0; wi < 4; ++wi) {                     // 8 codes
                    const uint32_t w = wi == 0 ? w4.x : (wi == 1 ? w4.y : (wi == 2 ? w4.z : w4.w));
                    uint32_t v[4];
#pragma unroll
                    for (int bj = 0; bj < 4; ++bj) v[bj] = lds32(dp4a_u(w, 0x80u << (8 * bj), tcol));
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        const uint4 xv = lds128(xg0 + (uint32_t)(((pc * 4 + wi) * B + b) * 16));
                        fma_pair(part[b][0], part[b][1], v[0], xv.x);
                        fma_pair(part[b][2], part[b][3], v[1], xv.y);
                        fma_pair(part[b][0], part[b][1], v[2], xv.z);
                        fma_pair(part[b][2], part[b][3], v[3], xv.w);
                    }
                }
            }
            const float sc = __half2float(__ushort_as_half(scale_raw));
#pragma unroll
            for (int b = 0; b < B; ++b)
                acc[b] = fmaf((part[b][0] + part[b][1]) + (part[b][2] + part[b][3]), sc, acc[b]);
            }
            __syncwarp();
            fence_async_smem();
            issue();
        }
        if (!ok) break;
        // ---- the other warps of the row set park their sums; the first keeps what it needs for the outputs
        if (h > 0) {
            float *ps = part_s + tparity * kPartStride;
#pragma unroll
            for (int b = 0; b < B; ++b) ps[((h - 1) * kLutTileM + r) * 2 + b] = acc[b];
        } else {
#pragma unroll
            for (int b = 0; b < B; ++b) { prev_acc[b] = acc[b]; prev_xsc[b] = xsc[b]; }
            prev_bias = bias; prev_row = row_raw; prev_N = p.N; prev_ldy = p.ldy; prev_y = p.y;
        }
        have_prev = true;
    }
    if (ok && have_prev && (ok = quarter_sync())) write_prev(tparity ^ 1);
    if (*err) {
        for (int i = 0; i < 400; ++i) __nanosleep(256);
    }
    __syncthreads();
    if (tid == 0 && s_err) atomicExch(status, s_err);
}


}  // namespace jqta

using namespace jqta;

// ---- host side -------------------------------------------------------------------
// plan layout: 12 ints [magic, n, grid, NB, tensor-map offset (bytes), B, fmt, problem offset (bytes),
// largest K, 0, 0, 0],
// tile_start[n + 1], cta_first[grid + 1], padding to 64 bytes, TaProblem[n], padding to 64 bytes, CUtensorMap[n]
static const int kTaMagic = 0x4a515441;
// fixed time per tile / per problem of the partition's cost model, in codes of one row, for gf4_lut2_kernel.  Swept on the 7B-shaped
// GF4 step (us per step on one GPU / for an eighth of it): bytes only 940 / 150.5; 384, 2048: 921.5 / 143.0;
// 768, 4096: 910.1 / 141.3; 1408, 6144: 900.1 / 140.1; 2304, 8192: 943.3 / 143.9.
static const double kLutTileCost = 1408, kLutProblemCost = 6144;
// The same for the tensor-memory kernels, whose loads and decode warps run across tile boundaries.  Swept in turn on one GPU, us
// per step, 7B-shaped GF4 (32 layers), 70B-shaped E2M1 (7 layers) and 7B-shaped E2M1 (16 layers):
//                    GF4, rows 8   24     48     E2M1 70B, rows 16   24    48      E2M1 7B, rows 24   48
//     1408, 6144          968     1613   2016                  918   971   1216                 522   702
//      700, 3000          935     1500   1989                  853   913   1166                 507   706
//      400, 3000          939     1494   2005                  849   908   1198                 511   711
//      300, 3000          943     1507   2004                  855   914   1193                 512   712
//        0,    0          957     1517   2009                  851   913   1192                 518   714
// (runs of one side differ by 1 to 3 % where the power cap holds the clock: all but GF4 with 24 rows)
static const double kTaTileCost = 400, kTaProblemCost = 3000;
static const int kTaHeader = 12;

// MMA N
static int ta_cols(int B) { return B <= 16 ? 16 : (B <= 32 ? 32 : (B <= 64 ? 64 : 0)); }

static bool ta_use_lut(int B, int maxK);
static size_t ta_align(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Tensor map over the packed rows of one matrix: bytes [N rows][ldw], boxes of rows x 128 bytes with the
// 128-byte swizzle; rows past N read as zeros.  The driver entry point is looked up once (no link-time
// dependency on the driver library).
static int ta_encode_map(CUtensorMap *out, const void *qw, int N, int ldw, int rows) {
    ta_encode_fn enc = ta_encoder();
    if (!enc) return JQ_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)ldw, (cuuint64_t)N};
    const cuuint64_t strides[1] = {(cuuint64_t)ldw};
    const cuuint32_t box[2] = {128, (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(qw), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? JQ_OK : JQ_ERR_CUDA_BASE - (int)cudaErrorInvalidValue;
}

static bool ta_shape_ok(int fmt, int N, int K, int g, int had) {
    if (N <= 0 || K < 512 || K % 256) return false;
    if (had != 0 && had != 128) return false;
    if (fmt == JQ_FMT_GF4) {
        const int gq = g >> 7;
        return g >= 128 && g % 128 == 0 && (gq & (gq - 1)) == 0 && K % g == 0;
    }
    return fmt == JQ_FMT_E2M1 && g == 32;
}

// batch 1 runs on the CUDA cores when the prepared activation of one problem fits its shared-memory buffer (K up to 12288).
// The line is older than the tensor-memory kernel of 24 warps, against whose predecessor this was 931 us to 1114 on the
// 7B-shaped step.  Now the CUDA cores are ahead for single calls of few tiles, which take one launch instead of two, and behind
// elsewhere (one row, us, CUDA cores / tensor memory): single calls 1024 x 1024 18.9 / 24.0, 4096 x 4096 14.7 / 17.3, 11008 x 4096
// 20.9 / 17.6, 4096 x 11008 21.2 / 17.6, 32000 x 4096 32.0 / 28.5; 7B-shaped step 956 / 836.  The two add a row's products in
// another order, so that moving the line changes last bits of one-row results.
static bool ta_use_lut(int B, int maxK) { return B == 1 && (size_t)maxK * 2 <= (size_t)LutSmem::kXBytes; }

extern "C" size_t jq_ta_workspace_bytes(const jq_problem *ph, int n, int B) {
    if (!ph || n <= 0 || B < 1 || B > 64) return 0;
    size_t total = kHeaderBytes;
    for (int i = 0; i < n; ++i) total += 256 + ta_align((size_t)ph[i].K * B * 2, 128);
    return total;
}

extern "C" size_t jq_ta_plan_bytes(int n) {
    if (n <= 0) return 0;
    return ta_align(ta_align(((size_t)kTaHeader + (size_t)(n + 1) + (size_t)jq_sm_count() + 1) * sizeof(int), 64) +
                        (size_t)n * sizeof(TaProblem), 64) + (size_t)n * sizeof(CUtensorMap);
}

static int ta_fill_problem(TaProblem &t, int fmt, const jq_problem &p, unsigned char *ws, size_t &off, int B) {
    if (!p.qweight || !p.x || !p.y || !p.scales) return JQ_ERR_NULL_PTR;
    if (fmt == JQ_FMT_GF4 && !p.codebook) return JQ_ERR_NULL_PTR;
    if (!ta_shape_ok(fmt, p.N, p.K, p.g, p.had_block)) return JQ_ERR_UNSUPPORTED;
    if (!jq_aligned16(p.qweight) || (fmt == JQ_FMT_GF4 && !jq_aligned16(p.codebook)) ||
        (reinterpret_cast<uintptr_t>(p.scales) & (fmt == JQ_FMT_E2M1 ? 15u : 1u)))
        return JQ_ERR_BAD_ALIGN;
    t.qw = reinterpret_cast<const uint8_t *>(p.qweight);
    t.scales = reinterpret_cast<const __half *>(p.scales);
    t.codebook = reinterpret_cast<const __half *>(p.codebook);
    t.x = p.x;
    t.bias = p.bias;
    t.y = p.y;
    t.xscale = reinterpret_cast<float *>(ws + off);
    off += 256;   // up to 64 batch rows
    t.xprep = reinterpret_cast<__half *>(ws + off);
    off += ta_align((size_t)p.K * B * 2, 128);
    t.N = p.N; t.K = p.K; t.g = p.g; t.had = p.had_block;
    t.ldw = p.K >> 1;
    t.lds = p.K / p.g;
    t.ldy = p.ldy > 0 ? p.ldy : p.N;
    t.tile0 = 0;
    return JQ_OK;
}

extern "C" int jq_ta_plan(int fmt, const jq_problem *ph, int n, int B, void *workspace_dev, size_t workspace_bytes,
                          void *plan_host, size_t plan_bytes) {
    if (!ph || !plan_host || !workspace_dev) return JQ_ERR_NULL_PTR;
    if (n <= 0 || B < 1) return JQ_ERR_BAD_SHAPE;
    if ((fmt != JQ_FMT_GF4 && fmt != JQ_FMT_E2M1) || !ta_cols(B)) return JQ_ERR_UNSUPPORTED;
    if (plan_bytes < jq_ta_plan_bytes(n) || workspace_bytes < jq_ta_workspace_bytes(ph, n, B)) return JQ_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(workspace_dev) & 127u) return JQ_ERR_BAD_ALIGN;
    const int grid = jq_sm_count();
    int *h = reinterpret_cast<int *>(plan_host);
    int *tile_start = h + kTaHeader, *cta_first = tile_start + n + 1;
    const size_t poff = ta_align(((size_t)kTaHeader + (n + 1) + grid + 1) * sizeof(int), 64);
    const size_t moff = ta_align(poff + (size_t)n * sizeof(TaProblem), 64);
    TaProblem *tp = reinterpret_cast<TaProblem *>(reinterpret_cast<unsigned char *>(plan_host) + poff);
    unsigned char *maps = reinterpret_cast<unsigned char *>(plan_host) + moff;
    size_t off = kHeaderBytes;
    double total = 0;
    int maxK = 0;
    for (int i = 0; i < n; ++i) maxK = ph[i].K > maxK ? ph[i].K : maxK;
    const bool lut = fmt == JQ_FMT_GF4 && ta_use_lut(B, maxK);
    const int tile_m = lut ? kLutTileM : kTileM;
    const double tile_cost = lut ? kLutTileCost : kTaTileCost, problem_cost = lut ? kLutProblemCost : kTaProblemCost;
    tile_start[0] = 0;
    for (int i = 0; i < n; ++i) {
        int st = ta_fill_problem(tp[i], fmt, ph[i], reinterpret_cast<unsigned char *>(workspace_dev), off, B);
        if (st) return st;
        CUtensorMap tm;
        st = ta_encode_map(&tm, ph[i].qweight, ph[i].N, ph[i].K >> 1, (lut || B > NB) ? 32 : kTileM);
        if (st) return st;
        memcpy(maps + (size_t)i * sizeof(CUtensorMap), &tm, sizeof(CUtensorMap));
        const int tiles = (ph[i].N + tile_m - 1) / tile_m;
        tp[i].tile0 = tile_start[i];
        tile_start[i + 1] = tile_start[i] + tiles;
        total += (double)tiles * (ph[i].K + tile_cost) + problem_cost;
    }
    // contiguous tile ranges of (nearly) equal cost: cut where the running cost passes c * total / grid.  A tile
    // costs its packed bytes plus a fixed part (table build, two syncs, outputs), a problem's first tile also the
    // switch of the activation buffer: with bytes alone a CTA of short rows ran 10 % longer than one of long rows.
    int cta = 0;
    double acc = 0;
    cta_first[0] = 0;
    for (int i = 0; i < n; ++i)
        for (int t = tile_start[i]; t < tile_start[i + 1]; ++t) {
            const double c = ph[i].K + tile_cost + (t == tile_start[i] ? problem_cost : 0);
            while (cta + 1 < grid && acc + 0.5 * c >= total * (cta + 1) / grid) cta_first[++cta] = t;
            acc += c;
        }
    while (cta < grid) cta_first[++cta] = tile_start[n];
    h[0] = kTaMagic; h[1] = n; h[2] = grid; h[3] = ta_cols(B); h[4] = (int)moff; h[5] = B; h[6] = fmt; h[7] = (int)poff;
    h[8] = maxK; h[9] = h[10] = h[11] = 0;
    return JQ_OK;
}

// launch configuration of a main kernel: allowed to start while the preparation kernel in front of it still runs;
// cluster: CTAs that share a tile
static void ta_pdl_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&attr)[2], int grid, int threads, int smem, int cluster,
                          cudaStream_t st) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
}

static int ta_prepare(const TaProblem *probs_dev, const TaProblem &single, int nblk, int B, int x_dtype, cudaStream_t st) {
    // up to two blocks of 32 warps per SM.  Single calls, with values loaded one by one by 8 warps before: 4096 x 11008 E2M1, 23
    // rows, 16.8 -> 14.8 us; 4096 x 14336, 16 rows, 18.0 -> 14.8; the 7B-shaped GF4 step with 8 rows (1792 blocks of 8 warps,
    // loads of four values) 1.3 % less.
    const bool wide = nblk <= 2 * jq_sm_count() || B <= 2;
    void (*const kernels[3][2])(const TaProblem *, TaProblem, int) = {
        {ta_prepare_kernel<256, float>, ta_prepare_kernel<1024, float>},
        {ta_prepare_kernel<256, __half>, ta_prepare_kernel<1024, __half>},
        {ta_prepare_kernel<256, __nv_bfloat16>, ta_prepare_kernel<1024, __nv_bfloat16>}};
    kernels[x_dtype][wide]<<<nblk, wide ? 1024 : 256, 0, st>>>(probs_dev, single, B);
    return jq_launch_status();
}

template <int FMT, int COLS>
static int ta_launch(const TaProblem *probs_dev, const CUtensorMap *maps_dev, const TaProblem &single,
                     const CUtensorMap &single_map, int nprob, const int *tile_start,
                     const int *cta_first, int grid, int B, int x_dtype, int y_dtype, const jqta::PeerInfo &peers,
                     int *status, cudaStream_t st) {
    const int s = ta_prepare(probs_dev, single, (nprob ? nprob : 1) * B, B, x_dtype, st);
    if (s) return s;
    void (*kern)(const TaProblem *, const CUtensorMap *, const TaProblem, const CUtensorMap, int, const int *, const int *, int, int,
                 jqta::PeerInfo, int, int *);
    int smem, threads;
    constexpr int parts = COLS == 64 ? 1 : 4;
    if constexpr (COLS == NB) {
        kern = gemm_ta_kernel<FMT>;
        smem = Smem<FMT == JQ_FMT_GF4>::kBytes;
        threads = kTaThreads;
    } else {
        kern = wide::gemm_ta_wide_kernel<FMT, COLS>;
        smem = wide::Smem::kBytes;
        threads = wide::kTaThreads;
    }
    // A single matrix with few tiles: 4 or 2 CTAs take parts of every row (N = 4096 is 32 tiles for 148 SMs)
    int split = 1;
    if (!nprob && parts == 4 && (single.K >> 8) >= kPartMinSteps)
        split = grid * 4 <= jq_sm_count() ? 4 : (grid * 2 <= jq_sm_count() ? 2 : 1);
    static jq_contexts done;
    JQ_CUDA_TRY(jq_allow_smem(reinterpret_cast<const void *>(kern), smem, done));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    ta_pdl_config(cfg, attr, grid * split, threads, smem, split, st);
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, probs_dev, maps_dev, single, single_map, nprob, tile_start, cta_first, B, y_dtype,
                                   peers, split, status));
    return jq_launch_status();
}

// One row whose outputs are written over (part of) its own activation.  Such a call has its activation prepared by a launch in
// front: where every CTA reads the row itself, another may already be writing to it.
static bool ta_outputs_on_inputs(const TaProblem &p, int x_dtype, int y_dtype) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(p.x), y = reinterpret_cast<uintptr_t>(p.y);
    return x < y + (uintptr_t)p.N * (y_dtype == JQ_F32 ? 4 : 2) && y < x + (uintptr_t)p.K * (x_dtype == JQ_F32 ? 4 : 2);
}

template <int B>
static int lut2_launch(const TaProblem *probs_dev, const CUtensorMap *maps_dev, const TaProblem &single,
                       const CUtensorMap &single_map, int nprob, const int *tile_start, const int *cta_first, int grid,
                       int x_dtype, int y_dtype, const jqta::PeerInfo &peers, int *status, cudaStream_t st) {
    const bool own = !nprob && !ta_outputs_on_inputs(single, x_dtype, y_dtype);
    if (!own) {
        const int s = ta_prepare(probs_dev, single, (nprob ? nprob : 1) * B, B, x_dtype, st);
        if (s) return s;
    }
    auto kern = own ? gf4_lut2_kernel<B, true> : gf4_lut2_kernel<B, false>;
    constexpr int smem = LutSmem::kBytes;
    static_assert(smem <= 227 * 1024, "shared memory");
    static jq_contexts done[2];
    JQ_CUDA_TRY(jq_allow_smem(reinterpret_cast<const void *>(kern), smem, done[own ? 1 : 0]));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    ta_pdl_config(cfg, attr, grid, kLutThreads, smem, 1, st);
    if (own) cfg.numAttrs = 0;         // the activation is read from the start: after everything in front of it
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, probs_dev, maps_dev, single, single_map, nprob, tile_start, cta_first, x_dtype,
                                   y_dtype, peers, status));
    return jq_launch_status();
}

static int ta_dispatch(int fmt, int nb, int maxK, const TaProblem *probs_dev, const CUtensorMap *maps_dev, const TaProblem &single,
                       const CUtensorMap &single_map, int nprob,
                       const int *tile_start, const int *cta_first, int grid, int B, int x_dtype, int y_dtype,
                       const jqta::PeerInfo &peers, int *status, cudaStream_t st) {
#define JQ_TA_ARGS probs_dev, maps_dev, single, single_map, nprob, tile_start, cta_first, grid, B, x_dtype, y_dtype, peers, status, st
    if (fmt == JQ_FMT_GF4) {
        if (ta_use_lut(B, maxK)) {
            return lut2_launch<1>(probs_dev, maps_dev, single, single_map, nprob, tile_start, cta_first, grid, x_dtype, y_dtype, peers, status, st);
        }
        if (nb == 16) return ta_launch<JQ_FMT_GF4, 16>(JQ_TA_ARGS);
        if (nb == 32) return ta_launch<JQ_FMT_GF4, 32>(JQ_TA_ARGS);
        if (nb == 64) return ta_launch<JQ_FMT_GF4, 64>(JQ_TA_ARGS);
        return JQ_ERR_UNSUPPORTED;
    }
    if (nb == 16) return ta_launch<JQ_FMT_E2M1, 16>(JQ_TA_ARGS);
    if (nb == 32) return ta_launch<JQ_FMT_E2M1, 32>(JQ_TA_ARGS);
    if (nb == 64) return ta_launch<JQ_FMT_E2M1, 64>(JQ_TA_ARGS);
#undef JQ_TA_ARGS
    return JQ_ERR_UNSUPPORTED;
}

extern "C" int jq_gemm_ta_grouped(const void *plan_host, const void *plan_dev, void *workspace_dev, int x_dtype,
                                  int y_dtype, int npeer, const int64_t *peer_delta, jq_stream_t stream) {
    if (!plan_host || !plan_dev || !workspace_dev || !peer_delta) return JQ_ERR_NULL_PTR;
    if (npeer < 1 || npeer > 8) return JQ_ERR_BAD_SHAPE;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return JQ_ERR_BAD_DTYPE;
    const int *h = reinterpret_cast<const int *>(plan_host);
    if (h[0] != kTaMagic) return JQ_ERR_BAD_SHAPE;
    jqta::PeerInfo peers;
    peers.n = npeer;
    for (int i = 0; i < 8; ++i) peers.delta[i] = i < npeer ? (long long)peer_delta[i] : 0;
    const int n = h[1], grid = h[2];
    const int *d = reinterpret_cast<const int *>(plan_dev);
    const TaProblem *probs = reinterpret_cast<const TaProblem *>(reinterpret_cast<const unsigned char *>(plan_dev) + h[7]);
    const CUtensorMap *maps = reinterpret_cast<const CUtensorMap *>(reinterpret_cast<const unsigned char *>(plan_dev) + h[4]);
    if (reinterpret_cast<uintptr_t>(maps) & 63u) return JQ_ERR_BAD_ALIGN;
    TaProblem none{};
    CUtensorMap nomap{};
    return ta_dispatch(h[6], h[3], h[8], probs, maps, none, nomap, n, d + kTaHeader, d + kTaHeader + n + 1, grid, h[5], x_dtype, y_dtype,
                       peers, reinterpret_cast<int *>(workspace_dev), reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int jq_gemm_ta(int fmt, const void *qweight, const void *scales, const void *codebook, const void *x,
                          const float *bias, void *y, int N, int K, int B, int g, int had_block, int x_dtype,
                          int y_dtype, void *workspace, size_t workspace_bytes, jq_stream_t stream) {
    if (!workspace) return JQ_ERR_NULL_PTR;
    if (B < 1) return JQ_ERR_BAD_SHAPE;
    if ((fmt != JQ_FMT_GF4 && fmt != JQ_FMT_E2M1) || !ta_cols(B)) return JQ_ERR_UNSUPPORTED;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return JQ_ERR_BAD_DTYPE;
    if (reinterpret_cast<uintptr_t>(workspace) & 127u) return JQ_ERR_BAD_ALIGN;
    jq_problem p{};
    p.qweight = qweight; p.scales = scales; p.codebook = codebook; p.x = x; p.bias = bias; p.y = y;
    p.N = N; p.K = K; p.g = g; p.had_block = had_block;
    if (workspace_bytes < jq_ta_workspace_bytes(&p, 1, B)) return JQ_ERR_WORKSPACE;
    TaProblem t;
    size_t off = kHeaderBytes;
    int st = ta_fill_problem(t, fmt, p, reinterpret_cast<unsigned char *>(workspace), off, B);
    if (st) return st;
    CUtensorMap tm;
    const bool lut = fmt == JQ_FMT_GF4 && ta_use_lut(B, K);
    st = ta_encode_map(&tm, qweight, N, K >> 1, (lut || B > NB) ? 32 : kTileM);
    if (st) return st;
    jqta::PeerInfo peers;
    peers.n = 1;
    for (int i = 0; i < 8; ++i) peers.delta[i] = 0;
    int grid = jq_sm_count();
    const int tile_m = lut ? kLutTileM : kTileM;
    const int tiles = (N + tile_m - 1) / tile_m;
    if (grid > tiles) grid = tiles;
    return ta_dispatch(fmt, ta_cols(B), K, nullptr, nullptr, t, tm, 0, nullptr, nullptr, grid, B, x_dtype, y_dtype, peers,
                       reinterpret_cast<int *>(workspace), reinterpret_cast<cudaStream_t>(stream));
}

// The status word is sticky: kernels only ever raise it.  Reading it synchronises the stream; clear != 0
// also resets it (stream-ordered) after the read.
extern "C" int jq_ta_status(void *workspace, int clear, jq_stream_t stream) {
    if (!workspace) return JQ_ERR_NULL_PTR;
    int v = 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    JQ_CUDA_TRY(cudaMemcpyAsync(&v, workspace, sizeof(int), cudaMemcpyDeviceToHost, st));
    JQ_CUDA_TRY(cudaStreamSynchronize(st));
    if (clear && v) JQ_CUDA_TRY(cudaMemsetAsync(workspace, 0, sizeof(int), st));
    return v;
}

// ---- bounded-wait self test ------------------------------------------------------
// One CTA waits, the way the pipelines above wait, on an mbarrier that nothing ever arrives on.  The wait
// has to give up after the given number of polls, raise the status word and let the kernel return; the
// device stays usable.  (This is how the failure path is exercised without faulting or hanging a GPU.)
namespace jqta {
__global__ void __launch_bounds__(64) bounded_wait_selftest_kernel(int *status, uint32_t limit) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int s_err;
    if (threadIdx.x == 0) {
        s_err = 0;
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    volatile int *err = &s_err;
    if (threadIdx.x == 32) {          // one waiter; nobody arrives
        bool ok = false;
        for (uint32_t i = 0; i < limit; ++i) {
            if (mbar_try(smem_u32(&bar), 0)) { ok = true; break; }
            if (i > 64) __nanosleep(64);
        }
        if (!ok) *err = JQ_ERR_TIMEOUT;
    }
    __syncthreads();
    if (threadIdx.x == 0) *status = s_err;
}
}  // namespace jqta

extern "C" int jq_selftest_bounded_wait(int *status_dev, unsigned int polls, jq_stream_t stream) {
    if (!status_dev) return JQ_ERR_NULL_PTR;
    if (polls == 0 || polls > (1u << 20)) return JQ_ERR_BAD_SHAPE;   // at most ~0.1 s of polling
    jqta::bounded_wait_selftest_kernel<<<1, 64, 0, reinterpret_cast<cudaStream_t>(stream)>>>(status_dev, polls);
    return jq_launch_status();
}
