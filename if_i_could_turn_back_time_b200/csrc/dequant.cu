// Packed 4-bit -> dense fp32 (bit-exact: one fp32 multiply per weight), and
// the stand-alone block Hadamard rotation.
#include "common.cuh"

namespace jq {

__constant__ float kE2M1[16] = {0.f, 0.5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f,
                                -0.f, -0.5f, -1.f, -1.5f, -2.f, -3.f, -4.f, -6.f};

// A warp turns 1024 consecutive codes of one row into fp32, 128 per step: lane l holds codes 4 l .. 4 l + 3 of a step, so
// that the warp's 16-byte stores cover 512 consecutive bytes (the kernel is bound by writing the dense matrix, eight
// times the bytes it reads).  The 16 values of the row's table sit in the lanes and are looked up with shuffles.
// Rows of the packed matrix are padded to 32 codes; the dense output has no padding, so rows that are not a multiple of
// four floats, or start off a 16-byte boundary, are stored element by element.
constexpr int kDequantSteps = 8;
template <int FMT>
__global__ void __launch_bounds__(256) dequant_kernel(const uint8_t *__restrict__ qw, const __half *__restrict__ scales,
                                                       const __half *__restrict__ codebook, float *__restrict__ out,
                                                       int N, int K, int g) {
    const int lane = threadIdx.x & 31;
    const int per_row = (K + 128 * kDequantSteps - 1) / (128 * kDequantSteps);
    const long long units = (long long)N * per_row;
    const int row_bytes = jq_row_stride_codes(K) >> 1, G = g ? K / g : 0;
    const bool vec = (K & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    for (long long u = blockIdx.x * 8LL + (threadIdx.x >> 5); u < units; u += gridDim.x * 8LL) {
        const int n = (int)(u / per_row), k0 = (int)(u - (long long)n * per_row) * (128 * kDequantSteps) + lane * 4;
        const uint8_t *row = qw + (size_t)n * row_bytes;
        uint32_t w[kDequantSteps];
        float s[kDequantSteps];
#pragma unroll
        for (int i = 0; i < kDequantSteps; ++i) {
            const int k = k0 + 128 * i;
            w[i] = k < K ? *reinterpret_cast<const unsigned short *>(row + (k >> 1)) : 0u;
            s[i] = (g && k < K) ? __half2float(scales[(size_t)n * G + k / g]) : 1.f;   // g % 32 == 0: one group per 4 codes
        }
        float entry;
        if (FMT == JQ_FMT_E2M1) entry = kE2M1[lane & 15];
        else entry = __half2float(codebook[(size_t)n * 16 + (lane & 15)]);
        float *o = out + (size_t)n * K;
#pragma unroll
        for (int i = 0; i < kDequantSteps; ++i) {
            const int k = k0 + 128 * i;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float t = __shfl_sync(0xffffffffu, entry, (w[i] >> (4 * j)) & 0xfu);
                v[j] = g ? __fmul_rn(t, s[i]) : t;
            }
            if (vec) {
                if (k < K) __stcs(reinterpret_cast<float4 *>(o + k), make_float4(v[0], v[1], v[2], v[3]));
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k + j < K) o[k + j] = v[j];
            }
        }
    }
}

// One warp per 128-block.
__global__ void __launch_bounds__(256) fwht_kernel(const void *__restrict__ x, float *__restrict__ y, long long nblocks,
                                                    int x_dtype) {
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long blk = warp; blk < nblocks; blk += nwarps) {
        float v[4];
        const size_t k0 = (size_t)blk * 128 + lane * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = load_act(x, k0 + j, x_dtype);
        fwht128_warp(v, lane);
        *reinterpret_cast<float4 *>(y + k0) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

}  // namespace jq

using namespace jq;

static int dequant_common(int fmt, const void *qw, const void *scales, const void *codebook, float *out, int N, int K,
                          int g, jq_stream_t stream) {
    if (!qw || !out) return JQ_ERR_NULL_PTR;
    if (fmt == JQ_FMT_GF4 && !codebook) return JQ_ERR_NULL_PTR;
    if (N <= 0 || K <= 0) return JQ_ERR_BAD_SHAPE;
    if (fmt == JQ_FMT_E2M1 && g == 0) return JQ_ERR_BAD_SHAPE;
    if (g < 0 || (g && (g % 32 || K % g))) return JQ_ERR_BAD_SHAPE;
    if (g && !scales) return JQ_ERR_NULL_PTR;
    if (!jq_aligned16(qw)) return JQ_ERR_BAD_ALIGN;
    if (reinterpret_cast<uintptr_t>(out) & 3u) return JQ_ERR_BAD_ALIGN;
    const long long units = (long long)N * ((K + 128 * kDequantSteps - 1) / (128 * kDequantSteps));
    long long blocks = (units + 7) / 8;
    const long long cap = 0x7fffffff;                  // one unit per warp: blocks that retire one by one keep loads and stores of different units overlapped
    if (blocks > cap) blocks = cap;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint8_t *q = reinterpret_cast<const uint8_t *>(qw);
    const __half *sc = reinterpret_cast<const __half *>(scales), *cb = reinterpret_cast<const __half *>(codebook);
    if (fmt == JQ_FMT_E2M1) dequant_kernel<JQ_FMT_E2M1><<<(int)blocks, 256, 0, st>>>(q, sc, nullptr, out, N, K, g);
    else dequant_kernel<JQ_FMT_GF4><<<(int)blocks, 256, 0, st>>>(q, sc, cb, out, N, K, g);
    return jq_launch_status();
}

extern "C" int jq_dequant_e2m1(const void *qweight, const void *scales, float *out, int N, int K, int g,
                               jq_stream_t stream) {
    return dequant_common(JQ_FMT_E2M1, qweight, scales, nullptr, out, N, K, g, stream);
}

extern "C" int jq_dequant_gf4(const void *qweight, const void *scales, const void *codebook, float *out, int N, int K,
                              int g, jq_stream_t stream) {
    return dequant_common(JQ_FMT_GF4, qweight, scales, codebook, out, N, K, g, stream);
}

extern "C" int jq_fwht_block(const void *x, float *y, int B, int K, int block, int x_dtype, jq_stream_t stream) {
    if (!x || !y) return JQ_ERR_NULL_PTR;
    if (B <= 0 || K <= 0) return JQ_ERR_BAD_SHAPE;
    if (block != 128) return JQ_ERR_UNSUPPORTED;
    if (K % block) return JQ_ERR_BAD_SHAPE;
    if (x_dtype != JQ_F32 && x_dtype != JQ_F16 && x_dtype != JQ_BF16) return JQ_ERR_BAD_DTYPE;
    if (!jq_aligned16(y)) return JQ_ERR_BAD_ALIGN;
    const long long nblocks = (long long)B * (K / 128);
    long long blocks = (nblocks + 7) / 8;
    const long long cap = (long long)jq_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    fwht_kernel<<<(int)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(x, y, nblocks, x_dtype);
    return jq_launch_status();
}
