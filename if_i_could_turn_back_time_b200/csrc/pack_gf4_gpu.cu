// Device-side GF4 packer: per-row 16-class Jenks natural breaks on the GPU,
// bit-identical to the host packer (pack_host.cpp) and to the CPU oracle.
//
// Two kernels per chunk of rows:
//   sort_rows_kernel, one small CTA per row, several per SM:
//     1. group scales (fp16_rn of the group absmax) and u = w / scale into shared memory;
//     2. bitonic sort of u (padded with +inf to a power of two);
//     3. run-length compression to distinct values and their start indices (= the prefix sums of the multiplicities);
//     4. float64 prefix sums, sequential in index order (the summation order is part of the format contract: codebooks
//        must come out bit-identical).  A chain of K dependent additions, some 44 clocks each: the other CTAs of the SM
//        fill the time.
//   jenks_rows_kernel, one CTA per SM:
//     5. the dynamic programme over 16 classes in its divide-and-conquer form (the left-most optimal split is monotone
//        in the prefix length), with the host's candidates and tie rule.  The recursion [lo, hi] -> mid,
//        [lo, mid - 1], [mid + 1, hi] is a fixed tree, walked level by level: a node's range of candidates lies between
//        the results next to its interval.  Groups of lanes take the nodes; ranges that are long for their group
//        are cut in pieces that all warps share;
//     6. back-track, class means -> fp16 codebook, codes by comparing each u with the classes' upper bounds.
// The objective is the k-class form of the one the reference evaluates for two
// classes (Python_Jenks_Test/Jenks_Tests/cuda_helpers.py:151-184).
//
// What bounds it: float64 arithmetic, 64 lanes per clock and SM, on about 15 x (log2(K) + 1) x K candidate splits of a
// row.  A candidate's cost has a division (some 20 float64 operations); it is estimated with a table of reciprocals
// first (6 operations), and only a thread's candidates within the estimate's error bound of its smallest are computed
// exactly, normally one.  The ranges of a level add up to K, but one node's can be most of it (weights with outliers): left
// to the node's own lanes, the longest range set the pace.  Measured: issue slots 54 %, float64 pipe 17 % busy, waits at
// the level barriers the top stall.  4096 x 4096: 92.3 ms with queues of nodes in global memory, one warp per node; 26.9 ms
// like this.  (Doubles permuted against bank conflicts: 30.8 ms, the index arithmetic costs more.  Costs compared as
// integers in the reductions over lanes: 0 to 3 % slower.)
#include "common.cuh"
#include <cfloat>

namespace jqg {

constexpr int kClasses = 16;
constexpr int kRowsPerSm = 8;             // rows of a chunk per SM, at most
// Workspace per SM: 152 bytes per value of a row padded to a power of two.  With eight rows per SM whatever their length it
// was 1.3 GB for rows of 32768 values.
constexpr size_t kSmBudget = 152;

__host__ __device__ inline size_t up16(size_t v) { return (v + 15) / 16 * 16; }

// a chunk row's slice of the workspace, written by the first kernel
struct RowData {
    double2 *P;          // [K + 1] prefix sums of n v and n v^2 over the distinct values
    int *C;              // [K + 1] prefix sums of n
    float *uv;           // [K]     distinct values
    int *m;              // how many
};
__host__ __device__ inline size_t row_bytes(int K) {
    return sizeof(double2) * ((size_t)K + 1) + up16(sizeof(int) * ((size_t)K + 1)) + up16(sizeof(float) * (size_t)K + 8);
}
// The second kernel reads P and C of its row first; their place then takes the split arguments of ten classes.  The
// other five classes' have a place of their own.
constexpr int kArgsInRow = (sizeof(double2) + sizeof(int)) / sizeof(unsigned short);
constexpr int kArgsBeside = kClasses - 1 - kArgsInRow;
__device__ inline RowData row_data(unsigned char *base, int K) {
    RowData r;
    r.P = reinterpret_cast<double2 *>(base); base += sizeof(double2) * ((size_t)K + 1);
    r.C = reinterpret_cast<int *>(base); base += up16(sizeof(int) * ((size_t)K + 1));
    r.m = reinterpret_cast<int *>(base);
    r.uv = reinterpret_cast<float *>(base) + 2;
    return r;
}

// the second kernel's arrays: where they lie (shared memory as far as they fit, the CTA's slice of the workspace
// otherwise), in the order of the traffic that a candidate causes
enum { kP1 = 0, kP2, kPrev, kCur, kRecip, kArg, kCount, kArrays };
struct Layout {
    size_t off[kArrays];
    unsigned shared;          // bit a: array a lies in shared memory
    size_t shared_bytes, cta_bytes;
};
__host__ inline Layout make_layout(int K, size_t shared_limit) {
    const size_t m1 = (size_t)K + 1, d = sizeof(double) * m1;
    const size_t bytes[kArrays] = {d, d, d, d, d, sizeof(unsigned short) * m1, sizeof(int) * m1};
    Layout L{};
    L.cta_bytes = up16(kArgsBeside * sizeof(unsigned short) * m1);
    for (int a = 0; a < kArrays; ++a) {
        const size_t b = up16(bytes[a]);
        if (L.shared_bytes + b <= shared_limit) { L.shared |= 1u << a; L.off[a] = L.shared_bytes; L.shared_bytes += b; }
        else { L.off[a] = L.cta_bytes; L.cta_bytes += b; }
    }
    return L;
}
constexpr size_t kSharedLimit = 200 * 1024;       // of the second kernel's CTAs on an SM together (besides their static arrays)

template <int kThreads>
__global__ void __launch_bounds__(kThreads) sort_rows_kernel(const float *__restrict__ W, int row0, int N, int K, int g,
                                                             __half *__restrict__ scales, unsigned char *__restrict__ ws, int npad) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *sv = reinterpret_cast<float *>(smem_raw);   // npad floats: the row being sorted
    constexpr int kWarps = kThreads / 32;
    __shared__ int s_scan[kWarps + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = row0 + blockIdx.x;
    const RowData rd = row_data(ws + (size_t)blockIdx.x * row_bytes(K), K);
    const int G = g ? K / g : 0;
    const float *wr = W + (size_t)row * K;
    // ---- 1. scales and normalised values
    if (g) {
        for (int gi = warp; gi < G; gi += kWarps) {
            float amax = 0.f;
            for (int k = lane; k < g; k += 32) amax = fmaxf(amax, fabsf(wr[gi * g + k]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            __half hs = __float2half_rn(amax);
            float s = __half2float(hs);
            if (amax == 0.f || s == 0.f || isinf(s) || isnan(s)) { hs = __float2half_rn(1.0f); s = 1.0f; }
            if (lane == 0) scales[(size_t)row * G + gi] = hs;
            for (int k = lane; k < g; k += 32) sv[gi * g + k] = __fdiv_rn(wr[gi * g + k], s);
        }
    } else {
        for (int k = tid; k < K; k += kThreads) sv[k] = wr[k];
    }
    for (int k = K + tid; k < npad; k += kThreads) sv[k] = __int_as_float(0x7f800000);  // +inf padding sorts last
    __syncthreads();
    // ---- 2. bitonic sort, ascending
    for (int size = 2; size <= npad; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < npad / 2; i += kThreads) {
                const int lo = 2 * i - (i & (stride - 1));
                const int hi = lo + stride;
                const bool up = (lo & size) == 0;
                const float a = sv[lo], b = sv[hi];
                if ((a > b) == up) { sv[lo] = b; sv[hi] = a; }
            }
            __syncthreads();
        }
    }
    // ---- 3. run-length compression of sv[0..K): a warp's 32 consecutive elements at a time
    int base = 0;                                          // distinct values so far
    for (int c0 = 0; c0 < K; c0 += kThreads) {
        const int i = c0 + tid;
        const bool head = i < K && (i == 0 || sv[i] != sv[i - 1]);
        const unsigned mask = __ballot_sync(0xffffffffu, head);
        if (lane == 0) s_scan[warp] = __popc(mask);
        __syncthreads();
        int before = base, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) { before += w < warp ? s_scan[w] : 0; all += s_scan[w]; }
        if (head) {
            const int t = before + __popc(mask & ((1u << lane) - 1u));
            rd.uv[t] = sv[i] + 0.0f;                       // -0.0 and +0.0 are one value: +0.0
            rd.C[t] = i;
        }
        base += all;
        __syncthreads();
    }
    const int m = base;
    if (tid == 0) { rd.C[m] = K; *rd.m = m; }
    __syncthreads();
    // ---- 4. the terms, then their sequential float64 prefix sums
    for (int t = tid; t < m; t += kThreads) {
        const double v = (double)rd.uv[t], n = (double)(rd.C[t + 1] - rd.C[t]);
        const double cv = __dmul_rn(n, v);
        rd.P[t + 1] = make_double2(cv, __dmul_rn(cv, v));
    }
    __syncthreads();
    if (warp == 0) {        // every lane carries the chain of additions along and keeps the sums of its own element
        double p1 = 0.0, p2 = 0.0;
        if (lane == 0) rd.P[0] = make_double2(0.0, 0.0);
        double2 nxt = lane < m ? rd.P[1 + lane] : make_double2(0.0, 0.0);
        for (int t0 = 0; t0 < m; t0 += 32) {
            const double2 now = nxt;
            double2 sums = now;
            if (t0 + 32 + lane < m) nxt = rd.P[t0 + 33 + lane];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                p1 = __dadd_rn(p1, __shfl_sync(0xffffffffu, now.x, i));
                p2 = __dadd_rn(p2, __shfl_sync(0xffffffffu, now.y, i));
                if (i == lane) sums = make_double2(p1, p2);
            }
            if (t0 + lane < m) rd.P[t0 + 1 + lane] = sums;
        }
    }
}

struct Dp {
    const double *P1, *P2;
    const int *C;             // null: all values are distinct, C[t] = t
    const double *recip;
    double margin;            // twice the error bound of an estimate

    __device__ __forceinline__ int count(int t) const { return C ? C[t] : t; }
    __device__ __forceinline__ double exact(const double *prev, int t, double p1, double p2, int cm) const {
        const double d1 = __dsub_rn(p1, P1[t]), d2 = __dsub_rn(p2, P2[t]);
        const double q = __ddiv_rn(__dmul_rn(d1, d1), (double)(cm - count(t)));
        const double seg = __dsub_rn(d2, q);
        return prev ? __dadd_rn(prev[t], seg) : seg;
    }
    // the same with the reciprocal of the count rounded first
    __device__ __forceinline__ double estimate(const double *prev, int t, double p1, double p2, int cm) const {
        const double d1 = __dsub_rn(p1, P1[t]), d2 = __dsub_rn(p2, P2[t]);
        const double q = __dmul_rn(__dmul_rn(d1, d1), recip[cm - count(t)]);
        return __dadd_rn(prev[t], __dsub_rn(d2, q));
    }
    // first minimum of prev[t] + cost(t, mid) over t = t0 + first, t0 + first + step, ... <= t1; kAhead estimates at a
    // time hide each other's latency
    template <int kAhead>
    __device__ __forceinline__ void scan(const double *prev, int t0, int t1, int first, int step, int mid, double &best, int &bt) const {
        const double p1 = P1[mid], p2 = P2[mid];
        const int cm = count(mid);
        double low = __longlong_as_double(0x7ff0000000000000LL), limit = low;
        int pos = -1;
        bool several = false;             // more than one candidate may be the minimum
        const bool one_each = kAhead > 1 && t1 - t0 < step;        // a candidate per lane needs no estimate
        if (one_each && t0 + first <= t1) pos = t0 + first;
        for (int tb = one_each ? t1 + 1 : t0 + first; tb <= t1; tb += kAhead * step) {
            double e[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) e[i] = estimate(prev, min(tb + i * step, t1), p1, p2, cm);
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int t = tb + i * step;
                if (t > t1) break;
                const double a = e[i];
                if (a < low) {
                    several = pos >= 0 && !(__dadd_rn(a, margin) < low);
                    low = a; pos = t; limit = __dadd_rn(a, margin);
                } else if (!(a > limit)) {    // (also when something is not a number)
                    several = true;
                }
            }
        }
        best = DBL_MAX;
        bt = 0x7fffffff;
        if (several) {
            for (int t = t0 + first; t <= t1; t += step)
                if (!(estimate(prev, t, p1, p2, cm) > limit)) {
                    const double c = exact(prev, t, p1, p2, cm);
                    if (c < best) { best = c; bt = t; }
                }
        } else if (pos >= 0) {
            const double c = exact(prev, pos, p1, p2, cm);
            if (c < best) { best = c; bt = pos; }
        }
    }
};

__device__ __forceinline__ void take_first_min(double &best, int &bt, double ob, int ot) {
    if (ob < best || (ob == best && ot < bt)) { best = ob; bt = ot; }
}

// kAllShared: every array lies in shared memory (the compiler then knows the address space)
template <int kThreads, bool kAllShared>
__global__ void __launch_bounds__(kThreads) jenks_rows_kernel(const float *__restrict__ W, int row0, int rows, int K, int g,
                                                              uint8_t *__restrict__ qw, const __half *__restrict__ scales,
                                                              __half *__restrict__ codebook, unsigned char *row_ws,
                                                              unsigned char *cta_ws, const __grid_constant__ Layout L) {
    constexpr int kWarps = kThreads / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_zero, s_breaks[kClasses + 1];
    __shared__ float s_upper[kClasses];                // largest value of each class
    // ranges that all warps share: a level's long nodes, the pieces of their ranges and the pieces' results.  A range is
    // long from 32 candidates per lane of its group and 1/128 of the row, a piece at least 1/64 of the row, and a level's
    // ranges add up to at most twice the row, so that neither array overflows (what did would be scanned by its group)
    constexpr int kWide = kThreads / 4, kPieces = kThreads / 2;
    struct Wide { int first, count, mid, t0; };
    struct Piece { int t0, t1, mid; };
    __shared__ Wide s_wide[kWide];
    __shared__ Piece s_piece[kPieces];
    __shared__ double s_best[kPieces];
    __shared__ int s_bt[kPieces];
    __shared__ int s_count[2][2];                      // long nodes, pieces; by parity of the level, as warps leave a level without any at different times
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char *slice = cta_ws + (size_t)blockIdx.x * L.cta_bytes;
    auto array = [&](int a) -> unsigned char * {
        if (kAllShared) return smem_raw + L.off[a];
        return ((L.shared >> a) & 1u) ? smem_raw + L.off[a] : slice + L.off[a];
    };
    double *const table = reinterpret_cast<double *>(array(kRecip));
    const int G = g ? K / g : 0;
    const int stride_b = jq_row_stride_codes(K) >> 1;

    for (int i = tid; i <= K; i += kThreads) table[i] = i ? __ddiv_rn(1.0, (double)i) : 0.0;

    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const int row = row0 + r;
        const float *wr = W + (size_t)row * K;
        const RowData rd = row_data(row_ws + (size_t)r * row_bytes(K), K);
        // the split arguments of class j = 2 .. 16, for the back-track
        auto args_of = [&](int j) {
            return j - 2 < kArgsInRow ? reinterpret_cast<unsigned short *>(rd.P) + (size_t)(j - 2) * (K + 1)
                                      : reinterpret_cast<unsigned short *>(slice) + (size_t)(j - 2 - kArgsInRow) * (K + 1);
        };
        const int m = *rd.m;
        const int ke = m < kClasses ? m : kClasses;
        auto classify = [&](unsigned char *at_P1, unsigned char *at_P2, unsigned char *at_prev, unsigned char *at_cur,
                            unsigned char *at_C, unsigned char *at_arg, const double *recip) __attribute__((always_inline)) {
        double *P1 = reinterpret_cast<double *>(at_P1), *P2 = reinterpret_cast<double *>(at_P2);
        double *prev = reinterpret_cast<double *>(at_prev), *cur = reinterpret_cast<double *>(at_cur);
        int *C = reinterpret_cast<int *>(at_C);
        unsigned short *arg = reinterpret_cast<unsigned short *>(at_arg);
        for (int i = tid; i <= m; i += kThreads) {
            const double2 p = rd.P[i];
            P1[i] = p.x;
            P2[i] = p.y;
            C[i] = rd.C[i];
        }
        __syncthreads();
        // ---- 5. dynamic programme.  An estimate differs from the exact cost by a few roundings of terms that are at
        // most the row's sum of squares: 2^-49 of it, with room to spare 2^-46
        const Dp dp{P1, P2, m == K ? nullptr : C, recip, P2[m] * 0x1p-45};
        for (int i = tid; i <= m; i += kThreads) prev[i] = i >= 1 ? dp.exact(nullptr, 0, P1[i], P2[i], dp.count(i)) : DBL_MAX;
        __syncthreads();
        int parity = 0;
        if (tid < 4) s_count[tid >> 1][tid & 1] = 0;
        __syncthreads();
        for (int j = 2; j <= ke; ++j) {
            unsigned short *out_arg = args_of(j);
            auto write = [&](int mid, double best, int bt) {
                cur[mid] = best;
                arg[mid] = (unsigned short)bt;
                out_arg[mid] = (unsigned short)bt;
            };
            const int root = j == ke ? m : j, piece_len = max(128, m / 64);
            for (int level = 0; (1 << level) <= m - root + 1; ++level, parity ^= 1) {
                const int nodes = 1 << level, width = nodes <= kWarps ? 32 : max(kThreads >> level, 1);   // lanes per node
                const int long_range = max(32 * width, m / 128);
                const int in_group = lane & (width - 1), leader = lane - in_group;
                for (int base = 0; base < nodes; base += kThreads / width) {
                    const int node = base + tid / width;
                    int l = root, h = m;
                    for (int b = level - 1; b >= 0 && l <= h; --b) {
                        const int mid = (l + h) >> 1;
                        if ((node >> b) & 1) l = mid + 1; else h = mid - 1;
                    }
                    const bool live = node < nodes && l <= h;
                    if (!__any_sync(0xffffffffu, live)) continue;
                    const int mid = (l + h) >> 1;
                    int t0 = 0, t1 = -1;
                    if (live) {
                        t0 = max(l == root ? j - 1 : (int)arg[l - 1], j - 1);
                        t1 = min(mid - 1, h == m ? m - 1 : (int)arg[h + 1]);
                    }
                    int shared_out = 0;
                    if (t1 - t0 >= long_range && in_group == 0) {
                        const int n = (t1 - t0) / piece_len + 1;
                        const int slot = atomicAdd(&s_count[parity][0], 1), first = atomicAdd(&s_count[parity][1], n);
                        shared_out = slot < kWide && first + n <= kPieces;
                        if (slot < kWide) s_wide[slot] = Wide{first, shared_out ? n : 0, mid, t0};
                        for (int i = 0; i < n && first + i < kPieces; ++i) {
                            const int a = t0 + i * piece_len;
                            s_piece[first + i] = shared_out ? Piece{a, min(t1, a + piece_len - 1), mid} : Piece{1, 0, mid};
                        }
                    }
                    shared_out = __shfl_sync(0xffffffffu, shared_out, leader);
                    double best = DBL_MAX;
                    int bt = 0x7fffffff;
                    if (live && !shared_out) {
                        if (width >= 8) dp.scan<4>(prev, t0, t1, in_group, width, mid, best, bt);
                        else dp.scan<1>(prev, t0, t1, in_group, width, mid, best, bt);
                    }
                    __syncwarp();
                    for (int o = width >> 1; o > 0; o >>= 1)
                        take_first_min(best, bt, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bt, o));
                    // (an empty range or all DBL_MAX: the host keeps t0)
                    if (live && !shared_out && in_group == 0) write(mid, best, bt == 0x7fffffff ? t0 : bt);
                }
                __syncthreads();
                const int n_wide = min(s_count[parity][0], kWide), n_pieces = min(s_count[parity][1], kPieces);
                if (n_wide == 0) continue;             // (the same for all threads)
                for (int c = warp; c < n_pieces; c += kWarps) {
                    const Piece pc = s_piece[c];
                    double best;
                    int bt;
                    dp.scan<4>(prev, pc.t0, pc.t1, lane, 32, pc.mid, best, bt);
                    __syncwarp();
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
                        take_first_min(best, bt, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bt, o));
                    if (lane == 0) { s_best[c] = best; s_bt[c] = bt; }
                }
                __syncthreads();
                if (tid < n_wide) {
                    const Wide wd = s_wide[tid];
                    double best = DBL_MAX;
                    int bt = 0x7fffffff;
                    for (int i = 0; i < wd.count; ++i) take_first_min(best, bt, s_best[wd.first + i], s_bt[wd.first + i]);
                    if (wd.count) write(wd.mid, best, bt == 0x7fffffff ? wd.t0 : bt);
                }
                if (tid < 2) s_count[parity][tid] = 0;
                __syncthreads();
            }
            double *tswap = prev; prev = cur; cur = tswap;
        }
        // ---- 6. back-track, codebook, class upper bounds
        if (tid == 0) {
            s_breaks[ke] = m;
            for (int j = ke; j >= 2; --j) s_breaks[j - 1] = args_of(j)[s_breaks[j]];
            s_breaks[0] = 0;
            // index of the distinct value 0.0 (m if the row has no exact zero)
            int lo = 0, hi = m;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (rd.uv[mid] < 0.0f) lo = mid + 1; else hi = mid;
            }
            s_zero = (lo < m && rd.uv[lo] == 0.0f) ? lo : m;
        }
        __syncthreads();
        if (tid < kClasses) {
            const int c = tid < ke ? tid : ke - 1;
            const int a = s_breaks[c], b = s_breaks[c + 1];
            double mean = __ddiv_rn(__dsub_rn(P1[b], P1[a]), (double)(C[b] - C[a]));
            if (s_zero >= a && s_zero < b) mean = 0.0;   // the class holding an exact zero is pinned to 0 (as the host packer)
            codebook[(size_t)row * kClasses + tid] = __double2half(mean);
            s_upper[tid] = tid < ke ? rd.uv[b - 1] : __int_as_float(0x7f800000);
        }
        __syncthreads();
        // codes: class = number of class upper bounds below the value
        const int words = stride_b >> 2;
        for (int wi = tid; wi < words; wi += kThreads) {
            uint32_t word = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int k = wi * 8 + e;
                if (k < K) {
                    float u = wr[k];
                    if (g) {
                        float s = __half2float(scales[(size_t)row * G + k / g]);
                        u = __fdiv_rn(u, s);
                    }
                    int c = 0;
#pragma unroll
                    for (int q = 0; q < kClasses - 1; ++q) c += (u > s_upper[q]) ? 1 : 0;
                    word |= (uint32_t)c << (4 * e);
                }
            }
            reinterpret_cast<uint32_t *>(qw + (size_t)row * stride_b)[wi] = word;
        }
        __syncthreads();
        };
        if (!kAllShared) {
            // The layout is for rows of K distinct values.  A row of fewer may fit in shared memory after all, reciprocals
            // and all: the walk down a tree is then not a chain of L2 latencies (1000 x 8192, about 550 distinct values a
            // row: 4.8 -> 3.1 ms).  The code is there twice so that the compiler knows which arrays are in shared memory
            // (with pointers chosen per row, rows of many values took 11 % longer).
            const size_t room = ((L.shared >> kRecip) & 1u) ? L.off[kRecip] : L.shared_bytes;
            const size_t d = sizeof(double) * ((m + 2) & ~1), used = up16(4 * d + d / 2 + d / 4);
            if (used <= room) {
                const double *recip = table;
                if (room == L.shared_bytes && used + sizeof(double) * ((size_t)K + 1) <= room) {
                    double *copy = reinterpret_cast<double *>(smem_raw + used);
                    for (int i = tid; i <= K; i += kThreads) copy[i] = table[i];
                    recip = copy;
                }
                classify(smem_raw, smem_raw + d, smem_raw + 2 * d, smem_raw + 3 * d, smem_raw + 4 * d, smem_raw + 4 * d + d / 2, recip);
                continue;
            }
        }
        classify(array(kP1), array(kP2), array(kPrev), array(kCur), array(kCount), array(kArg), table);
    }
}

}  // namespace jqg

static int next_pow2(int v) { int p = 1; while (p < v) p <<= 1; return p; }

// CTAs of the second kernel per SM: short rows leave room for more of them, with fewer threads each
static int jenks_threads(int K) { return K <= 1024 ? 256 : (K <= 2048 ? 512 : 1024); }
static int jenks_ctas_per_sm(int K) { return 1024 / jenks_threads(K); }
static jqg::Layout jenks_layout(int K) { return jqg::make_layout(K, jqg::kSharedLimit / jenks_ctas_per_sm(K)); }

// Rows of a chunk: as many per SM as the budget holds beside the second kernel's slices, a multiple of its CTAs; and the
// CTAs that have work.
struct Chunk { int rows, ctas; };
static Chunk pack_chunk(int N, int K) {
    const int per_sm = jenks_ctas_per_sm(K), sms = jq_sm_count();
    const size_t budget = jqg::kSmBudget * (size_t)next_pow2(K), slices = jenks_layout(K).cta_bytes * (size_t)per_sm;
    size_t rows = budget > slices ? (budget - slices) / jqg::row_bytes(K) : 0;
    if (rows > (size_t)jqg::kRowsPerSm) rows = jqg::kRowsPerSm;
    rows = rows / per_sm * per_sm;
    if (rows < (size_t)per_sm) rows = per_sm;
    const long long chunk = (long long)rows * sms, ctas = (long long)per_sm * sms;
    return Chunk{(int)(N < chunk ? N : chunk), (int)(N < ctas ? N : ctas)};
}

extern "C" size_t jq_pack_gf4_workspace_bytes_rows(int N, int K) {
    if (N <= 0 || K <= 0) return 0;
    const Chunk c = pack_chunk(N, K);
    return jqg::row_bytes(K) * (size_t)c.rows + jenks_layout(K).cta_bytes * (size_t)c.ctas;
}

extern "C" size_t jq_pack_gf4_workspace_bytes(int K) { return jq_pack_gf4_workspace_bytes_rows(0x7fffffff, K); }

extern "C" int jq_pack_gf4(const float *W, int N, int K, int g, void *qweight, void *scales, void *codebook,
                           void *workspace, size_t workspace_bytes, jq_stream_t stream) {
    if (!W || !qweight || !codebook || !workspace) return JQ_ERR_NULL_PTR;
    if (N <= 0 || K <= 0 || g < 0 || (g && (g % 32 || K % g))) return JQ_ERR_BAD_SHAPE;
    if (g && !scales) return JQ_ERR_NULL_PTR;
    const int npad = next_pow2(K);
    const size_t sort_smem = (size_t)npad * sizeof(float);
    if (sort_smem > 200 * 1024) return JQ_ERR_UNSUPPORTED;   // rows longer than 32768 values
    if (workspace_bytes < jq_pack_gf4_workspace_bytes_rows(N, K)) return JQ_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255u) || !jq_aligned16(qweight) || (reinterpret_cast<uintptr_t>(W) & 3u))
        return JQ_ERR_BAD_ALIGN;
    const jqg::Layout L = jenks_layout(K);
    const bool all_shared = L.shared == (1u << jqg::kArrays) - 1u;
    const int threads = jenks_threads(K);
    auto kern = threads == 256 ? (all_shared ? jqg::jenks_rows_kernel<256, true> : jqg::jenks_rows_kernel<256, false>)
              : threads == 512 ? (all_shared ? jqg::jenks_rows_kernel<512, true> : jqg::jenks_rows_kernel<512, false>)
                               : (all_shared ? jqg::jenks_rows_kernel<1024, true> : jqg::jenks_rows_kernel<1024, false>);
    JQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.shared_bytes));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const Chunk chunk = pack_chunk(N, K);
    // 256 threads per row while several rows share an SM (the sequential sums of one run beside the sorting of others); 1024
    // for rows that have an SM to themselves, for want of rows or (from 16385 values) of shared memory for a second: 148 rows
    // of 11008 with 560 distinct values 182 -> 127 us, 300 of 28672 1176 -> 754
    const int sort_threads = chunk.rows <= jq_sm_count() || sort_smem > 64 * 1024 ? 1024 : 256;
    auto sort = sort_threads == 1024 ? jqg::sort_rows_kernel<1024> : jqg::sort_rows_kernel<256>;
    JQ_CUDA_TRY(cudaFuncSetAttribute(sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem));
    unsigned char *row_ws = reinterpret_cast<unsigned char *>(workspace);
    unsigned char *cta_ws = row_ws + jqg::row_bytes(K) * (size_t)chunk.rows;
    for (int row0 = 0; row0 < N; row0 += chunk.rows) {
        const int rows = N - row0 < chunk.rows ? N - row0 : chunk.rows;
        sort<<<rows, sort_threads, sort_smem, st>>>(W, row0, N, K, g, reinterpret_cast<__half *>(scales), row_ws, npad);
        const int grid = rows < chunk.ctas ? rows : chunk.ctas;
        kern<<<grid, threads, L.shared_bytes, st>>>(W, row0, rows, K, g, reinterpret_cast<uint8_t *>(qweight),
                                                    reinterpret_cast<const __half *>(scales), reinterpret_cast<__half *>(codebook),
                                                    row_ws, cta_ws, L);
    }
    return jq_launch_status();
}
