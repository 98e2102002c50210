// Short causal convolution over time, per channel, of a step's flat batch.
//
//   u_t = in_t + in_bias                          (the projected values, the projection's bias included)
//   y_t = act(sum_j taps[c][j] * u_{t-K+1+j} + conv_bias)      zeros before a sequence's start
//
// A request's tokens may arrive in portions: the last K-1 values of u of each sequence live in
// its state slot `tail` [rows, K-1, C] (float32) and stand in for the tokens before the portion.
// `short_conv` reads the tail as earlier steps left it; `short_conv_tail` then moves it on.
// The two are separate launches because every token of a portion may read the old tail.
//
// Channels are cut into up to three column ranges with a destination each: a dense matrix in the
// model dtype, or a paged pool [pages, heads, page_size, head_dim] written at the token's slot.
#include <math.h>

#include "common.cuh"

using namespace sb;

namespace {

constexpr int MAX_TAPS = 16;

struct ConvSeg {
    int begin, end;        // channels [begin, end)
    int paged;             // 0: dense [N, stride]; 1: paged pool
    void* dst;
    long long stride;      // dense: elements per row
    int heads, head_dim;   // paged
};

struct ConvArgs {
    const void* in;        // [N, in_stride] in T, channel c at column c
    long long in_stride;
    const float* in_bias;  // [C] or null
    const float* taps;     // [C, K]
    const float* conv_bias;   // [C] or null
    int act;               // 0 none, 1 silu
    const float* tail;     // [rows, K-1, C]
    int C, K, N;
    const int* token_rows;
    const int* positions;
    const int* block_table;
    int table_width, page_size;
    ConvSeg seg[3];
    int nseg;
};

template <typename T>
__global__ void __launch_bounds__(256) short_conv_kernel(ConvArgs a) {
    sb::pdl_launch_dependents();
    sb::pdl_wait();
    const int n = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.C) return;
    const int row = a.token_rows[n], pos = a.positions[n];
    const int K = a.K;
    // how many tokens directly before this one belong to the same request (at most K-1 matter)
    int same = 0;
    for (int b = 1; b < K; ++b) {
        if (n - b >= 0 && a.token_rows[n - b] == row) same = b;
        else break;
    }
    const T* in = (const T*)a.in;
    const float bias = a.in_bias ? a.in_bias[c] : 0.f;
    float acc = 0.f;
    for (int j = 0; j < K; ++j) {
        const int back = K - 1 - j;
        if (pos - back < 0) continue;                       // before the sequence's start
        float u;
        if (back <= same) u = to_float(in[(size_t)(n - back) * a.in_stride + c]) + bias;
        else u = a.tail[((size_t)row * (K - 1) + (K - 1 - back + same)) * a.C + c];
        acc = fmaf(a.taps[(size_t)c * K + j], u, acc);
    }
    if (a.conv_bias) acc += a.conv_bias[c];
    if (a.act == 1) acc = acc / (1.0f + expf(-acc));
    for (int s = 0; s < a.nseg; ++s) {
        const ConvSeg& g = a.seg[s];
        if (c < g.begin || c >= g.end) continue;
        const int e = c - g.begin;
        if (!g.paged) {
            ((T*)g.dst)[(size_t)n * g.stride + e] = from_float<T>(acc);
        } else {
            const int head = e / g.head_dim, x = e - head * g.head_dim;
            const int page = a.block_table[(size_t)row * a.table_width + pos / a.page_size];
            ((T*)g.dst)[(((size_t)page * g.heads + head) * a.page_size + pos % a.page_size) * g.head_dim + x] =
                from_float<T>(acc);
        }
    }
}

// The same for many tokens: a thread holds 16 bytes of neighbouring channels (VEC) and walks RUN tokens of the batch with the
// last K - 1 values in registers, so that a value is read once and not K times, in whole lines.  The sums are those of the
// kernel above, in its order (which call takes which: sb_short_conv_pays_runs).  A prompt of 1,500 tokens through 3,072 channels of 3 taps and 4,096 of 4, twice each: 237 us with a
// thread a value, 102 here.
constexpr int RUN = 8;

template <typename T> struct OutVec;
template <> struct OutVec<float> {
    static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct OutVec<__nv_bfloat16> {
    static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
        uint32_t r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
            r[q] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(r[0], r[1], r[2], r[3]);
    }
};

template <typename T, int K>
__global__ void __launch_bounds__(128) short_conv_runs_kernel(ConvArgs a) {
    sb::pdl_launch_dependents();
    constexpr int VEC = Vec16<T>::N;
    const int c = (blockIdx.x * 128 + threadIdx.x) * VEC;
    const int n0 = blockIdx.y * RUN;
    sb::pdl_wait();
    if (c >= a.C) return;
    const T* in = (const T*)a.in + c;
    Vec16<T> raw[RUN];
#pragma unroll
    for (int i = 0; i < RUN; ++i)
        if (n0 + i < a.N) raw[i].load(in + (size_t)(n0 + i) * a.in_stride);
    float tap[VEC * K], ib[VEC], cb[VEC];
#pragma unroll
    for (int i = 0; i < VEC * K; i += 4) *reinterpret_cast<float4*>(tap + i) = *reinterpret_cast<const float4*>(a.taps + (size_t)c * K + i);
#pragma unroll
    for (int e = 0; e < VEC; e += 4) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(ib + e) = a.in_bias ? *reinterpret_cast<const float4*>(a.in_bias + c + e) : zero;
        *reinterpret_cast<float4*>(cb + e) = a.conv_bias ? *reinterpret_cast<const float4*>(a.conv_bias + c + e) : zero;
    }
    int s = 0;                                              // the destination of these channels
    while (s < a.nseg - 1 && !(c >= a.seg[s].begin && c < a.seg[s].end)) ++s;
    const ConvSeg& g = a.seg[s];
    const bool lands = c >= g.begin && c < g.end;
    const int e0 = c - g.begin, head = g.paged ? e0 / g.head_dim : 0, x0 = e0 - head * g.head_dim;
    float hist[K][VEC];                                     // [b]: b + 1 tokens back (the last row is not used)
    int row_before = -1;
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
        const int n = n0 + i;
        if (n >= a.N) break;
        const int row = a.token_rows[n], pos = a.positions[n];
        if (i == 0 || row != row_before) {
            int same = 0;
            for (int b = 1; b < K; ++b) {
                if (n - b >= 0 && a.token_rows[n - b] == row) same = b;
                else break;
            }
#pragma unroll
            for (int b = 1; b < K; ++b) {
                if (pos - b < 0) continue;                  // before the sequence's start
                if (b <= same) {
                    Vec16<T> v;
                    v.load(in + (size_t)(n - b) * a.in_stride);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) hist[b - 1][e] = a.in_bias ? v.get(e) + ib[e] : v.get(e);
                } else {
                    const float* t = a.tail + ((size_t)row * (K - 1) + (K - 1 - b + same)) * a.C + c;
#pragma unroll
                    for (int e = 0; e < VEC; e += 4) *reinterpret_cast<float4*>(&hist[b - 1][e]) = *reinterpret_cast<const float4*>(t + e);
                }
            }
        }
        row_before = row;
        float out[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            const float u = a.in_bias ? raw[i].get(e) + ib[e] : raw[i].get(e);
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < K - 1; ++j)
                if (pos - (K - 1 - j) >= 0) acc = fmaf(tap[e * K + j], hist[K - 2 - j][e], acc);
            acc = fmaf(tap[e * K + K - 1], u, acc);
            if (a.conv_bias) acc += cb[e];
            if (a.act == 1) acc = acc / (1.0f + expf(-acc));
            out[e] = acc;
#pragma unroll
            for (int b = K - 1; b > 0; --b) hist[b][e] = hist[b - 1][e];
            hist[0][e] = u;
        }
        if (!lands) continue;
        if (!g.paged) {
            OutVec<T>::store((T*)g.dst + (size_t)n * g.stride + e0, out);
        } else {
            const int page = a.block_table[(size_t)row * a.table_width + pos / a.page_size];
            OutVec<T>::store((T*)g.dst + (((size_t)page * g.heads + head) * a.page_size + pos % a.page_size) * g.head_dim + x0, out);
        }
    }
}

// Whether the kernel above takes a call: 2 to 4 taps and whole 16-byte pieces of every row, range and head.
template <typename T> bool runs_take(const ConvArgs& a) {
    constexpr int VEC = Vec16<T>::N;
    uintptr_t bits = reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.taps) | reinterpret_cast<uintptr_t>(a.tail) |
                     reinterpret_cast<uintptr_t>(a.in_bias) | reinterpret_cast<uintptr_t>(a.conv_bias);
    bool ok = a.K >= 2 && a.K <= 4 && a.C % VEC == 0 && a.in_stride % VEC == 0;
    for (int s = 0; s < a.nseg; ++s) {
        bits |= reinterpret_cast<uintptr_t>(a.seg[s].dst);
        ok = ok && a.seg[s].begin % VEC == 0 && a.seg[s].end % VEC == 0 && a.seg[s].stride % VEC == 0 &&
             (!a.seg[s].paged || a.seg[s].head_dim % VEC == 0);
    }
    // a channel in two ranges goes to both in the kernel above
    for (int s = 1; s < a.nseg; ++s)
        for (int q = 0; q < s; ++q) ok = ok && (a.seg[s].begin >= a.seg[q].end || a.seg[q].begin >= a.seg[s].end);
    return ok && (bits & 15) == 0;
}
template <typename T> void launch_runs(const ConvArgs& a, cudaStream_t stream) {
    constexpr int VEC = Vec16<T>::N;
    const dim3 grid((a.C / VEC + 127) / 128, (a.N + RUN - 1) / RUN), block(128);
    if (a.K == 2) sb::launch(short_conv_runs_kernel<T, 2>, grid, block, 0, stream, a);
    else if (a.K == 3) sb::launch(short_conv_runs_kernel<T, 3>, grid, block, 0, stream, a);
    else sb::launch(short_conv_runs_kernel<T, 4>, grid, block, 0, stream, a);
}

// One thread per (request, channel): the new tail is the last K-1 values of (old tail, this portion).
template <typename T>
__global__ void __launch_bounds__(256) short_conv_tail_kernel(float* __restrict__ tail, const T* __restrict__ in,
                                                              long long in_stride, const float* __restrict__ in_bias,
                                                              int C, int K, const int* __restrict__ seq_starts,
                                                              const int* __restrict__ seq_rows) {
    sb::pdl_launch_dependents();
    sb::pdl_wait();
    const int r = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int n0 = seq_starts[r], n1 = seq_starts[r + 1], len = n1 - n0;
    const int row = seq_rows[r];
    const float bias = in_bias ? in_bias[c] : 0.f;
    float* t = tail + (size_t)row * (K - 1) * C + c;
    float v[MAX_TAPS];
#pragma unroll
    for (int i = 0; i < MAX_TAPS; ++i) {
        if (i >= K - 1) break;
        const int from_end = K - 1 - i;                     // this entry is the from_end-th value from the end
        if (from_end <= len) v[i] = to_float(in[(size_t)(n1 - from_end) * in_stride + c]) + bias;
        else v[i] = t[(size_t)(i + len) * C];
    }
#pragma unroll
    for (int i = 0; i < MAX_TAPS; ++i) {
        if (i >= K - 1) break;
        t[(size_t)i * C] = v[i];
    }
}

}  // namespace

// Whether N tokens of `requests` requests by C channels of K taps go by runs (short_conv_runs_kernel) where their layout allows
// it (1) or a value a thread (0).  A run is eight tokens one after another, 9 to 14 us whatever their number, and more where a
// run meets many requests (each starts with a round trip for its row and one for its tail); a thread a value takes a time in
// proportion to the values.  Runs / a thread a value (us), by millions (2^20) of values: 4 taps in bfloat16, one portion: 0.75
// 10.9 / 9.7, 1.0 11.4 / 12.4, 2.0 12.0 / 22.8; decoding requests: 0.25 12.9 / 4.7 (64 through 4,096 channels), 1.0 14.3 / 12.0,
// 1.25 14.6 / 14.4, 1.5 14.7 / 16.9; one decoding request in eight tokens: 1.0 13.8 / 12.3, 1.25 13.9 / 14.9; 2 taps, decoding:
// 1.25 11.8 / 10.8, 1.5 11.9 / 12.5.  float32, 4 taps: one portion 0.5 6.7 / 7.1; decoding 0.75 9.7 / 9.4, 1.0 9.9 / 11.8.
extern "C" int sb_short_conv_pays_runs(int N, int C, int K, int requests, int dtype) {
    long long least = requests <= 2 ? (dtype == SB_BF16 ? 1 << 20 : 1 << 19) : (dtype == SB_BF16 ? 5 << 18 : 7 << 17);
    if (K == 2) least += least / 4;
    return (long long)N * C >= least;
}

// seg_*: arrays of `nseg` entries describing the destinations (see ConvSeg).  `requests`: how many the tokens are of (for the
// choice of the kernel alone; as many as tokens where it is not known).
extern "C" int sb_short_conv(const void* in, long long in_stride, const float* in_bias, const float* taps,
                             const float* conv_bias, int act, const float* tail, int C, int K, int N,
                             const int* token_rows, const int* positions, const int* block_table,
                             int table_width, int page_size, int nseg, const int* seg_begin, const int* seg_end,
                             const int* seg_paged, void* const* seg_dst, const long long* seg_stride,
                             const int* seg_heads, const int* seg_head_dim, int requests, int dtype, cudaStream_t stream) {
    SB_REQUIRE(C > 0 && N >= 0 && K >= 1 && K <= MAX_TAPS, "short_conv: bad sizes C=%d N=%d taps=%d (at most %d)", C, N, K,
               MAX_TAPS);
    SB_REQUIRE(nseg >= 1 && nseg <= 3, "short_conv: %d destinations (1 to 3)", nseg);
    SB_REQUIRE(K == 1 || tail != nullptr, "short_conv: %d taps need a tail state", K);
    SB_REQUIRE(N <= 65535, "short_conv: %d tokens exceed one launch", N);
    if (N == 0) return 0;
    ConvArgs a;
    a.in = in; a.in_stride = in_stride; a.in_bias = in_bias; a.taps = taps; a.conv_bias = conv_bias; a.act = act;
    a.tail = tail; a.C = C; a.K = K; a.N = N; a.token_rows = token_rows; a.positions = positions;
    a.block_table = block_table; a.table_width = table_width; a.page_size = page_size; a.nseg = nseg;
    for (int s = 0; s < nseg; ++s) {
        a.seg[s].begin = seg_begin[s]; a.seg[s].end = seg_end[s]; a.seg[s].paged = seg_paged[s];
        a.seg[s].dst = seg_dst[s]; a.seg[s].stride = seg_stride[s]; a.seg[s].heads = seg_heads[s];
        a.seg[s].head_dim = seg_head_dim[s];
        SB_REQUIRE(!a.seg[s].paged || (block_table != nullptr && page_size > 0 && a.seg[s].head_dim > 0),
                   "short_conv: a paged destination needs a block table");
    }
    if (sb_short_conv_pays_runs(N, C, K, requests, dtype) &&
        ((dtype == SB_F32 && runs_take<float>(a)) || (dtype == SB_BF16 && runs_take<__nv_bfloat16>(a)))) {
        if (dtype == SB_F32) launch_runs<float>(a, stream);
        else launch_runs<__nv_bfloat16>(a, stream);
        SB_LAUNCH_CHECK();
    }
    dim3 grid((C + 255) / 256, N);
    if (dtype == SB_F32) sb::launch(short_conv_kernel<float>, grid, dim3(256), 0, stream, a);
    else if (dtype == SB_BF16) sb::launch(short_conv_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, a);
    else SB_REQUIRE(false, "short_conv: unknown dtype %d", dtype);
    SB_LAUNCH_CHECK();
}

extern "C" int sb_short_conv_tail(float* tail, const void* in, long long in_stride, const float* in_bias, int C,
                                  int K, const int* seq_starts, const int* seq_rows, int R, int dtype,
                                  cudaStream_t stream) {
    SB_REQUIRE(C > 0 && R >= 0 && K >= 1 && K <= MAX_TAPS, "short_conv_tail: bad sizes C=%d R=%d taps=%d", C, R, K);
    if (R == 0 || K == 1) return 0;
    dim3 grid((C + 255) / 256, R);
    if (dtype == SB_F32)
        sb::launch(short_conv_tail_kernel<float>, grid, dim3(256), 0, stream, tail, (const float*)in, in_stride, in_bias,
                   C, K, seq_starts, seq_rows);
    else if (dtype == SB_BF16)
        sb::launch(short_conv_tail_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, tail, (const __nv_bfloat16*)in,
                   in_stride, in_bias, C, K, seq_starts, seq_rows);
    else
        SB_REQUIRE(false, "short_conv_tail: unknown dtype %d", dtype);
    SB_LAUNCH_CHECK();
}
