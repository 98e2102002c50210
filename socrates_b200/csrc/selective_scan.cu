// Selective scan (Mamba): a diagonal state space per channel whose step size and input and
// output maps depend on the token.  Per channel c and state index n, S a float32 state carried
// from token to token in the request's slot [rows, inner, states]:
//   dt = softplus(dt_raw[c] + dt_bias[c])
//   S[c][n] = exp(dt * A[c][n]) * S[c][n] + dt * x[c] * B[n],      A = -exp(A_log)
//   y[c] = sum_n S[c][n] * C[n] + D[c] * x[c]
//   out[c] = y[c] * silu(z[c])
// Step sizes, decays, exponentials and the state are float32; x, z, B and C come in the model dtype.
//
// A block serves some channels of one request and walks its tokens of the step in order; TS
// threads share a channel and add their parts of y by shuffles in a fixed order.  B and C of a few
// tokens at a time go through shared memory.  selective_scan_quads_kernel serves the usual numbers of
// states (8, 16, 32 or 64, four neighbours a thread); selective_scan_kernel every other one.
#include <math.h>

#include "common.cuh"
#include "f32x2.cuh"

using namespace sb;

namespace {

// exp of a decay's exponent (dt * A <= 0).  The float32 engine uses expf; in the bfloat16 engine, whose
// activations carry 8 bits, the hardware exponential (a relative error near 1e-6) is far below what the
// activations' rounding leaves, and the kernel is bound by these instructions.
template <typename T> __device__ __forceinline__ float decay_exp(float x) { return expf(x); }
template <> __device__ __forceinline__ float decay_exp<__nv_bfloat16>(float x) { return __expf(x); }

constexpr int THREADS = 128;
constexpr int TOKENS = 16;       // tokens whose B and C are staged (and whose dt, x, z are loaded) at once
constexpr int NPT = 8;           // states per thread at most
constexpr int SEGMENT = 128;     // tokens per segment of the three-launch form (a multiple of TOKENS)

struct ScanArgs {
    const void* x;           // [N, x_stride] in T, channel c at column c
    long long x_stride;
    const void* z;           // [N, z_stride] in T
    long long z_stride;
    const float* dt_raw;     // [N, inner]
    const float* dt_bias;    // [inner]
    const void* bc;          // [N, bc_stride] in T: B (states) | C (states)
    long long bc_stride;
    const float* A_log;      // [inner, states]
    const float* D;          // [inner]
    float* state;            // [rows, inner, states]
    void* out;               // [N, inner] in T
    const int* seq_starts;
    const int* seq_rows;
    int inner, states, TS;
    int R, seg;              // requests of the step; tokens per segment of the three-launch form
    float* seg_state;        // [segments of the step, inner, states]
    float* seg_dt;           // [segments of the step, inner]: the sum of the step sizes in the segment
};

// The segments of a step in one list: request 0's, then request 1's, ...  Finds segment g's request and its
// number within the request; false if the step has fewer segments.
__device__ __forceinline__ bool find_segment(int g, const int* seq_starts, int R, int len, int& r, int& si) {
    for (r = 0; r < R; ++r) {
        const int ns = (seq_starts[r + 1] - seq_starts[r] + len - 1) / len;
        if (g < ns) { si = g; return true; }
        g -= ns;
    }
    return false;
}

// MODE 0: a block walks all tokens of its request (decode steps; many requests).  One long prompt has too
// few channels to fill the GPU that way (a warp per scheduler, every step's latency exposed), so it runs as
// three launches over segments of `seg` tokens, each segment a block row of its own:
// MODE 1: the segment from a zero state: its final state and the sum of its step sizes, to scratch;
// (selective_scan_join_kernel walks a request's segments: S <- exp(A * sum dt) S + contribution, and leaves
//  the state BEFORE each segment in scratch and the state after the last in the request's slot;)
// MODE 2: the segment again from the state before it, this time writing the outputs.
template <typename T, int MODE>
__global__ void __launch_bounds__(THREADS) selective_scan_kernel(ScanArgs a) {
    sb::pdl_launch_dependents();
    extern __shared__ float bcs[];          // TOKENS * 2 * states, then (dt, dt*x, D*x, silu(z)) per channel and token
    float* tok = bcs + TOKENS * 2 * a.states;
    const int TS = a.TS, states = a.states;
    const int tid = threadIdx.x;
    const int l = tid % TS;
    const int c = blockIdx.x * (THREADS / TS) + tid / TS;
    const bool live = c < a.inner;
    int r = blockIdx.y, si = 0;
    float A[NPT], S[NPT];
#pragma unroll
    for (int e = 0; e < NPT; ++e) {
        const int n = l + e * TS;
        A[e] = (live && n < states) ? -expf(a.A_log[(size_t)c * states + n]) : 0.f;
    }
    const float bias = live ? a.dt_bias[c] : 0.f;
    const float Dc = live ? a.D[c] : 0.f;
    sb::pdl_wait();
    if (MODE != 0 && !find_segment(blockIdx.y, a.seq_starts, a.R, a.seg, r, si)) return;
    const int n0 = MODE == 0 ? a.seq_starts[r] : a.seq_starts[r] + si * a.seg;
    const int n1 = MODE == 0 ? a.seq_starts[r + 1] : min(a.seq_starts[r + 1], n0 + a.seg);
    const int row = a.seq_rows[r];
    float* st = MODE == 0 ? a.state + ((size_t)row * a.inner + (live ? c : 0)) * states
                          : a.seg_state + ((size_t)blockIdx.y * a.inner + (live ? c : 0)) * states;
#pragma unroll
    for (int e = 0; e < NPT; ++e) {
        const int n = l + e * TS;
        S[e] = (MODE != 1 && live && n < states) ? st[n] : 0.f;
    }
    float dt_sum = 0.f;
    const T* xs = (const T*)a.x;
    const T* zs = (const T*)a.z;
    const T* bc = (const T*)a.bc;
    for (int t0 = n0; t0 < n1; t0 += TOKENS) {
        const int nt = min(TOKENS, n1 - t0);
        __syncthreads();
        for (int i = tid; i < nt * 2 * states; i += THREADS) {
            const int t = i / (2 * states), k = i - t * 2 * states;
            bcs[i] = to_float(bc[(size_t)(t0 + t) * a.bc_stride + k]);
        }
        __syncthreads();
        // The tokens' own values, made once per channel: lane l of a channel's group takes the tokens
        // t = l, l + TS, ... (loads first, all in flight), computes the step size, its product with x and
        // the output gate, and leaves them in shared memory for the group.
        {
            float raws[TOKENS], xv[TOKENS], zv[TOKENS];
#pragma unroll
            for (int k = 0; k < TOKENS; ++k) {
                const int t = l + k * TS;
                raws[k] = xv[k] = zv[k] = 0.f;
                if (live && t < nt) {
                    const int n = t0 + t;
                    raws[k] = a.dt_raw[(size_t)n * a.inner + c];
                    xv[k] = to_float(xs[(size_t)n * a.x_stride + c]);
                    zv[k] = to_float(zs[(size_t)n * a.z_stride + c]);
                }
            }
#pragma unroll
            for (int k = 0; k < TOKENS; ++k) {
                const int t = l + k * TS;
                if (t < nt) {
                    const float raw = raws[k] + bias;
                    const float dt = raw > 20.f ? raw : log1pf(expf(raw));
                    float* o = tok + ((tid / TS) * TOKENS + t) * 4;
                    dt_sum += dt;
                    o[0] = dt;
                    o[1] = dt * xv[k];
                    o[2] = Dc * xv[k];
                    o[3] = zv[k] / (1.0f + expf(-zv[k]));
                }
            }
        }
        __syncwarp();
#pragma unroll 4
        for (int t = 0; t < nt; ++t) {
            const float4 v = *reinterpret_cast<const float4*>(tok + ((tid / TS) * TOKENS + t) * 4);
            const float dt = v.x, dx = v.y;
            const float* Bt = bcs + t * 2 * states;
            const float* Ct = Bt + states;
            float y = 0.f;
#pragma unroll
            for (int e = 0; e < NPT; ++e) {
                const int k = l + e * TS;
                if (k < states) {
                    S[e] = fmaf(decay_exp<T>(dt * A[e]), S[e], dx * Bt[k]);
                    y = fmaf(S[e], Ct[k], y);
                }
            }
            if (MODE != 1) {
                for (int o = TS >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                if (live && l == 0) ((T*)a.out)[(size_t)(t0 + t) * a.inner + c] = from_float<T>((y + v.z) * v.w);
            }
        }
        __syncwarp();
    }
    if (MODE == 1) {
        for (int o = TS >> 1; o > 0; o >>= 1) dt_sum += __shfl_xor_sync(0xffffffffu, dt_sum, o);
        if (live && l == 0) a.seg_dt[(size_t)blockIdx.y * a.inner + c] = dt_sum;
    }
    if (live && MODE != 2) {
#pragma unroll
        for (int e = 0; e < NPT; ++e) {
            const int n = l + e * TS;
            if (n < states) st[n] = S[e];
        }
    }
}

// ----------------------------------------------------------------------------------------
// The usual numbers of states: TS = 2, 4, 8 or 16 threads a channel with four neighbouring states each, so that a token costs
// a thread one 16-byte load of B and one of C, two-wide multiply-adds and nothing that is not its own.  What bounds it is the
// exponential unit (one per state and token, 16 a clock and SM); everything else has to fit beside that:
//   * the tokens' own values (step size, its product with x, D x, the gate) are made by threads that lie along the channels
//     (whole lines of dt_raw, x and z), the next sixteen tokens' loads in flight while these are walked;
//   * A is held times log2(e), so that a decay is one product and one ex2 (bfloat16 engine);
//   * y is summed for TS tokens at once: each shuffle halves the tokens a lane keeps, so the group's lane l ends with the sum of
//     token l, gates and stores it (TS - 1 shuffles for TS tokens, the sums in the order of a butterfly).
// 1,500 tokens by 4,096 channels of 16 states, both passes and the join (bfloat16): 456 us with a thread's states TS apart, a
// shuffle tree a token and eight predicated states a thread whatever their number, 108 here (the exponentials alone, twice
// 98 M of them, are 44); 2,048 tokens 652 / 138, 187 tokens of two requests in one launch 99 / 27.
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    sb::fma2(c, a, b);
    return c;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& lo, float& hi) { lo = low(v); hi = high(v); }
// exp(dt * A) from dt * `unit`: the float32 engine's `unit` is A, the bfloat16 engine's A * log2(e) (see decay_exp)
template <typename T> __device__ __forceinline__ float decay_unit(float A) { return A; }
template <> __device__ __forceinline__ float decay_unit<__nv_bfloat16>(float A) { return A * 1.4426950408889634f; }
template <typename T> __device__ __forceinline__ float decay_of(float x) { return expf(x); }
template <> __device__ __forceinline__ float decay_of<__nv_bfloat16>(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <typename T, int MODE, int TS>
__global__ void __launch_bounds__(THREADS) selective_scan_quads_kernel(ScanArgs a) {
    sb::pdl_launch_dependents();
    constexpr int STATES = 4 * TS;
    constexpr int CH = THREADS / TS;                        // channels of a block
    constexpr int ITEMS = TOKENS / TS;                      // (token, channel) values that a thread makes of a stage
    __shared__ float2 steps[2][TOKENS][CH];                 // dt, dt * x
    __shared__ float2 gates[MODE == 1 ? 1 : 2][MODE == 1 ? 1 : TOKENS][CH];     // D * x, silu(z)
    __shared__ __align__(16) float bcs[2][TOKENS * 2 * STATES];
    const int tid = threadIdx.x;
    const int l = tid % TS, ch = tid / TS;                  // in the walk: states 4 l .. 4 l + 3 of channel ch
    const int mc = tid % CH, mt = tid / CH;                 // in the making: channel mc of tokens mt, mt + TS, ...
    const int c = blockIdx.x * CH + ch;
    const bool live = c < a.inner;
    const int cm = blockIdx.x * CH + mc;
    const bool making = cm < a.inner;
    float unit[4];
    {
        const float4 v = live ? *reinterpret_cast<const float4*>(a.A_log + (size_t)c * STATES + 4 * l) : make_float4(0.f, 0.f, 0.f, 0.f);
        unit[0] = decay_unit<T>(-expf(v.x));
        unit[1] = decay_unit<T>(-expf(v.y));
        unit[2] = decay_unit<T>(-expf(v.z));
        unit[3] = decay_unit<T>(-expf(v.w));
    }
    const unsigned long long unit01 = pair(unit[0], unit[1]), unit23 = pair(unit[2], unit[3]);
    const float bias = making ? a.dt_bias[cm] : 0.f;
    const float Dc = making ? a.D[cm] : 0.f;
    sb::pdl_wait();
    int r = blockIdx.y, si = 0;
    if (MODE != 0 && !find_segment(blockIdx.y, a.seq_starts, a.R, a.seg, r, si)) return;
    const int n0 = MODE == 0 ? a.seq_starts[r] : a.seq_starts[r] + si * a.seg;
    const int n1 = MODE == 0 ? a.seq_starts[r + 1] : min(a.seq_starts[r + 1], n0 + a.seg);
    float* st = (MODE == 0 ? a.state + ((size_t)a.seq_rows[r] * a.inner + (live ? c : 0)) * STATES
                           : a.seg_state + ((size_t)blockIdx.y * a.inner + (live ? c : 0)) * STATES) + 4 * l;
    unsigned long long S01 = 0ull, S23 = 0ull;
    if (MODE != 1 && live) {
        const float4 v = *reinterpret_cast<const float4*>(st);
        S01 = pair(v.x, v.y);
        S23 = pair(v.z, v.w);
    }
    const T* xs = (const T*)a.x;
    const T* zs = (const T*)a.z;
    const T* bc = (const T*)a.bc;
    float raws[ITEMS];
    T xv[ITEMS], zv[ITEMS], bv[TS];
    auto fetch = [&](int t0) {
        const int nt = min(TOKENS, n1 - t0);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int t = mt + k * TS;
            raws[k] = 0.f;
            xv[k] = zv[k] = from_float<T>(0.f);
            if (making && t < nt) {
                const size_t n = t0 + t;
                raws[k] = a.dt_raw[n * a.inner + cm];
                xv[k] = xs[n * a.x_stride + cm];
                if (MODE != 1) zv[k] = zs[n * a.z_stride + cm];
            }
        }
#pragma unroll
        for (int k = 0; k < TS; ++k) {
            const int i = tid + k * THREADS, t = i / (2 * STATES), col = i % (2 * STATES);
            bv[k] = t < nt ? bc[(size_t)(t0 + t) * a.bc_stride + col] : from_float<T>(0.f);
        }
    };
    float dt_sum = 0.f;
    if (n0 < n1) fetch(n0);
    int buf = 0;
    for (int t0 = n0; t0 < n1; t0 += TOKENS, buf ^= 1) {
        const int nt = min(TOKENS, n1 - t0);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int t = mt + k * TS;
            if (t < nt) {
                const float raw = raws[k] + bias, x = to_float(xv[k]), z = to_float(zv[k]);
                const float dt = raw > 20.f ? raw : log1pf(expf(raw));
                dt_sum += dt;
                steps[buf][t][mc] = make_float2(dt, dt * x);
                if constexpr (MODE != 1) gates[buf][t][mc] = make_float2(Dc * x, z / (1.0f + expf(-z)));
            }
        }
#pragma unroll
        for (int k = 0; k < TS; ++k) bcs[buf][tid + k * THREADS] = to_float(bv[k]);
        // (one barrier a stage: the buffer that the next stage writes was last read before this one)
        __syncthreads();
        if (t0 + TOKENS < n1) fetch(t0 + TOKENS);
        auto walk = [&](int t) {                            // token t of the stage; the thread's part of its y
            const float2 v = steps[buf][t][ch];
            const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(&bcs[buf][t * 2 * STATES + 4 * l]);
            const unsigned long long dt2 = pair(v.x, v.x), dx2 = pair(v.y, v.y);
            float e0, e1, e2, e3;
            unpair(mul2(dt2, unit01), e0, e1);
            unpair(mul2(dt2, unit23), e2, e3);
            S01 = fma2(pair(decay_of<T>(e0), decay_of<T>(e1)), S01, mul2(dx2, B.x));
            S23 = fma2(pair(decay_of<T>(e2), decay_of<T>(e3)), S23, mul2(dx2, B.y));
            float lo = 0.f, hi = 0.f;
            if constexpr (MODE != 1) {
                const ulonglong2 C = *reinterpret_cast<const ulonglong2*>(&bcs[buf][t * 2 * STATES + STATES + 4 * l]);
                unpair(fma2(S23, C.y, mul2(S01, C.x)), lo, hi);
            }
            return lo + hi;
        };
#pragma unroll 1
        for (int tb = 0; tb < nt; tb += TS) {
            float y[TS];
            if (tb + TS <= nt) {
#pragma unroll
                for (int j = 0; j < TS; ++j) y[j] = walk(tb + j);
            } else {
#pragma unroll
                for (int j = 0; j < TS; ++j) y[j] = tb + j < nt ? walk(tb + j) : 0.f;
            }
            if constexpr (MODE != 1) {
#pragma unroll
                for (int o = TS >> 1; o > 0; o >>= 1) {
                    const bool upper = (l & o) != 0;
#pragma unroll
                    for (int i = 0; i < o; ++i) {
                        const float keep = upper ? y[i + o] : y[i], send = upper ? y[i] : y[i + o];
                        y[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                if (live && tb + l < nt) {
                    const float2 g = gates[buf][tb + l][ch];
                    ((T*)a.out)[(size_t)(t0 + tb + l) * a.inner + c] = from_float<T>((y[0] + g.x) * g.y);
                }
            }
        }
    }
    if (MODE == 1) {
        __syncthreads();                                    // everybody is done with the steps
        float* sums = reinterpret_cast<float*>(steps);      // [TS][CH]
        sums[mt * CH + mc] = dt_sum;
        __syncthreads();
        if (mt == 0 && making) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < TS; ++k) s += sums[k * CH + mc];
            a.seg_dt[(size_t)blockIdx.y * a.inner + cm] = s;
        }
    }
    if (MODE != 2 && live) {
        float4 v;
        unpair(S01, v.x, v.y);
        unpair(S23, v.z, v.w);
        *reinterpret_cast<float4*>(st) = v;
    }
}

template <int MODE> void launch_scan(const ScanArgs& a, dim3 grid, size_t smem, bool quads, int dtype, cudaStream_t stream) {
    const dim3 block(THREADS);
#define SB_SCAN(T)                                                                                              \
    if (!quads) sb::launch(selective_scan_kernel<T, MODE>, grid, block, smem, stream, a);                        \
    else if (a.TS == 2) sb::launch(selective_scan_quads_kernel<T, MODE, 2>, grid, block, 0, stream, a);          \
    else if (a.TS == 4) sb::launch(selective_scan_quads_kernel<T, MODE, 4>, grid, block, 0, stream, a);          \
    else if (a.TS == 8) sb::launch(selective_scan_quads_kernel<T, MODE, 8>, grid, block, 0, stream, a);          \
    else sb::launch(selective_scan_quads_kernel<T, MODE, 16>, grid, block, 0, stream, a);
    if (dtype == SB_F32) { SB_SCAN(float) } else { SB_SCAN(__nv_bfloat16) }
#undef SB_SCAN
}

// Between MODE 1 and MODE 2: one thread per (channel, state) of a request walks its segments.
__global__ void __launch_bounds__(256) selective_scan_join_kernel(ScanArgs a) {
    sb::pdl_launch_dependents();
    const int i = blockIdx.x * 256 + threadIdx.x, r = blockIdx.y;
    const int size = a.inner * a.states;
    const float A = i < size ? -expf(a.A_log[i]) : 0.f;
    sb::pdl_wait();
    if (i >= size) return;
    int base = 0;
    for (int q = 0; q < r; ++q) base += (a.seq_starts[q + 1] - a.seq_starts[q] + a.seg - 1) / a.seg;
    const int ns = (a.seq_starts[r + 1] - a.seq_starts[r] + a.seg - 1) / a.seg;
    const int c = i / a.states;
    float* slot = a.state + (size_t)a.seq_rows[r] * size + i;
    float s = *slot;
    for (int g0 = 0; g0 < ns; g0 += 8) {                         // eight segments' loads in flight
        float u[8], d[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (g0 + k < ns) {
                u[k] = a.seg_state[(size_t)(base + g0 + k) * size + i];
                d[k] = a.seg_dt[(size_t)(base + g0 + k) * a.inner + c];
            }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (g0 + k < ns) {
                a.seg_state[(size_t)(base + g0 + k) * size + i] = s;
                s = fmaf(expf(A * d[k]), s, u[k]);
            }
    }
    *slot = s;
}

}  // namespace

extern "C" int sb_selective_scan(const void* x, long long x_stride, const void* z, long long z_stride,
                                 const float* dt_raw, const float* dt_bias, const void* bc, long long bc_stride,
                                 const float* A_log, const float* D, float* state, void* out,
                                 const int* seq_starts, const int* seq_rows, int R, int inner, int states, int N,
                                 float* scratch, long long scratch_floats, int dtype, cudaStream_t stream) {
    SB_REQUIRE(R >= 0 && inner > 0 && states > 0 && states <= 32 * NPT,
               "selective_scan: bad sizes R=%d inner=%d states=%d (at most %d)", R, inner, states, 32 * NPT);
    SB_REQUIRE(R <= 65535, "selective_scan: %d requests exceed one launch", R);
    if (R == 0) return 0;
    // threads a channel: a power of two, as few as hold the states at NPT each (what a thread does per token
    // beside its states is the same for every thread of a channel), but four where the states allow it
    int TS = 1;
    while (TS * NPT < states) TS *= 2;
    while (TS < 4 && TS * 2 <= states) TS *= 2;
    // the kernel of neighbouring states: 16-byte pieces of A_log and of the states
    const bool quads = (states == 8 || states == 16 || states == 32 || states == 64) &&
                       ((reinterpret_cast<uintptr_t>(A_log) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(scratch)) & 15) == 0;
    if (quads) TS = states / 4;
    ScanArgs a;
    a.x = x; a.x_stride = x_stride; a.z = z; a.z_stride = z_stride; a.dt_raw = dt_raw; a.dt_bias = dt_bias;
    a.bc = bc; a.bc_stride = bc_stride; a.A_log = A_log; a.D = D; a.state = state; a.out = out;
    a.seq_starts = seq_starts; a.seq_rows = seq_rows; a.inner = inner; a.states = states; a.TS = TS;
    const int per_block = THREADS / TS;
    dim3 grid((inner + per_block - 1) / per_block, R);
    const size_t smem = ((size_t)TOKENS * 2 * states + (size_t)per_block * TOKENS * 4) * sizeof(float);
    SB_REQUIRE(dtype == SB_F32 || dtype == SB_BF16, "selective_scan: unknown dtype %d", dtype);
    // few requests with long portions: segments in parallel (three launches) if the caller lent scratch
    const int segs = (N + SEGMENT - 1) / SEGMENT + R;
    const bool spread = scratch != nullptr && (int)grid.x * R < 4 * 148 && segs > 2 * R &&
                        (long long)segs * inner * (states + 1) <= scratch_floats;
    a.R = R; a.seg = SEGMENT; a.seg_state = scratch; a.seg_dt = scratch ? scratch + (size_t)segs * inner * states : nullptr;
    if (!spread) {
        launch_scan<0>(a, grid, smem, quads, dtype, stream);
        SB_LAUNCH_CHECK();
    }
    dim3 sgrid(grid.x, segs), jgrid((inner * states + 255) / 256, R);
    launch_scan<1>(a, sgrid, smem, quads, dtype, stream);
    sb::launch(selective_scan_join_kernel, jgrid, dim3(256), 0, stream, a);
    launch_scan<2>(a, sgrid, smem, quads, dtype, stream);
    SB_LAUNCH_CHECK();
}

// float32 elements of scratch with which a step of N tokens of R requests can run its segments in parallel.
extern "C" long long sb_selective_scan_scratch(int N, int R, int inner, int states) {
    return (long long)((N + SEGMENT - 1) / SEGMENT + R) * inner * (states + 1);
}
