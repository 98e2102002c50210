// C[M,N] = A[M,K] * W[N,K]^T in float32 on the CUDA cores: the products of the true 32-bit path.  gemm_simt.cu sends
// float32 operands with whole 16-byte pieces here and keeps mixed types, odd K and cut products.
//
// The order of an output's sum is a matter of K alone: K is cut into 4 groups of 4 segments (of whole 16-wide pieces); the
// products of a segment are added in the order of k by fused multiply-adds, segments to their group one after the other, and
// the result is (group 0 + group 1) + (group 2 + group 3).  Both kernels here have that order, in both of their forms: a
// row's numbers are the same bits alone and in any batch.  (Short chains also carry less rounding than one long one.)
//
//   * few rows (M <= 8): bound by the bytes of W.  A block serves 32 columns and its four warps a group each; a warp streams
//     its part of the 32 rows of W through a ring of its own (cp.async), a lane per column, without a barrier in its loop.
//     Decode steps and the head.
//   * many rows: bound by the multiply-adds.  A warp holds a 64 x 64 tile of outputs in registers, 16 x 8 a lane, so that 24
//     floats from shared memory feed 128 multiply-adds (fma.rn.f32x2 on pairs of rows; with 8 x 8 a lane the loads took as
//     long as the products).  Where there are tiles enough the warps of a block are the four groups; else a cluster of
//     four blocks is, whose warps are the segments, and the groups meet through distributed shared memory.
//
// Measured (us, the 64 x 64 tile kernel of gemm_simt.cu / here): 4 rows by 151,936 x 2,560 2,472 / 247 (1.56 GB: 6.3 TB/s);
// 256 rows by 19,456 x 2,560 890 / 638 (40 TFLOP/s), by 2,560 x 9,728 845 / 238 (54), by 2,560 x 4,096 354 / 112 (48).
#include "common.cuh"

using namespace sb;

namespace {

constexpr int PIECE = 16;               // k of a piece
constexpr int GROUPS = 4, SEGMENTS = 4; // groups of K, segments of a group
constexpr int COLS = 32;                // columns of a block of the few-rows kernel
constexpr int NTHR = 32 * GROUPS;

// The first piece of segment `s` (0..16) of `pieces`.
__device__ __forceinline__ int first_piece(int s, int pieces) { return (int)((long long)s * pieces / (GROUPS * SEGMENTS)); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// 16 bytes, or zeros (`bytes` 0: nothing is read)
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ----------------------------------------------------------------------------- few rows
constexpr int RING = 6;                 // pieces in flight or in use per warp
template <int MT> constexpr int few_stage_floats() { return COLS * PIECE + MT * PIECE; }
template <int MT> constexpr int few_smem() { return GROUPS * RING * few_stage_floats<MT>() * 4; }

// W_OLDER: what W holds is older than the kernel before this one on the stream.  (A template argument: with a branch on it
// the loop was scheduled otherwise, 2,560 x 4,096 by one row 16.6 -> 19.8 us.)
template <int MT, bool W_OLDER>
__global__ void __launch_bounds__(NTHR)
gemm_f32_few_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K) {
    sb::pdl_launch_dependents();
    extern __shared__ __align__(16) float smem[];
    constexpr int STAGE = few_stage_floats<MT>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * COLS;
    float* ring = smem + warp * RING * STAGE;
    const int pieces = (K + PIECE - 1) / PIECE;
    const int begin = first_piece(warp * SEGMENTS, pieces), end = first_piece((warp + 1) * SEGMENTS, pieces);
    // 16-byte part p of column n lies at part p ^ (n / 2 % 4) of its row: eight columns' same part then fill all banks
    auto load_w = [&](int i) {
        const int k0 = i * PIECE;
        float* st = ring + ((i - begin) % RING) * STAGE;
#pragma unroll
        for (int j = 0; j < COLS * 4 / 32; ++j) {
            const int idx = lane + 32 * j, n = idx >> 2, p = idx & 3;
            const bool ok = n0 + n < N && k0 + 4 * p < K;
            copy16(smem_addr(st + n * PIECE + ((p ^ ((n >> 1) & 3)) << 2)), ok ? W + (size_t)(n0 + n) * K + k0 + 4 * p : W,
                   ok ? 16 : 0);
        }
    };
    auto load_a = [&](int i) {
        const int k0 = i * PIECE;
        float* st = ring + ((i - begin) % RING) * STAGE + COLS * PIECE;
        if (lane < MT * 4) {
            const int m = lane >> 2, p = lane & 3;
            const bool ok = m < M && k0 + 4 * p < K;
            copy16(smem_addr(st + m * PIECE + 4 * p), ok ? A + (size_t)m * K + k0 + 4 * p : A, ok ? 16 : 0);
        }
    };
    // A, and W too unless it is older, may come from the kernel before this one
    if constexpr (!W_OLDER) sb::pdl_wait();
#pragma unroll
    for (int i = 0; i < RING - 1; ++i)
        if (begin + i < end) load_w(begin + i);
    if constexpr (W_OLDER) sb::pdl_wait();
#pragma unroll
    for (int i = 0; i < RING - 1; ++i) {
        if (begin + i < end) load_a(begin + i);
        copy_commit();                  // the first group holds all weights above
    }
    float total[MT], acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) total[m] = acc[m] = 0.f;
    int seg = 1, seg_end = first_piece(warp * SEGMENTS + 1, pieces);
    for (int i = begin; i < end; ++i) {
        copy_wait<RING - 2>();
        __syncwarp();                   // piece i is there for every lane; every lane is done with piece i - 1
        if (i + RING - 1 < end) {
            load_w(i + RING - 1);
            load_a(i + RING - 1);
        }
        copy_commit();
        while (i == seg_end) {          // a segment ends before this piece
#pragma unroll
            for (int m = 0; m < MT; ++m) { total[m] += acc[m]; acc[m] = 0.f; }
            seg_end = first_piece(warp * SEGMENTS + ++seg, pieces);
        }
        const float* st = ring + ((i - begin) % RING) * STAGE;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float4 w = *reinterpret_cast<const float4*>(st + lane * PIECE + ((p ^ ((lane >> 1) & 3)) << 2));
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(st + COLS * PIECE + m * PIECE + 4 * p);
                acc[m] = fmaf(x.x, w.x, acc[m]);
                acc[m] = fmaf(x.y, w.y, acc[m]);
                acc[m] = fmaf(x.z, w.z, acc[m]);
                acc[m] = fmaf(x.w, w.w, acc[m]);
            }
        }
    }
    copy_wait<0>();
    __syncthreads();
    float* sum = smem;                  // [GROUPS][MT][COLS]
#pragma unroll
    for (int m = 0; m < MT; ++m) sum[(warp * MT + m) * COLS + lane] = total[m] + acc[m];
    __syncthreads();
    for (int idx = threadIdx.x; idx < MT * COLS; idx += NTHR) {
        const int m = idx / COLS, n = n0 + idx % COLS;
        if (m < M && n < N)
            C[(size_t)m * N + n] = (sum[idx] + sum[MT * COLS + idx]) + (sum[2 * MT * COLS + idx] + sum[3 * MT * COLS + idx]);
    }
}

// ----------------------------------------------------------------------------- many rows
constexpr int TILE = 64;                // rows and columns of a tile
constexpr int WARP_FLOATS = TILE * TILE + 2 * PIECE * TILE;     // a warp's sums and its pieces of A and W
constexpr int TILE_SMEM = GROUPS * WARP_FLOATS * 4;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}

// CLUSTER: four blocks are the groups of a tile and the warps of a block its segments; else the warps are the groups.
template <bool CLUSTER>
__global__ void __launch_bounds__(NTHR, 2)
gemm_f32_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                     int row_tiles, int w_older) {
    sb::pdl_launch_dependents();
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = CLUSTER ? blockIdx.x / GROUPS : blockIdx.x, group = CLUSTER ? blockIdx.x % GROUPS : warp;
    // row tiles of the same columns are neighbours: W comes from memory once
    const int m0 = (tile % row_tiles) * TILE, n0 = (tile / row_tiles) * TILE;
    float* sums = smem + warp * TILE * TILE;                            // [TILE][TILE]
    float* as = smem + GROUPS * TILE * TILE + warp * 2 * PIECE * TILE;  // [PIECE][TILE], k-major
    float* ws = as + PIECE * TILE;
    const int pieces = (K + PIECE - 1) / PIECE;
    const int seg0 = group * SEGMENTS + (CLUSTER ? warp : 0), segs = CLUSTER ? 1 : SEGMENTS;
    const int begin = first_piece(seg0, pieces), end = first_piece(seg0 + segs, pieces);
    // a lane copies rows `lane` and `lane + 32`; rows past the end repeat the last one (their results are not written)
    const float* a0 = A + (size_t)min(m0 + lane, M - 1) * K;
    const float* a1 = A + (size_t)min(m0 + lane + 32, M - 1) * K;
    const float* w0 = W + (size_t)min(n0 + lane, N - 1) * K;
    const float* w1 = W + (size_t)min(n0 + lane + 32, N - 1) * K;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 ra[8], rw[8];
    auto fetch_w = [&](int i) {
        const int k0 = i * PIECE;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const bool ok = k0 + 4 * p < K;
            rw[p] = ok ? __ldg(reinterpret_cast<const float4*>(w0 + k0 + 4 * p)) : zero;
            rw[4 + p] = ok ? __ldg(reinterpret_cast<const float4*>(w1 + k0 + 4 * p)) : zero;
        }
    };
    auto fetch_a = [&](int i) {
        const int k0 = i * PIECE;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const bool ok = k0 + 4 * p < K;
            ra[p] = ok ? *reinterpret_cast<const float4*>(a0 + k0 + 4 * p) : zero;
            ra[4 + p] = ok ? *reinterpret_cast<const float4*>(a1 + k0 + 4 * p) : zero;
        }
    };
    if (w_older && begin < end) fetch_w(begin);             // W as in the kernel above
    sb::pdl_wait();
    if (!w_older && begin < end) fetch_w(begin);
    if (begin < end) fetch_a(begin);
    const int tx = lane & 7, ty = lane >> 3;                // columns 4 tx + 32 h + j, rows 4 ty + 16 i + e
    unsigned long long acc[8][8];                           // [pairs of rows: 2 i + e / 2][columns: 4 h + j]
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    // a segment's sums join those of the segments before it (FIRST: become them); each lane has places of its own
    auto flush = [&](bool first) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = 4 * ty + 16 * (i >> 1) + 2 * (i & 1);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4* lo = reinterpret_cast<float4*>(sums + row * TILE + 32 * h + 4 * tx);
                float4* hi = reinterpret_cast<float4*>(sums + (row + 1) * TILE + 32 * h + 4 * tx);
                float l[4], u[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    l[j] = __uint_as_float(static_cast<uint32_t>(acc[i][4 * h + j]));
                    u[j] = __uint_as_float(static_cast<uint32_t>(acc[i][4 * h + j] >> 32));
                    acc[i][4 * h + j] = 0ull;
                }
                const float4 pl = first ? zero : *lo, pu = first ? zero : *hi;
                *lo = make_float4(pl.x + l[0], pl.y + l[1], pl.z + l[2], pl.w + l[3]);
                *hi = make_float4(pu.x + u[0], pu.y + u[1], pu.z + u[2], pu.w + u[3]);
            }
        }
    };
    int i = begin;
    for (int s = 0; s < segs; ++s) {
        const int seg_end = first_piece(seg0 + s + 1, pieces);
        for (; i < seg_end; ++i) {
            __syncwarp();                                   // every lane is done with the piece before
#pragma unroll
            for (int p = 0; p < 4; ++p) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    as[(4 * p + e) * TILE + lane] = reinterpret_cast<const float*>(&ra[p])[e];
                    as[(4 * p + e) * TILE + lane + 32] = reinterpret_cast<const float*>(&ra[4 + p])[e];
                    ws[(4 * p + e) * TILE + lane] = reinterpret_cast<const float*>(&rw[p])[e];
                    ws[(4 * p + e) * TILE + lane + 32] = reinterpret_cast<const float*>(&rw[4 + p])[e];
                }
            }
            __syncwarp();
            if (i + 1 < end) {
                fetch_w(i + 1);
                fetch_a(i + 1);
            }
#pragma unroll 4
            for (int k = 0; k < PIECE; ++k) {
                unsigned long long x[8];
                float y[8];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<ulonglong2*>(x + 2 * q) = *reinterpret_cast<const ulonglong2*>(as + k * TILE + 16 * q + 4 * ty);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float4*>(y + 4 * h) = *reinterpret_cast<const float4*>(ws + k * TILE + 32 * h + 4 * tx);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned long long yy = twice(y[j]);
#pragma unroll
                    for (int r = 0; r < 8; ++r) fma2(acc[r][j], x[r], yy);
                }
            }
        }
        flush(s == 0);
    }
    __syncthreads();
    constexpr int T2 = TILE * TILE;
    if constexpr (CLUSTER) {
        // the segments to this group's sums, then this block's quarter of the tile from all four groups
        for (int idx = threadIdx.x; idx < T2; idx += NTHR) smem[idx] = ((smem[idx] + smem[T2 + idx]) + smem[2 * T2 + idx]) + smem[3 * T2 + idx];
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        for (int idx = group * (T2 / GROUPS) + threadIdx.x; idx < (group + 1) * (T2 / GROUPS); idx += NTHR) {
            float v[GROUPS];
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                uint32_t at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr(smem + idx)), "r"(g));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[g]) : "r"(at) : "memory");
            }
            const int m = m0 + idx / TILE, n = n0 + idx % TILE;
            if (m < M && n < N) C[(size_t)m * N + n] = (v[0] + v[1]) + (v[2] + v[3]);
        }
        // nobody leaves while another block may still read its shared memory
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        for (int idx = threadIdx.x; idx < T2; idx += NTHR) {
            const int m = m0 + idx / TILE, n = n0 + idx % TILE;
            if (m < M && n < N) C[(size_t)m * N + n] = (smem[idx] + smem[T2 + idx]) + (smem[2 * T2 + idx] + smem[3 * T2 + idx]);
        }
    }
}

template <int MT, bool W_OLDER> int launch_few_as(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    auto kernel = gemm_f32_few_kernel<MT, W_OLDER>;
    static sb::OncePerDevice once_per_device;
    bool& configured = once_per_device.flag();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, few_smem<MT>());
        if (e != cudaSuccess) { sb_set_error("gemm_f32: %s", cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    sb::launch(kernel, dim3((N + COLS - 1) / COLS), dim3(NTHR), few_smem<MT>(), stream, C, A, W, M, N, K);
    return 0;
}
template <int MT>
int launch_few(float* C, const float* A, const float* W, int M, int N, int K, int w_older, cudaStream_t stream) {
    return w_older ? launch_few_as<MT, true>(C, A, W, M, N, K, stream) : launch_few_as<MT, false>(C, A, W, M, N, K, stream);
}

}  // namespace

namespace sb {

// Whether the kernels of this file take the operands: whole, aligned 16-byte pieces (a matter of K and of the addresses, not
// of M, so that a row's kernel family never depends on the batch).
bool gemm_f32_takes(const void* C, const void* A, const void* W, int M, int N, int K) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W);
    const long long blocks = (long long)((M + TILE - 1) / TILE) * ((N + TILE - 1) / TILE) * GROUPS;
    return K % 4 == 0 && (bits & 15) == 0 && blocks <= 0x7fffffffLL;
}

// `w_older`: nothing that the kernel before this one on the stream writes is in W (see sb_gemm_simt).
int gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int w_older, cudaStream_t stream) {
    if (M <= 1) return launch_few<1>(C, A, W, M, N, K, w_older, stream);
    if (M <= 2) return launch_few<2>(C, A, W, M, N, K, w_older, stream);
    if (M <= 4) return launch_few<4>(C, A, W, M, N, K, w_older, stream);
    if (M <= 8) return launch_few<8>(C, A, W, M, N, K, w_older, stream);
    static sb::OncePerDevice once_per_device;
    bool& configured = once_per_device.flag();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(gemm_f32_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM);
        if (e != cudaSuccess) { sb_set_error("gemm_f32: %s", cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    const int row_tiles = (M + TILE - 1) / TILE, tiles = row_tiles * ((N + TILE - 1) / TILE);
    int dev = 0, num_sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    // Below three tiles for each of the GPU's places (two blocks an SM) whole tiles fill their last round badly: a tile is
    // dealt to four blocks then.
    if (tiles < 3 * 2 * num_sms)
        sb::launch_cluster(gemm_f32_tile_kernel<true>, dim3(tiles * GROUPS), dim3(NTHR), TILE_SMEM, stream, dim3(GROUPS), C, A, W,
                           M, N, K, row_tiles, w_older);
    else
        sb::launch(gemm_f32_tile_kernel<false>, dim3(tiles), dim3(NTHR), TILE_SMEM, stream, C, A, W, M, N, K, row_tiles,
                   w_older);
    return 0;
}

}  // namespace sb
