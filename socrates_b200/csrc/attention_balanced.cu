// Paged GQA attention of the requests of a step that bring ONE token (bfloat16, mma.sync m16n8k16,
// float32 accumulation), the keys of all of them dealt to the GPU's blocks in equal shares.
//
// What bounds it: the bytes of the cached keys and values (HBM).  The split-key kernel of attention_mma.cu
// cuts every row into the same number of partitions, a number that the batch width alone decides: with rows of
// different lengths the longest row's blocks run on when the others are done, and from 19 rows of 8 KV heads on
// a row is not cut at all.  Here the 64-key tiles of all rows are laid end to end (per KV head) and slot s of W
// takes tiles [s T / W, (s+1) T / W): W slots times the KV heads are as many blocks as fit the GPU at once, so
// all of them end within a tile of each other whatever the lengths are.  The cut is made on the device from the
// rows' positions, so a recorded graph stays valid.  Rows that are alike or short stay with the split-key kernel,
// which has no merge through memory (GQAAttention.prefers_shares says where the line lies).
//
// A block walks its share as one sequence of tiles through a ring of three stages (cp.async); the ring runs on
// across rows, so the copies of the next row's first tiles are in flight while a row is finished.  Page numbers are
// copied from the block table seven tiles ahead, by cp.async too (a read that misses L2 takes as long as a tile).
// A row that lies in one share is written by its block; a row that several shares cut leaves one partial result
// (max, sum, O) per share, and the block that finds the others' done joins them in the order of the keys and clears
// the count.
//
// Requests that bring more than one token have no tiles here: a step that mixes prompt portions with decoding
// requests runs this kernel for the latter and a tile kernel for the former.
//
// Measured (us a launch, cold keys, 32 query and 8 KV heads of 128, split-key kernel / this one): 19 rows of 437 to
// 7,001 keys (257 MB) 110 / 48, i.e. 5.3 TB/s; 64 rows evenly from 256 to 4,096 (572 MB) 109 / 98, 5.9 TB/s.
#include <math.h>

#include "attention_mma.cuh"
#include "score_map.cuh"

namespace {

constexpr int NW = 4;                    // warps of a block; a tile holds 16 keys for each
constexpr int STAGES = 3;
constexpr int AHEAD = 7;                 // tiles that page numbers are read ahead (their copies go out STAGES - 1 ahead)
constexpr int PAGE_SLOTS = 8;            // tiles whose page numbers are held: more than AHEAD, a power of two
constexpr int MAX_REQUESTS = 1024;       // requests of a step (their offsets live in shared memory)

struct BalancedArgs {
    bf16* out;
    float *part_o, *part_ml;             // [Hkv][W][2][G][D] and [Hkv][W][2][G][2]
    int* counters;                       // [R][Hkv], zero before and after
    const bf16 *q, *k_pool, *v_pool;
    const int *block_table, *seq_starts, *seq_rows, *seq_first_pos;
    int table_width, R, Hq, Hkv, BS, window, W;
    float scale_log2;
};

// Where a walk over the tiles of all rows stands: tiles [begin, end) belong to request r.
struct Cursor {
    int r, begin, end, pos, lo, first;   // first: the tile index inside the row of flat tile 0
    __device__ __forceinline__ void seek(int x, const int* pre, const int* spos, int window) {
        while (x >= pre[r + 1]) ++r;
        begin = pre[r];
        end = pre[r + 1];
        pos = spos[r];
        lo = sb::first_visible(pos, window, 0);
        first = lo / KT - begin;
    }
    __device__ __forceinline__ int tile_start(int x) const { return (first + x) * KT; }
};

template <int D, int NBQ> constexpr int balanced_smem(int R) {
    return (STAGES * 2 * KT * D + STAGES * 8 * NBQ * D) * 2 + PAGE_SLOTS * KT * 4 + (4 * R + 4) * 4;
}

template <int D, int NBQ>
__global__ void __launch_bounds__(32 * NW, 2)
attn_decode_balanced_kernel(const BalancedArgs a) {
    sb::pdl_launch_dependents();
    // Before pdl_wait(): the step's offsets, rows, positions and block table (host copies) and keys and values
    // below a row's newest position (earlier steps).
    constexpr int NTHR = 32 * NW;
    constexpr int QROWS = 8 * NBQ;
    constexpr int STAGE = 2 * KT * D;                       // elements of a stage: keys, then values
    extern __shared__ __align__(128) uint8_t smem[];
    bf16* ring = reinterpret_cast<bf16*>(smem);
    bf16* qring = ring + STAGES * STAGE;                    // the query of the row that begins with the stage's tile
    int* pages = reinterpret_cast<int*>(qring + STAGES * QROWS * D);     // [PAGE_SLOTS][64] physical pages of a tile
    int* pre = pages + PAGE_SLOTS * KT;                     // [R + 1] tiles before each request
    int* spos = pre + a.R + 1;                              // [R]
    int* stok = spos + a.R;                                 // [R]
    int* srow = stok + a.R;                                 // [R]
    __shared__ float w_m[NW][16], w_l[NW][16];
    __shared__ int s_scan[NW], s_row0, s_last, s_others, s_first_last;

    const int G = a.Hq / a.Hkv;
    const int bs_log2 = 31 - __clz(a.BS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kh = blockIdx.x % a.Hkv, slot = blockIdx.x / a.Hkv;

    // ---- tiles of every request and their running sum
    int total = 0;
    for (int base = 0; base < a.R; base += NTHR) {
        const int r = base + tid;
        int t = 0;
        if (r < a.R) {
            const int s0 = a.seq_starts[r], pos = a.seq_first_pos[r];
            spos[r] = pos;
            stok[r] = s0;
            srow[r] = a.seq_rows[r];
            if (a.seq_starts[r + 1] - s0 == 1) t = pos / KT - sb::first_visible(pos, a.window, 0) / KT + 1;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += up;
        }
        if (lane == 31) s_scan[warp] = t;
        __syncthreads();
        int before = total;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const int n = s_scan[w];
            if (w < warp) before += n;
            total += n;
        }
        if (r < a.R) pre[r + 1] = before + t;
        __syncthreads();
    }
    if (tid == 0) pre[0] = 0;
    __syncthreads();
    const int T = total;
    const int W = max(1, min(a.W, T));
    if (slot >= W || T == 0) {
        sb::pdl_wait();
        return;
    }
    const int x0 = (int)((long long)slot * T / W), x1 = (int)((long long)(slot + 1) * T / W);
    for (int r = tid; r < a.R; r += NTHR)
        if (pre[r] <= x0 && x0 < pre[r + 1]) s_row0 = r;
    __syncthreads();

    const int n_pages = max(1, KT >> bs_log2);              // logical pages a tile touches
    // Bring the physical page of entry e of tile x to its slot (0 where the row does not reach: such keys are never
    // read, see load_kv_tile).  Asynchronous: part of the commit group that is open.
    auto fetch_page = [&](const Cursor& c, int x, int e) {
        const int logical = (c.tile_start(x) >> bs_log2) + e;
        const bool valid = logical <= (c.pos >> bs_log2);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                     ::"r"(smem_u32(pages + ((x - x0) % PAGE_SLOTS) * KT + e)),
                       "l"(a.block_table + (size_t)srow[c.r] * a.table_width + (valid ? logical : 0)), "r"(valid ? 4 : 0)
                     : "memory");
    };
    for (int i = tid; i < AHEAD * n_pages; i += NTHR) {
        const int x = x0 + i / n_pages;
        if (x < x1) {
            Cursor c;
            c.r = s_row0;
            c.seek(x, pre, spos, a.window);
            fetch_page(c, x, i % n_pages);
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    auto load_query = [&](const Cursor& c, int stage) {
        constexpr int CH = D / 8;
        bf16* qs = qring + stage * QROWS * D;
        for (int idx = tid; idx < QROWS * CH; idx += NTHR) {
            const int row = idx / CH, ch = idx - row * CH;
            const bool valid = row < G;
            cp_async16(smem_u32(qs + tile_off<D>(row, ch)),
                       a.q + ((size_t)stok[c.r] * a.Hq + kh * G + (valid ? row : 0)) * D + ch * 8, valid ? 16 : 0);
        }
    };

    // ---- the first tiles: those below their row's newest key before the wait, the others after it
    Cursor cl;                                              // of the tile whose copies go out
    cl.r = s_row0;
    cl.seek(x0, pre, spos, a.window);
    const Cursor c0 = cl;
#pragma unroll
    for (int late = 0; late < 2; ++late) {
        if (late) sb::pdl_wait();
        cl = c0;
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) {
            const int x = x0 + s;
            if (x >= x1) break;
            if (x >= cl.end) cl.seek(x, pre, spos, a.window);
            const int ts = cl.tile_start(x);
            if ((ts + KT > cl.pos) == (late != 0))
                load_kv_tile<D, KT, NTHR>(ring + s * STAGE, ring + s * STAGE + KT * D, a.k_pool, a.v_pool, pages + s * KT,
                                          ts >> bs_log2, bs_log2, a.Hkv, kh, ts, cl.lo, cl.pos + 1);
            if (late && (s == 0 || x == cl.begin)) load_query(cl, s);
        }
    }
    cp_async_commit();
#pragma unroll
    for (int s = 1; s < STAGES - 1; ++s) cp_async_commit();

    // the shares [first_share, end_share) that the tiles [begin, end) of a row fall into, and the place of a share's
    // partial result
    auto first_share = [&](int begin) { return (int)(((long long)(begin + 1) * W + T - 1) / T) - 1; };
    auto end_share = [&](int end) { return (int)(((long long)end * W + T - 1) / T); };
    auto piece_of = [&](int s, int begin) {
        return ((size_t)kh * a.W + s) * 2 + (begin <= (int)((long long)s * T / W) ? 0 : 1);
    };
    // Four neighbouring outputs of head `row` out of the partial results of all shares, in the order of the keys; share
    // `mine`'s (-1: none) are the M, L and o that come in: the numbers do not depend on which share came last.
    auto join = [&](int begin, int end, int mine, int row, int idx, float& M, float& L, float4& o) {
        constexpr int U = 8;                                // partial results in flight
        const float2 my_ml = make_float2(M, L);
        const float4 my_o = o;
        M = -INFINITY;
        L = 0.f;
        o = make_float4(0.f, 0.f, 0.f, 0.f);
        const int s_end = end_share(end);
        for (int s0 = first_share(begin); s0 < s_end; s0 += U) {
            float2 ml[U];
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = s0 + u;
                ml[u] = make_float2(-INFINITY, 0.f);
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (s == mine) {
                    ml[u] = my_ml;
                    v[u] = my_o;
                } else if (s < s_end) {
                    const size_t p = piece_of(s, begin);
                    ml[u] = __ldcg(reinterpret_cast<const float2*>(a.part_ml + (p * G + row) * 2));
                    v[u] = __ldcg(reinterpret_cast<const float4*>(a.part_o + p * G * D + idx));
                }
            }
            float top = M;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (ml[u].y > 0.f) top = fmaxf(top, ml[u].x);
            const float keep = L > 0.f ? exp2f(M - top) : 0.f;
            L *= keep;
            o.x *= keep; o.y *= keep; o.z *= keep; o.w *= keep;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (ml[u].y > 0.f) {
                    const float f = exp2f(ml[u].x - top);
                    L += f * ml[u].y;
                    o.x += f * v[u].x; o.y += f * v[u].y; o.z += f * v[u].z; o.w += f * v[u].w;
                }
            M = top;
        }
    };
    auto write4 = [&](int r, int idx, float L, const float4& o) {
        __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(a.out + ((size_t)stok[r] * a.Hq + kh * G) * D + idx);
        d[0] = __floats2bfloat162_rn(o.x / L, o.y / L);
        d[1] = __floats2bfloat162_rn(o.z / L, o.w / L);
    };
    // One thread, once every thread's part of a partial result is written: count it in.  1 for the last to come.
    auto count_in = [&](int r, int begin, int end) {
        int* counter = a.counters + (size_t)r * a.Hkv + kh;
        __threadfence();
        const bool last = atomicAdd(counter, 1) == end_share(end) - first_share(begin) - 1;
        if (last) *counter = 0;
        __threadfence();
        return last ? 1 : 0;
    };

    const WholeTileCopy<D, KT, NTHR> copy(ring, ring + KT * D, STAGE, a.k_pool, a.v_pool, bs_log2, a.Hkv, kh);
    ColState<D, NBQ> st;
    st.init();
    uint32_t qf[D / 16][4];
    Cursor cc = c0, ct = c0;                                // of the tile that is computed, and of the page read-ahead
    // The share's first row may be the rest of a row that the shares before it began: its partial result is counted
    // in one tile later (behind the barrier that the loop has anyway), and whether it came last is looked up at the end.
    int first_r = -1, first_begin = 0, first_end = 0;
    bool count_first = false;
    int stage = STAGES - 1;                                 // of tile x: (x - x0) % STAGES
    for (int x = x0; x < x1; ++x) {
        stage = stage == STAGES - 1 ? 0 : stage + 1;
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                    // tile x is there; everybody is done with tile x - 1
        if (count_first) {
            if (tid == NTHR - 1) s_first_last = count_in(first_r, first_begin, first_end);
            count_first = false;
        }
        const int xt = x + AHEAD, xl = x + STAGES - 1;
        if (xl < x1 && xl >= cl.end) cl.seek(xl, pre, spos, a.window);
        if (xt < x1) {
            if (xt >= ct.end) ct.seek(xt, pre, spos, a.window);
            if (tid < n_pages) fetch_page(ct, xt, tid);
        }
        if (x >= cc.end) cc.seek(x, pre, spos, a.window);
        const bool whole = cc.begin >= x0 && cc.end <= x1;  // the row lies in this share
        const bool ends = x + 1 == x1 || x + 1 == cc.end;
        int others = 0;
        if (ends && !whole && tid == 0) {                   // looked up now, needed when the tile is done
            const int* counter = a.counters + (size_t)cc.r * a.Hkv + kh;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(others) : "l"(counter) : "memory");
        }
        if (x == x0 || x == cc.begin) {
            const bf16* qs = qring + stage * QROWS * D;
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
                ldmatrix_x4(qf[kk], smem_u32(qs + tile_off<D>(NBQ == 1 ? lane & 7 : lane & 15, kk * 2 + (lane >> 4))));
        }
        // the copies of tile xl: in doses between the phases of tile x, or (a tile at a row's edge) at once
        const int stage_l = stage == 0 ? STAGES - 1 : stage - 1;
        const int* pg_l = pages + ((xl - x0) % PAGE_SLOTS) * KT;
        const int tl = cl.tile_start(xl);
        bool doses = false;
        if (xl < x1) {
            doses = tl >= cl.lo && tl + KT <= cl.pos + 1;
            if (!doses) {
                bf16* ks = ring + stage_l * STAGE;
                load_kv_tile<D, KT, NTHR>(ks, ks + KT * D, a.k_pool, a.v_pool, pg_l, tl >> bs_log2, bs_log2, a.Hkv, kh, tl,
                                          cl.lo, cl.pos + 1);
            }
            if (xl == cl.begin) load_query(cl, stage_l);
        }
        auto between = [&](int part) {
            if (doses) copy.dose(part, stage_l, pg_l - (tl >> bs_log2), tl);
        };
        const int ts = cc.tile_start(x);
        const bf16* ks = ring + stage * STAGE;
        warp_tile_decode<D, NBQ>(st, qf, ks, ks + KT * D, warp * 16, ts, cc.pos, cc.lo, cc.pos + 1, a.scale_log2,
                                 ts < cc.lo || ts + KT > cc.pos + 1, between);
        cp_async_commit();
        if (!ends) continue;

        // ---- the row, or this share of it, ends: merge the warps through the stage that was just read
        if (tid == 0) s_others = others;
        __syncthreads();
        float* wo = reinterpret_cast<float*>(ring + stage * STAGE);        // [NW][16][D]: exactly a stage
#pragma unroll
        for (int nb = 0; nb < NBQ; ++nb) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 2 * nb + e;
                float l = st.l[c];
                l += __shfl_xor_sync(0xffffffffu, l, 4);
                l += __shfl_xor_sync(0xffffffffu, l, 8);
                l += __shfl_xor_sync(0xffffffffu, l, 16);
                const int row = 8 * nb + 2 * (lane & 3) + e;
                if (lane < 4) { w_m[warp][row] = st.m[c]; w_l[warp][row] = l; }
#pragma unroll
                for (int mb = 0; mb < D / 16; ++mb) {
                    float* dst = wo + ((size_t)(warp * 16 + row)) * D + mb * 16 + (lane >> 2);
                    dst[0] = st.o[mb][nb][e];
                    dst[8] = st.o[mb][nb][e + 2];
                }
            }
        }
        __syncthreads();
        st.init();
        // the other shares' results are all there: join them to this one without writing it
        const bool finish = !whole && s_others == end_share(cc.end) - first_share(cc.begin) - 1;
        for (int idx = tid * 4; idx < G * D; idx += NTHR * 4) {
            const int row = idx / D;
            float M = -INFINITY, L = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < NW; ++w) M = w_l[w][row] > 0.f ? fmaxf(M, w_m[w][row]) : M;
#pragma unroll
            for (int w = 0; w < NW; ++w) {                  // a warp without a visible key has weight 0
                if (w_l[w][row] > 0.f) {
                    const float f = ex2_approx((w_m[w][row] - M) * a.scale_log2);
                    const float4 v = *reinterpret_cast<const float4*>(wo + (size_t)w * 16 * D + idx);
                    L += f * w_l[w][row];
                    o.x += f * v.x; o.y += f * v.y; o.z += f * v.z; o.w += f * v.w;
                }
            }
            M *= a.scale_log2;
            if (finish) join(cc.begin, cc.end, slot, row, idx, M, L, o);
            if (whole || finish) {
                write4(cc.r, idx, L, o);
            } else {
                const size_t p = piece_of(slot, cc.begin);
                *reinterpret_cast<float4*>(a.part_o + p * G * D + idx) = o;
                if (idx == row * D) *reinterpret_cast<float2*>(a.part_ml + (p * G + row) * 2) = make_float2(M, L);
            }
        }
        if (whole) continue;
        if (finish) {
            if (tid == 0) a.counters[(size_t)cc.r * a.Hkv + kh] = 0;
            continue;
        }
        if (x + 1 < x1) {                                   // the rest of an earlier share's row
            first_r = cc.r; first_begin = cc.begin; first_end = cc.end;
            count_first = true;
            continue;
        }
        __syncthreads();
        if (tid == 0) s_last = count_in(cc.r, cc.begin, cc.end);
        __syncthreads();
        if (!s_last) continue;
        for (int idx = tid * 4; idx < G * D; idx += NTHR * 4) {
            float M = -INFINITY, L = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            join(cc.begin, cc.end, -1, idx / D, idx, M, L, o);
            write4(cc.r, idx, L, o);
        }
    }
    cp_async_wait<0>();
    if (first_r >= 0) {
        __syncthreads();
        if (s_first_last)
            for (int idx = tid * 4; idx < G * D; idx += NTHR * 4) {
                float M = -INFINITY, L = 0.f;
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                join(first_begin, first_end, -1, idx / D, idx, M, L, o);
                write4(first_r, idx, L, o);
            }
    }
}

template <int D, int NBQ>
int launch_balanced(const BalancedArgs& a, cudaStream_t stream) {
    auto kernel = attn_decode_balanced_kernel<D, NBQ>;
    static sb::OncePerDevice once_per_device;
    bool& configured = once_per_device.flag();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             balanced_smem<D, NBQ>(MAX_REQUESTS));
        if (e != cudaSuccess) { sb_set_error("attention_balanced: %s", cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    sb::launch(kernel, dim3(a.W * a.Hkv), dim3(32 * NW), balanced_smem<D, NBQ>(a.R), stream, a);
    return 0;
}

}  // namespace

extern "C" int sb_attention_mma_supports(int Hq, int Hkv, int D, int page_size, int decode);

// 1 if the kernel takes this shape (bfloat16 only) with up to `requests` requests a step, else 0.
extern "C" int sb_attention_balanced_supports(int Hq, int Hkv, int D, int page_size, int requests) {
    return sb_attention_mma_supports(Hq, Hkv, D, page_size, 1) && requests > 0 && requests <= MAX_REQUESTS;
}

// Shares a KV head's tiles are cut into: as many blocks as the GPU holds at once.
extern "C" int sb_attention_balanced_shares(int Hq, int Hkv, int D, int requests, int num_sms) {
    if (Hkv <= 0 || Hq < Hkv || requests <= 0) return 1;
    const int nbq = Hq / Hkv <= 8 ? 1 : 2;
    const int smem = (STAGES * 2 * KT * D + STAGES * 8 * nbq * D) * 2 + PAGE_SLOTS * KT * 4 + (4 * requests + 4) * 4;
    const int fit = (227 * 1024) / (smem + 2048);
    const int per_sm = fit < 1 ? 1 : (fit > 4 ? 4 : fit);
    const int w = num_sms * per_sm / Hkv;
    return w < 1 ? 1 : w;
}

// Requests r = 0..R-1 bring tokens seq_starts[r] .. seq_starts[r+1]-1 at positions seq_first_pos[r]... of cache row
// seq_rows[r]; those with one token are served, the others' rows of `out` are left alone.  Scratch for `shares`
// shares: part_o Hkv*shares*2*G*D floats, part_ml Hkv*shares*2*G*2, and R*Hkv counters that are zero before the first
// call (the kernel leaves them zero).  What the kernel before this one on the stream may write: q, the newest key and
// value of each row; everything else it reads must be older than that kernel.
extern "C" int sb_attention_balanced(void* out, float* part_o, float* part_ml, int* counters, const void* q,
                                     const void* k_pool, const void* v_pool, const int* block_table, int table_width,
                                     const int* seq_starts, const int* seq_rows, const int* seq_first_pos, int R, int Hq,
                                     int Hkv, int D, int page_size, int window, float scale, int shares,
                                     cudaStream_t stream) {
    SB_REQUIRE(sb_attention_balanced_supports(Hq, Hkv, D, page_size, R),
               "attention_balanced: Hq=%d Hkv=%d head_dim=%d with %d requests is not supported", Hq, Hkv, D, R);
    SB_REQUIRE(window >= 0 && table_width > 0 && shares > 0 && (long long)shares * Hkv <= 0x7fffffffLL,
               "attention_balanced: bad sizes (table of %d, %d shares)", table_width, shares);
    SB_REQUIRE(part_o != nullptr && part_ml != nullptr && counters != nullptr, "attention_balanced: scratch is missing");
    const BalancedArgs a{(bf16*)out, part_o, part_ml, counters, (const bf16*)q, (const bf16*)k_pool, (const bf16*)v_pool,
                         block_table, seq_starts, seq_rows, seq_first_pos, table_width, R, Hq, Hkv, page_size, window,
                         shares, scale * LOG2E};
    const bool wide = Hq / Hkv > 8;
    int rc;
    switch (D) {
        case 16: rc = wide ? launch_balanced<16, 2>(a, stream) : launch_balanced<16, 1>(a, stream); break;
        case 32: rc = wide ? launch_balanced<32, 2>(a, stream) : launch_balanced<32, 1>(a, stream); break;
        case 64: rc = wide ? launch_balanced<64, 2>(a, stream) : launch_balanced<64, 1>(a, stream); break;
        default: rc = wide ? launch_balanced<128, 2>(a, stream) : launch_balanced<128, 1>(a, stream); break;
    }
    if (rc != 0) return rc;
    SB_LAUNCH_CHECK();
}
