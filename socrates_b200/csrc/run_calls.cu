// Runs a recorded list of entry points: the launches of a whole layer from ONE call of the host language.
//
// A step that is not replayed from a graph (prompt portions, mixed steps) launches eight or nine kernels a layer, and what
// the host needs for one through Python and ctypes (argument checks, conversions, look-ups of buffers) is three times what the
// driver's launch takes.  Layers of one shape launch the same kernels with the same arguments but for the addresses of their
// weights and pages, so the host records one layer's calls and hands the other layers' over as words.
//
// A call is [entry point, word 0, word 1, ...]: pointers and whole numbers as they are, floats as their bits.
#include <stdint.h>
#include <string.h>

#include <utility>

#include "common.cuh"

extern "C" {
int sb_add_rmsnorm(float*, const float*, int, long long, const float*, void*, const int*, int, int, float, int, cudaStream_t);
int sb_gemm_tcgen05(void*, const void*, const void*, int, int, int, int, int*, int*, int, int, const void*, long long, cudaStream_t);
int sb_gemm_simt(void*, const void*, const void*, int, int, int, int, int, int, int, int, cudaStream_t);
int sb_qk_norm_rope_kvwrite(const void*, const float*, int, long long, void*, void*, void*, const float*, const float*,
                            const float*, int, const int*, const int*, const int*, int, int, float, int, int, int, int, int, int,
                            int, int, int, const float*, int, float, int, int, int, float, float*, cudaStream_t);
int sb_silu_mul(void*, const void*, int, int, int, int, int, cudaStream_t);
int sb_attention_simt(void*, float*, float*, const void*, const void*, const void*, const int*, int, const int*, const int*, int,
                      int, int, int, int, int, float, int, int, cudaStream_t);
int sb_attention_prefill_tcgen05(void*, const void*, const void*, const void*, int, const int*, int, const int*, const int*,
                                 const int*, int, int, int, int, int, int, int, float, int*, const void*, long long, int, int,
                                 float, int, float*, float, const float*, int, int, const float*, int, int, cudaStream_t);
int sb_attention_prefill_mma(void*, const void*, const void*, const void*, const int*, int, const int*, const int*, const int*,
                             int, int, int, int, int, int, int, float, cudaStream_t);
int sb_attention_balanced(void*, float*, float*, int*, const void*, const void*, const void*, const int*, int, const int*,
                          const int*, const int*, int, int, int, int, int, int, float, int, cudaStream_t);
int sb_attention_decode_mma(void*, float*, float*, const void*, const void*, const void*, const int*, int, const int*,
                            const int*, int, int, int, int, int, int, float, int, int, float, const float*, int, cudaStream_t);
int sb_attention_decode_stream(void*, float*, float*, int*, const void*, const void*, const void*, const int*, int, const int*,
                               const int*, int, int, int, int, int, int, float, int, int, int, cudaStream_t);
}

namespace {

template <typename T> T from_word(int64_t w) {
    T v;
    static_assert(sizeof(T) <= 8, "an argument is a word");
    memcpy(&v, &w, sizeof(T));          // little-endian: a float or an int is the low half
    return v;
}
template <typename... Args, size_t... I>
int call(int (*fn)(Args...), const int64_t* w, std::index_sequence<I...>) { return fn(from_word<Args>(w[I])...); }
template <typename... Args> int call(int (*fn)(Args...), const int64_t* w) {
    return call(fn, w, std::index_sequence_for<Args...>{});
}
template <typename... Args> constexpr int arity(int (*)(Args...)) { return (int)sizeof...(Args); }

}  // namespace

#define SB_ENTRIES(X)                                                                                              \
    X(0, sb_add_rmsnorm) X(1, sb_gemm_tcgen05) X(2, sb_gemm_simt) X(3, sb_qk_norm_rope_kvwrite) X(4, sb_silu_mul)   \
    X(5, sb_attention_simt) X(6, sb_attention_prefill_tcgen05) X(7, sb_attention_prefill_mma)                       \
    X(8, sb_attention_balanced) X(9, sb_attention_decode_mma) X(10, sb_attention_decode_stream)

// Words that entry point `id` takes, or -1 (host only).
extern "C" int sb_run_calls_arity(int id) {
    switch (id) {
#define X(ID, FN) case ID: return arity(&FN);
        SB_ENTRIES(X)
#undef X
        default: return -1;
    }
}

// Runs the calls in `words` one after the other; the first one that fails ends it with its code (and its text in
// sb_last_error()).  *done: how many calls succeeded.
extern "C" int sb_run_calls(const int64_t* words, int n_words, int* done) {
    SB_REQUIRE(words != nullptr && done != nullptr && n_words >= 0, "run_calls: bad list");
    *done = 0;
    for (int at = 0; at < n_words;) {
        const int id = (int)words[at], n = sb_run_calls_arity(id);
        SB_REQUIRE(n >= 0 && at + 1 + n <= n_words, "run_calls: word %d names no entry point or the list is cut", at);
        int rc = 0;
        switch (id) {
#define X(ID, FN) case ID: rc = call(&FN, words + at + 1); break;
            SB_ENTRIES(X)
#undef X
        }
        if (rc != 0) return rc;
        ++*done;
        at += 1 + n;
    }
    return 0;
}
