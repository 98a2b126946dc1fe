// The end of a greedy decode step: the largest logit of each row.
#pragma once
#include "abi_check.cuh"
#include "blocks.cuh"

namespace sk {
namespace {

// Is (a, i) picked over (b, j): NaN before all, then the larger value, then the smaller index
__device__ __forceinline__ bool picked(float a, int i, float b, int j) {
    const bool na = a != a, nb = b != b;
    if (na != nb) return na;
    if (!na && a != b) return a > b;
    return i < j;
}

// One CTA per sequence.  32768 bf16 logits: 6.6 us at the end of a decoded token, where argmax, copy and two increments by
// the library take 17.
template <typename T, int V>
__global__ void __launch_bounds__(1024)
pick_token_kernel(const T* logits, int64_t ld, int vocab, int64_t* token, int64_t* pos, int32_t* seqlens) {
    pdl_begin();
    __shared__ float best_s[32];
    __shared__ int at_s[32];
    const int b = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const T* row = logits + b * ld;
    float best = -INFINITY;
    int at = vocab;                                           // behind every index: a row of -inf alone picks its first
    constexpr int U = 4;
    for (int i0 = t * V; i0 < vocab; i0 += U * 1024 * V) {
        float v[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * 1024 * V < vocab) load_vec<T, V>(row + i0 + u * 1024 * V, v[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int i = i0 + u * 1024 * V + e;
                if (i < vocab && picked(v[u][e], i, best, at)) {
                    best = v[u][e];
                    at = i;
                }
            }
    }
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const float x = __shfl_xor_sync(FULL, best, o);
            const int i = __shfl_xor_sync(FULL, at, o);
            if (picked(x, i, best, at)) {
                best = x;
                at = i;
            }
        }
    };
    reduce();
    if (lane == 0) {
        best_s[warp] = best;
        at_s[warp] = at;
    }
    __syncthreads();
    if (warp == 0) {
        best = best_s[lane];
        at = at_s[lane];
        reduce();
        if (lane == 0) {
            token[b] = at;
            if (seqlens != nullptr) seqlens[b] += 1;
            if (b == 0 && pos != nullptr) pos[0] += 1;
        }
    }
}

template <typename T>
int pick_dispatch(const void* logits, int64_t ld, int batch, int vocab, int64_t* token, int64_t* pos, int32_t* seqlens,
                  cudaStream_t st) {
    constexpr int V = 16 / sizeof(T);
    const bool vec = vocab % V == 0 && ld % V == 0 && (uintptr_t)logits % 16 == 0;
    auto kern = vec ? pick_token_kernel<T, V> : pick_token_kernel<T, 1>;
    return check_chained(launch_after(kern, dim3((unsigned)batch), dim3(1024), 0, st, (const T*)logits, ld, vocab, token, pos, seqlens),
                         "pick_token_kernel");
}

}  // namespace

int pick_token(const void* logits, int dtype, int64_t ld, int batch, int vocab, int64_t* token, int64_t* pos, int32_t* seqlens,
               cudaStream_t st) {
    SK_REQUIRE(logits && token && valid_dtype(dtype) && batch > 0 && vocab > 0 && ld >= vocab, "pick_token: null pointer, bad sizes or dtype");
    if (dtype == SK_F32) return pick_dispatch<float>(logits, ld, batch, vocab, token, pos, seqlens, st);
    return dtype == SK_BF16 ? pick_dispatch<__nv_bfloat16>(logits, ld, batch, vocab, token, pos, seqlens, st)
                            : pick_dispatch<__half>(logits, ld, batch, vocab, token, pos, seqlens, st);
}

}  // namespace sk
