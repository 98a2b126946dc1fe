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

// A cluster of eight CTAs per sequence, each an eighth of the row; the first one joins what they found.  32768 logits: one CTA
// took 6.6 us at the end of a decoded token.  A short row is one larger CTA's: 1000 logits 2.7 us, by a cluster 3.2.
constexpr int PT_CLUSTER = 8, PT_ALONE = 4096;
template <int CL> constexpr int PT_THREADS = CL == 1 ? 1024 : 256;
template <typename T, int V, int CL>
__global__ void __launch_bounds__(PT_THREADS<CL>)
pick_token_kernel(const T* logits, int64_t ld, int vocab, int64_t* token, int64_t* pos, int32_t* seqlens) {
    pdl_begin();
    constexpr int WARPS = PT_THREADS<CL> / 32;
    __shared__ float best_s[CL * WARPS];
    __shared__ int at_s[CL * WARPS];
    if (CL > 1) cluster_arrive();
    const int rank = blockIdx.x, b = blockIdx.y, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const T* row = logits + b * ld;
    float best = -INFINITY;
    int at = vocab;                                           // behind every index: a row of -inf alone picks its first
    constexpr int U = CL == 1 ? 1 : 4, STEP = CL * PT_THREADS<CL> * V;      // elements of the cluster's one load each
    for (int64_t i0 = (rank * PT_THREADS<CL> + t) * V; i0 < vocab; i0 += U * STEP) {
        float v[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * STEP < vocab) load_vec<T, V>(row + i0 + u * STEP, v[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int64_t i = i0 + u * STEP + e;
                if (i < vocab && picked(v[u][e], (int)i, best, at)) {
                    best = v[u][e];
                    at = (int)i;
                }
            }
    }
    auto join = [&](float x, int i) {
        if (picked(x, i, best, at)) {
            best = x;
            at = i;
        }
    };
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const float x = __shfl_xor_sync(FULL, best, o);
            const int i = __shfl_xor_sync(FULL, at, o);
            join(x, i);
        }
    };
    reduce();
    if (CL > 1) {
        cluster_wait();                                       // every CTA of the cluster has begun
        if (lane == 0) {
            store_first_cta(best_s + rank * WARPS + warp, best);
            store_first_cta(at_s + rank * WARPS + warp, (uint32_t)at);
        }
        cluster_arrive();
        cluster_wait();
    } else {
        if (lane == 0) {
            best_s[warp] = best;
            at_s[warp] = at;
        }
        __syncthreads();
    }
    if (rank == 0 && warp == 0) {
        static_assert(CL * WARPS % 32 == 0, "as many results for every lane");
        best = best_s[lane];
        at = at_s[lane];
        if (CL * WARPS > 32) join(best_s[(lane + 32) % (CL * WARPS)], at_s[(lane + 32) % (CL * WARPS)]);
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
    const int cl = vocab <= PT_ALONE ? 1 : PT_CLUSTER;
    auto kern = cl == 1 ? (vec ? pick_token_kernel<T, V, 1> : pick_token_kernel<T, 1, 1>)
                        : (vec ? pick_token_kernel<T, V, PT_CLUSTER> : pick_token_kernel<T, 1, PT_CLUSTER>);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(cl == 1 ? PT_THREADS<1> : PT_THREADS<PT_CLUSTER>);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cl;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cl > 1 ? 2 : 1;
    for (int b0 = 0; b0 < batch; b0 += 65535) {               // the grid's second dimension
        cfg.gridDim = dim3((unsigned)cl, (unsigned)(batch - b0 < 65535 ? batch - b0 : 65535));
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (const T*)logits + b0 * ld, ld, vocab, token + b0, b0 == 0 ? pos : (int64_t*)nullptr,
                                                 seqlens != nullptr ? seqlens + b0 : (int32_t*)nullptr);
        if (int rc = check_chained(e, "pick_token_kernel")) return rc;
    }
    return SK_OK;
}

// What a decode step begins with, in one launch: the current tokens, the position, and the lengths.
constexpr int BT_LENGTHS = 64;
struct BtLengths {
    int32_t* at[BT_LENGTHS];
};
__global__ void __launch_bounds__(128)
begin_token_kernel(const int64_t* first, int64_t* token, int batch, int64_t* pos, int32_t* seqlens, int64_t position,
                   const __grid_constant__ BtLengths lengths, int n) {
    for (int b = threadIdx.x; b < batch; b += 128) {
        token[b] = first[b];
        seqlens[b] = (int32_t)position;
    }
    if (threadIdx.x == 0) pos[0] = position;
    for (int i = threadIdx.x; i < n; i += 128) *lengths.at[i] = (int32_t)position;
}

}  // namespace

int pick_token(const void* logits, int dtype, int64_t ld, int batch, int vocab, int64_t* token, int64_t* pos, int32_t* seqlens,
               cudaStream_t st) {
    SK_REQUIRE(logits && token && valid_dtype(dtype) && batch > 0 && vocab > 0 && ld >= vocab, "pick_token: null pointer, bad sizes or dtype");
    if (dtype == SK_F32) return pick_dispatch<float>(logits, ld, batch, vocab, token, pos, seqlens, st);
    return dtype == SK_BF16 ? pick_dispatch<__nv_bfloat16>(logits, ld, batch, vocab, token, pos, seqlens, st)
                            : pick_dispatch<__half>(logits, ld, batch, vocab, token, pos, seqlens, st);
}

int begin_token(const int64_t* first, int64_t* token, int batch, int64_t* pos, int32_t* seqlens, int64_t position, int32_t* const* lengths,
                int n, cudaStream_t st) {
    SK_REQUIRE(first && token && pos && seqlens && batch > 0 && position >= INT32_MIN && position <= INT32_MAX && n >= 0 && (n == 0 || lengths),
               "begin_token: null pointer or bad sizes");
    int i = 0;
    do {                                                      // more lengths than a launch takes: the rest by themselves
        BtLengths part{};
        int m = 0;
        for (; m < BT_LENGTHS && i < n; ++m, ++i) {
            SK_REQUIRE(lengths[i] != nullptr, "begin_token: null length");
            part.at[m] = lengths[i];
        }
        begin_token_kernel<<<1, 128, 0, st>>>(first, token, batch, pos, seqlens, position, part, m);
        if (int rc = check_launch("begin_token_kernel")) return rc;
    } while (i < n);
    return SK_OK;
}

}  // namespace sk
