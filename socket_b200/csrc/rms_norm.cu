// RMS norm of rows in the model's type: the norms of a decode step.
#include "abi_check.cuh"
#include "blocks.cuh"

namespace sk {
namespace {

// One CTA per row, the row in registers.  Latency-bound: one pass over 8 KB (4096 x bf16), 2.9 us inside a decoded token
// where the library's norm takes 6.3.  EARLY: the weights are requested with the row, one trip to memory; of more rows than SMs they would keep
// other rows off (3000 rows of 8192: 47 us early, 28 late).
template <typename T, int V, int NV, bool EARLY>
__global__ void __launch_bounds__(512)
rms_norm_rows_kernel(const T* x, const T* w, int width, float eps, T* __restrict__ out) {
    pdl_begin();
    __shared__ float red[32];
    const int64_t row = blockIdx.x;
    const int nt = blockDim.x, t = threadIdx.x;
    float v[NV][V], ss = 0.f;
    Raw<T, V> g[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int i = (n * nt + t) * V;
        if (i < width) {
            load_vec<T, V>(x + row * width + i, v[n]);
            if (EARLY) g[n] = load_raw<T, V>(w + i);
        }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n)
        if ((n * nt + t) * V < width)
#pragma unroll
            for (int e = 0; e < V; ++e) ss = fmaf(v[n][e], v[n][e], ss);
    const float inv = 1.f / sqrtf(block_sum(ss, red) / (float)width + eps);
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int i = (n * nt + t) * V;
        if (i < width) {
            if (!EARLY) g[n] = load_raw<T, V>(w + i);
#pragma unroll
            for (int e = 0; e < V; ++e) v[n][e] *= inv * to_f32(g[n].e[e]);
            store_vec<T, V>(out + row * width + i, v[n]);
        }
    }
}

// Rows too long for registers: read twice, the second time mostly from L2.
template <typename T, int V>
__global__ void __launch_bounds__(512)
rms_norm_long_rows_kernel(const T* x, const T* w, int width, float eps, T* __restrict__ out) {
    pdl_begin();
    __shared__ float red[32];
    const int64_t row = blockIdx.x, step = (int64_t)blockDim.x * V;
    float ss = 0.f;
    for (int64_t i = threadIdx.x * V; i < width; i += step) {
        float v[V];
        load_vec<T, V>(x + row * width + i, v);
#pragma unroll
        for (int e = 0; e < V; ++e) ss = fmaf(v[e], v[e], ss);
    }
    const float inv = 1.f / sqrtf(block_sum(ss, red) / (float)width + eps);
    for (int64_t i = threadIdx.x * V; i < width; i += step) {
        float v[V], g[V];
        load_vec<T, V>(x + row * width + i, v);
        load_vec<T, V>(w + i, g);
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] *= inv * g[e];
        store_vec<T, V>(out + row * width + i, v);
    }
}

template <typename T>
int rms_dispatch(const void* x, const void* w, int64_t rows, int width, float eps, void* out, cudaStream_t st) {
    constexpr int V = 16 / sizeof(T);
    const bool vec = width % V == 0 && ((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) % 16 == 0;
    const int vecs = vec ? width / V : width;
    int nt = 512;
    while (nt > 32 && nt / 2 >= vecs) nt /= 2;
    const int nv = (vecs + nt - 1) / nt;
    auto run = [&](auto kern) {
        return check_chained(launch_after(kern, dim3((unsigned)rows), dim3((unsigned)nt), 0, st, (const T*)x, (const T*)w, width, eps,
                                          (T*)out), "rms_norm_rows_kernel");
    };
    const bool few = rows <= sm_count();
    if (vec && nv <= 1) return run(rms_norm_rows_kernel<T, V, 1, true>);
    if (vec && nv <= 4) return few ? run(rms_norm_rows_kernel<T, V, 4, true>) : run(rms_norm_rows_kernel<T, V, 4, false>);
    if (!vec && nv <= 4) return few ? run(rms_norm_rows_kernel<T, 1, 4, true>) : run(rms_norm_rows_kernel<T, 1, 4, false>);
    return vec ? run(rms_norm_long_rows_kernel<T, V>) : run(rms_norm_long_rows_kernel<T, 1>);
}

}  // namespace

int rms_norm_rows(const void* x, const void* w, int dtype, int64_t rows, int width, float eps, void* out, cudaStream_t st) {
    SK_REQUIRE(x && w && out && valid_dtype(dtype) && rows > 0 && width > 0, "sk_rms_norm: null pointer, bad sizes or dtype");
    if (dtype == SK_F32) return rms_dispatch<float>(x, w, rows, width, eps, out, st);
    return dtype == SK_BF16 ? rms_dispatch<__nv_bfloat16>(x, w, rows, width, eps, out, st) : rms_dispatch<__half>(x, w, rows, width, eps, out, st);
}

}  // namespace sk
