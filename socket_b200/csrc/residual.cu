// Everything between two matrix products that touches the fp32 residual stream: the scaled embedding,
// the residual update with a norm on the sublayer's output fused with the norm of the next sublayer's
// input, and the gated units of the feed-forwards.
#include <type_traits>

#include "blocks.cuh"

namespace sk {
namespace {

template <typename T, int V>
__global__ void __launch_bounds__(256)
embed_rows_kernel(const int64_t* __restrict__ tokens, const T* __restrict__ table, int64_t vocab, int width, float scale,
                  float* __restrict__ x, float* __restrict__ x_copy, int32_t* status) {
    // launched unchained, the first kernel of a stack: those behind it may rely on all earlier work being complete
    pdl_launch_dependents();
    const int64_t row = blockIdx.x;
    const int i = (blockIdx.y * 256 + threadIdx.x) * V;
    const int64_t tok = tokens[row];
    const bool ok = tok >= 0 && tok < vocab;              // outside the table: flagged, the row reads zero
    if (!ok && i == 0 && status != nullptr) atomicOr(status, SK_DEV_INDEX_OUT_OF_RANGE);
    if (i >= width) return;
    float v[V];
    if (ok) load_vec<T, V>(table + tok * width + i, v);
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = ok ? v[e] * scale : 0.f;
    store_vec<float, V>(x + row * width + i, v);
    if (x_copy != nullptr) store_vec<float, V>(x_copy + row * width + i, v);
}

// One CTA per row; the row lives in registers (NV vectors of V elements per thread).
//   in_mode  0: x stays; 1: x += rms(y) * w_in; 2: x = y + w_in; 3: x += y
//   out_mode 0: nothing; 1: out = rms(x) * w_out; 2: out = [x ; x0]; 3: out = layer norm of x * w_out
// EARLY: a decoded token's rows are bound by latency: everything is requested at once, as with each norm's weights requested behind its sum
// a row of 4096 waited for memory three times.  Other rows are bound by memory, and the registers that would hold the weights keep
// rows in flight instead (290 rows of 4096, 1024 threads each: 5.3 us early, 4.0 late, two rows an SM); vectors of 8 leave every other 16
// bytes of the fp32 stream to a second access (8000 rows of 4096: 125 us, so 95).
// IN: false where in_mode is 0, which then takes fewer registers (32000 rows of 4096 with a norm out: 129 us, so 113)
template <typename T, typename TY, int V, int NV, bool EARLY, bool IN>
__global__ void __launch_bounds__(1024, !EARLY && NV <= 4 && V * NV <= 8 ? 2 : 1)
residual_norm_kernel(sk_residual_params p) {
    __shared__ float red[3][32];
    const int64_t row = blockIdx.x;
    const int W = p.width, nt = blockDim.x, t = threadIdx.x;
    pdl_begin();                                          // the projection that reads `out` may request its weights
    float* xr = p.x + row * W;
    const T* w_in = (const T*)p.w_in;
    const T* w_out = (const T*)p.w_out;
    const TY* yr = (const TY*)p.y + row * p.y_ld;
    const bool norm_out = p.out_mode == 1 || p.out_mode == 3;
    Raw<TY, V> yw[NV];
    Raw<float, V> xw[NV], x0w[NV];
    Raw<T, V> wi[NV], wo[NV];
    auto request = [&](bool wanted, auto* from, auto& raw) {
        if (!wanted) return;
#pragma unroll
        for (int n = 0; n < NV; ++n)
            if ((n * nt + t) * V < W) raw[n] = load_raw<std::remove_const_t<std::remove_pointer_t<decltype(from)>>, V>(from + (n * nt + t) * V);
    };
    request(IN && p.in_mode != 0, yr, yw);                    // (known to be true, the registers of four vectors spill)
    request(p.in_mode != 2, xr, xw);
    if (EARLY) {
        request(IN && (p.in_mode == 1 || p.in_mode == 2), w_in, wi);
        request(norm_out, w_out, wo);
        request(p.out_mode == 2, p.x0 + row * W, x0w);
    }
    float xv[NV][V];
    if (IN && p.in_mode != 0) {
        float inv = 1.f;
        if (p.in_mode == 1) {
            float ss = 0.f;
#pragma unroll
            for (int n = 0; n < NV; ++n)
                if ((n * nt + t) * V < W)
#pragma unroll
                    for (int e = 0; e < V; ++e) ss = fmaf(to_f32(yw[n].e[e]), to_f32(yw[n].e[e]), ss);
            inv = 1.f / sqrtf(block_sum(ss, red[0]) / (float)W + p.eps);
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int i = (n * nt + t) * V;
            if (i < W) {
                if (!EARLY && p.in_mode != 3) wi[n] = load_raw<T, V>(w_in + i);
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const float y = to_f32(yw[n].e[e]);
                    xv[n][e] = p.in_mode == 1 ? xw[n].e[e] + y * inv * to_f32(wi[n].e[e])
                                              : (p.in_mode == 2 ? y + to_f32(wi[n].e[e]) : xw[n].e[e] + y);
                }
                store_vec<float, V>(xr + i, xv[n]);
            }
        }
    } else {
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
            for (int e = 0; e < V; ++e) xv[n][e] = xw[n].e[e];
    }
    if (norm_out) {
        float mean = 0.f;
        if (p.out_mode == 3) {                            // centred in registers; the stream itself is written already
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < NV; ++n)
                if ((n * nt + t) * V < W)
#pragma unroll
                    for (int e = 0; e < V; ++e) sum += xv[n][e];
            mean = block_sum(sum, red[2]) / (float)W;
        }
        float ss = 0.f;
#pragma unroll
        for (int n = 0; n < NV; ++n)
            if ((n * nt + t) * V < W)
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    xv[n][e] -= mean;
                    ss = fmaf(xv[n][e], xv[n][e], ss);
                }
        const float inv = 1.f / sqrtf(block_sum(ss, red[1]) / (float)W + p.eps);
        T* o = (T*)p.out + row * W;
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int i = (n * nt + t) * V;
            if (i < W) {
                float r[V];
                if (!EARLY) wo[n] = load_raw<T, V>(w_out + i);
#pragma unroll
                for (int e = 0; e < V; ++e) r[e] = xv[n][e] * inv * to_f32(wo[n].e[e]);
                store_vec<T, V>(o + i, r);
            }
        }
    } else if (p.out_mode == 2) {
        T* o = (T*)p.out + row * 2 * W;
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int i = (n * nt + t) * V;
            if (i < W) {
                if (!EARLY) x0w[n] = load_raw<float, V>(p.x0 + row * W + i);
                float r[V];
#pragma unroll
                for (int e = 0; e < V; ++e) r[e] = x0w[n].e[e];
                store_vec<T, V>(o + i, xv[n]);
                store_vec<T, V>(o + W + i, r);
            }
        }
    }
}

// KIND SKB_GLU_CLAMPED: y = g * sigmoid(slope * g) * (u + 1), g and u clamped; SKB_GLU_SILU: y = g * sigmoid(g) * u
template <typename T, int V, int KIND>
__global__ void __launch_bounds__(256)
glu_kernel(const T* gate, const T* up, int64_t rows, int ff, int64_t ld, float limit, float slope, T* __restrict__ out,
           int64_t out_ld) {
    pdl_begin();
    const int i = (blockIdx.x * 256 + threadIdx.x) * V;
    if (i >= ff) return;
    for (int64_t row = blockIdx.y; row < rows; row += gridDim.y) {
        float g[V], u[V], r[V];
        load_vec<T, V>(gate + row * ld + i, g);
        load_vec<T, V>(up + row * ld + i, u);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            if (KIND == SKB_GLU_CLAMPED) {
                const float a = fminf(g[e], limit), b = fminf(fmaxf(u[e], -limit), limit);
                r[e] = a * sigmoid_scaled<T>(a, slope) * (b + 1.f);
            } else {
                r[e] = silu<T>(g[e]) * u[e];
            }
        }
        store_vec<T, V>(out + row * out_ld + i, r);
    }
}

// The newest tokens of a portion, from token s0 on, into a ring of `ring` rows (row of position p: p % ring).
// s0 leaves out what no later token sees, so that no two tokens of a portion meet in one row.
// E: the unit of a copy, as large as rows and strides allow: 4096 tokens of 1024 + 1024 elements of 2 bytes in 14 us, one element at
// a time 34
template <typename E>
__global__ void __launch_bounds__(256)
ring_append_kernel(const E* k, const E* v, int64_t k_bs, int64_t k_ss, int64_t v_bs,
                   int64_t v_ss, int k_row, int v_row, int ring, const int64_t* pos, int64_t start, int s0,
                   E* __restrict__ k_cache, E* __restrict__ v_cache) {
    pdl_begin();
    const int s = s0 + blockIdx.x, b = blockIdx.y;
    const E* ks = k + b * k_bs + s * k_ss;
    const E* vs = v + b * v_bs + s * v_ss;                    // v_row is zero without values
    const int i = threadIdx.x, j = i - k_row;                 // the first piece is requested with the position
    E first;
    if (i < k_row) first = ks[i];
    else if (j < v_row) first = vs[j];
    const int64_t slot = position_mod(first_position(pos, start) + s, ring);
    E* kd = k_cache + ((int64_t)b * ring + slot) * k_row;
    E* vd = v_cache + ((int64_t)b * ring + slot) * v_row;
    if (i < k_row) kd[i] = first;
    else if (j < v_row) vd[j] = first;
    for (int n = i + blockDim.x; n < k_row + v_row; n += blockDim.x) {
        if (n < k_row) kd[n] = ks[n];
        else vd[n - k_row] = vs[n - k_row];
    }
}

template <typename T, typename TY, int V>
int residual_dispatch(const sk_residual_params& p, cudaStream_t st) {
    const int vecs = (p.width + V - 1) / V;
    // few rows: one vector per thread (latency); many rows: smaller blocks, more of them per SM, with two to four vectors per thread: of one,
    // 8000 rows of 1024 took 20.0 us (of two 16.6), of eight, whose registers spill, 8000 rows of 5120 119 us (of four 86)
    int nt = p.rows < 296 ? 1024 : 256;
    while (nt > 32 && nt / 2 >= vecs) nt /= 2;
    if (p.rows >= 2048 && nt >= vecs && nt > 64) nt /= 2;         // (400 rows of 512: 2.7 us of one vector a thread, 3.1 of two)
    if (vecs > 4 * nt) nt = vecs > 4 * 1024 ? 1024 : (vecs + 127) / 128 * 32;
    while (nt < 1024 && (vecs + nt - 1) / nt > 8) nt *= 2;
    const int nv = (vecs + nt - 1) / nt;
    // Weights early (us, cold, of 2048 or 4096 elements): 8 rows of both norms 3.5, late 3.7, 100 rows 4.0 and 3.8; without a second norm 2.6 and 2.3; of
    // two vectors a thread (5120) 4.2 and 4.9; small rows (54) 2.2 and 2.9
    const bool few = p.rows <= sm_count(), own = p.out_mode == 2 && p.x0 == p.x;      // the stream itself as x0 is read behind its update
    const bool early = !own && (nt <= 128 || (few && (nv > 1 || p.in_mode == 0 || p.out_mode == 2 || (p.out_mode != 0 && p.rows <= 32))));
    void (*kern)(sk_residual_params) = nullptr;
    auto pick = [&](auto in) {
        constexpr bool IN = decltype(in)::value;
        if (nv <= 1) kern = early ? residual_norm_kernel<T, TY, V, 1, true, IN> : residual_norm_kernel<T, TY, V, 1, false, IN>;
        else if (nv <= 2) kern = early ? residual_norm_kernel<T, TY, V, 2, true, IN> : residual_norm_kernel<T, TY, V, 2, false, IN>;
        else if (nv <= 4) kern = early && V == 1 ? residual_norm_kernel<T, TY, V, 4, V == 1, IN> : residual_norm_kernel<T, TY, V, 4, false, IN>;
        else if (nv <= 8) kern = residual_norm_kernel<T, TY, V, 8, false, IN>;
    };
    if (p.in_mode != 0) pick(std::true_type{});
    else pick(std::false_type{});
    if (kern == nullptr) return fail(SK_ERR_UNSUPPORTED, "sk_residual_norm: width %d is too large", p.width);
    return check_chained(launch_after(kern, dim3((unsigned)p.rows), dim3((unsigned)nt), 0, st, p), "residual_norm_kernel");
}

}  // namespace

int launch_embed_rows(const int64_t* tokens, const void* table, int dtype, int64_t rows, int64_t vocab, int width,
                      float scale, float* x, float* x_copy, int32_t* status, cudaStream_t st) {
    const int V = width % 4 == 0 ? 4 : 1;
    dim3 grid((unsigned)rows, (unsigned)((width + 256 * V - 1) / (256 * V)));
#define SK_EMBED(T, V) embed_rows_kernel<T, V><<<grid, 256, 0, st>>>(tokens, (const T*)table, vocab, width, scale, x, x_copy, status)
    if (dtype == SK_BF16) { if (V == 4) SK_EMBED(__nv_bfloat16, 4); else SK_EMBED(__nv_bfloat16, 1); }
    else { if (V == 4) SK_EMBED(float, 4); else SK_EMBED(float, 1); }
#undef SK_EMBED
    return check_launch("embed_rows_kernel");
}

int launch_residual_norm(const sk_residual_params& p, cudaStream_t st) {
    const bool v4 = p.width % 4 == 0 && p.y_ld % 4 == 0;
    if (p.dtype == SK_F32) return v4 ? residual_dispatch<float, float, 4>(p, st) : residual_dispatch<float, float, 1>(p, st);
    using bf = __nv_bfloat16;
    if (p.y_dtype == SK_F32) return v4 ? residual_dispatch<bf, float, 4>(p, st) : residual_dispatch<bf, float, 1>(p, st);
    return v4 ? residual_dispatch<bf, bf, 4>(p, st) : residual_dispatch<bf, bf, 1>(p, st);
}

int launch_glu(const void* gate, const void* up, int dtype, int64_t rows, int ff, int64_t ld, int kind, float limit, float slope,
               void* out, int64_t out_ld, cudaStream_t st) {
    const size_t es = dtype == SK_BF16 ? 2 : 4;
    auto vec = [&](int v) {
        return ff % v == 0 && ld % v == 0 && out_ld % v == 0 &&
               ((uintptr_t)gate | (uintptr_t)up | (uintptr_t)out) % (v * es) == 0;
    };
    const bool v4 = vec(4), v8 = dtype == SK_BF16 && vec(8);
    const int V = v8 ? 8 : (v4 ? 4 : 1);
    dim3 grid((unsigned)((ff + 256 * V - 1) / (256 * V)), (unsigned)(rows < 32768 ? rows : 32768));
#define SK_GLU(T, V)                                                                                                       \
    do {                                                                                                                   \
        auto kern = kind == SKB_GLU_CLAMPED ? glu_kernel<T, V, SKB_GLU_CLAMPED> : glu_kernel<T, V, SKB_GLU_SILU>;          \
        return check_chained(launch_after(kern, grid, dim3(256), 0, st, (const T*)gate, (const T*)up, rows, ff, ld, limit, slope, \
                                          (T*)out, out_ld), "glu_kernel");                                                 \
    } while (0)
    if (dtype == SK_BF16) { if (v8) SK_GLU(__nv_bfloat16, 8); else if (v4) SK_GLU(__nv_bfloat16, 4); else SK_GLU(__nv_bfloat16, 1); }
    else { if (v4) SK_GLU(float, 4); else SK_GLU(float, 1); }
#undef SK_GLU
}

int launch_ring_append(const void* k, const void* v, int dtype, int B, int S, int64_t k_bs, int64_t k_ss, int64_t v_bs,
                       int64_t v_ss, int k_row, int v_row, int ring, int keep, const int64_t* pos, int64_t start, void* k_cache,
                       void* v_cache, cudaStream_t st) {
    // first position to write: of the last block of `ring` positions, or of the last `ring` positions
    const int64_t first = keep == SKB_RING_CHUNK ? (start + S - 1) / ring * ring : start + S - ring;
    const int s0 = pos == nullptr && first > start ? (int)(first - start) : 0;   // a device position: one token
    const int es = dtype == SK_BF16 ? 2 : 4, e16 = 16 / es;
    const bool vec = k_row % e16 == 0 && k_bs % e16 == 0 && k_ss % e16 == 0 && ((uintptr_t)k | (uintptr_t)k_cache) % 16 == 0 &&
                     (v == nullptr || (v_row % e16 == 0 && v_bs % e16 == 0 && v_ss % e16 == 0 && ((uintptr_t)v | (uintptr_t)v_cache) % 16 == 0));
    if (v == nullptr) v_row = 0;
    auto run = [&](auto unit, int per) {                       // `per` elements in a unit
        using E = decltype(unit);
        const int pieces = k_row / per + v_row / per;
        const unsigned nt = pieces >= 256 ? 256u : (unsigned)((pieces + 31) / 32 * 32);
        return check_chained(launch_after(ring_append_kernel<E>, dim3((unsigned)(S - s0), (unsigned)B), dim3(nt), 0, st, (const E*)k,
                                          (const E*)v, k_bs / per, k_ss / per, v_bs / per, v_ss / per, k_row / per, v_row / per, ring, pos,
                                          start, s0, (E*)k_cache, (E*)v_cache), "ring_append_kernel");
    };
    if (vec) return run(uint4{}, e16);
    return dtype == SK_BF16 ? run(uint16_t{}, 1) : run(uint32_t{}, 1);
}

}  // namespace sk
