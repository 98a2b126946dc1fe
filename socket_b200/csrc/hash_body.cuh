// Device code shared by the hashing kernels: exact sign-random-projection codes of up
// to four rows at a time, and the write of one new token into the KV cache.
//
// fp64 arithmetic runs at about five lanes a cycle here (a warp instruction keeps an SM's unit for 6.6 cycles), so 32 fp64 dot
// products a warp took most of an append: 4.4 of the 5.7 us of a decode step's first kernel, 1980 us for 65536 rows.  The
// sign of a dot product is taken from its fp32 sum where that sum is beyond any rounding error, which leaves one in ten
// thousand to fp64; the norm of a value likewise, where fp32 decides its fp16 rounding.
#pragma once
#include "common.cuh"

namespace sk {

constexpr int HASH_THREADS = 256;
constexpr int HASH_WARPS = HASH_THREADS / 32;
constexpr int HASH_ROWS = 4;  // rows hashed together by one CTA

template <typename T, int EPL>
__device__ __forceinline__ void load_row_f64(const T* row, int lane, double (&dst)[EPL]) {
#pragma unroll
    for (int i = 0; i < EPL; ++i) dst[i] = (double)to_f32(row[lane * EPL + i]);
}
// EPL elements of a lane, raw; `vec`: the row starts at a multiple of their size, so that one load takes them all
template <typename T, int EPL> struct alignas(sizeof(T) * EPL) Lane {
    T e[EPL];
};
template <typename T, int EPL>
__device__ __forceinline__ Lane<T, EPL> load_lane(const T* row, int lane, bool vec) {
    Lane<T, EPL> r;
    if (vec) {
        r = *reinterpret_cast<const Lane<T, EPL>*>(row + lane * EPL);
    } else {
#pragma unroll
        for (int i = 0; i < EPL; ++i) r.e[i] = row[lane * EPL + i];
    }
    return r;
}
template <typename T, int EPL>
__device__ __forceinline__ void store_lane(T* row, int lane, bool vec, const Lane<T, EPL>& r) {
    if (vec) {
        *reinterpret_cast<Lane<T, EPL>*>(row + lane * EPL) = r;
    } else {
#pragma unroll
        for (int i = 0; i < EPL; ++i) row[lane * EPL + i] = r.e[i];
    }
}
template <typename T, int EPL> __device__ __forceinline__ bool lane_aligned(const T* p) {
    return (reinterpret_cast<uintptr_t>(p) & (sizeof(T) * EPL - 1)) == 0;
}
template <typename T, int EPL>
__device__ __forceinline__ void load_row_f32(const T* row, int lane, float (&dst)[EPL]) {
    const Lane<T, EPL> r = load_lane<T, EPL>(row, lane, lane_aligned<T, EPL>(row));
#pragma unroll
    for (int i = 0; i < EPL; ++i) dst[i] = to_f32(r.e[i]);
}

// Sum of SLOTS per-lane values for each of SLOTS (16 or 32) slots; lane j ends up with the total of slot j mod SLOTS.
template <int SLOTS, typename F>
__device__ __forceinline__ F transpose_reduce(F (&v)[SLOTS], int lane) {
#pragma unroll
    for (int step = SLOTS / 2; step >= 1; step >>= 1) {
        const bool upper = (lane & step) != 0;
#pragma unroll
        for (int i = 0; i < step; ++i) {
            const F send = upper ? v[i] : v[i + step];
            const F keep = upper ? v[i + step] : v[i];
            v[i] = keep + __shfl_xor_sync(FULL, send, step);
        }
    }
    return SLOTS == 16 ? v[0] + __shfl_xor_sync(FULL, v[0], 16) : v[0];
}

__device__ __forceinline__ double warp_sum_f64(double x) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
    return x;
}

// The fp16 rounding of a norm computed in fp32 (a dozen rounded squares and sums, far below 24 units of its last place off) is
// that of the fp64 norm rounded to fp32: not within 24 units of the middle between two fp16 numbers, and inside both normal ranges.
__device__ __forceinline__ bool norm_decides_f16(float norm) {
    return norm >= 6.2e-5f && norm <= 65000.f && (__float_as_uint(norm) & 0x1fffu) - 0x1000u + 24u > 48u;
}

__device__ __forceinline__ void store_code(void* base, int code_bytes, int l, unsigned code) {
    if (code_bytes == 1) static_cast<uint8_t*>(base)[l] = (uint8_t)code;
    else static_cast<int16_t*>(base)[l] = (int16_t)code;
}

// The 8 planes of table `l`, EPL elements per lane each.
template <typename PT, int EPL>
__device__ __forceinline__ void load_planes8(const PT* __restrict__ planes, int l, int lane,
                                             float (&pd)[8][EPL]) {
    constexpr int D = EPL * 32;
    const PT* pl = planes + (size_t)l * 8 * D;
    const bool vec = lane_aligned<PT, EPL>(planes);
    Lane<PT, EPL> raw[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) raw[p] = load_lane<PT, EPL>(pl + (size_t)p * D, lane, vec);
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int i = 0; i < EPL; ++i) pd[p][i] = to_f32(raw[p].e[i]);
}

constexpr float HASH_BAND = 1.52587890625e-05f;       // 2^-16: twice the error of 128 fp32 products and sums against |k| |p|
constexpr float HASH_TINY = 1e-30f;                   // sums of squares below it may have lost terms

// One warp, P == 8: codes of one table for HASH_ROWS rows; keys and planes are in registers.
// code_ptr[r] == nullptr marks an absent row.
template <int EPL>
__device__ __forceinline__ void hash_rows_planes8(const float (&kd)[HASH_ROWS][EPL],
                                                  const float (&pd)[8][EPL],
                                                  void* const (&code_ptr)[HASH_ROWS], int l,
                                                  int code_bytes, int lane) {
    // slot j = r*8 + (7-p): after the ballot, byte r of the mask is row r's code
    float v[32], sq[16];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < EPL; ++i) s = fmaf(kd[r][i], pd[p][i], s);
            v[r * 8 + (7 - p)] = s;
        }
    }
    const float tot = transpose_reduce<32>(v, lane);
    // squared norms: slots 0..3 the rows, 8..15 the planes in the order of the slots above
#pragma unroll
    for (int x = 0; x < 16; ++x) sq[x] = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) sq[r] = fmaf(kd[r][i], kd[r][i], sq[r]);
#pragma unroll
        for (int p = 0; p < 8; ++p) sq[8 + (7 - p)] = fmaf(pd[p][i], pd[p][i], sq[8 + (7 - p)]);
    }
    const float norms = transpose_reduce<16>(sq, lane);
    const float nk = __shfl_sync(FULL, norms, lane >> 3), np = __shfl_sync(FULL, norms, 8 + (lane & 7));
    // false for sums, norms or products outside fp32, and for rows and planes of zeros
    const bool sure = fabsf(tot) > HASH_BAND * (sqrtf(nk) * sqrtf(np)) && fabsf(tot) < INFINITY && nk > HASH_TINY && np > HASH_TINY;
    bool absent = false;
#pragma unroll
    for (int r = 0; r < HASH_ROWS; ++r) absent |= (lane >> 3) == r && code_ptr[r] == nullptr;
    unsigned bits = __ballot_sync(FULL, tot >= 0.f), open = __ballot_sync(FULL, !(sure || absent));
    if (open != 0) {                                   // one warp in a few hundred
        // rows and planes of zeros: their sums are exact
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) {
            bool any = false;
#pragma unroll
            for (int i = 0; i < EPL; ++i) any |= kd[r][i] != 0.f;
            if (!__any_sync(FULL, any)) open &= ~(0xffu << (8 * r));
        }
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            bool any = false;
#pragma unroll
            for (int i = 0; i < EPL; ++i) any |= pd[p][i] != 0.f;
            if (!__any_sync(FULL, any)) open &= ~(0x01010101u << (7 - p));
        }
#pragma unroll 1
        for (; open != 0; open &= open - 1) {
            const int j = __ffs(open) - 1;
            float k[EPL], q[EPL];
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                k[i] = q[i] = 0.f;
#pragma unroll
                for (int r = 0; r < HASH_ROWS; ++r) k[i] = (j >> 3) == r ? kd[r][i] : k[i];
#pragma unroll
                for (int p = 0; p < 8; ++p) q[i] = (j & 7) == 7 - p ? pd[p][i] : q[i];
            }
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < EPL; ++i) s = fma((double)k[i], (double)q[i], s);
            bits = warp_sum_f64(s) >= 0.0 ? bits | 1u << j : bits & ~(1u << j);
        }
    }
#pragma unroll
    for (int r = 0; r < HASH_ROWS; ++r)
        if (lane == r && code_ptr[r] != nullptr) store_code(code_ptr[r], code_bytes, l, (bits >> (8 * r)) & 0xffu);
}

// One warp, any P <= 15: plane by plane.
template <typename PT, int EPL>
__device__ __forceinline__ void hash_rows_generic(const float (&kd)[HASH_ROWS][EPL],
                                                  void* const (&code_ptr)[HASH_ROWS],
                                                  const PT* __restrict__ planes, int l, int P,
                                                  int code_bytes, int lane) {
    constexpr int D = EPL * 32;
    const PT* pl = planes + (size_t)l * P * D;
    unsigned code[HASH_ROWS];
#pragma unroll
    for (int r = 0; r < HASH_ROWS; ++r) code[r] = 0;
    for (int p = 0; p < P; ++p) {
        double pd[EPL];
        load_row_f64<PT, EPL>(pl + (size_t)p * D, lane, pd);
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) {
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < EPL; ++i) s = fma((double)kd[r][i], pd[i], s);
            s = warp_sum_f64(s);
            code[r] = code[r] * 2u + (s >= 0.0 ? 1u : 0u);
        }
    }
#pragma unroll
    for (int r = 0; r < HASH_ROWS; ++r)
        if (lane == 0 && code_ptr[r] != nullptr) store_code(code_ptr[r], code_bytes, l, code[r]);
}

// One warp: codes of table `l` for HASH_ROWS rows whose elements are already in registers.
template <typename PT, int EPL>
__device__ __forceinline__ void hash_table_rows(const float (&kd)[HASH_ROWS][EPL],
                                                void* const (&code_ptr)[HASH_ROWS],
                                                const PT* __restrict__ planes, int l, int P,
                                                int code_bytes, int lane) {
    if (P == 8) {
        float pd[8][EPL];
        load_planes8<PT, EPL>(planes, l, lane, pd);
        hash_rows_planes8<EPL>(kd, pd, code_ptr, l, code_bytes, lane);
    } else {
        hash_rows_generic<PT, EPL>(kd, code_ptr, planes, l, P, code_bytes, lane);
    }
}

// KV-cache append of new (b, s, kvh) rows, HASH_ROWS at a time, from row `n0` on in steps of `step`: this CTA hashes
// them against tables [l0, l0 + HASH_WARPS) (one table per warp, whose planes stay in registers); the CTAs with l0 == 0 also
// copy K and V, store ||v|| as fp16 and advance prefill_len.
template <typename KT, typename PT, int EPL>
__device__ __forceinline__ void kv_append_body(
    const KT* __restrict__ k_new, const KT* __restrict__ v_new, const int64_t* __restrict__ input_pos,
    const PT* __restrict__ planes, KT* __restrict__ k_cache, KT* __restrict__ v_cache,
    uint8_t* __restrict__ codes, __half* __restrict__ v_norm, int32_t* prefill_len, int32_t* status,
    int B, int S, int Hkv, int64_t Tcap, int L, int P, int64_t n0, int64_t step, int l0) {
    constexpr int D = EPL * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t N = (int64_t)B * S * Hkv;
    const int l = l0 + warp;
    const bool fast = (P == 8) && (l < L);
    const bool vec_in = lane_aligned<KT, EPL>(k_new) && lane_aligned<KT, EPL>(v_new);
    const bool vec_out = lane_aligned<KT, EPL>(k_cache) && lane_aligned<KT, EPL>(v_cache);
    float pd[8][EPL];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int i = 0; i < EPL; ++i) pd[p][i] = 0.f;
#pragma unroll 1
    for (bool first = true; n0 < N; n0 += step, first = false) {
        // Every global load is issued before the first one is consumed, so a group costs one memory
        // round trip: the new K rows and this warp's V row (their addresses do not depend on
        // input_pos), the positions, and once the planes.
        const bool mover = l0 == 0 && warp < HASH_ROWS && n0 + warp < N;      // warp r moves row r
        Lane<KT, EPL> kraw[HASH_ROWS], vraw;
        int64_t posv[HASH_ROWS];
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) {
            const int64_t n = n0 + r;
            posv[r] = -1;
#pragma unroll
            for (int i = 0; i < EPL; ++i) kraw[r].e[i] = from_f32<KT>(0.f);
            if (n < N) {
                kraw[r] = load_lane<KT, EPL>(k_new + n * D, lane, vec_in);
                posv[r] = input_pos[S == 1 ? 0u : (uint32_t)n / (uint32_t)Hkv % (uint32_t)S];
            }
        }
#pragma unroll
        for (int i = 0; i < EPL; ++i) vraw.e[i] = from_f32<KT>(0.f);
        if (mover) vraw = load_lane<KT, EPL>(v_new + (n0 + warp) * D, lane, vec_in);
        if (first && fast) load_planes8<PT, EPL>(planes, l, lane, pd);

        float kd[HASH_ROWS][EPL];
        void* code_ptr[HASH_ROWS];
        int64_t cache_row[HASH_ROWS];
#pragma unroll
        for (int r = 0; r < HASH_ROWS; ++r) {
            const int64_t n = n0 + r;
            code_ptr[r] = nullptr;
            cache_row[r] = -1;
#pragma unroll
            for (int i = 0; i < EPL; ++i) kd[r][i] = 0.f;
            if (n < N) {
                const uint32_t bs = (uint32_t)n / (uint32_t)Hkv, b = bs / (uint32_t)S;     // 2^32 rows are a terabyte
                const int kvh = (int)((uint32_t)n - bs * (uint32_t)Hkv);
                const int64_t pos = posv[r];
                if (pos < 0 || pos >= Tcap) {
                    if (status != nullptr && threadIdx.x == 0 && l0 == 0) atomicOr(status, SK_DEV_POS_OUT_OF_RANGE);
                } else {
                    cache_row[r] = ((int64_t)b * Hkv + kvh) * Tcap + pos;
                    code_ptr[r] = codes + cache_row[r] * L;
#pragma unroll
                    for (int i = 0; i < EPL; ++i) kd[r][i] = to_f32(kraw[r].e[i]);
                    if (threadIdx.x == 0 && l0 == 0 && kvh == 0 && b == 0) atomicMax(prefill_len, (int32_t)(pos + 1));
                }
            }
        }
        if (fast) hash_rows_planes8<EPL>(kd, pd, code_ptr, l, 1, lane);
        else if (l < L) hash_rows_generic<PT, EPL>(kd, code_ptr, planes, l, P, 1, lane);
        if (mover) {
            // static indexing of the per-row arrays
#pragma unroll
            for (int r = 0; r < HASH_ROWS; ++r) {
                if (warp != r || cache_row[r] < 0) continue;
                store_lane<KT, EPL>(k_cache + cache_row[r] * D, lane, vec_out, kraw[r]);
                store_lane<KT, EPL>(v_cache + cache_row[r] * D, lane, vec_out, vraw);
                float ss = 0.f;
#pragma unroll
                for (int i = 0; i < EPL; ++i) ss = fmaf(to_f32(vraw.e[i]), to_f32(vraw.e[i]), ss);
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) ss += __shfl_xor_sync(FULL, ss, o);
                float norm = sqrtf(ss);
                if (!norm_decides_f16(norm)) {             // the same for the whole warp
                    double sd = 0.0;
#pragma unroll
                    for (int i = 0; i < EPL; ++i) sd = fma((double)to_f32(vraw.e[i]), (double)to_f32(vraw.e[i]), sd);
                    norm = (float)sqrt(warp_sum_f64(sd));
                }
                if (lane == 0) v_norm[cache_row[r]] = __float2half_rn(norm);
            }
        }
    }
}

}  // namespace sk
