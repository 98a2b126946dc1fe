// State-space recurrence over a prompt portion on the 5th-generation tensor cores (bf16), in chunks of 128 tokens.  With
// cum_t the running sum of the log decays inside a chunk (log2 units) and dt_s the step sizes,
//   y_t   = 2^cum_t q_t^T S_in + sum_{s <= t} 2^(cum_t - cum_s) dt_s (q_t . k_s) x_s + D x_t
//   S_out = 2^cum_end S_in + U,   U = sum_s 2^(cum_end - cum_s) dt_s k_s x_s^T
// (k = B, q = C of the mixer).  A CTA owns 64 value columns of one head and walks the chunks in order.  Only
// S_out = f S_in + U depends on the chunk before, and S lives in fp32 registers of four warps (a key column per thread):
// scores, weights and U of later chunks are made while a chunk's outputs still run, so the chain between chunks is one
// fused multiply-add, a store to shared memory and one product.
//   warps 0-7   scores -> weights (two threads per token, 64 keys each), and the finished outputs
//   warps 8-11  the state;  12, 13, 16, 17 the weighted values;  14 MMA;  15 TMA
// (warp w runs on scheduler w % 4 and can reach the accumulator rows 32 (w % 4) on only; later tokens have more keys, so the
// weighted values, which any warp can make, go to the schedulers of the earlier tokens.)
// Whatever carries a decay or the state enters a product as two bf16 numbers, value and remainder (16 significant bits);
// sums are fp32, and so is the skip D x_t, added to the finished ones (8000 tokens, 128
// heads, with the convolution 291 us; as an addition to the weight of a token with itself, 16 bits of D, 280; with x read again from
// global memory 298).
// Measured (one GPU, inside a decoder; the form in blocks of 64 tokens in brackets): 8000 tokens, 128 heads of 128 x 64, 245 us
// (904); 1501 tokens, 64 heads, 45 us (105).  A chunk takes about 5000 cycles: 80 KiB come in over L2 (3000 cycles when 128
// blocks do so), and the 56 MMAs read 290 KiB of operands from shared memory (3400).  The roles' code has to stay small:
// with every loop of a chunk unrolled (90 KiB of instructions, of which each warp walks its own part once per chunk) a chunk
// took 6900 cycles.
// Every wait is bounded; if one runs out, all roles leave, the head's columns of y and its state become NaN, and the status word says so.
#include "blocks.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"
#include "warp_mma.cuh"

namespace sk {
namespace {

constexpr int TS_TOK = 128, TS_P = 64;                        // tokens of a chunk, value columns of a CTA
constexpr int TS_THREADS = 18 * 32, TS_MMA_WARP = 14, TS_TMA_WARP = 15;
constexpr uint32_t TS_PANEL = TS_TOK * 128;                   // 128 rows x 64 bf16
constexpr uint32_t TS_STAGE = 5 * TS_PANEL;                   // q and k (two panels each), x
constexpr uint32_t TS_IDLE_LIMIT = 1u << 22;                  // rounds of polls without anything to issue: about a second
constexpr float TS_LOG2E = 1.4426950408889634f;

struct TsShape {
    const float *dt, *cum;            // [B, H, chunks, 128]
    const float* skip;
    float* state;                     // [B, H, N, P]
    int32_t* status;
    __nv_bfloat16* y;                 // [B S, H P]
    int64_t start;
    int S, H, P, N, rep, chunks;
};

struct TsShared {
    float cum[2][TS_TOK], dt[2][TS_TOK];
    float fac[TS_TOK];                // 2^(cum at the end of the token's 32 - cum) dt
    uint64_t full[2], empty[2], sc_full[2], p_full[2], u_full[2], f_full, wv_full, wv_empty, s_full, s_empty, y_full, y_empty, drained;
    uint32_t tmem_base;
    int failed;
};
constexpr uint32_t TS_SMEM = 2 * TS_STAGE + 4 * TS_PANEL + sizeof(TsShared);     // stages; state and weighted values, two parts each
static_assert(TS_SMEM <= 232448, "one CTA's shared memory");

// dt = softplus(step column + bias), cum = running sum of -exp(A_log) dt log2(e) inside t's chunk, summed in fp64 so that it
// is rounded once; tokens past the portion's end get dt = 0 and leave the sum as it is.  A CTA: 128 tokens of 16 heads.
constexpr int TS_HEADS = 16;
__global__ void __launch_bounds__(256)
ssm_tc_decay_kernel(sk_ssm_params p, int chunks, float* __restrict__ dt, float* __restrict__ cum) {
    __shared__ float tile[TS_HEADS][TS_TOK + 4];
    const int c = blockIdx.x, h0 = blockIdx.y * TS_HEADS, b = blockIdx.z, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int e = t; e < TS_TOK * TS_HEADS; e += 256) {
        const int s = e / TS_HEADS, k = e % TS_HEADS, h = h0 + k, tok = c * TS_TOK + s;
        float d = 0.f;
        if (h < p.H && tok < p.S)
            d = softplus_f32(to_f32(((const __nv_bfloat16*)p.dt_in)[((int64_t)b * p.S + tok) * p.in_ld + h]) + p.dt_bias[h]);
        tile[k][s] = d;
    }
    __syncthreads();
    for (int k = warp; k < TS_HEADS && h0 + k < p.H; k += 8) {
        const float rate = -expf(p.A_log[h0 + k]) * TS_LOG2E;
        float d[4], run[4];
        double acc = 0.0, part[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            d[e] = tile[k][4 * lane + e];
            acc += (double)rate * (double)d[e];
            part[e] = acc;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double x = __shfl_up_sync(FULL, acc, o);
            if (lane >= o) acc += x;
        }
        const double before = acc - part[3];
#pragma unroll
        for (int e = 0; e < 4; ++e) run[e] = (float)(before + part[e]);
        const int64_t at = (((int64_t)b * p.H + h0 + k) * chunks + c) * TS_TOK + 4 * lane;
        store_vec<float, 4>(dt + at, d);
        store_vec<float, 4>(cum + at, run);
    }
}

__global__ void __launch_bounds__(TS_THREADS, 1)
ssm_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ TsShape p) {
    extern __shared__ __align__(1024) char ts_raw[];
    char* stage_s = ts_raw;                                   // [2][q, q, k, k, x]
    char* st_s = stage_s + 2 * TS_STAGE;                      // the state a chunk starts with: [value, remainder][128 n][64]
    char* wv_s = st_s + 2 * TS_PANEL;                         // weighted values: [value, remainder][128 tokens][64]
    TsShared& sh = *reinterpret_cast<TsShared*>(wv_s + 2 * TS_PANEL);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p0 = blockIdx.x * TS_P, h = blockIdx.y, b = blockIdx.z, g = h / p.rep;
    const int64_t head = (int64_t)b * p.H + h;
    volatile int* failed = &sh.failed;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init_count(&sh.full[s], 1);
            mbar_init_count(&sh.empty[s], 1);
            mbar_init_count(&sh.sc_full[s], 1);
            mbar_init_count(&sh.p_full[s], 8);
            mbar_init_count(&sh.u_full[s], 1);
        }
        mbar_init_count(&sh.f_full, 4);
        mbar_init_count(&sh.wv_full, 4);
        mbar_init_count(&sh.wv_empty, 1);
        mbar_init_count(&sh.s_full, 4);
        mbar_init_count(&sh.s_empty, 1);
        mbar_init_count(&sh.y_full, 1);
        mbar_init_count(&sh.y_empty, 8);
        mbar_init_count(&sh.drained, 1);
        sh.failed = (smem_addr(ts_raw) & 1023u) != 0;         // the swizzled panels need it; the linker aligns the array
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TS_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // columns: scores of two chunks, weights written over them | U of two chunks | q S | weights x
    const uint32_t t_sc = sh.tmem_base, t_u = t_sc + 256, t_qs = t_sc + 384, t_wx = t_sc + 448;
    auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(FULL, mbar_wait_bounded(bar, parity)) != 0; };
    auto gone = [&]() { return __any_sync(FULL, *failed != 0) != 0; };
    bool ok = !gone();

    if (warp < 8) {
        // ---- thread = token and half of the keys (of the value columns in the end)
        const int quarter = warp & 3, half = warp >> 2, t = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const float skip = p.skip[h];
        float carry = 0.f, next = 0.f;
        uint4 x_own[4], x_out[4];                             // the token's x, 32 columns: of this chunk, and of the one before
#pragma unroll 1
        for (int c = 0; ok && c <= p.chunks; ++c) {
            if (c < p.chunks) {
                // Weights of chunk c over its scores: 32 keys in 32 columns, the values' bf16 pairs and then the remainders'.
                // Among the warp's own tokens every weight has an exponential of its own; for 32 keys before them it is a
                // factor of the token times a factor of the key, both relative to the last of these keys, so that neither
                // exponent is above zero.
                const int st = c & 1;
                const uint32_t par = (uint32_t)((c >> 1) & 1);
                ok = wait_all(&sh.full[st], par) && wait_all(&sh.f_full, (uint32_t)(c & 1)) && wait_all(&sh.sc_full[st], par);
                if (!ok) break;
                tc_fence_after();
                const float ct = sh.cum[st][t];
                next = exp2_fast(ct);
#pragma unroll 1
                for (int j = half * 2; j < half * 2 + 2; ++j) {
                    const uint32_t col = t_sc + st * 128 + lane_base + j * 32;
                    uint32_t w[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) w[e] = 0;    // keys later than all of the warp's tokens
                    if (j <= quarter) {
                        float s[32];
                        tmem_ld32(col, reinterpret_cast<uint32_t(&)[32]>(s));
                        if (j < quarter) {
                            const float ft = exp2_fast(ct - sh.cum[st][j * 32 + 31]);
#pragma unroll
                            for (int e = 0; e < 32; e += 4) {
                                const float4 f = *reinterpret_cast<const float4*>(&sh.fac[j * 32 + e]);
                                s[e] *= f.x * ft;
                                s[e + 1] *= f.y * ft;
                                s[e + 2] *= f.z * ft;
                                s[e + 3] *= f.w * ft;
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 32; e += 4) {
                                const float4 cs = *reinterpret_cast<const float4*>(&sh.cum[st][j * 32 + e]);
                                const float4 ds = *reinterpret_cast<const float4*>(&sh.dt[st][j * 32 + e]);
                                const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, dv[4] = {ds.x, ds.y, ds.z, ds.w};
#pragma unroll
                                for (int q = 0; q < 4; ++q) {
                                    const float v = s[e + q] * (exp2_fast(ct - cv[q]) * dv[q]);
                                    s[e + q] = e + q <= lane ? v : 0.f;
                                }
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 16; ++e) split_bf16(s[2 * e], s[2 * e + 1], w[e], w[16 + e]);
                    }
                    tmem_st32(col, w);
                }
                // the skip is added to the finished sums, when the stage may be gone; it stays until this warp's weights are there
                const char* x_s = stage_s + st * TS_STAGE + 4 * TS_PANEL + t * 128;
#pragma unroll
                for (int e = 0; e < 4; ++e) x_own[e] = *reinterpret_cast<const uint4*>(x_s + (((half * 4 + e) ^ (t & 7)) << 4));
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.p_full[st]);
            }
            if (c > 0) {                                      // the outputs of the chunk before
                ok = wait_all(&sh.y_full, (uint32_t)((c - 1) & 1)) && !gone();
                if (!ok) break;
                tc_fence_after();
                const int tok = (c - 1) * TS_TOK + t;
                const int cols = tok < p.S ? p.P - p0 - half * 32 : 0;
                __nv_bfloat16* o = p.y + (((int64_t)b * p.S + tok) * p.H + h) * p.P + p0 + half * 32;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    float x[16], y[16];
                    tmem_ld(t_qs + lane_base + half * 32 + q * 16, reinterpret_cast<uint32_t(&)[16]>(x));
                    tmem_ld(t_wx + lane_base + half * 32 + q * 16, reinterpret_cast<uint32_t(&)[16]>(y));
                    if (q == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.y_empty);
                    }
#pragma unroll
                    for (int e = 0; e < 16; e += 8) {
                        const uint4 own = x_out[q * 2 + e / 8];
                        const uint32_t w[4] = {own.x, own.y, own.z, own.w};
                        float r[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float xt = __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
                            r[j] = fmaf(skip, xt, fmaf(carry, x[e + j], y[e + j]));
                        }
                        if (q * 16 + e < cols) store_vec<__nv_bfloat16, 8>(o + q * 16 + e, r);       // P is a multiple of 8
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) x_out[e] = x_own[e];
            carry = next;
        }
    } else if (warp < 12) {
        // ---- the state: thread = key column n
        const int r = (warp - 8) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((warp - 8) * 32) << 16;
        float* gst = p.state + (head * p.N + r) * p.P + p0;
        const int cols = r >= p.N ? 0 : (p.P - p0 < TS_P ? p.P - p0 : TS_P);
        float s[TS_P];
#pragma unroll
        for (int j = 0; j < TS_P; ++j) s[j] = p.start > 0 && j < cols ? gst[j] : 0.f;
#pragma unroll 1
        for (int c = 0; ok && c < p.chunks; ++c) {
            const int st = c & 1;
            ok = wait_all(&sh.full[st], (uint32_t)((c >> 1) & 1)) && (c == 0 || wait_all(&sh.s_empty, (uint32_t)((c - 1) & 1))) && !gone();
            if (!ok) break;
            const float f = exp2_fast(sh.cum[st][TS_TOK - 1]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                uint4 hi, lo;
                split_bf16(s[8 * j], s[8 * j + 1], hi.x, lo.x);
                split_bf16(s[8 * j + 2], s[8 * j + 3], hi.y, lo.y);
                split_bf16(s[8 * j + 4], s[8 * j + 5], hi.z, lo.z);
                split_bf16(s[8 * j + 6], s[8 * j + 7], hi.w, lo.w);
                char* dst = st_s + r * 128 + ((j ^ (r & 7)) << 4);
                *reinterpret_cast<uint4*>(dst) = hi;
                *reinterpret_cast<uint4*>(dst + TS_PANEL) = lo;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();                                // U of the chunk before has been read
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.s_full);
            ok = wait_all(&sh.u_full[st], (uint32_t)((c >> 1) & 1));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float u[32];
                tmem_ld32(t_u + st * 64 + lane_base + q * 32, reinterpret_cast<uint32_t(&)[32]>(u));
#pragma unroll
                for (int j = 0; j < 32; ++j) s[q * 32 + j] = fmaf(f, s[q * 32 + j], u[j]);
            }
        }
        tc_fence_before();
        if (ok) {
#pragma unroll
            for (int j = 0; j < TS_P; j += 4)
                if (j < cols) *reinterpret_cast<float4*>(gst + j) = make_float4(s[j], s[j + 1], s[j + 2], s[j + 3]);
        }
    } else if (warp == 12 || warp == 13 || warp >= 16) {
        // ---- the keys' factors; weighted values: eight lanes along a token's 64 columns, in the swizzled places they came to
        const int at = (warp < 16 ? warp - 12 : warp - 14) * 32 + lane;
#pragma unroll 1
        for (int c = 0; ok && c < p.chunks; ++c) {
            const int st = c & 1;
            ok = wait_all(&sh.full[st], (uint32_t)((c >> 1) & 1)) && (c == 0 || wait_all(&sh.p_full[st ^ 1], (uint32_t)(((c - 1) >> 1) & 1)));
            if (!ok) break;
            sh.fac[at] = exp2_fast(sh.cum[st][at | 31] - sh.cum[st][at]) * sh.dt[st][at];
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.f_full);
            ok = (c == 0 || wait_all(&sh.wv_empty, (uint32_t)((c - 1) & 1))) && !gone();
            if (!ok) break;
            const char* x_s = stage_s + st * TS_STAGE + 4 * TS_PANEL;
            const float end = sh.cum[st][TS_TOK - 1];
#pragma unroll 2
            for (int it = 0; it < 8; ++it) {
                const int s = it * 16 + (at >> 3);
                const float w = exp2_fast(end - sh.cum[st][s]) * sh.dt[st][s];
                const uint4 raw = *reinterpret_cast<const uint4*>(x_s + it * 2048 + at * 16);
                uint4 hi, lo;
                split_bf16(__uint_as_float(raw.x << 16) * w, __uint_as_float(raw.x & 0xffff0000u) * w, hi.x, lo.x);
                split_bf16(__uint_as_float(raw.y << 16) * w, __uint_as_float(raw.y & 0xffff0000u) * w, hi.y, lo.y);
                split_bf16(__uint_as_float(raw.z << 16) * w, __uint_as_float(raw.z & 0xffff0000u) * w, hi.z, lo.z);
                split_bf16(__uint_as_float(raw.w << 16) * w, __uint_as_float(raw.w & 0xffff0000u) * w, hi.w, lo.w);
                char* dst = wv_s + it * 2048 + at * 16;
                *reinterpret_cast<uint4*>(dst) = hi;
                *reinterpret_cast<uint4*>(dst + TS_PANEL) = lo;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.wv_full);
        }
    } else if (warp == TS_TMA_WARP) {
        if (lane == 0) {
            const int64_t e_at = head * p.chunks * TS_TOK;
            int c = 0;
#pragma unroll 1
            for (; ok && c < p.chunks && !*failed; ++c) {
                const int st = c & 1;
                if (c >= 2 && !mbar_wait_bounded(&sh.empty[st], (uint32_t)(((c >> 1) - 1) & 1))) {
                    ok = false;
                    break;
                }
                char* dst = stage_s + st * TS_STAGE;
                mbar_expect(&sh.full[st], TS_STAGE + 2 * TS_TOK * 4);
                for (int q = 0; q < 2; ++q) {
                    tma_load_4d(dst + q * TS_PANEL, &map_q, q * 64, g, c * TS_TOK, b, &sh.full[st]);
                    tma_load_4d(dst + (2 + q) * TS_PANEL, &map_k, q * 64, g, c * TS_TOK, b, &sh.full[st]);
                }
                tma_load_4d(dst + 4 * TS_PANEL, &map_v, p0, h, c * TS_TOK, b, &sh.full[st]);
                bulk_load(sh.cum[st], p.cum + e_at + (int64_t)c * TS_TOK, TS_TOK * 4, &sh.full[st]);
                bulk_load(sh.dt[st], p.dt + e_at + (int64_t)c * TS_TOK, TS_TOK * 4, &sh.full[st]);
            }
            if (c < p.chunks)                                 // left early: no copy stays in flight
                for (int q = c > 2 ? c - 2 : 0; q < c; ++q) mbar_wait_bounded(&sh.full[q & 1], (uint32_t)((q >> 1) & 1));
        }
        ok = __all_sync(FULL, ok) != 0;
    } else {
        // ---- MMAs: the warp stays converged, one lane issues (see umma_ss_by)
        const bool leader = elect_one();
        const uint32_t id_k = umma_idesc_bf16(TS_TOK, false), id_mn = umma_idesc_bf16(TS_P, true), id_u = id_mn | UMMA_A_MN;
        const uint64_t q_k = umma_desc_sw128(smem_addr(stage_s)), k_k = umma_desc_sw128(smem_addr(stage_s + 2 * TS_PANEL)),
                       k_mn = umma_desc_sw128_mn(smem_addr(stage_s + 2 * TS_PANEL), TS_PANEL),
                       x_mn = umma_desc_sw128_mn(smem_addr(stage_s + 4 * TS_PANEL), TS_PANEL),
                       s_mn = umma_desc_sw128_mn(smem_addr(st_s), TS_PANEL), w_mn = umma_desc_sw128_mn(smem_addr(wv_s), TS_PANEL);
        const int k16 = (p.N + 15) / 16;
        // Four products per chunk, each kind in order and each issued as soon as its operands are there: an order fixed in
        // advance waits for the next chunk's copy while products of this one could run.
        int ns = 0, nu = 0, nq = 0, nw = 0;                   // chunks issued: scores, U, q S, weights x
        uint32_t idle = 0;
        auto ready = [&](uint64_t* bar, uint32_t parity) { return mbar_test(bar, parity); };
#pragma unroll 1
        while (ok && (nu < p.chunks || nq < p.chunks || nw < p.chunks)) {
            bool any = false;
            // over the weights of the chunk before the last, whose product has been issued
            if (ns < p.chunks && ns <= nw + 1 && ready(&sh.full[ns & 1], (uint32_t)((ns >> 1) & 1))) {
                const int st = __shfl_sync(FULL, ns & 1, 0);       // uniform to the compiler as well
                const uint32_t at = st * (TS_STAGE >> 4);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t off = at + (uint32_t)(k >> 2) * (TS_PANEL >> 4) + (k & 3) * 2;
                    if (k < k16) umma_ss_by(leader, t_sc + st * 128, umma_desc_at(q_k, off), umma_desc_at(k_k, off), id_k, k > 0);
                }
                umma_commit_by(leader, &sh.sc_full[st]);
                ++ns;
                any = true;
            }
            // the state warps have read the U of the chunk before the last when they publish the state after it
            if (nu < ns && (nu < 2 || nu <= nq) && ready(&sh.wv_full, (uint32_t)(nu & 1))) {
                const int st = __shfl_sync(FULL, nu & 1, 0);
                const uint32_t at = st * (TS_STAGE >> 4);
                tc_fence_after();
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int k = 0; k < TS_TOK / 16; ++k)
                        umma_ss_by(leader, t_u + st * 64, umma_desc_at(k_mn, at + k * (2048 >> 4)),
                                   umma_desc_at(w_mn, part * (TS_PANEL >> 4) + k * (2048 >> 4)), id_u, part > 0 || k > 0);
                umma_commit_by(leader, &sh.u_full[st]);
                umma_commit_by(leader, &sh.wv_empty);
                if (nq > nu && nw > nu) umma_commit_by(leader, &sh.empty[st]);
                ++nu;
                any = true;
            }
            if (nq < p.chunks && nq < ns && ready(&sh.s_full, (uint32_t)(nq & 1)) &&
                (nq == 0 || ready(&sh.y_empty, (uint32_t)((nq - 1) & 1)))) {
                const int st = __shfl_sync(FULL, nq & 1, 0);
                const uint32_t at = st * (TS_STAGE >> 4);
                tc_fence_after();
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k < k16)
                            umma_ss_by(leader, t_qs, umma_desc_at(q_k, at + (uint32_t)(k >> 2) * (TS_PANEL >> 4) + (k & 3) * 2),
                                       umma_desc_at(s_mn, part * (TS_PANEL >> 4) + k * (2048 >> 4)), id_mn, part > 0 || k > 0);
                umma_commit_by(leader, &sh.s_empty);
                if (nw > nq) umma_commit_by(leader, &sh.y_full);
                if (nu > nq && nw > nq) umma_commit_by(leader, &sh.empty[st]);
                ++nq;
                any = true;
            }
            if (nw < ns && ready(&sh.p_full[nw & 1], (uint32_t)((nw >> 1) & 1)) &&
                (nw == 0 || ready(&sh.y_empty, (uint32_t)((nw - 1) & 1)))) {
                const int st = __shfl_sync(FULL, nw & 1, 0);
                const uint32_t at = st * (TS_STAGE >> 4);
                tc_fence_after();
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int k = 0; k < TS_TOK / 16; ++k)
                        // rows before these 16 keys have weights of zero for them, which an infinite or NaN x would not leave without
                        // effect: they are left out (k = 0, which all rows take, comes first)
                        umma_ts_from(leader, t_wx, t_sc + st * 128 + (k >> 1) * 32 + part * 16 + (k & 1) * 8,
                                     umma_desc_at(x_mn, at + k * (2048 >> 4)), id_mn, part > 0 || k > 0, k * 16);
                if (nq > nw) umma_commit_by(leader, &sh.y_full);
                if (nu > nw && nq > nw) umma_commit_by(leader, &sh.empty[st]);
                ++nw;
                any = true;
            }
            idle = any ? 0 : idle + 1;
            if (idle > TS_IDLE_LIMIT || gone()) ok = false;
        }
        umma_commit_by(leader, &sh.drained);                  // leave no MMA and no barrier arrival in flight
        mbar_wait_bounded(&sh.drained, 0);
    }
    if (!ok && lane == 0) *failed = 1;
    __syncthreads();
    if (sh.failed) {
        if (tid == 0 && p.status != nullptr) atomicOr(p.status, SK_DEV_WAIT_TIMEOUT);
        const int c = tid & (TS_P - 1);
        if (p0 + c < p.P) {
#pragma unroll 1
            for (int r = tid / TS_P; r < p.S; r += TS_THREADS / TS_P) p.y[(((int64_t)b * p.S + r) * p.H + h) * p.P + p0 + c] = __float2bfloat16_rn(NAN);
#pragma unroll 1
            for (int r = tid / TS_P; r < p.N; r += TS_THREADS / TS_P) p.state[(head * p.N + r) * p.P + p0 + c] = NAN;
        }
    }
    if (warp == TS_MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem_base), "r"(512u) : "memory");
}

int ts_chunks(int S) { return (S + TS_TOK - 1) / TS_TOK; }

}  // namespace

size_t ssm_tc_workspace(const sk_ssm_params& p) {             // step sizes and running decays
    return (size_t)2 * p.B * p.H * ts_chunks(p.S) * TS_TOK * sizeof(float);
}

bool ssm_tc_applicable(const sk_ssm_params& p) {
    // step sizes and decays are written and copied 16 bytes at a time (no workspace yet: a query)
    if ((uintptr_t)p.workspace % 16 != 0) return false;
    if (p.dtype != SK_BF16 || p.pos != nullptr || p.N % 8 != 0 || p.N > 128 || p.P % 8 != 0) return false;
    const __nv_bfloat16* x = (const __nv_bfloat16*)p.xbc;
    const __nv_bfloat16* k = x + (int64_t)p.H * p.P;
    const int64_t bs = (int64_t)p.S * p.xbc_ld;
    return p.B <= 65535 && p.H <= 65535 && head_map_ok(x, p.P, p.P, p.xbc_ld, bs) && head_map_ok(k, p.N, p.N, p.xbc_ld, bs) &&
           head_map_ok(k + (int64_t)p.G * p.N, p.N, p.N, p.xbc_ld, bs) && (uintptr_t)p.y % 16 == 0 && (uintptr_t)p.state % 16 == 0;
}

int launch_ssm_tc(const sk_ssm_params& p, cudaStream_t st) {
    const int chunks = ts_chunks(p.S);
    float* dt = (float*)p.workspace;
    float* cum = dt + (size_t)p.B * p.H * chunks * TS_TOK;
    const __nv_bfloat16* x = (const __nv_bfloat16*)p.xbc;     // row: [x (H P) | B (G N) | C (G N)]
    const __nv_bfloat16* k = x + (int64_t)p.H * p.P;
    const int64_t bs = (int64_t)p.S * p.xbc_ld;
    CUtensorMap mq, mk, mv;
    if (int rc = make_head_map(&mq, k + (int64_t)p.G * p.N, p.N, p.G, p.S, p.B, p.N, p.xbc_ld, bs, TS_TOK)) return rc;
    if (int rc = make_head_map(&mk, k, p.N, p.G, p.S, p.B, p.N, p.xbc_ld, bs, TS_TOK)) return rc;
    if (int rc = make_head_map(&mv, x, p.P, p.H, p.S, p.B, p.P, p.xbc_ld, bs, TS_TOK)) return rc;
    const cudaError_t e = cudaFuncSetAttribute(ssm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS_SMEM);
    if (e != cudaSuccess) return fail(SK_ERR_CUDA, "ssm_tc_kernel smem attribute: %s", cudaGetErrorString(e));
    ssm_tc_decay_kernel<<<dim3((unsigned)chunks, (unsigned)((p.H + TS_HEADS - 1) / TS_HEADS), (unsigned)p.B), 256, 0, st>>>(p, chunks, dt, cum);
    if (int rc = check_launch("ssm_tc_decay_kernel")) return rc;
    TsShape s{};
    s.dt = dt;
    s.cum = cum;
    s.skip = p.D;
    s.state = p.state;
    s.status = p.status;
    s.y = (__nv_bfloat16*)p.y;
    s.start = p.start;
    s.S = p.S;
    s.H = p.H;
    s.P = p.P;
    s.N = p.N;
    s.rep = p.H / p.G;
    s.chunks = chunks;
    ssm_tc_kernel<<<dim3((unsigned)((p.P + TS_P - 1) / TS_P), (unsigned)p.H, (unsigned)p.B), TS_THREADS, TS_SMEM, st>>>(mq, mk, mv, s);
    return check_launch("ssm_tc_kernel");
}

}  // namespace sk
