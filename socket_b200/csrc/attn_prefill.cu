// Softmax attention of a prompt portion on the 5th-generation tensor cores (bf16).
//
// A CTA owns 256 consecutive queries of one head as two tiles of 128.  One warp feeds 128-key tiles of K
// and V by TMA (128-byte swizzle), one thread issues the MMAs: S = Q K^T into tensor memory (fp32,
// shared-memory operands), O += P V with P read from tensor memory.  Each query tile has eight softmax warps, two
// threads per query row with 64 of its 128 scores each: they scale / bias / mask them, keep the running maximum (which
// the two exchange) and their sum, and write the weights back over their own scores as bf16.  While one tile is in its
// softmax the tensor core works on the other.  The accumulator is rescaled only when a row's maximum has grown by more
// than 2^8 since the last time (the final division by the sum makes the choice of reference invisible).  Scores under
// a cap are bounded, so weights are taken relative to zero: no maximum, no exchange, no rescaling.
//
// Visibility is causal, optionally restricted to the query's own chunk of positions or to a sliding window; tiles
// that no row of a query tile can see are not visited.  Out-of-range rows and columns of a tile are zero-filled by TMA.
// Every wait is bounded; one that runs out makes all roles leave, and is reported in the status word.
//
// Bound: the softmax arithmetic of a tile (the exponential's unit and the issue slots of 16 warps) beside 2 x 512 cycles of
// MMAs.  Measured, one GPU, L2 flushed (with four warps per tile, one thread per row, and the MMAs built and issued in one
// lane's loop: in brackets): 8000 tokens, 32 / 8 heads of 128, chunk and bias 586 us (996); 32 heads of 192 / 128 with
// sinks 677 us (1098); 32000 tokens, 16 heads, window 4096 and cap 1136 us (1739); 1501 tokens behind 2500, 16 heads,
// bias 94 us (133).
#include "blocks.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace sk {
namespace {

constexpr int FP_TILE = 128;                                  // queries of a tile = keys of a tile
constexpr int FP_HALF = FP_TILE / 2;                          // keys of a softmax thread
constexpr int FP_SOFTMAX_WARPS = 16;                          // warp: 8 tile + 4 half + quarter of the rows
constexpr int FP_TMA_WARP = 16, FP_MMA_WARP = 17;
constexpr int FP_THREADS = 32 * (FP_SOFTMAX_WARPS + 4);       // the last two warps idle: registers are dealt to groups of four
// Registers a thread: 96 at launch (640 threads), then 112 for the softmax warps and 32 for the others
// (512 x 112 + 128 x 32 = 61440, all that the block was launched with; with 104 and 64 the first two figures above are 655
// and 900 us).  64 scores and their weights do not quite fit: 270 to 360 bytes a thread are spilled in every form.
constexpr int FP_REGS_SOFTMAX = 112, FP_REGS_OTHER = 32;
constexpr uint32_t FP_PANEL = FP_TILE * 128;                  // 128 rows x 64 bf16
constexpr int FP_BIAS_SPAN = 96;                              // distances a warp's 32 rows x 64 keys can have
constexpr uint32_t FP_BIAS_BYTES = FP_SOFTMAX_WARPS * FP_BIAS_SPAN * sizeof(float);
constexpr float FP_RESCALE = 8.f;                             // log2 units
constexpr float FP_LOG2E = 1.4426950408889634f;

struct FpShared {
    uint64_t q_full;
    uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
    uint64_t s_full[2], p_full[2], o_full[2];
    uint64_t drained;
    uint32_t tmem_base;
    int failed;
    float xch[FP_SOFTMAX_WARPS][32];         // what the two threads of a row tell each other
};

// Dynamic shared memory: operand tiles, bias, FpShared.  Its start is a multiple of 1024 when there is no static shared
// data; a launch adds what is left of the limit, up to 1008 bytes, for a start that is not.
constexpr uint32_t FP_SMEM_LIMIT = 232448;

struct FpShape {            // what the kernel needs beside the tensor maps
    void* out;
    const float *bias, *sink;
    int32_t* status;
    int64_t o_bs, o_ss, o_hs, start, kv_start, bias_len;
    int S, H, G, dqk, dv, chunk, window, nk, nv;      // nk, nv: stages of the K and V rings
    int q_blocks;                             // blocks of 256 queries
    float scale_log2, cap_in, cap_out;        // softcap: s <- cap_out tanh(s cap_in), log2 units
    float cap_poly[5], cap_small;             // the same for s^2 <= cap_small: s times a polynomial in s^2
};
// Softcap: none, any, or one so low that exp of a capped score and sums of it stay far inside the fp32 range
enum { FP_CAP_NONE = 0, FP_CAP = 1, FP_CAP_BOUND = 2 };
constexpr float FP_CAP_BOUND_LOG2 = 80.f;

// first key row (counted from kv_start: rows of the call, below 2^30, whatever the positions are) that query row i sees
__device__ __forceinline__ int fp_first_row(const FpShape& p, int i) {
    int64_t lo = -p.kv_start;
    if (p.chunk > 0) lo = (i + p.kv_start) / p.chunk * p.chunk - p.kv_start;
    if (p.window > 0 && i - p.window + 1 > lo) lo = i - p.window + 1;
    return (int)max(lo, (int64_t)0);
}

// s <- cap_out tanh(s cap_in) for 16 scores from c0 on; the caller's loops are unrolled
template <int N> __device__ __forceinline__ void fp_cap16(const FpShape& p, float (&s)[N], int c0) {
    uint64_t t[8];
    float top[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint64_t x = pack2(s[c0 + 2 * i], s[c0 + 2 * i + 1]);
        t[i] = mul2(x, x);
        float a, b;
        unpack2(t[i], a, b);
        top[i & 1] = max3(top[i & 1], a, b);
    }
    if (__any_sync(FULL, !(fmaxf(top[0], top[1]) <= p.cap_small))) {
#pragma unroll
        for (int c = 0; c < 16; ++c) s[c0 + c] = p.cap_out * tanh_exp2(s[c0 + c] * p.cap_in);
    } else {
        const uint64_t k0 = pack2(p.cap_poly[0], p.cap_poly[0]), k1 = pack2(p.cap_poly[1], p.cap_poly[1]),
                       k2 = pack2(p.cap_poly[2], p.cap_poly[2]), k3 = pack2(p.cap_poly[3], p.cap_poly[3]),
                       k4 = pack2(p.cap_poly[4], p.cap_poly[4]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint64_t r = fma2(t[i], k4, k3);
            r = fma2(t[i], r, k2);
            r = fma2(t[i], r, k1);
            r = fma2(t[i], r, k0);
            r = mul2(r, pack2(s[c0 + 2 * i], s[c0 + 2 * i + 1]));
            unpack2(r, s[c0 + 2 * i], s[c0 + 2 * i + 1]);
        }
    }
}

template <bool BIAS, int CAP>
__global__ void __launch_bounds__(FP_THREADS, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const FpShape p) {
    extern __shared__ __align__(1024) char fp_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(fp_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // heads side by side, long rows first: the last blocks to start are short ones.  (Heads in groups whose keys and values fit
    // the L2 end in a short group of long rows: 24000 tokens, 16 heads of 192 / 128 in groups of 3: 2975 us, so 2643; 8000
    // tokens, 32 heads in groups of 9: 699 us, so 677.  16000 tokens, 16 heads were 1177 us in groups and are 1207 so.)
    const int b = blockIdx.y, back = blockIdx.x / p.H, h = blockIdx.x - back * p.H, g = h / (p.H / p.G);
    const int np = (p.dqk + 63) / 64, nvp = (p.dv + 63) / 64;
    char* q_s = tiles;                                        // [tile][panel]
    char* k_s = q_s + 2 * np * FP_PANEL;                      // [stage][panel]
    char* v_s = k_s + p.nk * np * FP_PANEL;
    float* bias_s = reinterpret_cast<float*>(v_s + p.nv * nvp * FP_PANEL);
    FpShared& sh = *reinterpret_cast<FpShared*>(reinterpret_cast<char*>(bias_s) + (BIAS ? FP_BIAS_BYTES : 0));

    // query tiles, and the range [beg, end) of key tiles each of them visits; key rows count from kv_start
    const int q0 = (p.q_blocks - 1 - back) * 2 * FP_TILE;
    int i0[2], beg[2], end[2], base = 0;                      // rows of a call: below 2^30
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int first = q0 + t * FP_TILE;
        i0[t] = (int)(p.start - p.kv_start) + first;
        const int lo = fp_first_row(p, i0[t]);
        if (t == 0) base = lo;
        const int rows = p.S - first < FP_TILE ? p.S - first : FP_TILE;
        beg[t] = (lo - base) / FP_TILE;
        end[t] = rows > 0 ? (i0[t] + rows - 1 - base) / FP_TILE + 1 : 0;
        if (rows <= 0) beg[t] = 0;
    }
    const int n = end[1] > end[0] ? end[1] : end[0];
    uint32_t room;                                            // the tiles end inside what was launched, wherever shared memory begins
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(room));
    const uint32_t used = (uint32_t)((char*)(&sh + 1) - fp_raw);
    if (used > room) {
        if (tid == 0 && p.status != nullptr) atomicOr(p.status, SK_DEV_WAIT_TIMEOUT);
        return;
    }

    if (tid == 0) {
        mbar_init_count(&sh.q_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init_count(&sh.k_full[s], 1);
            mbar_init_count(&sh.k_empty[s], 1);
            mbar_init_count(&sh.v_full[s], 1);
            mbar_init_count(&sh.v_empty[s], 1);
            mbar_init_count(&sh.s_full[s], 1);
            mbar_init_count(&sh.p_full[s], 8);
            mbar_init_count(&sh.o_full[s], 1);
        }
        mbar_init_count(&sh.drained, 1);
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == FP_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;                       // columns: S0 | S1 | O0 | O1, 128 each
    volatile int* failed = &sh.failed;

    if (warp >= FP_SOFTMAX_WARPS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FP_REGS_OTHER));
    if (warp == FP_TMA_WARP) {
        // ---- TMA producer
        if (lane == 0) {
            const uint32_t k_bytes = np * FP_PANEL, v_bytes = nvp * FP_PANEL;
            mbar_expect(&sh.q_full, 2 * k_bytes);
            for (int t = 0; t < 2; ++t)
                for (int c = 0; c < np; ++c)
                    tma_load_4d(q_s + (t * np + c) * FP_PANEL, &map_q, c * 64, h, q0 + t * FP_TILE, b, &sh.q_full);
            int j = 0;
            bool k_sent = false;
            for (; j < n && !*failed; ++j) {
                const int ks = j % p.nk, vs = j % p.nv, row = base + j * FP_TILE;
                if (j >= p.nk && !mbar_wait_bounded(&sh.k_empty[ks], (uint32_t)((j / p.nk - 1) & 1))) { *failed = 1; break; }
                mbar_expect(&sh.k_full[ks], k_bytes);
                for (int c = 0; c < np; ++c)
                    tma_load_4d(k_s + (ks * np + c) * FP_PANEL, &map_k, c * 64, g, row, b, &sh.k_full[ks]);
                k_sent = true;
                if (j >= p.nv && !mbar_wait_bounded(&sh.v_empty[vs], (uint32_t)((j / p.nv - 1) & 1))) { *failed = 1; break; }
                mbar_expect(&sh.v_full[vs], v_bytes);
                for (int c = 0; c < nvp; ++c)
                    tma_load_4d(v_s + (vs * nvp + c) * FP_PANEL, &map_v, c * 64, g, row, b, &sh.v_full[vs]);
                k_sent = false;
            }
            if (*failed) {                                    // leave no copy in flight
                mbar_wait_bounded(&sh.q_full, 0);
                const int nk_sent = j + (k_sent ? 1 : 0);
                for (int i = nk_sent > p.nk ? nk_sent - p.nk : 0; i < nk_sent; ++i)
                    mbar_wait_bounded(&sh.k_full[i % p.nk], (uint32_t)((i / p.nk) & 1));
                for (int i = j > p.nv ? j - p.nv : 0; i < j; ++i)
                    mbar_wait_bounded(&sh.v_full[i % p.nv], (uint32_t)((i / p.nv) & 1));
            }
        }
    } else if (warp == FP_MMA_WARP) {
        // ---- MMA issuer.  The whole warp walks the tiles and waits, one lane issues: operands then are warp-uniform, and an
        // MMA costs an addition per descriptor (built in one lane's loop, each took about 200 cycles to issue and 64 to run)
        const bool leader = elect_one();
        const uint32_t idesc_s = umma_idesc_bf16(FP_TILE, false), idesc_o = umma_idesc_bf16((p.dv + 15) / 16 * 16, true);
        const int k_steps = (p.dqk + 15) / 16;
        const uint64_t q_desc = umma_desc_sw128(smem_addr(q_s)), k_desc = umma_desc_sw128(smem_addr(k_s)),
                       v_desc = umma_desc_sw128_mn(smem_addr(v_s), FP_PANEL);
        const uint32_t k_stage = np * FP_PANEL >> 4, v_stage = nvp * FP_PANEL >> 4, k_mask = p.nk - 1, v_mask = p.nv - 1;
        auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(FULL, mbar_wait_bounded(bar, parity)) != 0; };
        auto step = [&](uint32_t d, uint64_t qd, uint64_t kd, int k) {
            const uint32_t off = (uint32_t)(k >> 2) * (FP_PANEL >> 4) + (k & 3) * 2;
            umma_ss_by(leader, d, umma_desc_at(qd, off), umma_desc_at(kd, off), idesc_s, k > 0);
        };
        auto scores = [&](int t, int j) {                     // S_t = Q_t K_j^T
            const uint64_t qd = umma_desc_at(q_desc, t * k_stage), kd = umma_desc_at(k_desc, (j & k_mask) * k_stage);
            const uint32_t d = tmem + t * FP_TILE;
            if (k_steps == 8) {
#pragma unroll
                for (int k = 0; k < 8; ++k) step(d, qd, kd, k);
            } else if (k_steps == 12) {
#pragma unroll
                for (int k = 0; k < 12; ++k) step(d, qd, kd, k);
            } else {
                for (int k = 0; k < k_steps; ++k) step(d, qd, kd, k);
            }
            umma_commit_by(leader, &sh.s_full[t]);
        };
        bool ok = wait_all(&sh.q_full, 0) && wait_all(&sh.k_full[0], 0);
        if (ok) {
            tc_fence_after();
            for (int t = 0; t < 2; ++t)
                if (beg[t] == 0 && end[t] > 0) scores(t, 0);
            umma_commit_by(leader, &sh.k_empty[0]);
        }
        for (int j = 0; ok && j < n && !__any_sync(FULL, *failed != 0); ++j) {
            const bool more = j + 1 < n;
            if (more) ok = wait_all(&sh.k_full[(j + 1) & k_mask], p.nk == 1 ? (uint32_t)((j + 1) & 1) : (uint32_t)(((j + 1) >> 1) & 1));
            ok = ok && wait_all(&sh.v_full[j & v_mask], p.nv == 1 ? (uint32_t)(j & 1) : (uint32_t)((j >> 1) & 1));
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (ok && j >= beg[t] && j < end[t]) {
                    ok = wait_all(&sh.p_full[t], (uint32_t)((j - beg[t]) & 1));
                    if (ok) {
                        tc_fence_after();
                        const uint64_t vd = umma_desc_at(v_desc, (j & v_mask) * v_stage);
#pragma unroll
                        for (int k = 0; k < FP_TILE / 16; ++k)
                            umma_ts_by(leader, tmem + 2 * FP_TILE + t * FP_TILE, tmem + t * FP_TILE + (k >> 2) * FP_HALF + (k & 3) * 8,
                                       umma_desc_at(vd, k * (2048 >> 4)), idesc_o, k > 0 || j > beg[t]);
                        if (j + 1 == end[t]) umma_commit_by(leader, &sh.o_full[t]);
                    }
                }
                // the scores of the next key tile replace weights that the MMAs above still read: same
                // issuing thread, so they execute in order
                if (t == 1 && ok) umma_commit_by(leader, &sh.v_empty[j & v_mask]);     // V goes on its way meanwhile
                if (ok && more && j + 1 >= beg[t] && j + 1 < end[t]) scores(t, j + 1);
            }
            if (ok && more) umma_commit_by(leader, &sh.k_empty[(j + 1) & k_mask]);
        }
        if (!ok && lane == 0) *failed = 1;
        umma_commit_by(leader, &sh.drained);                  // leave no MMA and no barrier arrival in flight
        mbar_wait_bounded(&sh.drained, 0);
    } else if (warp < FP_SOFTMAX_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FP_REGS_SOFTMAX));
        // ---- softmax: two threads per query row, 64 keys each
        const int t = warp >> 3, half = (warp >> 2) & 1, quad = warp & 3, a = quad * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        // the weights of a half go over the first 32 columns of its own scores
        const uint32_t s_addr = tmem + lane_base + t * FP_TILE + half * FP_HALF;
        const uint32_t o_addr = tmem + lane_base + 2 * FP_TILE + t * FP_TILE;
        const int i = i0[t] + a;                              // query row in key-row coordinates
        const float cc = BIAS || CAP != FP_CAP_NONE ? 1.f : p.scale_log2;    // log2 units per unit of s below
        const int lo_row = fp_first_row(p, i), lo_last = fp_first_row(p, i0[t] + quad * 32 + 31);
        float* bt = bias_s + warp * FP_BIAS_SPAN;
        const float* bias_h = BIAS ? p.bias + (int64_t)h * p.bias_len : nullptr;
        const int bias_last = (int)(p.bias_len < (1 << 30) ? p.bias_len : 1 << 30) - 1;
        // this warp's distances in tile j: row - key = bias_first(j) + 0 .. 94
        auto bias_first = [&](int j) { return i0[t] + quad * 32 - (base + j * FP_TILE + half * FP_HALF) - (FP_HALF - 1); };
        auto bias_at = [&](int d) { return __ldg(bias_h + min(max(d, 0), bias_last)) * FP_LOG2E; };
        float bias_next[FP_BIAS_SPAN / 32], bias_far = 0.f;   // requested a tile ahead
        if (BIAS && end[t] > 0) {
            bias_far = bias_at(bias_last);
#pragma unroll
            for (int e = 0; e < FP_BIAS_SPAN / 32; ++e) bias_next[e] = bias_at(bias_first(beg[t]) + lane + 32 * e);
        }
        // both warps of a row quarter come here equally often, whatever happened to the waits; between two turns lies a wait
        // for MMAs that the other warp has let go, so it has read what the turn before left
        auto partner = [&](float v) {
            sh.xch[warp][lane] = v;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quad) : "memory");
            return sh.xch[warp ^ 4][lane];
        };
        float m = CAP == FP_CAP_BOUND ? 0.f : -INFINITY, l = 0.f;
        bool ok = true;                                       // a wait that ran out: no more waits, the rest runs through
        for (int j = beg[t]; j < end[t]; ++j) {
            const int it = j - beg[t];
            const int r0 = base + j * FP_TILE + half * FP_HALF;
            bool far = false;                                 // every distance is beyond the table
            if (BIAS) {
                far = bias_first(j) >= bias_last;
                if (!far) {
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < FP_BIAS_SPAN / 32; ++e) bt[lane + 32 * e] = bias_next[e];
                    __syncwarp();
                }
                if (bias_first(j + 1) < bias_last) {
#pragma unroll
                    for (int e = 0; e < FP_BIAS_SPAN / 32; ++e) bias_next[e] = bias_at(bias_first(j + 1) + lane + 32 * e);
                }
            }
            if (ok) ok = __all_sync(FULL, mbar_wait_bounded(&sh.s_full[t], (uint32_t)(it & 1)));
            tc_fence_after();
            const bool partial = r0 + FP_HALF - 1 > i0[t] + quad * 32 || r0 < lo_last;     // some row does not see all these keys
            const int hi_c = i - r0, lo_c = lo_row - r0;
            float s[FP_HALF];
            tmem_ld64(s_addr, reinterpret_cast<uint32_t(&)[FP_HALF]>(s));
            if (CAP != FP_CAP_NONE) {                         // small scores: a polynomial, off the exponential's unit
#pragma unroll
                for (int c = 0; c < FP_HALF; c += 16) fp_cap16(p, s, c);
            }
            if (BIAS) {
                const float sc = CAP != FP_CAP_NONE ? 1.f : p.scale_log2;
                if (far) {
                    const uint64_t sc2 = pack2(sc, sc), far2 = pack2(bias_far, bias_far);
#pragma unroll
                    for (int c = 0; c < FP_HALF; c += 2) unpack2(fma2(pack2(s[c], s[c + 1]), sc2, far2), s[c], s[c + 1]);
                } else {
                    const float* at = bt + lane + FP_HALF - 1;
#pragma unroll
                    for (int c = 0; c < FP_HALF; ++c) s[c] = fmaf(s[c], sc, at[-c]);
                }
            }
            if (partial) {
#pragma unroll
                for (int c = 0; c < FP_HALF; ++c)
                    if (c > hi_c || c < lo_c) s[c] = -INFINITY;
            }
            if constexpr (CAP != FP_CAP_BOUND) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < FP_HALF; c += 2) mx[(c >> 1) & 3] = max3(mx[(c >> 1) & 3], s[c], s[c + 1]);
                const float own = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                const float mn = fmaxf(m, fmaxf(own, partner(own)));
                if (it == 0) {
                    m = mn;
                } else if (__any_sync(FULL, (mn - m) * cc > FP_RESCALE)) {      // the same for both warps of the rows
                    // the scores of this tile were issued after the previous tile's P V, so O is complete
                    const float f = mn == -INFINITY ? 1.f : exp2_fast((m - mn) * cc);
                    l *= f;
                    m = mn;
                    for (int c = half * FP_HALF; c < p.dv && c < (half + 1) * FP_HALF; c += 32) {
                        uint32_t r[32];
                        tmem_ld32(o_addr + c, r);
#pragma unroll
                        for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * f);
                        tmem_st32(o_addr + c, r);
                    }
                }
            }
            const float mc = m == -INFINITY ? 0.f : m * cc;
            const uint64_t scale2 = pack2(cc, cc), shift2 = pack2(-mc, -mc);
            uint64_t ls[2] = {0, 0};
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                uint32_t w[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    float x = s[part * 32 + 2 * c], y = s[part * 32 + 2 * c + 1];
                    if (CAP != FP_CAP_BOUND) unpack2(fma2(pack2(x, y), scale2, shift2), x, y);
                    x = exp2_fast(x);
                    y = exp2_fast(y);
                    ls[c & 1] = add2(ls[c & 1], pack2(x, y));
                    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
                    w[c] = *reinterpret_cast<const uint32_t*>(&v);
                }
                tmem_st16(s_addr + part * 16, w);
            }
            float l0, l1;
            unpack2(add2(ls[0], ls[1]), l0, l1);
            l += l0 + l1;
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.p_full[t]);
        }
        if (end[t] > 0) {
            if (ok) ok = __all_sync(FULL, mbar_wait_bounded(&sh.o_full[t], 0));
            const float other = partner(l);
            l = half == 0 ? l + other : other + l;
            if (ok) {
                tc_fence_after();
                const float mc = m == -INFINITY ? 0.f : m * cc;
                if (p.sink != nullptr) l += exp2f(p.sink[h] * FP_LOG2E - mc);
                const float inv = 1.f / l;
                const int row = q0 + t * FP_TILE + a;
                __nv_bfloat16* o = (__nv_bfloat16*)p.out + (int64_t)b * p.o_bs + (int64_t)row * p.o_ss + h * p.o_hs;
                for (int c = half * FP_HALF; c < p.dv && c < (half + 1) * FP_HALF; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(o_addr + c, r);
                    if (row < p.S) {
#pragma unroll
                        for (int e = 0; e < 32; e += 8) {
                            if (c + e < p.dv) {
                                uint32_t w[4];
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[e + 2 * k]) * inv,
                                                                                   __uint_as_float(r[e + 2 * k + 1]) * inv);
                                    w[k] = *reinterpret_cast<const uint32_t*>(&v);
                                }
                                *reinterpret_cast<uint4*>(o + c + e) = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        }
                    }
                }
            }
        }
        if (!ok) *failed = 1;
        tc_fence_before();
    }
    __syncthreads();
    if (tid == 0 && sh.failed && p.status != nullptr) atomicOr(p.status, SK_DEV_WAIT_TIMEOUT);
    if (warp == FP_MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// Stages of the two rings and the dynamic shared memory they take; 0 bytes when the shape does not fit
uint32_t plan_smem(int dqk, int dv, bool bias, int* nk, int* nv) {
    const uint32_t np = (dqk + 63) / 64, nvp = (dv + 63) / 64, extra = bias ? FP_BIAS_BYTES : 0;
    const int plans[3][2] = {{2, 2}, {2, 1}, {1, 1}};
    for (auto& pl : plans) {
        const uint32_t bytes = ((2 + pl[0]) * np + pl[1] * nvp) * FP_PANEL + extra + (uint32_t)sizeof(FpShared);
        if (bytes <= FP_SMEM_LIMIT) {
            *nk = pl[0];
            *nv = pl[1];
            return FP_SMEM_LIMIT - bytes < 1008 ? FP_SMEM_LIMIT : bytes + 1008;
        }
    }
    return 0;
}

}  // namespace

bool attn_prefill_tc_applicable(const sk_attn_params& p) {
    int nk, nv;
    return p.dtype == SK_BF16 && p.pos == nullptr && !p.ring && p.dv <= 128 && p.dqk <= 256 && p.scale > 0.f &&
           p.start >= p.kv_start && p.kv_rows < (int64_t)1 << 30 && head_map_ok(p.q, p.dqk, p.q_hs, p.q_ss, p.q_bs) &&
           head_map_ok(p.k, p.dqk, p.k_hs, p.k_ts, p.k_bs) && head_map_ok(p.v, p.dv, p.v_hs, p.v_ts, p.v_bs) &&
           head_map_ok(p.out, p.dv, p.o_hs, p.o_ss, p.o_bs) && plan_smem(p.dqk, p.dv, p.bias != nullptr, &nk, &nv) > 0;
}

int launch_attn_prefill_tc(const sk_attn_params& p, cudaStream_t st) {
    FpShape f;
    f.out = p.out;
    f.bias = p.bias;
    f.sink = p.sink;
    f.status = p.status;
    f.o_bs = p.o_bs;
    f.o_ss = p.o_ss;
    f.o_hs = p.o_hs;
    f.start = p.start;
    f.kv_start = p.kv_start;
    f.bias_len = p.bias_len;
    f.S = p.S;
    f.H = p.H;
    f.G = p.G;
    f.dqk = p.dqk;
    f.dv = p.dv;
    f.chunk = p.chunk;
    f.window = p.window;
    f.scale_log2 = p.scale * FP_LOG2E;
    f.cap_in = p.softcap > 0.f ? p.scale / p.softcap : 0.f;
    f.cap_out = p.softcap * FP_LOG2E;
    double c = p.scale * 1.4426950408889634, c2 = (double)f.cap_in * f.cap_in;
    for (int k = 0; k < 5; ++k, c *= c2) f.cap_poly[k] = (float)(TANH_POLY[k] * c);
    f.cap_small = f.cap_in > 0.f ? (TANH_POLY_RANGE / f.cap_in) * (TANH_POLY_RANGE / f.cap_in) : 0.f;
    const uint32_t smem = plan_smem(p.dqk, p.dv, p.bias != nullptr, &f.nk, &f.nv);
    CUtensorMap mq, mk, mv;
    if (int rc = make_head_map(&mq, p.q, p.dqk, p.H, p.S, p.B, p.q_hs, p.q_ss, p.q_bs, FP_TILE)) return rc;
    if (int rc = make_head_map(&mk, p.k, p.dqk, p.G, p.kv_rows, p.B, p.k_hs, p.k_ts, p.k_bs, FP_TILE)) return rc;
    if (int rc = make_head_map(&mv, p.v, p.dv, p.G, p.kv_rows, p.B, p.v_hs, p.v_ts, p.v_bs, FP_TILE)) return rc;
    auto kern = p.bias != nullptr ? attn_prefill_kernel<true, FP_CAP_NONE> : attn_prefill_kernel<false, FP_CAP_NONE>;
    if (p.softcap > 0.f)
        kern = p.bias != nullptr ? attn_prefill_kernel<true, FP_CAP>
                                 : (f.cap_out <= FP_CAP_BOUND_LOG2 ? attn_prefill_kernel<false, FP_CAP_BOUND> : attn_prefill_kernel<false, FP_CAP>);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(SK_ERR_CUDA, "attn_prefill_kernel smem attribute: %s", cudaGetErrorString(e));
    f.q_blocks = (p.S + 2 * FP_TILE - 1) / (2 * FP_TILE);
    dim3 grid((unsigned)(p.H * f.q_blocks), (unsigned)p.B);
    kern<<<grid, FP_THREADS, smem, st>>>(mq, mk, mv, f);
    return check_launch("attn_prefill_kernel");
}

}  // namespace sk
