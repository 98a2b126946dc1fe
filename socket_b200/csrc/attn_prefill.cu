// Softmax attention of a prompt portion on the 5th-generation tensor cores (bf16).
//
// A CTA owns 256 consecutive queries of one head as two tiles of 128.  One warp feeds 128-key tiles of K
// and V by TMA (128-byte swizzle), one warp issues the MMAs: S = Q K^T into tensor memory (fp32,
// shared-memory operands), O += P V with P read from tensor memory.  The softmax threads of a query row scale / bias / mask
// its scores, keep the running maximum and their sum, and write the weights back over the scores as bf16, in two parts: the
// MMAs of the first run beside the exponentials of the second.  While one tile is in its softmax the tensor core works on
// the other.  The accumulator is rescaled only when a row's maximum has grown by more than 2^8 since the last time (the
// final division by the sum makes the choice of reference invisible); so the first weights of a tile are taken relative to
// the last reference before the tile's maximum is known, and taken again in the rare case.  Scores under a low cap are
// bounded, so their weights are taken relative to zero: no maximum, no rescaling.
//
// Visibility is causal, optionally restricted to the query's own chunk of positions or to a sliding window; tiles
// that no row of a query tile can see are not visited.  Out-of-range rows and columns of a tile are zero-filled by TMA.
// Every wait is bounded; one that runs out makes all roles leave, and is reported in the status word.
//
// Bound: a tile's chain - scores, exponentials, the product of the last weights - against 2 x 1024 cycles of MMAs for two
// tiles of 128 / 128; a plain causal pair takes 3050, with the clock below its maximum under the power limit.  Measured,
// one GPU, L2 flushed (in brackets: two threads per row for every form, K asked for together with V, 270 bytes a thread
// spilled by the roles of 32 registers): 8000 tokens, 32 / 8 heads of 128, chunk and bias 473 us (551); 32 heads of 192 /
// 128 with sinks 532 us (684); 32000 tokens, 16 heads, window 4096 and cap 1016 us (1151); 8000 tokens, 16 heads 224 us
// (265), with a cap of 100 302 us (349), with cap and bias 328 us (387); 1501 tokens behind 2500, 16 heads, bias 76 us (86).
#include "blocks.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace sk {
namespace {

constexpr int FP_TILE = 128;                                  // queries of a tile = keys of a tile
// PER: softmax threads of a query row.  One, with all 128 scores in its registers, needs no exchange between threads; two do the
// arithmetic of a cap (six packed operations a pair of scores) on twice the warps: 32000 tokens, window and low cap 1016 us with two, 1065
// with one; 8000 tokens, 16 heads without a cap 224 us with one, 242 with two.
template <int PER> struct FpRoles {
    static constexpr int KEYS = FP_TILE / PER;                // keys of a softmax thread
    static constexpr int SOFTMAX_WARPS = 8 * PER;             // warp: 4 PER tile + 4 part of the keys + quarter of the rows
    static constexpr int TMA_WARP = SOFTMAX_WARPS, MMA_WARP = TMA_WARP + 1;
    static constexpr int THREADS = 32 * (SOFTMAX_WARPS + 4);  // the last two warps idle: registers are dealt to groups of four
    // Registers a thread at launch, and dealt out again: 384 x 168 = 256 x 216 + 128 x 72, 640 x 96 = 512 x 112 + 128 x 32
    static constexpr int REGS_SOFTMAX = PER == 1 ? 216 : 112, REGS_OTHER = PER == 1 ? 72 : 32;
    static constexpr int BIAS_SPAN = KEYS + 32;               // distances a warp's 32 rows and its keys can have
    static constexpr uint32_t BIAS_BYTES = SOFTMAX_WARPS * BIAS_SPAN * sizeof(float);
};
constexpr uint32_t FP_PANEL = FP_TILE * 128;                  // 128 rows x 64 bf16
constexpr float FP_RESCALE = 8.f;                             // log2 units
constexpr float FP_LOG2E = 1.4426950408889634f;

struct FpShared {
    uint64_t q_full[2];
    uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
    uint64_t s_full[2], p_full[2][2], o_full[2];
    uint64_t drained;
    uint32_t tmem_base;
    int failed;
    float xch[FP_TILE * 4];                  // what the threads of a row, or the CTAs of a block, tell each other
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
__host__ __device__ __forceinline__ int fp_first_row(const FpShape& p, int i) {
    int64_t lo = -p.kv_start;
    if (p.chunk > 0) lo = position_div(i + p.kv_start, p.chunk) * p.chunk - p.kv_start;
    if (p.window > 0 && i - p.window + 1 > lo) lo = i - p.window + 1;
    return (int)(lo > 0 ? lo : 0);
}
// the range [beg, end) of key tiles that each of the two query tiles from query q0 on visits; tiles count from key row `base`
__host__ __device__ __forceinline__ void fp_tiles(const FpShape& p, int q0, int (&i0)[2], int (&beg)[2], int (&end)[2], int& base) {
    base = 0;
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
}
__device__ __forceinline__ float4 load_cta(const void* local, int rank) {      // shared memory of the cluster's CTA `rank`, in its place here
    uint32_t at;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr(local)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    return v;
}
__device__ __forceinline__ float load_cta1(const void* local, int rank) {
    uint32_t at;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}

// s <- cap_out tanh(s cap_in): two small scores
__device__ __forceinline__ void fp_cap_pair(const FpShape& p, float& a, float& b) {
    const uint64_t x = pack2(a, b), t = mul2(x, x);
    uint64_t r = fma2(t, pack2(p.cap_poly[4], p.cap_poly[4]), pack2(p.cap_poly[3], p.cap_poly[3]));
    r = fma2(t, r, pack2(p.cap_poly[2], p.cap_poly[2]));
    r = fma2(t, r, pack2(p.cap_poly[1], p.cap_poly[1]));
    r = fma2(t, r, pack2(p.cap_poly[0], p.cap_poly[0]));
    unpack2(mul2(r, x), a, b);
}
// 16 scores from c0 on; the caller's loops are unrolled
template <int N> __device__ __forceinline__ void fp_cap16(const FpShape& p, float (&s)[N], int c0) {
    float top[2] = {0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 16; c += 2) top[(c >> 1) & 1] = max3_abs(top[(c >> 1) & 1], s[c0 + c], s[c0 + c + 1]);
    const float all = fmaxf(top[0], top[1]);
    if (__any_sync(FULL, !(all * all <= p.cap_small))) {
#pragma unroll
        for (int c = 0; c < 16; ++c) s[c0 + c] = p.cap_out * tanh_exp2(s[c0 + c] * p.cap_in);
    } else {
#pragma unroll
        for (int c = 0; c < 16; c += 2) fp_cap_pair(p, s[c0 + c], s[c0 + c + 1]);
    }
}

// the same for all of a thread's scores: as a rule all are small, and one vote says so
template <int N> __device__ __forceinline__ void fp_cap_all(const FpShape& p, float (&s)[N]) {
    float top[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < N; c += 2) top[(c >> 1) & 3] = max3_abs(top[(c >> 1) & 3], s[c], s[c + 1]);
    const float all = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
    if (__all_sync(FULL, all * all <= p.cap_small)) {
#pragma unroll
        for (int c = 0; c < N; c += 2) fp_cap_pair(p, s[c], s[c + 1]);
    } else {
#pragma unroll
        for (int c = 0; c < N; c += 16) fp_cap16(p, s, c);
    }
}

// SPLIT: CTAs, a cluster, that share a block's keys
template <bool BIAS, int CAP, int PER, int SPLIT>
__global__ void __launch_bounds__(FpRoles<PER>::THREADS, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const FpShape p) {
    using Roles = FpRoles<PER>;
    constexpr int KEYS = Roles::KEYS, BIAS_SPAN = Roles::BIAS_SPAN;
    extern __shared__ __align__(1024) char fp_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(fp_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // heads side by side, long rows first: the last blocks to start are short ones.  (Heads in groups whose keys and values fit
    // the L2 end in a short group of long rows: 24000 tokens, 16 heads of 192 / 128 in groups of 3: 2975 us, so 2643; 8000
    // tokens, 32 heads in groups of 9: 699 us, so 677.  16000 tokens, 16 heads were 1177 us in groups and are 1207 so.)
    const int unit = blockIdx.x / SPLIT, rank = blockIdx.x % SPLIT;
    const int b = blockIdx.y, back = unit / p.H, h = unit - back * p.H, g = h / (p.H / p.G);
    const int np = (p.dqk + 63) / 64, nvp = (p.dv + 63) / 64;
    char* q_s = tiles;                                        // [tile][panel]
    char* k_s = q_s + 2 * np * FP_PANEL;                      // [stage][panel]
    char* v_s = k_s + p.nk * np * FP_PANEL;
    float* bias_s = reinterpret_cast<float*>(v_s + p.nv * nvp * FP_PANEL);
    FpShared& sh = *reinterpret_cast<FpShared*>(reinterpret_cast<char*>(bias_s) + (BIAS ? Roles::BIAS_BYTES : 0));

    // query tiles, and the range [beg, end) of key tiles each of them visits; key rows count from kv_start
    const int q0 = (p.q_blocks - 1 - back) * 2 * FP_TILE;
    int i0[2], beg[2], end[2], base;                          // rows of a call: below 2^30
    fp_tiles(p, q0, i0, beg, end, base);
    int n = end[1] > end[0] ? end[1] : end[0];
    if constexpr (SPLIT > 1) {                                        // this CTA's share of them
        const int first = n * rank / SPLIT;
        n = n * (rank + 1) / SPLIT - first;
        base += first * FP_TILE;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            beg[t] = max(beg[t] - first, 0);
            end[t] = min(end[t] - first, n);
            if (end[t] <= beg[t]) beg[t] = end[t] = 0;
        }
    }
    // all threads of the cluster, warp by warp
    auto meet = [] {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    };
    uint32_t room;                                            // the tiles end inside what was launched, wherever shared memory begins
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(room));
    const uint32_t used = (uint32_t)((char*)(&sh + 1) - fp_raw);
    if (used > room) {
        if (tid == 0 && p.status != nullptr) atomicOr(p.status, SK_DEV_WAIT_TIMEOUT);
        return;
    }

    const uint32_t k_bytes = np * FP_PANEL, v_bytes = nvp * FP_PANEL;
    auto load_q = [&](int t) {
        mbar_expect(&sh.q_full[t], k_bytes);
        for (int c = 0; c < np; ++c)
            tma_load_4d(q_s + (t * np + c) * FP_PANEL, &map_q, c * 64, h, q0 + t * FP_TILE, b, &sh.q_full[t]);
    };
    auto load_k = [&](int k) {
        const int ks = k % p.nk;
        mbar_expect(&sh.k_full[ks], k_bytes);
        for (int c = 0; c < np; ++c)
            tma_load_4d(k_s + (ks * np + c) * FP_PANEL, &map_k, c * 64, g, base + k * FP_TILE, b, &sh.k_full[ks]);
    };
    if (warp == Roles::TMA_WARP && lane == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init_count(&sh.q_full[s], 1);
            mbar_init_count(&sh.k_full[s], 1);
            mbar_init_count(&sh.k_empty[s], 1);
            mbar_init_count(&sh.v_full[s], 1);
            mbar_init_count(&sh.v_empty[s], 1);
            mbar_init_count(&sh.s_full[s], 1);
            mbar_init_count(&sh.p_full[s][0], 4 * PER);
            mbar_init_count(&sh.p_full[s][1], 4 * PER);
            mbar_init_count(&sh.o_full[s], 1);
        }
        mbar_init_count(&sh.drained, 1);
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        load_q(0);                                            // on their way while the block assembles
        load_k(0);
        load_q(1);
    }
    if (warp == Roles::MMA_WARP) {
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

    if (warp >= Roles::SOFTMAX_WARPS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Roles::REGS_OTHER));
    if (warp == Roles::TMA_WARP) {
        // ---- TMA producer
        if (lane == 0) {
            int k = 1, v = 0;                                 // tiles of K and V sent
            while (v < n && !*failed) {
                // K leads by its ring: its stage is free when a tile's scores are done, which is before V's is
                if (k < n && k < v + p.nk) {
                    const int ks = k % p.nk;
                    if (k >= p.nk && !mbar_wait_bounded(&sh.k_empty[ks], (uint32_t)((k / p.nk - 1) & 1))) { *failed = 1; break; }
                    load_k(k++);
                } else {
                    const int vs = v % p.nv;
                    if (v >= p.nv && !mbar_wait_bounded(&sh.v_empty[vs], (uint32_t)((v / p.nv - 1) & 1))) { *failed = 1; break; }
                    mbar_expect(&sh.v_full[vs], v_bytes);
                    for (int c = 0; c < nvp; ++c)
                        tma_load_4d(v_s + (vs * nvp + c) * FP_PANEL, &map_v, c * 64, g, base + v * FP_TILE, b, &sh.v_full[vs]);
                    ++v;
                }
            }
            if (*failed) {                                    // leave no copy in flight
                for (int t = 0; t < 2; ++t) mbar_wait_bounded(&sh.q_full[t], 0);
                for (int i = k > p.nk ? k - p.nk : 0; i < k; ++i)
                    mbar_wait_bounded(&sh.k_full[i % p.nk], (uint32_t)((i / p.nk) & 1));
                for (int i = v > p.nv ? v - p.nv : 0; i < v; ++i)
                    mbar_wait_bounded(&sh.v_full[i % p.nv], (uint32_t)((i / p.nv) & 1));
            }
        }
        if constexpr (SPLIT > 1) {
            meet();
            meet();
        }
    } else if (warp == Roles::MMA_WARP) {
        // ---- MMA issuer.  The whole warp walks the tiles and waits, one lane issues: operands then are warp-uniform, and an
        // MMA costs an addition per descriptor (built in one lane's loop, each took about 200 cycles to issue and 64 to run)
        const bool leader = elect_one();
        const uint32_t tmem = __shfl_sync(FULL, sh.tmem_base, 0);
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
            if (PER == 1 && k_steps == 8) {                   // (32 registers do not hold the operands of unrolled steps)
#pragma unroll
                for (int k = 0; k < 8; ++k) step(d, qd, kd, k);
            } else if (PER == 1 && k_steps == 12) {
#pragma unroll
                for (int k = 0; k < 12; ++k) step(d, qd, kd, k);
            } else {
#pragma unroll 4
                for (int k = 0; k < k_steps; ++k) step(d, qd, kd, k);
            }
            umma_commit_by(leader, &sh.s_full[t]);
        };
        bool ok = wait_all(&sh.k_full[0], 0);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            ok = ok && wait_all(&sh.q_full[t], 0);
            tc_fence_after();
            if (ok && beg[t] == 0 && end[t] > 0) scores(t, 0);
        }
        if (ok) umma_commit_by(leader, &sh.k_empty[0]);
        for (int j = 0; ok && j < n && !__any_sync(FULL, *failed != 0); ++j) {
            const bool more = j + 1 < n;
            if (more) ok = wait_all(&sh.k_full[(j + 1) & k_mask], p.nk == 1 ? (uint32_t)((j + 1) & 1) : (uint32_t)(((j + 1) >> 1) & 1));
            ok = ok && wait_all(&sh.v_full[j & v_mask], p.nv == 1 ? (uint32_t)(j & 1) : (uint32_t)((j >> 1) & 1));
            const uint64_t vd = umma_desc_at(v_desc, (j & v_mask) * v_stage);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (ok && j >= beg[t] && j < end[t]) {
                    // the weights come in two parts, half of each softmax thread's keys: the first is multiplied while the second is computed
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        ok = ok && wait_all(&sh.p_full[t][part], (uint32_t)((j - beg[t]) & 1));
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int k = 0; k < (PER == 2 ? 4 : part == 0 ? 6 : 2); ++k) {
                            // 16 keys; a softmax thread's weights begin where its scores did
                            const int ks = PER == 1 ? part * 6 + k : (k >> 1) * 4 + part * 2 + (k & 1);
                            umma_ts_by(leader, tmem + 2 * FP_TILE + t * FP_TILE, tmem + t * FP_TILE + (PER == 1 ? ks * 8 : (ks >> 2) * KEYS + (ks & 3) * 8),
                                       umma_desc_at(vd, ks * (2048 >> 4)), idesc_o, part > 0 || k > 0 || j > beg[t]);
                        }
                    }
                    if (ok && j + 1 == end[t]) umma_commit_by(leader, &sh.o_full[t]);
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
        if constexpr (SPLIT > 1) {
            meet();
            meet();
        }
    } else if (warp < Roles::SOFTMAX_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Roles::REGS_SOFTMAX));
        // ---- softmax
        const int t = warp / (4 * PER), half = PER == 1 ? 0 : (warp >> 2) & 1, quad = warp & 3, a = quad * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        // a thread's weights go over the first columns of its own scores
        const uint32_t s_addr = tmem + lane_base + t * FP_TILE + half * KEYS;
        const uint32_t o_addr = tmem + lane_base + 2 * FP_TILE + t * FP_TILE;
        const int i = i0[t] + a;                              // query row in key-row coordinates
        const float sc = CAP != FP_CAP_NONE ? 1.f : p.scale_log2;            // log2 units per unit of s below
        const int lo_row = fp_first_row(p, i), lo_last = fp_first_row(p, i0[t] + quad * 32 + 31);
        float* bt = bias_s + warp * BIAS_SPAN;
        const float* bias_h = BIAS ? p.bias + (int64_t)h * p.bias_len : nullptr;
        const int bias_last = (int)(p.bias_len < (1 << 30) ? p.bias_len : 1 << 30) - 1;
        // this warp's distances in tile j: row - key = bias_first(j) + 0 .. KEYS + 30
        auto bias_first = [&](int j) { return i0[t] + quad * 32 - (base + j * FP_TILE + half * KEYS) - (KEYS - 1); };
        auto bias_at = [&](int d) { return __ldg(bias_h + min(max(d, 0), bias_last)) * FP_LOG2E; };
        float bias_next[BIAS_SPAN / 32], bias_far = 0.f;   // requested a tile ahead
        if (BIAS && end[t] > 0) {
            bias_far = bias_at(bias_last);
#pragma unroll
            for (int e = 0; e < BIAS_SPAN / 32; ++e) bias_next[e] = bias_at(bias_first(beg[t]) + lane + 32 * e);
        }
        float m = CAP == FP_CAP_BOUND ? 0.f : -INFINITY, l = 0.f;
        bool ok = true;                                       // a wait that ran out: no more waits, the rest runs through
        for (int j = beg[t]; j < end[t]; ++j) {
            const int it = j - beg[t];
            const int r0 = base + j * FP_TILE + half * KEYS;
            bool far = false;                                 // every distance is beyond the table
            if (BIAS) {
                far = bias_first(j) >= bias_last;
                if (!far) {
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < BIAS_SPAN / 32; ++e) bt[lane + 32 * e] = bias_next[e];
                    __syncwarp();
                }
                if (bias_first(j + 1) < bias_last) {
#pragma unroll
                    for (int e = 0; e < BIAS_SPAN / 32; ++e) bias_next[e] = bias_at(bias_first(j + 1) + lane + 32 * e);
                }
            }
            if (ok) ok = __all_sync(FULL, mbar_wait_bounded(&sh.s_full[t], (uint32_t)(it & 1)));
            tc_fence_after();
            const bool partial = r0 + KEYS - 1 > i0[t] + quad * 32 || r0 < lo_last;     // some row does not see all these keys
            const int hi_c = i - r0, lo_c = lo_row - r0;
            // weights: 2^(s * cs + off), in log2 units
            float cs = sc, off = 0.f;
            float s[KEYS];
            if constexpr (PER == 1) {
                tmem_ld64(s_addr, *reinterpret_cast<uint32_t(*)[64]>(s));
                tmem_ld64(s_addr + 64, *reinterpret_cast<uint32_t(*)[64]>(s + 64));
            } else {
                tmem_ld64(s_addr, reinterpret_cast<uint32_t(&)[KEYS]>(s));
            }
            if (CAP != FP_CAP_NONE) fp_cap_all(p, s);
            if (BIAS) {
                if (far) {
                    off = bias_far;
                } else {
                    const float* at = bt + lane + KEYS - 1;
#pragma unroll
                    for (int c = 0; c < KEYS; ++c) s[c] = fmaf(s[c], sc, at[-c]);
                    cs = 1.f;
                }
            }
            if (partial) {
#pragma unroll
                for (int c = 0; c < KEYS; ++c)
                    if (c > hi_c || c < lo_c) s[c] = -INFINITY;
            }
            uint64_t ls[2];
            // the weights of one half of the keys, relative to 2^ref, and their sum
            auto weights = [&](int part, float ref) {
                const uint64_t scale2 = pack2(cs, cs), shift2 = pack2(off - ref, off - ref);
#pragma unroll
                for (int q = 0; q < (PER == 1 && part == 0 ? 2 : 1); ++q) {
                    const int c0 = part * 32 + q * 32;
                    uint32_t w[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        float x = s[c0 + 2 * c], y = s[c0 + 2 * c + 1];
                        if (CAP != FP_CAP_BOUND) unpack2(fma2(pack2(x, y), scale2, shift2), x, y);
                        x = exp2_fast(x);
                        y = exp2_fast(y);
                        ls[c & 1] = add2(ls[c & 1], pack2(x, y));
                        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
                        w[c] = *reinterpret_cast<const uint32_t*>(&v);
                    }
                    tmem_st16(s_addr + c0 / 2, w);
                }
            };
            auto publish = [&](int part) {
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.p_full[t][part]);
            };
            // The first weights are taken relative to the reference that the tiles before have left, beside the search for
            // the maximum; where that is too low, they are taken again.
            const float ref = m == -INFINITY ? 0.f : m;
            ls[0] = ls[1] = 0;
            weights(0, ref);
            if constexpr (CAP != FP_CAP_BOUND) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < KEYS; c += 2) mx[(c >> 1) & 3] = max3(mx[(c >> 1) & 3], s[c], s[c + 1]);
                const float own = fmaf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), cs, off);
                if (__any_sync(FULL, own - m > FP_RESCALE)) {
                    const float mn = fmaxf(m, own), f = exp2_fast(m - mn);      // not -inf in one of the lanes; NaN or 1 where m is
                    if (it > 0) {
                        // the scores of this tile were issued after the previous tile's P V, so O is complete
                        l *= mn == -INFINITY ? 1.f : f;
                        for (int c = 0; c < p.dv; c += 32) {
                            uint32_t r[32];
                            tmem_ld32(o_addr + c, r);
#pragma unroll
                            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * (mn == -INFINITY ? 1.f : f));
                            tmem_st32(o_addr + c, r);
                        }
                    }
                    m = mn;
                    ls[0] = ls[1] = 0;
                    tmem_wait_st();                           // the first weights are in place, and so replaced
                    weights(0, m == -INFINITY ? 0.f : m);
                }
            }
            const float ref1 = m == -INFINITY ? 0.f : m;
            if (PER == 1) {
                weights(2, ref1);
                publish(0);
                weights(3, ref1);
            } else {
                publish(0);
                weights(1, ref1);
            }
            publish(1);
            float l0, l1;
            unpack2(add2(ls[0], ls[1]), l0, l1);
            l += l0 + l1;
        }
        if constexpr (SPLIT > 1) {
            // ---- the CTAs' parts of a block: each leaves its sums and unscaled rows of O where its operands were (no product
            // is in flight any more), then takes every SPLIT-th row of all of them
            const int pitch = nvp * 64, row = t * FP_TILE + a;               // floats of a row, 16-byte pieces permuted
            float* rows = reinterpret_cast<float*>(tiles);
            ok = __all_sync(FULL, mbar_wait_bounded(&sh.drained, 0)) && ok;
            sh.xch[PER == 1 ? row : half * 2 * FP_TILE + row] = PER == 1 ? m : l;
            if (PER == 1) sh.xch[2 * FP_TILE + row] = l;
            if (ok && end[t] > 0) {
                tc_fence_after();
                for (int c = half * KEYS; c < p.dv && c < (half + 1) * KEYS; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(o_addr + c, r);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        *reinterpret_cast<uint4*>(rows + row * pitch + (((c >> 2) + e) ^ (row & 7)) * 4) =
                            make_uint4(r[4 * e], r[4 * e + 1], r[4 * e + 2], r[4 * e + 3]);
                }
            }
            meet();
            {
                constexpr int N = SPLIT;
                float wt[N], sum[N], top = -INFINITY, total = 0.f;
                uint32_t seen = 0;                            // parts with visible keys; the others have no rows either
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    wt[q] = load_cta1(&sh.xch[row], q);
                    sum[q] = load_cta1(&sh.xch[2 * FP_TILE + row], q);
                }
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    if (PER == 2) {
                        sum[q] += wt[q];
                        wt[q] = 0.f;
                    }
                    if (sum[q] != 0.f) {
                        seen |= 1u << q;
                        wt[q] = fmaxf(wt[q], -3.0e38f);       // of NaN alone there is no maximum, but a sum
                        top = fmaxf(top, wt[q]);
                    }
                }
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    wt[q] = seen >> q & 1 ? exp2_fast(wt[q] - top) : 0.f;
                    total = fmaf(wt[q], sum[q], total);
                }
                if (p.sink != nullptr) total += exp2f(p.sink[h] * FP_LOG2E - top);
                const float inv = 1.f / total;
                // a row at a time, its columns along the lanes: another CTA's memory is read in whole rows, four of them requested together
                constexpr int STEP = N * PER, U = 4;
                for (int e0 = rank + (PER == 1 ? 0 : half * N); e0 < 32; e0 += STEP * U) {
                    float4 x[U][N];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int r1 = row - lane + ((e0 + u * STEP) & 31);
#pragma unroll
                        for (int q = 0; q < N; ++q) x[u][q] = load_cta(rows + r1 * pitch + (((lane * 4 < pitch ? lane : 0)) ^ (r1 & 7)) * 4, q);
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int e = e0 + u * STEP, s_row = q0 + row - lane + e;
                        const float inv1 = __shfl_sync(FULL, inv, e & 31);
                        const uint32_t seen1 = __shfl_sync(FULL, seen, e & 31);
                        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int q = 0; q < N; ++q) {
                            const float w = __shfl_sync(FULL, wt[q], e & 31);
                            if (seen1 >> q & 1) {
                                v[0] = fmaf(w, x[u][q].x, v[0]);
                                v[1] = fmaf(w, x[u][q].y, v[1]);
                                v[2] = fmaf(w, x[u][q].z, v[2]);
                                v[3] = fmaf(w, x[u][q].w, v[3]);
                            }
                        }
                        if (e < 32 && s_row < p.S && lane * 4 < p.dv) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) v[k] *= inv1;
                            store_vec<__nv_bfloat16, 4>((__nv_bfloat16*)p.out + (int64_t)b * p.o_bs + (int64_t)s_row * p.o_ss + h * p.o_hs + lane * 4, v);
                        }
                    }
                }
            }
            meet();                                           // nobody leaves while its rows are read
        } else if (end[t] > 0) {
            if (ok) ok = __all_sync(FULL, mbar_wait_bounded(&sh.o_full[t], 0));
            if (PER == 2) {                                   // the sum of both threads of a row
                sh.xch[warp * 32 + lane] = l;
                asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quad) : "memory");
                const float other = sh.xch[(warp ^ 4) * 32 + lane];
                l = half == 0 ? l + other : other + l;
            }
            if (ok) {
                tc_fence_after();
                const float mc = m == -INFINITY ? 0.f : m;
                if (p.sink != nullptr) l += exp2f(p.sink[h] * FP_LOG2E - mc);
                const float inv = 1.f / l;
                const int row = q0 + t * FP_TILE + a;
                __nv_bfloat16* o = (__nv_bfloat16*)p.out + (int64_t)b * p.o_bs + (int64_t)row * p.o_ss + h * p.o_hs;
                for (int c = half * KEYS; c < p.dv && c < (half + 1) * KEYS; c += 32) {
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
    } else if (SPLIT > 1) {
        meet();
        meet();
    }
    __syncthreads();
    if (tid == 0 && sh.failed && p.status != nullptr) atomicOr(p.status, SK_DEV_WAIT_TIMEOUT);
    if (warp == Roles::MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// Stages of the two rings and the dynamic shared memory they take; 0 bytes when the shape does not fit
uint32_t plan_smem(int dqk, int dv, bool bias, int* nk, int* nv) {
    const uint32_t np = (dqk + 63) / 64, nvp = (dv + 63) / 64, extra = bias ? FpRoles<1>::BIAS_BYTES : 0;
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

// CTAs that share a block's keys.  A call of few blocks leaves most SMs idle while its blocks walk over all keys: where two or four CTAs
// a block find a place at once, they share it: half as many pairs as there are SMs do, and two clusters of four for nine SMs (33 on 148, as
// each GPC may leave some SMs over).  What joining costs shows where they don't: 8000
// tokens, 16 heads are 512 blocks, 222 us alone, 266 by pairs, 401 by fours.  By the longest block's key tiles (one CTA | two | four):
// 28 tiles, 32 blocks 65 | 45 | 35 us; 35 tiles of 192 / 128, 64 blocks 82 | 55 us; 16 tiles under a cap, 64 blocks 47 | 34 us; 6 tiles of
// 256 / 128, 24 blocks 28.7 | 22.5 | 22.5 us.
int fp_split(const FpShape& f, int B) {
    const int64_t blocks = (int64_t)B * f.H * f.q_blocks, sms = sm_count();
    const int np = (f.dqk + 63) / 64, nvp = (f.dv + 63) / 64;
    if (2 * blocks > sms || (2 + f.nk) * np + f.nv * nvp < 4 * nvp) return 1;             // O's rows take the operands' place
    int most = 0;
    for (int k = 0; k < f.q_blocks; ++k) {
        int i0[2], beg[2], end[2], base;
        fp_tiles(f, k * 2 * FP_TILE, i0, beg, end, base);
        for (int e : end) most = e > most ? e : most;
    }
    return most < 6 ? 1 : most < 16 || 9 * blocks > 2 * sms ? 2 : 4;
}

template <int SPLIT> auto fp_kernel(bool bias, float softcap, bool bound) {
    if (softcap > 0.f)
        return bias ? attn_prefill_kernel<true, FP_CAP, 1, SPLIT>
                    : bound ? attn_prefill_kernel<false, FP_CAP_BOUND, 2, SPLIT> : attn_prefill_kernel<false, FP_CAP, 1, SPLIT>;
    return bias ? attn_prefill_kernel<true, FP_CAP_NONE, 1, SPLIT> : attn_prefill_kernel<false, FP_CAP_NONE, 1, SPLIT>;
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
    const bool bound = p.softcap > 0.f && p.bias == nullptr && f.cap_out <= FP_CAP_BOUND_LOG2;
    f.q_blocks = (p.S + 2 * FP_TILE - 1) / (2 * FP_TILE);
    const int split = fp_split(f, p.B);
    const auto kern = split == 1 ? fp_kernel<1>(p.bias != nullptr, p.softcap, bound)
                    : split == 2 ? fp_kernel<2>(p.bias != nullptr, p.softcap, bound) : fp_kernel<4>(p.bias != nullptr, p.softcap, bound);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(SK_ERR_CUDA, "attn_prefill_kernel smem attribute: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.H * f.q_blocks * split), (unsigned)p.B);
    cfg.blockDim = dim3(bound ? FpRoles<2>::THREADS : FpRoles<1>::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = split > 1 ? 1 : 0;
    return check_chained(cudaLaunchKernelEx(&cfg, kern, mq, mk, mv, f), "attn_prefill_kernel");
}

}  // namespace sk
