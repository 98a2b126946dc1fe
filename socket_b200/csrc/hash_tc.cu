// Bulk key hashing and bulk cache writes on the 5th-generation tensor cores (prefill: thousands of rows, 16-bit keys).
//
// codes = sign( K[N,128] . planes^T[128, L*P = 256] ) packed 8 planes -> one byte per table.
// Persistent CTAs, one per SM, walk the 128-row tiles of K.  The 256 plane rows stay in shared
// memory; TMA (cp.async.bulk.tensor, 128-byte swizzle) feeds a ring of K tiles, one elected thread
// issues eight tcgen05.mma.kind::f16 (M=128, N=256, K=16) per tile into one of two fp32
// accumulators in tensor memory, and the epilogue warps (sixteen, four threads per row; eight and two
// with APPEND) read the other accumulator back with tcgen05.ld, take the signs and write 32 code bytes
// per row, so loading, multiplying and the epilogue of consecutive tiles overlap.
//
// The same kernel with APPEND writes the rest of a cache append: eight warps move K (from the tile in
// shared memory) and V (straight through registers) to their cache rows and take ||v||, so K is read
// once and an append of bf16 or fp16 rows is one launch.  Its floor is memory, 1 KiB read and written per
// row.  Measured: 8192 tokens of 8 heads, bf16, 26 us, where six launches took 56 (copy 21, hash 16, exact
// decisions 9, check for too many of them 6, cache rows and counter 4), fp16 28 us, where the exact kernel
// took 1857; 384000 rows 98 us (4.1 TB/s), before 200.  What cost most on the way: fp64 sums of ||v||^2 (38 us
// for the 65536 rows) and the roles' unrolled code, 112 KiB, which missed the instruction cache (35 us).
//
// Exactness.  16-bit products are exact in fp32, only the accumulation rounds, so a sign
// can be wrong only when |acc| is tiny compared with |k|.|p|.  Every projection with
// |acc| <= 2^-16 |k| |p| (a bound far above the accumulation error of 128 terms) is marked in a
// bit mask of the tile and decided again from the exact fp64 dot product, which patches the bit: with APPEND
// by the norm warps from the rows in shared memory, without by eight warps of their own that read the key from
// global memory again.  ~1e-4 of the projections (five per tile) take that path, and a mask has room for all of
// them.  Rows of zeros hash to all-ones bytes directly.
#include <cuda.h>

#include "hash_body.cuh"
#include "tcgen05.cuh"

namespace sk {
namespace {

constexpr int TC_ROWS = 128;          // rows of K per CTA (MMA M)
constexpr int TC_N = 256;             // L * P (MMA N)
constexpr int TC_D = 128;             // head dim (MMA K total)
constexpr int TC_KHALF = 64;          // bf16 elements per 128-byte swizzle row
constexpr uint32_t TC_A_HALF_BYTES = TC_ROWS * 128;   // 16 KiB
constexpr uint32_t TC_B_HALF_BYTES = TC_N * 128;      // 32 KiB
constexpr uint32_t TC_PIPE_SMEM = 2 * TC_B_HALF_BYTES + 4 * 2 * TC_A_HALF_BYTES;   // planes + four K tiles: 192 KiB
constexpr int64_t TC_MAX_ROWS = 1 << 24;
constexpr float TC_TINY = 1e-30f;                     // sums of squares below it may have lost terms
constexpr float TC_BAND = 1.52587890625e-05f;         // 2^-16

// kind::f16, A = B of one 16-bit type (K-major), D = fp32, M = 128, N = 256
template <typename T> struct TcType;
template <> struct TcType<__nv_bfloat16> {
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((TC_N >> 3) << 17) | ((TC_ROWS >> 4) << 24);
    static constexpr CUtensorMapDataType MAP = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    static __device__ __forceinline__ float2 pair(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
};
template <> struct TcType<__half> {
    static constexpr uint32_t IDESC = (1u << 4) | ((TC_N >> 3) << 17) | ((TC_ROWS >> 4) << 24);
    static constexpr CUtensorMapDataType MAP = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    static __device__ __forceinline__ float2 pair(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
};

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

constexpr int TC_STAGES = 2;          // accumulators in tensor memory
constexpr int TC_MASKS = 4;           // masks of near-zero projections: tiles whose decisions may be outstanding
constexpr int TC_ARING = 4;           // K tiles in flight
constexpr int TC_NSLOTS = 8;          // norm slots
constexpr int TC_NORM_WARPS = 4;      // one thread per row of the K tile: its norm, and with APPEND later its near-zero projections
// two threads per accumulator row, 128 columns each; four of 64 where no warps move rows
template <bool APPEND> constexpr int TC_EPI_WARPS = APPEND ? 8 : 16;
constexpr int TC_MOVE_WARPS = 8;      // APPEND: 16 rows each
// Without APPEND: one thread per row of every second tile, for its near-zero projections.  Bulk hashing is bound by the tiles' roles, not by
// memory, and decisions take longest: 4194304 rows 638 us by the norm warps, 525 by four warps of their own, 444 with the masks of four
// tiles instead of two and keys from global memory, 386 by eight.
constexpr int TC_FIX_WARPS = 8;
// TMA warp, MMA warp, norm warps, epilogue warps, moving or deciding warps
template <bool APPEND> constexpr int TC_THREADS = 32 * (2 + TC_NORM_WARPS + TC_EPI_WARPS<APPEND> + (APPEND ? TC_MOVE_WARPS : TC_FIX_WARPS));
constexpr int TC_FIX_TOGETHER = 256;  // up to so many near-zero projections of 32 rows, a warp takes them one by one

struct TcShared {
    uint64_t b_full;                   // planes have landed (once)
    uint64_t a_full[TC_ARING];         // K tile of the ring slot has landed
    uint64_t a_empty[TC_ARING];        // MMAs, near-zero decisions and moves are done with the slot's K tile
    uint64_t norm_full[TC_NSLOTS];     // row norms of tile i are in knorm[i % 8]
    uint64_t acc_full[TC_STAGES];      // accumulator is complete
    uint64_t acc_empty[TC_STAGES];     // accumulator has been read back
    uint64_t near_full[TC_MASKS];     // codes are written and the mask is complete
    uint64_t near_empty[TC_MASKS];    // the mask has been read
    uint32_t tmem_base;
    int failed;                        // some bounded wait ran out
    float plane_norm[TC_N + 1];        // [TC_N] = the largest norm
    float knorm[TC_NSLOTS][TC_ROWS];   // |k| * 1.001 of the rows of tile i in slot i % 8 (inf: decide every bit exactly)
    __align__(16) uint32_t near_zero[TC_MASKS][TC_ROWS][TC_N / 32];   // bit k of word c: column 32 c + k
};

// Where an append writes; unused fields without APPEND
struct TcAppend {
    const uint4* v_new;
    const int64_t* input_pos;
    uint4 *k_cache, *v_cache;
    __half* v_norm;
    int32_t* prefill_len;
    int S, Hkv;
    int64_t Tcap;
    // cache row of new row n = (b, s, kvh); -1 for a position outside the cache
    __device__ __forceinline__ int64_t row(int64_t n, int64_t& pos) const {
        const uint32_t bs = (uint32_t)n / (uint32_t)Hkv, kvh = (uint32_t)n - bs * (uint32_t)Hkv;     // n < 2^24
        const uint32_t b = bs / (uint32_t)S;
        pos = __ldg(input_pos + (bs - b * (uint32_t)S));
        return pos >= 0 && pos < Tcap ? ((int64_t)b * Hkv + kvh) * Tcap + pos : -1;
    }
};

// The careful version of one 32-column chunk of one accumulator row (see the epilogue): signs, near-zero columns.
__device__ __noinline__ uint2 slow_chunk(uint32_t taddr, int c, float thr, float knorm, const float* plane_norm_s) {
    uint32_t r[32];
    tmem_ld32(taddr, r);
    uint32_t word = 0, mark = 0;
#pragma unroll 1
    for (int k = 0; k < 32; ++k) {
        const float acc = __uint_as_float(r[k]);
        if (acc >= 0.f) word |= 1u << (8 * (k >> 3) + 7 - (k & 7));
        // an accumulator that overflowed to NaN is marked too
        if (knorm > 0.f && !(fabsf(acc) > thr * plane_norm_s[c * 32 + k])) mark |= 1u << k;
    }
    return make_uint2(word, mark);
}

// d + the exact products of four elements
template <typename Ty> __device__ __forceinline__ double dot4(uint2 a, uint2 b, double d) {
    const float2 a0 = Ty::pair(a.x), a1 = Ty::pair(a.y), b0 = Ty::pair(b.x), b1 = Ty::pair(b.y);
    d = fma((double)a0.x, (double)b0.x, d);
    d = fma((double)a0.y, (double)b0.y, d);
    d = fma((double)a1.x, (double)b1.x, d);
    return fma((double)a1.y, (double)b1.y, d);
}

// Eight bytes of a 128-byte row of a swizzled tile: piece q = 0..15
__device__ __forceinline__ uint2 tile_piece(const char* half_tile, int row, int q) {
    return *reinterpret_cast<const uint2*>(half_tile + row * 128 + (((q >> 1) ^ (row & 7)) << 4) + (q & 1) * 8);
}

__device__ __forceinline__ void patch_code(uint8_t* row_codes, int col, bool set) {
    uint8_t* byte = row_codes + (col >> 3);
    uint32_t* word = reinterpret_cast<uint32_t*>(reinterpret_cast<uintptr_t>(byte) & ~(uintptr_t)3);
    const uint32_t m = 1u << (8 * (int)(reinterpret_cast<uintptr_t>(byte) & 3) + 7 - (col & 7));
    if (set) atomicOr(word, m); else atomicAnd(word, ~m);
}

// Persistent, warp-specialised: every CTA keeps the 256 plane rows in shared memory and walks the
// K tiles blockIdx.x, blockIdx.x + gridDim.x, ...  Warp 0 feeds a ring of K tiles by TMA, warp 1 issues the
// MMAs into one of two accumulators in tensor memory, the eight (APPEND) or sixteen warps from 6 on read the other accumulator back
// (tcgen05.ld), take the signs, apply the near-zero test and write the code bytes; warps 2-5 compute the
// row norms that test needs from the K tile in shared memory, and one tile later decide its near-zero
// projections (APPEND; else the last eight warps do); warps 14-21 (APPEND) move the rows.  So the load of tile i+1, the MMAs of tile i+1 and the
// epilogue of tile i overlap.  Every wait is bounded; a wait that runs out raises `failed`, which makes
// every role leave its loop, and the status flag.
template <typename T, bool APPEND>
__global__ void __launch_bounds__(TC_THREADS<APPEND>, 1)
hash_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_p,
               const T* __restrict__ planes, const T* __restrict__ keys, int64_t key_row_stride, int64_t N, uint8_t* codes, int64_t code_row_stride,
               const int64_t* __restrict__ dst_row, const __grid_constant__ TcAppend ap, int32_t* status) {
    extern __shared__ char tc_raw[];
    __shared__ TcShared ts;
    using Ty = TcType<T>;
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~(uintptr_t)1023);
    char* b_half[2] = {tiles, tiles + TC_B_HALF_BYTES};
    char* a_base = tiles + 2 * TC_B_HALF_BYTES;                 // [ring slot][half][16 KiB]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t n_tiles = (N + TC_ROWS - 1) / TC_ROWS;
    const int64_t my_tiles = (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;     // >= 1: grid <= n_tiles

    if (tid == 0) {
        mbar_init_count(&ts.b_full, 1);
        for (int s = 0; s < TC_ARING; ++s) {
            mbar_init_count(&ts.a_full[s], 1);
            // MMA commit, one arrival per norm warp and per moving warp
            mbar_init_count(&ts.a_empty[s], 1 + TC_NORM_WARPS + (APPEND ? TC_MOVE_WARPS : 0));
        }
        for (int s = 0; s < TC_NSLOTS; ++s) mbar_init_count(&ts.norm_full[s], TC_NORM_WARPS);
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init_count(&ts.acc_full[s], 1);
            mbar_init_count(&ts.acc_empty[s], TC_EPI_WARPS<APPEND>);
        }
        for (int s = 0; s < TC_MASKS; ++s) {
            mbar_init_count(&ts.near_full[s], TC_EPI_WARPS<APPEND>);
            mbar_init_count(&ts.near_empty[s], 4);               // four warps decide a tile
        }
        ts.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&ts.tmem_base)),
                     "r"((uint32_t)(TC_STAGES * TC_N))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ts.tmem_base;
    volatile int* failed = &ts.failed;
    // |plane| * 1.001 of the 256 planes, by the norm and the epilogue warps while the first tiles come in (every CTA
    // computes them for itself: 64 KiB from L2, cheaper than a launch of its own)
    constexpr int NORMERS = TC_NORM_WARPS + TC_EPI_WARPS<APPEND>;
    if (warp >= 2 && warp < 2 + NORMERS) {
        constexpr int U = 4;                                  // planes in flight per warp
        for (int n0 = (warp - 2) * U; n0 < TC_N; n0 += NORMERS * U) {
            uint2 raw[U];
#pragma unroll
            for (int u = 0; u < U; ++u) raw[u] = __ldg(reinterpret_cast<const uint2*>(planes + (size_t)(n0 + u) * TC_D) + lane);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float2 x = Ty::pair(raw[u].x), y = Ty::pair(raw[u].y);
                float sq = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(y.x, y.x, y.y * y.y)));
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) sq += __shfl_xor_sync(FULL, sq, o);
                // squares that may have left fp32's range: an infinite norm, and every projection on the plane is decided exactly
                const bool any = __any_sync(FULL, ((raw[u].x | raw[u].y) & 0x7fff7fffu) != 0);
                if (lane == 0) ts.plane_norm[n0 + u] = sq < TC_TINY && any ? INFINITY : sqrtf(sq) * 1.001f;
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NORMERS * 32) : "memory");
        if (warp == 2) {                                      // the largest, for the cheap first test
            float v = 0.f;
            for (int n = lane; n < TC_N; n += 32) v = fmaxf(v, ts.plane_norm[n]);
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL, v, o));
            if (lane == 0) ts.plane_norm[TC_N] = v;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NORMERS * 32) : "memory");
    }
    // a warp's common answer to a wait; a wait that ran out makes every role leave
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        const bool ok = __all_sync(FULL, mbar_wait_bounded(bar, parity)) != 0;
        if (!ok) *failed = 1;
        return ok;
    };
    auto gone = [&]() { return __any_sync(FULL, *failed != 0) != 0; };
    auto first_row = [&](int64_t i) { return (blockIdx.x + i * gridDim.x) * TC_ROWS; };
    // row of `codes` that row n of the call goes to, -1: not to be written
    auto code_row = [&](int64_t n) -> int64_t {
        int64_t pos;
        if (n >= N) return -1;
        if (APPEND) return ap.row(n, pos);
        return dst_row != nullptr ? dst_row[n] : n;
    };

    // near-zero projections of 32 rows of tile j, whose codes are written: exact fp64 dot products patch their bits
    auto decide = [&](int64_t j, int quad) {
        const int s = (int)(j % TC_MASKS), ra = (int)(j % TC_ARING), r_in_tile = quad * 32 + lane;
        const int64_t dst = code_row(first_row(j) + r_in_tile);
        if (!wait_all(&ts.near_full[s], (uint32_t)((j / TC_MASKS) & 1))) return false;
        uint32_t left[TC_N / 32];
        int mine = 0;
#pragma unroll
        for (int w = 0; w < TC_N / 32; w += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(&ts.near_zero[s][r_in_tile][w]);
            left[w] = x.x;
            left[w + 1] = x.y;
            left[w + 2] = x.z;
            left[w + 3] = x.w;
            mine += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
        }
        if (dst < 0) mine = 0;
        const int count = __reduce_add_sync(FULL, mine);
        __syncwarp();
        if (lane == 0) mbar_arrive(&ts.near_empty[s]);                 // the mask is in registers
        // this lane's next projection
        auto next = [&]() {
            int col = 0;
            bool found = false;
#pragma unroll
            for (int w = 0; w < TC_N / 32; ++w)
                if (!found && left[w] != 0) {
                    col = w * 32 + __ffs(left[w]) - 1;
                    left[w] &= left[w] - 1;
                    found = true;
                }
            --mine;
            return col;
        };
        const char* a = a_base + (size_t)ra * 2 * TC_A_HALF_BYTES;
        // four elements of a row of the tile: of an append, whose K tiles wait for the moving warps anyhow, from shared memory; else
        // from global memory, which leaves the tile to the next load
        auto key_piece = [&](int row, int i4) {
            if constexpr (APPEND) return tile_piece(a + (i4 >> 4) * TC_A_HALF_BYTES, row, i4 & 15);
            else return __ldg(reinterpret_cast<const uint2*>(keys + (first_row(j) + row) * key_row_stride) + i4);
        };
        const int h = lane >> 4, q = lane & 15;
        if (count <= TC_FIX_TOGETHER) {                                // a projection at a time, four elements per lane
            for (unsigned have = __ballot_sync(FULL, mine > 0); have != 0; have = __ballot_sync(FULL, mine > 0)) {
                const int src = __ffs(have) - 1, row = quad * 32 + src;
                const int col = __shfl_sync(FULL, lane == src ? next() : 0, src);
                const uint2 kr = key_piece(row, lane), pr = tile_piece(tiles + h * TC_B_HALF_BYTES, col, q);
                const double d = warp_sum_f64(dot4<Ty>(kr, pr, 0.0));
                if (lane == src) patch_code(codes + dst * code_row_stride, col, d >= 0.0);
            }
        } else {                                                       // hostile inputs: every lane its own row
            while (mine > 0) {
                const int col = next();
                double d = 0.0;
#pragma unroll 2
                for (int i4 = 0; i4 < 32; ++i4)
                    d = dot4<Ty>(key_piece(r_in_tile, i4), tile_piece(tiles + (i4 >> 4) * TC_B_HALF_BYTES, col, i4 & 15), d);
                patch_code(codes + dst * code_row_stride, col, d >= 0.0);
            }
            __syncwarp();
        }
        if (APPEND) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&ts.a_empty[ra]);
        }
        return true;
    };

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            mbar_expect(&ts.b_full, 2 * TC_B_HALF_BYTES);
            tma_load_2d(b_half[0], &map_p, 0, 0, &ts.b_full);
            tma_load_2d(b_half[1], &map_p, TC_KHALF, 0, &ts.b_full);
            int64_t i = 0;
#pragma unroll 1
            for (; i < my_tiles && !*failed; ++i) {
                const int ra = (int)(i % TC_ARING);
                if (i >= TC_ARING && !mbar_wait_bounded(&ts.a_empty[ra], (uint32_t)((i / TC_ARING - 1) & 1))) {
                    *failed = 1;
                    break;
                }
                const int row0 = (int)first_row(i);
                char* a = a_base + (size_t)ra * 2 * TC_A_HALF_BYTES;
                mbar_expect(&ts.a_full[ra], 2 * TC_A_HALF_BYTES);
                tma_load_2d(a, &map_k, 0, row0, &ts.a_full[ra]);
                tma_load_2d(a + TC_A_HALF_BYTES, &map_k, TC_KHALF, row0, &ts.a_full[ra]);
            }
            if (i < my_tiles) {                                 // left early: no copy stays in flight
                mbar_wait_bounded(&ts.b_full, 0);
                for (int64_t q = i > TC_ARING ? i - TC_ARING : 0; q < i; ++q)
                    mbar_wait_bounded(&ts.a_full[q % TC_ARING], (uint32_t)((q / TC_ARING) & 1));
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            if (!mbar_wait_bounded(&ts.b_full, 0)) *failed = 1;
#pragma unroll 1
            for (int64_t i = 0; i < my_tiles && !*failed; ++i) {
                const int s = (int)(i & 1), ra = (int)(i % TC_ARING);
                const uint32_t par = (uint32_t)((i >> 1) & 1);
                if (!mbar_wait_bounded(&ts.a_full[ra], (uint32_t)((i / TC_ARING) & 1)) ||
                    (i >= TC_STAGES && !mbar_wait_bounded(&ts.acc_empty[s], par ^ 1u))) {
                    *failed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_addr = smem_addr(a_base + (size_t)ra * 2 * TC_A_HALF_BYTES);
#pragma unroll
                for (int k = 0; k < TC_D / 16; ++k) {
                    const int half = k >> 2, kb = k & 3;           // 16 elements = 32 bytes along the swizzled row
                    const uint64_t da = umma_desc_sw128(a_addr + half * TC_A_HALF_BYTES + kb * 32);
                    const uint64_t db = umma_desc_sw128(smem_addr(b_half[half]) + kb * 32);
                    umma_f16(tmem + (uint32_t)s * TC_N, da, db, Ty::IDESC, k > 0 ? 1u : 0u);
                }
                umma_commit(&ts.acc_full[s]);                       // accumulator complete ...
                umma_commit(&ts.a_empty[ra]);                       // ... and the K tile no longer read by the MMAs
            }
        }
    } else if (warp < 2 + TC_NORM_WARPS) {
        // ---- one thread per row of the K tile, read from the swizzled tile in shared memory
        // (16-byte chunk c of row r sits at chunk c ^ (r & 7))
        const int r_in_tile = (warp - 2) * 32 + lane;
        bool ok = wait_all(&ts.b_full, 0);                             // the near-zero decisions (APPEND) read the planes
#pragma unroll 1
        for (int64_t i = 0; ok && i < my_tiles + (APPEND ? 1 : 0) && !gone(); ++i) {
            // norms of tile i.  They go to slot i % 8, which has a barrier of its own (these warps may be
            // ahead of the epilogue, and a barrier must not complete two phases ahead of a waiter): tile i
            // can only have been loaded after the MMAs of tile i-4 were done, which started after the
            // epilogue of tile i-6 had finished, so the last reader of the slot (tile i-8) is long gone.
            if (i < my_tiles) {
                const int ra = (int)(i % TC_ARING);
                if (!(ok = wait_all(&ts.a_full[ra], (uint32_t)((i / TC_ARING) & 1)))) break;
                float ss = 0.f;
                uint32_t any = 0;
                const char* a = a_base + (size_t)ra * 2 * TC_A_HALF_BYTES + (size_t)r_in_tile * 128;
#pragma unroll(APPEND ? 1 : 2)         // the roles of an append together have to fit the instruction cache
                for (int h = 0; h < 2; ++h) {
#pragma unroll(APPEND ? 4 : 8)
                    for (int c = 0; c < 8; ++c) {
                        const uint4 w = *reinterpret_cast<const uint4*>(a + h * TC_A_HALF_BYTES + ((c ^ (r_in_tile & 7)) << 4));
                        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 x = Ty::pair(u[j]);
                            ss = fmaf(x.x, x.x, fmaf(x.y, x.y, ss));
                            any |= u[j];
                        }
                    }
                }
                float kn = sqrtf(ss) * 1.001f;
                // a row whose products could overflow fp32, or whose squares may have vanished, gets an infinite norm: every
                // projection of it is then decided exactly (a NaN norm stays NaN and is handled in the epilogue)
                if (kn * ts.plane_norm[TC_N] >= 1e38f || (ss < TC_TINY && (any & 0x7fff7fffu) != 0)) kn = INFINITY;
                ts.knorm[i % TC_NSLOTS][r_in_tile] = kn;
                __syncwarp();
                if (lane == 0) mbar_arrive(&ts.norm_full[i % TC_NSLOTS]);
            }
            if (!APPEND) {
                if (lane == 0) mbar_arrive(&ts.a_empty[i % TC_ARING]);
            } else if (i > 0) {
                ok = decide(i - 1, warp - 2);
            }
        }
    } else if (warp < 2 + TC_NORM_WARPS + TC_EPI_WARPS<APPEND>) {
        // ---- epilogue: the two or four warps with the same (warp % 4) share the 32 accumulator lanes of that
        // quarter, a part of the columns each; a thread owns one row and 128 or 64 columns
        constexpr int CHUNKS = 32 / TC_EPI_WARPS<APPEND>;       // of 32 columns, a thread
        const int quad = warp & 3, ch = (warp - 2 - TC_NORM_WARPS) >> 2;
        const int r_in_tile = quad * 32 + lane;
        bool ok = true;
#pragma unroll 1
        for (int64_t i = 0; ok && i < my_tiles && !gone(); ++i) {
            const int s = (int)(i & 1);
            const uint32_t par = (uint32_t)((i >> 1) & 1);
            const int64_t row = first_row(i) + r_in_tile;
            const bool valid = row < N;
            const int64_t dst = code_row(row);                      // requested before the waits below
            ok = wait_all(&ts.norm_full[i % TC_NSLOTS], (uint32_t)((i / TC_NSLOTS) & 1)) &&
                 (i < TC_MASKS || wait_all(&ts.near_empty[i % TC_MASKS], (uint32_t)((i / TC_MASKS - 1) & 1)));
            if (!ok) break;
            // rows behind the last must not look like rows of zeros, whose careful path costs a warp's tile 16 us
            const float knorm = valid ? ts.knorm[i % TC_NSLOTS][r_in_tile] : 1.f;
            const float thr = TC_BAND * knorm;
            const float thr_max = valid ? thr * ts.plane_norm[TC_N] : -1.f;  // cheap first test, exact test inside
            if (!(ok = wait_all(&ts.acc_full[s], par))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t words[CHUNKS] = {};
#pragma unroll(APPEND ? 1 : CHUNKS)
            for (int c4 = 0; c4 < CHUNKS; ++c4) {
                const int c = ch * CHUNKS + c4;
                const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)s * TC_N + c * 32;
                uint32_t r[32];
                tmem_ld32(at, r);
                // Fast path, two instructions per projection and no branch: the sign bits are shifted
                // into one register per table (first plane = most significant bit) and the smallest
                // |acc| of the chunk decides whether anything needs the near-zero treatment.  A finite
                // norm below the overflow guard means every accumulator is finite.
                uint32_t neg[4] = {0u, 0u, 0u, 0u};
                float mn[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    neg[k >> 3] = __funnelshift_l(r[k], neg[k >> 3], 1);
                    mn[k & 3] = fminf(mn[k & 3], fabsf(__uint_as_float(r[k])));
                }
                uint32_t word = ~(neg[0] | (neg[1] << 8) | (neg[2] << 16) | (neg[3] << 24)), mark = 0;
                const float m = fminf(fminf(mn[0], mn[1]), fminf(mn[2], mn[3]));
                if (m <= thr_max && knorm < INFINITY && knorm > 0.f) {
                    // some projection of this row is near zero (about one chunk in seven of a warp has one): mark
                    // it for the exact decision.  The bits above stay as they are - the only value whose
                    // sign bit disagrees with (acc >= 0) is -0, and that one is always marked.
#pragma unroll
                    for (int k = 0; k < 32; ++k)
                        if (fabsf(__uint_as_float(r[k])) <= thr_max && fabsf(__uint_as_float(r[k])) <= thr * ts.plane_norm[c * 32 + k])
                            mark |= 1u << k;
                }
                // warp-uniform: the reload in the careful path is a warp-wide instruction
                if (__any_sync(FULL, !(knorm < INFINITY) || knorm == 0.f)) {
                    // rare: a row that may overflow or holds NaN, or a row of zeros - decide every bit
                    // the plain way (a rolled loop over a second copy of the chunk, out of line)
                    const uint2 w2 = slow_chunk(at, c, thr, knorm, ts.plane_norm);
                    if (!(knorm < INFINITY) || knorm == 0.f) {
                        word = w2.x;
                        mark = w2.y;
                    }
                }
#pragma unroll
                for (int x = 0; x < CHUNKS; ++x) words[x] = x == c4 ? word : words[x];
                ts.near_zero[i % TC_MASKS][r_in_tile][c] = mark;
            }
            // the accumulator is free again
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&ts.acc_empty[s]);
            if (dst >= 0) {                                        // negative = row not to be written
                if constexpr (CHUNKS == 4) reinterpret_cast<uint4*>(codes + dst * code_row_stride)[ch] = make_uint4(words[0], words[1], words[2], words[3]);
                else reinterpret_cast<uint2*>(codes + dst * code_row_stride)[ch] = make_uint2(words[0], words[1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ts.near_full[i % TC_MASKS]);          // releases the codes to the warps that may patch them
        }
    } else if (!APPEND) {
        // ---- decisions
        const int own = warp - 2 - TC_NORM_WARPS - TC_EPI_WARPS<APPEND>;
        bool ok = wait_all(&ts.b_full, 0);
#pragma unroll 1
        for (int64_t i = own >> 2; ok && i < my_tiles && !gone(); i += 2) ok = decide(i, own & 3);
    } else {
        // ---- APPEND: 16 rows of the tile to the cache, half a warp per row and 16 bytes per lane.  v_norm is the number the
        // general append stores, the fp64 norm rounded to fp32 and then to fp16; fp64 arithmetic runs at a few lanes a cycle
        // here (the sums alone took 9 of a tile's 10 us), so the norm is taken in fp32, whose error is far below 24 units of
        // its last place, and in fp64 only where that could change the rounding to fp16 (one row in 170), or fp32 or fp16
        // leaves its normal range.
        const int m0 = (warp - 2 - TC_NORM_WARPS - TC_EPI_WARPS<APPEND>) * 16, part = lane >> 4, piece = lane & 15;
        bool bad = false, ok = true;
        int32_t max_len = 0;
#pragma unroll 1
        for (int64_t i = 0; ok && i < my_tiles && !gone(); ++i) {
            const int ra = (int)(i % TC_ARING);
            const int64_t n0 = first_row(i) + m0;
            int64_t dst = -1, pos = -1;
            if (lane < 16 && n0 + lane < N) {
                dst = ap.row(n0 + lane, pos);
                if (dst < 0) bad = true;
                else if (pos + 1 > max_len) max_len = (int32_t)(pos + 1);
            }
            uint4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int64_t n = n0 + 2 * j + part;
                v[j] = n < N ? __ldg(ap.v_new + n * 16 + piece) : make_uint4(0, 0, 0, 0);
            }
            if (!(ok = wait_all(&ts.a_full[ra], (uint32_t)((i / TC_ARING) & 1)))) break;
            const char* a = a_base + (size_t)ra * 2 * TC_A_HALF_BYTES + (piece >> 3) * TC_A_HALF_BYTES;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = m0 + 2 * j + part;
                const int64_t d = __shfl_sync(FULL, dst, 2 * j + part);
                const uint4 k = *reinterpret_cast<const uint4*>(a + r * 128 + (((piece & 7) ^ (r & 7)) << 4));
                if (d >= 0) {
                    ap.k_cache[d * 16 + piece] = k;
                    ap.v_cache[d * 16 + piece] = v[j];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ts.a_empty[ra]);
            float mine = 0.f;                                  // lane (part, piece < 8): ||v||^2 of row 2 piece + part
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                float ss = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = Ty::pair(w[e]);
                    ss = fmaf(x.y, x.y, fmaf(x.x, x.x, ss));
                }
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) ss += __shfl_xor_sync(FULL, ss, o);
                if (piece == j) mine = ss;
            }
            const float s = sqrtf(mine);
            const bool sure = norm_decides_f16(s);
            const int64_t dm = __shfl_sync(FULL, dst, (2 * piece + part) & 15);
            if (sure && piece < 8 && dm >= 0) ap.v_norm[dm] = __float2half_rn(s);
            uint32_t redo = __ballot_sync(FULL, !sure && piece < 8 && dm >= 0);
            redo = (redo | redo >> 16) & 0xffu;
#pragma unroll 1
            for (; redo != 0; redo &= redo - 1) {              // warp-uniform
                const int j = __ffs(redo) - 1;
                const int64_t n = n0 + 2 * j + part;
                const uint4 x = n < N ? __ldg(ap.v_new + n * 16 + piece) : make_uint4(0, 0, 0, 0);
                const uint32_t w[4] = {x.x, x.y, x.z, x.w};
                double ss = 0.0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 y = Ty::pair(w[e]);
                    ss = fma((double)y.x, (double)y.x, ss);
                    ss = fma((double)y.y, (double)y.y, ss);
                }
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) ss += __shfl_xor_sync(FULL, ss, o);
                const int64_t d = __shfl_sync(FULL, dst, 2 * j + part);
                if (piece == 0 && d >= 0) ap.v_norm[d] = __float2half_rn((float)sqrt(ss));
            }
        }
        max_len = __reduce_max_sync(FULL, max_len);
        bad = __any_sync(FULL, bad) != 0;
        if (lane == 0) {
            if (bad && status != nullptr) atomicOr(status, SK_DEV_POS_OUT_OF_RANGE);
            if (max_len > 0) atomicMax(ap.prefill_len, max_len);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && ts.failed && status != nullptr) atomicOr(status, SK_DEV_WAIT_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)(TC_STAGES * TC_N))
                     : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// [rows, 128] 16-bit row-major (row stride in elements) -> boxes of 64 columns x box_rows rows
int make_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t rows, int64_t row_stride, uint32_t box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (enc == nullptr) return fail(SK_ERR_CUDA, "sk_hash_keys_tc: cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {(cuuint64_t)TC_D, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
    const cuuint32_t box[2] = {(cuuint32_t)TC_KHALF, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, type, 2, const_cast<void*>(base), dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(SK_ERR_CUDA, "sk_hash_keys_tc: cuTensorMapEncodeTiled failed (%d)", (int)r);
    return SK_OK;
}

// grid: one persistent CTA per SM
template <typename T, bool APPEND>
int hash_tc_launch(const void* keys, int64_t key_row_stride, const void* planes, int64_t N, uint8_t* codes,
                   int64_t code_row_stride, const int64_t* dst_row, const TcAppend& ap, int32_t* status, cudaStream_t st) {
    CUtensorMap map_k, map_p;
    int rc = make_map(&map_k, TcType<T>::MAP, keys, (uint64_t)N, key_row_stride, TC_ROWS);
    if (rc != SK_OK) return rc;
    rc = make_map(&map_p, TcType<T>::MAP, planes, TC_N, TC_D, TC_N);
    if (rc != SK_OK) return rc;
    auto kern = hash_tc_kernel<T, APPEND>;
    const size_t smem = TC_PIPE_SMEM + 1024;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(SK_ERR_CUDA, "hash_tc_kernel smem attribute: %s", cudaGetErrorString(e));
    const int64_t tiles = (N + TC_ROWS - 1) / TC_ROWS;
    const unsigned n_cta = (unsigned)(tiles < sm_count() ? tiles : sm_count());
    kern<<<n_cta, TC_THREADS<APPEND>, smem, st>>>(map_k, map_p, static_cast<const T*>(planes), static_cast<const T*>(keys), key_row_stride, N, codes,
                                              code_row_stride, dst_row, ap, status);
    return check_launch("hash_tc_kernel");
}

}  // namespace

int launch_hash_keys_tc(const void* keys, int64_t key_row_stride, const void* planes, int64_t N, uint8_t* codes,
                        int64_t code_row_stride, const int64_t* dst_row, int32_t* status, cudaStream_t st) {
    if (N == 0) return SK_OK;
    if (N >= TC_MAX_ROWS) return fail(SK_ERR_UNSUPPORTED, "sk_hash_keys_tc: at most 2^24 - 1 rows per call");
    return hash_tc_launch<__nv_bfloat16, false>(keys, key_row_stride, planes, N, codes, code_row_stride, dst_row, TcAppend{}, status, st);
}

bool kv_append_tc_applicable(const void* k_new, const void* v_new, int kv_dtype, const void* planes, int plane_dtype,
                             const void* k_cache, const void* v_cache, const uint8_t* codes, int64_t N, int D, int L, int P) {
    return (kv_dtype == SK_BF16 || kv_dtype == SK_F16) && plane_dtype == kv_dtype && D == TC_D && L == TC_N / 8 && P == 8 &&
           N < TC_MAX_ROWS &&
           (((uintptr_t)k_new | (uintptr_t)v_new | (uintptr_t)planes | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)codes) & 15) == 0;
}

int launch_kv_append_tc(const void* k_new, const void* v_new, int kv_dtype, const int64_t* input_pos, const void* planes,
                        void* k_cache, void* v_cache, uint8_t* codes, uint16_t* v_norm, int32_t* prefill_len, int32_t* status,
                        int B, int S, int Hkv, int64_t Tcap, cudaStream_t st) {
    const int64_t N = (int64_t)B * S * Hkv;
    if (N >= TC_MAX_ROWS) return fail(SK_ERR_UNSUPPORTED, "sk_kv_append_tc: at most 2^24 - 1 rows per call");
    TcAppend ap;
    ap.v_new = static_cast<const uint4*>(v_new);
    ap.input_pos = input_pos;
    ap.k_cache = static_cast<uint4*>(k_cache);
    ap.v_cache = static_cast<uint4*>(v_cache);
    ap.v_norm = reinterpret_cast<__half*>(v_norm);
    ap.prefill_len = prefill_len;
    ap.S = S;
    ap.Hkv = Hkv;
    ap.Tcap = Tcap;
    return kv_dtype == SK_BF16 ? hash_tc_launch<__nv_bfloat16, true>(k_new, TC_D, planes, N, codes, TC_N / 8, nullptr, ap, status, st)
                               : hash_tc_launch<__half, true>(k_new, TC_D, planes, N, codes, TC_N / 8, nullptr, ap, status, st);
}

}  // namespace sk
