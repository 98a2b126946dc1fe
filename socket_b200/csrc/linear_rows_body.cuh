// out [rows, n] = x [rows, k] W [n, k]^T for at most 8 rows (a decode step's projections), bf16 or fp16.
//
// Every weight is read once and used at most 8 times, so the bound is the memory: what matters is that loads are in
// flight all the time.  A CTA walks tiles of 16 RT weight rows; its 8 warps divide k.  A lane holds 32 consecutive
// bytes of two rows of each 16-row tile (four lanes: 128 bytes of a row) in a ring of registers, refilled as soon as a
// piece has been used and across the ends of tiles, so the stream does not stop at a tile's reduction: 64 KB in flight
// per CTA, two CTAs per SM (or one of 16 warps, when there is at most one tile per SM).  The products are m16n8k16 MMAs,
// weight rows against the (up to) 8 rows of x; a sum over k may be taken in any order as long as both operands take the
// same one, so a lane's own 16 elements serve as they were loaded, without a shuffle or a pass through shared memory.
// The warps' sums meet in shared memory, in warp order, in fp32.
//
// Weights do not depend on the kernel before this one.  With `chained` the kernel may start while kernels before it still
// run, fills its ring with weights, and only then waits for x.  It lets its own successor in before that wait, and so do the
// kernels of the sparse step: a chained projection can reach back over several kernels.  The caller vouches that neither
// the stream's last unchained launch nor anything behind it writes the weights.
//
// Measured (one row, cold weights, back to back in a graph; chained / not / cuBLAS): 4096 x 14336 19.2 / 20.8 / 24.4 us
// (6.1 TB/s), 28672 x 4096 37.0 / 38.7 / 39.1 us, 4096 x 4096 6.1 / 7.9 / 12.9 us, 2048 x 2048 2.4 / 4.0 / 7.3 us; 8 rows:
// 4096 x 14336 19.6 / 21.4 us, 2048 x 5632 5.4 / 7.2 us (one row 4.6 / 6.7).
#pragma once
#include "abi_check.cuh"
#include "blocks.cuh"
#include "warp_mma.cuh"

namespace sk {
namespace {

constexpr int LR_MAX_ROWS = 8;

__device__ __forceinline__ void lr_load_weights(const void* p, bool live, uint32_t (&r)[8]) {
    if (live) {
        asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "l"(p));
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = 0u;
    }
}
__device__ __forceinline__ void lr_load_x(const void* p, bool live, uint32_t (&r)[8]) {
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    if (live) {
        a = reinterpret_cast<const uint4*>(p)[0];
        b = reinterpret_cast<const uint4*>(p)[1];
    }
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
    r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}

// Tiles 0 .. plain_tiles - 1: 16 RT consecutive rows of W, results to `out`.  The others (RT = 2): 16 rows of the gate
// and the same 16 of the up projection, results through the gated unit to `act`.
template <typename T, int RT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS)
linear_rows_kernel(const __grid_constant__ sk_linear_params p, int plain_tiles, int tiles) {
    // Two stages of four 32-byte loads of weights each.  (Four stages of two: 4.6 instead of 6.0 TB/s at 4736 x 14336.)
    constexpr int NS = 2, PIECES = 2 / RT, STEP = 64 * PIECES;
    constexpr int COLS = 16 * RT;
    __shared__ float red[2][WARPS][LR_MAX_ROWS][COLS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();
    const T* w = (const T*)p.w;
    const int n_kb = (p.k + STEP - 1) / STEP;
    const int kb0 = (int)((int64_t)warp * n_kb / WARPS), n_it = (int)((int64_t)(warp + 1) * n_kb / WARPS) - kb0;
    const int k_first = kb0 * STEP + 16 * t;                    // this lane's first element of the warp's part
    const int my_tiles = tiles > (int)blockIdx.x ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int total = my_tiles * n_it;

    // the loading end of the ring: piece l_it of tile l_tile
    const T* wl[2 * RT];
    int l_tile = blockIdx.x, l_it = 0;
    auto point = [&]() {                                      // rows past the end repeat the last one, their results are dropped
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = half * 8 + g;
                int64_t row;
                if (RT == 2 && l_tile >= plain_tiles) {
                    const int f = min((l_tile - plain_tiles) * 16 + r, p.ff - 1);
                    row = (rt == 0 ? p.gate_row : p.up_row) + f;
                } else {
                    row = min(l_tile * COLS + rt * 16 + r, p.n - 1);
                }
                wl[2 * rt + half] = w + row * p.w_ld + k_first;
            }
    };
    uint32_t wf[NS][PIECES][2 * RT][8], xf[NS][PIECES][8];
    int xl_it = 0;
    auto load_w = [&](int s) {
#pragma unroll
        for (int c = 0; c < PIECES; ++c)
#pragma unroll
            for (int i = 0; i < 2 * RT; ++i)
                lr_load_weights(wl[i] + l_it * STEP + c * 64, k_first + l_it * STEP + c * 64 < p.k, wf[s][c][i]);
        if (++l_it == n_it) {
            l_it = 0;
            l_tile += gridDim.x;
            if (l_tile < tiles) point();
        }
    };
    const T* xg = (const T*)p.x + (int64_t)(g < p.rows ? g : 0) * p.x_ld + k_first;
    auto load_x = [&](int s) {
#pragma unroll
        for (int c = 0; c < PIECES; ++c)
            lr_load_x(xg + xl_it * STEP + c * 64, g < p.rows && k_first + xl_it * STEP + c * 64 < p.k, xf[s][c]);
        if (++xl_it == n_it) xl_it = 0;
    };
    if (total > 0) point();
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < total) load_w(s);
    pdl_wait();                                               // x comes from the kernel before
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < total) load_x(s);

    float acc[RT][4];
    int tile = blockIdx.x, c_it = 0, parity = 0;
    auto clear = [&]() {
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[rt][e] = 0.f;
    };
    auto finish_tile = [&]() {                                // acc[rt]: (row g, x rows 2t, 2t + 1), (row g + 8, the same)
        float (*part)[LR_MAX_ROWS][COLS] = red[parity];
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[warp][2 * t + (e & 1)][rt * 16 + g + ((e >> 1) << 3)] = acc[rt][e];
        __syncthreads();                                      // the next tile's sums go to the other half of `red`
        auto sum = [&](int row, int c) {
            float v = 0.f;
#pragma unroll
            for (int k = 0; k < WARPS; ++k) v += part[k][row][c];
            return v;
        };
        if (RT == 2 && tile >= plain_tiles) {
            const int row = tid >> 4, c = tid & 15, f = (tile - plain_tiles) * 16 + c;
            if (row < p.rows && f < p.ff) {
                const float gate = sum(row, c), up = sum(row, 16 + c);
                float v;
                if (p.glu == SKB_GLU_CLAMPED) {
                    const float a = fminf(gate, p.limit), b = fminf(fmaxf(up, -p.limit), p.limit);
                    v = a * sigmoid_scaled<T>(a, p.slope) * (b + 1.f);
                } else {
                    v = silu<T>(gate) * up;
                }
                ((T*)p.act)[(int64_t)row * p.act_ld + f] = from_f32<T>(v);
            }
        } else {
            const int row = tid / COLS, c = tid % COLS, n = tile * COLS + c;
            if (row < p.rows && n < p.n) {
                float v = sum(row, c);
                if (p.res != nullptr) v += to_f32(((const T*)p.res)[(int64_t)row * p.res_ld + n]);
                if (p.out_f32) ((float*)p.out)[(int64_t)row * p.out_ld + n] = v;
                else ((T*)p.out)[(int64_t)row * p.out_ld + n] = from_f32<T>(v);
            }
        }
        parity ^= 1;
        tile += gridDim.x;
    };
    static_assert(32 * WARPS >= LR_MAX_ROWS * COLS, "a thread per result of a tile");
    clear();
    if (n_it == 0) {                                          // fewer pieces than warps: nothing to add
        for (int i = 0; i < my_tiles; ++i) finish_tile();
        return;
    }
    for (int base = 0; base < total; base += NS) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            if (base + s < total) {
#pragma unroll
                for (int c = 0; c < PIECES; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt)
                            mma16816(acc[rt], wf[s][c][2 * rt][2 * j], wf[s][c][2 * rt + 1][2 * j], wf[s][c][2 * rt][2 * j + 1],
                                   wf[s][c][2 * rt + 1][2 * j + 1], xf[s][c][2 * j], xf[s][c][2 * j + 1], (const T*)nullptr);
                if (base + s + NS < total) {
                    load_w(s);
                    load_x(s);
                }
                if (++c_it == n_it) {
                    c_it = 0;
                    finish_tile();
                    clear();
                }
            }
        }
    }
}

template <typename T>
int linear_dispatch(const sk_linear_params& p, cudaStream_t st) {
    // 16 rows a tile while that leaves every tile its own CTA, else 32; 16 warps when an SM has one CTA anyway (2048 x 5632:
    // 4.8 instead of 8.3 us).  Grids are evened out: 224 CTAs x 4 tiles of 896 take 38.2 us, 296 of which 8 have a fourth, 41.5.
    const int sms = sm_count(), tiles16 = (p.n + 15) / 16 + 2 * ((p.ff + 15) / 16);
    const bool two = p.ff > 0 || tiles16 > 2 * sms, wide = !two && tiles16 <= sms;
    const int plain = two ? (p.n + 31) / 32 : (p.n + 15) / 16, tiles = plain + (p.ff + 15) / 16, room = wide ? sms : 2 * sms;
    const int rounds = (tiles + room - 1) / room;
    const dim3 grid((unsigned)((tiles + rounds - 1) / rounds)), block(wide ? 512u : 256u);
    cudaError_t e;
    auto kern = wide ? linear_rows_kernel<T, 1, 16> : two ? linear_rows_kernel<T, 2, 8> : linear_rows_kernel<T, 1, 8>;
    if (p.chained) {
        e = launch_after(kern, grid, block, 0, st, p, plain, tiles);
    } else {
        kern<<<grid, block, 0, st>>>(p, plain, tiles);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(SK_ERR_CUDA, "linear_rows_kernel: %s", cudaGetErrorString(e));
    return SK_OK;
}

}  // namespace

bool linear_rows_applicable(const sk_linear_params& p) {
    return p.rows > 0 && p.rows <= LR_MAX_ROWS && p.k > 0 && p.x_ld >= p.k && p.w_ld >= p.k && (p.dtype == SK_BF16 || p.dtype == SK_F16) &&
           p.k % 16 == 0 && p.w_ld % 16 == 0 && p.x_ld % 8 == 0 && (uintptr_t)p.w % 32 == 0 && (uintptr_t)p.x % 16 == 0;
}

int linear_rows(const sk_linear_params* p, cudaStream_t st) {
    SK_REQUIRE(p && p->x && p->w && p->rows > 0 && p->k > 0 && p->n >= 0 && p->ff >= 0 && p->n + p->ff > 0,
               "linear_rows: null pointer or empty product");
    SK_REQUIRE((p->n == 0 || (p->out && p->out_ld >= p->n)) && (p->res == nullptr || p->res_ld >= p->n) && p->x_ld >= p->k && p->w_ld >= p->k,
               "linear_rows: output missing or row stride smaller than row");
    SK_REQUIRE(p->ff == 0 || (p->act && p->act_ld >= p->ff && p->gate_row >= 0 && p->up_row >= 0 &&
                              (p->glu == SKB_GLU_CLAMPED || p->glu == SKB_GLU_SILU)), "linear_rows: gated unit incomplete");
    if (!linear_rows_applicable(*p))
        return fail(SK_ERR_UNSUPPORTED, "linear_rows: at most 8 rows of bf16 or fp16, k and the weights' row stride multiples of 16, aligned rows");
    return p->dtype == SK_BF16 ? linear_dispatch<__nv_bfloat16>(*p, st) : linear_dispatch<__half>(*p, st);
}

}  // namespace sk
