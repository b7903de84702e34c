// The two products of routed experts (see experts.cu) for few rows an expert (decoded tokens), bfloat16 with float32 sums on
// the tensor cores: a tile of 8, 16 or 32 listed rows, all of one expert, by 16 weight rows (gated: 16 gate and the 16
// matching up rows) or 32 (not gated) a warp.  Bound by the weights' bytes: a weight goes from memory to a register once, sixteen
// bytes a lane, and from there into mma.sync (m16n8k16: weight rows as M, listed rows as N) with no stop in shared memory.  That
// works because a product does not care in which order K is taken: lane t of a row's four holds elements 8 t .. 8 t + 7 of every
// 32, and the listed rows' lanes hold the same ones, so the pairs that the instruction multiplies are the right ones.  A warp asks
// for 64 elements of K of its 32 weight rows ahead of those that it multiplies; KW warps share a group's K and add their sums in
// order through shared memory.  Both products of
// 16 tokens with 4 of 32 experts: width 4,096, inner 1,536 298 -> 189 us (CUDA cores before; 168 us for the bytes); width 2,048,
// inner 1,024 129 -> 70 us (56); 128 tokens, which went through mma.sync from shared memory, 557 -> 300 us.
#include "common.cuh"
#include "activations.cuh"

namespace {

constexpr int THREADS = 256, WARPS = THREADS / 32, KSTEP = 64;

__device__ __forceinline__ uint4 load16(const bf16* p, bool live) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (live) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// NT: tiles of 8 listed rows.  A group of weight rows is 16 output columns (gated) or 32; a block has WARPS / KW of them.
template <bool GATED, int NT, int KW>
__global__ void __launch_bounds__(THREADS, 2) moe_product_few_kernel(const bf16* __restrict__ x, const int* __restrict__ sorted_rows,
                                                                     const int* __restrict__ tile_expert, const bf16* __restrict__ weight,
                                                                     bf16* __restrict__ out, int n, int k, int top, int block, int act) {
    constexpr int TILE = 8 * NT, GROUPS = WARPS / KW, COLS = GATED ? 16 : 32;
    __shared__ float sums[WARPS][2][16][TILE + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int expert = tile_expert[blockIdx.x];
    if (expert < 0) return;
    const int row0 = blockIdx.x * TILE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int group = warp / KW, part = warp % KW;
    const int col0 = (blockIdx.y * GROUPS + group) * COLS;
    if (col0 < n) {
        // weight rows of this lane: half 0 and 1, rows g and g + 8 of each (columns beyond the last repeat it and are not stored)
        const bf16* w = weight + (size_t)expert * (GATED ? 2 : 1) * n * k + 8 * t;
        const bf16* w_row[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int col = min(col0 + (GATED ? 0 : 16 * h) + g + 8 * u, n - 1);
                const int row = !GATED ? col : (block ? col / block * 2 * block + col % block + h * block : h * n + col);
                w_row[h][u] = w + (size_t)row * k;
            }
        const bf16* x_row[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int pair = sorted_rows[row0 + 8 * j + g];
            x_row[j] = pair >= 0 ? x + (size_t)(GATED ? pair / top : row0 + 8 * j + g) * k + 8 * t : nullptr;
        }
        float acc[2][NT][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[h][j][e] = 0.0f;
        uint4 wv[2][2][2][2];                            // [buffer][half][row][32 elements of K]
        const int steps = (k + KSTEP - 1) / KSTEP;
        const int first = part * steps / KW, last = (part + 1) * steps / KW;
        auto ask = [&](int buffer, int step) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int at = step * KSTEP + 32 * c;
                const bool live = step < last && at + 8 * t < k;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int u = 0; u < 2; ++u) wv[buffer][h][u][c] = load16(w_row[h][u] + at, live);
            }
        };
        auto multiply = [&](int buffer, int step) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int at = step * KSTEP + 32 * c;
                uint4 xv[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    xv[j] = make_uint4(0u, 0u, 0u, 0u);
                    if (x_row[j] && at + 8 * t < k) xv[j] = *reinterpret_cast<const uint4*>(x_row[j] + at);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint4 lo = wv[buffer][h][0][c], hi = wv[buffer][h][1][c];
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        mma_bf16(acc[h][j], lo.x, hi.x, lo.y, hi.y, xv[j].x, xv[j].y);
                        mma_bf16(acc[h][j], lo.z, hi.z, lo.w, hi.w, xv[j].z, xv[j].w);
                    }
                }
            }
        };
        ask(0, first);
        for (int step = first; step < last; step += 2) {
            ask(1, step + 1);
            multiply(0, step);
            ask(0, step + 2);
            if (step + 1 < last) multiply(1, step + 1);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) sums[warp][h][g + 8 * (e >> 1)][8 * j + 2 * t + (e & 1)] = acc[h][j][e];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < GROUPS * COLS * TILE; i += THREADS) {
        const int c = i % COLS, r = i / COLS % TILE, b = i / (COLS * TILE);
        const int pair = sorted_rows[row0 + r], col = (blockIdx.y * GROUPS + b) * COLS + c;
        if (pair < 0 || col >= n) continue;
        float v = 0.0f, u = 0.0f;
#pragma unroll
        for (int q = 0; q < KW; ++q) {
            v += sums[b * KW + q][GATED ? 0 : c >> 4][c & 15][r];
            if (GATED) u += sums[b * KW + q][1][c][r];
        }
        if (GATED) {
            const float gate = round_bf16(v);            // the projections' own rounding
            v = gate / (1.0f + expf(-gate)) * round_bf16(u);
        } else if (act >= 0) {
            v = mrs_activate(v, act);
        }
        out[(size_t)(GATED || act >= 0 ? row0 + r : pair) * n + col] = __float2bfloat16_rn(v);
    }
}

}  // namespace

// As mrs_moe_product_rows, bfloat16 only, lists in tiles of `tile` rows: 8, 16 or 32.  k a multiple of 8, x and weight on 16-byte
// boundaries.
MRS_EXPORT int mrs_moe_product_few(int gated, const void* x, const int* sorted_rows, const int* tile_expert, const void* weight, void* out,
                                   int capacity, int tile, int n, int k, int top, int block, int act, void* stream) {
    if (capacity <= 0) return 0;
    if ((tile != 8 && tile != 16 && tile != 32) || capacity % tile || n <= 0 || k <= 0 || k % 8 || top <= 0 || block < 0 ||
        (block && (!gated || n % block)) || act > 4 || (gated && act >= 0) || (((uintptr_t)x | (uintptr_t)weight) & 15))
        return MRS_BAD_ARGUMENT;
    // warps that share a group's K: a warp then walks 8 steps of 64 elements and more, and asks for 16 KB ahead
    const int kw = k >= 4096 ? 8 : (k >= 2048 ? 4 : (k >= 1024 ? 2 : 1));
    const int cols = (gated ? 16 : 32) * (WARPS / kw);
    const dim3 grid(capacity / tile, (n + cols - 1) / cols);
#define MRS_MOE_FEW(GATED, NT, KW)                                                                                              \
    MRS_LAUNCH((moe_product_few_kernel<GATED, NT, KW>), grid, THREADS, 0, stream, (const bf16*)x, sorted_rows, tile_expert, \
               (const bf16*)weight, (bf16*)out, n, k, top, block, act)
#define MRS_MOE_FEW_KW(GATED, NT)                  \
    switch (kw) {                                  \
        case 8: MRS_MOE_FEW(GATED, NT, 8); break;  \
        case 4: MRS_MOE_FEW(GATED, NT, 4); break;  \
        case 2: MRS_MOE_FEW(GATED, NT, 2); break;  \
        default: MRS_MOE_FEW(GATED, NT, 1); break; \
    }
#define MRS_MOE_FEW_NT(GATED)                           \
    if (tile == 8) {                                    \
        MRS_MOE_FEW_KW(GATED, 1)                        \
    } else if (tile == 16) {                            \
        MRS_MOE_FEW_KW(GATED, 2)                        \
    } else {                                            \
        MRS_MOE_FEW_KW(GATED, 4)                        \
    }
    if (gated) {
        MRS_MOE_FEW_NT(true)
    } else {
        MRS_MOE_FEW_NT(false)
    }
#undef MRS_MOE_FEW_NT
#undef MRS_MOE_FEW_KW
#undef MRS_MOE_FEW
    MRS_RETURN_LAUNCH_STATUS();
}
