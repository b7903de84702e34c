// float32 matrix product C[M,N] = A[M,K] . W[N,K]^T on the tcgen05 tensor cores, without giving up a bit of the inputs: every
// projection of the 32-bit path.
//
// A float32 is the sum of three bfloat16 (8 + 8 + 8 bits of its significand), so a product of two is nine products of bfloat16, each
// exact in float32.  Six of them are computed; the other three are at most 2^-24 of the product.  The MMAs add 32
// elements of K at a time into a fresh accumulator in tensor memory, small products first, and from there on a sum is ordinary
// float32 addition in registers: 32-element sums into one of four ranges of K, the four ranges in order.  An element's bits depend
// on K alone: not on M, not on the tile or the cut that the sizes chose, and a token's result does not change with what else is in the
// batch.  Results that the parts cannot be trusted with are computed again in float64 from the inputs: those that are no number or
// infinite, so that infinities and NaN are those of the sum of the products; those below 2^-100, whose smallest products lie near the end
// of float32's range (`store_column`; products down to 2^-120 come as close to 64 bits as ordinary ones, 2^-125 a little less); and those of
// rows with an element below some 2^-110, which has bits under bfloat16's range (2^-133), where the result is below 2^-60 or the other
// row has an element from 2^24 on (`mend_lost`).  Elsewhere K such bits are less than K 2^-48 of the result.  Looking for them takes 0.4 to
// 0.8 us of a call of up to 128 rows (K = 1,024 to 3,072), none that shows of 777; where one token has one, 777 rows take 102 us, where all
// have, 111.
//
// What bounds it: the workers' instructions (a float32 into three bfloat16 is some twenty-five instructions for four elements, and the
// sums), then shared memory (both matrices pass through it; parts of W lie in tensor memory, which took a step of 96 tokens from 0.80 to
// 0.70 us).  One turn of writers instead of two that overlap: 24 against 19 us for 8 rows in one CTA a tile.  Tiles of 128 tokens
// spill registers (90 against 63 us for 777 rows, N 4,096, K 1,024).
// The kernel from a cold L2, before (multiply-adds on the CUDA cores) and now: N 4,096, K 1,024: 1 row 12.0 -> 12.3 us, 8 rows 12.3 -> 12.6, 64
// rows 23 -> 13.8, 128 rows 38 -> 19, 777 rows 171 -> 67; N 1,024, K 2,048: 8 rows 18.4 -> 14.3, 777 rows 101 -> 36; N 6,144, K 1,024, 777
// rows 267 -> 97.  Error against 64 bits (relative, normal inputs): K = 1,024 5.7e-7 -> 0.9e-7, K = 3,072 1.0e-6 -> 1.2e-7.
//             (reference: cuBLAS, kernels/src/lib.rs:298-321)
#include <cooperative_groups.h>

#include <cfloat>

#include "parts3.cuh"
#include "tcgen05.cuh"

namespace {
namespace cg = cooperative_groups;

constexpr int BM = 128;              // weight rows of a tile: the M of the MMA, a lane of tensor memory each
constexpr int BK = 32;               // elements of K of a step: 64 bytes of bfloat16, one swizzled row
constexpr int RANGES = 4;            // of K, added in order
constexpr int WORKERS = 512, TURNS = 2, WRITERS = WORKERS / TURNS, THREADS = WORKERS + 32 * TURNS;
constexpr int PARTS = 3;             // bfloat16 of a float32

// Of a step: a weight row's parts in tensor memory (A of the MMA), the tokens' in shared memory (B); STAGES of both, two
// accumulators, and a ring of float32 pieces on their way.
template <int BN>
struct Tile {
    static constexpr int W_MINE = BM * BK / 4 / WRITERS, A_PIECES = BN * BK / 4, A_MINE = (A_PIECES + WRITERS - 1) / WRITERS;    // sixteen bytes each
    static constexpr int W_BYTES = BM * BK * 4, RAW_BYTES = W_BYTES + A_PIECES * 16;
    static constexpr int PART_BYTES = BN * BK * 2, STAGE_BYTES = PARTS * PART_BYTES;
    static constexpr int STAGES = BN == 96 ? 3 : 4, DEPTH = BN >= 64 ? 2 : 4;                         // DEPTH: of each turn's steps
    static constexpr int COLUMNS = BN / 4;                                                            // of a thread's row
    static constexpr uint32_t W_COLUMNS = PARTS * BK / 2, TMEM = 2 * BN + STAGES * W_COLUMNS <= 256 ? 256 : 512;
    static constexpr int SUM_BYTES = BM * BN * 4;                                                     // a range's sums
    static constexpr size_t SMEM = 1024 + STAGES * (size_t)STAGE_BYTES + TURNS * (size_t)DEPTH * RAW_BYTES + 2 * STAGES * sizeof(uint64_t) + 16;
    static_assert(SMEM <= 232448 && 2 * SUM_BYTES <= STAGES * STAGE_BYTES + TURNS * DEPTH * RAW_BYTES, "shared memory of an SM");
    static_assert(2 * BN + STAGES * W_COLUMNS <= TMEM, "tensor memory of an SM");
};

template <int PIECE>
__device__ __forceinline__ void copy_piece(uint32_t to, const float* from, bool live) {
    if (PIECE == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(from), "r"(live ? 16 : 0));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to), "l"(from), "r"(live ? 4 : 0));
}

// Rows of 64 bytes in groups of 8, sixteen-byte pieces xor-ed with half the row's number: the 64-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t address) {
    return (uint64_t)((address & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

__device__ __forceinline__ void tmem_load_4_async(uint32_t address, float* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(address) : "memory");
}
__device__ __forceinline__ void tmem_load_8_async(uint32_t address, float* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(address) : "memory");
}
template <int C>
__device__ __forceinline__ void add_columns(uint32_t address, float (&sum)[C]) {
    constexpr int STEP = C % 16 == 0 ? 16 : C < 8 ? C : 8;
#pragma unroll
    for (int c = 0; c < C; c += STEP) {
        float v[STEP];
        if constexpr (STEP == 16) tmem_load_16_async(address + c, v);
        else if constexpr (STEP == 8) tmem_load_8_async(address + c, v);
        else tmem_load_4_async(address + c, v);
        tmem_load_wait();
#pragma unroll
        for (int e = 0; e < STEP; e += 2) add_pair(sum[c + e], sum[c + e + 1], v[e], v[e + 1]);
    }
}

// 16 lanes x 8 columns: a thread has two columns, 2 (lane % 4) and the next, of lanes lane / 4 and 8 further.
__device__ __forceinline__ void tmem_store_16x8(uint32_t address, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The whole warp: a . w over K in float64.
__device__ __noinline__ float exact_dot(const float* __restrict__ a, const float* __restrict__ w, int K) {
    double sum = 0.0;
    for (int k = threadIdx.x & 31; k < K; k += 32) sum = fma((double)a[k], (double)w[k], sum);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return (float)sum;
}

// What a row's elements say of its results: some have bits under bfloat16's range; some are large enough for the other row's such bits
// to show.  The whole warp.
constexpr unsigned LOST = 1, LARGE = 2;
constexpr float LEAST = 0x1p-100f, LEAST_OF_LOST = 0x1p-60f;
__device__ __noinline__ unsigned row_facts(const float* __restrict__ row, int K) {
    uint32_t rest = 0;
    float top = 0.0f;
    for (int k = threadIdx.x & 31; k < K; k += 32) {
        float x = row[k], none = 0.0f;
        uint32_t parts[PARTS];
        top = fmaxf(top, fabsf(x));
        three_parts(x, none, parts);
        rest |= __float_as_uint(x);
    }
    return (__any_sync(0xffffffffu, rest & LOST_BITS) ? LOST : 0) | (__any_sync(0xffffffffu, top >= 0x1p24f) ? LARGE : 0);
}

// The tile's results of LOST rows, once they are stored: 128 weight rows from n0 on, `tokens` tokens from m0 on.  The facts are read from the
// rows themselves over the whole of K, so that a result depends on its own two rows alone.  The whole block; `facts`: BM + tokens.
__device__ __noinline__ void mend_lost(unsigned char* facts, const float* __restrict__ A, const float* __restrict__ W, float* C, int m0, int n0,
                                       int tokens, int M, int N, int K) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tokens = min(tokens, M - m0);
    for (int r = warp; r < BM + tokens; r += THREADS / 32) {
        const unsigned f = r >= BM ? row_facts(A + (size_t)(m0 + r - BM) * K, K) : n0 + r < N ? row_facts(W + (size_t)(n0 + r) * K, K) : 0;
        if (lane == 0) facts[r] = (unsigned char)f;
    }
    __syncthreads();                                         // the facts are there, and the results
    for (int task = warp; task < tokens * (BM / 32); task += THREADS / 32) {
        const int row = task % (BM / 32) * 32 + lane, n = n0 + row, m = m0 + task / (BM / 32);
        const unsigned w = facts[row], a = facts[BM + m - m0];
        const bool lost = (w | a) & LOST, shows = ((w & LARGE) && (a & LOST)) || ((w & LOST) && (a & LARGE));
        unsigned odd = __ballot_sync(0xffffffffu, n < N && lost && (shows || fabsf(C[(size_t)m * N + n]) < LEAST_OF_LOST));
        while (odd) {
            const int of = __ffs(odd) - 1;
            odd &= odd - 1;
            const float v = exact_dot(A + (size_t)m * K, W + (size_t)__shfl_sync(0xffffffffu, n, of) * K, K);
            if (lane == of) C[(size_t)m * N + n] = v;
        }
    }
}

// Stores the warp's 32 weight rows' results for one token; those that are no number, infinite or too small are computed again.
__device__ __forceinline__ void store_column(float v, const float* __restrict__ A, const float* __restrict__ W, float* C, int m, int n, int M, int N,
                                             int K) {
    if (m >= M) return;                                      // the same for the whole warp
    const float size = fabsf(v);
    unsigned odd = __ballot_sync(0xffffffffu, n < N && !(size <= FLT_MAX && size >= LEAST) && v != 0.0f);
    while (odd) {
        const int lane = __ffs(odd) - 1;
        odd &= odd - 1;
        const float again = exact_dot(A + (size_t)m * K, W + (size_t)__shfl_sync(0xffffffffu, n, lane) * K, K);
        if ((int)(threadIdx.x & 31) == lane) v = again;
    }
    if (n < N) C[(size_t)m * N + n] = v;
}

// A CTA has a tile of 128 weight rows x BN tokens, or (a cluster of 2 or 4) some of the tile's ranges of K.  Sixteen warps copy the
// float32 rows into shared memory (cp.async; a thread reads back only what it copied itself), write their parts as bfloat16 tiles
// and add finished accumulators to their sums; two more warps issue the MMAs of every other step.
// VEC: sixteen-byte copies (K a multiple of 4, both matrices on 16-byte boundaries), else four-byte ones.
template <int BN, bool VEC>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* C, int M,
                                                              int N, int K, int m_tiles, int cut) {
    using T = Tile<BN>;
    constexpr int STAGES = T::STAGES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* raw = smem + STAGES * T::STAGE_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(raw + TURNS * T::DEPTH * T::RAW_BYTES);       // a stage's parts are written
    uint64_t* done = full + STAGES;                                                    // a stage's MMAs have finished
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + STAGES);

    __shared__ unsigned char facts[BM + BN];                                           // of the tile's weight rows, then of its tokens
    __shared__ int met_lost;                                                           // read by the cluster

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x / cut, rank = blockIdx.x % cut;
    const int m0 = tile % m_tiles * BN, n0 = tile / m_tiles * BM;
    const int steps = (K + BK - 1) / BK, range = (steps + RANGES - 1) / RANGES, ranges = RANGES / cut;
    const int first = min(rank * ranges * range, steps), count = min((rank + 1) * ranges * range, steps) - first;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], WORKERS / 32);
            mbar_init(&done[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == WORKERS / 32) {
        tmem_alloc(tmem_slot, T::TMEM);
        tmem_relinquish_alloc_permit();
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    tcgen05_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();

    const int row = (warp & 3) * 32 + lane, column0 = (warp >> 2) * T::COLUMNS;        // of a worker's sums
    if (warp >= WORKERS / 32) {
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc_bf16_f32(BM, BN);
        for (int i = warp - WORKERS / 32; i < count; i += TURNS) {
            const int s = i % STAGES;
            mbar_wait(&full[s], i / STAGES & 1);
            tcgen05_fence_after_sync();
            const uint32_t stage = smem_u32(smem + s * T::STAGE_BYTES), parts = tmem_base + 2 * BN + s * T::W_COLUMNS, d = tmem_base + (i & 1) * BN;
            if (leader) {
                // (part of W, part of A): products of 2^-16, then 2^-8, then the leading parts
                constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
#pragma unroll
                for (int j = 0; j < 6; ++j) {
                    const uint32_t w = parts + order[j][0] * (BK / 2);
                    const uint64_t a = smem_desc_sw64(stage + order[j][1] * T::PART_BYTES);
                    umma_bf16_a_tmem(d, w, a, idesc, j > 0);
                    umma_bf16_a_tmem(d, w + 8, a + 2, idesc, true);
                }
                umma_commit(&done[s]);
            }
            __syncwarp();
        }
    }
    uint32_t rest = 0;                                       // what three parts leave of this thread's elements: LOST_BITS of it
    float now[T::COLUMNS], before[T::COLUMNS];               // the running range, the ranges before it (one CTA a tile: their sum)
#pragma unroll
    for (int c = 0; c < T::COLUMNS; ++c) now[c] = before[c] = 0.0f;
    if (warp < WORKERS / 32) {
        // A step's writers: of W, sixteen bytes of rows lane / 4 + 8 j of the warp's lanes of tensor memory, half of the step's K a
        // warp; of A, sixteen bytes of rows line + 32 j.
        const int turn = tid / WRITERS, writer = tid % WRITERS, half = writer / (WRITERS / 2), line = writer >> 3;
        const int w_line = (warp & 3) * 32 + (lane >> 2), w_k = half * 16 + (lane & 3) * 4, a_k = (writer & 7) * 4;
        const uint32_t to_w = tmem_base + 2 * BN + ((uint32_t)((warp & 3) * 32) << 16) + half * 8;
        const uint32_t to_a = smem_u32(smem) + line * 64 + (((a_k >> 3) ^ ((line >> 1) & 3)) << 4) + (a_k & 4) * 2;
        raw += turn * (T::DEPTH * T::RAW_BYTES) + writer * 16;
        const float* w_tile = W + (size_t)n0 * K;
        const float* a_tile = A + (size_t)m0 * K;
        const int w_last = N - 1 - n0, a_last = M - 1 - m0;  // rows beyond the last repeat it and are not stored
        int issued = turn, issue_slot = 0;                   // the next step to ask for
        auto copy = [&](uint32_t to, const float* row, int k) {
            if (VEC) {
                copy_piece<16>(to, row + (k < K ? k : 0), k < K);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) copy_piece<4>(to + 4 * e, row + (k + e < K ? k + e : 0), k + e < K);
            }
        };
        auto issue = [&]() {
            if (issued < count) {
                const int k0 = (first + issued) * BK;
                const uint32_t to = smem_u32(raw) + issue_slot * T::RAW_BYTES;
#pragma unroll
                for (int j = 0; j < T::W_MINE; ++j) copy(to + j * WRITERS * 16, w_tile + (size_t)min(w_line + 8 * j, w_last) * K, k0 + w_k);
#pragma unroll
                for (int j = 0; j < T::A_MINE; ++j)
                    if (T::A_PIECES % WRITERS == 0 || writer + j * WRITERS < T::A_PIECES)
                        copy(to + T::W_BYTES + j * WRITERS * 16, a_tile + (size_t)min(line + WRITERS / 8 * j, a_last) * K, k0 + a_k);
            }
            asm volatile("cp.async.commit_group;\n" ::);
            issued += TURNS;
            issue_slot = issue_slot + 1 == T::DEPTH ? 0 : issue_slot + 1;
        };
        for (int i = 0; i < T::DEPTH - 1; ++i) issue();
        bool kept = false;
        int stage = 0, slot = 0, left = range;               // stage of step i, slot of this turn's next step, steps to a range's end
        int done_stage = 0;                                  // of step i - 2
        uint32_t parity = 0;
#pragma unroll 1
        for (int i = 0; i < count + 2; ++i) {
            if (i < count && i % TURNS == turn) {            // the stage's last step, i - STAGES, is over: waited for below
                issue();
                asm volatile("cp.async.wait_group %0;\n" ::"n"(T::DEPTH - 1) : "memory");
                const unsigned char* from = raw + slot * T::RAW_BYTES;
                const uint32_t w = to_w + stage * T::W_COLUMNS, a = to_a + stage * T::STAGE_BYTES;
#pragma unroll
                for (int j = 0; j < T::W_MINE; j += 2) {     // 16 lanes
                    float4 x = *reinterpret_cast<const float4*>(from + j * WRITERS * 16), y = *reinterpret_cast<const float4*>(from + (j + 1) * WRITERS * 16);
                    uint32_t x0[PARTS], x1[PARTS], y0[PARTS], y1[PARTS];
                    three_parts(x.x, x.y, x0), three_parts(x.z, x.w, x1), three_parts(y.x, y.y, y0), three_parts(y.z, y.w, y1);
                    rest |= left_bits(x) | left_bits(y);
#pragma unroll
                    for (int part = 0; part < PARTS; ++part)
                        tmem_store_16x8(w + ((uint32_t)(8 * j) << 16) + part * (BK / 2), x0[part], x1[part], y0[part], y1[part]);
                }
#pragma unroll
                for (int j = 0; j < T::A_MINE; ++j)
                    if (T::A_PIECES % WRITERS == 0 || writer + j * WRITERS < T::A_PIECES) {
                        float4 x = *reinterpret_cast<const float4*>(from + T::W_BYTES + j * WRITERS * 16);
                        uint32_t low[PARTS], high[PARTS];
                        three_parts(x.x, x.y, low), three_parts(x.z, x.w, high);
                        rest |= left_bits(x);
#pragma unroll
                        for (int part = 0; part < PARTS; ++part)
                            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a + part * T::PART_BYTES + j * (WRITERS / 8 * BK * 2)), "r"(low[part]), "r"(high[part]));
                    }
                fence_async_shared();
                tmem_store_wait();
                slot = slot + 1 == T::DEPTH ? 0 : slot + 1;
            }
            if (i >= 2) {                                    // step i - 2 is over: frees its stage and its accumulator
                mbar_wait(&done[done_stage], parity);
                __syncwarp();
                tcgen05_fence_after_sync();
                add_columns(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (i & 1) * BN + column0, now);
                if (++done_stage == STAGES) {
                    done_stage = 0;
                    parity ^= 1;
                }
                if (--left == 0 || i - 1 == count) {         // a range's end
                    left = range;
                    if (cut == 1 || (cut == 2 && !kept)) {
                        kept = true;
#pragma unroll
                        for (int c = 0; c < T::COLUMNS; ++c) {
                            before[c] += now[c];
                            now[c] = 0.0f;
                        }
                    }
                }
            }
            if (i < count) {
                // all warps arrive: the step's MMAs write an accumulator that each of them has read its columns of
                tcgen05_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[stage]);
            }
            if (++stage == STAGES) stage = 0;
        }
    }
    int some = __syncthreads_or(rest & LOST_BITS), mine = 0, of_mine = BN;     // some thread met LOST bits; this CTA's tokens
    if (cut == 1) {
        if (warp < WORKERS / 32) {
#pragma unroll
            for (int c = 0; c < T::COLUMNS; ++c) store_column(before[c], A, W, C, m0 + column0 + c, n0 + row, M, N, K);
        }
    } else {
        // every CTA leaves its ranges' sums in its shared memory and adds up a slice of the columns
        cg::cluster_group cluster = cg::this_cluster();
        if (tid == 0) met_lost = some;
        float* sums = reinterpret_cast<float*>(smem);
        if (warp < WORKERS / 32) {
#pragma unroll
            for (int c = 0; c < T::COLUMNS; ++c) {
                const int at = (column0 + c) * BM + row;
                sums[at] = cut == 2 ? before[c] : now[c];
                if (cut == 2) sums[BM * BN + at] = now[c];
            }
        }
        cluster.sync();
        of_mine = BN / cut, mine = rank * of_mine;
        some = 0;
#pragma unroll
        for (int r = 0; r < RANGES; ++r) some |= *cluster.map_shared_rank(&met_lost, r % cut);      // wanted only behind the columns
        if (warp < WORKERS / 32) {
            for (int c = mine + (warp >> 2); c < mine + of_mine; c += WORKERS / BM) {
                float v = 0.0f;
#pragma unroll
                for (int r = 0; r < RANGES; ++r) v += cluster.map_shared_rank(sums, r / ranges)[r % ranges * (BM * BN) + c * BM + row];
                store_column(v, A, W, C, m0 + c, n0 + row, M, N, K);
            }
        }
        cluster.sync();                                      // no CTA leaves while another reads its sums
    }
    if (some && m0 + mine < M) mend_lost(facts, A, W, C, m0 + mine, n0, of_mine, M, N, K);
    tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == WORKERS / 32) {
        tcgen05_fence_after_sync();
        tmem_dealloc(tmem_base, T::TMEM);
    }
}

template <int BN, bool VEC>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int cut, void* stream) {
    static PerDevice configured;
    auto kernel = gemm_f32_kernel<BN, VEC>;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile<BN>::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    const long long m_tiles = ((long long)M + BN - 1) / BN, ctas = m_tiles * (((long long)N + BM - 1) / BM) * cut;
    if (ctas > 0x7fffffffll) return MRS_BAD_ARGUMENT;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)ctas);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = Tile<BN>::SMEM;
    config.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attributes[2];
    static const bool plain = getenv("MRS_PLAIN_LAUNCH") != nullptr;
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = cut;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = plain ? 1 : 2;
    const cudaError_t e = cudaLaunchKernelEx(&config, kernel, A, W, C, M, N, K, (int)m_tiles, cut);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

template <bool VEC>
int launch_tile(int bn, const float* A, const float* W, float* C, int M, int N, int K, int cut, void* stream) {
    switch (bn) {
        case 16: return launch<16, VEC>(A, W, C, M, N, K, cut, stream);
        case 32: return launch<32, VEC>(A, W, C, M, N, K, cut, stream);
        case 64: return launch<64, VEC>(A, W, C, M, N, K, cut, stream);
        default: return launch<96, VEC>(A, W, C, M, N, K, cut, stream);
    }
}

}  // namespace

MRS_EXPORT int mrs_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return MRS_BAD_ARGUMENT;
    const bool vec = K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    // A round of CTAs takes a line over a CTA's steps, in microseconds, measured alone at N = 1,024 to 6,144, K = 1,024 to 3,072 and
    // M = 1 to 777 (within a tenth nearly everywhere): 8 rows of N 4,096, K 1,024 18.7, 13.1 and 11.0 us with 1, 2 and 4 CTAs a tile; 777
    // rows 63 us with tiles of 96 tokens in two rounds, 73 with 64 in three.  Clusters of 4 do not come onto every SM.
    constexpr int widths[4] = {16, 32, 64, 96};
    constexpr double fixed[4] = {6.0, 6.5, 8.0, 9.3}, each[4] = {0.43, 0.45, 0.57, 0.70};
    const int sms = mrs_sm_count(), range = ((K + BK - 1) / BK + RANGES - 1) / RANGES;
    double best = 0.0;
    int bn = 0, cut = 1;
    for (int i = 0; i < 4; ++i) {
        const long long tiles = ((long long)N + BM - 1) / BM * (((long long)M + widths[i] - 1) / widths[i]);
        for (int c = 1; c <= RANGES; c *= 2) {
            const long long held = c == 4 ? sms * 7 / 8 / 4 * 4 : sms / c * c, rounds = held ? (tiles * c + held - 1) / held : tiles * c;
            const double time = (double)rounds * (fixed[i] + each[i] * (RANGES / c) * range);
            if (bn == 0 || time < best) best = time, bn = widths[i], cut = c;
        }
    }
    return vec ? launch_tile<true>(bn, A, W, C, M, N, K, cut, stream) : launch_tile<false>(bn, A, W, C, M, N, K, cut, stream);
}

MRS_EXPORT int mrs_gemm_f32_take_error(unsigned int* word) { return mrs_take_error_word(word); }
// Mirrors the error word into a word of pinned host memory from now on.
MRS_EXPORT int mrs_gemm_f32_mirror_errors(unsigned int* host_word) { return mrs_set_error_mirror(host_word); }
