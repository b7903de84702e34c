// Latent attention for prompt portions on the tcgen05 tensor cores: every query head reads the same cache rows, a row being a
// latent of R elements and r rotated ones, and the latent is the value too.  -DMRS_LATENT=R (64, 128, 192 or 256)
// -DMRS_ROTARY=r (0, 32 or 64; R + r at most 288).
//
// A CTA works on one tile of 128 query rows, 128 / heads consecutive tokens of one request times all heads (the rows that a
// number of heads which does not divide 128 leaves over are zeroed, masked and never stored), and walks the keys in blocks of 64:
//   warp 0     fetches the queries and, page by page through the request's block table, the rows of every block with bulk
//              tensor copies into a ring of stages, groups of 64 elements in the 128-byte swizzle and 32 rotated ones in
//              the 64-byte one; a block is fetched once and read by both products;
//   warp 1     issues S = Q.K^T (K-major, R + r elements) into one of four score buffers in tensor memory;
//   warp 2     issues O += P.V: P from tensor memory, where it lies over its scores, V the same stage's first R elements as
//              the MN-major operand, O 128 x R in tensor memory;
//   warps 4-7  softmax, one thread a query row: scores from tensor memory, mask, running maximum and sum in float32,
//              probabilities back as pairs of bfloat16; the accumulator is rescaled only when a row's maximum grew by more
//              than 2^8, after the last P.V issued has been added.
// A weight of 0 does not keep a row out of P.V when the row is not finite (0 x inf is no number), so the rows that no query of the
// tile sees are zeros in shared memory: pages behind the last key or given back are copied from behind the cache, where the copy
// fills zeros, and the others' rows before the window and behind the last key are cleared once the scores were made.  (A row that
// one token of a tile sees reaches the tile's other tokens when it is not finite.)
// Two warps issue because a commit holds its issuer some 400 clocks and a block's MMAs run 1,300: 18 of 45 clocks for the
// scores (N 64), 4 of 128 for the values (N 256); at the full rate they would run 1,090.  Four stages and four score buffers let scores
// run ahead of softmax, which with its trips to tensor memory sets the pace: a block takes some 3,300 clocks (tensor pipe 33% of an
// SM's active clocks).  A prompt of 2,048 tokens, 16 heads, R 256, r 32, a window of 1,024: 50 us (mma.sync in tiles of 64 rows
// 197), 256 tiles on 148 SMs.
// Every wait is bounded (tma.cuh).
#include "tcgen05.cuh"

#if !defined(MRS_LATENT) || !defined(MRS_ROTARY)
#error "compile with -DMRS_LATENT=<elements of the latent> -DMRS_ROTARY=<rotated elements>"
#endif

namespace {

constexpr int R = MRS_LATENT, ROT = MRS_ROTARY, ROW = R + ROT;
static_assert(R % 64 == 0 && R >= 64 && R <= 256 && (ROT == 0 || ROT == 32 || ROT == 64) && ROW <= 288, "sizes that this kernel takes");
constexpr int BM = 128, BN = 64, STAGES = 4, THREADS = 256;
constexpr int CHUNKS = R / 64 + (ROT == 64 ? 1 : 0);            // groups of 64 elements of a row
constexpr bool TAIL = ROT == 32;                                 // and one of 32
constexpr int Q_CHUNK = BM * 128, Q_BYTES = CHUNKS * Q_CHUNK + (TAIL ? BM * 64 : 0);
constexpr int K_CHUNK = BN * 128, K_BYTES = CHUNKS * K_CHUNK + (TAIL ? BN * 64 : 0);
static_assert(K_BYTES % 1024 == 0 && Q_BYTES % 1024 == 0, "swizzled tiles begin at multiples of 1,024 bytes");
constexpr int TMEM_COLUMNS = 512, O_COLUMN = STAGES * BN;        // a score buffer a stage, then the accumulator
constexpr float RESCALE_THRESHOLD = 8.0f;                        // in powers of two
constexpr float LOG2E = 1.4426950408889634f;

struct Tile {
    int seq, first_token, tokens, pad;
};

struct Barriers {
    uint64_t q_full, k_full[STAGES], pv_done[STAGES], s_full[STAGES], p_ready[STAGES];
};
constexpr size_t SMEM_BYTES = 1024 + Q_BYTES + STAGES * K_BYTES + sizeof(Barriers) + 16;

// 2^x in one instruction of the special-function unit (2 ulp; -inf gives 0).
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// A tile of rows of 32 bfloat16 (64 bytes, rows of 8 in 512-byte groups, 16-byte pieces xor-ed with half the row: the 64-byte
// swizzle of a bulk tensor copy), K-major; `address` 512-byte aligned, plus 32 bytes for the second 16 elements of K.
__device__ __forceinline__ uint64_t umma_smem_desc_sw64(uint32_t address) {
    uint64_t desc = 0;
    desc |= (uint64_t)((address & 0x3FFFF) >> 4);
    desc |= (uint64_t)1 << 16;
    desc |= (uint64_t)(512 >> 4) << 32;
    desc |= (uint64_t)1 << 46;
    desc |= (uint64_t)4 << 61;
    return desc;
}

__global__ void __launch_bounds__(THREADS, 1) attention_latent_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap q_tail_map, const __grid_constant__ CUtensorMap k_map,
    const __grid_constant__ CUtensorMap k_tail_map, const int* __restrict__ positions, const int* __restrict__ block_table, int table_width,
    const Tile* __restrict__ tiles, bf16* __restrict__ out, const float* __restrict__ gate, const float* __restrict__ sinks, int heads,
    int page_size, int page_shift, int cache_pages, float scale_log2, int window) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* q_smem = smem;                                // [chunk][128 rows][64], then [128 rows][32]
    unsigned char* k_smem = q_smem + Q_BYTES;                    // [stage][chunk][64 keys][64], then [64 keys][32]
    Barriers* bars = reinterpret_cast<Barriers*>(k_smem + STAGES * K_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int used_rows = BM / heads * heads;                    // rows that a copy of queries fills
    if (used_rows < BM) {
        constexpr int PIECES = CHUNKS * 8 + (TAIL ? 4 : 0);      // sixteen bytes each
        for (int idx = threadIdx.x; idx < (BM - used_rows) * PIECES; idx += THREADS) {
            const int row = used_rows + idx / PIECES, piece = idx % PIECES;
            unsigned char* to = piece < CHUNKS * 8 ? q_smem + (piece >> 3) * Q_CHUNK + row * 128 + (piece & 7) * 16
                                                   : q_smem + CHUNKS * Q_CHUNK + row * 64 + (piece - CHUNKS * 8) * 16;
            *reinterpret_cast<uint4*>(to) = make_uint4(0, 0, 0, 0);
        }
        fence_async_shared();
    }
    if (threadIdx.x == 0) {
        mbar_init(&bars->q_full, 1);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&bars->k_full[s], 1);
            mbar_init(&bars->pv_done[s], 1);
            mbar_init(&bars->s_full[s], 1);
            mbar_init(&bars->p_ready[s], 4);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLUMNS);
        tmem_relinquish_alloc_permit();
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    tcgen05_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();                                                  // the tile list, queries and newest rows come from kernels before

    const Tile work = tiles[blockIdx.x];
    const int tokens = min(work.tokens, BM / heads);
    const int first_pos = tokens > 0 ? positions[work.first_token] : 0, key_end = first_pos + tokens;
    const int first_seen = window > 0 ? max(0, first_pos - window + 1) : 0, block_first = first_seen / BN;
    const int blocks = tokens > 0 ? (key_end + BN - 1) / BN - block_first : 0;
    const int* pages = block_table + (size_t)work.seq * table_width;

    if (warp == 0 && blocks > 0) {
        // ------------------------------------------------------------------ copies
        if (lane == 0) {
            mbar_arrive_expect_tx(&bars->q_full, used_rows * ROW * 2);
            for (int c = 0; c < CHUNKS; ++c) tma_load_3d(q_smem + c * Q_CHUNK, &q_map, &bars->q_full, c * 64, 0, work.first_token);
            if (TAIL) tma_load_3d(q_smem + CHUNKS * Q_CHUNK, &q_tail_map, &bars->q_full, 0, 0, work.first_token);
        }
        __syncwarp();
        const int rows_per_copy = min(page_size, BN), copies = BN / rows_per_copy;       // pages of a block: 1 to 8
        // lane p reads the number of a block's page p a block ahead; where there is none (keys past the end, a page that was given
        // back) the copy takes the page behind the cache's last: zeros
        auto page_of = [&](int j) {
            const int key = (block_first + j) * BN + lane * rows_per_copy;
            return (lane < copies && key < key_end) ? pages[key >> page_shift] : -1;
        };
        int next_page = page_of(0);
        constexpr int PARTS = CHUNKS + (TAIL ? 1 : 0);
        for (int j = 0; j < blocks; ++j) {
            const int s = j % STAGES, pages_here = next_page;
            if (j + 1 < blocks) next_page = page_of(j + 1);
            if (lane == 0) {
                if (j >= STAGES) mbar_wait(&bars->pv_done[s], ((j / STAGES) & 1) ^ 1);
                mbar_arrive_expect_tx(&bars->k_full[s], K_BYTES);
            }
            __syncwarp();                                        // the stage is free and the barrier armed
            unsigned char* stage = k_smem + s * K_BYTES;
            for (int base = 0; base < copies * PARTS; base += 32) {                       // a lane issues the copy of a part of a page
                const int idx = base + lane, p = idx % copies, c = idx / copies;
                const int page = __shfl_sync(0xffffffffu, pages_here, p);
                if (idx >= copies * PARTS) continue;
                const int key = (block_first + j) * BN + p * rows_per_copy, row = key & (page_size - 1), from = page < 0 ? cache_pages : page;
                if (c < CHUNKS) tma_load_3d(stage + c * K_CHUNK + p * rows_per_copy * 128, &k_map, &bars->k_full[s], c * 64, row, from);
                else tma_load_3d(stage + CHUNKS * K_CHUNK + p * rows_per_copy * 64, &k_tail_map, &bars->k_full[s], 0, row, from);
            }
            __syncwarp();
        }
    } else if (warp == 1 && blocks > 0) {
        // ------------------------------------------------------------------ scores
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc_bf16_f32(BM, BN);
        const uint32_t q_addr = smem_u32(q_smem);
        mbar_wait(&bars->q_full, 0);
        for (int j = 0; j < blocks; ++j) {
            const int s = j % STAGES;
            // the stage was fetched after P.V of block j - STAGES was done, so the score buffer of that block is free as well
            mbar_wait(&bars->k_full[s], (j / STAGES) & 1);
            __syncwarp();
            tcgen05_fence_after_sync();
            const uint32_t k_addr = smem_u32(k_smem + s * K_BYTES), s_tmem = tmem_base + s * BN;
            if (leader) {
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t q_desc = umma_smem_desc_sw128(q_addr + c * Q_CHUNK + k * 32), k_desc = umma_smem_desc_sw128(k_addr + c * K_CHUNK + k * 32);
                        if (c == 0 && k == 0) umma_bf16_first(s_tmem, q_desc, k_desc, idesc);
                        else umma_bf16_more(s_tmem, q_desc, k_desc, idesc);
                    }
                if (TAIL) {
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        umma_bf16_more(s_tmem, umma_smem_desc_sw64(q_addr + CHUNKS * Q_CHUNK + k * 32), umma_smem_desc_sw64(k_addr + CHUNKS * K_CHUNK + k * 32), idesc);
                }
                umma_commit(&bars->s_full[s]);
            }
            __syncwarp();
        }
    } else if (warp == 2 && blocks > 0) {
        // ------------------------------------------------------------------ values
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc_bf16_f32(BM, R, true);
        const uint32_t o_tmem = tmem_base + O_COLUMN;
        for (int j = 0; j < blocks; ++j) {
            const int s = j % STAGES;
            mbar_wait(&bars->k_full[s], (j / STAGES) & 1);
            mbar_wait(&bars->p_ready[s], (j / STAGES) & 1);
            __syncwarp();
            tcgen05_fence_after_sync();
            const uint32_t v_addr = smem_u32(k_smem + s * K_BYTES), p_tmem = tmem_base + s * BN;
            if (leader) {
#pragma unroll
                for (int k = 0; k < BN / 16; ++k)
                    umma_bf16_a_tmem(o_tmem, p_tmem + k * 8, umma_smem_desc_sw128_mn(v_addr + k * 2048, K_CHUNK), idesc, k > 0 || j > 0);
                umma_commit(&bars->pv_done[s]);
            }
            __syncwarp();
        }
    } else if (warp >= 4 && blocks > 0) {
        // ------------------------------------------------------------------ softmax, one thread a query row
        const int quarter = warp & 3, row = quarter * 32 + lane, rows = tokens * heads;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const int pos = row < rows ? first_pos + row / heads : -1;
        const int lowest = window > 0 ? pos - window + 1 : 0;    // first key this row sees
        float reference = -CUDART_INF_F, sum = 0.0f;             // the maximum that probabilities and the accumulator are scaled by
        for (int j = 0; j < blocks; ++j) {
            const int s = j % STAGES, key0 = (block_first + j) * BN;
            const uint32_t s_tmem = lane_base + s * BN;
            mbar_wait(&bars->s_full[s], (j / STAGES) & 1);
            __syncwarp();                                        // the loads below are collective: the warp goes on together
            tcgen05_fence_after_sync();
            // rows of the block that no query of the tile sees: before the window of the first, behind the last key
            const int live_from = max(0, first_seen - key0), live_to = min(BN, key_end - key0);
            if (live_from > 0 || live_to < BN) {                 // the scores have read the keys, and P.V waits for this warp below
                mbar_wait(&bars->k_full[s], (j / STAGES) & 1);   // complete: the copies' writes come before those here
                for (int idx = threadIdx.x - 128; idx < (R / 64) * BN * 8; idx += 128) {
                    const int c = idx / (BN * 8), row_of = idx / 8 % BN;     // a row's 128 bytes of a chunk stay its own in the swizzle
                    if (row_of < live_from || row_of >= live_to)
                        *reinterpret_cast<uint4*>(k_smem + s * K_BYTES + c * K_CHUNK + idx % (BN * 8) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_async_shared();
                __syncwarp();
            }
            const bool edge = key0 + BN - 1 > first_pos || (window > 0 && key0 < key_end - window);
            float x[BN];
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 32) tmem_load_32_async(s_tmem + c0, x + c0);
            tmem_load_wait();
            float part_max[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
            if (edge) {
#pragma unroll
                for (int c = 0; c < BN; ++c) {
                    const int key = key0 + c;
                    x[c] = (key <= pos && key >= lowest) ? x[c] : -CUDART_INF_F;
                    part_max[c & 3] = fmaxf(part_max[c & 3], x[c]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < BN; c += 8)
#pragma unroll
                    for (int k = 0; k < 4; ++k) part_max[k] = max3(part_max[k], x[c + k], x[c + 4 + k]);
            }
            const float block_max = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])) * scale_log2;
            float alpha = 1.0f;
            const bool moved = block_max > reference + RESCALE_THRESHOLD;
            if (moved) {
                alpha = fast_exp2(reference - block_max);        // 0 when the reference was -inf
                reference = block_max;
            }
            const float base = reference == -CUDART_INF_F ? 0.0f : reference;
            if (j > 0 && __any_sync(0xffffffffu, moved)) {
                mbar_wait(&bars->pv_done[(j - 1) % STAGES], ((j - 1) / STAGES) & 1);        // every P.V issued so far has been added
                __syncwarp();
                tcgen05_fence_after_sync();
#pragma unroll 4
                for (int c = 0; c < R; c += 16) {
                    float o[16];
                    tmem_load_16(lane_base + O_COLUMN + c, o);
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] *= alpha;
                    tmem_store_16(lane_base + O_COLUMN + c, o);
                }
            }
            float part_sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t packed[16];
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const float p0 = fast_exp2(fmaf(x[c0 + c], scale_log2, -base)), p1 = fast_exp2(fmaf(x[c0 + c + 1], scale_log2, -base));
                    part_sum[c & 2] += p0;
                    part_sum[(c & 2) + 1] += p1;
                    __nv_bfloat162 two = __floats2bfloat162_rn(p0, p1);
                    packed[c / 2] = *reinterpret_cast<uint32_t*>(&two);
                }
                tmem_store_16_words(s_tmem + c0 / 2, packed);    // over the scores
            }
            sum = sum * alpha + ((part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]));
            tmem_store_wait();
            tcgen05_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_ready[s]);
        }
        mbar_wait(&bars->pv_done[(blocks - 1) % STAGES], ((blocks - 1) / STAGES) & 1);
        __syncwarp();
        tcgen05_fence_after_sync();
        const int head = row % heads, token = work.first_token + row / heads;
        float inv = 0.0f;
        if (row < rows) {
            if (sinks) sum += exp2f(sinks[head] * LOG2E - reference);      // beyond a float's range the row's weights are 0 anyway
            inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            if (gate) inv *= gate[(size_t)token * heads + head];
        }
        bf16* dst = out + ((size_t)token * heads + head) * R;
#pragma unroll 2
        for (int c = 0; c < R; c += 32) {
            float o[32];
            tmem_load_32_async(lane_base + O_COLUMN + c, o);     // collective: rows past the tile's end drop what they read
            tmem_load_wait();
            if (row < rows) {
#pragma unroll
                for (int e = 0; e < 32; e += 8) {
                    uint32_t w[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        __nv_bfloat162 two = __floats2bfloat162_rn(o[e + 2 * p] * inv, o[e + 2 * p + 1] * inv);
                        w[p] = *reinterpret_cast<uint32_t*>(&two);
                    }
                    *reinterpret_cast<uint4*>(dst + c + e) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        }
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after_sync();
        tmem_dealloc(tmem_base, TMEM_COLUMNS);
    }
}

// Tensor maps of the step's queries [tokens, heads, R + r] for copies of (128 / heads tokens, rounded down) x (heads): groups of 64
// elements, and the last 32 (r = 32).
int query_maps(const void* q, long long tokens, int heads, CUtensorMap* maps) {
    if (tokens <= 0 || ((uintptr_t)q & 15)) return MRS_BAD_ARGUMENT;
    const uint64_t strides[2] = {(uint64_t)ROW * 2, (uint64_t)heads * ROW * 2};
    const uint64_t dims[3] = {(uint64_t)CHUNKS * 64, (uint64_t)heads, (uint64_t)tokens};
    const uint32_t box[3] = {64, (uint32_t)heads, (uint32_t)(BM / heads)};
    const int code = mrs_make_tensor_map_bf16(&maps[0], q, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (code != 0 || !TAIL) return code;
    const uint64_t tail_dims[3] = {32, dims[1], dims[2]};
    const uint32_t tail_box[3] = {32, box[1], box[2]};
    return mrs_make_tensor_map_bf16(&maps[1], (const bf16*)q + CHUNKS * 64, 3, tail_dims, strides, tail_box, CU_TENSOR_MAP_SWIZZLE_64B);
}

int page_shift_of(int page_size) {
    int shift = 0;
    while ((1 << shift) < page_size) ++shift;
    return (1 << shift) == page_size ? shift : -1;
}

}  // namespace

MRS_EXPORT int mrs_attention_latent_tc_rows() { return BM; }

// Tensor maps of the cache's rows [pages, 1, page_size, R + r] for copies of up to 64 rows of a page: groups of 64 elements, and the
// last 32 (r = 32).  `map_out`: two maps of 128 bytes, 64-byte aligned.
MRS_EXPORT int mrs_attention_latent_tc_cache_maps(const void* cache, long long pages, int page_size, void* map_out) {
    if (page_shift_of(page_size) < 0 || page_size < 8 || pages <= 0 || ((uintptr_t)cache & 15)) return MRS_BAD_ARGUMENT;
    CUtensorMap* maps = reinterpret_cast<CUtensorMap*>(map_out);
    const uint64_t strides[2] = {(uint64_t)ROW * 2, (uint64_t)page_size * ROW * 2};
    const uint64_t dims[3] = {(uint64_t)CHUNKS * 64, (uint64_t)page_size, (uint64_t)pages};
    const uint32_t box[3] = {64, (uint32_t)(page_size < BN ? page_size : BN), 1};
    int code = mrs_make_tensor_map_bf16(&maps[0], cache, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (code != 0 || !TAIL) return code;
    const uint64_t tail_dims[3] = {32, dims[1], dims[2]};
    const uint32_t tail_box[3] = {32, box[1], 1};
    return mrs_make_tensor_map_bf16(&maps[1], (const bf16*)cache + CHUNKS * 64, 3, tail_dims, strides, tail_box, CU_TENSOR_MAP_SWIZZLE_64B);
}

// Tiles of up to 128 / heads consecutive tokens of one request each: (sequence, first token, tokens, 0).  out [tokens, heads, R];
// `gate` [tokens, heads] or null multiplies a head's result; `sinks` [heads] or null: one more term exp(sink) in the denominator.
// `cache_pages`: the pages that the cache's maps cover.  The queries' maps are made here: q is another buffer in every call.
MRS_EXPORT int mrs_attention_latent_tc(const void* q, long long tokens, const void* cache_maps, const int* positions, const int* block_table,
                                       int table_width, const int* tiles, int num_tiles, void* out, const float* gate, const float* sinks,
                                       int heads, int page_size, long long cache_pages, float scale, int window, void* stream) {
    if (num_tiles <= 0) return 0;
    const int shift = page_shift_of(page_size);
    if (shift < 0 || page_size < 8 || cache_pages <= 0 || cache_pages >= 0x7fffffff || heads <= 0 || heads > BM ||
        !(scale > 0.0f) || window < 0 || ((uintptr_t)out & 15))
        return MRS_BAD_ARGUMENT;
    static PerDevice configured;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(attention_latent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    CUtensorMap queries[2];
    const int code = query_maps(q, tokens, heads, queries);
    if (code != 0) return code;
    const CUtensorMap* k = reinterpret_cast<const CUtensorMap*>(cache_maps);
    MRS_LAUNCH(attention_latent_kernel, num_tiles, THREADS, SMEM_BYTES, stream, queries[0], queries[TAIL ? 1 : 0], k[0], k[TAIL ? 1 : 0], positions, block_table,
               table_width, (const Tile*)tiles, (bf16*)out, gate, sinks, heads, page_size, shift, (int)cache_pages, scale * LOG2E, window);
    MRS_RETURN_LAUNCH_STATUS();
}

MRS_EXPORT int mrs_attention_latent_tc_take_error(unsigned int* word) { return mrs_take_error_word(word); }
// Mirrors the error word into a word of pinned host memory from now on.
MRS_EXPORT int mrs_attention_latent_tc_mirror_errors(unsigned int* host_word) { return mrs_set_error_mirror(host_word); }

MRS_EXPORT const char* mrs_attention_latent_tc_error_string(int code) {
    if (code == MRS_BAD_ARGUMENT) return "arguments outside what the kernel supports (page size below 8 or no power of two, more than 128 heads, unaligned rows)";
    if (code == MRS_TENSOR_MAP_FAILED) return "the driver refused the tensor map (address, sizes or strides)";
    return cudaGetErrorString((cudaError_t)code);
}
