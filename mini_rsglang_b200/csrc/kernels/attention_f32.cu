// Paged causal grouped-query attention in float32 for heads of a multiple of 4 elements: the attention of the 32-bit path.
// (attention_simt.cu takes the other sizes, and bfloat16.)                                   (reference: ops.cu:101-147)
//
// A block takes one tile of rows, up to 64 (token, head of one key/value head's group) pairs of consecutive tokens of one
// request, and walks their keys in blocks of 32 through shared memory: scores, then the row's maximum, exponentials and sum,
// then the weighted values, all float32 multiply-adds.  The copies of the next keys run beside the exponentials and the values,
// those of the next values beside the scores.  Tiles begin where a request's position is a multiple of the tile's tokens, found
// by each block from the step's positions, so that no list has to be planned.
//
// A row's result has the same bits however its request is cut into steps and whatever lies beside it: a score is one chain over
// d in ascending order, blocks of keys begin at multiples of 32, keys are taken in chunks that begin at multiples of CHUNK, and
// the chunks' results (maximum, sum, weighted values) are joined in ascending order by the same arithmetic whether one block
// walked them all or each had a block of its own (few rows with long contexts; a second kernel then joins them).
//
// Heads of 128 elements run on the tensor cores (below).  The other sizes: bound by the multiply-add pipe and shared memory for prompts;
// for decoded tokens by a tile's chain of page numbers, keys, scores, weights and values.  Up to 8 rows take steps of two blocks: a warp
// a row and a block of scores, a column a thread, keys of two steps and values of one ahead, page numbers three.  Chunks of 256 keys, with
// the joining, from a cold L2, 16 query and 8 key/value heads of 64 and of 256: of 512, 400 tokens walk 13 blocks in a row on a third of
// the SMs (52 and 139 us against 50 and 105), 20 tokens behind 980 take 49 and 113 against 29 and 64; of 128, the joining outweighs it
// (880 tokens behind 1,420 361 and 1,319 against 322 and 1,153).
#include "parts3.cuh"
#include "tcgen05.cuh"

#include <type_traits>

namespace {

constexpr int ROWS = 64, KEYS = 32, CHUNK = 256, THREADS = 256, FEW_ROWS = 8;
constexpr int P_PITCH = KEYS + 4;

constexpr int FEW_KEYS = 2 * KEYS, FEW_PITCH = FEW_KEYS + 4, AHEAD = 4;

// shared memory of the walks over many and over few rows, each with the running sums of the chunks that !SPLIT keeps
template <int D, bool SPLIT> constexpr int smem_floats() {
    const int many = ROWS * (D + 4) + KEYS * (D + 4) + KEYS * D + ROWS * P_PITCH + (SPLIT ? 0 : ROWS * D);
    const int few = FEW_ROWS * (D + 4) + 2 * FEW_KEYS * (D + 4) + FEW_KEYS * D + FEW_ROWS * FEW_PITCH + (SPLIT ? 0 : FEW_ROWS * D);
    return many > few ? many : few;
}

__device__ __forceinline__ void copy16(float* to, const float* from, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(live ? 16 : 0));
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// exp(a - b) where a may be -inf (nothing there): 0
__device__ __forceinline__ float ratio(float a, float b) { return a == -CUDART_INF_F ? 0.0f : expf(a - b); }
// what both ways of joining chunks compute for an element
__device__ __forceinline__ float join(float total, float keep, float part, float take) { return fmaf(part, take, total * keep); }

struct Args {
    const float *q, *k, *v;
    const int *positions, *seq_of_token, *table;
    float *out, *part_o, *part_ml;               // [tokens, nq, chunks, d], [tokens, nq, chunks, 2]
    int tokens, nq, nkv, d, page_size, table_width, window, tile_tokens, chunks;
    float scale;
};

// The first token of the step's `tile`-th tile from the end (late tiles walk the most keys: they start first), its tokens in found[1];
// -1: there are fewer tiles.  The whole block; what it used of shared memory before has been read.
template <int BLOCK>
__device__ int find_tile(const Args& A, int tile, int* found, int* warp_count) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto begins = [&](int t) {
        if (t >= A.tokens) return true;
        const int pos = A.positions[t];
        return t == 0 || pos % A.tile_tokens == 0 || A.seq_of_token[t] != A.seq_of_token[t - 1] || pos != A.positions[t - 1] + 1;
    };
    __syncthreads();
    if (tid == 0) found[0] = -1;
    __syncthreads();
    int before = 0;
    for (int base = (A.tokens - 1) / BLOCK * BLOCK; base >= 0; base -= BLOCK) {
        const int t = base + tid;
        const bool first = t < A.tokens && begins(t);
        const int here = __syncthreads_count(first);
        if (before + here > tile) {
            const int wanted = here - 1 - (tile - before);               // from the front of these
            const unsigned mask = __ballot_sync(0xffffffffu, first);
            if (lane == 0) warp_count[warp] = __popc(mask);
            __syncthreads();
            int ahead = 0;
            for (int w = 0; w < warp; ++w) ahead += warp_count[w];
            if (first && ahead + __popc(mask & ((1u << lane) - 1u)) == wanted) found[0] = t;
            break;
        }
        before += here;
    }
    __syncthreads();
    const int t0 = found[0];
    if (t0 < 0) return -1;
    if (tid < 32) {                                          // tokens of the tile
        int count = A.tile_tokens;
        for (int i = 1 + lane; i < A.tile_tokens; i += 32)
            if (begins(t0 + i)) { count = i; break; }
        count = __reduce_min_sync(0xffffffffu, count);
        if (lane == 0) found[1] = count;
    }
    __syncthreads();
    return t0;
}

// SPLIT: a block takes one chunk (blockIdx.z) of its tiles' keys and leaves its parts in part_o and part_ml; otherwise all of them.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(THREADS, D <= 128 ? 2 : 1) attention_f32_kernel(const Args A) {
    constexpr int PITCH = D + 4, COLS = D / 16;          // columns of the output a thread has (rows in fours)
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;                                   // [ROWS][PITCH]
    float* k_s = q_s + ROWS * PITCH;                     // [KEYS][PITCH]
    float* v_s = k_s + KEYS * PITCH;                     // [KEYS][D]
    float* p_s = v_s + KEYS * D;                         // [ROWS][P_PITCH]
    __shared__ float keep_s[ROWS], take_s[ROWS];
    __shared__ long long place_s[AHEAD * FEW_KEYS];       // where cached rows begin, of the steps (few rows) or blocks that come next; -1: not seen
    __shared__ int found[2], warp_count[THREADS / 32];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = blockIdx.y, group = A.nq / A.nkv, d = A.d;
    for (int tile = blockIdx.x;; tile += gridDim.x) {
        const int t0 = find_tile<THREADS>(A, tile, found, warp_count);
        if (t0 < 0) return;
        const int tokens = found[1], rows = tokens * group;
        const int pos0 = A.positions[t0], end_key = pos0 + tokens;
        int begin = A.window > 0 ? max(0, pos0 + 1 - A.window) : 0, end = end_key;       // keys that some row sees
        if (SPLIT) {
            begin = max(begin, (int)blockIdx.z * CHUNK);     // keys beyond the last chunk that was planned go with it
            if ((int)blockIdx.z + 1 < A.chunks) end = min(end, ((int)blockIdx.z + 1) * CHUNK);
            if (begin >= end) continue;
        }
        const int* pages = A.table + (size_t)A.seq_of_token[t0] * A.table_width;
        // row r: token t0 + r / group, head g * group + r % group
        for (int i = tid; i < rows * (D / 4); i += THREADS) {
            const int r = i / (D / 4), c = i % (D / 4) * 4;
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (c < d) x = *reinterpret_cast<const float4*>(A.q + ((size_t)(t0 + r / group) * A.nq + g * group + r % group) * d + c);
            *reinterpret_cast<float4*>(q_s + r * PITCH + c) = x;
        }
        // where the row of key p begins in the cache.  The page's number comes from memory: it is asked for a step before the
        // copies want it (a lookup in front of every copy was half the time of a block)
        auto place_of = [&](int p) -> long long {
            if (p < begin || p >= end) return -1;
            return (((long long)pages[p / A.page_size] * A.nkv + g) * A.page_size + p % A.page_size) * d;
        };
        // rows to shared memory, zeros for those that are not seen
        auto fetch = [&](auto count, const float* __restrict__ cache, float* to, int pitch, const long long* places) {
            constexpr int MINE = decltype(count)::value * (D / 4) / THREADS;
            long long place[MINE];
#pragma unroll
            for (int i = 0; i < MINE; ++i) place[i] = places[(tid + i * THREADS) / (D / 4)];
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
                const int j = (tid + i * THREADS) / (D / 4), c = (tid + i * THREADS) % (D / 4) * 4;
                const bool live = place[i] >= 0 && c < d;
                copy16(to + j * pitch + c, cache + (live ? place[i] + c : 0), live);
            }
            copies_commit();
        };
        constexpr std::integral_constant<int, KEYS> block_rows;
        constexpr std::integral_constant<int, FEW_KEYS> step_rows;
        const bool few = rows <= FEW_ROWS;
        float* total_s = few ? smem + FEW_ROWS * PITCH + 2 * FEW_KEYS * PITCH + FEW_KEYS * D + FEW_ROWS * FEW_PITCH : p_s + ROWS * P_PITCH;      // !SPLIT: [4 * COLS][THREADS], few rows [FEW_OWN][THREADS]: a thread's own
        // scores: a warp has 16 rows x 16 keys, lanes 4 x 8; few rows: a warp a row and a block, a lane a key
        const int s_row = (warp >> 1) * 16 + (lane >> 3), s_key = (warp & 1) * 16 + (lane & 7);
        // values: a thread has rows o_row .. o_row + 3 and COLS columns in pieces of 4, 64 apart; few rows: a column of every
        // FEW_STEP-th row
        const int o_row = (warp * 2 + (lane >> 4)) * 4, o_col = (lane & 15) * 4;
        constexpr int FEW_STEP = THREADS / D, FEW_OWN = FEW_ROWS / FEW_STEP;
        const int f_col = tid % D, f_row = tid / D;
        float o[4][COLS];                                // few rows: o_few[i] is row f_row + i * FEW_STEP
        float* o_few = &o[0][0];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                o[i][c] = 0.0f;
                if (!SPLIT && (!few || i * COLS + c < FEW_OWN)) total_s[(i * COLS + c) * THREADS + tid] = 0.0f;
            }
        // a row's maximum and sum: four threads a row, eight keys of a block each
        const int m_row = tid >> 2, m_key = (tid & 3) * 8;
        float m = -CUDART_INF_F, l = 0.0f, m_all = -CUDART_INF_F, l_all = 0.0f;
        const int m_pos = m_row < rows ? pos0 + m_row / group : -1;      // rows beyond the last see nothing
        const int m_first = A.window > 0 ? max(0, m_pos + 1 - A.window) : 0;

        // the chunk joins those before it
        auto join_chunk = [&]() {
            __syncthreads();                             // keep_s has been read
            if ((tid & 3) == 0) {
                const float next = fmaxf(m_all, m), keep = m_all == next ? 1.0f : ratio(m_all, next), take = ratio(m, next);
                l_all = join(l_all, keep, l, take);
                m_all = next;
                keep_s[m_row] = keep;
                take_s[m_row] = take;
            }
            m = -CUDART_INF_F, l = 0.0f;
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4 * COLS; ++i) {
                if (few && i >= FEW_OWN) continue;
                const int r = few ? min(f_row + i * FEW_STEP, ROWS - 1) : o_row + i / COLS;
                float& total = total_s[i * THREADS + tid];
                total = join(total, keep_s[r], o[i / COLS][i % COLS], take_s[r]);
                o[i / COLS][i % COLS] = 0.0f;
            }
        };
        // a thread's eight scores of a block that begins at key `at`: masked, the row's maximum, exponentials in their place and their
        // sum; returns what the sums before are multiplied with.  The four threads of a row lie in one warp and come here together.
        auto weigh = [&](float* p, int at) {
            float x[8], top = -CUDART_INF_F;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int key = at + m_key + u;
                x[u] = key <= m_pos && key >= m_first ? p[u] * A.scale : -CUDART_INF_F;
                top = fmaxf(top, x[u]);
            }
            const unsigned quad = 0xfu << (lane & 28);
            top = fmaxf(top, __shfl_xor_sync(quad, top, 1));
            top = fmaxf(top, __shfl_xor_sync(quad, top, 2));
            const float next = fmaxf(m, top), alpha = m == next ? 1.0f : ratio(m, next);
            float sum = 0.0f;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float e = ratio(x[u], next);
                p[u] = e;
                sum += e;
            }
            sum += __shfl_xor_sync(quad, sum, 1);
            sum += __shfl_xor_sync(quad, sum, 2);
            l = l * alpha + sum;
            m = next;
            return alpha;
        };
        // where some row does not see all of the block's keys, weights of zero are skipped: a value that a row does not see never
        // reaches it, not even one that is no number
        auto some_unseen = [&](int at) { return at + KEYS > pos0 + 1 || (A.window > 0 && at < end_key - A.window); };

        int at = begin / KEYS * KEYS;
        if (few) {
            // Steps of up to two blocks of keys (they end at multiples of FEW_KEYS).  The keys of the next two steps and the values
            // of the next are on their way while one is worked on.
            float* fk_s = smem + FEW_ROWS * PITCH;       // [2][FEW_KEYS][PITCH], behind q
            float* fv_s = fk_s + 2 * FEW_KEYS * PITCH;   // [FEW_KEYS][D]
            float* fp_s = fv_s + FEW_KEYS * D;           // [FEW_ROWS][FEW_PITCH]
            auto keys_of = [&](int from) { return from < end ? (from % FEW_KEYS ? KEYS : FEW_KEYS) : 0; };
            auto after = [&](int from) { return from + (from % FEW_KEYS ? KEYS : FEW_KEYS); };
            const int second = after(at), third = after(second);
            if (tid < 3 * FEW_KEYS) place_s[tid] = place_of((tid < FEW_KEYS ? at : tid < 2 * FEW_KEYS ? second : third) + tid % FEW_KEYS);
            __syncthreads();
            int coming = after(third);                   // the step whose places come next, AHEAD - 1 ahead of the running one
            fetch(step_rows, A.k, fk_s, PITCH, place_s);
            fetch(step_rows, A.v, fv_s, D, place_s);
            fetch(step_rows, A.k, fk_s + FEW_KEYS * PITCH, PITCH, place_s + FEW_KEYS);
            for (int step = 0; at < end; ++step) {
                const int blocks = keys_of(at) / KEYS;
                const long long later = tid < FEW_KEYS ? place_of(coming + tid) : -1;
                copies_wait<2>();
                __syncthreads();                         // the step's keys are there (and q)
                const float* k_now = fk_s + (step & 1) * FEW_KEYS * PITCH;
                for (int task = warp; task < rows * blocks; task += THREADS / 32) {
                    const int r = task % rows, b = task / rows;
                    float s = 0.0f;
#pragma unroll 16
                    for (int e = 0; e < D; e += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(q_s + r * PITCH + e);
                        const float4 y = *reinterpret_cast<const float4*>(k_now + (b * KEYS + lane) * PITCH + e);
                        s = fmaf(x.x, y.x, s), s = fmaf(x.y, y.y, s), s = fmaf(x.z, y.z, s), s = fmaf(x.w, y.w, s);
                    }
                    fp_s[r * FEW_PITCH + b * KEYS + lane] = s;
                }
                __syncthreads();                         // the scores are there, the keys have been read
                fetch(step_rows, A.k, fk_s + (step & 1) * FEW_KEYS * PITCH, PITCH, place_s + (step + 2) % AHEAD * FEW_KEYS);
                if (m_row < rows)
                    for (int b = 0; b < blocks; ++b) {
                        const float alpha = weigh(fp_s + m_row * FEW_PITCH + b * KEYS + m_key, at + b * KEYS);
                        if ((tid & 3) == 0) keep_s[b * FEW_ROWS + m_row] = alpha;
                    }
                if (tid < FEW_KEYS) place_s[(step + AHEAD - 1) % AHEAD * FEW_KEYS + tid] = later;
                coming = after(coming);
                copies_wait<1>();
                __syncthreads();                         // the weights and the values are there
                // rows beyond the last add what nothing reads
                auto values = [&](auto own, auto skip, int b) {
                    constexpr int OWN = decltype(own)::value;
                    float f[OWN];
#pragma unroll
                    for (int i = 0; i < OWN; ++i) f[i] = o_few[i] * keep_s[b * FEW_ROWS + f_row + i * FEW_STEP];
                    const float* p = fp_s + f_row * FEW_PITCH + b * KEYS;
#pragma unroll 4
                    for (int j = 0; j < KEYS; j += 4) {
                        float y[4], w[OWN][4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) y[u] = fv_s[(b * KEYS + j + u) * D + f_col];
#pragma unroll
                        for (int i = 0; i < OWN; ++i) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(p + i * FEW_STEP * FEW_PITCH + j);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int i = 0; i < OWN; ++i)
                                if (!decltype(skip)::value || w[i][u] != 0.0f) f[i] = fmaf(w[i][u], y[u], f[i]);
                    }
#pragma unroll
                    for (int i = 0; i < OWN; ++i) o_few[i] = f[i];
                };
                for (int b = 0; b < blocks; ++b) {
                    const bool masked = some_unseen(at + b * KEYS);
                    if (rows <= FEW_STEP) masked ? values(std::integral_constant<int, 1>{}, std::true_type{}, b) : values(std::integral_constant<int, 1>{}, std::false_type{}, b);
                    else masked ? values(std::integral_constant<int, FEW_OWN>{}, std::true_type{}, b) : values(std::integral_constant<int, FEW_OWN>{}, std::false_type{}, b);
                }
                at = after(at);
                if (!SPLIT && (at >= end || at % CHUNK == 0)) join_chunk();
                __syncthreads();                         // values, weights and factors have been read
                fetch(step_rows, A.v, fv_s, D, place_s + (step + 1) % AHEAD * FEW_KEYS);
            }
        } else {
            // A block's keys and values are asked for while the block before it is worked on, their places one block earlier.
            if (tid < 2 * KEYS) place_s[tid] = place_of(at + tid);
            __syncthreads();
            fetch(block_rows, A.k, k_s, PITCH, place_s);
            fetch(block_rows, A.v, v_s, D, place_s);
            for (int block = 0; at < end; ++block, at += KEYS) {
                const long long later = tid < KEYS ? place_of(at + 2 * KEYS + tid) : -1;
                const long long* next_places = place_s + ((block + 1) & 1) * KEYS;
                const bool more = at + KEYS < end;
                copies_wait<1>();
                __syncthreads();                         // the keys are there (and q)
                if ((warp >> 1) * 16 < rows) {
                    float s[4][2] = {};
#pragma unroll 4
                    for (int e = 0; e < D; e += 4) {
                        float4 y[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) y[j] = *reinterpret_cast<const float4*>(k_s + (s_key + 8 * j) * PITCH + e);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 x = *reinterpret_cast<const float4*>(q_s + (s_row + 4 * i) * PITCH + e);
#pragma unroll
                            for (int j = 0; j < 2; ++j) s[i][j] = fmaf(x.x, y[j].x, s[i][j]);
#pragma unroll
                            for (int j = 0; j < 2; ++j) s[i][j] = fmaf(x.y, y[j].y, s[i][j]);
#pragma unroll
                            for (int j = 0; j < 2; ++j) s[i][j] = fmaf(x.z, y[j].z, s[i][j]);
#pragma unroll
                            for (int j = 0; j < 2; ++j) s[i][j] = fmaf(x.w, y[j].w, s[i][j]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j) p_s[(s_row + 4 * i) * P_PITCH + s_key + 8 * j] = s[i][j];
                }
                __syncthreads();                         // the scores are there, the keys have been read
                if (more) fetch(block_rows, A.k, k_s, PITCH, next_places);
                else copies_commit();
                const float alpha = weigh(p_s + m_row * P_PITCH + m_key, at);
                if ((tid & 3) == 0) keep_s[m_row] = alpha;
                copies_wait<1>();
                __syncthreads();                         // the weights and the values are there
                const bool masked = some_unseen(at);
                if (o_row < rows) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float alpha = keep_s[o_row + i];
#pragma unroll
                        for (int c = 0; c < COLS; ++c) o[i][c] *= alpha;
                    }
                    auto keys = [&](auto skip) {
#pragma unroll 2
                        for (int j = 0; j < KEYS; j += 4) {
                            float w[4][4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(p_s + (o_row + i) * P_PITCH + j);
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int c = 0; c < COLS; c += 4) {
                                    float y[4];
                                    *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(v_s + (j + u) * D + o_col + 16 * c);
#pragma unroll
                                    for (int i = 0; i < 4; ++i)
#pragma unroll
                                        for (int b = 0; b < 4; ++b)
                                            if (!decltype(skip)::value || w[i][u] != 0.0f) o[i][c + b] = fmaf(w[i][u], y[b], o[i][c + b]);
                                }
                        }
                    };
                    if (masked) keys(std::true_type{});
                    else keys(std::false_type{});
                }
                if (!SPLIT && (at + KEYS >= end || (at + KEYS) % CHUNK == 0)) join_chunk();
                if (tid < KEYS) place_s[(block & 1) * KEYS + tid] = later;
                __syncthreads();                         // values, weights and factors have been read
                if (more) fetch(block_rows, A.v, v_s, D, next_places);
                else copies_commit();
            }
        }
        copies_wait<0>();
        auto row_of = [&](int r) { return (size_t)(t0 + r / group) * A.nq + g * group + r % group; };
        if (SPLIT) {
            auto place = [&](int r) { return row_of(r) * A.chunks + blockIdx.z; };
            if ((tid & 3) == 0 && m_row < rows) {
                A.part_ml[2 * place(m_row)] = m;
                A.part_ml[2 * place(m_row) + 1] = l;
            }
            if (few) {
#pragma unroll
                for (int i = 0; i < FEW_OWN; ++i)
                    if (f_row + i * FEW_STEP < rows && f_col < d) A.part_o[place(f_row + i * FEW_STEP) * d + f_col] = o_few[i];
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (o_row + i >= rows) continue;
#pragma unroll
                    for (int c = 0; c < COLS; c += 4)
                        if (o_col + 16 * c < d)
                            *reinterpret_cast<float4*>(A.part_o + place(o_row + i) * d + o_col + 16 * c) = make_float4(o[i][c], o[i][c + 1], o[i][c + 2], o[i][c + 3]);
                }
            }
            continue;
        }
        __syncthreads();
        if ((tid & 3) == 0) keep_s[m_row] = 1.0f / l_all;
        __syncthreads();
        if (few) {
#pragma unroll
            for (int i = 0; i < FEW_OWN; ++i) {
                const int r = f_row + i * FEW_STEP;
                if (r < rows && f_col < d) A.out[row_of(r) * d + f_col] = total_s[i * THREADS + tid] * keep_s[r];
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (o_row + i >= rows) continue;
                const float inv = keep_s[o_row + i];
#pragma unroll
                for (int c = 0; c < COLS; c += 4) {
                    if (o_col + 16 * c >= d) continue;
                    float x[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) x[b] = total_s[(i * COLS + c + b) * THREADS + tid] * inv;
                    *reinterpret_cast<float4*>(A.out + row_of(o_row + i) * d + o_col + 16 * c) = make_float4(x[0], x[1], x[2], x[3]);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Heads of 128 elements on the tcgen05 tensor cores, with every bit of the inputs: a float32 is three bfloat16 (parts3.cuh), a product
// of two is six products of parts (the other three are at most 2^-24 of it).  A block takes a tile of up to 128 rows and walks their keys
// in blocks of 64:
//   warps 0-7   two threads a row, 32 scores and 64 columns each: scores from tensor memory, maximum, exponentials, the weights' parts
//               back into tensor memory; a block's weighted values (a fresh accumulator) are added to the row's in registers, in
//               float32.  Between a block's scores and its softmax they write the next block's keys as bfloat16 tiles, so that its MMAs
//               run under the softmax
//   warps 8-10  the values' tiles (rows come by cp.async a block ahead, page numbers four)
//   warp 11     issues the MMAs: scores = q parts (tensor memory) . keys, values = weights (tensor memory) . values
// A row's result has the same bits however its request is cut: blocks of keys begin at multiples of 64, chunks at multiples of CHUNK, and
// what a tile holds beside a row touches neither its scores nor its sums.  Values that the parts cannot be trusted with (infinite, NaN, from
// 2^64 on, beside which a weight's bits under bfloat16's range would show, or so small that their own last part lies under it) are zeros in
// the tiles and added by the rows that see them.  A score that is no number or infinite is computed again from its row and key, so that
// what a row does not see never reaches it, and so is one of a row with bits under bfloat16's range (2^-133) and one with an element
// from 2^64 on.  (Elsewhere such bits are 2^-62 of a score at most; of weights, 2^-134, they show in sums below 2^-110.)
//
// What bounds it: the parts' instructions and the chain of a block (some 7,000 clocks, of which the MMAs run 3,000), a CTA an SM.  With the
// joining, from a cold L2, 16 query and 8 key/value heads of 128, on the CUDA cores (the kernel above) and here: a prompt of 777 tokens
// 159 -> 76 us, 880 tokens behind 1,420 514 -> 229, 20 behind 980 41 -> 31.  Decoded tokens pay for 128 rows: one behind 4,000 24 -> 32, 4
// requests at 3,000 47 -> 81, 30 at 400 46 -> 92; they take this kernel for the bits' sake.  Error of the layer against 64 bits:
// 1.26e-6 -> 1.24e-6 (777 tokens).
// Tried: all conversions in the copying warps (100 us at 777 tokens), masks and exponentials with a branch an element (softmax 10,700
// clocks a block, 2,000 now).
// ------------------------------------------------------------------------------------------------
constexpr int TC_D = 128, TC_ROWS = 128, TC_KEYS = 64, TC_ROW_WARPS = 8, TC_COPY_WARPS = 3, TC_THREADS = (TC_ROW_WARPS + TC_COPY_WARPS + 1) * 32;
constexpr int TC_PART = TC_KEYS * TC_D * 2, TC_RAW = TC_KEYS * TC_D * 4;         // bytes of a block's part, of its float32 rows
constexpr int TC_S = 0, TC_O = TC_KEYS, TC_Q = TC_O + TC_D, TC_P = TC_Q + 3 * TC_D / 2, TC_TMEM = 512;      // columns of tensor memory
constexpr size_t TC_SMEM = 1024 + 6 * (size_t)TC_PART + 2 * (size_t)TC_RAW + TC_KEYS * TC_ROWS * 4;
static_assert(TC_P + 3 * TC_KEYS / 2 <= TC_TMEM, "tensor memory");
static_assert(CHUNK % TC_KEYS == 0, "whole blocks a chunk");
constexpr int TC_PLACES = 8, TC_AHEAD = 4;                               // blocks whose places are held; how far ahead they are looked up
constexpr float LARGE = 0x1p64f, SMALL = 0x1p-96f;
__device__ __forceinline__ bool has_parts(float v) { return fabsf(v) < LARGE && !(fabsf(v) < SMALL && v != 0.0f); }

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// What was met among floats that became parts: bits that three parts leave (of a NaN, which arithmetic makes of what is infinite, all of
// them), and the largest size.  (Maxima of the first parts, pairs of bfloat16, take longer: 880 tokens behind 1,420 209 us, with these 206.5,
// with neither 204.)
struct Met {
    uint32_t rest = 0;
    float top = 0.0f;
    __device__ __forceinline__ bool lost() const { return rest & LOST_BITS; }
    __device__ __forceinline__ bool large() const { return top >= LARGE; }
};
// four floats as two words of each part
__device__ __forceinline__ void split4(float4 v, uint2 (&parts)[3], Met& met) {
    uint32_t low[3], high[3];
    met.top = fmaxf(fmaxf(met.top, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    three_parts(v.x, v.y, low), three_parts(v.z, v.w, high);
#pragma unroll
    for (int p = 0; p < 3; ++p) parts[p] = make_uint2(low[p], high[p]);
    met.rest |= left_bits(v);
}

// a row and a key that the parts cannot be trusted with
__device__ __noinline__ float whole_score(const float* q, const float* k) {
    float s = 0.0f;
    for (int e = 0; e < TC_D; ++e) s = fmaf(q[e], k[e], s);
    return s;
}

template <bool SPLIT>
__global__ void __launch_bounds__(TC_THREADS, 1) attention_f32_tc_kernel(const Args A) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *k_parts = smem, *v_parts = smem + 3 * TC_PART, *k_raw = smem + 6 * TC_PART, *v_raw = k_raw + TC_RAW;
    float* weights = reinterpret_cast<float*>(v_raw + TC_RAW);           // [TC_KEYS][TC_ROWS], read where values have no parts
    // v_full: two in turn, so that the rows too may wait for it (what the copying warps left for them is then there)
    __shared__ uint64_t k_full, s_full, p_full, v_full[2], o_full;
    __shared__ uint32_t tmem_slot;
    __shared__ long long place_s[TC_PLACES][TC_KEYS];                    // where cached rows begin; -1: not seen
    __shared__ float met[2][2][TC_ROWS];
    __shared__ unsigned odd_values[2][TC_KEYS / 32];                     // keys whose values have no parts
    // rows that met something: of the queries LOST and LARGE_ONE by halves; of a block's keys, by the warp that wrote them, a bit a key that
    // lost bits and, eight bits further, one a key with a large element
    __shared__ unsigned char q_facts[2][TC_ROWS];
    __shared__ __align__(16) unsigned short key_facts[2][TC_ROW_WARPS];
    constexpr unsigned LOST = 1, LARGE_ONE = 2;
    __shared__ int found[2], warp_count[TC_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int ISSUER = TC_ROW_WARPS + TC_COPY_WARPS;
    if (tid == 0) {
        mbar_init(&k_full, TC_ROW_WARPS);
        for (int b = 0; b < 2; ++b) mbar_init(&v_full[b], TC_COPY_WARPS);
        mbar_init(&s_full, 1);
        mbar_init(&p_full, TC_ROW_WARPS);
        mbar_init(&o_full, 1);
        mbar_fence_init();
    }
    if (warp == ISSUER) {
        tmem_alloc(&tmem_slot, TC_TMEM);
        tmem_relinquish_alloc_permit();
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    tcgen05_fence_after_sync();
    const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    pdl_launch_dependents();
    pdl_wait();
    const int g = blockIdx.y, group = A.nq / A.nkv;
    int it = 0;                                                          // blocks of keys so far, over all tiles
    for (int tile = blockIdx.x;; tile += gridDim.x) {
        const int t0 = find_tile<TC_THREADS>(A, tile, found, warp_count);
        if (t0 < 0) break;
        const int tokens = found[1], rows = tokens * group;
        const int pos0 = A.positions[t0], end_key = pos0 + tokens;
        int begin = A.window > 0 ? max(0, pos0 + 1 - A.window) : 0, end = end_key;
        if (SPLIT) {
            begin = max(begin, (int)blockIdx.z * CHUNK);                 // keys beyond the last chunk that was planned go with it
            if ((int)blockIdx.z + 1 < A.chunks) end = min(end, ((int)blockIdx.z + 1) * CHUNK);
            if (begin >= end) continue;
        }
        const int at0 = begin / TC_KEYS * TC_KEYS, blocks = (end - at0 + TC_KEYS - 1) / TC_KEYS;
        const int* pages = A.table + (size_t)A.seq_of_token[t0] * A.table_width;
        auto place_of = [&](int p) -> long long {
            if (p < begin || p >= end) return -1;
            return (((long long)pages[p / A.page_size] * A.nkv + g) * A.page_size + p % A.page_size) * TC_D;
        };
        if (tid < TC_AHEAD * TC_KEYS) place_s[(it + tid / TC_KEYS) % TC_PLACES][tid % TC_KEYS] = place_of(at0 + tid);
        __syncthreads();
        // rows `mine`, mine + COUNT, ... of a block: a lane four of a row's elements, which it fetches and converts itself
        auto fetch = [&](auto count, const float* cache, unsigned char* raw, int mine, int i, bool wanted) {
            constexpr int COUNT = decltype(count)::value;
            if (wanted) {
#pragma unroll 4
                for (int row = mine; row < TC_KEYS; row += COUNT) {
                    const long long place = place_s[i % TC_PLACES][row];
                    copy16(reinterpret_cast<float*>(raw) + row * TC_D + 4 * lane, cache + (place >= 0 ? place + 4 * lane : 0), place >= 0);
                }
            }
            copies_commit();
        };
        const uint32_t part_at = (lane >> 4) * (TC_PART / 2) + (lane & 1) * 8, piece = (lane & 15) >> 1;
        auto put = [&](unsigned char* to, int row, float4 v, Met& met) {
            uint2 parts[3];
            split4(v, parts, met);
            to += part_at + row * 128 + ((piece ^ (row & 7)) << 4);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(to + p * TC_PART) = parts[p];
        };
        auto raw_of = [&](const unsigned char* raw, int row) { return *reinterpret_cast<const float4*>(raw + row * TC_D * 4 + 16 * lane); };
        // some read together; what was met
        auto convert = [&](auto count, unsigned char* to, const unsigned char* raw, int mine) {
            constexpr int COUNT = decltype(count)::value, TOGETHER = 4;
            Met met;
#pragma unroll 1
            for (int first = mine; first < TC_KEYS; first += TOGETHER * COUNT) {
                float4 v[TOGETHER];
#pragma unroll
                for (int r = 0; r < TOGETHER; ++r) v[r] = raw_of(raw, min(first + r * COUNT, TC_KEYS - 1));
#pragma unroll
                for (int r = 0; r < TOGETHER; ++r)
                    if (first + r * COUNT < TC_KEYS) put(to, first + r * COUNT, v[r], met);
            }
            return met;
        };
        constexpr std::integral_constant<int, TC_ROW_WARPS> by_rows;
        constexpr std::integral_constant<int, TC_COPY_WARPS> by_copies;
        if (warp == ISSUER) {
            const bool leader = elect_one();
            constexpr uint32_t s_desc = umma_idesc_bf16_f32(TC_ROWS, TC_KEYS), o_desc = umma_idesc_bf16_f32(TC_ROWS, TC_D, true);
            constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};      // (part of A, part of B): small products first
            auto scores = [&](int i) {
                mbar_wait(&k_full, i & 1);
                tcgen05_fence_after_sync();
                if (leader) {
#pragma unroll 1
                    for (int j = 0; j < 6; ++j) {
                        const uint32_t a = tmem + TC_Q + order[j][0] * (TC_D / 2), b = smem_u32(k_parts) + order[j][1] * TC_PART;
#pragma unroll
                        for (int k = 0; k < TC_D / 16; ++k)              // two groups of 64 columns
                            umma_bf16_a_tmem(tmem + TC_S, a + 8 * k, umma_smem_desc_sw128(b + (k / 4) * (TC_PART / 2)) + 2 * (k % 4), s_desc, j > 0 || k > 0);
                    }
                    umma_commit(&s_full);
                }
                __syncwarp();
            };
            scores(it);
            for (int n = 0; n < blocks; ++n) {
                if (n + 1 < blocks) scores(it + n + 1);
                mbar_wait(&p_full, (it + n) & 1);
                mbar_wait(&v_full[(it + n) & 1], (it + n) >> 1 & 1);
                tcgen05_fence_after_sync();
                if (leader) {
#pragma unroll 1
                    for (int j = 0; j < 6; ++j) {
                        const uint32_t a = tmem + TC_P + order[j][0] * (TC_KEYS / 2), b = smem_u32(v_parts) + order[j][1] * TC_PART;
#pragma unroll
                        for (int k = 0; k < TC_KEYS / 16; ++k)
                            umma_bf16_a_tmem(tmem + TC_O, a + 8 * k, umma_smem_desc_sw128_mn(b + k * 16 * 128, TC_PART / 2), o_desc, j > 0 || k > 0);
                    }
                    umma_commit(&o_full);
                }
                __syncwarp();
            }
        } else if (warp >= TC_ROW_WARPS) {
            const int mine = warp - TC_ROW_WARPS, ct = tid - TC_ROW_WARPS * 32;
            fetch(by_copies, A.v, v_raw, mine, it, true);
            for (int n = 0; n < blocks; ++n) {
                const int i = it + n;
                const long long later = ct < TC_KEYS ? place_of(at0 + (n + TC_AHEAD) * TC_KEYS + ct) : -1;
                copies_wait<0>();
                if (i > 0) mbar_wait(&o_full, (i - 1) & 1);              // the values' parts have been read, and the odd values two blocks before
                if (ct < TC_KEYS / 32) odd_values[i & 1][ct] = 0u;
                if (ct < TC_KEYS) place_s[(i + TC_AHEAD) % TC_PLACES][ct] = later;
                bar_sync(1, TC_COPY_WARPS * 32);
                const Met all = convert(by_copies, v_parts, v_raw, mine);
                if (__any_sync(0xffffffffu, all.lost() || all.large())) {
#pragma unroll 1
                    for (int row = mine; row < TC_KEYS; row += TC_COPY_WARPS) {
                        float4 v = raw_of(v_raw, row);
                        Met met;
                        put(v_parts, row, v, met);
                        if (!__any_sync(0xffffffffu, met.lost() || met.large())) continue;      // a row's lanes agree: its readers ask each value
                        if (!has_parts(v.x)) v.x = 0.0f;
                        if (!has_parts(v.y)) v.y = 0.0f;
                        if (!has_parts(v.z)) v.z = 0.0f;
                        if (!has_parts(v.w)) v.w = 0.0f;
                        put(v_parts, row, v, met);
                        if (lane == 0) atomicOr(&odd_values[i & 1][row / 32], 1u << (row % 32));
                    }
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_full[i & 1]);
                fetch(by_copies, A.v, v_raw, mine, i + 1, n + 1 < blocks);
            }
            copies_wait<0>();
        } else {
            const int row = (warp & 3) * 32 + lane, half = warp >> 2, pair_bar = 2 + (warp & 3);
            const bool live = row < rows;
            const size_t row_at = (size_t)(t0 + (live ? row / group : 0)) * A.nq + g * group + (live ? row % group : 0);
            const float* q = A.q + row_at * TC_D;
            fetch(by_rows, A.k, k_raw, warp, it, true);
            Met of_q;
#pragma unroll 1
            for (int c = 0; c < 64; c += 32) {
                uint32_t words[3][16];
#pragma unroll
                for (int e = 0; e < 32; e += 4) {
                    uint2 parts[3];
                    split4(live ? *reinterpret_cast<const float4*>(q + half * 64 + c + e) : make_float4(0.0f, 0.0f, 0.0f, 0.0f), parts, of_q);
#pragma unroll
                    for (int p = 0; p < 3; ++p) words[p][e / 2] = parts[p].x, words[p][e / 2 + 1] = parts[p].y;
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_store_16_words(lanes + TC_Q + p * (TC_D / 2) + half * 32 + c / 2, words[p]);
            }
            tmem_store_wait();
            q_facts[half][row] = (of_q.lost() ? LOST : 0) | (of_q.large() ? LARGE_ONE : 0);
            // block i's keys as parts: q is there, and the scores of the block before have been read
            auto keys_ready = [&](int i, bool more) {
                copies_wait<0>();
                const Met all = convert(by_rows, k_parts, k_raw, warp);
                unsigned met_keys = 0;
                if (__any_sync(0xffffffffu, all.lost() || all.large())) {
#pragma unroll 1
                    for (int b = 0; b < TC_KEYS / TC_ROW_WARPS; ++b) {
                        Met met;
                        uint2 parts[3];
                        split4(raw_of(k_raw, warp + b * TC_ROW_WARPS), parts, met);
                        met_keys |= (__any_sync(0xffffffffu, met.lost()) ? 1u : 0u) << b | (__any_sync(0xffffffffu, met.large()) ? 256u : 0u) << b;
                    }
                }
                if (lane == 0) key_facts[i & 1][warp] = (unsigned short)met_keys;
                fence_async_shared();
                tcgen05_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&k_full);
                fetch(by_rows, A.k, k_raw, warp, i + 1, more);
            };
            keys_ready(it, blocks > 1);
            const int my_pos = live ? pos0 + row / group : -1, my_first = A.window > 0 ? max(0, my_pos + 1 - A.window) : 0;
            float o[64];
#pragma unroll
            for (int c = 0; c < 64; ++c) o[c] = 0.0f;
            float m = -CUDART_INF_F, l = 0.0f, m_all = -CUDART_INF_F, l_all = 0.0f;
            bool joined = false;
            // block i's weighted values join the row's
            auto take_values = [&](int i) {
                mbar_wait(&v_full[i & 1], i >> 1 & 1);
                mbar_wait(&o_full, i & 1);
                __syncwarp();
                tcgen05_fence_after_sync();
#pragma unroll
                for (int c = 0; c < 64; c += 16) {
                    float v[16];
                    tmem_load_16_async(lanes + TC_O + half * 64 + c, v);
                    tmem_load_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[c + e] += v[e];
                }
                if (odd_values[i & 1][0] | odd_values[i & 1][1]) {
                    bar_sync(pair_bar, 64);                              // the other half's weights are there
#pragma unroll 1
                    for (int k = 0; k < TC_KEYS; ++k) {
                        if (!(odd_values[i & 1][k / 32] >> (k % 32) & 1u)) continue;
                        const float w = weights[k * TC_ROWS + row];
                        const long long place = place_s[i % TC_PLACES][k];
                        if (w == 0.0f || place < 0) continue;
#pragma unroll
                        for (int c = 0; c < 64; ++c) {
                            const float v = A.v[place + half * 64 + c];
                            if (!has_parts(v)) o[c] = fmaf(w, v, o[c]);
                        }
                    }
                    bar_sync(pair_bar, 64);
                }
            };
            // both halves' sums, behind block i: through that block's place in `met`, which is written again only behind the barrier of
            // the block after it (the other place is written ahead of that barrier, when the other half may not have read these yet)
            auto whole_sum = [&](int i) {
                bar_sync(pair_bar, 64);                                  // block i's maxima have been read
                met[i & 1][half][row] = l;
                bar_sync(pair_bar, 64);
                return met[i & 1][0][row] + met[i & 1][1][row];
            };
            float* out = A.out + row_at * TC_D + half * 64;
            auto join_chunk = [&](int i) {                               // !SPLIT: the chunk that ends with block i joins those before it, which lie in `out`
                const float sum = whole_sum(i);
                const float next = fmaxf(m_all, m), keep = m_all == next ? 1.0f : ratio(m_all, next), take = ratio(m, next);
                l_all = join(l_all, keep, sum, take);
                m_all = next;
                if (live) {
#pragma unroll
                    for (int c = 0; c < 64; c += 4) {
                        float4 total = joined ? *reinterpret_cast<const float4*>(out + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        total = make_float4(join(total.x, keep, o[c], take), join(total.y, keep, o[c + 1], take), join(total.z, keep, o[c + 2], take),
                                            join(total.w, keep, o[c + 3], take));
                        *reinterpret_cast<float4*>(out + c) = total;
                    }
                }
                joined = true;
                m = -CUDART_INF_F, l = 0.0f;
#pragma unroll
                for (int c = 0; c < 64; ++c) o[c] = 0.0f;
            };
            bool pending = false;                                        // a block's values are still to come
#pragma unroll 1
            for (int n = 0; n < blocks; ++n) {
                const int i = it + n, at = at0 + n * TC_KEYS;
                if (!SPLIT && n > 0 && at % CHUNK == 0) {
                    take_values(i - 1);
                    join_chunk(i - 1);
                    pending = false;
                }
                float x[32], top = -CUDART_INF_F;
                mbar_wait(&s_full, i & 1);
                __syncwarp();
                tcgen05_fence_after_sync();
                tmem_load_32(lanes + TC_S + half * 32, x);
                const uint4 met_keys = *reinterpret_cast<const uint4*>(key_facts[i & 1]);      // block i + 2's come when all warps are here
                if (n + 1 < blocks) keys_ready(i + 1, n + 2 < blocks);
                bool odd = met_keys.x | met_keys.y | met_keys.z | met_keys.w;
#pragma unroll
                for (int u = 0; u < 32; ++u) odd |= !(fabsf(x[u]) <= 3.402823466e38f);
                if (__any_sync(0xffffffffu, odd)) {                      // parts that cannot be trusted: the rows and the keys themselves
                    const unsigned f = q_facts[0][row] | q_facts[1][row], words[4] = {met_keys.x, met_keys.y, met_keys.z, met_keys.w};
#pragma unroll
                    for (int u = 0; u < 32; ++u) {
                        const int key = at + half * 32 + u;
                        const unsigned of_key = words[u % 8 / 2] >> (u % 2 * 16 + half * 4 + u / 8);      // written by warp u % 8, its row half * 4 + u / 8
                        const bool shows = ((of_key & 1u) && (f & LARGE_ONE)) || ((of_key & 256u) && (f & LOST));
                        if (key <= my_pos && key >= my_first && (shows || !(fabsf(x[u]) <= 3.402823466e38f)))
                            x[u] = whole_score(q, A.k + place_s[i % TC_PLACES][half * 32 + u]);
                    }
                }
                if (at + TC_KEYS > pos0 + 1 || (A.window > 0 && at < end_key - A.window)) {       // some row does not see all of the block
                    const int last = my_pos - (at + half * 32), first = my_first - (at + half * 32);
#pragma unroll
                    for (int u = 0; u < 32; ++u) x[u] = u <= last && u >= first ? x[u] * A.scale : -CUDART_INF_F;
                } else if (live) {
#pragma unroll
                    for (int u = 0; u < 32; ++u) x[u] *= A.scale;
                } else {
#pragma unroll
                    for (int u = 0; u < 32; ++u) x[u] = -CUDART_INF_F;
                }
#pragma unroll
                for (int u = 0; u < 32; ++u) top = fmaxf(top, x[u]);
                met[i & 1][half][row] = top;
                bar_sync(pair_bar, 64);
                top = fmaxf(top, met[i & 1][half ^ 1][row]);
                const float next = fmaxf(m, top), alpha = m == next ? 1.0f : ratio(m, next);
                float sum = 0.0f;
                const float from = next == -CUDART_INF_F ? 0.0f : next;  // nothing seen yet: zeros
#pragma unroll
                for (int u = 0; u < 32; ++u) x[u] = expf(x[u] - from);
#pragma unroll
                for (int u = 0; u < 32; ++u) sum += x[u];
                l = l * alpha + sum;
                m = next;
                if (pending) take_values(i - 1);
#pragma unroll
                for (int c = 0; c < 64; ++c) o[c] *= alpha;
#pragma unroll
                for (int u = 0; u < 32; ++u) weights[(half * 32 + u) * TC_ROWS + row] = x[u];
                uint32_t words[3][16];
#pragma unroll
                for (int u = 0; u < 32; u += 2) {
                    uint32_t parts[3];
                    three_parts(x[u], x[u + 1], parts);
#pragma unroll
                    for (int p = 0; p < 3; ++p) words[p][u / 2] = parts[p];
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_store_16_words(lanes + TC_P + p * (TC_KEYS / 2) + half * 16, words[p]);
                tmem_store_wait();
                tcgen05_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full);
                pending = true;
            }
            copies_wait<0>();
            take_values(it + blocks - 1);
            if (SPLIT) {
                const float sum = whole_sum(it + blocks - 1);
                if (live) {
                    const size_t place = row_at * A.chunks + blockIdx.z;
                    if (half == 0) A.part_ml[2 * place] = m, A.part_ml[2 * place + 1] = sum;
#pragma unroll
                    for (int c = 0; c < 64; c += 4)
                        *reinterpret_cast<float4*>(A.part_o + place * TC_D + half * 64 + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
                }
            } else {
                join_chunk(it + blocks - 1);
                const float inv = 1.0f / l_all;
                if (live) {
#pragma unroll
                    for (int c = 0; c < 64; c += 4) {
                        const float4 total = *reinterpret_cast<const float4*>(out + c);
                        *reinterpret_cast<float4*>(out + c) = make_float4(total.x * inv, total.y * inv, total.z * inv, total.w * inv);
                    }
                }
            }
        }
        it += blocks;
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == ISSUER) {
        tcgen05_fence_after_sync();
        tmem_dealloc(tmem, TC_TMEM);
    }
}

// Joins a row's chunks in ascending order: a warp a (token, head).
__global__ void attention_f32_join_kernel(const Args A) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= (long long)A.tokens * A.nq) return;
    const int pos = A.positions[row / A.nq];
    const int first = min((A.window > 0 ? max(0, pos + 1 - A.window) : 0) / CHUNK, A.chunks - 1), last = min(pos / CHUNK, A.chunks - 1);
    const float* ml = A.part_ml + 2 * row * A.chunks;
    float m_all = -CUDART_INF_F, l_all = 0.0f, total[8] = {};
    constexpr int BATCH = 4;                             // chunks whose parts are loaded together
    for (int c0 = first; c0 <= last; c0 += BATCH) {
        float m[BATCH], l[BATCH], o[BATCH][8];
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            const int c = min(c0 + b, last);
            m[b] = ml[2 * c], l[b] = ml[2 * c + 1];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[b][i] = lane + 32 * i < A.d ? A.part_o[(row * A.chunks + c) * A.d + lane + 32 * i] : 0.0f;
        }
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            if (c0 + b > last) break;
            const float next = fmaxf(m_all, m[b]), keep = m_all == next ? 1.0f : ratio(m_all, next), take = ratio(m[b], next);
            l_all = join(l_all, keep, l[b], take);
            m_all = next;
#pragma unroll
            for (int i = 0; i < 8; ++i) total[i] = join(total[i], keep, o[b][i], take);
        }
    }
    const float inv = 1.0f / l_all;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (lane + 32 * i < A.d) A.out[row * A.d + lane + 32 * i] = total[i] * inv;
}

template <int D, bool SPLIT>
int launch(const Args& A, int tiles, void* stream) {
    constexpr int SMEM = smem_floats<D, SPLIT>() * (int)sizeof(float);
    static PerDevice configured;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<D, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    MRS_LAUNCH((attention_f32_kernel<D, SPLIT>), dim3(tiles, A.nkv, SPLIT ? A.chunks : 1), THREADS, SMEM, stream, A);
    MRS_RETURN_LAUNCH_STATUS();
}

template <bool SPLIT>
int launch_tc(const Args& A, int tiles, void* stream) {
    static PerDevice configured;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_tc_kernel<SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    MRS_LAUNCH(attention_f32_tc_kernel<SPLIT>, dim3(tiles, A.nkv, SPLIT ? A.chunks : 1), TC_THREADS, TC_SMEM, stream, A);
    MRS_RETURN_LAUNCH_STATUS();
}

}  // namespace

MRS_EXPORT int mrs_attention_f32_take_error(unsigned int* word) { return mrs_take_error_word(word); }
// Mirrors the error word into a word of pinned host memory from now on.
MRS_EXPORT int mrs_attention_f32_mirror_errors(unsigned int* host_word) { return mrs_set_error_mirror(host_word); }

MRS_EXPORT int mrs_attention_f32_chunk() { return CHUNK; }

// `parts`: null, or scratch of tokens * nq * chunks * (d + 2) floats; then every chunk of mrs_attention_f32_chunk() keys of a tile has
// a block of its own (keys beyond `chunks` of them go with the last one: right, but no longer the same bits as in one walk).  `sequences`: rows of the block table.
MRS_EXPORT int mrs_attention_f32(const float* q, const float* k_cache, const float* v_cache, const int* positions, const int* seq_of_token,
                                 const int* block_table, float* out, float* parts, int chunks, int tokens, int sequences, int nq, int nkv, int d,
                                 int page_size, int table_width, float scale, int window, void* stream) {
    if (tokens <= 0) return 0;
    if (d <= 0 || d % 4 || d > 256 || nkv <= 0 || nkv > 65535 || nq <= 0 || nq % nkv || nq / nkv > ROWS || page_size <= 0 || sequences < 0 ||
        (parts && (chunks <= 0 || chunks > 65535)) || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out | (uintptr_t)parts) & 15))
        return MRS_BAD_ARGUMENT;
    Args A = {};
    A.q = q, A.k = k_cache, A.v = v_cache, A.positions = positions, A.seq_of_token = seq_of_token, A.table = block_table, A.out = out;
    A.tokens = tokens, A.nq = nq, A.nkv = nkv, A.d = d, A.page_size = page_size, A.table_width = table_width, A.window = window, A.scale = scale;
    const bool tc = d == TC_D;
    A.tile_tokens = (tc ? TC_ROWS : ROWS) / (nq / nkv);
    A.chunks = parts ? chunks : 1;
    A.part_o = parts, A.part_ml = parts ? parts + (size_t)tokens * nq * chunks * d : nullptr;
    // a request's rows make at most two tiles that are not whole; rows that lie otherwise make more, and blocks take several
    const long long most = (long long)tokens / A.tile_tokens + 2LL * sequences + 1;
    const int tiles = (int)(most < tokens ? most : tokens);
    const int code = tc ? (parts ? launch_tc<true>(A, tiles, stream) : launch_tc<false>(A, tiles, stream))
                   : d <= 64 ? (parts ? launch<64, true>(A, tiles, stream) : launch<64, false>(A, tiles, stream))
                   : d <= 128 ? (parts ? launch<128, true>(A, tiles, stream) : launch<128, false>(A, tiles, stream))
                              : (parts ? launch<256, true>(A, tiles, stream) : launch<256, false>(A, tiles, stream));
    if (code != 0 || !parts) return code;
    MRS_LAUNCH(attention_f32_join_kernel, (unsigned)(((long long)tokens * nq + 3) / 4), 128, 0, stream, A);
    MRS_RETURN_LAUNCH_STATUS();
}
