// Token selection on the device: arg-max, and seeded temperature / top-k / top-p sampling.
//
// The reference takes the arg-max on the GPU (ops.cu:152-162: larger logit wins, the smaller id
// on a tie) and samples on the host in float64 after sorting the whole row
// (crates/engine/src/lib.rs:207-244).  Here a row never leaves the device.  The set that may be
// drawn is the reference's: rows ordered by descending logit with ties by ascending id, cut to
// the first top_k, then to the shortest prefix whose weight exp((x - max)/T) reaches top_p times
// the weight of the top_k set.  Such a prefix is {x > threshold} plus the first few ids of
// {x == threshold}; the threshold is found by a radix descent over the float's bits (by count
// for top_k, by weight for top_p) in place of a sort.  The draw is the inverse CDF over the
// kept set in id order with u from a counter-based generator keyed by (seed, draw index), so a
// request's tokens do not depend on what else is in the batch.
#include "common.cuh"
#include <cooperative_groups.h>

#include <cstring>
namespace cg = cooperative_groups;

#define ARGMAX_THREADS 1024

__device__ __forceinline__ unsigned ordered_key(float x) {
    const unsigned b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_value(unsigned key) {
    return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

// u in [0, 1) from (seed, draw index): the splitmix64 finaliser over a Weyl sequence.
__host__ __device__ __forceinline__ float uniform_from_counter(unsigned long long seed, unsigned long long index) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (index + 1ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

struct Best {
    float value;
    int id;
};
__device__ __forceinline__ Best better(Best a, Best b) {
    return (b.value > a.value || (b.value == a.value && b.id < a.id)) ? b : a;
}

// The best of the block's threads; result valid in every thread.
__device__ Best block_best(Best best, Best* scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best other = {__shfl_xor_sync(0xffffffffu, best.value, o), __shfl_xor_sync(0xffffffffu, best.id, o)};
        best = better(best, other);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = best;
    __syncthreads();
    if (warp == 0) {
        Best b = lane < (int)(blockDim.x >> 5) ? scratch[lane] : Best{-CUDART_INF_F, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            Best other = {__shfl_xor_sync(0xffffffffu, b.value, o), __shfl_xor_sync(0xffffffffu, b.id, o)};
            b = better(b, other);
        }
        if (lane == 0) scratch[32] = b;
    }
    __syncthreads();
    return scratch[32];
}

// Arg-max of one row by the whole block; result valid in every thread.
__device__ Best block_argmax(const float* __restrict__ row, int vocab, Best* scratch) {
    Best best = {-CUDART_INF_F, 0x7fffffff};
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) best = better(best, Best{row[i], i});
    return block_best(best, scratch);
}

// One row per thread-block cluster: every block of the cluster takes a share of the row, block 0
// gathers the shares' results through distributed shared memory.  A row of 150k logits is then
// read by eight SMs instead of one.
__global__ void __launch_bounds__(ARGMAX_THREADS) argmax_kernel(const float* __restrict__ logits, int* __restrict__ out,
                                                                int vocab) {
    __shared__ Best scratch[33];
    __shared__ Best shares[16];
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank(), blocks = cluster.num_blocks();
    const int row = blockIdx.x / blocks;
    const int share = (vocab + blocks - 1) / blocks;
    const int begin = min(vocab, (int)rank * share), end = min(vocab, begin + share);
    Best b = block_argmax(logits + (size_t)row * vocab + begin, end - begin, scratch);
    if (threadIdx.x == 0) {
        if (b.id != 0x7fffffff) b.id += begin;
        cluster.map_shared_rank(shares, 0)[rank] = b;
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
        Best best = shares[0];
        for (unsigned r = 1; r < blocks; ++r) best = better(best, shares[r]);
        out[row] = best.id;
    }
}

MRS_EXPORT int mrs_argmax(const float* logits, int* out, int rows, int vocab, void* stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0) return MRS_BAD_ARGUMENT;
    const unsigned blocks = vocab >= 65536 ? 8 : (vocab >= 16384 ? 4 : 1);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(rows * blocks);
    config.blockDim = dim3(ARGMAX_THREADS);
    config.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = blocks;
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&config, argmax_kernel, logits, out, vocab);
    if (e != cudaSuccess) return (int)e;
    MRS_RETURN_LAUNCH_STATUS();
}

// ------------------------------------------------------------------------------------------------
// Sampling.  A row belongs to a thread-block cluster (1, 4 or 8 CTAs): every CTA brings its share of the row into shared
// memory once, and everything after that (largest logit, the two thresholds, the draw) reads it there; the CTAs meet
// through distributed shared memory.  A threshold that at most SAMPLE_LIST candidates decide takes one histogram of the cluster and
// a sort in every CTA; others (more equals at the edge, temperatures that crowd a row into one bin, rows read from memory) take three
// digits of 11, 11 and 10 bits with two meetings each.  What bounds it is the chain: of some 60,000 clocks of a row with top-p the
// largest logit takes 8,000, the weights' histogram 14,000 (an exponential and two or three additions in shared memory an element), its
// meetings and scan 9,000, the candidates 12,000, the draw 15,000.
// Rows of 151,936 logits, three digits always and now: 24 with top-p 69 -> 50 us, top-k and top-p 68 -> 36, top-k 35 -> 34, temperature
// alone 23 -> 24; one row 48 -> 31, 47 -> 27, 25 -> 23, 17 -> 16; 24 of 32,768 with top-p 47 -> 27.  (One CTA a row, which read it
// from L2 some fifteen times with 8-bit digits, took 1,626 us for 24 rows.)
//
// The weights of the kept set are summed in 32 segments of a row, in id order, whatever the cluster's size: a row's token
// does not depend on how many CTAs shared it.
// ------------------------------------------------------------------------------------------------
#define SAMPLE_CTA_THREADS 512
#define SAMPLE_CTA_WARPS (SAMPLE_CTA_THREADS / 32)
#define SAMPLE_MAX_BLOCKS 8
#define SAMPLE_SEGMENTS 32
#define SAMPLE_BINS 2048
#define SAMPLE_SHARE_BYTES (160 * 1024)                        // of a row in a CTA's shared memory, at most (up to 77 KB two CTAs fit an SM)
#define SAMPLE_PIECE 32768                                     // elements of a longer share whose weights are added at a time
#define SAMPLE_NOT_KEPT (-1.0f)
static_assert(SAMPLE_SHARE_BYTES / 4 <= 65535 && SAMPLE_PIECE <= 65535, "parts of weights fit 32 bits");

// Which elements are kept: keys above `low`, and the first `quota` ids among keys equal to `low`.
struct Cut {
    unsigned low;
    int quota;
};

// A weight (0 .. 1) as a whole number of 2^-48 in three parts of 16 bits, whose sums over up to 65,535 elements fit 32 bits each
// (native additions in shared memory; sums of whole numbers do not depend on their order).  A float32 from 2^-25 on is such a number
// itself; a smaller one is off by 2^-49 at most, a million of them together by 2^-29 of the largest weight.  Bins are added up
// across CTAs and along the row in float64, in a fixed order.
struct Fixed {
    unsigned high, mid, low;
};
__device__ __forceinline__ Fixed fixed_weight(float w) {
    const float x = w * 65536.0f, high = floorf(x), y = (x - high) * 65536.0f, mid = floorf(y);      // all exact
    return Fixed{(unsigned)high, (unsigned)mid, __float2uint_rn((y - mid) * 65536.0f)};
}
__device__ __forceinline__ double fixed_value(unsigned high, unsigned mid, unsigned low) {
    return (double)(((unsigned long long)high << 32) + ((unsigned long long)mid << 16) + low) * (1.0 / 281474976710656.0);
}

struct SampleShared {
    Best warp_best[33];                              // block_best's
    Best best;                                       // of this CTA's share; read by the whole cluster, as are the next eight
    int bad;
    // This CTA's histogram.  By count it is `high`; by weight it is the three parts, which give their place (`high` and `mid`) to the
    // words of a float64 when the walk is over; the last digit, of half as many bins, also counts, in the upper half of `high`.
    alignas(16) unsigned high[SAMPLE_BINS];
    alignas(16) unsigned mid[SAMPLE_BINS];
    alignas(16) unsigned low[SAMPLE_BINS];
    unsigned slice_count[SAMPLE_BINS / 4];           // this CTA's slice of the bins, summed over the cluster
    double slice_weight[SAMPLE_BINS / 4];
    int seg_ties[SAMPLE_SEGMENTS];                   // this CTA's segments
    float seg_weight[SAMPLE_SEGMENTS];
    unsigned warp_count[SAMPLE_CTA_WARPS];           // scan over the bins
    double warp_weight[SAMPLE_CTA_WARPS];
    int first, lowest;                               // places in descending order of the bins
    unsigned edge_count, above_count;
    double above_weight;
    int all_ties[SAMPLE_SEGMENTS];
    float all_weight[SAMPLE_SEGMENTS];
    unsigned listed;                                 // of this CTA's candidates (in `high`); read by the whole cluster
};

// What the digit search knows: keys that match `prefix` under `mask` hold the edge, `above` of them (by count or weight)
// lie above it.
struct Edge {
    unsigned prefix, mask, count;     // `count`: elements of the last digit's bin
    unsigned above_count;
    double above_weight, target;      // `target`: the weight that the edge has to reach
};

// One digit of BITS bits.  `walk_elements(piece, add)` walks this CTA's elements of a piece (at most 65,535 of them) and calls
// add(key, w) for those to be counted, w() being an element's weight (the digit's place is applied here); by weight the first bin (from
// the top) whose running weight reaches `share` of all the weight (a float32 product) is chosen, by count the first whose running
// count reaches `wanted`.  By weight a bin without weight counts as empty.  `extra_key`, `extra_weight`: a run of equal keys that the
// elements leave out, added to its bin once.
template <bool BY_WEIGHT, int BITS, typename Walk>
__device__ void sample_digit(cg::cluster_group& cluster, SampleShared& s, unsigned rank, unsigned blocks, int shift, Edge& e,
                             Walk walk_elements, int pieces, float share, unsigned wanted, bool has_extra, unsigned extra_key,
                             double extra_weight) {
    constexpr int BINS = 1 << BITS, OWN = BINS / SAMPLE_CTA_THREADS;      // bins, and bins a thread looks at when the edge is searched
    constexpr bool COUNTED = !BY_WEIGHT || 2 * BINS <= SAMPLE_BINS;
    static_assert(BINS <= SAMPLE_BINS && OWN * SAMPLE_CTA_THREADS == BINS, "whole bins a thread");
    unsigned* count = BY_WEIGHT ? s.high + SAMPLE_BINS / 2 : s.high;
    double held[OWN];                                // weights of bins threadIdx.x, + CTA_THREADS, ...
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int b = threadIdx.x + j * SAMPLE_CTA_THREADS;
        held[j] = 0.0;
        if (COUNTED) count[b] = 0u;
        if (BY_WEIGHT) s.high[b] = 0u, s.mid[b] = 0u, s.low[b] = 0u;
    }
    if (threadIdx.x == 0) s.first = 0x7fffffff, s.lowest = -1;
    __syncthreads();
    for (int piece = 0; piece < pieces; ++piece) {
        walk_elements(piece, [&](unsigned key, auto weight) {
            if ((key & e.mask) != e.prefix) return;
            const unsigned b = (key >> shift) & (BINS - 1u);
            if (COUNTED) atomicAdd(&count[b], 1u);
            if (BY_WEIGHT) {
                const Fixed w = fixed_weight(weight());
                if (w.high) atomicAdd(&s.high[b], w.high);
                if (w.mid) atomicAdd(&s.mid[b], w.mid);
                if (w.low) atomicAdd(&s.low[b], w.low);
            }
        });
        if (!BY_WEIGHT) continue;
        __syncthreads();
        const bool last = piece + 1 == pieces;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int b = threadIdx.x + j * SAMPLE_CTA_THREADS;
            held[j] += fixed_value(s.high[b], s.mid[b], s.low[b]);
            s.high[b] = last ? (unsigned)__double2hiint(held[j]) : 0u;
            s.mid[b] = last ? (unsigned)__double2loint(held[j]) : 0u;
            s.low[b] = 0u;
        }
        if (!last) __syncthreads();
    }
    const bool extra = BY_WEIGHT && has_extra && (extra_key & e.mask) == e.prefix;
    const int extra_bin = (int)((extra_key >> shift) & (BINS - 1u));
    auto weight_in = [&](unsigned r, int bin) {
        return __hiloint2double((int)cluster.map_shared_rank(s.high, r)[bin], (int)cluster.map_shared_rank(s.mid, r)[bin]);
    };
    const int slice = BINS / blocks;
    if (blocks > 1) {
        cluster.sync();
        if ((int)threadIdx.x < slice) {
            const int b = (int)rank * slice + (int)threadIdx.x;
            unsigned c = 0u;
            double w = 0.0;
#pragma unroll
            for (unsigned r = 0; r < SAMPLE_MAX_BLOCKS; ++r) {       // all loads under way together
                if (r >= blocks) continue;
                if (COUNTED) c += cluster.map_shared_rank(count, r)[b];
                if (BY_WEIGHT) w += weight_in(r, b);
            }
            s.slice_count[threadIdx.x] = c;
            if (BY_WEIGHT) s.slice_weight[threadIdx.x] = w;
        }
        cluster.sync();
    } else {
        __syncthreads();
    }
    // bins from the top: thread t has places OWN t .. OWN t + OWN - 1, place p is bin BINS - 1 - p
    unsigned c[OWN], c_sum = 0u;
    double w[OWN], w_sum = 0.0;
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int bin = BINS - 1 - ((int)threadIdx.x * OWN + j);
        c[j] = 0u;
        w[j] = 0.0;
        if (blocks > 1) {
            if (COUNTED) c[j] = cluster.map_shared_rank(s.slice_count, bin / slice)[bin % slice];
            if (BY_WEIGHT) w[j] = cluster.map_shared_rank(s.slice_weight, bin / slice)[bin % slice];
        } else {
            if (COUNTED) c[j] = count[bin];
            if (BY_WEIGHT) w[j] = weight_in(0, bin);
        }
        if (extra && bin == extra_bin) c[j] += 1u, w[j] += extra_weight;
        c_sum += c[j];
        w_sum += w[j];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned c_run = c_sum;
    double w_run = w_sum, w_before = 0.0, w_total = 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        if (!BY_WEIGHT) {
            const unsigned cu = __shfl_up_sync(0xffffffffu, c_run, o);
            if (lane >= o) c_run += cu;
        } else {
            const double wu = __shfl_up_sync(0xffffffffu, w_run, o);
            if (lane >= o) w_run += wu;
        }
    }
    if (BY_WEIGHT) {
        w_before = __shfl_up_sync(0xffffffffu, w_run, 1);
        if (lane == 0) w_before = 0.0;
    }
    if (lane == 31) s.warp_count[warp] = c_run, s.warp_weight[warp] = w_run;
    __syncthreads();
    unsigned c_before = c_run - c_sum;
    for (int i = 0; i < SAMPLE_CTA_WARPS; ++i) {
        if (!BY_WEIGHT && i < warp) c_before += s.warp_count[i];
        if (BY_WEIGHT) {
            if (i == warp) w_before += w_total;
            w_total += s.warp_weight[i];
        }
    }
    if (BY_WEIGHT && e.mask == 0u) e.target = (double)(share * (float)w_total);
    const double goal = BY_WEIGHT ? e.target - e.above_weight : 0.0;
    const unsigned need = wanted - e.above_count;
    {
        unsigned ca = c_before;
        double wa = w_before;
        int found = 0x7fffffff, last = -1;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            if (BY_WEIGHT ? w[j] == 0.0 : c[j] == 0u) continue;
            last = (int)threadIdx.x * OWN + j;
            if (found == 0x7fffffff && (BY_WEIGHT ? wa + w[j] >= goal : ca + c[j] >= need)) found = last;
            ca += c[j];
            wa += w[j];
        }
        if (found != 0x7fffffff) atomicMin(&s.first, found);
        if (last >= 0) atomicMax(&s.lowest, last);
    }
    __syncthreads();
    const int place = s.first != 0x7fffffff ? s.first : max(s.lowest, 0);      // rounding left the sum a hair short: the last bin holds the edge
    if (place / OWN == (int)threadIdx.x) {
        unsigned ca = c_before, here = 0u;
        double wa = w_before;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            if ((int)threadIdx.x * OWN + j < place) ca += c[j], wa += w[j];
            if ((int)threadIdx.x * OWN + j == place) here = c[j];
        }
        s.edge_count = here;
        s.above_count = ca;
        s.above_weight = wa;
    }
    __syncthreads();
    e.prefix |= (unsigned)(BINS - 1 - place) << shift;
    e.mask |= (BINS - 1u) << shift;
    e.count = s.edge_count;
    if (!BY_WEIGHT) e.above_count += s.above_count;
    e.above_weight += s.above_weight;
    // the histogram is written again after the next barrier of the cluster's first kind: every CTA has read its slices by then
}

// Candidates of a threshold.  Elements are binned by how many 64ths of a (natural) logarithm their weight lies below the largest: a
// function that never rises with the key, and that spreads a row over some hundred bins where the keys' first 11 bits (sign, exponent
// and two bits) crowd it into some ten.  What the edge's bin holds (by count: all bins down to it) is then few enough to be sorted in
// every CTA, which finds the threshold without another meeting of the cluster.
#define SAMPLE_LIST 1024
__device__ __forceinline__ float log_steps(float v, float top, float inv_t) { return (top - v) * inv_t * 64.0f; }
__device__ __forceinline__ unsigned log_bin(float v, float top, float inv_t) { return (unsigned)fminf(log_steps(v, top, inv_t), (float)(SAMPLE_BINS - 1)); }

// f(index, value) for this CTA's elements, in shared memory on a 16-byte boundary, four at a time
template <typename F>
__device__ __forceinline__ void each_shared(const float* x, int length, F f) {
#pragma unroll 2
    for (int i = threadIdx.x; i < length / 4; i += SAMPLE_CTA_THREADS) {
        const float4 v = reinterpret_cast<const float4*>(x)[i];
        f(4 * i, v.x), f(4 * i + 1, v.y), f(4 * i + 2, v.z), f(4 * i + 3, v.w);
    }
    const int i = (length & ~3) + threadIdx.x;
    if (i < length) f(i, x[i]);
}

// Gathers the keys for which `wanted(v)` holds from all CTAs and sorts them, largest first, into candidates(s): their count, or -1 if
// they are more than SAMPLE_LIST.  Every CTA gets the same.  The CTA's own go through s.high, all of them through s.mid.
__device__ __forceinline__ unsigned* candidates(SampleShared& s) { return s.mid + SAMPLE_LIST; }
template <typename Wanted>
__device__ int sample_candidates(cg::cluster_group& cluster, SampleShared& s, unsigned blocks, const float* x, int length, Wanted wanted) {
    if (threadIdx.x == 0) s.listed = 0u;
    __syncthreads();
    each_shared(x, length, [&](int, float v) {
        if (!wanted(v)) return;
        const unsigned at = atomicAdd(&s.listed, 1u);
        if (at < SAMPLE_LIST) s.high[at] = ordered_key(v);
    });
    if (blocks > 1) cluster.sync();
    else __syncthreads();
    constexpr int TEAM = SAMPLE_CTA_THREADS / SAMPLE_MAX_BLOCKS;          // threads that bring a CTA's
    const unsigned team = threadIdx.x / TEAM;
    unsigned n = 0u, from = 0u, count = 0u;
#pragma unroll
    for (unsigned r = 0; r < SAMPLE_MAX_BLOCKS; ++r) {
        const unsigned c = r < blocks ? *cluster.map_shared_rank(&s.listed, r) : 0u;
        if (r < team) from += c;
        if (r == team) count = c;
        n += c;
    }
    if (n > SAMPLE_LIST) return -1;
    if (count > 0u) {
        const unsigned* list = cluster.map_shared_rank(s.high, team);
        for (unsigned i = threadIdx.x % TEAM; i < count; i += TEAM) s.mid[from + i] = list[i];
    }
    if (threadIdx.x < (n + 3u) / 4u * 4u - n) s.mid[n + threadIdx.x] = 0u;      // no finite float's key
    __syncthreads();
    // a key's place: how many are larger, or equal and before it; of keys before those of its warp, how many are larger than key - 1
    for (unsigned i = threadIdx.x; i < n; i += SAMPLE_CTA_THREADS) {
        const unsigned key = s.mid[i], base = i & ~31u;
        unsigned place = 0u;
        auto larger = [&](unsigned from, unsigned to, unsigned than) {
#pragma unroll 4
            for (unsigned j = from; j < to; j += 4) {
                const uint4 k = *reinterpret_cast<const uint4*>(s.mid + j);
                place += (unsigned)(k.x > than) + (unsigned)(k.y > than) + (unsigned)(k.z > than) + (unsigned)(k.w > than);
            }
        };
        larger(0u, base, key - 1u);
        for (unsigned j = base; j < min(base + 32u, n); ++j) place += (unsigned)(s.mid[j] > key || (s.mid[j] == key && j < i));
        larger(base + 32u, n, key);
        candidates(s)[place] = key;
    }
    __syncthreads();
    return (int)n;
}

// The first of `n` sorted candidates at which their running weight reaches `goal` (where rounding left the sum a hair short: the last
// that has a weight).  key, the weight of the candidates above it and the count of its equals (among all `listed`).
struct Reached {
    unsigned key;
    int equals;
    double above;
};
__device__ __forceinline__ unsigned long long fixed_units(float w) {
    const Fixed f = fixed_weight(w);
    return ((unsigned long long)f.high << 32) + ((unsigned long long)f.mid << 16) + f.low;
}
// Running sums of the candidates' weights in units of 2^-48 (whole numbers), in place of what `sums` held; their total.
template <typename Weight>
__device__ unsigned long long sample_running(SampleShared& s, int n, Weight weight_of_key, unsigned long long* sums) {
    constexpr int OWN = SAMPLE_LIST / SAMPLE_CTA_THREADS;
    unsigned long long* warps = reinterpret_cast<unsigned long long*>(s.warp_weight);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long own[OWN], run = 0ull;
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int i = threadIdx.x * OWN + j;
        run += i < n ? fixed_units(weight_of_key(candidates(s)[i])) : 0ull;
        own[j] = run;
    }
    unsigned long long before = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += up;
    }
    if (lane == 31) warps[warp] = before;
    before -= run;
    __syncthreads();
    unsigned long long total = 0ull;
    for (int i = 0; i < SAMPLE_CTA_WARPS; ++i) {
        if (i < warp) before += warps[i];
        total += warps[i];
    }
#pragma unroll
    for (int j = 0; j < OWN; ++j) sums[threadIdx.x * OWN + j] = before + own[j];
    if (threadIdx.x == 0) s.first = 0x7fffffff, s.lowest = -1;
    __syncthreads();
    return total;
}
__device__ Reached sample_reached(SampleShared& s, int n, int listed, const unsigned long long* sums, double goal) {
    constexpr double UNIT = 1.0 / 281474976710656.0;
    for (int i = threadIdx.x; i < n; i += SAMPLE_CTA_THREADS) {
        const unsigned long long below = i > 0 ? sums[i - 1] : 0ull;
        if (sums[i] == below) continue;
        atomicMax(&s.lowest, i);
        if ((double)sums[i] * UNIT >= goal && !(i > 0 && (double)below * UNIT >= goal)) atomicMin(&s.first, i);
    }
    __syncthreads();
    const int place = s.first != 0x7fffffff ? s.first : max(s.lowest, 0);
    const unsigned* list = candidates(s);
    const unsigned key = list[place];
    int above = 0, equals = 0;
    for (int base = 0; base < listed; base += SAMPLE_CTA_THREADS) {
        const int i = base + threadIdx.x;
        above += __syncthreads_count(i < listed && list[i] > key);
        equals += __syncthreads_count(i < listed && list[i] == key);
    }
    return Reached{key, equals, above > 0 ? (double)sums[above - 1] * UNIT : 0.0};
}

// The parameters of up to ROWS rows, in the launch itself: reading them from pinned memory takes a row 10 us (24 rows 57 instead of
// 45), a copy to the device a launch.
template <int ROWS>
struct SampleWords {
    unsigned long long seed[ROWS];
    float temperature[ROWS];
    int top_k[ROWS];
    float top_p[ROWS];
    int draw_index[ROWS];
};

// IN_SHARED: the CTA's share of the row lies in shared memory (and gives its place to the weights of the kept set);
// otherwise a row is too long for that and is read from memory each time.
template <bool IN_SHARED, int ROWS>
__global__ void __launch_bounds__(SAMPLE_CTA_THREADS, 2) sample_kernel(
    const float* __restrict__ logits, int vocab, int per_segment, const __grid_constant__ SampleWords<ROWS> params, int* __restrict__ out,
    int* __restrict__ copy) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float share[];
    __shared__ SampleShared s;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank(), blocks = cluster.num_blocks();
    const int r = blockIdx.x / blocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int own_segments = SAMPLE_SEGMENTS / blocks;
    const int begin = min(vocab, (int)rank * own_segments * per_segment);
    const int length = min(vocab, begin + own_segments * per_segment) - begin;      // of this CTA's share
    const float* row = logits + (size_t)r * vocab + begin;
    const float temp = params.temperature[r], p_raw = params.top_p[r];
    const int k_raw = params.top_k[r];

    auto answer = [&](int token) {
        out[r] = token;
        copy[r] = token;
    };
    // Largest logit (also the greedy answer) and a check that the row is finite.
    int bad = 0;
    Best mine = {-CUDART_INF_F, 0x7fffffff};
    auto see = [&](float x, int i) {
        bad |= !(fabsf(x) <= 3.402823466e38f);
        mine = better(mine, Best{x, i});
    };
    int vectors = 0;
    if (((uintptr_t)row & 15) == 0) {
        vectors = length / 4;
#pragma unroll 5
        for (int i = threadIdx.x; i < vectors; i += SAMPLE_CTA_THREADS) {
            const float4 v = reinterpret_cast<const float4*>(row)[i];
            if (IN_SHARED) reinterpret_cast<float4*>(share)[i] = v;
            see(v.x, begin + 4 * i), see(v.y, begin + 4 * i + 1), see(v.z, begin + 4 * i + 2), see(v.w, begin + 4 * i + 3);
        }
    }
#pragma unroll 4
    for (int i = 4 * vectors + threadIdx.x; i < length; i += SAMPLE_CTA_THREADS) {
        const float v = row[i];
        if (IN_SHARED) share[i] = v;
        see(v, begin + i);
    }
    bad = __syncthreads_or(bad);
    mine = block_best(mine, s.warp_best);
    if (threadIdx.x == 0) s.best = mine, s.bad = bad;
    if (blocks > 1) cluster.sync();
    else __syncthreads();
    Best top = s.best;
#pragma unroll
    for (unsigned q = 0; q < SAMPLE_MAX_BLOCKS; ++q) {
        if (q >= blocks) continue;
        top = better(top, *cluster.map_shared_rank(&s.best, q));
        bad |= *cluster.map_shared_rank(&s.bad, q);
    }
    // the same in every CTA of the cluster: they leave together, and none while another still reads its shared memory
    const float inv_t = 1.0f / temp;                 // beyond a float's range: as temperature 0
    if (bad || temp == 0.0f || k_raw == 1 || isinf(inv_t)) {
        if (rank == 0 && threadIdx.x == 0) answer(bad ? -1 : top.id);
        if (blocks > 1) cluster.sync();
        return;
    }
    const float* x = IN_SHARED ? share : row;
    auto weight_of = [&](float v) { return expf((v - top.value) * inv_t); };

    // ---- top_k: the k-th largest key by count ------------------------------------------------
    // Kept are the keys from cut.low on; of those equal to it, where there are more than `quota`, the first ids.
    Cut cut = {0u, 0x7fffffff};
    int ties = 0;                                    // elements of the row whose key is cut.low, where some of them may be left out
    const bool by_count = k_raw > 0 && k_raw < vocab;
    // how many equals of weight `one` it takes from `above` to `target`; a weight of nothing: all of them
    auto equals_to = [](double target, double above, double one) {
        const double missing = (target - above) / one;
        return missing < 2147483647.0 ? max(1, (int)ceil(missing)) : 0x7fffffff;
    };
    bool found = false;                              // both thresholds, from candidates
    if (IN_SHARED && (by_count ? k_raw <= SAMPLE_LIST : p_raw < 1.0f)) {
        Edge e = {0u, 0u, 0u, 0u, 0.0, 0.0};
        auto each = [&](int, auto add) {
            each_shared(x, length, [&](int, float v) { add((SAMPLE_BINS - 1 - log_bin(v, top.value, inv_t)) << 21, [&] { return weight_of(v); }); });
        };
        unsigned long long* sums = reinterpret_cast<unsigned long long*>(s.low);
        static_assert(sizeof(s.low) >= SAMPLE_LIST * sizeof(*sums), "running sums of the candidates");
        auto weight_of_key = [&](unsigned key) { return weight_of(key_value(key)); };
        if (by_count) {
            sample_digit<false, 11>(cluster, s, rank, blocks, 21, e, each, 1, 0.0f, (unsigned)k_raw, false, 0u, 0.0);
            const unsigned edge = SAMPLE_BINS - 1 - (e.prefix >> 21);
            const float end = (float)(edge + 1u);
            const int n = edge + 1u < SAMPLE_BINS && e.above_count + e.count <= SAMPLE_LIST        // the last bin's end is open
                ? sample_candidates(cluster, s, blocks, x, length, [&](float v) { return log_steps(v, top.value, inv_t) < end; }) : -1;
            if (n >= 0) {
                found = true;
                const unsigned* list = candidates(s);
                cut.low = list[k_raw - 1];
                int above = 0;
                for (int base = 0; base < n; base += SAMPLE_CTA_THREADS) {
                    const int i = base + threadIdx.x;
                    above += __syncthreads_count(i < n && list[i] > cut.low);
                    ties += __syncthreads_count(i < n && list[i] == cut.low);
                }
                cut.quota = k_raw - above;
                if (p_raw < 1.0f) {
                    const double total = (double)sample_running(s, k_raw, weight_of_key, sums) * (1.0 / 281474976710656.0);
                    const double target = (double)(p_raw * (float)total);
                    const Reached at = sample_reached(s, k_raw, n, sums, target);
                    const int need = equals_to(target, at.above, (double)fixed_units(weight_of_key(at.key)) * (1.0 / 281474976710656.0));
                    if (at.key == cut.low) {
                        cut.quota = min(cut.quota, need);
                    } else {
                        cut.low = at.key;
                        cut.quota = need;
                        ties = at.equals;
                    }
                }
            }
        } else {
            sample_digit<true, 11>(cluster, s, rank, blocks, 21, e, each, 1, p_raw, 0u, false, 0u, 0.0);
            const unsigned edge = SAMPLE_BINS - 1 - (e.prefix >> 21);
            const float start = (float)edge, end = (float)(edge + 1u);
            const int n = edge + 1u < SAMPLE_BINS
                ? sample_candidates(cluster, s, blocks, x, length,
                                    [&](float v) { const float at = log_steps(v, top.value, inv_t); return at >= start && at < end; }) : -1;
            if (n >= 0) {
                found = true;
                sample_running(s, n, weight_of_key, sums);
                const Reached at = sample_reached(s, n, n, sums, e.target - e.above_weight);
                cut.low = at.key;
                cut.quota = equals_to(e.target, e.above_weight + at.above, (double)fixed_units(weight_of_key(at.key)) * (1.0 / 281474976710656.0));
                ties = at.equals;
            }
        }
        if (!found) {                                // the digits' histograms take the lists' place: no CTA reads them any more
            if (blocks > 1) cluster.sync();
            else __syncthreads();
        }
    }
    if (!found && by_count) {
        Edge e = {0u, 0u, 0u, 0u, 0.0, 0.0};
        auto each = [&](int, auto add) {
#pragma unroll 4
            for (int i = threadIdx.x; i < length; i += SAMPLE_CTA_THREADS) add(ordered_key(x[i]), [] { return 0.0f; });
        };
        sample_digit<false, 11>(cluster, s, rank, blocks, 21, e, each, 1, 0.0f, (unsigned)k_raw, false, 0u, 0.0);
        sample_digit<false, 11>(cluster, s, rank, blocks, 10, e, each, 1, 0.0f, (unsigned)k_raw, false, 0u, 0.0);
        if (e.above_count + e.count == (unsigned)k_raw) {
            cut.low = e.prefix;                      // all keys of the bin are kept, whatever their last digit
        } else {
            sample_digit<false, 10>(cluster, s, rank, blocks, 0, e, each, 1, 0.0f, (unsigned)k_raw, false, 0u, 0.0);
            cut.low = e.prefix;
            cut.quota = k_raw - (int)e.above_count;
            ties = (int)e.count;
        }
    }

    // ---- top_p: the key at which the running weight reaches top_p times the top_k set's weight ---
    if (!found && p_raw < 1.0f) {
        Edge e = {0u, 0u, 0u, 0u, 0.0, 0.0};
        auto counted = [&](float w) {                // a weight as the histograms count it
            const Fixed f = fixed_weight(w);
            return fixed_value(f.high, f.mid, f.low);
        };
        const bool some = cut.quota < ties;          // only some of the equals at the cut: they are added as one
        const unsigned low = cut.low;
        const double low_weight = some ? counted(weight_of(key_value(low))) * cut.quota : 0.0;
        const int pieces = IN_SHARED ? 1 : (length + SAMPLE_PIECE - 1) / SAMPLE_PIECE;
        auto each = [&](int piece, auto add) {
            const int from = IN_SHARED ? 0 : piece * SAMPLE_PIECE, to = IN_SHARED ? length : min(length, from + SAMPLE_PIECE);
#pragma unroll 4
            for (int i = from + threadIdx.x; i < to; i += SAMPLE_CTA_THREADS) {
                const float v = x[i];
                const unsigned key = ordered_key(v);
                if (some ? key > low : key >= low) add(key, [&] { return weight_of(v); });
            }
        };
        sample_digit<true, 11>(cluster, s, rank, blocks, 21, e, each, pieces, p_raw, 0u, some, low, low_weight);
        sample_digit<true, 11>(cluster, s, rank, blocks, 10, e, each, pieces, p_raw, 0u, some, low, low_weight);
        sample_digit<true, 10>(cluster, s, rank, blocks, 0, e, each, pieces, p_raw, 0u, some, low, low_weight);
        const double one = counted(weight_of(key_value(e.prefix)));
        const int need = equals_to(e.target, e.above_weight, one);
        if (some && e.prefix == cut.low) {
            cut.quota = min(cut.quota, need);
        } else {
            cut.low = e.prefix;
            cut.quota = need;
            ties = (int)e.count;
        }
    }

    // ---- the kept set's weights, segment by segment in id order -------------------------------------
    // Where only some of the equals at the cut are kept (the first ids), a segment has to know how many come before it.
    const bool ranked = cut.quota < ties;
    const int first_segment = (int)rank * own_segments;
    auto share_segments = [&]() {                     // every CTA gets all segments' numbers
        if (blocks > 1) cluster.sync();
        else __syncthreads();
    };
    if (ranked) {
        for (int g = warp; g < own_segments; g += SAMPLE_CTA_WARPS) {
            const int from = g * per_segment, to = min(length, from + per_segment);
            int n = 0;
            for (int i = from + lane; i < to; i += 32) n += ordered_key(x[i]) == cut.low;
            n = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0) s.seg_ties[g] = n;
        }
        share_segments();
        if (threadIdx.x < SAMPLE_SEGMENTS) s.all_ties[threadIdx.x] = cluster.map_shared_rank(s.seg_ties, threadIdx.x / own_segments)[threadIdx.x % own_segments];
        __syncthreads();
    }
    // f(i, weight or SAMPLE_NOT_KEPT) for 32 neighbouring elements of segment g at a time
    auto walk = [&](int g, auto f) {
        const int from = g * per_segment, to = min(length, from + per_segment);
        int seen = 0;
        if (ranked)
            for (int j = 0; j < first_segment + g; ++j) seen += s.all_ties[j];
        for (int base = from; base < to; base += 32) {
            const int i = base + lane;
            const bool live = i < to;
            const float v = live ? x[i] : 0.0f;
            const unsigned key = live ? ordered_key(v) : 0u;
            bool kept = live && key >= cut.low;
            if (ranked) {
                const bool tie = live && key == cut.low;
                const unsigned tie_mask = __ballot_sync(0xffffffffu, tie);
                if (tie) kept = seen + __popc(tie_mask & ((1u << lane) - 1u)) < cut.quota;
                seen += __popc(tie_mask);
            }
            f(i, live, kept ? weight_of(v) : SAMPLE_NOT_KEPT);
        }
    };
    if (IN_SHARED) {                                  // the weights take the logits' place
        if (ranked) {
            for (int g = warp; g < own_segments; g += SAMPLE_CTA_WARPS)
                walk(g, [&](int i, bool live, float w) { if (live) share[i] = w; });
        } else {
            each_shared(share, length, [&](int i, float v) { share[i] = ordered_key(v) >= cut.low ? weight_of(v) : SAMPLE_NOT_KEPT; });
        }
        __syncthreads();
    }
    auto weights = [&](int g, auto f) {
        if constexpr (IN_SHARED) {
            const int from = g * per_segment, to = min(length, from + per_segment);
#pragma unroll 8
            for (int base = from; base < to; base += 32) f(base + lane, base + lane < to, base + lane < to ? share[base + lane] : SAMPLE_NOT_KEPT);
        } else {
            walk(g, f);
        }
    };
    for (int g = warp; g < own_segments; g += SAMPLE_CTA_WARPS) {
        float local = 0.0f;
        weights(g, [&](int, bool, float w) { local += w >= 0.0f ? w : 0.0f; });
        local = warp_sum(local);
        if (lane == 0) s.seg_weight[g] = local;
    }
    share_segments();
    if (threadIdx.x < SAMPLE_SEGMENTS) s.all_weight[threadIdx.x] = cluster.map_shared_rank(s.seg_weight, threadIdx.x / own_segments)[threadIdx.x % own_segments];
    if (blocks > 1) cluster.sync();                   // behind it no CTA reads another's shared memory
    else __syncthreads();

    // ---- inverse CDF over the kept set in id order ------------------------------------------------
    float of_segment[SAMPLE_SEGMENTS], retained = 0.0f;
#pragma unroll
    for (int g = 0; g < SAMPLE_SEGMENTS; ++g) of_segment[g] = s.all_weight[g];
#pragma unroll
    for (int g = 0; g < SAMPLE_SEGMENTS; ++g) retained += of_segment[g];
    const float u = uniform_from_counter(params.seed[r], (unsigned long long)params.draw_index[r]) * retained;
    float run = 0.0f, before_last = 0.0f;
    int chosen = -1, last = 0;
#pragma unroll
    for (int g = 0; g < SAMPLE_SEGMENTS; ++g) {
        if (chosen >= 0 || of_segment[g] <= 0.0f) continue;
        const float with = run + of_segment[g];
        last = g;
        before_last = with - of_segment[g];
        if (with > u) chosen = g;
        else run = with;
    }
    if (chosen < 0) {
        chosen = last;
        run = before_last;
    }
    if (chosen / own_segments != (int)rank) return;
    chosen %= own_segments;
    // running weights of 32 neighbouring elements
    auto scan = [&](float w) {
        float cum = w >= 0.0f ? w : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, cum, o);
            if (lane >= o) cum += up;
        }
        return cum;
    };
    if constexpr (IN_SHARED) {
        // Every warp scans some of the segment's groups of 32; one thread then adds the groups' weights in order and stops at the
        // group that u falls into: some kept element's running weight is above it, which the largest tells.
        const int from = chosen * per_segment, to = min(length, from + per_segment), groups = (to - from + 31) / 32;      // at most BINS
        float *weight = reinterpret_cast<float*>(s.high), *largest = reinterpret_cast<float*>(s.low);
        for (int g = warp; g < groups; g += SAMPLE_CTA_WARPS) {
            const int i = from + 32 * g + lane;
            const float w = i < to ? share[i] : SAMPLE_NOT_KEPT, cum = scan(w);
            const float top_cum = warp_max(w >= 0.0f ? cum : -1.0f);
            if (lane == 31) weight[g] = cum, largest[g] = top_cum;
        }
        __syncthreads();
        if (warp != 0) return;
        int group = -1, last_group = 0;
        for (int base = 0; base < groups && group < 0; base += 32) {         // 32 groups' numbers in the lanes; every lane adds them
            const float mine = base + lane < groups ? weight[base + lane] : 0.0f, top_mine = base + lane < groups ? largest[base + lane] : -1.0f;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const float step = __shfl_sync(0xffffffffu, mine, k), top_step = __shfl_sync(0xffffffffu, top_mine, k);
                if (group >= 0) continue;
                if (top_step >= 0.0f) {
                    last_group = base + k;
                    if (run + top_step > u) group = base + k;
                }
                if (group < 0) run += step;
            }
        }
        const int g = group >= 0 ? group : last_group, i = from + 32 * g + lane;
        const float w = i < to ? share[i] : SAMPLE_NOT_KEPT, cum = scan(w);
        const unsigned hit = __ballot_sync(0xffffffffu, w >= 0.0f && run + cum > u), kept = __ballot_sync(0xffffffffu, w >= 0.0f);
        if (lane == 0) answer(begin + from + 32 * g + (group >= 0 ? __ffs(hit) - 1 : 31 - __clz(kept)));
    } else {
        if (warp != 0) return;
        int picked = -1, last_kept = -1;
        walk(chosen, [&](int i, bool, float w) {
            const float cum = scan(w);
            const unsigned hit = __ballot_sync(0xffffffffu, w >= 0.0f && run + cum > u), kept = __ballot_sync(0xffffffffu, w >= 0.0f);
            if (picked < 0 && hit) picked = begin + i - lane + (__ffs(hit) - 1);
            if (kept) last_kept = begin + i - lane + (31 - __clz(kept));
            run += __shfl_sync(0xffffffffu, cum, 31);
        });
        if (lane == 0) answer(picked >= 0 ? picked : last_kept);
    }
}

template <int ROWS>
static int launch_sample(const float* logits, int rows, int vocab, const SampleWords<ROWS>& params, int* out, int* copy, void* stream) {
    const int per_segment = (int)((((long long)vocab + SAMPLE_SEGMENTS - 1) / SAMPLE_SEGMENTS + 31) & ~31LL);
    // short rows gain nothing from more CTAs: their meetings cost more than the walks
    const int blocks = vocab >= 65536 ? 8 : (vocab >= 8192 ? 4 : 1);
    const size_t share = (size_t)per_segment * (SAMPLE_SEGMENTS / blocks) * sizeof(float);
    const bool in_shared = share <= SAMPLE_SHARE_BYTES;
    static PerDevice configured;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(sample_kernel<true, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_SHARE_BYTES);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)rows * blocks);
    config.blockDim = dim3(SAMPLE_CTA_THREADS);
    config.dynamicSmemBytes = in_shared ? share : 0;
    config.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = blocks, attributes[0].val.clusterDim.y = 1, attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    static const bool plain = getenv("MRS_PLAIN_LAUNCH") != nullptr;
    config.attrs = attributes;
    config.numAttrs = plain ? 1 : 2;
    const cudaError_t e = in_shared ? cudaLaunchKernelEx(&config, sample_kernel<true, ROWS>, logits, vocab, per_segment, params, out, copy)
                                    : cudaLaunchKernelEx(&config, sample_kernel<false, ROWS>, logits, vocab, per_segment, params, out, copy);
    if (e != cudaSuccess) return (int)e;
    MRS_RETURN_LAUNCH_STATUS();
}

template <int ROWS>
static int launch_sample_words(const float* logits, int first, int count, int rows, int vocab, const unsigned char* words, int* out, int* copy,
                               void* stream) {
    SampleWords<ROWS> w = {};
    const size_t n = (size_t)rows, bytes = 4 * (size_t)count;
    memcpy(w.seed, words + 8 * (size_t)first, 2 * bytes);
    memcpy(w.temperature, words + 8 * n + 4 * (size_t)first, bytes);
    memcpy(w.top_k, words + 12 * n + 4 * (size_t)first, bytes);
    memcpy(w.top_p, words + 16 * n + 4 * (size_t)first, bytes);
    memcpy(w.draw_index, words + 20 * n + 4 * (size_t)first, bytes);
    return launch_sample(logits + (size_t)first * vocab, count, vocab, w, out + first, copy + first, stream);
}

// `words`, in the host's memory and read before this returns: all rows' seeds, then their temperatures, top_k (<= 0: off), top_p and draw
// indices.  out[r] = the token, or -1 when the row holds a NaN or an infinity; copy[r] = out[r], in pinned memory: complete when the
// stream has come here.
MRS_EXPORT int mrs_sample_words(const float* logits, int rows, int vocab, const unsigned char* words, int* out, int* copy, void* stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0 || rows > 0x7fffffff / 8 || !words || !copy) return MRS_BAD_ARGUMENT;
    constexpr int FEW = 32, MANY = 160;                      // 4 KB of arguments
    for (int first = 0; first < rows; first += MANY) {
        const int count = rows - first < MANY ? rows - first : MANY;
        const int code = count <= FEW ? launch_sample_words<FEW>(logits, first, count, rows, vocab, words, out, copy, stream)
                                      : launch_sample_words<MANY>(logits, first, count, rows, vocab, words, out, copy, stream);
        if (code != 0) return code;
    }
    return 0;
}
