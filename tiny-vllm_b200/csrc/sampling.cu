// Next-token sampling, a cluster of 8 CTAs per row of logits (each takes an eighth of the
// vocabulary; partial results meet through distributed shared memory): greedy argmax, or
// temperature with optional top-k and top-p and an exponential race as the draw.
//
// Follows tinyvllm/sampling.py: argmax for temperature 0 (:42-43); scores =
// (logits - max) / temperature in float32 (:82-104); the k largest scores stay
// (:107-112); softmax over them; a token stays under top-p while the mass of the
// tokens sorted before it does not exceed top_p (:125-139); the draw is
// argmax(p / noise), noise ~ Exp(1) (:141-157).  Ties go to the smaller token id.
// Ties exactly at the top-p boundary all stay.
//
// The noise is counter-based instead of a generator carried from step to step:
// token i of draw number n of a request with seed s takes word i % 4 of
// Philox-4x32-10(counter = (i / 4, n_lo, n_hi, 0), key = (s_lo, s_hi)),
// u = ((word >> 9) + 0.5) / 2^23, noise = -log(u).  A request's tokens thus do not
// depend on what else is in the batch or on the order of the rows.
//
// No sort: the thresholds are found three bits of the ordered bit pattern at a time.  A pass counts (top-k) or adds
// up (top-p) the tokens of the eight continuations of the bits found so far; eleven passes settle all 32 bits, and
// the last one also says how many tokens equal the threshold.  A CTA keeps its part of the row's scores in shared
// memory, each thread its own four tokens of every 2,048, so a pass reads nothing from global memory and costs two block barriers and
// one of the cluster.  Rows too long for that (more than about 430,000 tokens) read the logits in every pass.
//
// Bound by the passes' barriers and compares.  Measured over 151,936 tokens (us; one bit a pass over the logits in L2 /
// this): 48 rows, half of them greedy, a quarter top-k 50, a quarter top-p 0.95 680 / 128; one row of top-k 50 496 / 52,
// of top-p 0.95 645 / 77, of both 1,013 / 89; 64 rows of both 1,083 / 343.  Greedy rows alone are slower for it: one
// 4.1 / 4.4, 32 4.9 / 5.9, 37 5.1 / 9.6 (33 clusters of this shared memory fit at once), 38 5.1 / 7.5, 64 6.1 / 8.8.
#include "common.cuh"

#include <cstdint>

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define SAMPLE_THREADS 512
#define SAMPLE_WARPS (SAMPLE_THREADS / 32)
#define SAMPLE_CTAS 8           // CTAs (one cluster) that share a row
#define SAMPLE_DIGIT 3          // bits of the threshold that a pass settles
#define SAMPLE_BINS (1 << SAMPLE_DIGIT)
#define SAMPLE_STAGED_BYTES (208 * 1024)
#define SAMPLE_ROWS_AT_ONCE (2 * 148 / SAMPLE_CTAS)

__device__ __forceinline__ uint32_t ordered_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                              uint32_t k0, uint32_t k1, uint32_t out[4]) {
#pragma unroll
    for (int round = 0; round < 10; ++round) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// What the CTAs of a row's cluster tell one another: every reduction below ends with each CTA's
// partial result in slot [buffer][rank] of every CTA's copy, written through distributed shared
// memory, and one cluster barrier; the buffers alternate, so a slot is not written again before
// every CTA has read it (it has to pass the barrier in between).
struct SampleShared {
    uint32_t warp_key[SAMPLE_WARPS];
    int warp_i[SAMPLE_WARPS];
    uint32_t part_key[2][SAMPLE_CTAS];
    int part_i[2][SAMPLE_CTAS];
    uint32_t warp_bins[SAMPLE_BINS][SAMPLE_WARPS];
    uint32_t part_bins[2][SAMPLE_CTAS][SAMPLE_BINS];       // counts, or sums as their bits
};

struct RowTeam {
    cg::cluster_group cluster;
    SampleShared* sh;
    int rank;
    int phase;
    bool joined;                            // the cluster's CTAs all run: waited for before the first remote store

    // count of this CTA alone
    __device__ __forceinline__ int local_sum(int v) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        v = __reduce_add_sync(0xffffffffu, v);
        __syncthreads();
        if (lane == 0) sh->warp_i[warp] = v;
        __syncthreads();
        int total = 0;
#pragma unroll
        for (int w = 0; w < SAMPLE_WARPS; ++w) total += sh->warp_i[w];
        return total;
    }

    // The eight bins of every thread, added up: lanes, warps, then CTAs, in a fixed order.  part_bins[the phase returned]
    // holds every CTA's sums afterwards; it stays until the next but one call.
    template <typename V> __device__ __forceinline__ int sum_bins(const V* bins, V* totals) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int b = 0; b < SAMPLE_BINS; ++b) {
            uint32_t bits;
            if constexpr (sizeof(V) == 4 && V(0.5f) != V(0)) bits = __float_as_uint(warp_sum(bins[b]));
            else bits = __reduce_add_sync(0xffffffffu, (uint32_t)bins[b]);
            if (lane == b) sh->warp_bins[b][warp] = bits;
        }
        __syncthreads();
        if (warp == 0) {
            const int b = lane % SAMPLE_BINS;
            V total = 0;
#pragma unroll
            for (int w = 0; w < SAMPLE_WARPS; ++w) total = add(total, value_of<V>(sh->warp_bins[b][w]));
            // lanes 8 r .. 8 r + 7 write to the CTAs r and r + 4
#pragma unroll
            for (int r = lane / SAMPLE_BINS; r < SAMPLE_CTAS; r += 32 / SAMPLE_BINS)
                cluster.map_shared_rank(sh, r)->part_bins[phase][rank][b] = bits_of(total);
        }
        cluster.sync();
#pragma unroll
        for (int b = 0; b < SAMPLE_BINS; ++b) {
            V total = value_of<V>(sh->part_bins[phase][0][b]);
#pragma unroll
            for (int r = 1; r < SAMPLE_CTAS; ++r) total = add(total, value_of<V>(sh->part_bins[phase][r][b]));
            totals[b] = total;
        }
        const int used = phase;
        phase ^= 1;
        return used;
    }
    static __device__ __forceinline__ int add(int a, int b) { return a + b; }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ uint32_t bits_of(int v) { return (uint32_t)v; }
    static __device__ __forceinline__ uint32_t bits_of(float v) { return __float_as_uint(v); }
    template <typename V> static __device__ __forceinline__ V value_of(uint32_t bits) {
        if constexpr (V(0.5f) != V(0)) return __uint_as_float(bits); else return (int)bits;
    }

    // (key, index) of the largest key, the smaller index among equals
    static __device__ __forceinline__ void warp_best(uint32_t& key, int& index) {
        const uint32_t top = __reduce_max_sync(0xffffffffu, key);
        index = (int)__reduce_min_sync(0xffffffffu, key == top ? (uint32_t)index : 0x7fffffffu);
        key = top;
    }

    // argmax of (value, smaller index wins ties) of values that are numbers or -inf; every thread of every CTA gets it
    __device__ __forceinline__ void argmax(float& value, int& index) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t key = ordered_key(__fadd_rn(value, 0.0f));       // -0 and 0 are equals
        warp_best(key, index);
        __syncthreads();
        if (lane == 0) { sh->warp_key[warp] = key; sh->warp_i[warp] = index; }
        __syncthreads();
        if (warp == 0) {
            key = sh->warp_key[lane % SAMPLE_WARPS];
            index = sh->warp_i[lane % SAMPLE_WARPS];
            warp_best(key, index);
            if (lane < SAMPLE_CTAS) {                             // lane r tells CTA r
                SampleShared* other = cluster.map_shared_rank(sh, lane);
                other->part_key[phase][rank] = key;
                other->part_i[phase][rank] = index;
            }
        }
        cluster.sync();
        key = sh->part_key[phase][lane % SAMPLE_CTAS];
        index = sh->part_i[phase][lane % SAMPLE_CTAS];
        warp_best(key, index);
        value = __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
        phase ^= 1;
    }
};

// The token of one row.  ARGMAX: greedy rows alone, others are left; else STAGED says whether the scores stay in shared
// memory (room for this CTA's part of the row).
template <typename T, bool STAGED, bool ARGMAX>
__device__ __forceinline__ void sample_row(RowTeam& team, SampleShared& shared, float* staged, int row, const T* logits,
                                           int64_t row_stride, int vocab, const int* __restrict__ packed, int capacity,
                                           int* __restrict__ tokens) {
    const int tid = threadIdx.x;
    const T* x = logits + (int64_t)row * row_stride;
    // this CTA's part of the row: whole groups of four tokens (they share a block of noise)
    const int part = ((vocab + SAMPLE_CTAS - 1) / SAMPLE_CTAS + 3) / 4 * 4;
    const int begin = min(vocab, team.rank * part), end = min(vocab, begin + part);
    const int first_quad = begin / 4 + tid, quads_end = (end + 3) / 4;       // begin < end: begin is a multiple of four
    const bool any = begin < end;
    const bool wide = sizeof(T) == 4 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    // a token that is not there: a bit pattern below every score's (no arithmetic gives it)
    const float absent = __uint_as_float(0xffffffffu);

    auto load_quad = [&](int quad, float* v) {
        if (wide && quad * 4 + 4 <= end) {
            const float4 f = reinterpret_cast<const float4*>(x)[quad];
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = quad * 4 + e < end ? to_float<T>(x[quad * 4 + e]) : absent;
        }
    };
    float best = -INFINITY;
    int best_index = 0x7fffffff;
    const float temp = __int_as_float(packed[row]);
    const bool greedy = !(temp > 0.0f);
    auto meet = [&](int quad, const float* v) {
        if (STAGED && !ARGMAX && !greedy) reinterpret_cast<float4*>(staged)[quad - begin / 4] = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (v[e] > best) { best = v[e]; best_index = 4 * quad + e; }     // (absent is greater than nothing)
    };
    // whole words without a condition between their loads, so that several are in flight; then what is left
    int quad = first_quad;
    if (any && wide)
#pragma unroll 5
        for (; quad < end / 4; quad += SAMPLE_THREADS) {
            const float4 f = reinterpret_cast<const float4*>(x)[quad];
            const float v[4] = {f.x, f.y, f.z, f.w};
            meet(quad, v);
        }
    for (; any && quad < quads_end; quad += SAMPLE_THREADS) {
        float v[4];
        load_quad(quad, v);
        meet(quad, v);
    }
    if (!team.joined) {
        cluster_wait();
        team.joined = true;
    }
    team.argmax(best, best_index);
    if (ARGMAX || greedy || best_index == 0x7fffffff) {           // the same in every CTA of the row
        if (tid == 0 && team.rank == 0) tokens[row] = best_index == 0x7fffffff ? 0 : best_index;
        return;
    }
    if constexpr (!ARGMAX) {
    const float row_max = best;
    // Four scores of this thread; a token past the row's end comes as `absent`, whose key is 0.
    auto make_scores = [&](int quad, float* v) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            v[e] = quad * 4 + e < end ? __fdiv_rn(__fsub_rn(v[e], row_max), temp) : absent;
    };
    if constexpr (STAGED) {                                      // every thread its own: no barrier
        for (int quad = first_quad; any && quad < quads_end; quad += SAMPLE_THREADS) {
            float4& at = reinterpret_cast<float4*>(staged)[quad - begin / 4];
            float v[4] = {at.x, at.y, at.z, at.w};
            make_scores(quad, v);
            at = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    auto scores_of = [&](int quad, float* v) {
        if constexpr (STAGED) {
            const float4 f = reinterpret_cast<const float4*>(staged)[quad - begin / 4];
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
            load_quad(quad, v);
            make_scores(quad, v);
        }
    };

    // ---- top-k: the k-th largest key, then how many of its equals stay
    const int k = packed[2 * capacity + row];
    const bool use_k = k > 0 && k < vocab;
    uint32_t k_key = 0;
    int k_index_limit = vocab;
    if (use_k) {
        int above = 0, equal = 0, used = 0;
        for (int shift = 30; shift >= 0; shift -= SAMPLE_DIGIT) {            // 2 bits, then ten times 3
            int bins[SAMPLE_BINS], totals[SAMPLE_BINS];
#pragma unroll
            for (int b = 0; b < SAMPLE_BINS; ++b) bins[b] = 0;
            const uint32_t found = shift == 30 ? 0u : k_key >> (shift + SAMPLE_DIGIT);
            int quad = any ? first_quad : quads_end;
            while (quad < quads_end) {
                unsigned long long packed_bins = 0;                          // a byte a bin
                for (int n = 0; n < 63 && quad < quads_end; ++n, quad += SAMPLE_THREADS) {
                    float v[4];
                    scores_of(quad, v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint32_t digits = ordered_key(v[e]) >> shift;
                        const bool in = quad * 4 + e < end && (shift == 30 || digits >> SAMPLE_DIGIT == found);
                        packed_bins += in ? 1ull << (8 * (digits & (SAMPLE_BINS - 1))) : 0ull;
                    }
                }
#pragma unroll
                for (int b = 0; b < SAMPLE_BINS; ++b) bins[b] += (int)(packed_bins >> (8 * b)) & 255;
            }
            used = team.sum_bins(bins, totals);
            // the largest digit from which on k tokens lie
            int digit = 0;
            int larger = above;
#pragma unroll
            for (int b = SAMPLE_BINS - 1; b > 0; --b)
                if (digit == 0) {
                    if (larger + totals[b] >= k) digit = b; else larger += totals[b];
                }
            above = larger;
            k_key |= (uint32_t)digit << shift;
#pragma unroll
            for (int b = 0; b < SAMPLE_BINS; ++b) if (b == digit) equal = totals[b];
        }
        int wanted = k - above;
        if (equal > wanted) {              // ties: the first `wanted` of them by token id
            const int last_digit = k_key & (SAMPLE_BINS - 1);
            for (int r = 0; r < team.rank; ++r) wanted -= (int)shared.part_bins[used][r][last_digit];
            // of this CTA's equals the first `wanted` stay (none, or all, where that says so)
            if (wanted <= 0) k_index_limit = begin;
            else if (wanted >= (int)shared.part_bins[used][team.rank][last_digit]) k_index_limit = end;
            else {
                int lo = begin, hi = end;
                while (lo < hi) {
                    const int mid = lo + (hi - lo) / 2;
                    int count = 0;
                    for (int quad = first_quad; quad < quads_end && quad * 4 < mid; quad += SAMPLE_THREADS) {
                        float v[4];
                        scores_of(quad, v);
#pragma unroll
                        for (int e = 0; e < 4; ++e) count += quad * 4 + e < mid && ordered_key(v[e]) == k_key;
                    }
                    if (team.local_sum(count) >= wanted) hi = mid; else lo = mid + 1;
                }
                k_index_limit = lo;
            }
        }
    }
#define KEPT_K(key, i) (!use_k || (key) > k_key || ((key) == k_key && (i) < k_index_limit))

    // ---- top-p: the smallest key kappa with mass(keys above kappa) <= top_p
    const float p_limit = __int_as_float(packed[capacity + row]);
    uint32_t p_key = 0;
    if (p_limit < 1.0f) {
        float above = 0.0f, total = 0.0f;
        for (int shift = 30; shift >= 0; shift -= SAMPLE_DIGIT) {
            float bins[SAMPLE_BINS], totals[SAMPLE_BINS];
#pragma unroll
            for (int b = 0; b < SAMPLE_BINS; ++b) bins[b] = 0.0f;
            const uint32_t found = shift == 30 ? 0u : p_key >> (shift + SAMPLE_DIGIT);
            for (int quad = first_quad; any && quad < quads_end; quad += SAMPLE_THREADS) {
                float v[4];
                scores_of(quad, v);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t key = ordered_key(v[e]), digits = key >> shift;
                    if ((shift == 30 || digits >> SAMPLE_DIGIT == found) && quad * 4 + e < end && KEPT_K(key, quad * 4 + e)) {
                        const float mass = expf(v[e]);
                        const uint32_t digit = digits & (SAMPLE_BINS - 1);
#pragma unroll
                        for (int b = 0; b < SAMPLE_BINS; ++b) bins[b] = __fadd_rn(bins[b], digit == b ? mass : 0.0f);
                    }
                }
            }
            team.sum_bins(bins, totals);
            if (shift == 30) {
#pragma unroll
                for (int b = SAMPLE_BINS - 1; b >= 0; --b) total = __fadd_rn(total, totals[b]);
            }
            // the smallest digit above all of whose keys no more than top_p lies
            int digit = shift == 30 ? 3 : SAMPLE_BINS - 1;
            float larger = above;
#pragma unroll
            for (int b = SAMPLE_BINS - 1; b > 0; --b)
                if (digit == b) {
                    const float next = __fadd_rn(larger, totals[b]);
                    if (__fdiv_rn(next, total) <= p_limit) { digit = b - 1; larger = next; }
                }
            above = larger;
            p_key |= (uint32_t)digit << shift;
        }
    }

    // ---- the race
    const uint32_t seed_lo = (uint32_t)packed[3 * capacity + row], seed_hi = (uint32_t)packed[4 * capacity + row];
    const uint32_t draw_lo = (uint32_t)packed[5 * capacity + row], draw_hi = (uint32_t)packed[6 * capacity + row];
    float win = -INFINITY;
    int win_index = 0x7fffffff;
    // a thread takes four consecutive tokens at a time: they share one Philox block
    for (int quad = first_quad; any && quad < quads_end; quad += SAMPLE_THREADS) {
        float v[4];
        scores_of(quad, v);
        bool in[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t key = ordered_key(v[e]);
            in[e] = quad * 4 + e < end && key >= p_key && KEPT_K(key, quad * 4 + e);
        }
        if (!(in[0] || in[1] || in[2] || in[3])) continue;
        uint32_t words[4];
        philox4x32_10((uint32_t)quad, draw_lo, draw_hi, 0u, seed_lo, seed_hi, words);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (!in[e]) continue;
            const float u = __fmul_rn(__fadd_rn((float)(words[e] >> 9), 0.5f), 1.0f / 8388608.0f);
            const float ratio = __fdiv_rn(expf(v[e]), -logf(u));
            if (ratio > win) { win = ratio; win_index = quad * 4 + e; }
        }
    }
    team.argmax(win, win_index);
    if (tid == 0 && team.rank == 0) tokens[row] = win_index == 0x7fffffff ? best_index : win_index;
#undef KEPT_K
    }
}

// Which rows a launch takes: all of them, the greedy ones, or the others (a cluster then takes several in turn).
enum SampleRows { ALL_ROWS, GREEDY_ROWS, OTHER_ROWS };

template <typename T, bool STAGED, SampleRows WHICH>
__global__ void __launch_bounds__(SAMPLE_THREADS, WHICH == GREEDY_ROWS ? 4 : 2)
sample_rows_kernel(const T* logits, int64_t row_stride, int rows, int vocab,   // logits: from a kernel before
                   const int* __restrict__ packed, int capacity, int* __restrict__ tokens) {
    __shared__ SampleShared shared;
    extern __shared__ __align__(16) float staged[];
    RowTeam team{cg::this_cluster(), &shared, (int)(blockIdx.x % SAMPLE_CTAS), 0, false};
    cluster_arrive();                       // this CTA runs; waited for before the first remote store
    if (WHICH != OTHER_ROWS) pdl_wait();
    // What both launches read is there: the one for the other rows may begin, to see whether it has any, and waits
    // for this one where it does.
    if (WHICH == GREEDY_ROWS) pdl_launch_dependents();
    for (int row = blockIdx.x / SAMPLE_CTAS; row < rows; row += gridDim.x / SAMPLE_CTAS) {
        const bool greedy = !(__int_as_float(packed[row]) > 0.0f);
        if ((WHICH == GREEDY_ROWS && !greedy) || (WHICH == OTHER_ROWS && greedy)) continue;
        if (WHICH == OTHER_ROWS && !team.joined) pdl_wait();
        sample_row<T, STAGED, WHICH == GREEDY_ROWS>(team, shared, staged, row, logits, row_stride, vocab, packed, capacity, tokens);
    }
    if (!team.joined) {
        // A CTA without a row of its own waits too: with nothing but greedy rows this grid would else end, and what follows
        // it start, while the launch for the greedy ones still writes its tokens.
        if (WHICH == OTHER_ROWS) pdl_wait();
        cluster_wait();
    }
}

// bytes of shared memory that a CTA's part of a row takes; 0: more than there is
static int staged_bytes(int vocab) {
    const long long part = (((long long)vocab + SAMPLE_CTAS - 1) / SAMPLE_CTAS + 3) / 4 * 4;
    return part * 4 <= SAMPLE_STAGED_BYTES ? (int)part * 4 : 0;
}

static bool two_launches(int rows, int vocab) { return rows > SAMPLE_ROWS_AT_ONCE && staged_bytes(vocab) > 0; }

// pdl: 1 for the programmatic launch behind the kernel before, 2 for that of the second launch behind the first
template <typename T>
static cudaError_t launch_sample_rows(const void* logits, long long row_stride, int rows, int vocab, const int* packed,
                                      int capacity, int* tokens, int pdl, cudaStream_t s) {
    const int bytes = staged_bytes(vocab);
    auto launch = [&](auto kernel, int clusters, int shared, int pdl) -> cudaError_t {
        // (one limit for all sizes: a smaller one could come between another thread's limit and its launch)
        cudaError_t e = shared ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_STAGED_BYTES) : cudaSuccess;
        if (e != cudaSuccess) return e;
        TvbLaunch launch(dim3(clusters * SAMPLE_CTAS), dim3(SAMPLE_THREADS), shared, s, pdl, SAMPLE_CTAS);
        return cudaLaunchKernelEx(&launch.config, kernel, (const T*)logits, (int64_t)row_stride, rows, vocab, packed, capacity, tokens);
    };
    // The shared memory leaves room for two CTAs an SM.  Rows beyond those that fit at once would make greedy rows,
    // which do not use it, wait in line: they get a launch without it (64 greedy rows of 151,936 tokens: 17.6 us in one
    // launch, 8.8 in two).  With the line at the 33 clusters that fit, 34 to 44 rows were up to 15 % quicker with one kind
    // of sampling, but mixed rows 9 % slower and 48 rows up to 6 %.
    if (!two_launches(rows, vocab))
        return bytes ? launch(sample_rows_kernel<T, true, ALL_ROWS>, rows, bytes, pdl & 1)
                     : launch(sample_rows_kernel<T, false, ALL_ROWS>, rows, 0, pdl & 1);
    const cudaError_t e = launch(sample_rows_kernel<T, false, GREEDY_ROWS>, rows, 0, pdl & 1);
    return e != cudaSuccess ? e : launch(sample_rows_kernel<T, true, OTHER_ROWS>, SAMPLE_ROWS_AT_ONCE, bytes, pdl >> 1);
}

// launches that sampling so many rows takes
extern "C" int tvb_sample_rows_launches(int rows, int vocab) { return rows <= 0 ? 0 : two_launches(rows, vocab) ? 2 : 1; }

// packed: int32 [7, capacity], field-major: temperature and top_p as float bits, top_k,
// seed low/high word, draw-counter low/high word; row r reads column r.
extern "C" int tvb_sample_rows(const void* logits, long long row_stride, int rows, int vocab,
                               const int* packed, int capacity, int* tokens, int dtype, int pdl,
                               void* stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0 || capacity < rows) return TVB_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (dtype == TVB_F32) e = launch_sample_rows<float>(logits, row_stride, rows, vocab, packed, capacity, tokens, pdl, s);
    else if (dtype == TVB_BF16) e = launch_sample_rows<bf16>(logits, row_stride, rows, vocab, packed, capacity, tokens, pdl, s);
    else return TVB_BAD_ARGUMENT;
    return e == cudaSuccess ? tvb_last_error() : (int)e;
}
