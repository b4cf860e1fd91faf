// Float32 attention for heads of 64 or 128 without any extra (bias, cap, sink, gate, kept keys): the arithmetic of
// the row kernel, a block of keys at a time.
//
// A row's keys are cut into chunks of ATTN_CHUNK at absolute multiples, as in the row kernel.  Within a chunk: scores
// are chains over the dimension; the weights are taken relative to the largest score of the chunk; their sum is 32
// ascending chains (keys l, l + 32, ...) and a tree over those; an output is the sum of one chain over each 64 keys, in
// ascending order; chunks are merged in ascending order by merge_partial.  All kernels below follow that order to
// the bit, so a position's result depends neither on the batch nor on how the tokens were cut into steps.
//
// Tokens are attended in one of two ways:
//  * F32Token: a CTA a (token, kv head): decoded tokens.  Bound by reading the keys and values once; all of a chunk's keys
//    and half its values are in flight at once.
//  * f32_tile: a CTA a kv head and 32 query rows (32 / group consecutive tokens with the group's heads), keys and values in
//    halves of a chunk through two buffers: runs of four tokens of a request and more within such a tile (prompt portions).
//    Bound by the float32 cores and shared memory (a thread owns 4 x 4 scores, then 4 x 4 outputs).
// Mode split has a launch for each, a CTA a chunk.  In mode rows, where a CTA walks all chunks, one launch has both: the first
// CTAs deal out the tokens outside of runs among themselves, the others have a tile each.  (Tiles that took single tokens
// in line, each at the cost of 32 rows, needed 358 us for 32 decoded tokens of 200 keys, and 1,547 for 24 of 1,000 keys
// beside a prompt of 300; these need 16 and 96.)
//
// Measured (16 query heads, 8 kv heads of 128, us a layer; one warp a (token, head) that reads every key's row by a lane of
// its own / these): three prompts of 301, 226 and 151 tokens 373 / 67, one of 600 837 / 119, one of 2,048 8,545 / 840, one
// of 9 8.5 / 4.5, one of 31 17.9 / 15.7; decoding, mode split: 4 requests of 701 tokens 126 / 13, 48 of 701 309 / 83; mode
// rows: 4 of 200 98 / 8.3, 32 of 200 100 / 16, 256 of 100 246 / 74, 24 of 1,000 beside a prompt of 300 1,090 / 96.  Prompts of
// a few tokens each are slower than with a warp a row: 64 of 3 tokens 11 / 31, 32 of 8 15 / 25.
#pragma once

#define F32_THREADS 256
#define F32_ROWS 32                        // query rows of a tile
#define F32_HALF 128                       // keys of a buffer
#define F32_SUB 64                         // keys of one chain of an output
#define F32_MIN_RUN 4                      // consecutive tokens of a request from which they are attended in a tile
#define F32_SCORE_ROW (ATTN_CHUNK + 4)
#define F32_SMS 148                        // one CTA of shared memory this large an SM

struct F32Args {
    const float* q;
    int64_t q_token_stride;
    const float* key_cache;
    const float* value_cache;
    const int* block_tables;
    int table_stride;
    const int* token_row;
    const int* positions;
    float* out;
    int64_t out_token_stride;
    float* scratch;                        // mode split: the partials
    int max_chunks, tokens, num_q, num_kv, page_size, window;
    float scale;
    int pdl;                               // the launch for single tokens in mode split
};

// Whether `token` is attended in a tile: its run of tokens of one request, within the tile of `tile_tokens` it
// falls into, is long enough.
__device__ __forceinline__ bool f32_in_long_run(const F32Args& a, int token, int tile_tokens) {
    const int from = token - token % tile_tokens, to = min(a.tokens, from + tile_tokens);
    const int request = a.token_row[token];
    int run = 1;
    for (int t = token - 1; run < F32_MIN_RUN && t >= from && a.token_row[t] == request; --t) ++run;
    for (int t = token + 1; run < F32_MIN_RUN && t < to && a.token_row[t] == request; ++t) ++run;
    return run >= F32_MIN_RUN;
}

__device__ __forceinline__ int64_t f32_slot(const F32Args& a, const int* table, int kv_head, int j) {
    return ((int64_t)table[j / a.page_size] * a.num_kv + kv_head) * a.page_size + j % a.page_size;
}

// Scores of one row's chunk (in place, from shared memory) -> weights; (max, sum) to every lane.  Keys outside
// [lo, position] weigh nothing, whatever their score slot holds.
__device__ __forceinline__ void f32_weights(float* scores, int begin, int lo, int position, int lane, float& max, float& sum) {
    float s[ATTN_CHUNK / 32];
    max = -INFINITY;
#pragma unroll
    for (int i = 0; i < ATTN_CHUNK / 32; ++i) {
        const int j = begin + lane + 32 * i;
        s[i] = scores[lane + 32 * i];
        if (j >= lo && j <= position) max = fmaxf(max, s[i]);
    }
    max = warp_max(max);
    sum = 0.0f;
#pragma unroll
    for (int i = 0; i < ATTN_CHUNK / 32; ++i) {
        const int j = begin + lane + 32 * i;
        const float p = j >= lo && j <= position ? expf(__fsub_rn(s[i], max)) : 0.0f;
        scores[lane + 32 * i] = p;
        sum = __fadd_rn(sum, p);
    }
    sum = warp_sum(sum);
}

// What a CTA keeps in static shared memory
struct F32Shared {
    int64_t slots[ATTN_CHUNK];
    int row_position[F32_ROWS];                                    // tiles: -1: not a row of this run
    float row_max[F32_ROWS], row_sum[F32_ROWS];
};

// One token, one kv head, one chunk: leaves (max, sum) of the group's heads in sh.row_max, sh.row_sum and the sums over 64
// keys each in `subs`, with a barrier behind.
template <int D, int GROUP> struct F32Token {
    static constexpr int PITCH = D + 4;                            // 16 bytes more, for the banks
    static constexpr int shared_floats = ATTN_CHUNK * PITCH + F32_HALF * D + GROUP * D + GROUP * F32_SCORE_ROW;
    static_assert(F32_HALF * D + ATTN_CHUNK / F32_SUB * GROUP * D <= ATTN_CHUNK * PITCH, "the sums take the keys' place");
    float* keys;                                                   // [ATTN_CHUNK][PITCH]; later the values from F32_HALF on
    float* values;                                                 // [F32_HALF][D]
    float* q;                                                      // [GROUP][D]
    float* scores;                                                 // [GROUP][F32_SCORE_ROW]
    float* subs;                                                   // [ATTN_CHUNK / F32_SUB][GROUP][D], behind the values in keys

    __device__ __forceinline__ explicit F32Token(float* shared) {
        keys = shared;
        values = keys + ATTN_CHUNK * PITCH;
        q = values + F32_HALF * D;
        scores = q + GROUP * D;
        subs = keys + F32_HALF * D;
    }

    __device__ __forceinline__ void load_q(const F32Args& a, int token, int kv_head) {
        const float* q_rows = a.q + (int64_t)token * a.q_token_stride + (int64_t)kv_head * GROUP * D;
        for (int i = threadIdx.x; i < GROUP * D; i += F32_THREADS) q[i] = q_rows[i];
    }

    __device__ __forceinline__ void chunk(const F32Args& a, F32Shared& sh, const int* table, int kv_head, int chunk, int lo,
                                          int position) {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const int begin = chunk * ATTN_CHUNK;
        const int first = max(lo, begin) - begin, count = min(position - begin + 1, ATTN_CHUNK);      // keys first..count-1
        if (tid >= first && tid < count) sh.slots[tid] = f32_slot(a, table, kv_head, begin + tid);
        __syncthreads();
        auto load = [&](float* dst, int pitch, const float* cache, int from, int to) {
            from = max(from, first);
            to = min(to, count);
            for (int i = from * (D / 4) + tid; i < to * (D / 4); i += F32_THREADS) {
                const int j = i / (D / 4), part = i % (D / 4) * 4;
                cp_async_16(dst + j * pitch + part, cache + sh.slots[j] * D + part, true);
            }
            cp_async_commit();
        };
        load(keys, PITCH, a.key_cache, 0, ATTN_CHUNK);
        load(values, D, a.value_cache, 0, F32_HALF);
        cp_async_wait<1>();
        __syncthreads();
        if (tid >= first && tid < count) {
            float dot[GROUP];
#pragma unroll
            for (int g = 0; g < GROUP; ++g) dot[g] = 0.0f;
            const float4* k4 = reinterpret_cast<const float4*>(keys + tid * PITCH);
#pragma unroll 8
            for (int i = 0; i < D / 4; ++i) {
                const float4 k = k4[i];
#pragma unroll
                for (int g = 0; g < GROUP; ++g) {
                    const float4 v = reinterpret_cast<const float4*>(q + g * D)[i];
                    dot[g] = __fmaf_rn(v.x, k.x, dot[g]);
                    dot[g] = __fmaf_rn(v.y, k.y, dot[g]);
                    dot[g] = __fmaf_rn(v.z, k.z, dot[g]);
                    dot[g] = __fmaf_rn(v.w, k.w, dot[g]);
                }
            }
#pragma unroll
            for (int g = 0; g < GROUP; ++g) scores[g * F32_SCORE_ROW + tid] = __fmul_rn(dot[g], a.scale);
        }
        __syncthreads();                                           // the keys are read: the other values take their place
        load(keys - F32_HALF * D, D, a.value_cache, F32_HALF, ATTN_CHUNK);
        if (warp < GROUP) {
            float max, sum;
            f32_weights(scores + warp * F32_SCORE_ROW, begin, lo, position, lane, max, sum);
            if (lane == 0) { sh.row_max[warp] = max; sh.row_sum[warp] = sum; }
        }
        cp_async_wait<0>();
        __syncthreads();
        const int dim = tid % D;
        for (int sub = tid / D; sub < ATTN_CHUNK / F32_SUB; sub += F32_THREADS / D) {
            float acc[GROUP];
#pragma unroll
            for (int g = 0; g < GROUP; ++g) acc[g] = 0.0f;
            const int from = max(sub * F32_SUB, first), to = min((sub + 1) * F32_SUB, count);
            const float* v = (sub * F32_SUB < F32_HALF ? values : keys - F32_HALF * D) + dim;
#pragma unroll 8
            for (int j = from; j < to; ++j) {
                const float value = v[j * D];
#pragma unroll
                for (int g = 0; g < GROUP; ++g) acc[g] = __fmaf_rn(scores[g * F32_SCORE_ROW + j], value, acc[g]);
            }
#pragma unroll
            for (int g = 0; g < GROUP; ++g) subs[(sub * GROUP + g) * D + dim] = acc[g];
        }
        __syncthreads();
    }

    // output i (of GROUP * D) of the chunk
    __device__ __forceinline__ float output(int i) const {
        float o = subs[i];
#pragma unroll
        for (int sub = 1; sub < ATTN_CHUNK / F32_SUB; ++sub) o = __fadd_rn(o, subs[sub * GROUP * D + i]);
        return o;
    }
};

template <int D, int GROUP>
__device__ __forceinline__ void f32_zero_token(const F32Args& a, int token, int kv_head) {
    for (int i = threadIdx.x; i < GROUP * D; i += F32_THREADS)
        a.out[(int64_t)token * a.out_token_stride + (int64_t)kv_head * GROUP * D + i] = 0.0f;
}

// Mode split: a CTA a (token, kv head, chunk), partials to scratch; tile_tokens > 0: but for the tokens of long runs.
template <int D, int GROUP>
__global__ void __launch_bounds__(F32_THREADS) attention_f32_token_kernel(F32Args a, int tile_tokens) {
    extern __shared__ __align__(16) float f32_shared[];
    __shared__ F32Shared sh;
    const int tid = threadIdx.x, token = blockIdx.x / a.num_kv, kv_head = blockIdx.x % a.num_kv, chunk = blockIdx.y;
    pdl_launch_dependents();
    pdl_wait();
    const int position = a.positions[token], request = a.token_row[token];
    if (request < 0 || position < 0) {                             // padding row of a captured batch
        if (chunk == 0) f32_zero_token<D, GROUP>(a, token, kv_head);
        return;
    }
    const int lo = a.window > 0 ? max(0, position - a.window + 1) : 0;
    if (!chunk_visible(chunk, lo, 0, position)) return;
    if (tile_tokens > 0 && f32_in_long_run(a, token, tile_tokens)) return;
    F32Token<D, GROUP> work(f32_shared);
    work.load_q(a, token, kv_head);
    work.chunk(a, sh, a.block_tables + (int64_t)request * a.table_stride, kv_head, chunk, lo, position);
    const int64_t row0 = (int64_t)token * a.num_q + kv_head * GROUP;
    for (int i = tid; i < GROUP * D; i += F32_THREADS) {
        float* dst = a.scratch + ((row0 + i / D) * a.max_chunks + chunk) * (int64_t)(D + 2);
        if (i % D == 0) { dst[0] = sh.row_max[i / D]; dst[1] = sh.row_sum[i / D]; }
        dst[2 + i % D] = work.output(i);
    }
}

// Mode rows, one token and kv head: its chunks one after the other, merged as they come.
template <int D, int GROUP>
__device__ __forceinline__ void f32_whole_token(const F32Args& a, float* shared, F32Shared& sh, int token, int kv_head) {
    const int position = a.positions[token], request = a.token_row[token];
    if (request < 0 || position < 0) {
        f32_zero_token<D, GROUP>(a, token, kv_head);
        return;
    }
    constexpr int EACH = (GROUP * D + F32_THREADS - 1) / F32_THREADS;      // outputs of a thread
    const int lo = a.window > 0 ? max(0, position - a.window + 1) : 0;
    F32Token<D, GROUP> work(shared);
    Partial<1> total[EACH];
#pragma unroll
    for (int e = 0; e < EACH; ++e) total[e] = Partial<1>{-INFINITY, 0.0f, {0.0f}};
    __syncthreads();                                               // the token before is finished with shared memory
    work.load_q(a, token, kv_head);
    for (int chunk = lo / ATTN_CHUNK; chunk <= position / ATTN_CHUNK; ++chunk) {
        work.chunk(a, sh, a.block_tables + (int64_t)request * a.table_stride, kv_head, chunk, lo, position);
#pragma unroll
        for (int e = 0; e < EACH; ++e) {
            const int i = threadIdx.x + e * F32_THREADS;
            if (i < GROUP * D) merge_partial(total[e], Partial<1>{sh.row_max[i / D], sh.row_sum[i / D], {work.output(i)}});
        }
        __syncthreads();                                           // the sums are read
    }
    float* to = a.out + (int64_t)token * a.out_token_stride + (int64_t)kv_head * GROUP * D;
#pragma unroll
    for (int e = 0; e < EACH; ++e) {
        const int i = threadIdx.x + e * F32_THREADS;
        if (i < GROUP * D) to[i] = __fdiv_rn(total[e].out[0], total[e].sum);
    }
}

// A tile's runs of F32_MIN_RUN tokens and more.  SPLIT false: all their chunks; SPLIT: chunk blockIdx.y, partials to scratch.
template <int D, int GROUP> struct F32Tile {
    static constexpr int PITCH = D + 4;
    static constexpr int TOKENS = F32_ROWS / GROUP;
    static constexpr int shared_floats = 2 * F32_HALF * PITCH + F32_ROWS * PITCH + F32_ROWS * F32_SCORE_ROW;
};

template <int D, int GROUP, bool SPLIT>
__device__ __forceinline__ void f32_tile(const F32Args& a, float* shared, F32Shared& sh, int block) {
    constexpr int PITCH = F32Tile<D, GROUP>::PITCH, TOKENS = F32Tile<D, GROUP>::TOKENS;
    constexpr int RT = D / 32;                                     // rows of a thread's outputs (times 4 dims)
    constexpr int DIM_GROUPS = D / 4, ROW_GROUPS = F32_THREADS / DIM_GROUPS;
    float* buffer[2] = {shared, shared + F32_HALF * PITCH};        // [F32_HALF][PITCH] each
    float* q = shared + 2 * F32_HALF * PITCH;                      // [F32_ROWS][PITCH]
    float* scores = q + F32_ROWS * PITCH;                          // [F32_ROWS][F32_SCORE_ROW]
    int64_t* slots = sh.slots;
    int* row_position = sh.row_position;
    float* row_max = sh.row_max;
    float* row_sum = sh.row_sum;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kv_head = block % a.num_kv, first_token = block / a.num_kv * TOKENS;
    const int tile_end = min(a.tokens, first_token + TOKENS);
    const int score_row = (warp & 1) * 4 + (lane & 3), score_key = (warp >> 1) * 8 + (lane >> 2);      // + 8 i, + 32 j
    const int out_row = tid / DIM_GROUPS, out_dim = tid % DIM_GROUPS * 4;                               // + ROW_GROUPS i

    int taken_to = first_token;                                    // the end of the last run that is taken here
    for (int run = first_token, run_end; run < tile_end; run = run_end) {
        const int request = a.token_row[run];
        int largest = a.positions[run], smallest = largest;
        for (run_end = run + 1; run_end < tile_end && a.token_row[run_end] == request; ++run_end) {
            largest = max(largest, a.positions[run_end]);
            smallest = min(smallest, a.positions[run_end]);
        }
        if (run_end > taken_to) {                                  // (equal: the rest of a run that was cut below)
            if (run_end - run < F32_MIN_RUN) continue;             // its tokens are attended one by one
            taken_to = run_end;
        }
        if (request < 0 || smallest < 0) {
            // padding: zeros (a run that mixes padding with tokens of a request is cut at every token)
            if (smallest < 0) run_end = run + 1;
            if (request < 0 || a.positions[run] < 0) {
                if (!SPLIT || blockIdx.y == 0)
                    for (int i = tid; i < (run_end - run) * GROUP * D; i += F32_THREADS)
                        a.out[(int64_t)(run + i / (GROUP * D)) * a.out_token_stride + (int64_t)kv_head * GROUP * D +
                              i % (GROUP * D)] = 0.0f;
                continue;
            }
            largest = smallest = a.positions[run];
        }
        // the keys every row of the run sees: [shared_from, smallest]; any: [lowest, largest]
        const int lowest = a.window > 0 ? max(0, smallest - a.window + 1) : 0;
        const int shared_from = a.window > 0 ? max(0, largest - a.window + 1) : 0;
        const int* table = a.block_tables + (int64_t)request * a.table_stride;
        const int chunk_from = SPLIT ? (int)blockIdx.y : lowest / ATTN_CHUNK;
        const int chunk_to = SPLIT ? (int)blockIdx.y : largest / ATTN_CHUNK;
        if (SPLIT && !chunk_visible(chunk_from, lowest, 0, largest)) continue;

        __syncthreads();                                           // the run before is finished with shared memory
        if (tid < F32_ROWS) {
            const int token = first_token + tid / GROUP;
            row_position[tid] = token >= run && token < run_end ? a.positions[token] : -1;
        }
        for (int i = tid; i < F32_ROWS * D; i += F32_THREADS) {
            const int row = i / D, token = first_token + row / GROUP;
            q[row * PITCH + i % D] = token >= run && token < run_end
                ? a.q[(int64_t)token * a.q_token_stride + (int64_t)(kv_head * GROUP + row % GROUP) * D + i % D] : 0.0f;
        }
        float total_max[RT], total_sum[RT], total[RT][4];
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            total_max[i] = -INFINITY;
            total_sum[i] = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; ++e) total[i][e] = 0.0f;
        }
        for (int chunk = chunk_from; chunk <= chunk_to; ++chunk) {
            const int begin = chunk * ATTN_CHUNK;
            const int first = max(lowest - begin, 0), count = min(largest - begin + 1, ATTN_CHUNK);        // keys first..count-1
            if (tid >= first && tid < count) slots[tid] = f32_slot(a, table, kv_head, begin + tid);
            __syncthreads();                                       // ... and the buffers of the chunk before are read
            auto load = [&](int half, int pitch, const float* cache) {
                const int from = max(half * F32_HALF, first), to = min((half + 1) * F32_HALF, count);
                for (int i = from * (D / 4) + tid; i < to * (D / 4); i += F32_THREADS) {
                    const int j = i / (D / 4), part = i % (D / 4) * 4;
                    cp_async_16(buffer[half] + (j - half * F32_HALF) * pitch + part, cache + slots[j] * D + part, true);
                }
                cp_async_commit();
            };
            load(0, PITCH, a.key_cache);
            load(1, PITCH, a.key_cache);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                cp_async_wait<1>();
                __syncthreads();
                if (half * F32_HALF < count && (half + 1) * F32_HALF > first) {
                    float dot[4][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) dot[i][j] = 0.0f;
                    const float* qp = q + score_row * PITCH;
                    const float* kp = buffer[half] + score_key * PITCH;
#pragma unroll 2
                    for (int d = 0; d < D; d += 4) {
                        float4 qv[4], kv[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(qp + i * 8 * PITCH + d);
#pragma unroll
                        for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(kp + j * 32 * PITCH + d);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                dot[i][j] = __fmaf_rn(qv[i].x, kv[j].x, dot[i][j]);
                                dot[i][j] = __fmaf_rn(qv[i].y, kv[j].y, dot[i][j]);
                                dot[i][j] = __fmaf_rn(qv[i].z, kv[j].z, dot[i][j]);
                                dot[i][j] = __fmaf_rn(qv[i].w, kv[j].w, dot[i][j]);
                            }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j)                // keys that were not loaded are masked by position
                            scores[(score_row + 8 * i) * F32_SCORE_ROW + half * F32_HALF + score_key + 32 * j] =
                                __fmul_rn(dot[i][j], a.scale);
                }
                __syncthreads();
                load(half, D, a.value_cache);
            }
            for (int row = warp; row < F32_ROWS; row += F32_THREADS / 32) {
                const int position = row_position[row];
                float max, sum;
                f32_weights(scores + row * F32_SCORE_ROW, begin, a.window > 0 ? position - a.window + 1 : 0, position, lane,
                            max, sum);
                if (lane == 0) { row_max[row] = max; row_sum[row] = sum; }
            }
            float part[RT][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (half == 0) cp_async_wait<1>(); else cp_async_wait<0>();
                __syncthreads();
#pragma unroll
                for (int sub = 0; sub < F32_HALF / F32_SUB; ++sub) {
                    const int sub_at = half * F32_HALF + sub * F32_SUB;
                    float acc[RT][4];
#pragma unroll
                    for (int i = 0; i < RT; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[i][e] = 0.0f;
                    const int from = max(sub_at, first), to = min(sub_at + F32_SUB, count);
                    for (int at = from & ~3; at < to; at += 4) {
                        float4 p[RT];
#pragma unroll
                        for (int i = 0; i < RT; ++i)
                            p[i] = *reinterpret_cast<const float4*>(scores + (out_row + i * ROW_GROUPS) * F32_SCORE_ROW + at);
                        const float* v = buffer[half] + (at - half * F32_HALF) * D + out_dim;
                        if (at >= from && at + 4 <= to && begin + at >= shared_from && begin + at + 3 <= smallest) {
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const float4 value = *reinterpret_cast<const float4*>(v + u * D);
#pragma unroll
                                for (int i = 0; i < RT; ++i) {
                                    const float w = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                                    acc[i][0] = __fmaf_rn(w, value.x, acc[i][0]);
                                    acc[i][1] = __fmaf_rn(w, value.y, acc[i][1]);
                                    acc[i][2] = __fmaf_rn(w, value.z, acc[i][2]);
                                    acc[i][3] = __fmaf_rn(w, value.w, acc[i][3]);
                                }
                            }
                        } else {                                   // a key that a row does not see must not touch it, whatever it holds
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int j = at + u;
                                if (j < from || j >= to) continue;
                                const float4 value = *reinterpret_cast<const float4*>(v + u * D);
#pragma unroll
                                for (int i = 0; i < RT; ++i) {
                                    const int position = row_position[out_row + i * ROW_GROUPS];
                                    if (begin + j > position || (a.window > 0 && begin + j <= position - a.window)) continue;
                                    const float w = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                                    acc[i][0] = __fmaf_rn(w, value.x, acc[i][0]);
                                    acc[i][1] = __fmaf_rn(w, value.y, acc[i][1]);
                                    acc[i][2] = __fmaf_rn(w, value.z, acc[i][2]);
                                    acc[i][3] = __fmaf_rn(w, value.w, acc[i][3]);
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < RT; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            part[i][e] = half == 0 && sub == 0 ? acc[i][e] : __fadd_rn(part[i][e], acc[i][e]);
                }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int row = out_row + i * ROW_GROUPS, token = first_token + row / GROUP;
                if (SPLIT) {
                    if (token < run || token >= run_end) continue;
                    const int lo = a.window > 0 ? max(0, row_position[row] - a.window + 1) : 0;
                    if (!chunk_visible(chunk, lo, 0, row_position[row])) continue;
                    float* dst = a.scratch + (((int64_t)token * a.num_q + kv_head * GROUP + row % GROUP) * a.max_chunks + chunk) *
                                                 (int64_t)(D + 2);
                    if (out_dim == 0) { dst[0] = row_max[row]; dst[1] = row_sum[row]; }
#pragma unroll
                    for (int e = 0; e < 4; ++e) dst[2 + out_dim + e] = part[i][e];
                } else {
                    Partial<4> so_far{total_max[i], total_sum[i], {total[i][0], total[i][1], total[i][2], total[i][3]}};
                    const Partial<4> more{row_max[row], row_sum[row], {part[i][0], part[i][1], part[i][2], part[i][3]}};
                    merge_partial(so_far, more);
                    total_max[i] = so_far.max;
                    total_sum[i] = so_far.sum;
#pragma unroll
                    for (int e = 0; e < 4; ++e) total[i][e] = so_far.out[e];
                }
            }
        }
        if (!SPLIT) {
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int row = out_row + i * ROW_GROUPS, token = first_token + row / GROUP;
                if (token < run || token >= run_end) continue;
                float* to = a.out + (int64_t)token * a.out_token_stride + (int64_t)(kv_head * GROUP + row % GROUP) * D + out_dim;
#pragma unroll
                for (int e = 0; e < 4; ++e) to[e] = __fdiv_rn(total[i][e], total_sum[i]);
            }
        }
    }
}

template <int D, int GROUP>
__global__ void __launch_bounds__(F32_THREADS, D == 64 ? 2 : 1) attention_f32_tile_kernel(F32Args a) {
    extern __shared__ __align__(16) float f32_shared[];
    __shared__ F32Shared sh;
    f32_tile<D, GROUP, true>(a, f32_shared, sh, blockIdx.x);
}

// Mode rows.  The first `token_ctas` CTAs deal out the tokens outside of long runs (tile_tokens == 0: all tokens) by kv
// head, the others have a tile each.  A thread looks at one (token, kv head) of its CTA's share at a time.
template <int D, int GROUP>
__global__ void __launch_bounds__(F32_THREADS, D == 64 ? 2 : 1) attention_f32_rows_kernel(F32Args a, int token_ctas, int tile_tokens) {
    extern __shared__ __align__(16) float f32_shared[];
    __shared__ F32Shared sh;
    __shared__ uint32_t taken[F32_THREADS / 32];
    if ((int)blockIdx.x >= token_ctas) {
        f32_tile<D, GROUP, false>(a, f32_shared, sh, blockIdx.x - token_ctas);
        return;
    }
    const int items = a.tokens * a.num_kv;
    for (int64_t base = blockIdx.x; base < items; base += (int64_t)token_ctas * F32_THREADS) {
        const int64_t at = base + (int64_t)token_ctas * threadIdx.x;
        const bool mine = at < items && (tile_tokens == 0 || !f32_in_long_run(a, (int)at / a.num_kv, tile_tokens));
        const uint32_t bits = __ballot_sync(0xffffffffu, mine);
        __syncthreads();                                           // the share before is read
        if (threadIdx.x % 32 == 0) taken[threadIdx.x / 32] = bits;
        __syncthreads();
        for (int w = 0; w < F32_THREADS / 32; ++w)
            for (uint32_t left = taken[w]; left; left &= left - 1) {
                const int item = (int)(base + (int64_t)token_ctas * (w * 32 + __ffs(left) - 1));
                f32_whole_token<D, GROUP>(a, f32_shared, sh, item / a.num_kv, item % a.num_kv);
            }
    }
}

template <int D, int GROUP>
static int launch_f32(const F32Args& a, cudaStream_t s) {
    constexpr int TOKENS = F32Tile<D, GROUP>::TOKENS;
    constexpr int tile_shared = 4 * F32Tile<D, GROUP>::shared_floats, token_shared = 4 * F32Token<D, GROUP>::shared_floats;
    constexpr int rows_shared = tile_shared > token_shared ? tile_shared : token_shared;
    const long long tiles = (long long)((a.tokens + TOKENS - 1) / TOKENS) * a.num_kv;
    if (tiles > 2147483647LL - F32_SMS || (long long)a.tokens * a.num_kv > 2147483647LL) return TVB_BAD_ARGUMENT;
    cudaError_t e;
    // Up to TOKENS tokens each gets a CTA (a chunk) of its own; with more, runs of one request share their keys' reads.
    if (a.max_chunks == 0) {
        // ... from as many on as would go to an SM three at a time: two single tokens take an SM about as long as a tile
        const int items = a.tokens * a.num_kv;
        const bool tiled = a.tokens > TOKENS && items > 2 * F32_SMS;
        auto kernel = attention_f32_rows_kernel<D, GROUP>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_shared);
        if (e != cudaSuccess) return (int)e;
        const int token_ctas = tiled ? F32_SMS : items;
        kernel<<<(unsigned)(token_ctas + (tiled ? tiles : 0)), F32_THREADS, tiled ? rows_shared : token_shared, s>>>(
            a, token_ctas, tiled ? TOKENS : 0);
        return tvb_last_error();
    }
    const bool tiled = a.tokens > TOKENS;
    auto kernel = attention_f32_token_kernel<D, GROUP>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, token_shared);
    if (e != cudaSuccess) return (int)e;
    TvbLaunch launch(dim3((unsigned)(a.tokens * a.num_kv), a.max_chunks), dim3(F32_THREADS), token_shared, s, a.pdl);
    e = cudaLaunchKernelEx(&launch.config, kernel, a, tiled ? TOKENS : 0);
    if (e != cudaSuccess) return (int)e;
    if (tiled) {
        auto tile_kernel = attention_f32_tile_kernel<D, GROUP>;
        e = cudaFuncSetAttribute(tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_shared);
        if (e != cudaSuccess) return (int)e;
        tile_kernel<<<dim3((unsigned)tiles, a.max_chunks), F32_THREADS, tile_shared, s>>>(a);
    }
    return tvb_last_error();
}

static int launch_f32_of(int head_dim, int group, const F32Args& a, cudaStream_t s) {
#define F32_OF(D)                                                                                       \
    (group == 1 ? launch_f32<D, 1>(a, s) : group == 2 ? launch_f32<D, 2>(a, s) : group == 4 ? launch_f32<D, 4>(a, s) \
                                                                                : launch_f32<D, 8>(a, s))
    return head_dim == 64 ? F32_OF(64) : F32_OF(128);
#undef F32_OF
}
