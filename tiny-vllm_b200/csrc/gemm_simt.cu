// C[M,N] = A[M,K] . W[N,K]^T on the float32 cores: the matrix product of the true
// 32-bit path (no tensor cores, no reduced-precision mode), for any M, N, K.
//
// float32 operands.  The sum of an output element has one order, whatever M is and whichever of the
// two kernels below (float32 cores) runs: K is cut into segments of 128; a segment is a chain over its even k and one over
// its odd k (one fused multiply-add per k, ascending; the packed instruction on pairs of floats does both),
// then their sum; four segments are added in ascending order to a group, the groups in ascending
// order to the result.  A row's result does not depend on which other rows are in the batch, and
// the shorter chains are closer to the 64-bit sums than one chain over K.  Stands where the
// reference calls F.linear (tinyvllm/layers.py:84-85).
//
//  * gemm_f32_few_kernel: up to 8 rows (decode).  Bound by reading W once: x stays in shared memory, W comes
//    through a ring of cp.async stages of 8 or 16 columns x 1,024 k, a thread owns one (column, segment).
//  * gemm_f32_tile_kernel: more rows (beyond 32 narrow products and rows off the 16-byte boundary; the others have
//    gemm_f32_tc.cu, in another order).  Bound by the float32 cores: tiles of up to 64 x 64, a thread
//    owns up to 8 x 4 outputs, three to four stages of 32 k in flight, groups of 512 k spread over the grid
//    where the tiles alone leave SMs idle (their sums meet in a second kernel, in the fixed order).
//
// Measured (us, one 64 x 64 tile kernel with scalar loads and one chain a sum / these): 4 rows 4,096 x 1,024 76 / 7.8,
// 1,024 x 3,072 229 / 9.5, 151,936 x 1,024 709 / 150 (one row: 703 / 118, 5.3 TB/s); 64 rows 6,144 x 1,024 80 / 58;
// 677 rows 4,096 x 1,024 251 / 176, 1,024 x 2,048 215 / 93, 6,144 x 1,024 390 / 260 (33 TFLOP/s; 2,048 rows 37.5: three
// 64-bit operands keep the packed instruction at about 44 on this part, scalar ones on the same layout were slower).
// In a decode step of 4 rows (28 layers of the 0.6B sizes) the products of up to 8 rows are launched programmatically and ask
// for their first stages (64 KB a CTA of 16 columns) while the kernel before runs: with the small kernels between them
// launched the same way, and the norm below, 1,780 to 1,500 us a step.
// Error against 64-bit sums (2-norm): 5.7e-7 at k = 1,024 and 9.9e-7 at k = 3,072 before, 1.6e-7 at both.
//
// bfloat16 operands (sizes the tensor-core products do not take): one plain tile kernel, one ascending chain.
#include "common.cuh"

#include <algorithm>

// ------------------------------------------------------------------------------------------ bfloat16 operands
#define TILE_M 64
#define TILE_N 64
#define TILE_K 16

template <typename TI, typename TO>
__global__ void __launch_bounds__(256)
gemm_nt_simt_kernel(const TI* __restrict__ a, int64_t lda, const TI* __restrict__ w, int64_t ldw,
                    TO* __restrict__ c, int64_t ldc, int m, int n, int k) {
    __shared__ float a_tile[TILE_K][TILE_M + 4];
    __shared__ float w_tile[TILE_K][TILE_N + 4];
    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * TILE_M, col0 = blockIdx.x * TILE_N;
    const int ty = tid / 16, tx = tid % 16;           // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    const int load_row = tid / 4;                      // 64 rows, 4 threads per row
    const int load_k = (tid % 4) * 4;                  // 4 consecutive k per thread
    for (int k0 = 0; k0 < k; k0 += TILE_K) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int kk = k0 + load_k + i;
            const int ar = row0 + load_row, wr = col0 + load_row;
            a_tile[load_k + i][load_row] = (ar < m && kk < k) ? to_float<TI>(a[(int64_t)ar * lda + kk]) : 0.0f;
            w_tile[load_k + i][load_row] = (wr < n && kk < k) ? to_float<TI>(w[(int64_t)wr * ldw + kk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TILE_K; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = a_tile[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = w_tile[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __fmaf_rn(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= m) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = col0 + tx * 4 + j;
            if (col < n) c[(int64_t)r * ldc + col] = from_float<TO>(acc[i][j]);
        }
    }
}

// ------------------------------------------------------------------------------------------ float32 operands
#define SEGMENT 128                     // k of one pair of chains
#define GROUP_SEGMENTS 4
#define GROUP (SEGMENT * GROUP_SEGMENTS)

typedef unsigned long long f32x2;       // two float32 in a 64-bit register pair
__device__ __forceinline__ void fma_pair(f32x2& acc, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum_pair(f32x2 v) {
    return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}

// Four floats row[k0..k0+3] of a row of k floats to shared memory, zero beyond k (or all zero): one 16-byte copy
// (ALIGNED: the row starts on a 16-byte boundary and k is a multiple of four), else four 4-byte ones.
template <bool ALIGNED>
__device__ __forceinline__ void copy_four(float* dst, const float* row, int k0, int k, bool valid) {
    if constexpr (ALIGNED) {
        const bool in = valid && k0 < k;
        cp_async_16(dst, in ? row + k0 : row, in);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool in = valid && k0 + e < k;
            const int bytes = in ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_address(dst + e)),
                         "l"(in ? row + k0 + e : row), "r"(bytes));
        }
    }
}

// ---- up to 8 rows
#define FEW_K 1024                                   // k of a stage: 8 segments
#define FEW_SEGMENTS (FEW_K / SEGMENT)
#define FEW_ROW (FEW_K + 4)                          // floats from one column of a stage to the next: 16 bytes more,
                                                     // so that the 8 columns of a quarter warp differ in banks
#define X_SEGMENT (SEGMENT + 4)                      // the same for the segments of x

template <int ROWS, int COLS, int STAGES, bool ALIGNED>
__global__ void __launch_bounds__(COLS * FEW_SEGMENTS)
gemm_f32_few_kernel(const float* a, int64_t lda, const float* w, int64_t ldw, float* c, int64_t ldc, int m, int n, int k,
                    int w_constant) {
    constexpr int THREADS = COLS * FEW_SEGMENTS;
    static_assert(ROWS * COLS <= THREADS, "one thread folds one output");
    extern __shared__ __align__(16) float few_shared[];
    const int segments = (k + SEGMENT - 1) / SEGMENT;
    const int x_row = segments * X_SEGMENT;
    float* ring = few_shared;                                    // [STAGES][COLS][FEW_ROW]
    float* parts = ring + STAGES * COLS * FEW_ROW;               // [FEW_SEGMENTS][ROWS][COLS]
    float* x = parts + FEW_SEGMENTS * ROWS * COLS;               // [ROWS][segments][X_SEGMENT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = (lane & 7) + (COLS > 8 ? (warp & 1) * 8 : 0);
    const int part = (lane >> 3) + (COLS > 8 ? warp >> 1 : warp) * 4;
    const int chunks = (k + FEW_K - 1) / FEW_K, tiles = (n + COLS - 1) / COLS;
    const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;      // tiles of this CTA
    const int items = mine * chunks;

    int load_tile = blockIdx.x, load_chunk = 0, load_stage = 0;      // the item that is loaded next
    auto load = [&]() {
        const int k0 = load_chunk * FEW_K, first = load_tile * COLS;
        float* to = ring + load_stage * COLS * FEW_ROW + tid * 4;
        const float* from = w + (int64_t)first * ldw;
        // only the segments that exist are read later
        const int quads = min(FEW_K, segments * SEGMENT - k0) / 4;
#pragma unroll
        for (int column = 0; column < COLS; ++column) {
#pragma unroll
            for (int q = 0; q < FEW_K / 4; q += THREADS)
                if (q + tid < quads) copy_four<ALIGNED>(to + q * 4, from, k0 + (q + tid) * 4, k, first + column < n);
            to += FEW_ROW;
            if (first + column + 1 < n) from += ldw;
        }
        load_stage = load_stage + 1 == STAGES ? 0 : load_stage + 1;
        if (++load_chunk == chunks) { load_chunk = 0; load_tile += gridDim.x; }
    };
    // Under programmatic dependent launch this kernel may run beside the one before it, and lets the next one do the same.
    // A weight that no kernel in flight writes is asked for at once, before the wait for the rows of x.
    pdl_launch_dependents();
    if (!w_constant) pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < items) load();
    if (w_constant) pdl_wait();
#pragma unroll
    for (int row = 0; row < ROWS; ++row) {
        const float* from = a + (int64_t)min(row, m - 1) * lda;
        for (int q = tid; q < segments * (SEGMENT / 4); q += THREADS)
            copy_four<ALIGNED>(x + row * x_row + (q / (SEGMENT / 4)) * X_SEGMENT + (q % (SEGMENT / 4)) * 4, from, q * 4, k, row < m);
    }
    // x and the first stages are one group, the oldest; the others of the ring's start are empty
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) cp_async_commit();
    float total = 0.0f;
    int tile = blockIdx.x, chunk = 0, at_stage = 0;
    for (int item = 0; item < items; ++item) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                          // the stage is whole; the one before is read
        if (item + STAGES - 1 < items) load();
        cp_async_commit();
        const int segment = chunk * FEW_SEGMENTS + part;
        if (segment < segments) {
            const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(
                ring + (at_stage * COLS + col) * FEW_ROW + part * SEGMENT);
            const float* xp = x + segment * X_SEGMENT;
            f32x2 acc[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = 0;
#pragma unroll 8
            for (int q = 0; q < SEGMENT / 4; ++q) {
                const ulonglong2 wv = wp[q];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const ulonglong2 xv = reinterpret_cast<const ulonglong2*>(xp + r * x_row)[q];
                    fma_pair(acc[r], xv.x, wv.x);
                    fma_pair(acc[r], xv.y, wv.y);
                }
            }
#pragma unroll
            for (int r = 0; r < ROWS; ++r) parts[(part * ROWS + r) * COLS + col] = sum_pair(acc[r]);
        }
        __syncthreads();
        if (tid < ROWS * COLS) {
            const int have = min(FEW_SEGMENTS, segments - chunk * FEW_SEGMENTS);
            if (chunk == 0) total = 0.0f;
#pragma unroll
            for (int g = 0; g < FEW_SEGMENTS / GROUP_SEGMENTS; ++g) {
                if (g * GROUP_SEGMENTS >= have) break;
                float sum = parts[g * GROUP_SEGMENTS * ROWS * COLS + tid];
#pragma unroll
                for (int s = 1; s < GROUP_SEGMENTS; ++s)
                    if (g * GROUP_SEGMENTS + s < have)
                        sum = __fadd_rn(sum, parts[(g * GROUP_SEGMENTS + s) * ROWS * COLS + tid]);
                total = chunk == 0 && g == 0 ? sum : __fadd_rn(total, sum);
            }
            if (chunk == chunks - 1) {
                const int row = tid / COLS, at = tile * COLS + tid % COLS;
                if (row < m && at < n) c[(int64_t)row * ldc + at] = total;
            }
        }
        at_stage = at_stage + 1 == STAGES ? 0 : at_stage + 1;
        if (++chunk == chunks) { chunk = 0; tile += gridDim.x; }
    }
    cp_async_wait<0>();
}

// ---- more rows
#define BN 64                                        // columns of a tile
#define TN 4                                         // ... and of a thread
#define STEP 32                                      // k of a stage
#define TILE_ROW (STEP + 4)                          // floats from row to row: 16 bytes more, for the banks
#define TILE_STAGES 4

// Groups [z * groups_per, ...) of the sum of one BM x BN tile, TM x TN outputs a thread.  partial == nullptr: the CTA has
// every group and adds them up in c; else group g goes to partial[g][m][n].
template <int BM, int TM, bool ALIGNED>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 3)
gemm_f32_tile_kernel(const float* __restrict__ a, int64_t lda, const float* __restrict__ w, int64_t ldw,
                     float* c, int64_t ldc, float* partial, int groups_per, int m, int n, int k) {
    constexpr int RY = BM / TM, RX = BN / TN, THREADS = RY * RX;
    static_assert(RY % 4 == 0 && RX % 8 == 0, "a warp is 4 x 8 threads");
    extern __shared__ __align__(16) float tile_shared[];          // [TILE_STAGES][BM + BN][TILE_ROW]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Neighbouring lanes share a row of a or of w: a 16-byte read of shared memory then takes two wavefronts
    // instead of four (measured: lanes of a quarter warp on 8 different rows took four, whoever shared them).
    const int ty = (warp % (RY / 4)) * 4 + ((lane & 1) | (lane >> 1 & 2));
    const int tx = (warp / (RY / 4)) * 8 + ((lane >> 1 & 1) | (lane >> 2 & 6));
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int k_from = blockIdx.z * groups_per * GROUP, k_to = min(k, k_from + groups_per * GROUP);
    const int steps = (k_to - k_from + STEP - 1) / STEP;

    auto load = [&](int step) {
        float* stage = tile_shared + (step % TILE_STAGES) * (BM + BN) * TILE_ROW;
        const int k0 = k_from + step * STEP;
#pragma unroll
        for (int i = tid; i < (BM + BN) * (STEP / 4); i += THREADS) {
            const int row = i / (STEP / 4), q = i % (STEP / 4);
            const bool of_a = row < BM;
            const int at = of_a ? row0 + row : col0 + row - BM, last = (of_a ? m : n) - 1;
            const float* from = of_a ? a + (int64_t)min(at, last) * lda : w + (int64_t)min(at, last) * ldw;
            copy_four<ALIGNED>(stage + row * TILE_ROW + q * 4, from, k0 + q * 4, k, at <= last);
        }
    };
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < steps) load(s);
        cp_async_commit();
    }
    f32x2 acc[TM][TN];
    float group[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0;
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<TILE_STAGES - 2>();
        __syncthreads();
        if (step + TILE_STAGES - 1 < steps) load(step + TILE_STAGES - 1);
        cp_async_commit();
        const float* stage = tile_shared + (step % TILE_STAGES) * (BM + BN) * TILE_ROW;
        const float* ap = stage + ty * TILE_ROW;
        const float* wp = stage + (BM + tx) * TILE_ROW;
#pragma unroll 2
        for (int q = 0; q < STEP / 4; ++q) {
            ulonglong2 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(ap + i * RY * TILE_ROW + q * 4);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(wp + j * RX * TILE_ROW + q * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma_pair(acc[i][j], av[i].x, wv.x);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma_pair(acc[i][j], av[i].y, wv.y);
            }
        }
        const bool last = step + 1 == steps;
        if ((step + 1) % (SEGMENT / STEP) != 0 && !last) continue;
        const int segment = step / (SEGMENT / STEP);              // of this CTA's range
        const bool opens = segment % GROUP_SEGMENTS == 0, closes = (segment + 1) % GROUP_SEGMENTS == 0 || last;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float sum = sum_pair(acc[i][j]);
                group[i][j] = opens ? sum : __fadd_rn(group[i][j], sum);
                acc[i][j] = 0;
            }
        if (!closes) continue;
        const int g = segment / GROUP_SEGMENTS;
        float* to = partial ? partial + (int64_t)(blockIdx.z * groups_per + g) * m * n : c;
        const int64_t ld = partial ? n : ldc;
        const bool add = !partial && g > 0;                       // to this thread's own sum so far
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int row = row0 + ty + i * RY;
            if (row >= m) continue;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int col = col0 + tx + j * RX;
                if (col >= n) continue;
                float* at = to + row * ld + col;
                *at = add ? __fadd_rn(*at, group[i][j]) : group[i][j];
            }
        }
    }
    cp_async_wait<0>();
}

// c = the sum of the groups' partial products, in ascending order
__global__ void __launch_bounds__(256)
gemm_f32_fold_kernel(const float* __restrict__ partial, int groups, float* __restrict__ c, int64_t ldc, int m, int n) {
    const int64_t size = (int64_t)m * n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x) {
        float total = partial[i];
        for (int g = 1; g < groups; ++g) total = __fadd_rn(total, partial[g * size + i]);
        c[(i / n) * ldc + i % n] = total;
    }
}

// ---------------------------------------------------------------------------------------------- launches
#define SMS 148
#define FEW_ROWS 8
#define SHARED_LIMIT (227 * 1024)

// 16 columns a CTA (twice the warps for one copy of x) as soon as that gives every SM one
static int few_columns(int n) { return n >= 16 * SMS ? 16 : 8; }

static long long few_shared_bytes(int rows, int columns, int stages, int k) {
    const int segments = (k + SEGMENT - 1) / SEGMENT;
    return 4LL * (stages * columns * FEW_ROW + FEW_SEGMENTS * rows * columns + (long long)rows * segments * X_SEGMENT);
}

static int few_template_rows(int m) { return m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : 8; }

static bool takes_few(int m, int n, int k) {
    return m <= FEW_ROWS && few_shared_bytes(few_template_rows(m), few_columns(n), 2, k) <= SHARED_LIMIT;
}

// How a product runs in tiles: rows of a tile, groups a CTA, CTAs a tile, groups in all, columns of c a launch.
// us: about what it takes.
struct TilePlan { int bm, groups_per, splits, groups, cols; double us; };

#define SCRATCH_FLOATS (16LL << 20)                  // the most that partial sums take

// Time (us) of one group of k in `ctas` tiles spread over the SMs: the busiest SM runs three CTAs side by side, then what
// is left.  Measured for one, two and three CTAs an SM (4,096 x 12,288 and 1,024 x 2,048 at 12 to 2,048 rows).
// `even`: many short CTAs, whose rounds run into one another: the mean of that and of an even spread.
static double group_us(long long ctas, int bm, bool even) {
    static const double together[3][3] = {{11.5, 14.5, 19.0}, {13.0, 20.0, 28.0}, {28.0, 40.0, 50.0}};
    const double* us = together[bm == 16 ? 0 : bm == 32 ? 1 : 2];
    const long long most = (ctas + SMS - 1) / SMS;
    const double rounds = (double)(most / 3) * us[2] + (most % 3 ? us[most % 3 - 1] : 0.0);
    return most <= 3 || !even ? rounds : 0.5 * (rounds + (double)ctas / (3 * SMS) * us[2]);
}

// k is cut over the grid where that is quicker by these times, with 3 us a launch more for adding up the partial sums and
// what writing and reading them takes (6 TB/s).  They take up to 64 MiB: a product whose sums would take more runs a
// range of columns at a time.  The order of a sum is the same in all plans.
// Measured (us, whole / cut): 64 x 6,144 x 1,024 58 / 43, 300 x 1,024 x 2,048 111 / 59, 677 x 6,144 x 1,024 269 / 260,
// 300 x 4,096 x 12,288 1,299 / 902 in two ranges; not cut: 2,048 x 6,144 x 1,024 690 / 739, 1,024 x 4,096 x 1,024 243 / 246.
static TilePlan tile_plan(int m, int n, int k) {
    TilePlan plan;
    plan.bm = m <= 16 ? 16 : m <= 32 ? 32 : 64;
    plan.groups = plan.groups_per = (k + GROUP - 1) / GROUP;
    plan.cols = n;
    const long long tile_rows = (m + plan.bm - 1) / plan.bm;
    const double whole = plan.groups * group_us((n + BN - 1) / BN * tile_rows, plan.bm, false);
    plan.us = plan.groups > 1 ? whole : 2.0 + (whole - 2.0) * ((k + STEP - 1) / STEP * STEP) / GROUP;
    const long long fit = SCRATCH_FLOATS / ((long long)plan.groups * m) / BN * BN;      // columns that the scratch holds
    if (fit > 0) {
        const long long ranges = (n + fit - 1) / fit;
        const int cols = (int)(((n + ranges - 1) / ranges + BN - 1) / BN) * BN;
        double best = 0.985 * whole;
        for (int per = plan.groups - 1; per >= 1; --per) {
            const int splits = (plan.groups + per - 1) / per;
            if (splits > 65535) break;
            const double cost = (double)((n + cols - 1) / cols) * (per * group_us(cols / BN * tile_rows * splits, plan.bm, true) + 3.0) +
                                8.0 * plan.groups * m * n / 6e6;
            if (cost < best) { plan.us = best = cost; plan.groups_per = per; plan.cols = std::min(n, cols); }
        }
    }
    plan.splits = (plan.groups + plan.groups_per - 1) / plan.groups_per;
    return plan;
}

template <int ROWS, int COLS, int STAGES, bool ALIGNED>
static int launch_few(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, int m, int n,
                      int k, int pdl, int w_constant, cudaStream_t s) {
    auto kernel = gemm_f32_few_kernel<ROWS, COLS, STAGES, ALIGNED>;
    const int shared = (int)few_shared_bytes(ROWS, COLS, STAGES, k);
    // (one limit for all k: a smaller one could come between another thread's limit and its launch)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SHARED_LIMIT);
    if (e != cudaSuccess) return (int)e;
    const int resident = std::max(1, SHARED_LIMIT / (shared + 1024));
    const int tiles = (n + COLS - 1) / COLS;
    // as many CTAs as run at once, each with the same number of tiles but for one
    const int turns = (tiles + SMS * resident - 1) / (SMS * resident);
    TvbLaunch launch(dim3((tiles + turns - 1) / turns), dim3(COLS * FEW_SEGMENTS), shared, s, pdl);
    e = cudaLaunchKernelEx(&launch.config, kernel, a, (int64_t)lda, w, (int64_t)ldw, c, (int64_t)ldc, m, n, k, w_constant);
    return e == cudaSuccess ? tvb_last_error() : (int)e;
}

template <int ROWS, bool ALIGNED>
static int few_of(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, int m, int n, int k,
                  int pdl, int w_constant, cudaStream_t s) {
    if (few_columns(n) == 16) return launch_few<ROWS, 16, 2, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
    if (few_shared_bytes(ROWS, 8, 3, k) <= SHARED_LIMIT) return launch_few<ROWS, 8, 3, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
    return launch_few<ROWS, 8, 2, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
}

template <int BM, int TM, bool ALIGNED>
static int launch_tiles(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, float* partial,
                        const TilePlan& plan, int m, int n, int k, cudaStream_t s) {
    auto kernel = gemm_f32_tile_kernel<BM, TM, ALIGNED>;
    constexpr int shared = TILE_STAGES * (BM + BN) * TILE_ROW * 4;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shared);
    if (e != cudaSuccess) return (int)e;
    for (int at = 0; at < n; at += plan.cols) {
        const int cols = std::min(plan.cols, n - at);
        const dim3 grid((cols + BN - 1) / BN, (m + BM - 1) / BM, plan.splits);
        if (grid.y > 65535) return TVB_BAD_ARGUMENT;
        kernel<<<grid, (BM / TM) * (BN / TN), shared, s>>>(a, lda, w + at * ldw, ldw, c + at, ldc,
                                                           plan.splits > 1 ? partial : nullptr, plan.groups_per, m, cols, k);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
        if (plan.splits > 1) {
            const long long size = (long long)m * cols;
            const int blocks = (int)std::min<long long>((size + 255) / 256, 8 * SMS);
            gemm_f32_fold_kernel<<<blocks, 256, 0, s>>>(partial, plan.groups, c + at, ldc, m, cols);
        }
    }
    return tvb_last_error();
}

template <bool ALIGNED>
static int gemm_f32(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, float* partial,
                    int m, int n, int k, int pdl, int w_constant, cudaStream_t s) {
    if (takes_few(m, n, k)) {
        switch (few_template_rows(m)) {
            case 1: return few_of<1, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
            case 2: return few_of<2, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
            case 4: return few_of<4, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
            default: return few_of<8, ALIGNED>(a, lda, w, ldw, c, ldc, m, n, k, pdl, w_constant, s);
        }
    }
    const TilePlan plan = tile_plan(m, n, k);
    if (plan.splits > 1 && !partial) return TVB_BAD_ARGUMENT;
    if (plan.bm == 16) return launch_tiles<16, 4, ALIGNED>(a, lda, w, ldw, c, ldc, partial, plan, m, n, k, s);
    if (plan.bm == 32) return launch_tiles<32, 4, ALIGNED>(a, lda, w, ldw, c, ldc, partial, plan, m, n, k, s);
    return launch_tiles<64, 8, ALIGNED>(a, lda, w, ldw, c, ldc, partial, plan, m, n, k, s);
}

// float32 of scratch that a product of float32 operands wants (0: none)
extern "C" long long tvb_gemm_f32_scratch_floats(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0 || takes_few(m, n, k)) return 0;
    const TilePlan plan = tile_plan(m, n, k);
    return plan.splits > 1 ? (long long)plan.groups * m * plan.cols : 0;
}

// kernels that a product of float32 operands launches
// About what a float32 product of more than 8 rows takes (us).  Measured / this: 677 x 128 x 1,024 28.7 / 31.1, 301 x 64 x 512
// 26.8 / 28.0, 8,192 x 64 x 2,048 76 / 73, 2,048 x 128 x 64 5.5 / 5.3.
extern "C" double tvb_gemm_f32_us(int m, int n, int k) {
    return m <= 0 || n <= 0 || k <= 0 ? 0.0 : tile_plan(m, n, k).us;
}

extern "C" int tvb_gemm_f32_launches(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    if (takes_few(m, n, k)) return 1;
    const TilePlan plan = tile_plan(m, n, k);
    return (n + plan.cols - 1) / plan.cols * (plan.splits > 1 ? 2 : 1);
}

// in_dtype: type of A and W; out_dtype: type of C (float32 output from bfloat16
// inputs serves the logits); scratch: tvb_gemm_f32_scratch_floats floats, for float32 operands.  pdl, w_constant: up to
// 8 rows of float32 run beside the end of the kernel before, which does not write w.
extern "C" int tvb_gemm_nt_simt(const void* a, long long lda, const void* w, long long ldw, void* c,
                                long long ldc, int m, int n, int k, int in_dtype, int out_dtype, float* scratch,
                                int pdl, int w_constant, void* stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0) return TVB_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    if (in_dtype == TVB_F32 && out_dtype == TVB_F32) {
        const bool aligned = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                             ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
        return aligned ? gemm_f32<true>((const float*)a, lda, (const float*)w, ldw, (float*)c, ldc, scratch, m, n, k, pdl, w_constant, s)
                       : gemm_f32<false>((const float*)a, lda, (const float*)w, ldw, (float*)c, ldc, scratch, m, n, k, pdl, w_constant, s);
    }
    dim3 grid((n + TILE_N - 1) / TILE_N, (m + TILE_M - 1) / TILE_M);
    if (grid.y > 65535) return TVB_BAD_ARGUMENT;
    if (in_dtype == TVB_BF16 && out_dtype == TVB_BF16)
        gemm_nt_simt_kernel<bf16, bf16><<<grid, 256, 0, s>>>((const bf16*)a, lda, (const bf16*)w, ldw,
                                                             (bf16*)c, ldc, m, n, k);
    else if (in_dtype == TVB_BF16 && out_dtype == TVB_F32)
        gemm_nt_simt_kernel<bf16, float><<<grid, 256, 0, s>>>((const bf16*)a, lda, (const bf16*)w, ldw,
                                                              (float*)c, ldc, m, n, k);
    else
        return TVB_BAD_ARGUMENT;
    return tvb_last_error();
}
