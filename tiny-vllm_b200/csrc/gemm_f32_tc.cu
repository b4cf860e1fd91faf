// C[m, n] = A[m, k] . W[n, k]^T of float32 operands with more than a few rows, on the fifth-generation tensor cores
// and with all 24 bits of the operands.  (Few rows, narrow products, and rows off the 16-byte boundary: gemm_simt.cu.)
//
// A float32 x times 2^16 is the sum of three bfloat16, exactly, from the smallest float32 to 2^111: x1 is rounded to 8 bits (so
// that the rest has either sign), x2 the first 8 bits of the rest and x3 what is left.  (Without the factor the lowest bits of
// operands below 2^-109 lie under bfloat16's smallest, 2^-133: an error of 5e-7 at 1e-34 and 3e-3 at 1e-38.)  The sums are
// multiplied by 2^-32 when they leave the registers.  A product of two such sums is nine products, of which the six largest
// are taken (x1 w1; x1 w2, x2 w1; x2 w2, x1 w3, x3 w1): what is left out is 2^-23 of |x w| at most, about 2^-26.7 on average
// and with either sign.  (x2 w3 and x3 w2 too: 1.10e-7 to 1.09e-7 below, 677 x 1,024 x 6,144 61 to 69 us.)
// Products of bfloat16 are exact in float32; the tensor cores add them up in tensor memory over 64 k, the small ones
// first, and every such sum is then added by the float32 cores to a sum in registers, in ascending order of k: the
// tensor cores cut off what does not fit instead of rounding it, which over all of k would shrink the sums.
//
// The sum of an output element has one order whatever m is: blocks of 64 k ascending inside a group of 1,024, the groups
// ascending.  It is not the order of gemm_simt.cu: an element's last bits depend on which of the two kernels takes the product.
// Infinities, NaN and values from 2^111 on have no such three parts, and a sum of 2^96 and more is beyond float32 with the
// factors (or NaN: x1 w2 may have the other sign than x1 w1).  All of it ends in a sum that is not finite: such an element is
// summed again by the float32 cores from the operands themselves, and has their bits.
//
// Error against 64-bit sums (2-norm, 1e-8; this / float32 cores), normal operands at k = 4, 8, 16, 64, 256, 1,024, 3,072, 25,600:
// 4.9 / 4.1, 4.9 / 4.8, 5.0 / 6.0, 7.9 / 10.7, 8.9 / 15.0, 11.0 / 15.5, 11.6 / 16.0, 14.6 / 20.1; of that 6 is what the tensor
// cores cut off.  Rows of one value (k = 64, 1,024): 5.2 / 23, 13 / 47.  Where all products have one sign the cuts add up: uniform
// operands in (0, 1) 8.4 / 6.7, 9.6 / 5.1, 8.9 / 4.9 at k = 64, 1,024, 3,072, and with few products that are most of the sum
// (e to twice a normal value, both operands) 53 / 10 at k = 64, 37 / 11 at 1,024; with weights of either sign 12 / 14 there.
//
// x is split once, by a small kernel; w on its way into shared memory, by the 16 warps that also add up the sums: its
// parts are never in memory, and a weight takes no more room than before.  Integer instructions split (the conversion
// to bfloat16 has a quarter of their rate).  A tile is 128 columns of c by 16 to 128 rows: with two stages of 96 KB no
// more fits.  A block of 64 k takes 1.25 us at 16 rows and 1.65 at 128, of which the products are 0.6 and 0.9: what bounds
// the kernel is the chain of splitting, handing over, products and sums, two blocks deep (tensor pipe active 46 %, issue slots
// 56 %, DRAM 5 %).  (Registers decide: at 96 a thread nothing may spill in the loop, since the stream of w evicts from what L1
// is left what is spilled: 2.2 us a block.  Eight warps that split beside eight that add up: 2.0.  Waits by
// one lane that tells the others: 1.4 and 1.9.)
//
// Measured (us, float32 cores / this, weights from memory): 64 rows 4,096 x 1,024 31 / 25, 6,144 x 1,024 43 / 26, 1,024 x
// 3,072 30 / 27; 301 rows 93 / 30, 127 / 32, 76 / 32; 677 rows 176 / 54, 260 / 61 (140 TFLOP/s), 139 / 37; 2,048 rows
// 464 / 119, 687 / 175 (147 TFLOP/s), 354 / 104.
#include <algorithm>
#include <initializer_list>

#include "tc5.cuh"

namespace {

constexpr int BW = 128;                 // rows of w of a tile = lanes of tensor memory
constexpr int MAX_X = 128;              // rows of x of a tile at most; a launch takes a multiple of 16
constexpr int BK = 64;                  // k of a stage: 64 bfloat16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int GROUP = 1024;             // k of a sum in registers
constexpr int GROUP_BLOCKS = GROUP / BK;
constexpr int WORK_WARPS = 16;          // split w and add up sums; one more warp copies x and issues the products
constexpr int WORKERS = 32 * WORK_WARPS;
constexpr int THREADS = WORKERS + 32;
constexpr int SUM_COLS = MAX_X / (WORK_WARPS / 4);       // rows of x whose sums a warp holds
constexpr int STAGES = 2;
constexpr int PART_BYTES = 128 * BK * 2;                 // one of the three parts of 128 rows
constexpr int STAGE_BYTES = 6 * PART_BYTES;              // of w, then of x
constexpr int BARRIERS = 4;
constexpr int SHARED_BYTES = STAGES * STAGE_BYTES + BARRIERS * 8 + 16 + 1024;
constexpr uint32_t TMEM_COLS = 2 * MAX_X;
constexpr int ROWS_A_PASS = WORKERS / (BK / 4);          // 32: a thread takes 4 k of every 32nd row of w
constexpr int PASSES = 128 / ROWS_A_PASS;

enum { GAVE_UP_FULL = 1, GAVE_UP_DONE = 2, GAVE_UP_FREE = 3 };

__device__ int tvb_gemm_f32_tc_status_word = 0;

// a * b + c on two float32 at once.
__device__ __forceinline__ float2 fma_two(float2 a, float2 b, float2 c) {
    union Pair { float2 f; unsigned long long u; } x{a}, y{b}, z{c}, r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(x.u), "l"(y.u), "l"(z.u));
    return r.f;
}

constexpr float PART_SCALE = 65536.0f, SUM_SCALE = 1.0f / (PART_SCALE * PART_SCALE);

__device__ __forceinline__ float2 scale_two(float2 a) {
    union Pair { float2 f; unsigned long long u; } x{a}, y{make_float2(PART_SCALE, PART_SCALE)}, r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(x.u), "l"(y.u));
    return r.f;
}

// Four float32 times 2^16 as three times four bfloat16.
__device__ __forceinline__ void split_four(const float4& x, uint2* part) {
    float2 rest[2] = {scale_two(make_float2(x.x, x.y)), scale_two(make_float2(x.z, x.w))};
    uint32_t* words = reinterpret_cast<uint32_t*>(part);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const uint32_t half = p == 0 ? 0x8000u : 0u;
            const uint32_t a = __float_as_uint(rest[j].x) + half, b = __float_as_uint(rest[j].y) + half;
            words[2 * p + j] = __byte_perm(a, b, 0x7632);
            if (p == 2) break;
            rest[j] = fma_two(make_float2(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u)),
                              make_float2(-1.0f, -1.0f), rest[j]);           // exact
        }
    }
}

// One lane of the warp, chosen so that the compiler keeps the control flow of the warp uniform.
__device__ __forceinline__ bool elect_lane() {
    uint32_t elected;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.b32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(elected));
    return elected != 0;
}

constexpr int AGAIN_K = 32, AGAIN_STRIDE = AGAIN_K + 4;  // k of a step, floats from row to row in shared memory (the banks)
constexpr int AGAIN_ROWS = 4;                           // rows of x at a time
template <int ROWS> constexpr int AGAIN_FLOATS = (32 + ROWS) * AGAIN_STRIDE;            // shared memory of a warp
static_assert(WORK_WARPS * AGAIN_FLOATS<AGAIN_ROWS> * 4 <= STAGES * STAGE_BYTES, "it lies where the stages were");

// Elements of c that are not finite, of ROWS rows from `row` on and a column a lane (bit i of `again`: row + i), are summed again
// from the operands by the float32 cores, in the order of gemm_simt.cu (segments of 128 k, a chain over the even and one over the
// odd k of each; four segments a group, the groups ascending): those with infinities, and those that are beyond float32 in parts
// or with the parts' factors although theirs need not be.  A row of x with a NaN has nothing but NaN already.
// What is left is finite again, or NaN from the next norm on, so that this runs rarely: 677 x 1,024 x 6,144 takes 61 us, with an
// infinity in one row 87, all NaN 74, all infinities or beyond 2^96 920 (the float32 cores 261); 677 x 3,072 x 1,024, added up from partial
// sums, 37, 460, 45 and 1,390 (139).
template <int ROWS>
__device__ __noinline__ void sum_again(unsigned again, int row, int col, const float* a, int64_t lda, const float* w, int64_t ldw,
                                       float* c, int64_t ldc, int m, int k, const int* nan_rows, float* tile) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (row + i < m && nan_rows[row + i]) again &= ~(1u << i);
    const unsigned cols = __ballot_sync(0xffffffffu, again != 0);
    if (cols == 0) return;
    float4 held[8];                                                  // of w: 4 k of every fourth column
    float held_x[ROWS];
    auto load = [&](int at) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int of = i * 4 + lane / 8, of_col = __shfl_sync(0xffffffffu, col, of), from = at + (lane & 7) * 4;
            held[i] = (cols >> of & 1) && from < k ? *reinterpret_cast<const float4*>(w + (int64_t)of_col * ldw + from)
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i) held_x[i] = row + i < m && at + lane < k ? a[(int64_t)(row + i) * lda + at + lane] : 0.0f;
    };
    float even[ROWS], odd[ROWS], group[ROWS], total[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) even[i] = odd[i] = group[i] = total[i] = 0.0f;
    load(0);
    for (int at = 0; at < k; at += AGAIN_K) {
        __syncwarp();                                                // (what is in the tile has been read)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(tile + (i * 4 + lane / 8) * AGAIN_STRIDE + (lane & 7) * 4) = held[i];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) tile[(32 + i) * AGAIN_STRIDE + lane] = held_x[i];
        __syncwarp();
        if (at + AGAIN_K < k) load(at + AGAIN_K);
#pragma unroll
        for (int q = 0; q < AGAIN_K; q += 4) {                       // (zeros behind k)
            const float4 wv = *reinterpret_cast<const float4*>(tile + lane * AGAIN_STRIDE + q);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const float4 xv = *reinterpret_cast<const float4*>(tile + (32 + i) * AGAIN_STRIDE + q);
                even[i] = __fmaf_rn(xv.z, wv.z, __fmaf_rn(xv.x, wv.x, even[i]));
                odd[i] = __fmaf_rn(xv.w, wv.w, __fmaf_rn(xv.y, wv.y, odd[i]));
            }
        }
        const int segment = at / 128;
        const bool last = at + AGAIN_K >= k;
        if ((at + AGAIN_K) % 128 != 0 && !last) continue;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float sum = __fadd_rn(even[i], odd[i]);
            group[i] = segment % 4 == 0 ? sum : __fadd_rn(group[i], sum);
            if (segment % 4 == 3 || last) total[i] = segment < 4 ? group[i] : __fadd_rn(total[i], group[i]);
            even[i] = odd[i] = 0.0f;
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (again >> i & 1) c[(int64_t)(row + i) * ldc + col] = total[i];
}

// A row of x a block: its three parts, [3][m][kp] with zeros from k on, and whether it holds a NaN.
__global__ void __launch_bounds__(128)
split_rows_kernel(const float* a, int64_t lda, uint2* parts, int* nan_rows, int m, int k, int kp) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x;
    bool nan = false;
    for (int at = threadIdx.x * 4; at < kp; at += 128 * 4) {
        const float4 x = at < k ? *reinterpret_cast<const float4*>(a + (int64_t)row * lda + at) : make_float4(0.f, 0.f, 0.f, 0.f);
        nan |= x.x != x.x || x.y != x.y || x.z != x.z || x.w != x.w;
        uint2 part[3];
        split_four(x, part);
#pragma unroll
        for (int i = 0; i < 3; ++i) parts[((int64_t)(i * m + row) * kp + at) / 4] = part[i];
    }
    const int any = __syncthreads_or(nan);
    if (threadIdx.x == 0) nan_rows[row] = any;
}

// One CTA: a tile of up to 128 columns of c and `nx` rows, over groups [z * groups_per, ...) of k.  partial == nullptr: all groups,
// whose sums meet in c; else group g goes to partial[g][m][n].  map_x: the parts of x.
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const int* nan_rows, const float* a, int64_t lda,
                   const float* w, int64_t ldw, float* c, int64_t ldc, float* partial, int groups_per, int m, int n, int k, int nx) {
    extern __shared__ uint8_t raw_shared[];
    const uint32_t base = (smem_address(raw_shared) + 1023u) & ~1023u;
    uint8_t* aligned = raw_shared + (base - smem_address(raw_shared));
    const uint32_t bars = base + STAGES * STAGE_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto done_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(aligned + STAGES * STAGE_BYTES + BARRIERS * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
    volatile int* not_finite = abort_flag + 1;          // whether an element of c is not
    int* status = &tvb_gemm_f32_tc_status_word;

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int col0 = blockIdx.x * BW, row0 = blockIdx.y * nx;
    const int k_from = blockIdx.z * groups_per * GROUP, k_to = min(k, k_from + groups_per * GROUP);
    const int blocks = (k_to - k_from + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), WORK_WARPS + 1); mbar_init(done_bar(s), 1); }
        *abort_flag = *not_finite = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        prefetch_tensormap(&map_x);
    }
    if (warp == 0) tmem_alloc(smem_address(tmem_base_slot), TMEM_COLS);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_base_slot;
    // waits of a whole warp
    auto warp_wait = [&](uint32_t bar, uint32_t parity, int code) {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code)) != 0;
    };

    if (warp < WORK_WARPS) {
        // ---- Operands: 4 k of every 32nd row of w a thread, the next block's values in flight while this one's are split.
        // Sums: the 32 lanes of tensor memory that the warp's number modulo 4 names, SUM_COLS of the rows of x.
        // Block b is split while the products of b - 1 run, then the sums of b - 1 are added up.  When those are done, the
        // stage that b + 1 goes to is free, and a warp that hands b + 1 over has read the accumulator it goes to.
        const int chunk = threadIdx.x & 15, r0 = threadIdx.x >> 4;
        const float* w_from = w + (int64_t)(col0 + r0) * ldw + k_from + chunk * 4;
        const uint32_t w_at = base + (uint32_t)(r0 * 128 + (((chunk >> 1) ^ (r0 & 7)) << 4) + (chunk & 1) * 8);   // (32 rows: the same)
        float4 held[PASSES];
        auto load = [&](int pass, int block) {
            const bool in = col0 + r0 + pass * ROWS_A_PASS < n && k_from + block * BK + chunk * 4 < k_to;
            held[pass] = in ? *reinterpret_cast<const float4*>(w_from + (int64_t)(pass * ROWS_A_PASS) * ldw + block * BK)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        const int quarter = warp & 3, first = (warp >> 2) * SUM_COLS;
        const int col = col0 + quarter * 32 + lane;
        const int rows = min(min(nx - first, SUM_COLS), m - row0 - first); // of this warp's sums; none where negative
        float sum[SUM_COLS];
#pragma unroll
        for (int j = 0; j < SUM_COLS; ++j) sum[j] = 0.0f;
#pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) load(pass, 0);
        for (int b = 0; b <= blocks; ++b) {
            if (b < blocks) {
#pragma unroll
                for (int pass = 0; pass < PASSES; ++pass) {
                    uint2 part[3];
                    split_four(held[pass], part);
                    if (b + 1 < blocks) load(pass, b + 1);
                    const uint32_t at = w_at + (uint32_t)((b & 1) * STAGE_BYTES + pass * ROWS_A_PASS * 128);
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at + (uint32_t)(i * PART_BYTES)), "r"(part[i].x),
                                     "r"(part[i].y) : "memory");
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(b & 1));
            }
            if (b == 0) continue;
            const int before = b - 1, acc = before & 1;
            if (!warp_wait(done_bar(acc), (before >> 1) & 1u, GAVE_UP_DONE)) break;
            tc_fence_after_sync();
#pragma unroll
            for (int at = 0; at < SUM_COLS; at += 8) {
                if (at >= rows) break;
                uint32_t v[8];
                tmem_load_8(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * MAX_X + first + at), v);
                tmem_load_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) sum[at + j] = __fadd_rn(sum[at + j], __uint_as_float(v[j]));
            }
            tc_fence_before_sync();
            if (b % GROUP_BLOCKS != 0 && b != blocks) continue;
            const int g = before / GROUP_BLOCKS;
            const int64_t ld = partial ? n : ldc;
            float* to = (partial ? partial + (int64_t)(blockIdx.z * groups_per + g) * m * n : c) + (int64_t)(row0 + first) * ld + col;
            if (col < n) {
#pragma unroll
                for (int j = 0; j < SUM_COLS; ++j) {
                    if (j < rows) {
                        const float scaled = __fmul_rn(sum[j], SUM_SCALE);
                        const float total = !partial && g > 0 ? __fadd_rn(*to, scaled) : scaled;    // (this thread's own sum so far)
                        *to = total;
                        if (!partial && !isfinite(total)) *not_finite = 1;          // (partial sums: when they are added up)
                    }
                    to += ld;
                }
            }
#pragma unroll
            for (int j = 0; j < SUM_COLS; ++j) sum[j] = 0.0f;
        }
    } else {
        // ---- copies of x, a block ahead, and products: of a block the smallest first
        const uint32_t idesc = instruction_descriptor_bf16(BW, nx, false);
        auto copy = [&](int b) {
            if (elect_lane()) {
                const uint32_t at = base + (b & 1) * STAGE_BYTES + 3 * PART_BYTES;
                mbar_arrive_expect(full_bar(b & 1), 3u * (uint32_t)nx * BK * 2);
#pragma unroll
                for (int i = 0; i < 3; ++i) tma_load_3d(at + i * PART_BYTES, &map_x, k_from + b * BK, row0, i, full_bar(b & 1));
            }
            __syncwarp();
        };
        pdl_wait();
        copy(0);
        if (blocks > 1) copy(1);
        for (int b = 0; b < blocks; ++b) {
            if (!warp_wait(full_bar(b & 1), (b >> 1) & 1u, GAVE_UP_FULL)) break;
            tc_fence_after_sync();
            if (elect_lane()) {
                const uint32_t w_at = base + (b & 1) * STAGE_BYTES, x_at = w_at + 3 * PART_BYTES;
                const uint32_t d_tmem = tmem_base + (uint32_t)((b & 1) * MAX_X);
                constexpr int W_PART[6] = {2, 0, 1, 1, 0, 0}, X_PART[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    const uint64_t w_desc = tile_descriptor(w_at + W_PART[p] * PART_BYTES);
                    const uint64_t x_desc = tile_descriptor(x_at + X_PART[p] * PART_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk) tc_mma(d_tmem, w_desc + 2u * kk, x_desc + 2u * kk, idesc, (p | kk) != 0);
                }
                tc_commit(done_bar(b & 1));
            }
            __syncwarp();
            if (b > 0 && b + 1 < blocks) {
                if (!warp_wait(done_bar((b - 1) & 1), ((b - 1) >> 1) & 1u, GAVE_UP_FREE)) break;
                copy(b + 1);
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    const bool gave_up = *abort_flag != 0;
    if (gave_up) {
        // copies or products may still be in flight from and to this CTA's memory: give them time
        const long long started = clock64();
        while (clock64() - started < 400000) __nanosleep(1000);
    }
    pdl_wait();
    if (*not_finite && !gave_up && warp < WORK_WARPS) {
        const int first = (warp >> 2) * SUM_COLS, col = col0 + (warp & 3) * 32 + lane;
        const int rows_to = min(min(row0 + nx, row0 + first + SUM_COLS), m);
        float* tile = reinterpret_cast<float*>(aligned) + warp * AGAIN_FLOATS<AGAIN_ROWS>;                // (the stages are free)
        for (int row = row0 + first; row < rows_to; row += AGAIN_ROWS) {
            unsigned again = 0;                                                         // of this thread's own elements
            for (int i = 0; i < AGAIN_ROWS; ++i)
                if (row + i < rows_to && col < n && !isfinite(c[(int64_t)(row + i) * ldc + col])) again |= 1u << i;
            if (__any_sync(0xffffffffu, again))
                sum_again<AGAIN_ROWS>(again, row, col, a, lda, w, ldw, c, ldc, m, k, nan_rows, tile);
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_free(tmem_base, TMEM_COLS);
    }
}

// What of c the warps of the kernel below have written and is not finite, summed again: a row of a warp's at a time.
template <int VEC>
__device__ __noinline__ void fold_again(float* c, int64_t ldc, int m, int n, const float* a, int64_t lda, const float* w,
                                        int64_t ldw, int k, const int* nan_rows, float* tile) {
    const int words = n / VEC, lane = threadIdx.x & 31;
    const int64_t total = (int64_t)m * words;
    for (int64_t from = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; from < total; from += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = min(from + lane, total - 1);
        const int row = (int)(i / words), at = (int)(i % words) * VEC;
        for (int j = 0; j < VEC; ++j) {
            unsigned again = __ballot_sync(0xffffffffu, from + lane < total && !isfinite(c[(int64_t)row * ldc + at + j]));
            while (again) {
                const int of_row = __shfl_sync(0xffffffffu, row, __ffs(again) - 1);
                const unsigned now = again & __ballot_sync(0xffffffffu, row == of_row);
                again &= ~now;
                sum_again<1>(now >> lane & 1, of_row, at + j, a, lda, w, ldw, c, ldc, m, k, nan_rows, tile);
            }
        }
    }
}

// c = the sum of the groups' partial products, in ascending order; VEC neighbouring columns a thread.
template <int VEC>
__global__ void __launch_bounds__(256, 4)
fold_groups_kernel(const float* __restrict__ partial, int groups, float* c, int64_t ldc, int m, int n, const float* a, int64_t lda,
                   const float* w, int64_t ldw, int k, const int* nan_rows) {
    __shared__ __align__(16) float tiles[256 / 32][AGAIN_FLOATS<1>];
    const int words = n / VEC;
    const int64_t size = (int64_t)m * n, total = (int64_t)m * words;
    bool again = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = total <= 0x7fffffff ? (uint32_t)i / (uint32_t)words : i / words;
        const int64_t at = (i - row * words) * VEC;
        float sum[VEC], more[VEC];
        load_values<VEC>(partial + row * n + at, sum);
        for (int g = 1; g < groups; ++g) {
            load_values<VEC>(partial + g * size + row * n + at, more);
#pragma unroll
            for (int j = 0; j < VEC; ++j) sum[j] = __fadd_rn(sum[j], more[j]);
        }
        store_values<VEC>(c + row * ldc + at, sum);
#pragma unroll
        for (int j = 0; j < VEC; ++j) again |= !isfinite(sum[j]);
    }
    if (__any_sync(0xffffffffu, again)) fold_again<VEC>(c, ldc, m, n, a, lda, w, ldw, k, nan_rows, tiles[threadIdx.x / 32]);
}

struct Plan { int nx, tiles_x, groups, groups_per, splits; double us; };

constexpr long long SCRATCH_FLOATS = 16LL << 20;      // the most that partial sums take

Plan plan_of(int m, int n, int k, int sms) {
    Plan best{};
    best.groups = (k + GROUP - 1) / GROUP;
    const long long tiles_w = (n + BW - 1) / BW;
    const int fewest = (m + MAX_X - 1) / MAX_X;
    double least = 0.0;
    for (int tiles = fewest; tiles <= fewest + 4 && tiles <= (m + 15) / 16; ++tiles) {
        const int nx = ((m + tiles - 1) / tiles + 15) / 16 * 16, tiles_x = (m + nx - 1) / nx;
        const double block_us = 1.2 + 0.0035 * nx;
        for (int per = best.groups; per >= 1; --per) {
            const int splits = (best.groups + per - 1) / per;
            if (splits > 1 && ((long long)best.groups * m * n > SCRATCH_FLOATS || splits > 65535)) break;
            const long long waves = (tiles_w * tiles_x * splits + sms - 1) / sms;
            const double us = waves * ((std::min(per * GROUP, k) + BK - 1) / BK * block_us + 4.0) +
                              (splits > 1 ? 3.0 + 8.0 * best.groups * m * n / 6e6 : 0.0);
            if (best.nx == 0 || us < least) {
                least = us;
                best.nx = nx; best.tiles_x = tiles_x; best.groups_per = per; best.splits = splits;
            }
        }
    }
    best.us = least;
    return best;
}

// Scratch of a product: partial sums, the parts of x, and a word a row of x.  Partial sums take up to 64 MiB and so do the
// parts (128 rows, where those take more): a product of more rows runs a range of rows at a time.
long long padded_k(int k) { return (k + BK - 1) / BK * BK; }
int range_rows(int m, int k) {
    const long long fit = std::max(128LL, SCRATCH_FLOATS * 4 / (6 * padded_k(k)) / 128 * 128);
    const long long ranges = (m + fit - 1) / fit;
    return ranges <= 1 ? m : (int)(((m + ranges - 1) / ranges + 127) / 128 * 128);
}
int plan_sms() {
    const int sms = tvb_sm_count();
    return sms > 0 ? sms : 148;                       // (asked for sizes without a device)
}
long long sum_bytes(const Plan& plan, int m, int n) {
    return plan.splits > 1 ? ((long long)plan.groups * m * n * 4 + 127) / 128 * 128 : 0;
}

}  // namespace

// 0, or which wait gave up in some launch since the last call (1 operands, 2 and 3 products); reading clears it.
// Synchronises the device.
extern "C" int tvb_gemm_f32_tc_status() {
    int value = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&value, tvb_gemm_f32_tc_status_word, sizeof(int)) != cudaSuccess) return -1;
    if (value != 0) cudaMemcpyToSymbol(tvb_gemm_f32_tc_status_word, &zero, sizeof(int));
    return value;
}

extern "C" long long tvb_gemm_f32_tc_scratch_bytes(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    const int rows = range_rows(m, k), last = m - (m - 1) / rows * rows;
    long long most = 0;
    for (int of : {rows, last})
        most = std::max(most, sum_bytes(plan_of(of, n, k, plan_sms()), of, n) + 3 * of * padded_k(k) * 2 + 4ll * of);
    return most;
}

// About what a product takes (us): its plan's estimate, and splitting x, at 1.2 ns a row or the rate of memory.
// Measured / this: 301 x 64 x 512 15.0 / 15.9, 8,192 x 64 x 2,048 89 / 92, 677 x 128 x 1,024 27.0 / 29.0.
extern "C" double tvb_gemm_f32_tc_us(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0.0;
    const int rows = range_rows(m, k), last = m - (m - 1) / rows * rows;
    auto range = [&](int of) { return plan_of(of, n, k, plan_sms()).us + 0.5 + of * std::max(0.0012, 1.4e-6 * k); };
    return (m - 1) / rows * range(rows) + range(last);
}

// kernels that a product launches
extern "C" int tvb_gemm_f32_tc_launches(int m, int n, int k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    const int rows = range_rows(m, k), last = m - (m - 1) / rows * rows;
    return (m - 1) / rows * (plan_of(rows, n, k, plan_sms()).splits > 1 ? 3 : 2) + (plan_of(last, n, k, plan_sms()).splits > 1 ? 3 : 2);
}

static int launch_range(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, int m, int n, int k,
                        uint8_t* scratch, int sms, int pdl, int w_constant, cudaStream_t s) {
    const Plan plan = plan_of(m, n, k, sms);
    if (plan.tiles_x > 65535) return TVB_BAD_ARGUMENT;
    float* partial = plan.splits > 1 ? reinterpret_cast<float*>(scratch) : nullptr;
    uint8_t* parts = scratch + sum_bytes(plan, m, n);
    const long long kp = padded_k(k);
    int* nan_rows = reinterpret_cast<int*>(parts + 3 * m * kp * 2);
    CUtensorMap map_x;
    {
        const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)m, 3};
        const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)(m * kp * 2)};
        const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)plan.nx, 1};
        if (!tvb_make_map(&map_x, parts, 3, dims, strides, box)) return (int)cudaErrorNotSupported;
    }
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SHARED_BYTES);
    if (e != cudaSuccess) return (int)e;
    // The product's kernel reads w without waiting: the kernel that splits x, which it follows, starts behind all launches
    // before, unless none of those that may still run writes w.
    TvbLaunch split(dim3(m), dim3(128), 0, s, pdl && w_constant);
    e = cudaLaunchKernelEx(&split.config, split_rows_kernel, a, (int64_t)lda, reinterpret_cast<uint2*>(parts), nan_rows, m, k, (int)kp);
    if (e != cudaSuccess) return (int)e;
    TvbLaunch launch(dim3((n + BW - 1) / BW, plan.tiles_x, plan.splits), dim3(THREADS), SHARED_BYTES, s, pdl);
    e = cudaLaunchKernelEx(&launch.config, gemm_f32_tc_kernel, map_x, (const int*)nan_rows, a, (int64_t)lda, w, (int64_t)ldw, c,
                           (int64_t)ldc, partial, plan.groups_per, m, n, k, plan.nx);
    if (e != cudaSuccess) return (int)e;
    if (plan.splits > 1) {
        const bool by_four = n % 4 == 0 && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
        const int blocks = (int)std::min<long long>(((long long)m * n / (by_four ? 4 : 1) + 255) / 256, 8LL * sms);
        auto fold = by_four ? fold_groups_kernel<4> : fold_groups_kernel<1>;
        fold<<<blocks, 256, 0, s>>>(partial, plan.groups, c, ldc, m, n, a, lda, w, ldw, k, nan_rows);
    }
    return tvb_last_error();
}

// c[m, n] = a . w^T; rows of a and w on 16-byte boundaries.  scratch: tvb_gemm_f32_tc_scratch_bytes, on a 128-byte
// boundary.  w_constant: no launch that may still run writes w.
extern "C" int tvb_gemm_f32_tc(const float* a, long long lda, const float* w, long long ldw, float* c, long long ldc, int m,
                               int n, int k, uint8_t* scratch, int pdl, int w_constant, void* stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0 || k % 4 || lda % 4 || ldw % 4 || !scratch ||
        ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) || (reinterpret_cast<uintptr_t>(scratch) & 127))
        return TVB_BAD_ARGUMENT;
    const int sms = tvb_sm_count();
    if (sms <= 0) return (int)cudaErrorInvalidDevice;
    const int rows = range_rows(m, k);
    for (int at = 0; at < m; at += rows) {
        const int status = launch_range(a + at * lda, lda, w, ldw, c + at * ldc, ldc, std::min(rows, m - at), n, k, scratch, sms,
                                        pdl, w_constant, (cudaStream_t)stream);
        if (status != 0) return status;
    }
    return 0;
}
