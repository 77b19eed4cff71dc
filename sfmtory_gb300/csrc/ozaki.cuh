// FP64 trailing update of the blocked Cholesky on the BF16 tensor cores, by
// error-free splitting (Ozaki, Ogita, Oishi & Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012).
//
// The update is A[I, J] -= P_I P_J^T with P the 64-column panel below the
// diagonal block. Each panel row r is scaled by 2^-e_r (e_r: the binary
// exponent of its largest entry, so |x| < 1) and cut into kOzSlices slices
// of 8 bits:
//   P[r, t] = 2^e_r sum_{i=1..7} s_i[r, t] 2^-8i,  s_i integer, |s_i| <= 255
// (exact to 56 bits >= 53). An integer of at most 8 significant bits is a
// BF16 value and a product of two is below 2^16, so a 64-term dot product
// of slices is an integer below 2^22 that the tensor cores' FP32
// accumulation holds exactly. The update is
//   (P P^T)[r, c] = 2^(e_r + e_c) sum_{i,j} 2^-8(i+j) G_ij[r, c],
//   G_ij = S_i[R] S_j[C]^T,
// of which the 28 terms with i + j <= 8 are kept. Products of one weight d =
// i + j share an FP32 accumulator G_d (exact for d <= 5: at most four products,
// < 2^24). The groups d <= 6 are combined exactly in 64-bit integers,
//   L = 2^32 G_2 + 2^24 G_3 + 2^16 G_4 + 2^8 G_5 + G_6   (< 2^55),
// the last two in FP32, T = G_7 + G_8 / 2^8, and
//   (P P^T)[r, c] = 2^(e_r + e_c - 48) (L + T / 2^8)
// is formed in FP64 (L rounds to 53 bits: the FP64 rounding of the product
// itself) and subtracted.
//
// Error, in units of s = 2^(e_r + e_c) (an entry of P P^T is below 64 s): the
// weights left out are below 2^-47.3 (six products of weight 9, each < 64 x
// 255^2 x 2^-72). G_6 may pass 2^24 when digits close to 255 share a sign; its
// last four accumulations then lose up to two units of 2^-48 each, 2^-45. T
// rounds below 2^-54, and digits of an entry below 2^-56 of its row's largest
// are cut off (2^-49 for 64 of both rows). With the result's own rounding the
// sum stays below 2^-44 (measured: 2^-45.3 for digits of 254 and 255, 2^-46.8 for
// random ones); 64 multiply-adds in FP64 are within 2^-41.
//
// The products run on the fifth-generation tensor cores: one block per 128 x 64
// tile, its slices fetched by bulk copies in the layout that tcgen05.mma reads
// (a 64-wide panel's BF16 row is the 128 bytes of a swizzle row), 112
// instructions of 128 x 64 x 16 into seven accumulators in tensor memory, one
// per weight. The epilogue reads them back a row a thread and assembles each
// entry's FP64 value in integers, so that one FP64 instruction is left of
// four (65 cycles a warp each). 65 us for the 741 64 x 64 tiles of n = 2560,
// against 102 us with warp-level mma.sync from 64 x 32 tiles and an FP64
// epilogue; the factor of n = 5000 takes 8.6 ms, 14.4 before. (Entries passed
// through shared memory to a row a warp: 57 us alone, but the factor 9.3 ms;
// the next diagonal block runs beside this kernel.)
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace sfmba {

constexpr int kOzSlices = 7;
constexpr int kOzK = 64;     // panel width (the Cholesky block)
constexpr int kOzRows = 128;  // rows of an output tile
constexpr int kOzCols = 64;   // columns of an output tile (32 where few tiles leave SMs idle)
constexpr int kOzThreads = 256;
// Slices of 64 panel rows: [kOzSlices][64 rows][64], the eight 16-byte pieces
// of a row permuted by its number mod 8 (the 128-byte swizzle).
constexpr int kOzSliceBytes = 64 * kOzK * 2;
constexpr size_t kOzBlockElems = (size_t)kOzSlices * 64 * kOzK;
// Shared: the rows' slices (two blocks each), the columns', 1024-byte aligned.
constexpr int kOzColsAt = kOzSlices * 2 * kOzSliceBytes;
constexpr size_t kOzSmem = (size_t)kOzColsAt + kOzSlices * kOzSliceBytes + 1024;
constexpr int kOzPolls = 1 << 18;  // bound of every wait

// Digit i (1..7) of |x| 2^-e in base 256, |x| < 2^e, from the bits of |x|:
// the significand shifted to 56 fractional bits, what lies below cut off.
__device__ __forceinline__ unsigned long long oz_fraction(unsigned long long abs_bits, int emax) {
    const int ex = (int)(abs_bits >> 52);
    const unsigned long long m = abs_bits & ((1ULL << 52) - 1);
    const unsigned long long sig = ex ? m | (1ULL << 52) : m;
    const int right = emax - max(ex, 1) - 3;
    return right <= 0 ? sig << -right : right < 64 ? sig >> right : 0;
}

// Slices and exponent of one panel row of nb <= 64 entries (one warp; lane
// owns columns lane and lane + 32; missing columns are zero).
// block: the 64-row block that it is row r of (kOzBlockElems). Integer
// arithmetic on the bits throughout (GB300's FP64 pipe takes 65 cycles for
// each of the ~60 multiplications, truncations and conversions that the same
// digits cost in FP64: 3.8 against 13 us for 2500 rows).
__device__ __forceinline__ void oz_split_row(const double *__restrict__ row, int nb, int lane,
                                             __nv_bfloat16 *__restrict__ block, int r, int *e_out) {
    constexpr unsigned long long kAbs = ~(1ULL << 63);
    const unsigned long long b0 = lane < nb ? (unsigned long long)__double_as_longlong(row[lane]) : 0;
    const unsigned long long b1 = lane + 32 < nb ? (unsigned long long)__double_as_longlong(row[lane + 32]) : 0;
    const int emax = __reduce_max_sync(0xffffffffu, max((int)((b0 & kAbs) >> 52), (int)((b1 & kAbs) >> 52)));
    // max |x| = f 2^e with f in [0.5, 1): |x| 2^-e < 1. A row of zeros and
    // subnormals takes e as if its largest were the smallest normal number.
    const int scale = max(emax, 1), e = scale - 1022;
    const unsigned long long m0 = oz_fraction(b0 & kAbs, scale), m1 = oz_fraction(b1 & kAbs, scale);
    const int at = (((lane >> 3) ^ (r & 7)) << 3) + (lane & 7);
    const float s0 = b0 >> 63 ? -1.0f : 1.0f, s1 = b1 >> 63 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < kOzSlices; ++i) {
        const unsigned d0 = (unsigned)(m0 >> (48 - 8 * i)) & 255u, d1 = (unsigned)(m1 >> (48 - 8 * i)) & 255u;
        block[(i * 64 + r) * kOzK + at] = __float2bfloat16_rn(s0 * (float)d0);
        block[(i * 64 + r) * kOzK + (at ^ 32)] = __float2bfloat16_rn(s1 * (float)d1);  // column lane + 32
    }
    if (lane == 0) *e_out = e;
}

// -2^x v for the products' value v = L + T / 2^8 rounded as above (L to 53 bits,
// then the sum): assembled from the bits of L and T in integers where L is
// below 2^53 and the result normal.
__device__ __forceinline__ double oz_value(long long L, float T, int x0) {
    int x = x0;
    // L + T / 2^8 = h + lo / 2^16; T is a multiple of 2^-8
    const int t = __float2int_rd(T);
    const unsigned lo = ((unsigned)(t & 255) << 8) | (unsigned)__float2int_rn((T - (float)t) * 256.0f);
    const long long h = L + (t >> 8);
    const unsigned long long neg = (unsigned long long)(h >> 63);
    unsigned long long mh = ((unsigned long long)h ^ neg) + (neg != 0 && lo == 0);  // |.|: mh + ml / 2^16
    unsigned ml = neg ? (0u - lo) & 0xffffu : lo;
    if (mh == 0) {  // rows that share little or nothing
        if (ml == 0) return -0.0;
        mh = ml;
        ml = 0;
        x -= 16;
    }
    const int lz = __clzll((long long)mh), e = 1085 - lz + x;
    if ((unsigned long long)(L + (1LL << 53)) > (1ULL << 54) || e < 1 || e > 2044)
        return ldexp(-fma((double)T, 0.00390625, (double)L), x0);
    const unsigned long long low = (unsigned long long)ml << 48;
    const unsigned long long m = (mh << lz) | (low >> (64 - lz));  // the top 64 bits, the last one set below
    const unsigned rest = (unsigned)(m & 0x7ff) | ((low << lz) != 0);
    unsigned long long bits = m >> 11;
    bits += (rest + 0x3ff + (unsigned)(bits & 1)) >> 11;  // to nearest, ties to even
    bits = (bits + ((unsigned long long)e << 52)) ^ (~neg << 63);
    return __longlong_as_double((long long)bits);
}

__device__ __forceinline__ unsigned oz_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool oz_wait(unsigned bar, int polls = kOzPolls) {
    for (int k = 0; k < polls; ++k) {
        unsigned ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(bar)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Eight columns of this warp's 32 accumulator rows, a row a lane; there after
// oz_wait_acc.
__device__ __forceinline__ void oz_load_acc(unsigned addr, unsigned (&u)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr));
}
template <int N>
__device__ __forceinline__ void oz_wait_acc(unsigned (&u)[N][8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int d = 0; d < N; ++d)
#pragma unroll
        for (int k = 0; k < 8; ++k) asm volatile("" : "+r"(u[d][k]));  // no use moves above the wait
}

// Descriptor of a K-major operand in rows of 128 swizzled bytes (groups of
// eight rows 1024 bytes apart) at shared address `at`.
__device__ __forceinline__ unsigned long long oz_operand(unsigned at) {
    return (unsigned long long)((at >> 4) & 0x3fff) | (1ULL << 16) | (64ULL << 32) | (1ULL << 46) | (2ULL << 61);
}

// One 128 x NC tile (NC 32 or 64) of the update, A[r, c] -= (P P^T)[r, c] for
// r < mi, c < mj, by kOzThreads threads with an SM's shared and tensor memory
// to themselves. A: the tile's first entry, row stride lda. diag: row c0 + c of
// the tile is its column c (only c0 + c <= r is written); otherwise c0 is its
// first column's place in a block of 64. slR / slC: the 64-row blocks of slices
// of its first rows (the next block follows) and of its columns. eR / eC: the
// exponents of its rows and columns. smem: kOzSmem bytes. False, and A as it
// was, if a wait (of `polls` attempts for a slice) gave up; the copies and
// products under way are awaited all the same.
template <int NC>
__device__ __forceinline__ bool oz_tile_update(double *A, size_t lda, int mi, int mj, bool diag, int c0,
                                               const __nv_bfloat16 *slR, const __nv_bfloat16 *slC, const int *eR,
                                               const int *eC, unsigned char *smem, int polls) {
    constexpr int kWarpCols = NC / 2;
    // slice i there; products done (tcgen05.commit) and issued (the thread that issues them)
    __shared__ alignas(8) unsigned long long bars[kOzSlices + 1];
    __shared__ unsigned tmem_at;
    __shared__ int missed;  // a slice did not come
    __shared__ int xC[NC];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned base = (oz_smem(smem) + 1023u) & ~1023u, there = oz_smem(&bars[0]), done = oz_smem(&bars[kOzSlices]);
    if (tid == 0) {
        for (int i = 0; i <= kOzSlices; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(there + 8 * i), "r"(i < kOzSlices ? 1 : 2)
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const int halves = mi > 64 ? 2 : 1;
        for (int i = 0; i < kOzSlices; ++i) {
            auto copy = [&](unsigned dst, const __nv_bfloat16 *src, int bytes) {
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                    "l"(src), "r"(bytes), "r"(there + 8 * i)
                    : "memory");
            };
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(there + 8 * i),
                         "r"(halves * kOzSliceBytes + (diag ? 0 : NC * kOzK * 2))
                         : "memory");
            for (int h = 0; h < halves; ++h)
                copy(base + (2 * i + h) * kOzSliceBytes, slR + h * kOzBlockElems + i * 64 * kOzK, kOzSliceBytes);
            if (!diag) copy(base + kOzColsAt + i * kOzSliceBytes, slC + (i * 64 + c0) * kOzK, NC * kOzK * 2);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(oz_smem(&tmem_at))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid >= 64 && tid < 64 + NC) xC[tid - 64] = tid - 64 < mj ? eC[tid - 64] : 0;
    const int r = 32 * (warp & 3) + lane, cw = kWarpCols * (warp >> 2);  // this thread's row and first column
    const int xr = r < mi ? eR[r] - 48 : 0;
    const int cols = (r < mi ? min(mj, diag ? r + 1 - c0 : mj) : 0) - cw;
    double *a = A + (size_t)r * lda + cw;
    double acc[kWarpCols];  // fetched while the products run
#pragma unroll
    for (int k = 0; k < kWarpCols; ++k) acc[k] = k < cols ? a[k] : 0.0;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = tmem_at;
    if (tid == 0) {
        // FP32 accumulators, BF16 operands, both K-major, 128 x NC
        constexpr unsigned kShape = (1u << 4) | (1u << 7) | (1u << 10) | ((NC / 8) << 17) | ((128 / 16) << 24);
        const unsigned cb = diag ? base + c0 * kOzK * 2 : base + kOzColsAt;
        const unsigned col_step = diag ? 2 * kOzSliceBytes : kOzSliceBytes;
        bool got = true, issued = false;
        for (int d = 2; d <= 8 && got; ++d) {  // weight 2^-8d: slices up to d - 1
            got = oz_wait(there + 8 * (d - 2), polls);
            issued = issued || got;
            for (int i = max(1, d - kOzSlices); i <= min(kOzSlices, d - 1) && got; ++i)
#pragma unroll
                for (int k = 0; k < kOzK / 16; ++k) {
                    const unsigned long long ad = oz_operand(base + (i - 1) * 2 * kOzSliceBytes + 32 * k);
                    const unsigned long long bd = oz_operand(cb + (d - i - 1) * col_step + 32 * k);
                    const unsigned more = i > max(1, d - kOzSlices) || k > 0;
                    asm volatile(
                        "{ .reg .pred p; setp.ne.u32 p, %4, 0;\n"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(tmem + (d - 2) * NC),
                        "l"(ad), "l"(bd), "r"(kShape), "r"(more)
                        : "memory");
                }
        }
        missed = !got;
        if (issued)
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(done)
                         : "memory");
        else
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(done) : "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(done) : "memory");
    }
    __syncwarp();
    const bool over = oz_wait(done), ok = __all_sync(0xffffffffu, over && !missed);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (int i = 0; !ok && tid == 0 && i < kOzSlices; ++i) oz_wait(there + 8 * i);  // no copy is under way at the end
    if (ok && __any_sync(0xffffffffu, cols > 0)) {
#pragma unroll
        for (int q = 0; q < kWarpCols; q += 8) {
            unsigned u[7][8];
            const unsigned at = tmem + ((unsigned)(32 * (warp & 3)) << 16) + cw + q;
#pragma unroll
            for (int d = 0; d < 7; ++d) oz_load_acc(at + d * NC, u[d]);
            oz_wait_acc(u);
            auto G = [&](int d, int k) { return __uint_as_float(u[d - 2][k]); };
            auto Gi = [&](int d, int k) { return __float2int_rn(G(d, k)); };
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int top = Gi(2, k) * 256 + Gi(3, k);
                const long long L = (long long)top * (1 << 24) + (long long)Gi(4, k) * (1 << 16) +
                                    (long long)Gi(5, k) * (1 << 8) + Gi(6, k);
                const float T = fmaf(G(8, k), 0.00390625f, G(7, k));
                if (q + k < cols) a[q + k] = acc[q + k] + oz_value(L, T, xr + xC[cw + q + k]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    return ok;
}

}  // namespace sfmba
