// Device bodies of the blocked Cholesky factorisations (k_dense.cu,
// k_batched.cu): the factor and inverse of a 64 x 64 diagonal block, the
// panel below it and the FP64 trailing update. Every entry of the factor sees
// its operations in one fixed order (the columns of a block ascending, one
// fused multiply-add per term), whatever the tile or the thread that does it.
//
// GB300 runs FP64 at half a lane per clock and SM sub-partition: a warp-wide
// FP64 instruction occupies its sub-partition for 65 cycles however many
// lanes are active, with 72 cycles to its result (one warp, clock64). Integer
// instructions, shared memory and barriers (36 cycles for 256 threads) are
// cheap beside that.
#pragma once

#include "common.cuh"

namespace sfmba {

constexpr int kBlkLD = 65;           // row stride of the 64-wide shared tiles

// Cholesky factor and factor inverse of one diagonal block of nb <= 64
// columns, by a cluster of three 256-thread blocks on as many SMs.
//
// Block 0 factors the leading 32 columns of the leading 32 rows and sends each
// column to block 1, which takes rows 32.. through the same steps a little
// behind and then factors its own 32 x 32 block. Block 2 carries the inverse
// along from the columns that both send. The chain of pivots (root,
// reciprocal, next pivot) so has little FP64 work beside it.
//
// A factoring block: warp 0 runs the chain. It scales what step j publishes by
// 1 / L_jj, forms pivot j + 1 from its own copy of L[j+1][j], and takes that
// pivot's root and reciprocal while the row warps apply step j. The six row
// warps sit on the three other sub-partitions and own the lower triangle in
// patches of 4 rows x 8 columns, a register per lane and patch. Warp 4, which
// would share warp 0's FP64 pipe, stores the columns and sends them
// (st.async, counted by one barrier per column at the receiver). Two named
// barriers a step: warp 0 only arrives where the others wait for its column
// and waits where they only arrive.
//
// Bound: the pivot chain. 48 us for 64 columns, against 87 us with factor
// and inverse swept together by one block, 67 us with only the inverse on a
// second block (in the first half of the steps the row warps' FP64 issue
// exceeded the chain), 62 us with the inverse on block 0 after its half and
// 55 us with that and pivot_root.
struct CholBlock {
    double col[64 * 64];          // column j of L at 64 j, 1 / L_jj on the diagonal
    unsigned long long full[64];  // completes when what the others send of column j is there
    double v[32], raw[32], diag[32], root;
    int failed;
};
constexpr int kCholCluster = 3;

constexpr int kBlkPolls = 1 << 18;   // bound of every wait for a column
enum CholStatus { kCholOk = 0, kCholBadPivot = 1, kCholGaveUp = 2 };  // 2: a wait ran out
constexpr double kBlkFailed = -1.0;  // in place of 1 / L_jj: pivot j or one before it failed

// x < 0 for the marks and reciprocals above, on the integer pipe.
__device__ __forceinline__ bool is_failed(double x) { return __double_as_longlong(x) < 0; }
// x > 0, on the integer pipe.
__device__ __forceinline__ bool is_positive(double x) {
    const long long b = __double_as_longlong(x);
    return b > 0 && b <= 0x7ff0000000000000LL;
}
// Barrier `id` of the block's 256 threads: wait, or only arrive.
__device__ __forceinline__ void bar_sync(int id) {
    __syncwarp();
    asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id) {
    __syncwarp();
    asm volatile("bar.arrive %0, 256;" ::"r"(id) : "memory");
}
constexpr int kRowWarps = 6;

// Row warp 0..5 of this thread's warp, -1 for warps 0 and 4.
__device__ __forceinline__ int row_warp() {
    const int warp = threadIdx.x >> 5;
    return warp == 0 || warp == 4 ? -1 : warp < 4 ? warp - 1 : warp - 2;
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Another block's columns and barriers.
struct CholPeer {
    unsigned col, full;

    __device__ __forceinline__ CholPeer(const CholBlock &sm, unsigned rank) {
        const unsigned c = (unsigned)__cvta_generic_to_shared(sm.col), f = (unsigned)__cvta_generic_to_shared(sm.full);
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(col) : "r"(c), "r"(rank));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(full) : "r"(f), "r"(rank));
    }
    // Entry i of column j; its 8 bytes count on the column's barrier.
    __device__ __forceinline__ void send(int j, int i, double x) const {
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                         col + 8u * (64 * j + i)),
                     "l"(__double_as_longlong(x)), "r"(full + 8u * j)
                     : "memory");
    }
};

// A block's barriers, before the cluster's first barrier: one arrival and the
// bytes of a column each (first: of columns 0 .. 31).
__device__ __forceinline__ void chol_expect(CholBlock &sm, int first, int second) {
    if (threadIdx.x < 64) {
        const unsigned bar = (unsigned)__cvta_generic_to_shared(&sm.full[threadIdx.x]);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(threadIdx.x < 32 ? first : second)
                     : "memory");
    }
}

__device__ __forceinline__ bool chol_wait(const CholBlock &sm, int j, int polls) {
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&sm.full[j]);
    for (int k = 0; k < polls; ++k) {
        unsigned ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(bar)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// sqrt(d) and 1 / sqrt(d), each the rounded quotient that sqrt and the division
// give, in integer arithmetic: 480 cycles for the pair against 935 in FP64
// (one warp, clock64).
//
// With d = m 4^k, m in [1, 4) and M = m 2^52 an integer: the rounded root
// of m is S 2^-52 for the integer S with S^2 - S < M 2^52 <= S^2 + S (never a
// tie), and its rounded reciprocal R 2^-53 for the integer R with
// |2^106 - 2 R S| < S (R = 2^53 for S = 2^52; never a tie otherwise). Y, a
// float reciprocal root y of m's leading bits after one step of third order in
// 61-bit fixed point, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - m y^2, is good to
// 2^-58, so that M Y is within a unit of S and Y within two of R, and both
// remainders, taken modulo 2^64, fit a word; the conditions settle the rest.
__device__ __forceinline__ void pivot_root(double d, double &root, double &recip) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(d), one = 1ULL << 52;
    const int ex = (int)(bits >> 52);
    if (ex == 0 || ex >= 2047) {  // subnormal, infinite, NaN or negative
        root = sqrt(d);
        recip = 1.0 / root;
        return;
    }
    const int k = (ex - 1023) >> 1, odd = (ex - 1023) & 1;  // m = 1.f or 2 * 1.f
    const unsigned long long f = bits & (one - 1), M = (f | one) << odd;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(((unsigned)(127 + odd) << 23) | (unsigned)(f >> 29))));
    y = fmaxf(y, 0.5f);  // in [0.5, 1 + 2^-22]
    const unsigned yb = __float_as_uint(y);
    const unsigned yi = ((yb & 0x7fffffu) | 0x800000u) << ((yb >> 23) - 126);              // y 2^24
    const long long e = (1LL << 61) - (long long)__umul64hi(M << 10, ((unsigned long long)yi * yi) << 15);  // e 2^61
    const long long e2 = (long long)(int)(e >> 20) * (int)(e >> 20) >> 21;                 // e^2 2^61
    const long long Y = ((long long)yi << 36) + ((((e >> 1) + ((3 * e2) >> 3)) >> 3) * (long long)yi >> 22);  // 2^60
    unsigned long long S = (__umul64hi(M << 10, (unsigned long long)Y << 3) + 256) >> 9;
    const long long r = (long long)((M << 52) - S * S);
    if (r > (long long)S) S += 1;
    else if (r <= -(long long)S) S -= 1;
    root = __longlong_as_double((long long)(S - one + ((unsigned long long)(1023 + k) << 52)));
    unsigned long long R = (unsigned long long)(Y + 64) >> 7;
    long long q = -(long long)(R * S);  // 2^105 - R S
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (2 * q > (long long)S) {
            R += 1;
            q -= (long long)S;
        } else if (2 * q < -(long long)S) {
            R -= 1;
            q += (long long)S;
        }
    }
    recip = __longlong_as_double((long long)(R - one + ((unsigned long long)(1022 - k) << 52)));
}

// The patches of 4 rows x 8 columns of an n x n lower triangle, n <= 32, that a
// row warp owns: patch p = 6 s + rw of those dealt column block by column
// block, block h holding the row groups 2 h .. G - 1.
constexpr int kTriPatches = 4;
struct TriPatches {
    double a[kTriPatches];
    int row[kTriPatches], col[kTriPatches], G, rw, last;

    __device__ __forceinline__ int start(int h) const { return h * (G - h + 1); }
    __device__ __forceinline__ int slot(int from) const {  // the first slot with p >= from
        return from <= rw ? 0 : (from - rw + kRowWarps - 1) / kRowWarps;
    }
    __device__ __forceinline__ TriPatches(const double *A, size_t ld, int n) : G((n + 3) >> 2), rw(row_warp()) {
        const int total = start((n + 7) >> 3), lane = threadIdx.x & 31;
        last = rw < 0 ? 0 : slot(total);
#pragma unroll
        for (int s = 0; s < kTriPatches; ++s) {
            const int p = kRowWarps * s + rw;
            int h = 0;
            while (h < 3 && start(h + 1) <= p) ++h;
            row[s] = s < last ? 4 * (2 * h + p - start(h)) + (lane >> 3) : 32;
            col[s] = 8 * h + (lane & 7);
            a[s] = row[s] < n && col[s] <= row[s] ? A[row[s] * ld + col[s]] : 0.0;
        }
    }
    // a -= v v^T on the patches of the column blocks from h on (jumps: a
    // predicated FP64 instruction would cost its 65 cycles all the same).
    __device__ __forceinline__ void apply(const double *v, int h) {
        if (rw < 0) return;
        switch (slot(start(h))) {
#define SFMBA_PATCH(s)                           \
    case s:                                      \
        if (s >= last) break;                    \
        a[s] = fma(-v[row[s]], v[col[s]], a[s]); \
        [[fallthrough]];
            SFMBA_PATCH(0)
            SFMBA_PATCH(1)
            SFMBA_PATCH(2)
            SFMBA_PATCH(3)
#undef SFMBA_PATCH
        default: break;
        }
    }
};

// Rows and columns r0 .. r0 + n - 1 (n <= 32) of the block, from the patches
// that hold them with every column before r0 applied. Column j goes to A (its
// entry (r0, r0)) and, through send(j, entry), to other blocks. Returns how
// many pivots were > 0 before one was not (0, negative and NaN all fail, as
// nalgebra's Cholesky::new).
template <typename Send>
__device__ __forceinline__ int chol_factor_half(double *A, size_t ld, int n, TriPatches &P, CholBlock &sm, Send send) {
    constexpr int kColumn = 1, kApplied = 2;  // column j is there; step j is applied
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 32) sm.raw[tid] = tid == 0 ? 1.0 : 0.0;
    if (tid == 0) sm.failed = 0;
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kTriPatches; ++s) {
        if (P.row[s] < 32 && P.row[s] > 0 && P.col[s] == 0) sm.raw[P.row[s]] = P.a[s];
        if (P.row[s] == P.col[s]) sm.diag[P.row[s]] = P.a[s];
    }
    __syncthreads();
    if (warp == 0) {
        double next = sm.diag[0];
        for (int j = 0; j < n; ++j) {
            const int n1 = j + 1;
            double sd, inv;
            const bool ok = is_positive(next);
            if (ok) pivot_root(next, sd, inv);
            if (j > 0) bar_sync(kApplied);
            if (!ok) {
                if (lane == 0) sm.failed = n1;
                bar_arrive(kColumn);
                break;
            }
            // v = raw / L_jj: column j of L below j, 1 / L_jj at j.
            const double dn = sm.diag[n1 & 31], v = sm.raw[lane] * inv;
            const double l = __shfl_sync(0xffffffffu, v, n1 & 31);
            sm.v[lane] = v;
            if (lane == 0) sm.root = sd;
            bar_arrive(kColumn);
            next = fma(-l, l, dn);
        }
    } else {
        for (int j = 0; j < n; ++j) {
            const int n1 = j + 1;
            bar_sync(kColumn);
            if (sm.failed) break;
            if (warp == 4) {
                const double v = sm.v[lane], sd = sm.root;
                send(j, lane, v);
                if (lane >= j && lane < n) A[lane * ld + j] = lane == j ? sd : v;
            } else if (n1 < n) {
                P.apply(sm.v, n1 >> 3);
                // What the next step scales, column j + 1 below its pivot, and the
                // diagonal entry of the pivot after it.
#pragma unroll
                for (int s = 0; s < kTriPatches; ++s) {
                    if (P.col[s] == n1 && P.row[s] > n1 && P.row[s] < 32) sm.raw[P.row[s]] = P.a[s];
                    if (P.row[s] == j + 2 && P.col[s] == j + 2) sm.diag[(j + 2) & 31] = P.a[s];
                }
                if (P.rw == 0 && lane == 0) sm.raw[n1] = 1.0;
            }
            if (n1 < n) bar_arrive(kApplied);
        }
    }
    __syncthreads();
    return sm.failed ? sm.failed - 1 : n;
}

// Block 1: rows 32.. of the block through block 0's 32 columns as they arrive,
// then their own factor. A wait that gives up ends it as a failed pivot does:
// block 2 gets a mark for every column, and what block 0 still sends is awaited.
__device__ __forceinline__ int chol_rows_behind(double *A, size_t ld, int nb, const CholPeer &inverse, CholBlock &sm,
                                                int polls) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = nb - 32;
    double *A2 = A + 32 * ld + 32;
    TriPatches P(A2, ld, n);
    // Left of them, slot s of warp w is the patch of rows 32 + 4 w .. and columns 8 s ..
    const int r = 4 * warp + (lane >> 3), c = lane & 7;
    double b[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) b[s] = r < n ? A[(32 + r) * ld + 8 * s + c] : 0.0;
    if (tid < 32) sm.raw[tid] = tid < n ? A[(32 + tid) * ld] : 0.0;
    if (tid == 0) sm.failed = 0;
    cluster_sync();
    for (int j = 0; j < 32; ++j) {
        const int n1 = j + 1;
        const double *L = sm.col + 64 * j;
        if (warp == 0) {
            const bool ok = __all_sync(0xffffffffu, chol_wait(sm, j, polls));
            const double inv = ok ? L[j] : kBlkFailed;
            if (is_failed(inv)) {
                if (lane == 0) sm.failed = ok ? kCholBadPivot : kCholGaveUp;
                for (int i = j; i < nb; ++i) inverse.send(i, 32 + lane, kBlkFailed);
                for (int i = j; i < 32; ++i) chol_wait(sm, i, kBlkPolls);  // nothing is under way when the block leaves
            } else {
                const double v = sm.raw[lane] * inv;
                sm.v[lane] = v;
                inverse.send(j, 32 + lane, v);
                if (lane < n) A[(32 + lane) * ld + j] = v;
            }
        }
        __syncthreads();
        if (sm.failed) return sm.failed;
        const double v = -sm.v[r];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (s < (n1 >> 3)) continue;
            b[s] = fma(v, L[8 * s + c], b[s]);
            if (8 * s + c == n1) sm.raw[r] = b[s];
        }
        P.apply(sm.v, 0);
        __syncthreads();
    }
    const int done = chol_factor_half(A2, ld, n, P, sm, [&](int j, int i, double x) { inverse.send(32 + j, 32 + i, x); });
    for (int i = done; warp == 4 && i < n; ++i) inverse.send(32 + i, 32 + lane, kBlkFailed);
    return done == n ? kCholOk : kCholBadPivot;
}

// Block 2: X = L^-1 ([64][64], zeros above the diagonal and outside nb), from
// the columns of L as they arrive. Warp w owns columns 4 w .. 4 w + 3 of
// either half, a lane the rows congruent to lane / 4 mod 8 of one of them:
// columns of an inverse do not depend on one another, so the warps meet
// nowhere. Returns a CholStatus, of the thread's warp.
__device__ __forceinline__ int chol_block_inverse(double *X, int nb, CholBlock &sm, int polls) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rs = lane >> 2;
    const int c = 4 * w + (lane & 3), d = 32 + c;
    double a[8], b[4];  // rows 8 s + rs of column c, rows 32 + 8 s + rs of column d: minus the sums so far
#pragma unroll
    for (int s = 0; s < 8; ++s) a[s] = 0.0;
#pragma unroll
    for (int s = 0; s < 4; ++s) b[s] = 0.0;
    bool ok = true;
    int status = kCholOk;
#pragma unroll
    for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = 8 * s + q;
            double x = 0.0, y = 0.0;
            if (ok && j < nb && j >= 4 * w) {
                ok = __all_sync(0xffffffffu, chol_wait(sm, j, polls));
                const double *L = sm.col + 64 * j;
                const double inv = ok ? L[j] : kBlkFailed;
                if (is_failed(inv)) {
                    status = ok ? kCholBadPivot : kCholGaveUp;
                    ok = false;
                }
                if (ok) {
                    x = (c == j ? 1.0 : a[s]) * inv;  // row j of X on the lanes of its residue
                    const double xb = __shfl_sync(0xffffffffu, x, 4 * q + (lane & 3));
#pragma unroll
                    for (int t = q == 7 ? s + 1 : s; t < 8; ++t) a[t] = fma(-L[8 * t + rs], xb, a[t]);
                    if (s >= 4 && j >= 32 + 4 * w) {
                        y = (d == j ? 1.0 : b[s & 3]) * inv;
                        const double yb = __shfl_sync(0xffffffffu, y, 4 * q + (lane & 3));
#pragma unroll
                        for (int t = q == 7 ? s + 1 : s; t < 8; ++t) b[t & 3] = fma(-L[8 * t + rs], yb, b[t & 3]);
                    }
                }
            }
            if (rs == q) {
                X[64 * j + c] = c <= j ? x : 0.0;
                X[64 * j + d] = d <= j ? y : 0.0;
            }
        }
    for (int j = 0; !ok && w == 0 && j < nb; ++j) chol_wait(sm, j, kBlkPolls);  // nothing is under way at the end
    return status;
}

// The diagonal block at A (row stride ld) by the blocks of a cluster: L below
// and on the diagonal, its inverse at X. *failed is set when it has none; A
// and X are then partly written. A wait of more than `polls` attempts gives up:
// it counts in *timeouts and sets *failed too. All blocks call it or none.
__device__ __forceinline__ void chol_block(double *A, size_t ld, int nb, double *X, CholBlock &sm, int *failed,
                                           int *timeouts, int polls) {
    const unsigned rank = cluster_rank();
    const CholPeer rows(sm, 1), inverse(sm, 2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool both = nb > 32;
    int status = kCholOk;
    chol_expect(sm, rank == 2 && both ? 512 : 256, 256);
    if (rank == 0) {
        const int n = min(32, nb);
        TriPatches P(A, ld, n);
        cluster_sync();
        auto send = [&](int j, int i, double x) {
            if (both) rows.send(j, i, x);
            inverse.send(j, i, x);
        };
        const int done = chol_factor_half(A, ld, n, P, sm, send);
        if (done < n) status = kCholBadPivot;
        for (int j = done; warp == 4 && j < n; ++j) send(j, lane, kBlkFailed);
    } else if (rank == 1 && both) {
        status = chol_rows_behind(A, ld, nb, inverse, sm, polls);
    } else {
        cluster_sync();
        if (rank == 2) status = chol_block_inverse(X, nb, sm, polls);
    }
    if (status != kCholOk && lane == 0) {
        *failed = 1;
        if (status == kCholGaveUp) atomicAdd(timeouts, 1);
    }
    cluster_sync();  // no block leaves while another sends to it
}

// Rows [r0, r0 + 8) (below row `end`) of the panel right of which the factor's
// columns k0.. are done: A[r, k-block] <- A[r, k-block] L_kk^-T, one warp per
// row of a 256-thread block. L: the matrix, row stride n; inv: L_kk^-1
// [64][64]; nb: columns of the block. Lane c takes column c and then column
// 63 - c, so that every lane runs the same 65 multiply-adds. Eight rows a
// block (4 us, FP64 pipe) instead of 32 (33 us): a panel of 600 rows reaches
// half of the SMs.
constexpr int kPanelRows = 8;
__device__ __forceinline__ void chol_panel_rows(double *L, int n, int k0, int nb, int r0, int end, const double *inv) {
    __shared__ double Li[64 * kBlkLD];
    __shared__ double R[kPanelRows][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = r0 + warp;
    for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) Li[(e >> 6) * kBlkLD + (e & 63)] = inv[e];
    double *row = L + (size_t)r * n + k0;
    if (r < end) {
        R[warp][lane] = lane < nb ? row[lane] : 0.0;
        R[warp][lane + 32] = lane + 32 < nb ? row[lane + 32] : 0.0;
    }
    __syncthreads();
    if (r >= end) return;
    double s = 0.0, first = 0.0;
    for (int k = 0; k < 65; ++k) {
        const bool second = k > lane;
        const int t = second ? k - lane - 1 : k, c = second ? 63 - lane : lane;
        if (k == lane + 1) {
            first = s;
            s = 0.0;
        }
        s = fma(R[warp][t], Li[c * kBlkLD + t], s);
    }
    if (lane < nb) row[lane] = first;
    if (63 - lane < nb) row[63 - lane] = s;
}

// A[ri.., rj..] -= P_i P_j^T for one TS x TS tile (mi x mj of it, the lower
// triangle only when ri == rj) of the trailing update of the 64 columns at
// k0, by 256 threads. The FP64 pipe bounds it at any tile size (65 cycles a
// warp instruction against a few for its two shared loads), so the tile is
// small to spread a short update over the SMs: 4, 16 and 66 us for a 16, 32
// and 64-wide tile on one SM.
template <int TS>
__device__ __forceinline__ void chol_update_tile(double *L, int n, int k0, int ri, int rj, int mi, int mj) {
    constexpr int E = TS / 16;
    __shared__ double Pi[TS * kBlkLD], Pj[TS * kBlkLD];
    for (int e = threadIdx.x; e < TS * 64; e += blockDim.x) {
        const int r = e >> 6, c = e & 63;
        Pi[r * kBlkLD + c] = r < mi ? L[(size_t)(ri + r) * n + k0 + c] : 0.0;
        Pj[r * kBlkLD + c] = r < mj ? L[(size_t)(rj + r) * n + k0 + c] : 0.0;
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[E][E];
#pragma unroll
    for (int a = 0; a < E; ++a)
#pragma unroll
        for (int b = 0; b < E; ++b) acc[a][b] = 0.0;
#pragma unroll 4
    for (int t = 0; t < 64; ++t) {
        double x[E], y[E];
#pragma unroll
        for (int a = 0; a < E; ++a) x[a] = Pi[(ty + 16 * a) * kBlkLD + t];
#pragma unroll
        for (int b = 0; b < E; ++b) y[b] = Pj[(tx + 16 * b) * kBlkLD + t];
#pragma unroll
        for (int a = 0; a < E; ++a)
#pragma unroll
            for (int b = 0; b < E; ++b) acc[a][b] = fma(x[a], y[b], acc[a][b]);
    }
#pragma unroll
    for (int a = 0; a < E; ++a) {
        const int r = ty + 16 * a;
        if (r >= mi) continue;
#pragma unroll
        for (int b = 0; b < E; ++b) {
            const int c = tx + 16 * b;
            if (c >= mj || (ri == rj && c > r)) continue;
            L[(size_t)(ri + r) * n + rj + c] -= acc[a][b];
        }
    }
}

// Tile width of the FP64 trailing update of `tiles` 64 x 64 tiles: 16 while
// that leaves at most four blocks per SM, 32 beyond.
inline int chol_tile(long long tiles) { return tiles <= 38 ? 16 : 32; }

}  // namespace sfmba
