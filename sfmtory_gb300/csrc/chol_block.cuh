// Device bodies of the blocked Cholesky factorisations (k_dense.cu,
// k_batched.cu): the factor and inverse of a 64 x 64 diagonal block, the
// panel below it and the FP64 trailing update. Every entry of the factor sees
// its operations in one fixed order (the columns of a block ascending, one
// fused multiply-add per term), whatever the tile or the thread that does it.
//
// GB300 runs FP64 at half a lane per clock and SM sub-partition: a warp-wide
// FP64 instruction occupies its sub-partition for 65 cycles however many
// lanes are active, with 72 cycles to its result; a square root with an
// addition takes 692 cycles, a reciprocal with an addition 449 (one warp,
// clock64). Shared memory and barriers (36 cycles for 256 threads) are cheap
// beside that.
#pragma once

#include "common.cuh"

namespace sfmba {

constexpr int kBlkLD = 65;           // row stride of the 64-wide shared tiles
constexpr int kBlkBuf = 194;         // scratch of chol_block_factor_invert (doubles)

// Cholesky factor and factor inverse of one diagonal block of nb <= 64
// columns by a 256-thread block.
//
// Warp 0 runs the chain of pivots: it scales what step j publishes by
// 1 / L_jj, forms pivot j + 1 from its own copy of L[j+1][j], and takes that
// pivot's square root and reciprocal while the row warps apply step j. Row
// i of the block holds the factor right of the current column and the
// inverse left of it: step j takes L[i][j] v from it, where v is column j of
// L below the pivot and row j of the inverse left of it, so factor and
// inverse come from one sweep of the same 64 steps. The six row warps sit on
// the three other sub-partitions (warp 4, which would share warp 0's FP64
// pipe, only keeps the barriers) and own the lower triangle in patches of
// 4 rows x 8 columns, a register per lane and patch, dealt in turn from the
// top: 72 warp instructions for the first step, fewer each time four rows are
// done (row by row it would be 95).
//
// Bound: the row warps' FP64 issue in the first third of the steps, the pivot
// chain (square root, reciprocal and three multiply-adds, ~1300 cycles) after
// it: 75 us for 64 columns and 14 us for 16, against 132 and 37 us with every
// warp in every step, both barriers inside the chain and a second sweep for
// the inverse.
//
// A: [64][kBlkLD] shared, lower triangle of the nb x nb block on entry, the
// factor on exit (below and on the diagonal). X: [64][kBlkLD] shared, L^-1 on
// exit (zeros above the diagonal and outside nb). buf: [kBlkBuf] shared.
// Returns false (and leaves A, X unspecified) if a pivot is not > 0 (0,
// negative and NaN all fail, as nalgebra's Cholesky::new). Every thread of
// the block must call it, after a barrier that follows the last write of A.
__device__ __forceinline__ bool chol_block_factor_invert(double *A, double *X, int nb, double *buf) {
    constexpr int kRowWarps = 6, kPatches = 12;  // patches of a row warp (72 in all)
    double *v = buf, *raw = buf + 64, *diag = buf + 128;
    int *failed = reinterpret_cast<int *>(buf + 192);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rw = warp == 0 || warp == 4 ? -1 : warp < 4 ? warp - 1 : warp - 2;  // row warp 0..5
    for (int e = tid; e < 64 * kBlkLD; e += blockDim.x) X[e] = 0.0;
    // Patch p = kRowWarps s + rw: patches in order of their rows; the two row
    // groups 2m and 2m + 1 have m + 1 patches each.
    double a[kPatches];
    int row[kPatches], col[kPatches];
    if (rw >= 0) {
#pragma unroll
        for (int s = 0; s < kPatches; ++s) {
            const int p = kRowWarps * s + rw;
            int m = 0;
            while ((m + 1) * (m + 2) <= p) ++m;
            const int q = p - m * (m + 1), g = q > m ? 1 : 0;  // group 2m + g, patch q - g (m + 1) of it
            row[s] = 4 * (2 * m + g) + (lane >> 3);
            col[s] = 8 * (q - g * (m + 1)) + (lane & 7);
            a[s] = row[s] < nb && col[s] <= row[s] ? A[row[s] * kBlkLD + col[s]] : 0.0;
        }
    }
    double sd = 0.0, inv = 0.0;
    if (tid < 64) {
        raw[tid] = tid == 0 ? 1.0 : tid < nb ? A[tid * kBlkLD] : 0.0;
        diag[tid] = tid < nb ? A[tid * kBlkLD + tid] : 0.0;
    }
    __syncthreads();  // before A is overwritten
    if (warp == 0) {
        const double d = diag[0];
        if (lane == 0) *failed = !(d > 0.0);
        sd = sqrt(d);
        inv = 1.0 / sd;
    }
    __syncthreads();
    if (*failed) return false;
    for (int j = 0; j < nb; ++j) {
        const int n1 = j + 1;
        double next = 0.0, v0 = 0.0, v1 = 0.0;  // the next pivot; this lane's entries of v
        if (warp == 0) {
            // v = raw / L_jj: column j of L below j, row j of the inverse up to j.
            const double r0 = raw[lane], r1 = raw[lane + 32], dn = diag[n1 & 63];
            double l;
            if (n1 < 32) {
                v0 = r0 * inv;
                v1 = r1 * inv;
                l = __shfl_sync(0xffffffffu, v0, n1);
            } else {
                v1 = r1 * inv;
                v0 = r0 * inv;
                l = __shfl_sync(0xffffffffu, v1, n1 & 31);
            }
            next = fma(-l, l, dn);
            v[lane] = v0;
            v[lane + 32] = v1;
        }
        __syncthreads();
        if (warp == 0) {
            if (lane <= j) X[j * kBlkLD + lane] = v0;
            else if (lane < nb) A[lane * kBlkLD + j] = v0;
            if (lane + 32 <= j) X[j * kBlkLD + lane + 32] = v1;
            else if (lane + 32 < nb) A[(lane + 32) * kBlkLD + j] = v1;
            if (lane == 0) A[j * kBlkLD + j] = sd;
        }
        if (n1 == nb) break;
        if (warp == 0) {
            if (lane == 0 && !(next > 0.0)) *failed = 1;
            sd = sqrt(next);
            inv = 1.0 / sd;
        } else if (rw >= 0) {
            // The patches with a row below j: those from `first` on, up to the
            // block's last row (jumps: a predicated FP64 instruction would cost
            // its 65 cycles all the same).
            const int g0 = n1 >> 2, g1 = (nb - 1) >> 2;
            auto start = [](int g) { return g & 1 ? ((g + 1) >> 1) * ((g + 1) >> 1) : (g >> 1) * ((g >> 1) + 1); };
            const int p0 = start(g0), p1 = start(g1 + 1);
            const int first = p0 <= rw ? 0 : (p0 - rw + kRowWarps - 1) / kRowWarps;
            const int last = p1 <= rw ? 0 : (p1 - rw + kRowWarps - 1) / kRowWarps;
            switch (first) {
#define SFMBA_PATCH(s)               \
    case s:                          \
        if (s >= last) break;        \
        a[s] = fma(-v[row[s]], v[col[s]], col[s] == j ? 0.0 : a[s]); /* the inverse's column j starts from 0 */ \
        [[fallthrough]];
                SFMBA_PATCH(0)
                SFMBA_PATCH(1)
                SFMBA_PATCH(2)
                SFMBA_PATCH(3)
                SFMBA_PATCH(4)
                SFMBA_PATCH(5)
                SFMBA_PATCH(6)
                SFMBA_PATCH(7)
                SFMBA_PATCH(8)
                SFMBA_PATCH(9)
                SFMBA_PATCH(10)
                SFMBA_PATCH(11)
#undef SFMBA_PATCH
            default: break;
            }
            // What the next step scales: column j + 1 below its pivot, row j + 1 of
            // the inverse; and the diagonal entry of the pivot after it.
#pragma unroll
            for (int s = 0; s < kPatches; ++s) {
                const bool in_col = col[s] == n1 && row[s] > n1, in_row = row[s] == n1 && col[s] <= j;
                if (in_col || in_row) raw[in_col ? row[s] : col[s]] = a[s];
                if (row[s] == j + 2 && col[s] == j + 2) diag[(j + 2) & 63] = a[s];
            }
            if (rw == 0 && lane == 0) raw[n1] = 1.0;
        }
        __syncthreads();
        if (*failed) return false;
    }
    __syncthreads();
    return true;
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
