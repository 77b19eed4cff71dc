// Partial-pivoting LU by rows (the dense solver's and the batch's fallback).
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace sfmba {

// Partial-pivoting LU of one or several systems in one cooperative launch with
// one grid barrier per column (k_dense.cu, k_batched.cu). The rows of all
// systems are numbered one system after another and dealt to the blocks in
// runs. No row is swapped: every block keeps the order of the rows of its
// systems (order[p]: the row at place p), finds the pivot of column k among the
// places from k on by itself (the first maximum |a|) and updates its own rows
// that are not pivots yet, a row a warp. A zero column is skipped, and with it
// the row at its place. A row's multiplier is stored after the next barrier:
// other blocks may still be searching the column it replaces. Every entry sees
// the operations of the swapping column loop in the same order.
//
// Bound: the chain of a column (barrier, column, pivot, division, row), not
// bandwidth: with its solve 8.8 ms for 652 unknowns, against 12.2 with pivots,
// swaps and divisions by one block between two barriers (7.0 against 13.1 for
// the window of a batch that needed it).
struct LuRow {
    double l;   // multiplier to store ..
    int lcol;   // .. in this column, -1: none
    int active; // not a pivot yet
};
struct LuWindow {
    int f, n, order, first, lo, hi;  // its order's place in shared memory; owned rows lo..hi, from the block's first on
};

inline size_t lu_coop_smem(long long rows, int max_n) {
    return (size_t)rows * (sizeof(LuRow) + sizeof(int)) + (size_t)(rows + 2) * sizeof(LuWindow) +
           (size_t)2 * max_n * sizeof(int);
}

struct LuSystem {
    double *A;  // [n][n]
    int *perm;  // receives the order
    int n;
};

// at(f): system f of nf; max_n: the largest; max_rows: rows a block may own.
// 256 threads, lu_coop_smem bytes of dynamic shared memory.
template <typename At>
__device__ __forceinline__ void lu_columns(int nf, int max_n, int max_rows, At at) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) unsigned char lu_sm[];
    LuRow *rows = reinterpret_cast<LuRow *>(lu_sm);
    LuWindow *wins = reinterpret_cast<LuWindow *>(rows + max_rows);
    int *orders = reinterpret_cast<int *>(wins + max_rows + 2);
    __shared__ unsigned long long best_key[8];
    __shared__ int best_at[8], nwin;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        long long total = 0;
        for (int f = 0; f < nf; ++f) total += at(f).n;
        const long long per = (total + gridDim.x - 1) / gridDim.x;
        const long long lo = min(total, per * blockIdx.x), hi = min(total, lo + per);
        int c = 0, place = 0;
        long long base = 0;
        for (int f = 0; f < nf && base < hi; ++f) {
            const int n = at(f).n;
            if (n > 0 && base + n > lo) {
                const int a = (int)(max(lo, base) - base), e = (int)(min(hi, base + n) - base);
                wins[c++] = {f, n, place, (int)(max(lo, base) - lo), a, e};
                place += n;
            }
            base += n;
        }
        nwin = c;
    }
    __syncthreads();
    for (int i = 0; i < nwin; ++i) {
        const LuWindow W = wins[i];
        for (int p = tid; p < W.n; p += blockDim.x) orders[W.order + p] = p;
        for (int r = W.lo + tid; r < W.hi; r += blockDim.x) rows[W.first + r - W.lo] = {0.0, -1, 1};
    }
    __syncthreads();
    for (int k = 0; k <= max_n; ++k) {  // the last turn stores the last multipliers
        for (int i = 0; i < nwin; ++i) {
            const LuWindow W = wins[i];
            if (k > W.n) continue;
            double *A = at(W.f).A;
            LuRow *mine = rows + W.first - W.lo;
            int *order = orders + W.order;
            for (int r = W.lo + tid; r < W.hi; r += blockDim.x)
                if (mine[r].lcol >= 0) {
                    A[(size_t)r * W.n + mine[r].lcol] = mine[r].l;
                    mine[r].lcol = -1;
                }
            if (k == W.n) continue;
            // The first maximum: |a| as an integer, 0 for NaN, which no comparison prefers.
            unsigned long long key = 0;
            int place = k;
            for (int p = k + tid; p < W.n; p += blockDim.x) {
                const double v = fabs(A[(size_t)order[p] * W.n + k]);
                const unsigned long long b = (unsigned long long)__double_as_longlong(v);
                const unsigned long long kv = b <= 0x7ff0000000000000ULL ? b + 1 : 0;
                if (kv > key) { key = kv; place = p; }
            }
            auto take = [&](unsigned long long ok, int oa) {
                if (ok > key || (ok == key && oa < place)) { key = ok; place = oa; }
            };
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                take(__shfl_xor_sync(0xffffffffu, key, off), __shfl_xor_sync(0xffffffffu, place, off));
            if (lane == 0) {
                best_key[warp] = key;
                best_at[warp] = place;
            }
            __syncthreads();  // also: the order as the last column left it, its readers done
            key = best_key[0];
            place = best_at[0];
#pragma unroll
            for (int q = 1; q < 8; ++q) take(best_key[q], best_at[q]);
            const int pr = order[place];
            const double *P = A + (size_t)pr * W.n;
            const double diag = P[k];
            const int kr = order[k];
            __syncthreads();
            if (diag == 0.0) {  // the column is skipped, and with it the row at its place
                if (tid == 0 && kr >= W.lo && kr < W.hi) mine[kr].active = 0;
            } else {
                if (tid == 0) {
                    order[place] = kr;
                    order[k] = pr;
                }
                for (int r = W.lo + warp; r < W.hi; r += 8) {
                    if (r == pr) {
                        if (lane == 0) mine[r].active = 0;
                        continue;
                    }
                    if (!mine[r].active) continue;
                    double *row = A + (size_t)r * W.n;
                    const double l = row[k] / diag;
                    if (lane == 0) {
                        mine[r].l = l;
                        mine[r].lcol = k;
                    }
                    // Eight loads of either row in flight (the compiler must
                    // assume that a store changes the next load).
                    for (int c0 = k + 1 + lane; c0 < W.n; c0 += 256) {
                        double u[8], v[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int c = c0 + 32 * q;
                            u[q] = c < W.n ? P[c] : 0.0;
                            v[q] = c < W.n ? row[c] : 0.0;
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int c = c0 + 32 * q;
                            if (c < W.n) row[c] = fma(-l, u[q], v[q]);
                        }
                    }
                }
            }
            __syncthreads();
        }
        grid.sync();
    }
    for (int i = 0; i < nwin; ++i) {
        const LuWindow W = wins[i];
        if (W.lo == 0)
            for (int p = tid; p < W.n; p += blockDim.x) at(W.f).perm[p] = orders[W.order + p];
    }
}

}  // namespace sfmba
