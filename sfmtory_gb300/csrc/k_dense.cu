// Dense reduced camera system:
//   * Schur reduction S_ij = [i==j] H_i - sum_p E_ip C_p^-1 E_jp^T, one warp
//     per image pair (FP32) or per chunk of its pairs (FP64, then a sum of the
//     chunks in order), walking the pair list grouped by image pair (the
//     visibility-sorted order), so no global atomics are used (reference:
//     lib.rs:114-211, :981-1043);
//   * fold of the image-level system onto the reference's slot order with
//     damping, per-parameter masks and symmetrisation (lib.rs:918-956,
//     :1051-1074);
//   * blocked right-looking FP64 Cholesky (64-wide panels) with triangular
//     solves and one FP64 refinement step, and a partial-pivoting LU
//     fallback (lib.rs:1081-1094). On the mixed path the trailing updates
//     run on the BF16 tensor cores by error-free splitting (ozaki.cuh), to
//     FP64 accuracy; the plain FP64 path keeps FP64 fused multiply-adds.
#include <cooperative_groups.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <type_traits>

#include "chol_block.cuh"
#include "kernels.cuh"
#include "lu_rows.cuh"
#include "ozaki.cuh"
#include "schur.cuh"

namespace sfmba {

namespace {

constexpr int kSchurWarps = 4;

// The FP32 reduction, one warp per image pair.
template <int D>
__global__ void __launch_bounds__(32 * kSchurWarps)
    k_schur_pairs(const float *__restrict__ rec, const int2 *__restrict__ pairs,
                  const int *__restrict__ group_start, const int2 *__restrict__ group_ij,
                  const int *__restrict__ group_order, int ngroups,
                  const int *__restrict__ ob_pt, const float *__restrict__ pt_Cinv,
                  const unsigned char *__restrict__ pt_ok, const double *__restrict__ img_H, int nID,
                  double *__restrict__ S_img) {
    constexpr int W = kSchurWarps;
    using Tile = SchurTile<float, D>;
    __shared__ float sA[W][32][Tile::LDS];
    __shared__ float sP[W][32][Tile::LDS];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x * W + wl >= ngroups) return;
    const int g = group_order[blockIdx.x * W + wl];
    const int2 ij = group_ij[g];
    double out[Tile::RH][Tile::CQ];
    schur_group<float, D>(rec, pairs, group_start[g], group_start[g + 1], ob_pt, pt_Cinv, pt_ok, sA[wl], sP[wl],
                          lane, out);
    if (lane >= Tile::LS) return;
    const int i = ij.x, j = ij.y;
    const int r0 = (lane >> 2) * Tile::RH, c0 = (lane & 3) * Tile::CQ;
#pragma unroll
    for (int a = 0; a < Tile::RH; ++a)
#pragma unroll
        for (int b = 0; b < Tile::CQ; ++b) {
            const int r = r0 + a, c = c0 + b;
            if (r >= D || c >= D) continue;
            const double v = out[a][b];
            if (i == j) {
                S_img[(size_t)(i * D + r) * nID + i * D + c] = img_H[(size_t)i * D * D + r * D + c] + v;
            } else {
                S_img[(size_t)(i * D + r) * nID + j * D + c] = v;
                S_img[(size_t)(j * D + c) * nID + i * D + r] = v;
            }
        }
}

// Chunks of each group, and its partial blocks: its chunks if it has several.
// Groups are taken by decreasing pair count (t: a group's place in that order),
// so that the chunks are launched with the shortest last.
__global__ void k_schur_count_chunks(const int *group_start, const int *group_order, int ngroups, int chunk,
                                     int *chunks, int *parts) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > ngroups) return;
    const int g = t < ngroups ? group_order[t] : 0;
    const int c = t < ngroups ? (group_start[g + 1] - group_start[g] + chunk - 1) / chunk : 0;
    chunks[t] = c;
    parts[t] = c > 1 ? c : 0;
}

// Chunks as {first pair, end, group, partial block or -1 for a whole group}.
__global__ void k_schur_list_chunks(const int *group_start, const int *group_order, int ngroups, int chunk,
                                    const int *chunk_off, const int *part_off, int4 *chunks) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ngroups) return;
    const int g = group_order[t], e = group_start[g + 1], c0 = chunk_off[t], c1 = chunk_off[t + 1];
    int s = group_start[g];
    for (int c = c0; c < c1; ++c, s += chunk)
        chunks[c] = make_int4(s, min(s + chunk, e), g, c1 - c0 == 1 ? -1 : part_off[t] + c - c0);
}

template <int D>
__device__ __forceinline__ void store_schur(int i, int j, int r, int c, double v, const double *img_H, int nID,
                                            double *S_img) {
    if (i == j) {
        S_img[(size_t)(i * D + r) * nID + i * D + c] = img_H[(size_t)i * D * D + r * D + c] + v;
    } else {
        S_img[(size_t)(i * D + r) * nID + j * D + c] = v;
        S_img[(size_t)(j * D + c) * nID + i * D + r] = v;
    }
}

// The FP64 reduction, one warp per chunk of a group's pairs: a warp's FP64
// instruction takes its sub-partition for 65 cycles, so one warp per group
// left a few long groups (an image with itself: all its observations) to run
// alone. 47 OPENCV images, 120 000 observations: 0.59 against 1.71
// ms; 16 images that see all of 2000 points: 0.21 against 0.80 ms; 500 images
// of 240 observations, 4500 groups: 0.73 either way. The FP32 form keeps one
// warp per group: its compensated sum over a group's rounds has one order.
template <int D>
__global__ void __launch_bounds__(64)
    k_schur_chunks(const double *__restrict__ rec, const int2 *__restrict__ pairs,
                   const int2 *__restrict__ group_ij, const int *__restrict__ nchunks,
                   const int4 *__restrict__ chunks, const int *__restrict__ ob_pt, const double *__restrict__ pt_Cinv, const unsigned char *__restrict__ pt_ok,
                   const double *__restrict__ img_H, int nID, double *__restrict__ part,
                   double *__restrict__ S_img) {
    using Tile = SchurTile<double, D>;
    __shared__ double sA[2][32][Tile::LDS];
    __shared__ double sP[2][32][Tile::LDS];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 2 + wl;
    if (c >= *nchunks) return;
    const int4 ch = chunks[c];
    double out[Tile::RH][Tile::CQ];
    schur_group<double, D>(rec, pairs, ch.x, ch.y, ob_pt, pt_Cinv, pt_ok, sA[wl], sP[wl], lane, out);
    if (lane >= Tile::LS) return;
    const bool whole = ch.w < 0;
    double *dst = part + (size_t)max(ch.w, 0) * D * D;
    const int2 ij = group_ij[ch.z];
    const int r0 = (lane >> 2) * Tile::RH, c0 = (lane & 3) * Tile::CQ;
#pragma unroll
    for (int a = 0; a < Tile::RH; ++a)
#pragma unroll
        for (int b = 0; b < Tile::CQ; ++b) {
            const int r = r0 + a, q = c0 + b;
            if (r >= D || q >= D) continue;
            if (whole) store_schur<D>(ij.x, ij.y, r, q, out[a][b], img_H, nID, S_img);
            else dst[r * D + q] = out[a][b];
        }
}

// Adds the partial blocks of the groups of several chunks (all among the first
// ngroups places), in order; one warp per group.
template <int D>
__global__ void __launch_bounds__(256) k_schur_combine(const int2 *group_ij, const int *group_order, int ngroups,
                                                       const int *part_off, const double *part, const double *img_H, int nID,
                                                       double *S_img) {
    const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t >= ngroups) return;
    const int a = part_off[t], b = part_off[t + 1];
    if (a == b) return;
    const int2 ij = group_ij[group_order[t]];
    for (int e = threadIdx.x & 31; e < D * D; e += 32) {
        double v = 0.0;
        for (int k = a; k < b; ++k) v += part[(size_t)k * D * D + e];
        store_schur<D>(ij.x, ij.y, e / D, e % D, v, img_H, nID, S_img);
    }
}

// S[a][b] = sym( sum_{u in pre(a), w in pre(b)} S_img[u][w] ) + [a==b] lambda diag(B)[a];
// masked parameters become identity rows/columns (lib.rs:1051-1070). With
// `list`, entries between two slots of more than kFoldList images each are
// left to k_fold_shared.
__global__ void k_fold(const double *__restrict__ S_img, int nID, const int *__restrict__ pre_start,
                       const int *__restrict__ pre, const unsigned char *__restrict__ masked,
                       const double *__restrict__ diagB, const LMState *__restrict__ st, int n, bool list,
                       double *__restrict__ S, double *__restrict__ L) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const int a = blockIdx.y;
    if (b >= n || a >= n) return;
    double v;
    if (masked[a] || masked[b]) {
        v = a == b ? 1.0 : 0.0;
    } else {
        double vab = 0.0, vba = 0.0;
        const int as = pre_start[a], ae = pre_start[a + 1], bs = pre_start[b], be = pre_start[b + 1];
        if (list && ae - as > kFoldList && be - bs > kFoldList) return;
        for (int x = as; x < ae; ++x)
            for (int y = bs; y < be; ++y) {
                vab += S_img[(size_t)pre[x] * nID + pre[y]];
                vba += S_img[(size_t)pre[y] * nID + pre[x]];
            }
        v = 0.5 * (vab + vba);
        if (a == b) v += diagB[a] * st->lambda;
    }
    S[(size_t)a * n + b] = v;
    L[(size_t)a * n + b] = v;
}

// Keys of the image pairs of both directions, grouped by the pair of shared
// cameras (shcam: an image's shared-camera index, -1 if it has its own); what
// is not such a pair, or a diagonal pair's second direction, gets a key past
// all others.
__global__ void k_fold_keys(const int2 *group_ij, int ngroups, const int *shcam, int nI, int nsh, uint64_t *keys) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    const int2 ij = group_ij[g];
    const int ci = shcam[ij.x], cj = shcam[ij.y];
    const bool both = ci >= 0 && cj >= 0;
    const uint64_t ab = (uint64_t)ci * nsh + cj, ba = (uint64_t)cj * nsh + ci;
    keys[2 * (size_t)g] = both ? (ab << 32) | ((uint64_t)ij.x * nI + ij.y) : ~(uint64_t)0;
    keys[2 * (size_t)g + 1] = both && ij.x != ij.y ? (ba << 32) | ((uint64_t)ij.y * nI + ij.x) : ~(uint64_t)0;
}

__device__ __forceinline__ int key_lower_bound(const uint64_t *keys, int n, uint64_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (keys[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Entries of k_fold between slots of cameras that many images share: the sum
// over image pairs runs over the pairs with a common point only (the blocks
// of all others are zero), in k_fold's order, so the result is k_fold's bit
// for bit. One warp per entry: the 32 lanes gather 256 blocks' terms ahead
// while lanes 0 and 1 add the previous 256 of S_ab and S_ba. A camera of a
// 300-image sequence (240 000 observations) took 20 ms a fold with one thread
// walking all 300 x 300 pairs per entry, and takes 0.6 ms now.
constexpr int kFoldBatch = 8;  // terms in flight per lane and direction
__global__ void __launch_bounds__(32) k_fold_shared(const double *__restrict__ S_img, int nID, int D, int nI, int nsh,
                                                    const uint64_t *__restrict__ keys, int nkeys,
                                                    const int *__restrict__ slots, int nslots,
                                                    const int *__restrict__ shcam,
                                                    const int *__restrict__ pre_start, const int *__restrict__ pre,
                                                    const unsigned char *__restrict__ masked,
                                                    const double *__restrict__ diagB, const LMState *__restrict__ st,
                                                    int n, double *__restrict__ S, double *__restrict__ L) {
    __shared__ double term[2][32 * kFoldBatch];
    const int a = slots[blockIdx.x / nslots], b = slots[blockIdx.x % nslots], lane = threadIdx.x;
    if (masked[a] || masked[b]) return;
    const int ua = pre[pre_start[a]], ub = pre[pre_start[b]];
    const int ra = ua % D, rb = ub % D;
    const uint64_t pair = (uint64_t)shcam[ua / D] * nsh + shcam[ub / D];
    const int k0 = key_lower_bound(keys, nkeys, pair << 32), k1 = key_lower_bound(keys, nkeys, (pair + 1) << 32);
    double tab[kFoldBatch], tba[kFoldBatch], sum = 0.0;
    auto gather = [&](int k) {
#pragma unroll
        for (int q = 0; q < kFoldBatch; ++q) {
            const int e = k + q * 32 + lane;
            tab[q] = tba[q] = 0.0;
            if (e < k1) {
                const unsigned xy = (unsigned)keys[e];
                const size_t u = (size_t)(xy / (unsigned)nI) * D + ra, w = (size_t)(xy % (unsigned)nI) * D + rb;
                tab[q] = S_img[u * nID + w];
                tba[q] = S_img[w * nID + u];
            }
        }
    };
    gather(k0);
    for (int k = k0; k < k1; k += 32 * kFoldBatch) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kFoldBatch; ++q) {
            term[0][q * 32 + lane] = tab[q];
            term[1][q * 32 + lane] = tba[q];
        }
        __syncwarp();
        gather(k + 32 * kFoldBatch);
        const int m = min(32 * kFoldBatch, k1 - k);
        if (lane < 2) {
#pragma unroll 8
            for (int q = 0; q < m; ++q) sum += term[lane][q];
        }
    }
    const double vba = __shfl_sync(0xffffffffu, sum, 1);
    if (lane == 0) {
        double v = 0.5 * (sum + vba);
        if (a == b) v += diagB[a] * st->lambda;
        S[(size_t)a * n + b] = v;
        L[(size_t)a * n + b] = v;
    }
}

__global__ void k_fold_rhs(const double *img_rhs, const int *pre_start, const int *pre,
                           const unsigned char *masked, int n, double *rhs) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    double v = 0.0;
    if (!masked[a])
        for (int x = pre_start[a]; x < pre_start[a + 1]; ++x) v += img_rhs[pre[x]];
    rhs[a] = v;
}

// ---------------------------------------------------------------- Cholesky

constexpr int NB = kCholNB;
constexpr int LD = NB + 1;

// Factor the diagonal block k0 (in place, lower) and write the inverse of its
// factor to Linv: one cluster of blocks. Sets state->factor_failed when a
// pivot is not > 0 (nalgebra Cholesky::new semantics: 0, negative and NaN all
// fail).
__global__ void __cluster_dims__(kCholCluster, 1, 1) __launch_bounds__(256)
    k_chol_diag(double *L, int n, int k0, double *Linv, LMState *st, int polls) {
    __shared__ CholBlock sm;
    if (st->factor_failed) return;
    chol_block(L + (size_t)k0 * n + k0, (size_t)n, min(NB, n - k0), Linv + (size_t)(k0 / NB) * NB * NB, sm,
               &st->factor_failed, &st->wait_timeouts, polls);
}

// Panel below the diagonal block k0.
__global__ void __launch_bounds__(256) k_chol_panel(double *L, int n, int k0, const double *Linv,
                                                     const LMState *st) {
    if (st->factor_failed) return;
    const int nb = min(NB, n - k0), r0 = k0 + nb + blockIdx.x * kPanelRows;
    if (r0 >= n) return;
    chol_panel_rows(L, n, k0, nb, r0, min(n, r0 + kPanelRows), Linv + (size_t)(k0 / NB) * NB * NB);
}

// Tile (ti, tj), tj <= ti, of block q of a trailing update launch. part 0:
// every lower tile; 1: the first tile column (tj = 0, the next diagonal
// block's column, updated first for the look-ahead); 2: the others.
__device__ __forceinline__ void trailing_tile(long long q, int part, int &ti, int &tj) {
    if (part == 1) {
        ti = (int)q;
        tj = 0;
        return;
    }
    int a = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while ((long long)(a + 1) * (a + 2) / 2 <= q) ++a;
    while ((long long)a * (a + 1) / 2 > q) --a;
    ti = a;
    tj = (int)(q - (long long)a * (a + 1) / 2);
    if (part == 2) {
        ++ti;
        ++tj;
    }
}

// Trailing update of the lower triangle right of panel k0 in TS x TS tiles:
// block q is tile q % S^2 (S = 64 / TS) of the 64 x 64 tile q / S^2.
template <int TS>
__global__ void __launch_bounds__(256) k_chol_update(double *L, int n, int k0, int part, const LMState *st) {
    constexpr int S = NB / TS;
    if (st->factor_failed) return;
    int ti, tj;
    trailing_tile(blockIdx.x / (S * S), part, ti, tj);
    const int sub = blockIdx.x % (S * S);
    const int ri = k0 + NB + ti * NB + (sub / S) * TS, rj = k0 + NB + tj * NB + (sub % S) * TS;
    if (ri >= n || rj > ri) return;
    chol_update_tile<TS>(L, n, k0, ri, rj, min(TS, n - ri), min(TS, n - rj));
}

// The column loop of k_lu_pivot / k_lu_update (below) in one cooperative
// launch (lu_rows.cuh); perm receives the order of the rows.
__global__ void __launch_bounds__(256) k_lu_coop(double *A, int n, int *perm, const LMState *st, int max_rows) {
    if (!st->factor_failed || st->solve_failed) return;
    lu_columns(1, n, max_rows, [&](int) { return LuSystem{A, perm, n}; });
}

// ------------------------------------------------ tensor-core trailing update
// Slices and exponents of the panel rows below the diagonal block k0 (one
// warp per row; ozaki.cuh). slices: a block of kOzBlockElems per 64 rows.
__global__ void __launch_bounds__(256) k_oz_split(const double *L, int n, int k0, __nv_bfloat16 *slices, int *exps,
                                                   const LMState *st) {
    if (st->factor_failed) return;
    const int nb = min(NB, n - k0);
    const int r = k0 + nb + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (r >= n) return;
    oz_split_row(L + (size_t)r * n + k0, nb, threadIdx.x & 31, slices + (size_t)(r / 64) * kOzBlockElems, r & 63,
                 exps + r);
}

// A[I, J] -= P_I P_J^T right of the panel, from the slices of k_oz_split
// (ozaki.cuh): block (p, q) has columns tj0 * 64 + q * NC .. of the trailing
// matrix and the pair of 64-row tiles 2 p and 2 p + 1 below their diagonal
// tile.
template <int NC>
__global__ void __launch_bounds__(kOzThreads, 1) k_oz_update(double *L, int n, int k0, int tj0,
                                                             const __nv_bfloat16 *slices, const int *exps,
                                                             LMState *st, int polls) {
    extern __shared__ unsigned char oz_sm[];
    // The next diagonal block may set the flag while this kernel runs: one
    // thread reads it, so that no warp waits for the tensor memory or the
    // barriers of another that left.
    if (__syncthreads_or(threadIdx.x == 0 && st->factor_failed)) return;
    const int c0 = (int)blockIdx.y * NC % 64;
    const int rj = k0 + NB + tj0 * 64 + (int)blockIdx.y * NC, ri = rj - c0 + (int)blockIdx.x * kOzRows;
    if (ri >= n || rj >= n) return;
    const bool ok = oz_tile_update<NC>(L + (size_t)ri * n + rj, (size_t)n, min(kOzRows, n - ri), min(NC, n - rj),
                                       blockIdx.x == 0, c0, slices + (size_t)(ri / 64) * kOzBlockElems,
                                       slices + (size_t)(rj / 64) * kOzBlockElems, exps + ri, exps + rj, oz_sm,
                                       polls);
    // Not factor_failed: the blocks of k_chol_diag read that beside this kernel and must agree.
    if (!ok && threadIdx.x == 0) atomicAdd(&st->wait_timeouts, 1);
}

// Both triangular solves of L L^T x = rhs as a flow of 64-wide blocks over one
// cooperative launch: block row K of the matrix belongs to thread block
// K mod gridDim.x, which subtracts the products with y_0, y_1, .. in order as
// they appear, multiplies by L_KK^-1 and publishes y_K; the backward sweep
// runs the same way from the last block up the columns. A block waits only
// for the block it needs next (a flag per block, read by one thread) instead
// of the whole grid, and the loads of L run a block ahead of the products.
//
// Sums keep one fixed order: forward, entry t of a row's 64 products belongs
// to lane t % 32 and the 32 lane sums meet in a butterfly (16, 8, 4, 2, 1),
// of which four threads per row each take the lanes of one residue mod 4;
// backward and with the block inverses, four interleaved sums over t % 4.
//
// Bound: the FP64 latency of the chain of block steps (products with the last
// block, inverse, publication). n = 4994: 0.68 ms for both sweeps, 3.2
// ms with a grid barrier per block step and every thread block forming the
// products with the inverse.
constexpr int kFlowPolls = 1 << 22;  // a few seconds; then the wait gives up

// Waits (thread 0) until block k is published; false, for every thread of the
// block, when the wait gave up (counted in LMState::wait_timeouts).
__device__ __forceinline__ bool flow_wait(const int *ready, int k, int *ok, LMState *st) {
    if (threadIdx.x == 0) {
        int v = 0;
        for (int i = 0; i < kFlowPolls && !v; ++i)
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(ready + k) : "memory");
        if (!v) atomicAdd(&st->wait_timeouts, 1);
        *ok = v;
    }
    __syncthreads();
    return *ok != 0;
}

// Publishes block k after every thread's stores to it.
__device__ __forceinline__ void flow_publish(int *ready, int k) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(ready + k), "r"(1) : "memory");
}

// ready: [2 * blocks] zero; y, x: [n].
__global__ void __launch_bounds__(256) k_trsv_flow(const double *L, int n, const double *Linv, const double *rhs,
                                                    double *y, double *x, int *ready, LMState *st) {
    __shared__ double Li[NB * LD], vk[NB], bk[NB], part[4][NB];
    __shared__ int ok;
    if (st->factor_failed) return;  // read-only here: every block takes the same branch
    const int nblk = (n + NB - 1) / NB, G = gridDim.x, tid = threadIdx.x;
    const int q = tid >> 6, c = tid & 63;  // (sum, entry) of the interleaved sums
    auto load_inverse = [&](int K) {
        for (int e = tid; e < NB * NB; e += blockDim.x) Li[(e >> 6) * LD + (e & 63)] = Linv[(size_t)K * NB * NB + e];
    };
    for (int K = blockIdx.x; K < nblk; K += G) {
        const int k0 = K * NB, nb = min(NB, n - k0), p = tid & 3, r = tid >> 2;
        const double *row = L + (size_t)(k0 + min(r, nb - 1)) * n + p;
        double acc = r < nb ? rhs[k0 + r] : 0.0, cur[16], nxt[16];
        load_inverse(K);
#pragma unroll
        for (int i = 0; i < 16; ++i) cur[i] = K > 0 ? row[4 * i] : 0.0;
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int i = 0; i < 16; ++i) nxt[i] = k + 1 < K ? row[(k + 1) * NB + 4 * i] : 0.0;
            if (!flow_wait(ready, k, &ok, st)) return;
            if (tid < NB) vk[tid] = __ldcg(y + k * NB + tid);
            __syncthreads();
            double d[8];  // lanes p, p + 4, .. p + 28
#pragma unroll
            for (int i = 0; i < 8; ++i)
                d[i] = fma(cur[i + 8], vk[4 * (i + 8) + p], fma(cur[i], vk[4 * i + p], 0.0));
#pragma unroll
            for (int h = 4; h > 0; h >>= 1)
#pragma unroll
                for (int i = 0; i < h; ++i) d[i] += d[i + h];
            double s = d[0];
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            acc -= s;
#pragma unroll
            for (int i = 0; i < 16; ++i) cur[i] = nxt[i];
            // the next flow_wait's barrier lies between these reads of vk and its next write
        }
        if (p == 0) bk[r] = acc;
        __syncthreads();
        double s = 0.0;  // y_K = L_KK^-1 b_K
        for (int t = q; t <= c; t += 4) s = fma(Li[c * LD + t], bk[t], s);
        part[q][c] = s;
        __syncthreads();
        if (tid < nb) y[k0 + tid] = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
        flow_publish(ready, K);
    }
    if ((int)blockIdx.x >= nblk) return;
    for (int K = blockIdx.x + (nblk - 1 - (int)blockIdx.x) / G * G; K >= 0; K -= G) {
        const int k0 = K * NB, nb = min(NB, n - k0);
        const double *col = L + k0 + min(c, nb - 1);
        double yv = c < nb ? y[k0 + c] : 0.0, cur[16], nxt[16];
        load_inverse(K);
        auto fetch = [&](int k, double (&v)[16]) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int t = k * NB + q + 4 * i;
                v[i] = k > K && t < n ? col[(size_t)t * n] : 0.0;
            }
        };
        fetch(nblk - 1, cur);
        for (int k = nblk - 1; k > K; --k) {
            fetch(k - 1, nxt);
            if (!flow_wait(ready + nblk, k, &ok, st)) return;
            if (tid < NB) vk[tid] = k * NB + tid < n ? __ldcg(x + k * NB + tid) : 0.0;
            __syncthreads();
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (k * NB + q + 4 * i < n) s = fma(cur[i], vk[q + 4 * i], s);
            part[q][c] = s;
            __syncthreads();
            yv -= (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
#pragma unroll
            for (int i = 0; i < 16; ++i) cur[i] = nxt[i];
        }
        if (q == 0) bk[c] = yv;
        __syncthreads();
        double s = 0.0;  // x_K = L_KK^-T y_K
        for (int t = c + q; t < nb; t += 4) s = fma(Li[t * LD + c], bk[t], s);
        part[q][c] = s;
        __syncthreads();
        if (tid < nb) x[k0 + tid] = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
        flow_publish(ready + nblk, K);
    }
}

// res = rhs - S x (one warp per row).
__global__ void k_residual(const double *S, int n, const double *x, const double *rhs, double *res,
                           const LMState *st) {
    if (st->factor_failed) return;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n) return;
    double s = 0.0;
    for (int c = lane; c < n; c += 32) s += S[(size_t)warp * n + c] * x[c];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) res[warp] = rhs[warp] - s;
}

__global__ void k_axpy_inplace(int n, const double *c, double *x, const LMState *st) {
    if (st->factor_failed) return;
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < n) x[a] += c[a];
}

// ---------------------------------------------------------------- LU fallback

// Column k: pivot on max |a| (first maximum), swap rows, scale the
// multipliers. A zero column is skipped (no swap, no elimination).
__global__ void __launch_bounds__(1024) k_lu_pivot(double *A, int n, int k, int *perm, const LMState *st) {
    __shared__ double bv[1024];
    __shared__ int bi[1024];
    if (!st->factor_failed || st->solve_failed) return;
    double best = -1.0;
    int besti = k;
    for (int r = k + threadIdx.x; r < n; r += blockDim.x) {
        const double v = fabs(A[(size_t)r * n + k]);
        if (v > best) { best = v; besti = r; }
    }
    bv[threadIdx.x] = best;
    bi[threadIdx.x] = besti;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            const double o = bv[threadIdx.x + w];
            const int oi = bi[threadIdx.x + w];
            if (o > bv[threadIdx.x] || (o == bv[threadIdx.x] && oi < bi[threadIdx.x])) {
                bv[threadIdx.x] = o;
                bi[threadIdx.x] = oi;
            }
        }
        __syncthreads();
    }
    const int piv = bi[0];
    const double diag = A[(size_t)piv * n + k];
    if (diag == 0.0) {
        if (threadIdx.x == 0) perm[k] = -1;  // zero column: skipped
        return;
    }
    if (piv != k)
        for (int c = threadIdx.x; c < n; c += blockDim.x) {
            const double t = A[(size_t)k * n + c];
            A[(size_t)k * n + c] = A[(size_t)piv * n + c];
            A[(size_t)piv * n + c] = t;
        }
    if (threadIdx.x == 0) perm[k] = piv;
    __syncthreads();
    for (int r = k + 1 + threadIdx.x; r < n; r += blockDim.x) A[(size_t)r * n + k] /= diag;
}

__global__ void k_lu_update(double *A, int n, int k, const int *perm, const LMState *st) {
    if (!st->factor_failed || st->solve_failed) return;
    if (perm[k] < 0) return;
    const int c = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int r = k + 1 + blockIdx.y;
    if (c >= n || r >= n) return;
    A[(size_t)r * n + c] -= A[(size_t)r * n + k] * A[(size_t)k * n + c];
}

// The rows' order (ordered: they lie where they were) or their swaps applied
// to rhs, then unit-lower and upper solves. A zero diagonal
// of U fails the solve (lambda then grows); success clears factor_failed so
// the back-substitution and trial kernels run.
// Sum of v over the 1024-thread block (warp sums, then the 32 warps' sums
// by warp 0), valid in every thread; two barriers.
__device__ __forceinline__ double block_sum_1024(double v, double *red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = (threadIdx.x & 31) < (blockDim.x >> 5) ? red[threadIdx.x & 31] : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    __syncthreads();  // red is reused by the next call
    return t;
}

__global__ void __launch_bounds__(1024) k_lu_solve(const double *A, int n, const int *perm,
                                                    const double *rhs, double *x, LMState *st, bool ordered) {
    __shared__ double red[32];
    __shared__ int bad;
    if (!st->factor_failed || st->solve_failed) return;
    if (threadIdx.x == 0) bad = 0;
    for (int a = threadIdx.x; a < n; a += blockDim.x) x[a] = rhs[ordered ? perm[a] : a];
    __syncthreads();
    if (threadIdx.x == 0 && !ordered)
        for (int k = 0; k < n; ++k)
            if (perm[k] >= 0 && perm[k] != k) {
                const double t = x[k];
                x[k] = x[perm[k]];
                x[perm[k]] = t;
            }
    __syncthreads();
    for (int i = 0; i < n; ++i) {
        const double *row = A + (size_t)(ordered ? perm[i] : i) * n;
        double s = 0.0;
        for (int k = threadIdx.x; k < i; k += blockDim.x) s += row[k] * x[k];
        s = block_sum_1024(s, red);
        if (threadIdx.x == 0) x[i] -= s;
        __syncthreads();
    }
    for (int i = n - 1; i >= 0; --i) {
        const double *row = A + (size_t)(ordered ? perm[i] : i) * n;
        double s = 0.0;
        for (int k = i + 1 + threadIdx.x; k < n; k += blockDim.x) s += row[k] * x[k];
        s = block_sum_1024(s, red);
        if (threadIdx.x == 0) {
            const double d = row[i];
            if (d == 0.0) bad = 1;
            else x[i] = (x[i] - s) / d;
        }
        __syncthreads();
        if (bad) break;
    }
    if (threadIdx.x == 0) {
        if (bad) st->solve_failed = 1;
        else st->factor_failed = 0;
    }
}

template <typename F>
void dispatch_D(int D, F &&f) {
    switch (D) {
    case 6: f(std::integral_constant<int, 6>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    case 11: f(std::integral_constant<int, 11>()); break;
    case 14: f(std::integral_constant<int, 14>()); break;
    default: throw Error(SFMBA_ERR_INTERNAL, "unsupported image block width");
    }
}


void set_smem_limits() {
    thread_local int done_dev = -1;
    int dev = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    if (done_dev == dev) return;
    allow_shared_memory(k_oz_update<32>);
    allow_shared_memory(k_oz_update<64>);
    allow_shared_memory(k_lu_coop);
    done_dev = dev;
}

}  // namespace

void launch_schur_pairs(const Bufs &b, cudaStream_t s) {
    if (b.ngroups == 0) return;
    dispatch_D(b.D, [&](auto dc) {
        constexpr int D = decltype(dc)::value;
        if (b.mixed)
            k_schur_pairs<D><<<div_up(b.ngroups, kSchurWarps), 32 * kSchurWarps, 0, s>>>(
                (const float *)b.rec, b.pairs, b.group_start, b.group_ij, b.group_order, b.ngroups, b.ob_pt,
                (const float *)b.pt_Cinv, b.pt_ok, b.img_H, b.nID, b.S_img);
        else {
            k_schur_chunks<D><<<div_up(b.schur_max_chunks, 2), 64, 0, s>>>(
                (const double *)b.rec, b.pairs, b.group_ij, b.schur_chunk_off + b.ngroups, b.schur_chunks, b.ob_pt,
                (const double *)b.pt_Cinv, b.pt_ok, b.img_H, b.nID, b.schur_part, b.S_img);
            SFMBA_LAUNCH_CHECK();
            // Groups of several chunks come first and have more pairs than a chunk each.
            const int several = (int)std::min<long long>(b.ngroups, b.npairs / (b.schur_chunk + 1));
            if (several > 0)
                k_schur_combine<D><<<div_up(several, 8), 256, 0, s>>>(b.group_ij, b.group_order, several,
                                                                      b.schur_part_off, b.schur_part, b.img_H, b.nID,
                                                                      b.S_img);
        }
    });
    SFMBA_LAUNCH_CHECK();
}

// Pairs per chunk: about eight chunks per SM, between one and eight rounds
// of 32 pairs (a chunk of one round is mostly staging; longer ones than eight
// leave a few SMs busy at the end).
int schur_chunk_pairs(long long npairs, int sms) {
    const long long c = (npairs / (8LL * sms) + 31) / 32 * 32;
    return (int)std::min<long long>(256, std::max<long long>(32, c));
}

// Chunks of the current groups (temp: CUB scratch). Where the groups alone are
// as many warps as the chunks aim at, none of two rounds of pairs is cut (60
// images of 30 points each that most of them see: 105 us cut at 32 pairs, 96 at
// 64 and more).
void launch_schur_chunks(Bufs &b, int sms, void *temp, size_t temp_bytes, cudaStream_t s) {
    if (b.ngroups == 0) return;
    if (b.ngroups >= 8 * sms)
        b.schur_chunk = std::max(b.schur_chunk, 64);
    b.schur_max_chunks = (int)(b.npairs / b.schur_chunk + b.ngroups);
    k_schur_count_chunks<<<div_up(b.ngroups + 1, 256), 256, 0, s>>>(
        b.group_start, b.group_order, b.ngroups, b.schur_chunk, b.schur_chunk_off, b.schur_part_off);
    SFMBA_LAUNCH_CHECK();
    for (int *v : {b.schur_chunk_off, b.schur_part_off}) {
        size_t need = 0;
        SFMBA_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, need, v, v, b.ngroups + 1, s));
        if (need > temp_bytes) throw Error(SFMBA_ERR_INTERNAL, "chunk scan temp too small");
        SFMBA_CUDA(cub::DeviceScan::ExclusiveSum(temp, need, v, v, b.ngroups + 1, s));
    }
    k_schur_list_chunks<<<div_up(b.ngroups, 256), 256, 0, s>>>(b.group_start, b.group_order, b.ngroups, b.schur_chunk,
                                                               b.schur_chunk_off, b.schur_part_off, b.schur_chunks);
    SFMBA_LAUNCH_CHECK();
}

size_t shared_fold_temp_bytes(long long nkeys) {
    size_t bytes = 0;
    SFMBA_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, bytes, (const uint64_t *)nullptr, (uint64_t *)nullptr,
                                              std::max<long long>(nkeys, 1)));
    return bytes;
}

void launch_shared_fold_setup(Bufs &b, uint64_t *keys, uint64_t *keys_tmp, void *temp, size_t temp_bytes,
                              cudaStream_t s) {
    k_fold_keys<<<div_up(b.ngroups, 256), 256, 0, s>>>(b.group_ij, b.ngroups, b.fold_shcam, b.nI, b.fold_nsh, keys_tmp);
    SFMBA_LAUNCH_CHECK();
    SFMBA_CUDA(cub::DeviceRadixSort::SortKeys(temp, temp_bytes, (const uint64_t *)keys_tmp, keys,
                                              2LL * b.ngroups, 0, 64, s));
    b.fold_keys = keys;
    b.fold_nkeys = 2 * b.ngroups;
}

void launch_fold_system(const Bufs &b, cudaStream_t s) {
    if (b.n == 0) return;
    dim3 grid(div_up(b.n, 128), b.n);
    k_fold<<<grid, 128, 0, s>>>(b.S_img, b.nID, b.slot_pre_start, b.slot_pre, b.slot_masked, b.diagB,
                                b.state, b.n, b.fold_nslots > 0, b.S, b.L);
    SFMBA_LAUNCH_CHECK();
    if (b.fold_nslots > 0) {
        k_fold_shared<<<(unsigned)(b.fold_nslots * b.fold_nslots), 32, 0, s>>>(
            b.S_img, b.nID, b.D, b.nI, b.fold_nsh, b.fold_keys, b.fold_nkeys, b.fold_slots, b.fold_nslots, b.fold_shcam,
            b.slot_pre_start, b.slot_pre, b.slot_masked, b.diagB, b.state, b.n, b.S, b.L);
        SFMBA_LAUNCH_CHECK();
    }
    k_fold_rhs<<<div_up(b.n, 256), 256, 0, s>>>(b.img_rhs, b.slot_pre_start, b.slot_pre, b.slot_masked,
                                                b.n, b.rhs);
    SFMBA_LAUNCH_CHECK();
}

void launch_fold_rhs(const Bufs &b, cudaStream_t s) {
    if (b.n == 0) return;
    k_fold_rhs<<<div_up(b.n, 256), 256, 0, s>>>(b.img_rhs, b.slot_pre_start, b.slot_pre, b.slot_masked, b.n,
                                                b.rhs);
    SFMBA_LAUNCH_CHECK();
}

namespace {

// Second stream and two events of the look-ahead, per host thread and device.
struct LookAhead {
    int device = -1;
    cudaStream_t s2 = nullptr;
    cudaEvent_t col_done = nullptr, next_ready = nullptr;
    ~LookAhead() {
        if (col_done) cudaEventDestroy(col_done);
        if (next_ready) cudaEventDestroy(next_ready);
        if (s2) cudaStreamDestroy(s2);
    }
};

LookAhead &look_ahead() {
    thread_local LookAhead la;
    int dev = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    if (la.device != dev) {
        if (la.s2) {
            cudaEventDestroy(la.col_done);
            cudaEventDestroy(la.next_ready);
            cudaStreamDestroy(la.s2);
        }
        la.device = dev;
        // The highest priority: the next panel's blocks are dispatched as soon
        // as the trailing update's blocks free an SM, not after all of them.
        int least = 0, greatest = 0;
        SFMBA_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        SFMBA_CUDA(cudaStreamCreateWithPriority(&la.s2, cudaStreamNonBlocking, greatest));
        SFMBA_CUDA(cudaEventCreateWithFlags(&la.col_done, cudaEventDisableTiming));
        SFMBA_CUDA(cudaEventCreateWithFlags(&la.next_ready, cudaEventDisableTiming));
    }
    return la;
}

}  // namespace

// Cooperative launch of kernel k with `want` blocks of 256 threads at most
// what the GPU holds at once (cap: co-resident blocks, queried once per
// device by the caller); false when none can be resident.
template <typename... Args>
bool launch_coop(void (*k)(Args...), int cap, int want, size_t smem, cudaStream_t s, Args... args) {
    if (cap < 1) return false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::max(1, std::min(cap, want)));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SFMBA_CUDA(cudaLaunchKernelEx(&cfg, k, args...));
    SFMBA_LAUNCH_CHECK();
    return true;
}

// Co-resident blocks of a 256-thread kernel with `smem` dynamic shared memory.
template <typename K>
int coop_capacity(K k, size_t smem) {
    int dev = 0, per_sm = 0, sms = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    SFMBA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, smem));
    SFMBA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return per_sm * sms;
}

// Blocked right-looking Cholesky with a look-ahead of one panel: after the
// panel of block k, the tile column of block k + 1 is updated first; then
// the diagonal factor, panel (and slices) of block k + 1 run on a second
// stream while the rest of block k's trailing update runs on s. The
// diagonal factor is the serial part (one cluster of three blocks, FP64-pipe
// bound), so it hides behind the bulk update. Tensor-core updates read the panel slices of
// their own step: two slice buffers alternate by step.
void launch_cholesky(const Bufs &b, cudaStream_t s) {
    set_smem_limits();
    const int n = b.n;
    if (n == 0) return;
    const bool oz = b.oz_slices != nullptr;
    const size_t slice_elems = div_up(n, 64) * kOzBlockElems;
    const int polls = b.give_up_tiles ? 0 : kOzPolls;
    auto slices = [&](int k0) { return (__nv_bfloat16 *)b.oz_slices + ((k0 / NB) & 1) * slice_elems; };
    auto exps = [&](int k0) { return b.oz_exp + ((k0 / NB) & 1) * (size_t)n; };
    // diagonal factor, panel and (tensor path) slices of block k0, on stream st
    auto head = [&](int k0, cudaStream_t st) {
        k_chol_diag<<<kCholCluster, 256, 0, st>>>(b.L, n, k0, b.Linv, b.state, b.give_up_columns ? 0 : kBlkPolls);
        SFMBA_LAUNCH_CHECK();
        const int rem = n - k0 - NB;
        if (rem <= 0) return;
        k_chol_panel<<<div_up(rem, kPanelRows), 256, 0, st>>>(b.L, n, k0, b.Linv, b.state);
        SFMBA_LAUNCH_CHECK();
        if (oz) {
            k_oz_split<<<div_up(rem, 8), 256, 0, st>>>(b.L, n, k0, slices(k0), exps(k0), b.state);
            SFMBA_LAUNCH_CHECK();
        }
    };
    auto update = [&](int k0, int part, cudaStream_t st) {
        const int tiles = div_up(n - k0 - NB, NB);
        const long long blocks = part == 1 ? tiles : (tiles - 1LL) * tiles / 2;
        if (oz) {
            // The next block's column is on the chain and few tiles: narrow ones (15 us
            // for n = 2560 against 22).
            if (part == 1)
                k_oz_update<32><<<dim3(div_up(tiles, 2), 2), kOzThreads, kOzSmem, st>>>(b.L, n, k0, 0, slices(k0),
                                                                                       exps(k0), b.state, polls);
            else
                k_oz_update<64><<<dim3(tiles / 2, tiles - 1), kOzThreads, kOzSmem, st>>>(b.L, n, k0, 1, slices(k0),
                                                                                        exps(k0), b.state, polls);
        } else if (chol_tile(blocks) == 16)
            k_chol_update<16><<<(unsigned)(16 * blocks), 256, 0, st>>>(b.L, n, k0, part, b.state);
        else
            k_chol_update<32><<<(unsigned)(4 * blocks), 256, 0, st>>>(b.L, n, k0, part, b.state);
        SFMBA_LAUNCH_CHECK();
    };
    head(0, s);
    for (int k0 = 0; k0 + NB < n; k0 += NB) {
        const long long tiles = div_up(n - k0 - NB, NB);
        const int k1 = k0 + NB;
        update(k0, 1, s);  // tile column of block k1
        if (tiles == 1) {
            head(k1, s);
            continue;
        }
        LookAhead &la = look_ahead();
        SFMBA_CUDA(cudaEventRecord(la.col_done, s));
        SFMBA_CUDA(cudaStreamWaitEvent(la.s2, la.col_done, 0));
        head(k1, la.s2);
        SFMBA_CUDA(cudaEventRecord(la.next_ready, la.s2));
        update(k0, 2, s);
        SFMBA_CUDA(cudaStreamWaitEvent(s, la.next_ready, 0));
    }
}

void launch_cholesky_solve(const Bufs &b, const double *rhs, double *x, cudaStream_t s) {
    const int n = b.n;
    if (n == 0) return;
    const int nblk = div_up(n, NB);
    SFMBA_CUDA(cudaMemsetAsync(b.trsv_ready, 0, sizeof(int) * 2 * (size_t)nblk, s));
    thread_local int cap_dev = -1, cap = 0;  // co-resident blocks
    int dev = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    if (cap_dev != dev) {
        cap = coop_capacity(k_trsv_flow, 0);
        cap_dev = dev;
    }
    if (!launch_coop(k_trsv_flow, cap, nblk, 0, s, (const double *)b.L, n, (const double *)b.Linv, rhs, b.work2, x,
                     b.trsv_ready, b.state))
        throw Error(SFMBA_ERR_INTERNAL, "the triangular solve does not fit the GPU");
}

void launch_refine(const Bufs &b, cudaStream_t s) {
    // One FP64 iterative-refinement step: res = rhs - S delta, solve, delta += c.
    k_residual<<<div_up((long long)b.n * 32, 256), 256, 0, s>>>(b.S, b.n, b.delta, b.rhs, b.ref_res, b.state);
    SFMBA_LAUNCH_CHECK();
    launch_cholesky_solve(b, b.ref_res, b.ref_corr, s);
    k_axpy_inplace<<<div_up(b.n, 256), 256, 0, s>>>(b.n, b.ref_corr, b.delta, b.state);
    SFMBA_LAUNCH_CHECK();
}

// Blocks (a row per SM sub-partition, whose FP64 pipe its division and products
// fill, at most one block per SM) and shared memory of k_lu_coop; false when
// the rows' order does not fit and the columns take a launch each.
static bool lu_coop_shape(int n, int &blocks, size_t &smem) {
    int dev = 0, sms = 0, most = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    SFMBA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SFMBA_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    blocks = std::min(sms, div_up(n, 4));
    smem = lu_coop_smem(div_up(n, blocks), n);
    return smem + 1024 <= (size_t)most;
}

void launch_lu_factor(const Bufs &b, cudaStream_t s) {
    const int n = b.n;
    SFMBA_CUDA(cudaMemcpyAsync(b.L, b.S, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, s));
    if (n == 0) return;
    int blocks = 0;
    size_t smem = 0;
    if (!b.lu_by_columns && lu_coop_shape(n, blocks, smem)) {
        set_smem_limits();
        launch_coop(k_lu_coop, blocks, blocks, smem, s, b.L, n, b.lu_perm, (const LMState *)b.state,
                    div_up(n, blocks));
        return;
    }
    for (int k = 0; k < n; ++k) {
        k_lu_pivot<<<1, 1024, 0, s>>>(b.L, n, k, b.lu_perm, b.state);
        SFMBA_LAUNCH_CHECK();
        if (k + 1 < n) {
            dim3 grid(div_up(n - k - 1, 128), n - k - 1);
            k_lu_update<<<grid, 128, 0, s>>>(b.L, n, k, b.lu_perm, b.state);
            SFMBA_LAUNCH_CHECK();
        }
    }
}

void launch_lu_solve(const Bufs &b, cudaStream_t s) {
    int blocks = 0;
    size_t smem = 0;
    const bool ordered = !b.lu_by_columns && b.n > 0 && lu_coop_shape(b.n, blocks, smem);
    k_lu_solve<<<1, 1024, 0, s>>>(b.L, b.n, b.lu_perm, b.rhs, b.delta, b.state, ordered);
    SFMBA_LAUNCH_CHECK();
}

}  // namespace sfmba
