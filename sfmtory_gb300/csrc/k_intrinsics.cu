// refine_intrinsics (crates/sfm-ba/src/intrinsics.rs:116-238): every camera's
// parameters refined by its own dense LM with poses and points held fixed.
// Per iteration the k x k normal equations of the robustly weighted residuals
// with central finite-difference Jacobians (step 1e-6 on each parameter),
// the damped system solved by one thread (Cholesky, LU fallback, else
// lambda x 3), the trial cost; accept iff finite and lower (lambda / 3, floor
// 1e-12), at most 8 tries, stop when none is accepted. Cameras with fewer
// than 8 observations keep their parameters. All arithmetic FP64.
//
// The loop ends where rounding decides whether a step lowers the cost, so
// the order of every sum is part of the result: observation k of a camera
// belongs to lane k % 128, each lane sums its own in order, and the 128 lane
// sums are combined in one fixed tree. Sums of two products are written as an
// explicit multiply-add, so that the rounding does not depend on the compiler.
// Two kernels keep that order, with the same bits:
//   * few or large cameras: one cooperative kernel takes all cameras through
//     the loop in step, its work spread over the whole GPU. A round is: the
//     terms of every observation (one thread each, the FP64-heavy part), the
//     lane sums (one 128-thread block per camera and quantity, reading the
//     terms), the small solves, and the same two steps for the trial costs;
//   * many small cameras: one block per camera for its whole loop, without
//     terms in memory and without waiting for the other cameras.
//
// Bound: the FP64 pipe (17 projections and 16 divisions per observation and
// iteration). One OPENCV camera seen in 120 000 observations: 13 ms a call in
// step, 640 ms by one block, which leaves 151 of 152 SMs idle. 2000 OPENCV
// cameras of 400 observations each: 36 ms in step, 18 ms by blocks.
#include <cooperative_groups.h>

#include <algorithm>

#include "camera.cuh"
#include "kernels.cuh"

namespace sfmba {

namespace {

constexpr int kRefineThreads = kRefineLanes;
constexpr double kFdStep = 1e-6;           // intrinsics.rs EPS
constexpr int kRefineSys = 8 * 9 / 2 + 8;  // upper triangle of J^T W J, then J^T W r
constexpr int kCarry = kRefineSys * kRefineLanes;

// Block sum in FP64, fixed order (warp shuffles, then the warps in order).
__device__ __forceinline__ double block_sum128(double v, double *sh) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    const double r = sh[0] + sh[1] + sh[2] + sh[3];
    return r;
}

// One camera's loop. mode: 0 ended, 1 the next round forms the system,
// 2 the next round retries it with more damping.
struct RefineState {
    double cur[8], trial[8], sys[kRefineSys];
    double lambda, cost;
    int it, tries, mode, solved;
};

struct RefineArgs {
    const double *poses, *points, *ob_xy;
    const int *ob_img, *ob_pt, *cam_model;
    const int *row_cam;    // [rows] camera of each 128-observation row
    const int *cam_row0;   // [nC + 1] first row of each camera
    const int *row_obs;    // [rows][128] observation, -1 past the camera's last
    double *terms;         // [kRefineSys + 1][chunk rows][128]
    double *lane_sum;      // [2][kRefineSys][128] lane sums of the one camera that crosses a chunk's end
    RefineState *st;       // [nC]
    int *active;           // cameras whose loop has not ended
    double *cams;
    int nC, rows, chunk_rows, max_iterations, loss;
    double lambda0, scale;
};

__device__ __forceinline__ bool obs_residual(const double *poses, const double *points, const int *ob_img,
                                             const int *ob_pt, const double *ob_xy, int o, int model,
                                             const double *cam, double &rx, double &ry) {
    const int i = ob_img[o], p = ob_pt[o];
    const double *X = points + 3 * (size_t)p;
    return residual64(poses + 7 * (size_t)i, model, cam, X[0], X[1], X[2], ob_xy[2 * (size_t)o],
                      ob_xy[2 * (size_t)o + 1], rx, ry);
}

// Residual r0, weight w and difference columns jx, jy of observation o at
// `cur`; false for a point behind the camera.
__device__ __forceinline__ bool obs_columns(const RefineArgs &q, int o, int model, const double *cur, double &r0x,
                                            double &r0y, double &w, double (&jx)[8], double (&jy)[8]) {
    const int np = model_dof(model);
    double pp[8];
    if (!obs_residual(q.poses, q.points, q.ob_img, q.ob_pt, q.ob_xy, o, model, cur, r0x, r0y)) return false;
    w = robust_weight<double>(sqrt(__fma_rn(r0x, r0x, __dmul_rn(r0y, r0y))), q.loss, q.scale);
#pragma unroll
    for (int k = 0; k < 8; ++k) pp[k] = cur[k];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        jx[a] = jy[a] = 0.0;
        if (a >= np) continue;
        double px = r0x, py = r0y, mx = r0x, my = r0y;
        pp[a] = cur[a] + kFdStep;
        if (!obs_residual(q.poses, q.points, q.ob_img, q.ob_pt, q.ob_xy, o, model, pp, px, py)) { px = r0x; py = r0y; }
        pp[a] = cur[a] - kFdStep;
        if (!obs_residual(q.poses, q.points, q.ob_img, q.ob_pt, q.ob_xy, o, model, pp, mx, my)) { mx = r0x; my = r0y; }
        pp[a] = cur[a];
        jx[a] = (px - mx) / (2.0 * kFdStep);
        jy[a] = (py - my) / (2.0 * kFdStep);
    }
    return true;
}

// Terms of observation o for the normal equations: the products each
// quantity sums and, last, the weight that multiplies them (all 0 for a
// point behind the camera or a row's padding, o < 0).
__device__ __forceinline__ void system_terms(const RefineArgs &q, int o, int model, const double *cur, double *out,
                                             size_t plane) {
    const int np = model_dof(model);
    double r0x = 0.0, r0y = 0.0, w = 0.0, jx[8], jy[8];
    if (o < 0 || !obs_columns(q, o, model, cur, r0x, r0y, w, jx, jy)) {
        r0x = r0y = w = 0.0;
#pragma unroll
        for (int a = 0; a < 8; ++a) jx[a] = jy[a] = 0.0;
    }
    int e = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = a; b < 8; ++b, ++e)
            if (b < np) out[e * plane] = __fma_rn(jx[a], jx[b], __dmul_rn(jy[a], jy[b]));
#pragma unroll
    for (int a = 0; a < 8; ++a)
        if (a < np) out[(36 + a) * plane] = __fma_rn(jx[a], r0x, __dmul_rn(jy[a], r0y));
    out[kRefineSys * plane] = w;
}

// Terms of observation o for the robust cost w n^2: w n and n (0 for a point
// behind the camera or a row's padding).
__device__ __forceinline__ void cost_terms(const RefineArgs &q, int o, int model, const double *cam, double &wn,
                                           double &n) {
    double rx, ry;
    wn = n = 0.0;
    if (o >= 0 && obs_residual(q.poses, q.points, q.ob_img, q.ob_pt, q.ob_xy, o, model, cam, rx, ry)) {
        n = sqrt(__fma_rn(rx, rx, __dmul_rn(ry, ry)));
        wn = robust_weight<double>(n, q.loss, q.scale) * n;
    }
}

// Solves A x = b (n <= 8, row-major, A symmetric): Cholesky, else LU with
// partial pivoting; false if both fail.
__device__ __forceinline__ bool solve_small(int n, const double *A, const double *b, double *x) {
    double L[64];
    bool chol = true;
    for (int j = 0; j < n && chol; ++j) {
        double d = A[j * n + j];
        for (int k = 0; k < j; ++k) d -= L[j * 8 + k] * L[j * 8 + k];
        if (!(d > 0.0)) { chol = false; break; }
        const double ljj = sqrt(d);
        L[j * 8 + j] = ljj;
        for (int i = j + 1; i < n; ++i) {
            double v = A[i * n + j];
            for (int k = 0; k < j; ++k) v -= L[i * 8 + k] * L[j * 8 + k];
            L[i * 8 + j] = v / ljj;
        }
    }
    if (chol) {
        double y[8];
        for (int i = 0; i < n; ++i) {
            double v = b[i];
            for (int k = 0; k < i; ++k) v -= L[i * 8 + k] * y[k];
            y[i] = v / L[i * 8 + i];
        }
        for (int i = n - 1; i >= 0; --i) {
            double v = y[i];
            for (int k = i + 1; k < n; ++k) v -= L[k * 8 + i] * x[k];
            x[i] = v / L[i * 8 + i];
        }
        return true;
    }
    double M[64], r[8];
    int perm[8];
    for (int i = 0; i < n; ++i) {
        perm[i] = i;
        r[i] = b[i];
        for (int j = 0; j < n; ++j) M[i * 8 + j] = A[i * n + j];
    }
    for (int k = 0; k < n; ++k) {
        int p = k;
        double best = fabs(M[k * 8 + k]);
        for (int i = k + 1; i < n; ++i)
            if (fabs(M[i * 8 + k]) > best) { best = fabs(M[i * 8 + k]); p = i; }
        if (best == 0.0) return false;
        if (p != k) {
            for (int j = 0; j < n; ++j) { const double t = M[k * 8 + j]; M[k * 8 + j] = M[p * 8 + j]; M[p * 8 + j] = t; }
            const double t = r[k]; r[k] = r[p]; r[p] = t;
            const int q = perm[k]; perm[k] = perm[p]; perm[p] = q;
        }
        for (int i = k + 1; i < n; ++i) {
            const double f = M[i * 8 + k] / M[k * 8 + k];
            for (int j = k; j < n; ++j) M[i * 8 + j] -= f * M[k * 8 + j];
            r[i] -= f * r[k];
        }
    }
    for (int i = n - 1; i >= 0; --i) {
        double v = r[i];
        for (int j = i + 1; j < n; ++j) v -= M[i * 8 + j] * x[j];
        x[i] = v / M[i * 8 + i];
    }
    return true;
}

// Trial parameters of a camera: cur plus the step of the system `sys` damped by
// lambda; cur itself, and false, if it has no solution. One thread.
__device__ __forceinline__ bool damped_step(const double *sys, int np, double lambda, const double *cur, double *trial) {
    double A[64], rhs[8], dx[8];
    int e = 0;
    for (int a = 0; a < 8; ++a)
        for (int b = a; b < 8; ++b, ++e)
            if (a < np && b < np) A[a * np + b] = A[b * np + a] = sys[e];
    for (int a = 0; a < np; ++a) {
        rhs[a] = -sys[36 + a];
        A[a * np + a] += lambda * fmax(A[a * np + a], 1e-12);
    }
    const bool solved = solve_small(np, A, rhs, dx);
    for (int a = 0; a < 8; ++a) trial[a] = cur[a] + (solved && a < np ? dx[a] : 0.0);
    return solved;
}

// The lane's running sum over rows [r0, r1) of a chunk: sum of x * y in order
// (t: the row-major terms of this lane, py: distance from x to y). Loads of
// eight rows are in flight ahead of the dependent multiply-adds.
__device__ __forceinline__ double lane_chain(const double *x, const double *y, int rows, double acc) {
    int r = 0;
    for (; r + 8 <= rows; r += 8) {
        double a[8], b[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            a[k] = x[(size_t)(r + k) * kRefineLanes];
            b[k] = y[(size_t)(r + k) * kRefineLanes];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) acc = fma(a[k], b[k], acc);
    }
    for (; r < rows; ++r) acc = fma(x[(size_t)r * kRefineLanes], y[(size_t)r * kRefineLanes], acc);
    return acc;
}

__global__ void __launch_bounds__(kRefineThreads) k_refine_intrinsics(RefineArgs q) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[4];
    const int lane = threadIdx.x;
    const size_t plane = (size_t)q.chunk_rows * kRefineLanes;
    const int chunks = (q.rows + q.chunk_rows - 1) / q.chunk_rows;

    // The loops' start states.
    for (int c = blockIdx.x; c < q.nC; c += gridDim.x) {
        RefineState &s = q.st[c];
        if (lane < 8) s.cur[lane] = s.trial[lane] = q.cams[8 * (size_t)c + lane];
        if (lane == 0) {
            s.lambda = q.lambda0;
            s.cost = 0.0;
            s.it = -1;  // the first round only evaluates the start cost
            s.tries = 0;
            s.solved = 1;
            s.mode = q.cam_row0[c + 1] > q.cam_row0[c] ? 2 : 0;  // intrinsics.rs:135-141: left as it is
        }
    }
    grid.sync();

    for (bool first = true;; first = false) {
        if (!first) {
            if (*(volatile int *)q.active == 0) break;
            for (int k = 0; k < chunks; ++k) {
                const int lo = k * q.chunk_rows, hi = min(q.rows, lo + q.chunk_rows);
                for (int row = lo + blockIdx.x; row < hi; row += gridDim.x) {
                    const int c = q.row_cam[row];
                    const RefineState &s = q.st[c];
                    if (s.mode != 1) continue;
                    system_terms(q, q.row_obs[(size_t)row * kRefineLanes + lane], q.cam_model[c], s.cur,
                                 q.terms + (size_t)(row - lo) * kRefineLanes + lane, plane);
                }
                grid.sync();
                const int c0 = q.row_cam[lo], c1 = q.row_cam[hi - 1];  // the chunk's cameras
                for (int t = blockIdx.x; t < (c1 - c0 + 1) * kRefineSys; t += gridDim.x) {
                    const int c = c0 + t / kRefineSys, e = t % kRefineSys;
                    RefineState &s = q.st[c];
                    const int r0 = max(lo, q.cam_row0[c]), r1 = min(hi, q.cam_row0[c + 1]);
                    if (s.mode != 1 || r0 >= r1) continue;
                    const int np = model_dof(q.cam_model[c]);
                    // entry e of the upper triangle (rows of 8, 7, .. entries) or of J^T W r
                    int a = 0, b = e;
                    for (; a < 8 && b >= 8 - a; ++a) b -= 8 - a;
                    if (e >= 36 ? e - 36 >= np : a + b >= np) continue;
                    double *carry = q.lane_sum + e * kRefineLanes + lane;
                    const double *in = q.terms + (size_t)(r0 - lo) * kRefineLanes + lane;
                    double acc = r0 == q.cam_row0[c] ? 0.0 : carry[((k - 1) & 1) * kCarry];
                    acc = lane_chain(in + kRefineSys * plane, in + e * plane, r1 - r0, acc);
                    if (r1 < q.cam_row0[c + 1]) {
                        carry[(k & 1) * kCarry] = acc;
                    } else {
                        const double v = block_sum128(acc, sh);
                        if (lane == 0) s.sys[e] = v;
                    }
                }
                grid.sync();
            }
            for (int c = blockIdx.x; c < q.nC; c += gridDim.x) {
                RefineState &s = q.st[c];
                if (lane != 0 || s.mode == 0) continue;
                s.solved = damped_step(s.sys, model_dof(q.cam_model[c]), s.lambda, s.cur, s.trial) ? 1 : 0;
                s.mode = 2;
                if (!s.solved) {  // intrinsics.rs:202-205
                    s.lambda *= 3.0;
                    if (++s.tries == 8) {
                        s.mode = 0;
                        atomicSub(q.active, 1);
                    }
                }
            }
            grid.sync();
        }
        for (int k = 0; k < chunks; ++k) {
            const int lo = k * q.chunk_rows, hi = min(q.rows, lo + q.chunk_rows);
            for (int row = lo + blockIdx.x; row < hi; row += gridDim.x) {
                const int c = q.row_cam[row];
                const RefineState &s = q.st[c];
                if (s.mode == 0 || !s.solved) continue;
                double *out = q.terms + (size_t)(row - lo) * kRefineLanes + lane;
                cost_terms(q, q.row_obs[(size_t)row * kRefineLanes + lane], q.cam_model[c], s.trial, out[0], out[plane]);
            }
            grid.sync();
            const int c0 = q.row_cam[lo], c1 = q.row_cam[hi - 1];
            for (int c = c0 + blockIdx.x; c <= c1; c += gridDim.x) {
                RefineState &s = q.st[c];
                const int r0 = max(lo, q.cam_row0[c]), r1 = min(hi, q.cam_row0[c + 1]);
                if (s.mode == 0 || !s.solved || r0 >= r1) continue;
                double *carry = q.lane_sum + lane;
                const double *in = q.terms + (size_t)(r0 - lo) * kRefineLanes + lane;
                double acc = r0 == q.cam_row0[c] ? 0.0 : carry[((k - 1) & 1) * kCarry];
                acc = lane_chain(in, in + plane, r1 - r0, acc);
                if (r1 < q.cam_row0[c + 1]) {
                    carry[(k & 1) * kCarry] = acc;
                    continue;
                }
                const double tc = block_sum128(acc, sh);
                if (lane == 0) {
                    bool next = false;  // an iteration is over: accepted, or the start cost
                    if (s.it < 0) {
                        s.cost = tc;
                        next = true;
                    } else if (isfinite(tc) && tc < s.cost) {
                        for (int a = 0; a < 8; ++a) s.cur[a] = s.trial[a];
                        s.cost = tc;
                        s.lambda = fmax(s.lambda / 3.0, 1e-12);
                        next = true;
                    } else {
                        s.lambda *= 3.0;
                        if (++s.tries == 8) {
                            s.mode = 0;
                            atomicSub(q.active, 1);
                        }
                    }
                    if (next) {
                        s.tries = 0;
                        s.mode = ++s.it < q.max_iterations ? 1 : 0;
                        if (s.mode == 0) atomicSub(q.active, 1);
                    }
                }
                __syncthreads();  // sh is reused by the block's next camera
            }
            grid.sync();
        }
    }
    for (int c = blockIdx.x; c < q.nC; c += gridDim.x)
        if (lane < 8) q.cams[8 * (size_t)c + lane] = q.st[c].cur[lane];
}

// Robust cost of the parameters `cam` over rows [r0, r1), by the block.
__device__ double block_cost(const RefineArgs &q, int r0, int r1, int model, const double *cam, double *sh) {
    double sum = 0.0;
    for (int r = r0; r < r1; ++r) {
        double wn, n;
        cost_terms(q, q.row_obs[(size_t)r * kRefineLanes + threadIdx.x], model, cam, wn, n);
        sum = fma(wn, n, sum);
    }
    return block_sum128(sum, sh);
}

// One block per camera for its whole loop.
__global__ void __launch_bounds__(kRefineThreads) k_refine_cameras(RefineArgs q) {
    __shared__ double sh[4], cur[8], trial[8], sys[kRefineSys];
    __shared__ int solved;
    const int c = blockIdx.x, lane = threadIdx.x, r0 = q.cam_row0[c], r1 = q.cam_row0[c + 1];
    if (r0 == r1) return;  // intrinsics.rs:135-141: left as it is
    const int model = q.cam_model[c], np = model_dof(model);
    if (lane < 8) cur[lane] = q.cams[8 * (size_t)c + lane];
    __syncthreads();
    double cost = block_cost(q, r0, r1, model, cur, sh), lambda = q.lambda0;
    for (int it = 0; it < q.max_iterations; ++it) {
        double acc[kRefineSys];
#pragma unroll
        for (int e = 0; e < kRefineSys; ++e) acc[e] = 0.0;
        for (int r = r0; r < r1; ++r) {
            const int o = q.row_obs[(size_t)r * kRefineLanes + lane];
            double r0x, r0y, w, jx[8], jy[8];
            if (o < 0 || !obs_columns(q, o, model, cur, r0x, r0y, w, jx, jy)) continue;
            int e = 0;
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int b = a; b < 8; ++b, ++e)
                    if (b < np) acc[e] = fma(w, __fma_rn(jx[a], jx[b], __dmul_rn(jy[a], jy[b])), acc[e]);
#pragma unroll
            for (int a = 0; a < 8; ++a, ++e)
                if (a < np) acc[e] = fma(w, __fma_rn(jx[a], r0x, __dmul_rn(jy[a], r0y)), acc[e]);
        }
        auto total = [&](int e, double v) {
            v = block_sum128(v, sh);
            if (lane == 0) sys[e] = v;
        };
        int e = 0;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = a; b < 8; ++b, ++e)
                if (b < np) total(e, acc[e]);
#pragma unroll
        for (int a = 0; a < 8; ++a, ++e)
            if (a < np) total(e, acc[e]);
        __syncthreads();
        bool accepted = false;
        for (int t = 0; t < 8; ++t) {
            if (lane == 0) solved = damped_step(sys, np, lambda, cur, trial);
            __syncthreads();
            if (solved) {
                const double tc = block_cost(q, r0, r1, model, trial, sh);
                if (isfinite(tc) && tc < cost) {
                    cost = tc;
                    accepted = true;
                    break;
                }
            }
            lambda *= 3.0;  // intrinsics.rs:202-205, for a system without a solution too
            __syncthreads();
        }
        if (!accepted) break;
        lambda = fmax(lambda / 3.0, 1e-12);
        if (lane < 8) cur[lane] = trial[lane];
        __syncthreads();
    }
    if (lane < 8) q.cams[8 * (size_t)c + lane] = cur[lane];
}

}  // namespace

// In step or a block per camera. In step pays for its barriers and for the
// (camera, quantity) sums of every round, a block for the rows of the largest
// camera, one after another. Measured, block time / time in step (SIMPLE_RADIAL,
// OPENCV alike): 1 camera of 1, 2, 4, 16 rows 0.98, 1.1, 1.7, 3.9; 50 cameras of
// 2, 4, 8, 32 rows 0.7, 1.05, 1.5, 2.9; 150 of 4, 8, 32 rows 0.8, 1.1, 1.2; 300 of
// 4 to 16 rows 0.7 to 0.9, however many rows: then the blocks fill the GPU, so
// the largest camera has to hold more than 3/5 of an SM's share of all rows.
bool refine_in_step(int cameras, int most_rows, int rows, int sms) {
    return cameras + 45LL <= 25LL * most_rows && 3LL * rows <= 5LL * most_rows * sms;
}

size_t refine_state_bytes() { return sizeof(RefineState); }

void launch_refine_intrinsics(const IntrinsicsBufs &q, int max_iterations, double lambda0, int loss, double scale,
                              cudaStream_t s) {
    if (q.nC == 0 || q.rows == 0) return;
    RefineArgs a;
    a.poses = q.poses; a.points = q.points; a.ob_xy = q.ob_xy;
    a.ob_img = q.ob_img; a.ob_pt = q.ob_pt; a.cam_model = q.cam_model;
    a.row_cam = q.row_cam; a.cam_row0 = q.cam_row0; a.row_obs = q.row_obs;
    a.terms = q.terms; a.lane_sum = q.lane_sum; a.st = (RefineState *)q.state; a.active = q.active;
    a.cams = q.cams;
    a.nC = q.nC; a.rows = q.rows; a.chunk_rows = std::min(q.rows, kRefineChunkRows);
    a.max_iterations = max_iterations; a.loss = loss; a.lambda0 = lambda0; a.scale = scale;
    if (!q.in_step) {
        k_refine_cameras<<<q.nC, kRefineThreads, 0, s>>>(a);
        SFMBA_LAUNCH_CHECK();
        return;
    }
    int dev = 0, per_sm = 0, sms = 0;
    SFMBA_CUDA(cudaGetDevice(&dev));
    SFMBA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine_intrinsics, kRefineThreads, 0));
    SFMBA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (per_sm < 1) throw Error(SFMBA_ERR_INTERNAL, "the intrinsics kernel does not fit an SM");
    // Blocks past one per row or lane sum would only add to the grid barriers.
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::min<long long>((long long)per_sm * sms,
                                                     std::max<long long>(a.rows, std::min<long long>(kRefineSys * (long long)q.nC, sms))));
    cfg.blockDim = dim3(kRefineThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SFMBA_CUDA(cudaLaunchKernelEx(&cfg, k_refine_intrinsics, a));
    SFMBA_LAUNCH_CHECK();
}

}  // namespace sfmba
