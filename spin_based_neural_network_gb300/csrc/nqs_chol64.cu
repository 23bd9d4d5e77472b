// FP64 Cholesky factorisation and solve of the plain MinSR path, T y = b, in one cooperative
// launch: T = L L^T (lower triangle, in place), L z = b beside it, then L^T y = z.
//
// 32-wide block columns, right-looking.  Step k:
//   panel     the rows below the factored diagonal block, x L_kk^T = a, and the right-hand side,
//             two or eight rows a warp with 16 or four lanes a row, spread over the CTAs so that
//             each SM's FP64 pipes take a share (a warp instruction takes 64 clocks of a quarter
//             SM's pipe however many lanes are active);
//   trailing  32 x 32 tiles of A -= P P^T (and of z -= P z_k, by the owners of the diagonal tiles)
//             on CTAs 1 .. G-1, while CTA 0 updates the next diagonal block and factors it.
// The step is bound by the FP64 pipes of all SMs while the trailing matrix is large and by the
// chain panel -> next diagonal block -> two grid barriers below n ~ 1000 (an FP64 instruction takes
// 64 clocks of a quarter SM's pipe and as long to return, so a chain of them is slow wherever it runs).
// Measured at n = 1000 (4x4 Heisenberg, 1000 samples): 1.23 ms for factor and solve against 5.85 ms
// as 157 launches of one kernel per block and phase.
#include <algorithm>

#include "nqs_grid.cuh"
#include "nqs_internal.cuh"

namespace nqs {

namespace {

constexpr int CB = 32, CT = 256;          // block width, threads

struct Chol64Args {
    double *T;                            // [n][n], lower triangle
    int n;
    const double *b;
    double *z, *y, *rd;                   // forward solution, result, reciprocal diagonal of L [n]
    int *status;                          // status[I_FAIL]: first non-positive pivot column, or -1
    unsigned *bar;
    int *err;
};

struct Chol64Smem {
    double A[CB][CB + 1], B[CB][CB + 1];  // [k][row] operands; the diagonal block
    double rinv[CB], x[CB];
    int fail;
};

// Lower-triangular tile t: row bi, column bj <= bi.
__device__ __forceinline__ void lower_tile(int t, int &bi, int &bj) {
    int r = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= t) r++;
    while (r * (r + 1) / 2 > t) r--;
    bi = r;
    bj = t - r * (r + 1) / 2;
}

// Factor the kb x kb block in S (lower triangle; rows kb .. 31 the identity) by the block, in panels of
// four columns: warp 0 (lane = row) runs the panel's pivots and their columns in registers, then all
// warps take the panel off the columns after it, so that the long part of the FP64 work is on the four
// pipes of the SM and warp 0 keeps the chain of pivots only (34 FP64 instructions a panel).  rinv gets
// the reciprocal pivots; *fail the first column whose pivot is not positive, or -1; the columns
// before it are finished in S (the pivot test of src/nqs/nqs_optimizer.c:1029-1031).
// Measured: order 1000, factor and solve 1.23 ms, 1.69 ms with the whole block by one warp (28 us each)
// and eight rows a warp in every panel.
__device__ void factor32(double (*S)[CB + 1], int kb, double *rinv, int *fail) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int j0 = 0; j0 < CB; j0 += 4) {
        if (warp == 0) {
            double d[4];
            int f = -1;
#pragma unroll
            for (int b = 0; b < 4; b++) d[b] = lane >= j0 + b ? S[lane][j0 + b] : 0.0;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                double p = __shfl_sync(0xffffffffu, d[b], j0 + b);
                if (f < 0 && j0 + b < kb && !(p > 0.0)) f = j0 + b;
                if (f >= 0) p = 1.0;                        // the sweep ends on a unit pivot
                const double y = rsqrt(p), l = d[b] * y;
                if (lane == j0 + b) rinv[j0 + b] = y;
                if (f < 0) d[b] = l;
#pragma unroll
                for (int c = b + 1; c < 4; c++) d[c] = fma(-l, __shfl_sync(0xffffffffu, l, j0 + c), d[c]);
            }
#pragma unroll
            for (int b = 0; b < 4; b++)
                if (lane >= j0 + b && (f < 0 || j0 + b < f)) S[lane][j0 + b] = d[b];
            if (lane == 0) *fail = f;
        }
        __syncthreads();
        if (*fail >= 0) return;                             // the same for the whole block
        const int r0 = j0 + 4, i = tid >> 3;
        if (4 * warp + 3 >= r0) {                           // warp w: rows 4 w .. 4 w + 3
            double l[4];
#pragma unroll
            for (int b = 0; b < 4; b++) l[b] = S[i][j0 + b];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = (tid & 7) + 8 * q;
                if (c >= r0 && c <= i) {
                    double v = S[i][c];
#pragma unroll
                    for (int b = 0; b < 4; b++) v = fma(-l[b], S[c][j0 + b], v);
                    S[i][c] = v;
                }
            }
        }
        __syncthreads();
    }
}

// x of one row from a (columns q + LR i a lane, LR lanes a row): x_j = a_j / L_jj, a -= x_j L_:j.
template <int LR>
__device__ __forceinline__ void row_solve(double (&s)[CB / LR], const double (*Ld)[CB + 1], const double *rinv, int kb,
                                          int lane) {
    const int q = lane % LR;
#pragma unroll
    for (int j = 0; j < CB; j++) {
        if (j >= kb) break;
        const int i = j / LR;
        const double x = __shfl_sync(0xffffffffu, s[i] * rinv[j], (lane & ~(LR - 1)) | (j % LR));
        if (q == j % LR) s[i] = x;
#pragma unroll
        for (int k = i; k < CB / LR; k++) s[k] = fma(-x, Ld[q + LR * k][j], s[k]);   // zero at and above the diagonal
    }
}

// The panel of the block at k0 (unit diagonal block Ld, reciprocal pivots rinv) and the right-hand
// side: 32 / LR rows a warp, dealt to the CTAs first.
template <int LR>
__device__ __forceinline__ void panel_solve(double *T, double *z, int n, int k0, int kb, const double (*Ld)[CB + 1],
                                            const double *rinv) {
    constexpr int RW = 32 / LR, C = CB / LR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k1 = k0 + kb, q = lane % LR;
    const int nun = (n - k1 + RW - 1) / RW;                 // unit nun is the right-hand side
    for (int u = blockIdx.x + gridDim.x * warp; u <= nun; u += gridDim.x * (CT / 32)) {
        const int row = k1 + u * RW + lane / LR;
        const bool ok = u < nun ? row < n : lane < LR;
        double *p = u < nun ? T + (size_t)row * n + k0 : z + k0;
        double s[C];
#pragma unroll
        for (int i = 0; i < C; i++) s[i] = ok && q + LR * i < kb ? __ldcg(p + q + LR * i) : 0.0;
        row_solve<LR>(s, Ld, rinv, kb, lane);
#pragma unroll
        for (int i = 0; i < C; i++)
            if (ok && q + LR * i < kb) p[q + LR * i] = s[i];
    }
}

__global__ void __launch_bounds__(CT, 1) k_chol64(Chol64Args a) {
    __shared__ Chol64Smem sm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bx = blockIdx.x, G = gridDim.x;
    const int n = a.n, nblk = (n + CB - 1) / CB;
    double *T = a.T;
    for (int i = bx * CT + tid; i < n; i += G * CT) a.z[i] = a.b[i];
    // CTA 0: the diagonal block at k0 from sm.A, factored and stored
    auto factor_store = [&](int k0) {
        const int kb = min(CB, n - k0);
        factor32(sm.A, kb, sm.rinv, &sm.fail);
        const int f = sm.fail, keep = f < 0 ? kb : f;
        for (int e = tid; e < CB * CB; e += CT) {
            const int r = e >> 5, c = e & 31;
            if (r < kb && c <= r && c < keep) T[(size_t)(k0 + r) * n + k0 + c] = sm.A[r][c];
        }
        if (tid < kb) a.rd[k0 + tid] = sm.rinv[tid];
        if (tid == 0 && f >= 0) a.status[I_FAIL] = k0 + f;
    };
    if (bx == 0) {
        for (int e = tid; e < CB * CB; e += CT) {
            const int r = e >> 5, c = e & 31;
            sm.A[r][c] = r < n && c <= r ? T[(size_t)r * n + c] : (r == c ? 1.0 : 0.0);
        }
        __syncthreads();
        factor_store(0);
    }
    if (!grid_barrier(a.bar, a.err, G)) return;
    for (int k = 0; k < nblk; k++) {
        const int k0 = k * CB, kb = min(CB, n - k0), k1 = k0 + kb, rest = n - k1;
        if (__ldcg(a.status + I_FAIL) >= 0) return;
        // ---- panel and right-hand side
        // two rows a warp while every row has a warp of its own SM's (the row's chain of dependent
        // operations bounds it: 3 us against 5), eight rows beyond (half the instructions a row)
        const bool few = rest <= 2 * G * (CT / 32);
        if (bx <= (few ? (rest + 1) / 2 : (rest + 7) / 8)) {
            for (int e = tid; e < CB * CB; e += CT) {
                const int r = e >> 5, c = e & 31;
                sm.B[r][c] = r < kb && c < r ? __ldcg(T + (size_t)(k0 + r) * n + k0 + c) : 0.0;
            }
            if (tid < CB) sm.rinv[tid] = tid < kb ? __ldcg(a.rd + k0 + tid) : 0.0;
            __syncthreads();
            if (few) panel_solve<16>(T, a.z, n, k0, kb, sm.B, sm.rinv);
            else panel_solve<4>(T, a.z, n, k0, kb, sm.B, sm.rinv);
        }
        if (rest <= 0) break;
        if (!grid_barrier(a.bar, a.err, G)) return;
        // ---- trailing update; the next diagonal block by CTA 0
        const int nb = (rest + CB - 1) / CB, ntile = nb * (nb + 1) / 2;
        const double *P = T + k0;                       // panel columns (row pitch n)
        if (bx == 0) {
            const int kn = min(CB, rest);
            for (int e = tid; e < CB * CB; e += CT) {
                const int r = e >> 5, c = e & 31;
                sm.B[r][c] = r < kn && c < kb ? __ldcg(P + (size_t)(k1 + r) * n + c) : 0.0;
                sm.A[r][c] = r < kn && c <= r ? __ldcg(T + (size_t)(k1 + r) * n + k1 + c) : (r == c ? 1.0 : 0.0);
            }
            if (tid < CB) sm.x[tid] = tid < kb ? __ldcg(a.z + k0 + tid) : 0.0;
            __syncthreads();
            // the ten lower 8 x 8 sub-blocks, an entry a thread
            for (int o = tid; o < 640; o += CT) {
                int br, bc;
                lower_tile(o >> 6, br, bc);
                const int r = 8 * br + ((o >> 3) & 7), c = 8 * bc + (o & 7);
                double s0 = sm.A[r][c], s1 = 0.0;
#pragma unroll
                for (int m = 0; m < CB; m += 2) {
                    s0 = fma(-sm.B[r][m], sm.B[c][m], s0);
                    s1 = fma(-sm.B[r][m + 1], sm.B[c][m + 1], s1);
                }
                sm.A[r][c] = s0 + s1;
            }
            if (warp == 7 && lane < kn) {
                double s = __ldcg(a.z + k1 + lane);
                for (int m = 0; m < CB; m++) s = fma(-sm.B[lane][m], sm.x[m], s);
                a.z[k1 + lane] = s;
            }
            __syncthreads();
            factor_store(k1);
        }
        const int own = G > 1 ? bx - 1 : 0, step = G > 1 ? G - 1 : 1;
        if (own >= 0 && own + 1 < ntile) {
            const int tx = tid & 15, ty = tid >> 4;
            double pa[4], pb[4], pc[4];
            int bi, bj;
            auto fetch = [&](int t) {                   // operands and old values of tile t into registers
                lower_tile(t, bi, bj);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int e = tid + CT * i, r = e >> 5, c = e & 31;
                    const int ra = k1 + bi * CB + r, rb = k1 + bj * CB + r;
                    pa[i] = ra < n && c < kb ? __ldcg(P + (size_t)ra * n + c) : 0.0;
                    pb[i] = rb < n && c < kb ? __ldcg(P + (size_t)rb * n + c) : 0.0;
                    const int ci = k1 + bi * CB + ty + 16 * (i >> 1), cj = k1 + bj * CB + tx + 16 * (i & 1);
                    pc[i] = ci < n && cj <= ci ? __ldcg(T + (size_t)ci * n + cj) : 0.0;
                }
            };
            fetch(own + 1);
            for (int t = own + 1; t < ntile; t += step) {
                __syncthreads();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int e = tid + CT * i, r = e >> 5, c = e & 31;
                    sm.A[c][r] = pa[i];
                    sm.B[c][r] = pb[i];
                }
                double acc[4] = {pc[0], pc[1], pc[2], pc[3]};
                const int ti = bi, tj = bj;
                if (ti == tj && tid < CB) sm.x[tid] = tid < kb ? __ldcg(a.z + k0 + tid) : 0.0;
                __syncthreads();
                if (t + step < ntile) fetch(t + step);
#pragma unroll
                for (int m = 0; m < CB; m++) {
                    const double a0 = -sm.A[m][ty], a1 = -sm.A[m][ty + 16], b0 = sm.B[m][tx], b1 = sm.B[m][tx + 16];
                    acc[0] = fma(a0, b0, acc[0]);
                    acc[1] = fma(a0, b1, acc[1]);
                    acc[2] = fma(a1, b0, acc[2]);
                    acc[3] = fma(a1, b1, acc[3]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int ci = k1 + ti * CB + ty + 16 * (i >> 1), cj = k1 + tj * CB + tx + 16 * (i & 1);
                    if (ci < n && cj <= ci) T[(size_t)ci * n + cj] = acc[i];
                }
                if (ti == tj && warp == 7 && k1 + ti * CB + lane < n) {
                    const int i = k1 + ti * CB + lane;
                    double s = __ldcg(a.z + i);
                    for (int m = 0; m < CB; m++) s = fma(-sm.A[m][lane], sm.x[m], s);
                    a.z[i] = s;
                }
            }
        }
        if (!grid_barrier(a.bar, a.err, G)) return;
    }
    if (!grid_barrier(a.bar, a.err, G)) return;
    // ---- L^T y = z, last block first; z_j -= sum_m L[k0 + m][j] y_m by column blocks
    for (int k = nblk - 1; k >= 0; k--) {
        const int k0 = k * CB, kb = min(CB, n - k0);
        for (int e = tid; e < CB * CB; e += CT) {
            const int r = e >> 5, c = e & 31;
            sm.B[r][c] = r < kb && c < r ? __ldcg(T + (size_t)(k0 + r) * n + k0 + c) : 0.0;
        }
        if (tid < CB) sm.rinv[tid] = tid < kb ? __ldcg(a.rd + k0 + tid) : 0.0;
        // the rows of this CTA's first column block do not depend on y: loaded before the barrier
        const int j = bx * CB + lane;
        double lv[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int m = warp * 4 + i;
            lv[i] = j < k0 && m < kb ? __ldcg(T + (size_t)(k0 + m) * n + j) : 0.0;
        }
        if (k < nblk - 1 && !grid_barrier(a.bar, a.err, G)) return;
        if (bx != 0 && bx * CB >= k0) continue;         // nothing left for this CTA but the barriers
        __syncthreads();
        if (warp == 0) {
            double v = lane < kb ? __ldcg(a.z + k0 + lane) : 0.0;
#pragma unroll 8
            for (int m = CB - 1; m >= 0; m--) {
                if (m >= kb) continue;
                const double x = __shfl_sync(0xffffffffu, v, m) * sm.rinv[m];
                if (lane == m) v = x;
                v = fma(-x, sm.B[m][lane], v);          // zero at and above the diagonal
            }
            sm.x[lane] = lane < kb ? v : 0.0;
            if (bx == 0 && lane < kb) a.y[k0 + lane] = v;
        }
        __syncthreads();
        for (int c0 = bx * CB; c0 < k0; c0 += G * CB) {
            double s = 0.0;
            if (c0 == bx * CB) {
#pragma unroll
                for (int i = 0; i < 4; i++) s = fma(lv[i], sm.x[warp * 4 + i], s);
            } else {
                for (int i = 0; i < 4; i++) {
                    const int m = warp * 4 + i;
                    if (m < kb) s = fma(__ldcg(T + (size_t)(k0 + m) * n + c0 + lane), sm.x[m], s);
                }
            }
            sm.A[warp][lane] = s;
            __syncthreads();
            if (warp == 0) {
                double v = __ldcg(a.z + c0 + lane);
#pragma unroll
                for (int w = 0; w < CT / 32; w++) v -= sm.A[w][lane];
                a.z[c0 + lane] = v;
            }
            __syncthreads();
        }
    }
}

}  // namespace

// T = L L^T and T y = b on the library stream; status[I_FAIL] (set to -1 by the caller) receives
// the first failing column, with the columns before it (of the rows down to its block's last) as
// the factorisation left them and y untouched.  *err_out (device) is raised when a barrier gave up.
bool chol64_factor_solve(double *T, int n, const double *b, double *y, int *status, int **err_out) {
    static DevBuf<double> z, rd;
    static DevBuf<unsigned> bar;
    Context &c = ctx();
    if (!z.ensure(n) || !rd.ensure(n) || !bar.ensure(2)) return false;
    if (!NQS_CUDA(cudaMemsetAsync(bar.p, 0, 2 * sizeof(unsigned), c.stream))) return false;
    *err_out = (int *)bar.p + 1;
    Chol64Args a{T, n, b, z.p, y, rd.p, status, bar.p, *err_out};
    // one CTA per SM, and no more than the first step's tiles or panel units can use
    const int nb = (n + CB - 1) / CB, grid = std::max(1, std::min(c.sm_count, std::max(nb * (nb - 1) / 2, n / 8) + 1));
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3(CT);
    lc.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    NQS_LAUNCH("chol_solve_fp64");
    return NQS_CUDA(cudaLaunchKernelEx(&lc, k_chol64, a));
}

bool chol64_set_barrier_budget(unsigned v, cudaStream_t st) {
    return NQS_CUDA(cudaMemcpyToSymbolAsync(g_barrier_budget, &v, sizeof(v), 0, cudaMemcpyHostToDevice, st)) &&
           NQS_CUDA(cudaStreamSynchronize(st));
}

}  // namespace nqs
