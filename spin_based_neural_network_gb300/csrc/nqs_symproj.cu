// Symmetry-projected RBM / complex RBM programs: log-amplitudes, gradients and local energies.
//
// psi(s) = sum_g chi_g cos(arg_g) |psi_base(g s)| / sqrt(G) (src/nqs/nqs_symproj.c:31-80).  One
// block per configuration, its warps over the group elements; with theta_h of g s,
// sigma_h = sign(Re theta_h) and r_h = exp(-2 sigma_h theta_h),
//   log 2 cosh theta_h = sigma_h theta_h + log(1 + r_h),   tanh theta_h = sigma_h (1 - r_h) / (1 + r_h),
// so an amplitude takes one exponential and one sine pair per hidden unit and one logarithm of
// prod (1 + r_h), and the ratio psi_base(g s') / psi_base(g s) of a connected configuration is the
// product of factors of nqs_local_energy.cu, here from tables over all pairs of sites (g maps a
// bond onto a pair).  The FP64 pipe (a warp instruction per 16 clocks and SM) bounds all of it.
//
// Measured (kagome 2x2, 8 elements, complex RBM M = 64, 1024 samples): local energies 308 us, complex
// gradient 165 us; kagome 3x3, 18 elements, M = 40, 500 configurations: log-amplitudes 133 us,
// gradient 194 us; before, with log 2 cosh of every unit of every amplitude and one warp per
// configuration: 3811, 625, 360 and 866 us.
#include <math.h>

#include "nqs_amp.cuh"

namespace nqs {

namespace {

constexpr double kPairRange = 350.0;       // as kFlipRange of nqs_local_energy.cu
constexpr int kMaxSymSmem = 160 * 1024;

__device__ __forceinline__ double sflip(double v, uint64_t bits, int i) {
    return __longlong_as_double(__double_as_longlong(v) ^ (long long)(((bits >> i) & 1ull) << 63));
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}

// prod (1 + r) runs down to 0.03^M and below (hidden biases near i pi / 2, where cosh acts as i sinh), past
// the range of a double at M = 144: log-amplitudes and gradients take factors 2^512 out of it below
// 2^-400 (e counts them; tested by exponent fields after every eighth unit: |1 + r_h| is 2^-62 at least, as cos of a double), energies leave a configuration with an element below kProdMin to the logarithms.
__device__ __forceinline__ void lift(double2 &P, int &e) {
    if (max(__double2hiint(P.x) & 0x7fffffff, __double2hiint(P.y) & 0x7fffffff) < (1023 - 400) << 20) {
        P.x *= 0x1p512;
        P.y *= 0x1p512;
        e++;
    }
}
// No product of the energies that matters in the sum underflows above it: a partial product below 1e-308 times
// the others' 2^256 e^350 at most is 1e-19 of 1e-60.
constexpr double kProdMin = 1e-60;
// A sum over the group that cancels to this share of its terms is rounding (a node: an element of the other
// sign maps the configuration to itself).  Energies leave it to the logarithms too, and amplitudes to the same sums:
// the residues of psi(s) and of its connected configurations, nodes as well, then have finite ratios, where sums in
// another order come out as 0 ten times as often and the ratios are infinite.
constexpr double kNodeMin = 1e-12;

__host__ __device__ inline int pair_rows(int N) { return N * (N - 1) / 2 + N; }
// row of the pair i < j, or of the single site i (j < 0)
__device__ __forceinline__ int pair_row(int N, int i, int j) {
    return j < 0 ? N * (N - 1) / 2 + i : i * (2 * N - i - 1) / 2 + (j - i - 1);
}

// exp(D_h), exp(-D_h) with D = 2 (W_i - W_j) (2 W_i for a single site) per hidden unit, and of the
// visible biases in column M; range_ok as in k_flip_tables.  One warp per row.
template <bool CPLX>
__global__ void __launch_bounds__(128) k_sym_pair_tables(DevAnsatz a, int rows, double *tab, int *range_ok) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= rows) return;
    constexpr int W = CPLX ? 4 : 2;
    const int M = a.M, N = a.N, np = N * (N - 1) / 2;
    int i = row - np, j = -1;
    if (row < np) {
        i = 0;
        j = row;
        while (j >= N - 1 - i) {
            j -= N - 1 - i;
            i++;
        }
        j += i + 1;
    }
    const double *aR = a.p, *aI = a.p + crbm_pr(a);
    double sum = 0.0;
    for (int h = lane; h <= M; h += 32) {
        double x = h < M ? a.wtr[(long)i * M + h] : aR[i], y = 0.0;
        if (j >= 0) x -= h < M ? a.wtr[(long)j * M + h] : aR[j];
        if (CPLX) {
            y = h < M ? a.wti[(long)i * M + h] : aI[i];
            if (j >= 0) y -= h < M ? a.wti[(long)j * M + h] : aI[j];
        }
        x *= 2.0;
        y *= 2.0;
        const double ep = exp(x), em = exp(-x);
        double *t = tab + ((size_t)row * (M + 1) + h) * W;
        if (CPLX) {
            double sn, cs;
            sincos(y, &sn, &cs);
            t[0] = ep * cs;
            t[1] = ep * sn;
            t[2] = em * cs;
            t[3] = -em * sn;
        } else {
            t[0] = ep;
            t[1] = em;
        }
        sum += fabs(x);
    }
    sum = warp_sum(sum);
    if (lane == 0) range_ok[row] = sum <= kPairRange;
}

// Shared memory of a block: per element the hidden units' values (r or tanh), the inverse of
// prod (1 + r), log|psi|, arg, weight, permuted configuration, signs of Re theta.
struct SymSmem {
    size_t val, pinv, lp, ag, w, pb, neg, inv, list, num, total;
};
__host__ __device__ inline SymSmem sym_smem(int G, int N, int M, int nm, int warps, bool vals) {
    SymSmem o;
    size_t p = 0;
    o.val = p;
    p += vals ? (size_t)G * M * 16 : 0;
    o.pinv = p;
    p += (size_t)G * 16;
    o.w = p;
    p += (size_t)G * 16;
    o.lp = p;
    p += (size_t)G * 8;
    o.ag = p;
    p += (size_t)G * 8;
    o.pb = p;
    p += (size_t)G * 8;
    o.num = p;
    p += (size_t)warps * nm * 8;
    o.neg = p;
    p += (size_t)G * 32;
    o.list = p;
    p += (size_t)(nm + 3) / 4 * 8;
    o.inv = p;
    p += nm ? (size_t)G * N : 0;
    o.total = (p + 15) / 16 * 16;
    return o;
}

// The configurations g s of all elements, by the whole block (the caller synchronises).
__device__ __forceinline__ void sym_configs(const DevAmp &A, uint64_t s, unsigned char *smb, const SymSmem &L) {
    for (int g = threadIdx.x >> 5; g < A.G; g += blockDim.x >> 5) {
        const uint64_t pb = permute_bits(s, A.perm + (long)g * A.a.N, A.a.N);
        if ((threadIdx.x & 31) == 0) ((uint64_t *)(smb + L.pb))[g] = pb;
    }
}

// The amplitudes of elements g0 .. g0 + 3 by one warp, eight lanes an element: prod (1 + r_h), the sums
// visible + sigma_h theta_h, and per hidden unit r_h (VALS = 1, with the signs of Re theta) or
// tanh theta_h (VALS = 2).
template <int VALS, bool CPLX>
__device__ __forceinline__ void sym_elements(const DevAmp &A, int g0, unsigned char *smb, const SymSmem &L) {
    const DevAnsatz &a = A.a;
    const int lane = threadIdx.x & 31, sl = lane & 7, g = g0 + (lane >> 3), M = a.M, N = a.N;
    const bool in = g < A.G;
    const long Pr = CPLX ? crbm_pr(a) : 0;
    const uint64_t pb = in ? ((const uint64_t *)(smb + L.pb))[g] : 0;
    double2 *val = (double2 *)(smb + L.val) + (size_t)g * M;
    unsigned char *neg = smb + L.neg + 32 * (size_t)g;              // bit h % 8 of byte h / 8
    double lr = 0.0, li = 0.0;
    double2 P = make_double2(1.0, 0.0);
    int pe = 0;
    if (in)
        for (int i = sl; i < N; i += 8) {
            lr += sflip(a.p[i], pb, i);
            if (CPLX) li += sflip(a.p[Pr + i], pb, i);
        }
    for (int j = 0; j * 8 < M; j++) {
        const int h = sl + 8 * j;
        double xr = 0.0, xi = 0.0;
        if (in && h < M) {
            xr = a.p[N + h];
            if (CPLX) xi = a.p[Pr + N + h];
            for (int i = 0; i < N; i++) {
                xr += sflip(a.wtr[(long)i * M + h], pb, i);
                if (CPLX) xi += sflip(a.wti[(long)i * M + h], pb, i);
            }
            const bool n = xr < 0.0;
            // r is kept for factors X of up to exp(350), so it has to be exact to its own size: from exp below 1/2,
            // from expm1, which the sums 1 + r and 1 - r take as it is, above (with exp there too the energies at weights
            // of 0.05 were 10 % further off; both functions cost the kernel 7 %).  (NaN for an infinite theta)
            double em1, e;
            if (VALS == 1 && fabs(xr) > 0.34657359) {
                e = exp(-2.0 * fabs(xr));
                em1 = e - 1.0;
            } else {
                em1 = expm1(-2.0 * fabs(xr));
                e = 1.0 + em1;
            }
            em1 += xr - xr;
            const double ep1 = 2.0 + em1;
            lr += fabs(xr);
            if (CPLX) {
                li += n ? -xi : xi;
                double sn, cs;
                sincos(xi, &sn, &cs);
                const double es = e * sn, u = 2.0 * es * sn;          // e (1 - cos 2y)
                const double v = (n ? 2.0 : -2.0) * es * cs;          // Im r
                const double2 d = make_double2(ep1 - u, v);           // 1 + r
                if (VALS == 1) val[h] = make_double2(e - u, v);
                if (VALS == 2) {
                    const double f = (n ? -1.0 : 1.0) / fma(d.x, d.x, d.y * d.y);
                    const double2 t = cmul(make_double2(u - em1, -v), make_double2(d.x, -d.y));
                    val[h] = make_double2(t.x * f, t.y * f);
                }
                P = cmul(P, d);
                if (VALS != 1 && (j & 7) == 7) lift(P, pe);
            } else {
                if (VALS == 1) val[h] = make_double2(e, 0.0);
                if (VALS == 2) val[h] = make_double2((n ? em1 : -em1) / ep1, 0.0);
                P.x *= ep1;
            }
        }
        if (VALS == 1) {
            const uint32_t b = __ballot_sync(0xffffffffu, xr < 0.0) >> (lane & 24);
            if (in && sl == 0) neg[j] = (unsigned char)b;
        }
    }
    if (CPLX && VALS != 1) lift(P, pe);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, P.x, o);
        if (CPLX) P = cmul(P, make_double2(x, __shfl_xor_sync(0xffffffffu, P.y, o)));
        else P.x *= x;
        lr += __shfl_xor_sync(0xffffffffu, lr, o);
        if (CPLX) li += __shfl_xor_sync(0xffffffffu, li, o);
        if (CPLX && VALS != 1) {
            pe += __shfl_xor_sync(0xffffffffu, pe, o);
            lift(P, pe);
        }
    }
    if (pe > 0) lr -= (double)pe * 354.89135644669200;              // 512 ln 2
    if (in && sl == 0) {
        ((double *)(smb + L.lp))[g] = lr;
        ((double *)(smb + L.ag))[g] = li;
        ((double2 *)(smb + L.pinv))[g] = P;
    }
}

// Weights w_g = chi_g exp(lp_g - max + i arg_g) by one warp, an element a lane (inner Marshall layers
// included; INV: pinv becomes 1 / prod (1 + r)); returns max and sum_g w_g (all lanes).  out, when given, says that
// the sum cancels to kNodeMin, or (INV) that a prod (1 + r) is below kProdMin or NaN.
template <bool INV, bool CPLX>
__device__ __forceinline__ double sym_weights(const DevAmp &A, unsigned char *smb, const SymSmem &L, double2 &sum,
                                              bool *out = nullptr) {
    const int lane = threadIdx.x & 31;
    double *lp = (double *)(smb + L.lp), *ag = (double *)(smb + L.ag);
    double2 *w = (double2 *)(smb + L.w), *pinv = (double2 *)(smb + L.pinv);
    const uint64_t *pb = (const uint64_t *)(smb + L.pb);
    double mx = -1e300;
    bool low = false;
    for (int g = lane; g < A.G; g += 32) {
        const double2 P = pinv[g];
        // |P| <= 2^256, and at least 2^-400 or (INV) not used below kProdMin: its square stays in range
        const double n2 = CPLX ? fma(P.x, P.x, P.y * P.y) : P.x * P.x;
        if (INV) low = low || !(n2 >= kProdMin * kProdMin);
        lp[g] += CPLX ? 0.5 * log(n2) : log(P.x);
        ag[g] = apply_marshall(ag[g] + (CPLX ? atan2(P.y, P.x) : 0.0), pb[g], A.n_inner, A.inner_mask);
        if (INV) pinv[g] = CPLX ? make_double2(P.x / n2, -P.y / n2) : make_double2(1.0 / P.x, 0.0);
        mx = fmax(mx, lp[g]);
    }
    mx = warp_max(mx);
    double sr = 0.0, si = 0.0, sa = 0.0;
    for (int g = lane; g < A.G; g += 32) {
        const double m = A.chars[g] * exp(lp[g] - mx);
        double sn, cs;
        sincos(ag[g], &sn, &cs);
        w[g] = make_double2(m * cs, m * sn);
        sr += m * cs;
        si += m * sn;
        sa += fabs(m);
    }
    sum = make_double2(warp_sum(sr), warp_sum(si));
    if (out) {
        sa = warp_sum(sa);
        *out = __any_sync(0xffffffffu, low) || !(fabs(sum.x) > kNodeMin * sa);
    }
    return mx;
}

// A node's amplitude, by the sums of the other programs' kernels.
__device__ __noinline__ void node_amplitude(const DevAmp &A, uint64_t s, double &la, double &ar) {
    warp_amp_eval(A, s, la, ar, nullptr);
}

template <bool CPLX>
__global__ void k_sym_log_amp(DevAmp A, const uint64_t *__restrict__ bits, double *la, double *ar) {
    extern __shared__ __align__(16) unsigned char smb[];
    const int warp = threadIdx.x >> 5, NW = blockDim.x >> 5, b = blockIdx.x;
    const SymSmem L = sym_smem(A.G, A.a.N, A.a.M, 0, NW, false);
    const uint64_t s = bits[b];
    sym_configs(A, s, smb, L);
    __syncthreads();
    for (int g = 4 * warp; g < A.G; g += 4 * NW) sym_elements<0, CPLX>(A, g, smb, L);
    __syncthreads();
    if (warp != 0) return;
    double2 sum;
    bool node;
    const double mx = sym_weights<false, CPLX>(A, smb, L, sum, &node);
    double l, p;
    if (node) {
        node_amplitude(A, s, l, p);
    } else {
        l = log(fabs(sum.x)) + mx - 0.5 * log((double)A.G);
        p = apply_marshall(sum.x < 0.0 ? kPi : 0.0, s, A.n_outer, A.outer_mask);
    }
    if ((threadIdx.x & 31) == 0) {
        if (la) la[b] = l;
        if (ar) ar[b] = p;
    }
}

// mode 1: real weights w_g = chi_g cos(arg_g) e^lp_g / sum and the real-projected base rows
// (src/nqs/nqs_symproj.c:82-155); mode 2: complex weights and the holomorphic rows (:157-261).
template <bool CPLX>
__global__ void k_sym_gradient(DevAmp A, const uint64_t *__restrict__ bits, int mode, double *O, double *Oi) {
    extern __shared__ __align__(16) unsigned char smb[];
    const int tid = threadIdx.x, warp = tid >> 5, NW = blockDim.x >> 5, b = blockIdx.x, nt = blockDim.x;
    const DevAnsatz &a = A.a;
    const int N = a.N, M = a.M, G = A.G;
    const SymSmem L = sym_smem(G, N, M, 0, NW, true);
    const long P = a.P, Pr = CPLX ? crbm_pr(a) : P;
    const uint64_t s = bits[b];
    sym_configs(A, s, smb, L);
    __syncthreads();
    for (int g = 4 * warp; g < G; g += 4 * NW) sym_elements<2, CPLX>(A, g, smb, L);
    __syncthreads();
    double2 *w = (double2 *)(smb + L.w), *val = (double2 *)(smb + L.val);
    const uint64_t *pb = (const uint64_t *)(smb + L.pb);
    __shared__ int zero;
    if (warp == 0) {
        double2 sum;
        sym_weights<false, CPLX>(A, smb, L, sum);
        if (mode == 1) sum.y = 0.0;
        const double d2 = fma(sum.x, sum.x, sum.y * sum.y);
        for (int g = tid; g < G; g += 32)
            w[g] = mode == 1 ? make_double2(w[g].x / sum.x, 0.0)
                             : make_double2((w[g].x * sum.x + w[g].y * sum.y) / d2, (w[g].y * sum.x - w[g].x * sum.y) / d2);
        if (tid == 0) zero = mode == 1 ? sum.x == 0.0 : d2 == 0.0;
    }
    __syncthreads();
    double *o = O + (size_t)b * P, *oi = Oi ? Oi + (size_t)b * P : nullptr;
    if (zero) {                                              // a node of the projected state: zero row
        for (long k = tid; k < P; k += nt) {
            o[k] = 0.0;
            if (oi) oi[k] = 0.0;
        }
        return;
    }
    // d log psi / d theta_k = x + i y of the real parameter k, and of its imaginary partner: i (x + i y)
    auto put = [&](long k, double x, double y) {
        o[k] = x;
        if (mode == 2) oi[k] = y;
        if (CPLX) {
            o[Pr + k] = -y;
            if (mode == 2) oi[Pr + k] = x;
        }
    };
    for (int e = tid; e < G * M; e += nt) {
        const double2 wg = w[e / M];
        val[e] = mode == 1 ? make_double2(wg.x * val[e].x, wg.x * val[e].y) : cmul(wg, val[e]);
    }
    for (int i = tid; i < N; i += nt) {
        double x = 0.0, y = 0.0;
        for (int g = 0; g < G; g++) {
            x += sflip(w[g].x, pb[g], i);
            y += sflip(w[g].y, pb[g], i);
        }
        put(i, x, mode == 1 ? 0.0 : y);
    }
    __syncthreads();
    for (int e = tid; e < M * (N + 1); e += nt) {            // hidden biases, then the weights
        const int h = e < M ? e : (e - M) / N, i = e < M ? -1 : (e - M) % N;
        double x = 0.0, y = 0.0;
        for (int g = 0; g < G; g++) {
            const double2 t = val[g * M + h];
            x += i < 0 ? t.x : sflip(t.x, pb[g], i);
            if (CPLX || mode == 2) y += i < 0 ? t.y : sflip(t.y, pb[g], i);
        }
        put(N + e, x, y);
    }
}

// Local energies; L, J as in k_local_prod.
template <int LN, int J, bool CPLX>
__global__ void k_sym_energy(DevAmp A, DevHam H, const uint64_t *__restrict__ bits, double *__restrict__ Er,
                             double *__restrict__ Ei, const double *__restrict__ tab, const int *__restrict__ range_ok,
                             int rows, int nm, int *done) {
    extern __shared__ __align__(16) unsigned char smb[];
    constexpr int W = CPLX ? 4 : 2, GR = 32 / LN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, NW = blockDim.x >> 5, b = blockIdx.x;
    const int sl = lane % LN, sg = lane / LN;
    const DevAnsatz &a = A.a;
    const int N = a.N, M = a.M, G = A.G;
    bool ok = true;
    for (int k = tid; k < rows; k += blockDim.x) ok = ok && range_ok[k] != 0;
    ok = __syncthreads_and(ok);
    if (!ok) {                                               // run by k_local_generic
        if (tid == 0) done[b] = 0;
        return;
    }
    const SymSmem L = sym_smem(G, N, M, nm, NW, true);
    unsigned char *inv = smb + L.inv;
    unsigned short *list = (unsigned short *)(smb + L.list);
    double *num = (double *)(smb + L.num);
    __shared__ int s_n, s_sum1, s_sum2, s_out;
    __shared__ double s_psi0;
    const uint64_t s = bits[b];
    const bool tfim = H.kind == NQS_HAM_TFIM;
    for (int e = tid; e < G * N; e += blockDim.x) inv[e / N * N + A.perm[e]] = (unsigned char)(e % N);
    if (warp == NW - 1) {                                    // connected configurations, as in k_local_prod
        int n = 0, sum1 = 0, sum2 = 0;
        for (int m0 = 0; m0 < nm; m0 += 32) {
            const int m = m0 + lane;
            int u = m, v = -1;
            if (!tfim && m < nm) {
                const int *bd = m < H.nb1 ? H.b1 + 2 * m : H.b2 + 2 * (m - H.nb1);
                u = bd[0];
                v = bd[1];
            }
            const bool anti = m < nm && (tfim || (((s >> u) ^ (s >> v)) & 1ull));
            const uint32_t am = __ballot_sync(0xffffffffu, anti);
            if (!tfim) {
                const uint32_t in = __ballot_sync(0xffffffffu, m < nm), g1 = __ballot_sync(0xffffffffu, m < H.nb1);
                sum1 += __popc(g1) - 2 * __popc(am & g1);
                sum2 += __popc(in & ~g1) - 2 * __popc(am & ~g1);
            }
            if (anti) list[n + __popc(am & ((1u << lane) - 1))] = (unsigned short)m;
            n += __popc(am);
        }
        if (tfim)
            for (int m0 = 0; m0 < H.nb1; m0 += 32) {
                const int k = m0 + lane;
                const bool in = k < H.nb1, anti = in && (((s >> H.b1[2 * k]) ^ (s >> H.b1[2 * k + 1])) & 1ull);
                sum1 += __popc(__ballot_sync(0xffffffffu, in)) - 2 * __popc(__ballot_sync(0xffffffffu, anti));
            }
        if (lane == 0) {
            s_n = n;
            s_sum1 = sum1;
            s_sum2 = sum2;
        }
    }
    sym_configs(A, s, smb, L);
    __syncthreads();
    for (int g = 4 * warp; g < G; g += 4 * NW) sym_elements<1, CPLX>(A, g, smb, L);
    for (int c = lane; c < nm; c += 32) num[warp * nm + c] = 0.0;
    __syncthreads();
    double2 *w = (double2 *)(smb + L.w);
    if (warp == 0) {
        double2 sum;
        bool out;
        sym_weights<true, CPLX>(A, smb, L, sum, &out);
        if (lane == 0) {
            s_psi0 = sum.x;
            s_out = out;
            done[b] = !out;
        }
        const double2 *pinv = (const double2 *)(smb + L.pinv);
        __syncwarp();
        for (int g = lane; g < G; g += 32) w[g] = cmul(w[g], pinv[g]);
    }
    __syncthreads();
    if (s_out) return;
    const int n = s_n;
    auto sites = [&](int m, int &u, int &v) {
        if (tfim) {
            u = m;
            v = -1;
        } else {
            const int *bd = m < H.nb1 ? H.b1 + 2 * m : H.b2 + 2 * (m - H.nb1);
            u = bd[0];
            v = bd[1];
        }
    };
    for (int g = warp; g < G; g += NW) {
        const uint64_t pb = ((const uint64_t *)(smb + L.pb))[g];
        const double2 *val = (const double2 *)(smb + L.val) + (size_t)g * M;
        const unsigned char *negs = smb + L.neg + 32 * (size_t)g;
        int par0 = 0;
        for (int m = 0; m < A.n_inner; m++) par0 += __popcll(pb & A.inner_mask[m]) & 1;
        double rr[J], ri[J];
        uint32_t neg = 0;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const int h = sl + LN * j;
            rr[j] = ri[j] = 0.0;
            if (h < M) {
                rr[j] = val[h].x;
                if (CPLX) ri[j] = val[h].y;
                neg |= ((negs[h >> 3] >> (h & 7)) & 1u) << j;
            }
        }
        const double2 wg = w[g];
        // pair row and the spin at its first site (1: down) of configuration c of this element
        auto element_row = [&](int c, int &row, int &down, uint64_t &flip) {
            int u, v;
            sites(list[c], u, v);
            int i = inv[g * N + u], j = v >= 0 ? inv[g * N + v] : -1;
            if (j >= 0 && j < i) {
                const int t = i;
                i = j;
                j = t;
            }
            row = pair_row(N, i, j);
            down = (int)((pb >> i) & 1ull);
            flip = (1ull << i) | (j >= 0 ? 1ull << j : 0ull);
        };
        for (int c0 = 0; c0 < n; c0 += 32) {
            double2 keep = make_double2(0.0, 0.0);
#pragma unroll 1
            for (int k = 0; k < LN && c0 + k * GR < n; k++) {
                const int c = c0 + k * GR + sg;
                double2 p = make_double2(1.0, 0.0);
                if (c < n) {
                    int row, down;
                    uint64_t flip;
                    element_row(c, row, down, flip);
                    const double *rp = tab + (size_t)row * (M + 1) * W;
                    const uint32_t sel = down ? ~neg : neg;
#pragma unroll
                    for (int j = 0; j < J; j++) {
                        const int h = sl + LN * j;
                        if (h < M) {
                            const bool q = (sel >> j) & 1u;
                            if (CPLX) {
                                const double2 *t = (const double2 *)(rp + (size_t)h * W);
                                const double2 Y = t[q ? 0 : 1], X = t[q ? 1 : 0];
                                p = cmul(p, make_double2(fma(X.x, rr[j], fma(-X.y, ri[j], Y.x)),
                                                         fma(X.x, ri[j], fma(X.y, rr[j], Y.y))));
                            } else {
                                const double2 t = *(const double2 *)(rp + (size_t)h * W);
                                p.x *= q ? fma(t.y, rr[j], t.x) : fma(t.x, rr[j], t.y);
                            }
                        }
                    }
                }
#pragma unroll
                for (int o = LN / 2; o > 0; o >>= 1) {
                    const double x = __shfl_xor_sync(0xffffffffu, p.x, o);
                    if (CPLX) p = cmul(p, make_double2(x, __shfl_xor_sync(0xffffffffu, p.y, o)));
                    else p.x *= x;
                }
                if (sl == k) keep = p;
            }
            const int c = c0 + sl * GR + sg;
            if (c < n) {
                int row, down;
                uint64_t flip;
                element_row(c, row, down, flip);
                const double *t = tab + ((size_t)row * (M + 1) + M) * W;
                int par = -par0;
                for (int m = 0; m < A.n_inner; m++) par += __popcll((pb ^ flip) & A.inner_mask[m]) & 1;
                const int q = down ? 0 : 1;
                double x;
                if (CPLX) x = cmul(cmul(keep, wg), ((const double2 *)t)[q]).x;
                else x = keep.x * wg.x * t[q];
                num[warp * nm + c] += (par & 1) ? -x : x;
            }
        }
    }
    __syncthreads();
    if (warp != 0) return;
    const int par0 = marshall_count(A, s);
    const double psi0 = s_psi0, c1 = tfim ? -H.Gamma : 0.5 * H.Jxy, c2 = 0.5 * H.J2;
    double off = 0.0;
    for (int c = lane; c < n; c += 32) {
        const int m = list[c];
        double x = 0.0;
        for (int q = 0; q < NW; q++) x += num[q * nm + c];
        int u, v;
        sites(m, u, v);
        const uint64_t s2 = s ^ (1ull << u) ^ (v >= 0 ? 1ull << v : 0ull);
        const double cf = m < H.nb1 || tfim ? c1 : c2;
        off = fma(((marshall_count(A, s2) - par0) & 1) ? -cf : cf, x, off);
    }
    off = warp_sum(off);
    if (lane == 0) {
        double diag = tfim ? -H.J * (double)s_sum1 : 0.25 * H.Jz * (double)s_sum1;
        if (H.nb2 > 0) diag += 0.25 * H.J2 * (double)s_sum2;
        if (Er) Er[b] = diag + off / psi0;
        if (Ei) Ei[b] = 0.0;
    }
}

bool sym_base(const DevAmp &A) { return A.G > 0 && (A.a.kind == KIND_RBM || A.a.kind == KIND_CRBM) && A.a.M <= 32 * kMaxJ; }

// Warps of a block: four elements a warp in the amplitudes, but an element a warp in the energies.
int sym_warps(int G) { return G < 8 ? G : 8; }
int amp_warps(int G) { return G < 32 ? (G + 3) / 4 : 8; }

template <typename K>
bool big_smem(K k, size_t bytes) {
    return bytes <= 48 * 1024 ||
           NQS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

}  // namespace

// One element uses 8 lanes of a warp where the kernel before takes a warp a configuration: amplitudes of one element
// (two of the complex RBM) and gradients of one stay there.  Measured, 3000 configurations, 64 units, complex: one
// element 131 us a call there and 216 us here, two 202 and 216, three 278 and 214; real: two 153 and 130; gradient
// of one configuration, 160 units: one element 110 and 121, two 184 and 123.
bool sym_log_amp_capable(const DevAmp &A) {
    return sym_base(A) && A.G >= (A.a.kind == KIND_CRBM ? 3 : 2) && sym_smem(A.G, A.a.N, A.a.M, 0, 8, false).total <= kMaxSymSmem;
}

bool launch_sym_log_amp(const DevAmp &A, const uint64_t *bits, int B, double *la, double *ar) {
    const int NW = amp_warps(A.G);
    const size_t sm = sym_smem(A.G, A.a.N, A.a.M, 0, NW, false).total;
    NQS_LAUNCH("log_amp_symproj");
    if (A.a.kind == KIND_CRBM) {
        if (!big_smem(k_sym_log_amp<true>, sm)) return false;
        k_sym_log_amp<true><<<B, 32 * NW, sm, ctx().stream>>>(A, bits, la, ar);
    } else {
        if (!big_smem(k_sym_log_amp<false>, sm)) return false;
        k_sym_log_amp<false><<<B, 32 * NW, sm, ctx().stream>>>(A, bits, la, ar);
    }
    return NQS_CUDA(cudaGetLastError());
}

bool sym_gradient_capable(const DevAmp &A) {
    return sym_base(A) && A.G >= 2 && sym_smem(A.G, A.a.N, A.a.M, 0, 8, true).total <= kMaxSymSmem;
}

// mode 1: real-projected rows O; mode 2: holomorphic rows (O, Oi).
bool launch_sym_gradient(const DevAmp &A, const uint64_t *bits, int B, int mode, double *O, double *Oi) {
    const int NW = 8;
    const size_t sm = sym_smem(A.G, A.a.N, A.a.M, 0, NW, true).total;
    NQS_LAUNCH(mode == 1 ? "symproj_gradient" : "symproj_gradient_complex");
    if (A.a.kind == KIND_CRBM) {
        if (!big_smem(k_sym_gradient<true>, sm)) return false;
        k_sym_gradient<true><<<B, 32 * NW, sm, ctx().stream>>>(A, bits, mode, O, Oi);
    } else {
        if (!big_smem(k_sym_gradient<false>, sm)) return false;
        k_sym_gradient<false><<<B, 32 * NW, sm, ctx().stream>>>(A, bits, mode, O, Oi);
    }
    return NQS_CUDA(cudaGetLastError());
}

bool sym_energy_capable(const DevAmp &A, const DevHam &H) {
    const int nm = H.kind == NQS_HAM_TFIM ? H.N : H.nb1 + H.nb2;
    return sym_base(A) && nm > 0 && sym_smem(A.G, A.a.N, A.a.M, nm, 8, true).total <= kMaxSymSmem;
}

// Local energies of the configurations; done[b] (device) is 0 where weights out of range, a small product or a
// node left one to k_local_generic.
bool launch_sym_energy(const DevAmp &A, const DevHam &H, const uint64_t *bits, int B, double *Er, double *Ei,
                       int **done) {
    static DevBuf<double> tab;
    static DevBuf<int> flags;
    const int N = A.a.N, M = A.a.M, rows = pair_rows(N), nm = H.kind == NQS_HAM_TFIM ? H.N : H.nb1 + H.nb2;
    const bool cx = A.a.kind == KIND_CRBM;
    if (!tab.ensure((size_t)rows * (M + 1) * (cx ? 4 : 2)) || !flags.ensure((size_t)rows + B)) return false;
    cudaStream_t st = ctx().stream;
    *done = flags.p + rows;
    {
        NQS_LAUNCH("symproj_tables");
        if (cx) k_sym_pair_tables<true><<<(rows + 3) / 4, 128, 0, st>>>(A.a, rows, tab.p, flags.p);
        else k_sym_pair_tables<false><<<(rows + 3) / 4, 128, 0, st>>>(A.a, rows, tab.p, flags.p);
    }
    const int NW = sym_warps(A.G);
    const size_t sm = sym_smem(A.G, N, M, nm, NW, true).total;
    NQS_LAUNCH("local_symproj");
#define NQS_CASE(LL, JJ)                                                                                            \
    case JJ:                                                                                                        \
        if (cx) {                                                                                                   \
            if (!big_smem(k_sym_energy<LL, JJ, true>, sm)) return false;                                            \
            k_sym_energy<LL, JJ, true><<<B, 32 * NW, sm, st>>>(A, H, bits, Er, Ei, tab.p, flags.p, rows, nm, *done); \
        } else {                                                                                                    \
            if (!big_smem(k_sym_energy<LL, JJ, false>, sm)) return false;                                           \
            k_sym_energy<LL, JJ, false><<<B, 32 * NW, sm, st>>>(A, H, bits, Er, Ei, tab.p, flags.p, rows, nm, *done); \
        }                                                                                                           \
        break;
    if (M <= 64) {
        switch ((M + 15) / 16 * 2) { NQS_CASE(8, 2) NQS_CASE(8, 4) NQS_CASE(8, 6) NQS_CASE(8, 8) }
    } else if (M <= 128) {
        switch ((M + 31) / 32 * 2) { NQS_CASE(16, 6) NQS_CASE(16, 8) }
    } else {
        switch ((M + 63) / 64 * 2) { NQS_CASE(32, 6) NQS_CASE(32, 8) }
    }
#undef NQS_CASE
    return NQS_CUDA(cudaGetLastError());
}

}  // namespace nqs
