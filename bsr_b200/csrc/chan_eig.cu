// The channel eigenproblems of diag_hd as the library's own batched kernels.
//
// Reference: src/bsr/BSR_HD3/diag_hd.f90:82-111 -- for every channel, LAPACK
// DSYGV('V','U') of (H_ii, S_ii) restricted to the splines l+2..ns (or ns-1).
// Here, for all channels at once (40 channels of n ~ 200 at the config-2 size):
//   1. chan_tridiag_kernel: the banded Cholesky S = L L^T (bandwidth ks), the
//      reduction C = L^-1 H L^-T by banded substitutions, and the Householder
//      tridiagonalisation of C (LAPACK dsytd2's lower-triangle convention:
//      C = Q T Q^T, Q = H_0 H_1 ... H_{n-3}) on C packed in shared memory;
//   2. chan_bisect_kernel: every eigenvalue of T by bisection on Sturm counts
//      (to a relative width of 2 eps, as far as the counts resolve);
//   3. chan_invit_kernel: its eigenvector by inverse iteration (LU of T - lambda I
//      with partial pivoting, three solves from a fixed pseudo-random start);
//   4. (host) symmetric orthogonalisation of the eigenvectors, twice:
//      Y <- Y (3/2 I - 1/2 Y^T Y) as batched FP64 tensor-core GEMMs.  Inverse
//      iteration leaves eigenvectors of close eigenvalues non-orthogonal by
//      ~eps ||T|| / gap; mixing y_j with y_i by that amount changes the residual
//      of y_j by ~eps ||T||, so the pairs stay accurate and become orthonormal;
//   5. chan_q_kernel: z = Q y; chan_solve_kernel: x = L^-T z.
// The eigenvectors come out S-orthonormal (x^T S x = 1) in ascending order of
// their eigenvalues, as DSYGV returns them (up to the sign of each vector).
#include <algorithm>
#include <cfloat>

#include "ctx.h"
#include "dgemm.h"

namespace bsrg {

constexpr int CH_THREADS = 512, CH_WARPS = CH_THREADS / 32;
constexpr int CH_NMAX = 256;                  // rows of a channel problem (eight 32-column chunks, 16 rows a warp)
constexpr int CH_Q = CH_NMAX / 32, CH_RED = 8;

__host__ __device__ inline size_t tri(int i) { return (size_t)i * (i + 1) / 2; }

__device__ inline double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sums of four values over the warp; lanes 8 t .. 8 t + 7 get that of s[t]
__device__ inline double warp_sum4(double (&s)[4], int lane)
{
#pragma unroll
    for (int h = 2; h > 0; h >>= 1) {
        const bool up = lane & (8 * h);
#pragma unroll
        for (int t = 0; t < h; t++) {
            const double give = up ? s[t] : s[t + h], keep = up ? s[t + h] : s[t];
            s[t] = keep + __shfl_xor_sync(0xffffffffu, give, 8 * h);
        }
    }
    double v = s[0];
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// S(i, j) of the channel restricted to rows/columns s0.. (sb: band (ns, ks), lower)
__device__ inline double s_restricted(const double *sb, int ns, int ks, int s0, int i, int j)
{
    const int hi = s0 + (i > j ? i : j), lo = s0 + (i > j ? j : i);
    return hi - lo < ks ? sb[hi + (size_t)ns * (lo - hi + ks - 1)] : 0.0;
}

// solve L y = b for one column: y_i from the window of the last KS - 1 values, the newest one last (only
// its product and the division are on the chain from one row to the next)
template <int KS>
__device__ __forceinline__ double band_step(const double *Lrow, double v, double (&win)[KS])
{
#pragma unroll
    for (int t = KS - 1; t > 0; t--) v = fma(-Lrow[KS - 1 - t], win[t - 1], v);
    v /= Lrow[KS - 1];
#pragma unroll
    for (int t = KS - 2; t > 0; t--) win[t] = win[t - 1];
    win[0] = v;
    return v;
}

// What bounds it: the chain of n - 2 dependent reflectors, each with one pass over the packed triangle in
// shared memory.  The pass applies the last reflector's rank-2 update and forms the product with the new
// reflector at once (a load and a store per entry); a warp takes four rows at a time, its lanes the columns, so
// the loads meet no bank conflict (triangular numbers run through all residues of 16 too: a column read down the
// rows meets none either), the columns' part of the product stays in registers.  One warp forms the next
// reflector (all sixteen for themselves, without that barrier, cost more: they share the FP64 units).
// Measured (40 channels of 195 rows, ks 10): 1459 -> 1029 us, of which Cholesky 95 and the substitutions 70.
template <int KS>
__global__ void __launch_bounds__(CH_THREADS)
chan_tridiag_kernel(int ns, int npad, const int *__restrict__ s0v, const int *__restrict__ nsolv,
                    const double *__restrict__ hcc, const double *__restrict__ sb, double *Xg, double *Lg,
                    double *Vg, double *dg, double *eg, double *taug, int *info)
{
    extern __shared__ __align__(16) double cs[];
    const int ich = blockIdx.x, n = nsolv[ich], s0 = s0v[ich];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const size_t np2 = (size_t)npad * npad, npk = tri(npad);
    double *vw = cs;                          // the last reflector v and its w, entry by entry (16-byte pairs)
    double *Cp = vw + 2 * (size_t)npad;       // C, packed lower (row i at tri(i))
    double *Lb = Cp + npk;                    // L band: row i, column j at i*KS + (j - i + KS - 1)
    double *xs = Lb + (size_t)npad * KS;      // the reflector
    double *ps = xs + npad;                   // its product with C
    double *red = ps + npad;                  // CH_RED rows of column sums
    int *bad = (int *)(red + (size_t)CH_RED * npad);
    const double *H = hcc + ((size_t)(ich + 1) * (ich + 2) / 2 - 1) * ns * ns;
    double *X = Xg + (size_t)ich * np2;
    for (int q = tid; q < npad * KS; q += CH_THREADS) {
        const int i = q / KS, j = i - (KS - 1) + q % KS;
        Lb[q] = i < n && j >= 0 ? s_restricted(sb, ns, KS, s0, i, j) : 0.0;
    }
    for (int q = tid; q < 2 * npad; q += CH_THREADS) vw[q] = 0.0;
    if (tid == 0) *bad = 0;
    __syncthreads();
    // ---- banded Cholesky, S to L in place: one warp, column by column, the KS rows that a column reaches in
    //      registers (row i with lane i mod KS, its entry of column c in r[c mod KS]) ----
    if (w == 0) {
        double r[KS];
#pragma unroll
        for (int c = 0; c < KS; c++) r[c] = lane < KS && lane < n && c <= lane ? Lb[lane * KS + c - lane + KS - 1] : 0.0;
        for (int j0 = 0; j0 < n; j0 += KS) {
#pragma unroll
            for (int jj = 0; jj < KS; jj++) {
                const int j = j0 + jj;
                if (j < n) {
                // the row that enters after this column, columns j+1 .. j+KS
                double nr[KS];
#pragma unroll
                for (int t = 1; t <= KS; t++) nr[t - 1] = j + KS < n ? Lb[(j + KS) * KS + t - 1] : 0.0;
                double dj = __shfl_sync(0xffffffffu, r[jj], jj);
                if (!(dj > 0.0)) {               // not positive definite: flagged, kept finite
                    if (lane == 0 && *bad == 0) *bad = j + 1;
                    dj = 1.0;
                }
                const double ljj = sqrt(dj), l = lane == jj ? ljj : r[jj] / ljj;
                const int i = j + (lane >= jj ? lane - jj : lane - jj + KS);
                if (lane < KS && i < n) Lb[i * KS + j - i + KS - 1] = l;
#pragma unroll
                for (int t = 1; t < KS; t++) {
                    const int c = (jj + t) % KS;
                    r[c] = fma(-l, __shfl_sync(0xffffffffu, l, c), r[c]);
                }
                if (lane == jj) {
#pragma unroll
                    for (int t = 1; t <= KS; t++) r[(jj + t) % KS] = nr[t - 1];
                }
                }
            }
        }
    }
    __syncthreads();
    // ---- X^T = (L^-1 H)^T (thread per column of H, which is symmetric: read along its rows) ----
    constexpr int PF = 8;                         // rows fetched ahead
    for (int c = tid; c < n; c += CH_THREADS) {
        double win[KS], nx[PF];
#pragma unroll
        for (int t = 0; t < KS; t++) win[t] = 0.0;
        const double *Hc = H + (s0 + c) + (size_t)ns * s0;
#pragma unroll
        for (int u = 0; u < PF; u++) nx[u] = u < n ? Hc[(size_t)ns * u] : 0.0;
        for (int i0 = 0; i0 < n; i0 += PF) {
            double cur[PF];
#pragma unroll
            for (int u = 0; u < PF; u++) cur[u] = nx[u];
#pragma unroll
            for (int u = 0; u < PF; u++) nx[u] = i0 + PF + u < n ? Hc[(size_t)ns * (i0 + PF + u)] : 0.0;
#pragma unroll
            for (int u = 0; u < PF; u++)
                if (i0 + u < n) X[(size_t)c * npad + i0 + u] = band_step<KS>(Lb + (i0 + u) * KS, cur[u], win);
        }
    }
    __syncthreads();
    // ---- C = L^-1 X^T, lower triangle packed in shared memory ----
    for (int c = tid; c < n; c += CH_THREADS) {
        double win[KS], nx[PF];
#pragma unroll
        for (int t = 0; t < KS; t++) win[t] = 0.0;
        const double *Xc = X + c;                     // X^T(i, c)
#pragma unroll
        for (int u = 0; u < PF; u++) nx[u] = u < n ? Xc[(size_t)u * npad] : 0.0;
        for (int i0 = 0; i0 < n; i0 += PF) {
            double cur[PF];
#pragma unroll
            for (int u = 0; u < PF; u++) cur[u] = nx[u];
#pragma unroll
            for (int u = 0; u < PF; u++) nx[u] = i0 + PF + u < n ? Xc[(size_t)(i0 + PF + u) * npad] : 0.0;
#pragma unroll
            for (int u = 0; u < PF; u++)
                if (i0 + u < n) {
                    const double v = band_step<KS>(Lb + (i0 + u) * KS, cur[u], win);
                    if (i0 + u >= c) Cp[tri(i0 + u) + c] = v;
                }
        }
    }
    __syncthreads();
    // ---- Householder tridiagonalisation (dsytd2, lower); column j = 32 q + lane is a lane's q-th ----
    double *dgc = dg + (size_t)ich * npad, *egc = eg + (size_t)ich * npad, *tgc = taug + (size_t)ich * npad;
    double last = 0.0;                        // tau of the last reflector (warp 0)
    for (int i = tid; i < n; i += CH_THREADS) xs[i] = ps[i] = 0.0;
    __syncthreads();
    for (int k = 0; k < n; k++) {
        if (w == 0) {
            // p and w of the last reflector v (zero before the first): w = tau p - (tau / 2) (tau p . v) v;
            // then column k with C - v w^T - w v^T applied, x_i, i >= k
            double v[CH_Q], x[CH_Q], dot = 0.0;
#pragma unroll
            for (int q = 0; q < CH_Q; q++) {
                const int j = 32 * q + lane;
                v[q] = j < n ? xs[j] : 0.0;
                x[q] = j >= min(k, n - 2) && j < n ? last * ps[j] : 0.0;
                dot = fma(x[q], v[q], dot);
            }
            const double gam = -0.5 * last * warp_sum(dot);
            double vk = 0.0, wk = 0.0, alpha = 0.0, sigma = 0.0;
#pragma unroll
            for (int q = 0; q < CH_Q; q++) {
                const int j = 32 * q + lane;
                x[q] = fma(gam, v[q], x[q]);
                if (j < n) *reinterpret_cast<double2 *>(vw + 2 * j) = make_double2(v[q], x[q]);
            }
            __syncwarp();
            {
                const double2 t = *reinterpret_cast<const double2 *>(vw + 2 * k);
                vk = t.x;
                wk = t.y;
            }
#pragma unroll
            for (int q = 0; q < CH_Q; q++) {
                const int i = 32 * q + lane;
                const double c = i >= k && i < n ? Cp[tri(i) + k] - (v[q] * wk + x[q] * vk) : 0.0;
                x[q] = c;
                if (i >= k + 2) sigma = fma(c, c, sigma);
                if (i == k) dgc[k] = c;
                if (i == k + 1 && i < n) egc[k] = c;           // of the last two rows; else the reflector's
            }
            if (k + 2 < n) {
                sigma = warp_sum(sigma);
#pragma unroll
                for (int q = 0; q < CH_Q; q++)
                    if (q == (k + 1) >> 5) alpha = __shfl_sync(0xffffffffu, x[q], (k + 1) & 31);
                // squares near the smallest normal number have lost their bits: the column scaled by 2^500 (exact)
                double down = 1.0;
                if (fma(alpha, alpha, sigma) < 0x1p-900) {
                    down = 0x1p-500;
                    alpha *= 0x1p500;
                    sigma = 0.0;
#pragma unroll
                    for (int q = 0; q < CH_Q; q++) {
                        x[q] *= 0x1p500;
                        if (32 * q + lane >= k + 2) sigma = fma(x[q], x[q], sigma);
                    }
                    sigma = warp_sum(sigma);
                }
                double beta, scal;
                if (sigma == 0.0) {
                    last = 0.0; beta = alpha; scal = 0.0;
                } else {
                    beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
                    last = (beta - alpha) / beta;
                    scal = 1.0 / (alpha - beta);
                }
                __syncwarp();
                if (lane == 0) { egc[k] = beta * down; tgc[k] = last; }
                // the new reflector (1, x(k+2..) scal), also kept below its first entry for the back-transform
#pragma unroll
                for (int q = 0; q < CH_Q; q++) {
                    const int i = 32 * q + lane;
                    const double t = x[q] * scal;
                    if (i < n) xs[i] = i == k + 1 ? 1.0 : i > k + 1 ? t : 0.0;
                    if (i > k + 1 && i < n) Cp[tri(i) + k] = t;
                }
            } else if (lane == 0) {
                tgc[k] = 0.0;
            }
        }
        if (k + 2 >= n) continue;
        __syncthreads();
        double v[CH_Q], wv[CH_Q], x[CH_Q], acc[CH_Q];
#pragma unroll
        for (int q = 0; q < CH_Q; q++) {
            const int j = 32 * q + lane;
            v[q] = wv[q] = x[q] = acc[q] = 0.0;
            if (j > k && j < n) {             // zero up to column k: what is there stays as it is
                const double2 t = *reinterpret_cast<const double2 *>(vw + 2 * j);
                v[q] = t.x;
                wv[q] = t.y;
                x[q] = xs[j];
            }
        }
        // four rows of a warp at a time
        for (int i0 = 4 * w; i0 < n; i0 += 4 * CH_WARPS) {
            if (i0 + 3 <= k) continue;
            double sr[4], vi[4], wi[4], xi[4];
            double *row[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int i = min(i0 + t, n - 1);
                const double2 u = *reinterpret_cast<const double2 *>(vw + 2 * i);
                vi[t] = u.x;
                wi[t] = u.y;
                xi[t] = xs[i];
                row[t] = Cp + tri(i) + lane;
                sr[t] = 0.0;
            }
#pragma unroll
            for (int q = 0; q < CH_Q; q++) {
                if (32 * q > i0 + 3 || 32 * q + 31 <= k) continue;
                if (32 * q + 31 < i0 && i0 + 3 < n) {
                    // below the diagonal
                    double c[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) c[t] = row[t][32 * q];
#pragma unroll
                    for (int t = 0; t < 4; t++) c[t] = fma(-vi[t], wv[q], fma(-wi[t], v[q], c[t]));
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        row[t][32 * q] = c[t];
                        sr[t] = fma(c[t], x[q], sr[t]);
                        acc[q] = fma(c[t], xi[t], acc[q]);
                    }
                } else {
                    const int j = 32 * q + lane;
                    double c[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) c[t] = row[t][j <= i0 + t ? 32 * q : -lane];   // any of the row's
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const bool in = j <= i0 + t && i0 + t < n;
                        const double u = fma(-vi[t], wv[q], fma(-wi[t], v[q], c[t]));
                        if (in) row[t][32 * q] = u;
                        sr[t] = fma(in ? u : 0.0, x[q], sr[t]);
                        acc[q] = fma(in && j < i0 + t ? u : 0.0, xi[t], acc[q]);
                    }
                }
            }
            const double t = warp_sum4(sr, lane);
            const int i = i0 + (lane >> 3);
            if ((lane & 7) == 0 && i > k && i < n) ps[i] = t;
        }
        // the columns' part: sixteen warps' sums by way of eight rows
        if (w >= CH_RED) {
#pragma unroll
            for (int q = 0; q < CH_Q; q++)
                if (32 * q + 31 > k && 32 * q + lane < n) red[(w - CH_RED) * npad + 32 * q + lane] = acc[q];
        }
        __syncthreads();
        if (w < CH_RED) {
#pragma unroll
            for (int q = 0; q < CH_Q; q++)
                if (32 * q + 31 > k && 32 * q + lane < n) red[w * npad + 32 * q + lane] += acc[q];
        }
        __syncthreads();
        for (int j = tid; j < n; j += CH_THREADS)
            if (j > k) {
                double t = ps[j];
#pragma unroll
                for (int r = 0; r < CH_RED; r++) t += red[r * npad + j];
                ps[j] = t;
            }
        __syncthreads();
    }
    __syncthreads();
    // ---- outputs: the reflectors (packed C) and L ----
    double *Vc = Vg + (size_t)ich * npk;
    for (size_t q = tid; q < tri(n); q += CH_THREADS) Vc[q] = Cp[q];
    double *Lc = Lg + (size_t)ich * npad * KS;
    for (int q = tid; q < n * KS; q += CH_THREADS) Lc[q] = Lb[q];
    if (tid == 0) info[ich] = *bad;
}

// pseudo-random start vector entry in [-1, 1) for eigenpair j, row i (a fixed integer hash)
__device__ inline double start_entry(int i, int j)
{
    unsigned h = (unsigned)i * 0x9E3779B1u ^ ((unsigned)j * 0x85EBCA77u + 0xC2B2AE3Du);
    h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
    return (double)h * (2.0 / 4294967296.0) - 1.0;
}

// The eigenvalues of channel blockIdx.x's tridiagonal T: CB_L lanes per eigenvalue count the eigenvalues below
// CB_L points of its interval at once (Sturm counts as the sign changes of the scaled leading minors, rescaled
// every fourth row; no division), until the interval is 2 eps of its ends wide.
// What bounds it: the issue slots of the counts.  Measured (40 channels of 195 rows): 167 us; with the
// inverse iteration below 1906 -> 392 us against one thread per eigenpair for both, bisecting by ratios.
constexpr int CB_T = 256, CB_L = 8, CB_PASSES = 48;
__global__ void __launch_bounds__(CB_T)
chan_bisect_kernel(int ns, int npad, const int *__restrict__ nsolv, const double *__restrict__ dg,
                   const double *__restrict__ eg, double *Wv)
{
    __shared__ double2 ch[CH_NMAX + 4];                      // (d_i, e_{i-1}^2), scaled by 2^-q
    __shared__ double wl[CB_T / 32], wu[CB_T / 32];
    const int ich = blockIdx.x, n = nsolv[ich], n4 = (n + 3) & ~3;
    const int tid = threadIdx.x, lane = tid & 31, sub = lane % CB_L, j = (blockIdx.y * CB_T + tid) / CB_L;
    const double *d = dg + (size_t)ich * npad, *e = eg + (size_t)ich * npad;
    // Gershgorin bounds
    double gl = DBL_MAX, gu = -DBL_MAX;
    for (int i = tid; i < n; i += CB_T) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
        gl = fmin(gl, d[i] - r);
        gu = fmax(gu, d[i] + r);
    }
    for (int o = 16; o > 0; o >>= 1) {
        gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
        gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
    }
    if (lane == 0) { wl[tid >> 5] = gl; wu[tid >> 5] = gu; }
    __syncthreads();
    for (int q = 0; q < CB_T / 32; q++) { gl = fmin(gl, wl[q]); gu = fmax(gu, wu[q]); }
    const double tnorm = fmax(fabs(gl), fabs(gu));
    int ex = 0;
    if (tnorm > 0.0) frexp(tnorm, &ex);
    for (int i = tid; i < n4; i += CB_T) {
        const double f = i > 0 && i < n ? scalbn(e[i - 1], -ex) : 0.0;
        // e^2 of 2^-140 at least (a shift of 2^-70 tnorm at most) keeps the minors in range between the
        // rescalings; beyond the end minors that keep their sign
        ch[i] = i < n ? make_double2(scalbn(d[i], -ex), fmax(f * f, 0x1p-140)) : make_double2(4.0, 0.0);
    }
    __syncthreads();
    const double eps = DBL_EPSILON;
    double lo = scalbn(gl, -ex) - 4.0 * eps, hi = scalbn(gu, -ex) + 4.0 * eps;
    bool done = j >= n;
    for (int pass = 0; pass < CB_PASSES; pass++) {
        done = done || hi - lo <= 2.0 * eps * fmax(fabs(lo), fabs(hi)) + 0x1p-128;
        if (__all_sync(0xffffffffu, done)) break;
        const double x = lo + (hi - lo) * ((sub + 1) * (1.0 / (CB_L + 1)));
        double p0 = 0.0, p1 = 1.0;
        int cnt = 0;
#pragma unroll 2
        for (int i = 0; i < n4; i += 4) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const double2 c = ch[i + q];
                const double p = fma(c.x - x, p1, -(c.y * p0));
                cnt += (unsigned)(__double2hiint(p) ^ __double2hiint(p1)) >> 31;
                p0 = p1;
                p1 = p;
            }
            const int h = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
            const double r = __hiloint2double(0x7fe00000 - h, 0);
            p0 *= r;
            p1 *= r;
        }
        const unsigned above = (__ballot_sync(0xffffffffu, cnt > j) >> (lane - sub)) & ((1u << CB_L) - 1);
        const int f = above ? __ffs(above) - 1 : CB_L;
        const double xl = __shfl_sync(0xffffffffu, x, lane - sub + (f > 0 ? f - 1 : 0));
        const double xh = __shfl_sync(0xffffffffu, x, lane - sub + (f < CB_L ? f : CB_L - 1));
        if (!done) {
            if (f > 0) lo = xl;
            if (f < CB_L) hi = xh;
        }
    }
    if (sub == 0 && j < n) Wv[(size_t)ich * ns + j] = scalbn(0.5 * (lo + hi), ex);
}

// Eigenvector j = blockIdx.y*32 + lane of channel blockIdx.x's T by inverse iteration: LU of T - lambda I with
// partial pivoting (rows i, i+1 at step i), three solves.  Y (row i, column j at Y[i*npad + j], i.e. the
// transposed eigenvector matrix in column-major terms) gets the unit eigenvector, zero outside the n x n block.
// What bounds it: the chains of seven sweeps over the rows, each row with a division in four of them.  The
// multipliers and the vector stay in shared memory, the pivots of the unpivoted rows in A (npad x npad per
// channel), one bit a row says which; a pivoted row of U is (e_i, d_{i+1} - lambda, e_{i+1}) again.
// Measured (40 channels of 195 rows): 225 us.
__global__ void __launch_bounds__(32)
chan_invit_kernel(int ns, int npad, const int *__restrict__ nsolv, const double *__restrict__ dg,
                  const double *__restrict__ eg, const double *__restrict__ Wv, double *__restrict__ Yg,
                  double *__restrict__ Ag)
{
    extern __shared__ __align__(16) double cs[];
    double *d = cs, *e = d + npad, *LL = e + npad, *Yv = LL + (size_t)32 * npad;
    const int ich = blockIdx.x, n = nsolv[ich], lane = threadIdx.x, j = blockIdx.y * 32 + lane;
    const size_t np2 = (size_t)npad * npad;
    double tn = 0.0;
    for (int i = lane; i < n; i += 32) {
        d[i] = dg[(size_t)ich * npad + i];
        e[i] = i + 1 < n ? eg[(size_t)ich * npad + i] : 0.0;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + fabs(e[i]);
        tn = fmax(tn, fmax(fabs(d[i] - r), fabs(d[i] + r)));
    }
    for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
    double *Y = Yg + (size_t)ich * np2, *A = Ag + (size_t)ich * np2;
    if (j >= npad) return;
    if (j >= n) {
        for (int i = 0; i < npad; i++) Y[(size_t)i * npad + j] = 0.0;
        return;
    }
    const double lam = Wv[(size_t)ich * ns + j], tiny = tn > 0.0 ? DBL_EPSILON * tn : DBL_MIN;
    LL += lane;
    Yv += lane;
    unsigned piv[CH_Q];                          // bit i & 31 of word i >> 5: row i was exchanged
    // ---- LU ----
    double ai = d[0] - lam, ui = e[0];
#pragma unroll
    for (int q = 0; q < CH_Q; q++) {
        unsigned bits = 0;
        const int i1 = min(32 * q + 32, n - 1);
        for (int i = 32 * q; i < i1; i++) {
            const double li = e[i], di1 = d[i + 1] - lam, ui1 = e[i + 1];
            const bool sw = !(fabs(ai) >= fabs(li));
            if (!sw && ai == 0.0) ai = tiny;
            const double mlt = (sw ? ai : li) / (sw ? li : ai);
            A[(size_t)i * npad + j] = ai;
            LL[32 * i] = mlt;
            bits |= (unsigned)sw << (i & 31);
            ai = sw ? ui - mlt * di1 : di1 - mlt * ui;
            ui = sw ? -mlt * ui1 : ui1;
        }
        piv[q] = bits;
    }
    if (ai == 0.0) ai = tiny;
    const double alast = ai;
    // ---- three solves, normalised ----
    double scale = 1.0;
    for (int it = 0; it < 3; it++) {
        // forward: y = L^-1 P b, b = the start vector or the previous x * scale
        double yc = it == 0 ? start_entry(0, j) : Yv[0] * scale;
#pragma unroll
        for (int q = 0; q < CH_Q; q++) {
            const int i1 = min(32 * q + 32, n - 1);
            const unsigned bits = piv[q];
#pragma unroll 4
            for (int i = 32 * q; i < i1; i++) {
                const double yn = it == 0 ? start_entry(i + 1, j) : Yv[32 * (i + 1)] * scale, mlt = LL[32 * i];
                const bool sw = bits >> (i & 31) & 1;
                Yv[32 * i] = sw ? yn : yc;
                yc = sw ? yc - mlt * yn : yn - mlt * yc;
            }
        }
        // back: U x = y, U with two superdiagonals
        double x1 = yc / alast, x2 = 0.0, ss = x1 * x1;
        Yv[32 * (n - 1)] = x1;
#pragma unroll
        for (int q = CH_Q - 1; q >= 0; q--) {
            const unsigned bits = piv[q], prev = q > 0 ? piv[q > 0 ? q - 1 : 0] >> 31 : 0;
#pragma unroll 4
            for (int i = min(32 * q + 31, n - 2); i >= 32 * q; i--) {
                const bool sw = bits >> (i & 31) & 1;
                const bool swp = (i & 31) ? bits >> ((i & 31) - 1) & 1 : prev;     // row i - 1 was exchanged
                const double a = sw ? e[i] : A[(size_t)i * npad + j];
                const double u = sw ? d[i + 1] - lam : swp ? -LL[32 * (i > 0 ? i - 1 : 0)] * e[i] : e[i];
                const double c2 = sw ? e[i + 1] : 0.0;
                const double x = (Yv[32 * i] - u * x1 - c2 * x2) / a;
                Yv[32 * i] = x;
                ss += x * x;
                x2 = x1;
                x1 = x;
            }
        }
        scale = 1.0 / sqrt(ss);
    }
    for (int i = 0; i < n; i++) Y[(size_t)i * npad + j] = Yv[32 * i] * scale;
    for (int i = n; i < npad; i++) Y[(size_t)i * npad + j] = 0.0;
}

// M = 3/2 I - 1/2 G for the symmetric orthogonalisation step; flag if G is far from I
__global__ void chan_lowdin_kernel(int npad, const int *__restrict__ nsolv, double *G, int *flag)
{
    const int ich = blockIdx.y, n = nsolv[ich];
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)npad * npad) return;
    const int r = (int)(q % npad), c = (int)(q / npad);
    double *g = G + (size_t)ich * npad * npad + q;
    const double id = r == c ? 1.0 : 0.0;
    if (r < n && c < n && fabs(*g - id) > 1e-3) atomicExch(flag, 1);
    *g = 1.5 * id - 0.5 * *g;
}

// z = Q y for every eigenvector of the channel, in place, Q y = H_0 (H_1 (... H_{n-3} y)).  A warp takes C
// vectors at a time, a lane every 32nd row of them in registers; the reflectors are read down a column of the
// packed triangle in shared memory (no bank conflict) and no barrier is met.
// What bounds it: the dependent reflectors (a sum over the warp and an update each).
// Measured (40 channels of 195 rows): 158 us, 3098 before with one CTA per channel,
// panel after panel, and the substitution below.
template <int NQ, int C, int Q0>
__device__ __forceinline__ void q_chunk(double (&z)[NQ][C], const double *const (&col)[NQ], const double *tau, int n,
                                        int lane)
{
    // the reflectors whose first row lies in chunk Q0
    const int k0 = min(n - 3, 32 * Q0 + 30), k1 = max(0, 32 * Q0 - 1);
    double v[NQ - Q0], nv[NQ - Q0];
    auto fetch = [&](int k) {
#pragma unroll
        for (int q = Q0; q < NQ; q++) {
            const int i = 32 * q + lane;
            nv[q - Q0] = (q > Q0 || i > k + 1) && i < n ? col[q][k] : q == Q0 && i == k + 1 ? 1.0 : 0.0;
        }
    };
    if (k0 >= k1) fetch(k0);
    for (int k = k0; k >= k1; k--) {
        const double tk = tau[k];
        double s[C] = {};
#pragma unroll
        for (int q = Q0; q < NQ; q++) {
            v[q - Q0] = nv[q - Q0];
#pragma unroll
            for (int c = 0; c < C; c++) s[c] = fma(v[q - Q0], z[q][c], s[c]);
        }
        if (k > k1) fetch(k - 1);
        if (C == 4) {
            double t[4];
#pragma unroll
            for (int c = 0; c < 4; c++) t[c] = s[c < C ? c : 0];
            const double a = warp_sum4(t, lane);
#pragma unroll
            for (int c = 0; c < C; c++) s[c] = __shfl_sync(0xffffffffu, a, 8 * c);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < C; c++) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
        }
#pragma unroll
        for (int c = 0; c < C; c++) {
            const double t = tk * s[c];
#pragma unroll
            for (int q = Q0; q < NQ; q++) z[q][c] = fma(-v[q - Q0], t, z[q][c]);
        }
    }
    if constexpr (Q0 > 0) q_chunk<NQ, C, Q0 - 1>(z, col, tau, n, lane);
}

template <int NQ, int C>
__global__ void __launch_bounds__(CH_THREADS)
chan_q_kernel(int npad, const int *__restrict__ nsolv, const double *__restrict__ Vg, const double *__restrict__ taug,
              double *Yg)
{
    extern __shared__ __align__(16) double cs[];
    const int ich = blockIdx.x, n = nsolv[ich], tid = threadIdx.x, lane = tid & 31;
    const size_t npk = tri(npad);
    double *Vp = cs, *tau = Vp + npk;
    for (size_t q = tid; q < tri(n); q += CH_THREADS) Vp[q] = Vg[(size_t)ich * npk + q];
    for (int q = tid; q < n; q += CH_THREADS) tau[q] = q + 2 < n ? taug[(size_t)ich * npad + q] : 0.0;
    __syncthreads();
    double *Y = Yg + (size_t)ich * npad * npad;
    const double *col[NQ];                       // row i = 32 q + lane of the packed triangle
#pragma unroll
    for (int q = 0; q < NQ; q++) col[q] = Vp + tri(min(32 * q + lane, n - 1));
    const int groups = (n + C - 1) / C;
    for (int g = blockIdx.y * CH_WARPS + (tid >> 5); g < groups; g += gridDim.y * CH_WARPS) {
        double z[NQ][C];
#pragma unroll
        for (int q = 0; q < NQ; q++)
#pragma unroll
            for (int c = 0; c < C; c++) {
                const int i = 32 * q + lane, j = C * g + c;
                z[q][c] = i < n && j < n ? Y[(size_t)i * npad + j] : 0.0;
            }
        if (n >= 3) q_chunk<NQ, C, NQ - 1>(z, col, tau, n, lane);
#pragma unroll
        for (int q = 0; q < NQ; q++)
#pragma unroll
            for (int c = 0; c < C; c++) {
                const int i = 32 * q + lane, j = C * g + c;
                if (i < n && j < n) Y[(size_t)i * npad + j] = z[q][c];
            }
    }
}

typedef void (*chan_q_fn)(int, const int *, const double *, const double *, double *);
template <int NQ> static chan_q_fn chan_q_of(int c)
{
    return c == 2 ? chan_q_kernel<NQ, 2> : c == 4 ? chan_q_kernel<NQ, 4> : chan_q_kernel<NQ, 5>;
}

// x = L^-T z, a thread per eigenvector, rows fetched ahead
constexpr int CL_T = 64;
template <int KS>
__global__ void __launch_bounds__(CL_T)
chan_solve_kernel(int ns, int npad, const int *__restrict__ nsolv, const double *__restrict__ Lg,
                  const double *__restrict__ Zg, double *__restrict__ AA)
{
    extern __shared__ __align__(16) double cs[];
    const int ich = blockIdx.x, n = nsolv[ich], tid = threadIdx.x, c = blockIdx.y * CL_T + tid;
    // L by columns: row i of U = L^T at Ub[i KS], its diagonal last, entry i + t at KS - 1 - t
    double *Ub = cs;
    for (int q = tid; q < n * KS; q += CL_T) {
        const int i = q / KS, t = KS - 1 - q % KS;
        Ub[q] = i + t < n ? Lg[(size_t)ich * npad * KS + (size_t)(i + t) * KS + KS - 1 - t] : 0.0;
    }
    __syncthreads();
    if (c >= n) return;
    const double *Z = Zg + (size_t)ich * npad * npad + c;
    double *X = AA + (size_t)ich * ns * ns + (size_t)ns * c;
    constexpr int PF = 8;
    double win[KS], nx[PF];
#pragma unroll
    for (int t = 0; t < KS; t++) win[t] = 0.0;
#pragma unroll
    for (int u = 0; u < PF; u++) nx[u] = n - 1 - u >= 0 ? Z[(size_t)(n - 1 - u) * npad] : 0.0;
    for (int i0 = n - 1; i0 >= 0; i0 -= PF) {
        double cur[PF];
#pragma unroll
        for (int u = 0; u < PF; u++) cur[u] = nx[u];
#pragma unroll
        for (int u = 0; u < PF; u++) nx[u] = i0 - PF - u >= 0 ? Z[(size_t)(i0 - PF - u) * npad] : 0.0;
#pragma unroll
        for (int u = 0; u < PF; u++)
            if (i0 - u >= 0) X[i0 - u] = band_step<KS>(Ub + (i0 - u) * KS, cur[u], win);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef void (*chan_tridiag_fn)(int, int, const int *, const int *, const double *, const double *, double *,
                                double *, double *, double *, double *, double *, int *);
typedef void (*chan_solve_fn)(int, int, const int *, const double *, const double *, double *);

template <int KS> static void chan_fns(chan_tridiag_fn *t, chan_solve_fn *b)
{
    *t = chan_tridiag_kernel<KS>;
    *b = chan_solve_kernel<KS>;
}

static bool chan_lookup(int ks, chan_tridiag_fn *t, chan_solve_fn *b)
{
    switch (ks) {
    case 2: chan_fns<2>(t, b); return true;
    case 3: chan_fns<3>(t, b); return true;
    case 4: chan_fns<4>(t, b); return true;
    case 5: chan_fns<5>(t, b); return true;
    case 6: chan_fns<6>(t, b); return true;
    case 7: chan_fns<7>(t, b); return true;
    case 8: chan_fns<8>(t, b); return true;
    case 9: chan_fns<9>(t, b); return true;
    case 10: chan_fns<10>(t, b); return true;
    case 11: chan_fns<11>(t, b); return true;
    case 12: chan_fns<12>(t, b); return true;
    case 13: chan_fns<13>(t, b); return true;
    case 14: chan_fns<14>(t, b); return true;
    case 15: chan_fns<15>(t, b); return true;
    case 16: chan_fns<16>(t, b); return true;
    default: return false;
    }
}

static size_t tridiag_smem(int npad, int ks)
{
    return sizeof(double) * (tri(npad) + (size_t)npad * ks + (CH_RED + 4) * (size_t)npad + 4);
}

bool chan_own_ok(int ns, int ks, int npad, int device)
{
    chan_tridiag_fn t;
    chan_solve_fn b;
    if (!chan_lookup(ks, &t, &b) || npad > CH_NMAX || npad < 1) return false;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    (void)ns;
    return tridiag_smem(npad, ks) <= (size_t)optin;
}

size_t chan_own_workspace_doubles(int nch, int npad, int ks)
{
    const size_t np2 = (size_t)npad * npad;
    // X, Y, Y', G | L band | reflectors | d, e, tau; the pivots of the inverse iteration take X's place
    return (size_t)nch * (4 * np2 + (size_t)npad * ks + tri(npad) + 3 * (size_t)npad) + 64;
}

int chan_own_solve(bsrg_ctx *c, const bsrg_basis *b, const double *hcc, int nch, int npad, const int *d_s0,
                   const int *d_nsol, double *AA, double *Wv, int *d_info, double *ws, int *d_flag)
{
    const int ns = b->ns, ks = b->ks;
    cudaStream_t s = c->stream;
    chan_tridiag_fn ktri;
    chan_solve_fn ksol;
    if (!chan_lookup(ks, &ktri, &ksol)) { set_error("channel solves: ks=%d outside 2..16", ks); return BSRG_ERR_ARG; }
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    const size_t sm1 = tridiag_smem(npad, ks), sm2 = sizeof(double) * 66 * npad;
    const size_t sm3 = sizeof(double) * (tri(npad) + npad);
    if (sm1 > (size_t)optin || npad > CH_NMAX) { set_error("channel solves: n=%d too large for shared memory", npad); return BSRG_ERR_ARG; }
    const size_t np2 = (size_t)npad * npad;
    double *X = ws, *Y = X + np2 * nch, *Y2 = Y + np2 * nch, *Gm = Y2 + np2 * nch;
    double *Lg = Gm + np2 * nch, *Vg = Lg + (size_t)npad * ks * nch, *dg = Vg + tri(npad) * nch;
    double *eg = dg + (size_t)npad * nch, *tg = eg + (size_t)npad * nch;
    cudaError_t e;
    if ((e = smem_attr(ktri, (int)sm1)) != cudaSuccess ||
        (e = smem_attr(chan_invit_kernel, (int)sm2)) != cudaSuccess)
        return cuda_fail(e, "channel solves: shared memory");
    if ((e = cudaMemsetAsync(d_flag, 0, 2 * sizeof(int), s)) != cudaSuccess) return cuda_fail(e, "channel solves: flag");
    ktri<<<nch, CH_THREADS, sm1, s>>>(ns, npad, d_s0, d_nsol, hcc, b->sb, X, Lg, Vg, dg, eg, tg, d_info);
    chan_bisect_kernel<<<dim3((unsigned)nch, (unsigned)((npad * CB_L + CB_T - 1) / CB_T)), CB_T, 0, s>>>(
        ns, npad, d_nsol, dg, eg, Wv);
    chan_invit_kernel<<<dim3((unsigned)nch, (unsigned)((npad + 31) / 32)), 32, sm2, s>>>(ns, npad, d_nsol, dg, eg, Wv,
                                                                                          Y, X);
    // two symmetric orthogonalisation steps; Y holds the eigenvectors as rows (Y^T column-major)
    double *src = Y, *dst = Y2;
    for (int pass = 0; pass < 2; pass++) {
        DgemmBatch g{};
        g.m = npad; g.n = npad; g.k = npad;
        g.A = src; g.lda = npad; g.sA = (long)np2;
        g.B = src; g.ldb = npad; g.sB = (long)np2;
        g.C = Gm; g.ldc = npad; g.sC = (long)np2;
        g.alpha = 1.0; g.beta = 0.0;
        int rc = dgemm_batched(false, true, g, nch, s);       // Gram matrix of the eigenvectors (rows)
        if (rc != BSRG_OK) return rc;
        dim3 gl((unsigned)((np2 + 255) / 256), (unsigned)nch);
        chan_lowdin_kernel<<<gl, 256, 0, s>>>(npad, d_nsol, Gm, pass == 0 ? d_flag : d_flag + 1);
        DgemmBatch u{};
        u.m = npad; u.n = npad; u.k = npad;
        u.A = Gm; u.lda = npad; u.sA = (long)np2;
        u.B = src; u.ldb = npad; u.sB = (long)np2;
        u.C = dst; u.ldc = npad; u.sC = (long)np2;
        u.alpha = 1.0; u.beta = 0.0;
        rc = dgemm_batched(false, false, u, nch, s);          // rows <- M rows
        if (rc != BSRG_OK) return rc;
        double *t = src; src = dst; dst = t;
    }
    // the reflectors of a channel fill an SM's shared memory: one CTA an SM
    // and as few vectors a warp as they allow
    const int slots = CH_WARPS * std::max(1, 148 / nch), cq = npad <= 2 * slots ? 2 : npad > 4 * slots && npad <= 5 * slots ? 5 : 4;
    const unsigned split = (unsigned)std::max(1, std::min((npad + cq * CH_WARPS - 1) / (cq * CH_WARPS), 148 / nch));
    const chan_q_fn kq = npad <= 64 ? chan_q_of<2>(cq) : npad <= 128 ? chan_q_of<4>(cq) : npad <= 224 ? chan_q_of<7>(cq)
                                                                                                    : chan_q_of<8>(cq);
    if ((e = smem_attr(kq, (int)sm3)) != cudaSuccess) return cuda_fail(e, "channel solves: shared memory");
    kq<<<dim3((unsigned)nch, split), CH_THREADS, sm3, s>>>(npad, d_nsol, Vg, tg, src);
    ksol<<<dim3((unsigned)nch, (unsigned)((npad + CL_T - 1) / CL_T)), CL_T, sizeof(double) * npad * ks, s>>>(
        ns, npad, d_nsol, Lg, src, AA);
    return cuda_fail(cudaGetLastError(), "channel solves");
}

}  // namespace bsrg
