// Symmetric tridiagonal eigensolver (divide and conquer) for sm_100a.
//
// The reference's DSYEV (LAP_DSYEV, src/libs/ZCOM/LAPACK_calls.f90:54-76,
// called from diag_hd.f90:312) reduces A to a tridiagonal T and diagonalises T
// by the implicit QL/QR algorithm (DSTEQR).  Here T is diagonalised by Cuppen's
// divide and conquer as in LAPACK's DSTEDC (the published algorithm; Gu and
// Eisenstat's recomputed z for orthogonal eigenvectors), laid out for the GPU:
//
//   * the tree is cut top-down into halves until the pieces have at most
//     DC_LEAF rows; every cut (s, m, e) tears T into T1 (+) T2 + |b| v v^T with
//     b = e(m-1), v = e_{m-1} + sign(b) e_m (the diagonal of both halves loses
//     |b| at the cut);
//   * leaves: one CTA each, cyclic Jacobi with tournament ordering on the dense
//     leaf in shared memory;
//   * merges, one tree level at a time, deepest first: per merge one CTA sorts the poles, finds the tolerance and
//     deflates -- small z components, and close poles merged by a Givens rotation; every thread tests its pairs,
//     only the rotations themselves are a chain -- and lays the surviving columns out by type (upper half only,
//     mixed, lower half only, deflated); the secular equation 1 + rho sum z_i^2 / (d_i - lambda) = 0 is solved per
//     root (two-pole rational iteration, every iterate kept inside a bracket, roots stored as pole + offset); z is
//     recomputed from the roots (Loewner's formula) and the eigenvectors of D + rho z z^T formed column by column;
//     all merged eigenvectors of a level, each half's rows against its column types, are one launch of FP64
//     tensor-core products that writes the columns to their ascending places.
//   The merges' sizes stay on the device (the launches cover the largest a merge can be), so nothing is read back
//   between the levels.
//   * eigenvalues alone: bisection on Sturm counts (tridiag_values).
#include <algorithm>
#include <cmath>
#include <vector>

#include "ctx.h"
#include "dmma.cuh"

namespace bsrg {
namespace {

constexpr int DC_LEAF = 32;
constexpr int DC_MAXK = 10240;   // largest merge (shared-memory deflation pass)

struct DcMerge {
    int s, k1, k2, pad;
    long off_g;     // Qg (k x k): gathered child columns, type-grouped, rotations applied
    long off_u;     // U (k x k): eigenvectors of D + rho z z^T (rows in Qg column order)
    long off_v;     // per-merge vectors (8k doubles)
    long off_i;     // per-merge int vectors (4k ints)
};

// per-merge scalars (ints): K, n1, n2, n3, nrot
constexpr int DC_NS = 8;

// ---------------------------------------------------------------------------
// tears and leaves
// ---------------------------------------------------------------------------
__global__ void dc_tear_kernel(int nsplit, const int *__restrict__ splits, double *d, const double *__restrict__ e)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nsplit) return;
    const int m = splits[q];
    const double b = fabs(e[m - 1]);
    d[m - 1] -= b;
    d[m] -= b;
}

// Cyclic Jacobi on one leaf (k <= DC_LEAF), tournament ordering: every round rotates k/2 disjoint
// pairs.  A thread applies both sides to the 2 x 2 block of a pair of pairs, so a round is the angles
// (a dependent chain of square roots and divisions) and one pass.  Eigenvalues are written ascending to
// w[s..s+k), eigenvectors to Z[s.., s..].  Measured: 1.42 ms a launch with 64 rows and a pass per side,
// 0.23 with 32 (n = 1713).
__global__ void __launch_bounds__(256) dc_leaf_kernel(const int *__restrict__ ls, const int *__restrict__ lk,
                                                      const double *__restrict__ d, const double *__restrict__ e,
                                                      double *w, double *Z, long ldz)
{
    __shared__ double A[DC_LEAF][DC_LEAF + 1], V[DC_LEAF][DC_LEAF + 1];
    __shared__ double rc[DC_LEAF / 2], rs[DC_LEAF / 2];
    __shared__ int rp[DC_LEAF / 2], rq[DC_LEAF / 2];
    __shared__ int rotated;
    __shared__ int rank[DC_LEAF];
    static_assert(DC_LEAF * DC_LEAF / 4 == 256, "a thread per pair of pairs");
    const int s = ls[blockIdx.x], k = lk[blockIdx.x], tid = threadIdx.x;
    for (int q = tid; q < DC_LEAF * DC_LEAF; q += blockDim.x) {
        const int r = q % DC_LEAF, c = q / DC_LEAF;
        double a = 0.0;
        if (r < k && c < k) {
            if (r == c) a = d[s + r];
            else if (r == c + 1) a = e[s + c];
            else if (c == r + 1) a = e[s + r];
        }
        A[r][c] = a;
        V[r][c] = (r == c) ? 1.0 : 0.0;
    }
    const int m = k + (k & 1), np = m / 2, bi = tid / (DC_LEAF / 2), bj = tid % (DC_LEAF / 2);
    const double eps = 2.220446049250313e-16;
    __syncthreads();
    for (int sweep = 0; sweep < 40 && m > 1; sweep++) {
        if (tid == 0) rotated = 0;
        __syncthreads();
        for (int r = 0; r < m - 1; r++) {
            if (tid < np) {
                int p, q;
                if (tid == 0) { p = 0; q = 1 + r % (m - 1); }
                else { p = 1 + (tid + r) % (m - 1); q = 1 + (m - 1 - tid + r) % (m - 1); }
                if (p > q) { int t = p; p = q; q = t; }
                double c = 1.0, sn = 0.0;
                if (q < k) {
                    const double apq = A[p][q], app = A[p][p], aqq = A[q][q];
                    if (apq != 0.0 && fabs(apq) > eps * sqrt(fabs(app * aqq))) {
                        const double tau = (aqq - app) / (2.0 * apq);
                        const double t = tau >= 0.0 ? 1.0 / (tau + sqrt(1.0 + tau * tau))
                                                    : -1.0 / (-tau + sqrt(1.0 + tau * tau));
                        c = 1.0 / sqrt(1.0 + t * t);
                        sn = t * c;
                        rotated = 1;
                    }
                }
                rp[tid] = p; rq[tid] = q; rc[tid] = c; rs[tid] = sn;
            }
            __syncthreads();
            if (bi < np && bj < np) {
                const int p = rp[bi], q = rq[bi], x = rp[bj], y = rq[bj];
                const double c = rc[bi], sn = rs[bi], cc = rc[bj], ss = rs[bj];
                const double apx = A[p][x], apy = A[p][y], aqx = A[q][x], aqy = A[q][y];
                const double lpx = c * apx - sn * aqx, lpy = c * apy - sn * aqy;       // rows
                const double lqx = sn * apx + c * aqx, lqy = sn * apy + c * aqy;
                A[p][x] = cc * lpx - ss * lpy;                                         // columns
                A[p][y] = ss * lpx + cc * lpy;
                A[q][x] = cc * lqx - ss * lqy;
                A[q][y] = ss * lqx + cc * lqy;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = bi + h * np;
                    const double vx = V[row][x], vy = V[row][y];
                    V[row][x] = cc * vx - ss * vy;
                    V[row][y] = ss * vx + cc * vy;
                }
            }
            __syncthreads();
        }
        if (!rotated) break;
        __syncthreads();
    }
    // ascending order: rank by value, ties by index
    if (tid < k) {
        const double v = A[tid][tid];
        int rk = 0;
        for (int j = 0; j < k; j++) {
            const double u = A[j][j];
            rk += (u < v) || (u == v && j < tid);
        }
        rank[tid] = rk;
        w[s + rk] = v;
    }
    __syncthreads();
    for (int q = tid; q < k * k; q += blockDim.x) {
        const int r = q % k, c = q / k;
        Z[(s + r) + ldz * (long)(s + rank[c])] = V[r][c];
    }
}

// ---------------------------------------------------------------------------
// merge step 1: sort, deflate, gather the columns (one CTA per merge)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double blk_max(double v, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int q = 0; q < (int)(blockDim.x + 31) / 32; q++) r = fmax(r, sh[q]);
    __syncthreads();
    return r;
}

// min(1, max |T(i, j)|), what the deflation's tolerance scales the entries of z with
__global__ void __launch_bounds__(1024) dc_norm_kernel(int n, const double *__restrict__ d, const double *__restrict__ e,
                                                       double *norm)
{
    __shared__ double red[32];
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fmax(fabs(d[i]), i + 1 < n ? fabs(e[i]) : 0.0));
    m = blk_max(m, red);
    if (threadIdx.x == 0) *norm = fmin(1.0, m);
}

// exclusive sum over the block's threads; the total in *all
__device__ __forceinline__ unsigned long long blk_scan(unsigned long long v, unsigned long long *sh,
                                                       unsigned long long *all)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    unsigned long long before = 0, total = 0;
    for (int q = 0; q < nw; q++) {
        if (q < warp) before += sh[q];
        total += sh[q];
    }
    *all = total;
    return before + x - v;
}

// Sort, deflate and group one merge's columns (one CTA).  LAPACK's rules: an entry of z below the tolerance
// deflates; of two neighbours among the others that are close, a rotation takes one out.  LAPACK's tolerance,
// 8 eps max(|d|, |z|), is that of a T scaled to 1; T is not scaled here, so where it is smaller the entries of z,
// which are not, count times its largest entry.  The rotations
// are a chain (an entry that a rotation has changed meets the next one), so one thread walks them, but only
// from the pairs that are close as they are: every thread has tested its pairs first.  The places of the
// columns are prefix sums over the threads' stretches.  (One thread in all of it took 1.6 ms in five merge
// levels at n = 1713 and 7.5 at n = 7810; 0.07 ms in six levels at 1713 so.)
// Shared layout (dynamic): dS[k] zS[k] (doubles), src[k] (int: child column), st[k] (char:
// 0 deflated, 1 upper, 2 mixed, 3 lower).  Outputs in the merge's vectors:
//   V: dd[K] poles ascending | zz[K] | dval[nd] deflated eigenvalues
//   I: pos[K] Qg column of pole i | gsrc[k] child column of Qg column t | rot (pairs of Qg columns) ...
__global__ void __launch_bounds__(512) dc_prep_kernel(const DcMerge *__restrict__ mg, const double *__restrict__ e,
                                                      const double *__restrict__ w, const double *__restrict__ Z,
                                                      long ldz, double *ws, int *iws, int *scal,
                                                      const double *__restrict__ norm)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ double red[32];
    __shared__ unsigned long long scan[32];
    __shared__ int s_nrot, s_unsorted;
    const DcMerge M = mg[blockIdx.x];
    const int k1 = M.k1, k = M.k1 + M.k2, s = M.s, tid = threadIdx.x, nt = blockDim.x;
    double *dS = (double *)dsm, *zS = dS + k;
    int *src = (int *)(zS + k);
    unsigned char *st = (unsigned char *)(src + k);
    double *V = ws + M.off_v;
    double *dd = V, *zz = V + k, *dval = V + 2 * k, *rotc = V + 3 * k, *rots = V + 4 * k;
    int *I = iws + M.off_i;
    int *pos = I, *gsrc = I + k, *rotp = I + 2 * k, *rotq = I + 3 * k, *dpos = I + 5 * k;
    int *sc = scal + DC_NS * blockIdx.x;
    const double beta = e[s + k1 - 1];
    const double sg = beta >= 0.0 ? 1.0 : -1.0;
    const double rsq2 = 0.70710678118654752440;
    if (tid == 0) { s_nrot = 0; s_unsorted = 0; }
    // (with a NaN among the values two of them can take one place: the places left over stay valid indices)
    for (int i = tid; i < k; i += nt) { dS[i] = zS[i] = 0.0; src[i] = i; st[i] = i < k1 ? 1 : 3; }
    __syncthreads();
    // merge the two ascending runs (stable: run 1 first on ties)
    for (int i = tid; i < k; i += nt) {
        double v;
        int rk;
        if (i < k1) {
            v = w[s + i];
            int lo = 0, hi = M.k2;   // count run-2 values < v
            while (lo < hi) { int md = (lo + hi) >> 1; if (w[s + k1 + md] < v) lo = md + 1; else hi = md; }
            rk = i + lo;
        } else {
            const int j = i - k1;
            v = w[s + i];
            int lo = 0, hi = k1;     // count run-1 values <= v
            while (lo < hi) { int md = (lo + hi) >> 1; if (w[s + md] <= v) lo = md + 1; else hi = md; }
            rk = j + lo;
        }
        const double zv = i < k1 ? Z[(s + k1 - 1) + ldz * (long)(s + i)] * rsq2
                                 : sg * Z[(s + k1) + ldz * (long)(s + i)] * rsq2;
        dS[rk] = v;
        zS[rk] = zv;
        src[rk] = i;
        st[rk] = i < k1 ? 1 : 3;
    }
    __syncthreads();
    double md = 0.0, mz = 0.0;
    for (int i = tid; i < k; i += nt) { md = fmax(md, fabs(dS[i])); mz = fmax(mz, fabs(zS[i])); }
    md = blk_max(md, red);
    mz = blk_max(mz, red);
    const double rho = 2.0 * fabs(beta);
    const double tol = 8.0 * 2.220446049250313e-16 * fmax(md, mz * *norm);
    const bool none = rho * mz <= tol;                      // all deflate
    // a thread's stretch of the sorted order
    const int per = (k + nt - 1) / nt, i0 = min(k, tid * per), i1 = min(k, i0 + per);
    unsigned long long total;
    // the entries that stay, in order: idx (in pos for now)
    int *idx = pos, *close = gsrc;
    {
        int cnt = 0;
        for (int i = i0; i < i1; i++) {
            if (none || rho * fabs(zS[i]) <= tol) st[i] = 0;
            cnt += st[i] != 0;
        }
        int at = (int)blk_scan((unsigned long long)cnt, scan, &total);
        for (int i = i0; i < i1; i++)
            if (st[i] != 0) idx[at++] = i;
    }
    const int m = (int)total;
    __syncthreads();
    // entry p of idx and the one before it: do they rotate?
    auto rotates = [&](int p, double &tau, double &c, double &sn) {
        const int j = idx[p], prev = idx[p - 1];
        const double sv = zS[prev], cv = zS[j], t = dS[j] - dS[prev];
        tau = hypot(cv, sv);
        c = cv / tau;
        sn = -sv / tau;
        return fabs(t * c * sn) <= tol;
    };
    int ncl;
    {
        const int perm = (m + nt - 1) / nt, p0 = max(1, min(m, tid * perm)), p1 = min(m, tid * perm + perm);
        int cnt = 0;
        double tau, c, sn;
        for (int p = p0; p < p1; p++) cnt += rotates(p, tau, c, sn);
        int at = (int)blk_scan((unsigned long long)cnt, scan, &total);
        if (cnt)
            for (int p = p0; p < p1; p++)
                if (rotates(p, tau, c, sn)) close[at++] = p;
        ncl = (int)total;
    }
    __syncthreads();
    if (tid == 0 && ncl > 0) {
        int nrot = 0, seen = 0;                             // entries up to seen have been tested as they are now
        for (int f = 0; f < ncl; f++) {
            int p = close[f];
            if (p <= seen) continue;
            for (; p < m; p++) {
                double tau, c, sn;
                seen = p;
                if (!rotates(p, tau, c, sn)) break;
                const int j = idx[p], prev = idx[p - 1];
                zS[j] = tau;
                zS[prev] = 0.0;
                st[j] = (unsigned char)(st[prev] == st[j] ? st[j] : 2);
                st[prev] = 0;
                const double tp = dS[prev] * c * c + dS[j] * sn * sn;
                dS[j] = dS[prev] * sn * sn + dS[j] * c * c;
                dS[prev] = tp;
                // columns (prev, j) rotated by (c, sn); indices mapped to Qg below
                rotp[nrot] = prev;
                rotq[nrot] = j;
                rotc[nrot] = c;
                rots[nrot] = sn;
                nrot++;
            }
        }
        s_nrot = nrot;
    }
    __syncthreads();
    // Qg column of each sorted position: by type, ascending within each type, deflated last; poles and
    // deflated values ascending.  Counts of types 1, 2, 3 and 0 in 16 bits each.
    unsigned long long mine = 0;
    for (int i = i0; i < i1; i++) mine += 1ull << (16 * ((st[i] + 3) & 3));
    const unsigned long long before = blk_scan(mine, scan, &total);
    const int n1 = (int)(total & 0xffff), n2 = (int)(total >> 16 & 0xffff), n3 = (int)(total >> 32 & 0xffff);
    const int K = n1 + n2 + n3;
    {
        int c1 = (int)(before & 0xffff), c2 = (int)(before >> 16 & 0xffff), c3 = (int)(before >> 32 & 0xffff);
        int nd = (int)(before >> 48), ip = c1 + c2 + c3;
        c2 += n1;
        c3 += n1 + n2;
        for (int i = i0; i < i1; i++) {
            if (st[i] != 0) {
                const int col = st[i] == 1 ? c1++ : (st[i] == 2 ? c2++ : c3++);
                gsrc[col] = i;             // sorted position feeding Qg column col
                dd[ip] = dS[i];
                zz[ip] = zS[i];
                pos[ip++] = col;
            } else {
                dval[nd] = dS[i];
                dpos[nd++] = i;
            }
        }
    }
    __syncthreads();
    // a rotation can leave close neighbours out of order
    if (s_nrot > 0) {
        for (int q = tid + 1; q < max(K, k - K); q += nt)
            if ((q < K && dd[q - 1] > dd[q]) || (q < k - K && dval[q - 1] > dval[q])) s_unsorted = 1;
        __syncthreads();
        if (s_unsorted && tid == 0) {
            for (int i = 1; i < K; i++) {
                const double x = dd[i], y = zz[i];
                const int c = pos[i];
                int q = i;
                while (q > 0 && dd[q - 1] > x) { dd[q] = dd[q - 1]; zz[q] = zz[q - 1]; pos[q] = pos[q - 1]; q--; }
                dd[q] = x; zz[q] = y; pos[q] = c;
            }
            for (int i = 1; i < k - K; i++) {
                const double x = dval[i];
                const int c = dpos[i];
                int q = i;
                while (q > 0 && dval[q - 1] > x) { dval[q] = dval[q - 1]; dpos[q] = dpos[q - 1]; q--; }
                dval[q] = x; dpos[q] = c;
            }
        }
        __syncthreads();
    }
    for (int q = tid; q < k - K; q += nt) gsrc[K + q] = dpos[q];
    if (tid == 0) { sc[0] = K; sc[1] = n1; sc[2] = n2; sc[3] = n3; sc[4] = s_nrot; }
    __syncthreads();
    // rotations recorded on sorted positions -> on Qg columns; child column of every Qg
    // column for the gather (int slab 5k..6k; the deflated positions there are done)
    int *colof = (int *)dS;       // dS has been copied out
    for (int c = tid; c < k; c += nt) colof[gsrc[c]] = c;
    __syncthreads();
    for (int t = tid; t < s_nrot; t += nt) { rotp[t] = colof[rotp[t]]; rotq[t] = colof[rotq[t]]; }
    for (int c = tid; c < k; c += nt) I[5 * k + c] = src[gsrc[c]];
    if (tid == 0) {
        double *pr = ws + M.off_v + 7 * (long)k;
        pr[0] = rho;
    }
}

// Qg(:, c) = child column feeding Qg column c (zero outside its half).  Threads run
// along rows (coalesced), each covering 32 columns.
__global__ void dc_gather_kernel(const DcMerge *__restrict__ mg, const double *__restrict__ Z, long ldz, double *ws,
                                 const int *__restrict__ iws)
{
    const DcMerge M = mg[blockIdx.z];
    const int k1 = M.k1, k = M.k1 + M.k2, s = M.s;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= k) return;
    const int c0 = blockIdx.y * 32;
    if (c0 >= k) return;
    const int *chcol = iws + M.off_i + 5 * (long)k;
    double *Qg = ws + M.off_g;
    const int c1 = min(c0 + 32, k);
    for (int c = c0; c < c1; c++) {
        const int sc = chcol[c];
        double v = 0.0;
        if ((sc < k1) == (r < k1)) v = Z[(s + r) + ldz * (long)(s + sc)];
        Qg[r + (long)k * c] = v;
    }
}

// the deflation rotations, in order, on every row of Qg (rows are independent)
__global__ void dc_rotate_kernel(const DcMerge *__restrict__ mg, const int *__restrict__ scal, double *ws,
                                 const int *__restrict__ iws)
{
    const DcMerge M = mg[blockIdx.y];
    const int k = M.k1 + M.k2;
    const int nrot = scal[DC_NS * blockIdx.y + 4];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= k || nrot == 0) return;
    const double *V = ws + M.off_v;
    const double *rotc = V + 3 * (long)k, *rots = V + 4 * (long)k;
    const int *rotp = iws + M.off_i + 2 * (long)k, *rotq = iws + M.off_i + 3 * (long)k;
    double *Qg = ws + M.off_g;
    for (int t = 0; t < nrot; t++) {
        const long a = rotp[t], b = rotq[t];
        const double c = rotc[t], sn = rots[t];
        const double x = Qg[r + k * a], y = Qg[r + k * b];
        Qg[r + k * a] = c * x + sn * y;
        Qg[r + k * b] = c * y - sn * x;
    }
}

// ---------------------------------------------------------------------------
// merge step 2: secular equation, one thread per root
// ---------------------------------------------------------------------------
// root j in (dd_j, dd_{j+1}) (the last in (dd_K, dd_K + rho |z|^2)) as origin index + offset
constexpr int SEC_WARPS = 16;          // roots per CTA of the secular kernel (a warp each)

__device__ __forceinline__ double warp_sum(double x)
{
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// one warp per root: the lanes split the sums over the poles, every lane then takes the same step
__global__ void __launch_bounds__(32 * SEC_WARPS) dc_secular_kernel(const DcMerge *__restrict__ mg,
                                                                    const int *__restrict__ scal, double *ws,
                                                                    int *iws, int kcap)
{
    extern __shared__ __align__(16) double sm2[];
    const int mi = blockIdx.y;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2;
    const int K = scal[DC_NS * mi];
    if ((int)blockIdx.x * SEC_WARPS >= K) return;
    double *V = ws + M.off_v;
    const double *dd = V, *zz = V + k;
    double *tau = V + 5 * (long)k;
    int *org = iws + M.off_i + 4 * (long)k;
    const double rho = V[7 * (long)k];
    double *sd = sm2, *sz = sm2 + kcap;
    for (int i = threadIdx.x; i < K; i += blockDim.x) { sd[i] = dd[i]; sz[i] = zz[i] * zz[i]; }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.x * SEC_WARPS + (threadIdx.x >> 5);
    if (j >= K) return;
    int o;
    double lo, hi;
    if (j < K - 1) {
        const double mid = 0.5 * (sd[j + 1] - sd[j]);
        double fp = 0.0;
        for (int i = lane; i < K; i += 32) fp += sz[i] / ((sd[i] - sd[j]) - mid);
        const double f = 1.0 + rho * warp_sum(fp);
        if (f >= 0.0) { o = j; lo = 0.0; hi = mid; }
        else { o = j + 1; lo = -mid; hi = 0.0; }
    } else {
        double zp = 0.0;
        for (int i = lane; i < K; i += 32) zp += sz[i];
        o = j; lo = 0.0; hi = rho * warp_sum(zp);
    }
    const double dov = sd[o];
    // Iterate on tau with the two-pole model of the secular function (the "middle way" of
    // R.-C. Li, 1993, as LAPACK dlaed4 uses it): psi (poles up to j) and phi (poles above j)
    // are each replaced by a constant plus their nearest pole, matched in value and slope;
    // the model's root in the bracket is the next iterate (the last root: one pole).  Every
    // iterate stays inside [lo, hi]; a step that would leave it bisects instead.
    double t = 0.5 * (lo + hi);
    const double dj = sd[j] - dov, dj1 = j < K - 1 ? sd[j + 1] - dov : 0.0;
    for (int it = 0; it < 100; it++) {
        double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
        for (int i = lane; i < K; i += 32) {
            const double r = 1.0 / ((sd[i] - dov) - t);
            const double q = sz[i] * r;
            if (i <= j) { psi += q; dpsi += q * r; }
            else { phi += q; dphi += q * r; }
        }
        psi = warp_sum(psi);
        dpsi = warp_sum(dpsi);
        phi = warp_sum(phi);
        dphi = warp_sum(dphi);
        const double eabs = 1.0 + rho * (fabs(psi) + fabs(phi));
        const double f = 1.0 + rho * (psi + phi);
        if (f < 0.0) lo = t; else hi = t;
        if (f == 0.0 || fabs(f) <= 8.0 * 2.220446049250313e-16 * K * eabs) break;
        const double Dj = dj - t;                      // distances to the two nearest poles
        double eta;
        if (j < K - 1) {
            const double Dj1 = dj1 - t;
            const double sj = rho * dpsi * Dj * Dj, sj1 = rho * dphi * Dj1 * Dj1;
            const double c = f - sj / Dj - sj1 / Dj1;
            // c eta^2 - (c (Dj + Dj1) + sj + sj1) eta + (c Dj Dj1 + sj Dj1 + sj1 Dj) = 0
            const double qa = c, qb = c * (Dj + Dj1) + sj + sj1, qc = c * Dj * Dj1 + sj * Dj1 + sj1 * Dj;
            // the model's root between the two poles, eta in (Dj, Dj1); both roots formed stably
            eta = 0.5 * (lo + hi) - t;
            if (qa == 0.0) {
                if (qb != 0.0) eta = qc / qb;
            } else {
                const double disc = sqrt(fmax(qb * qb - 4.0 * qa * qc, 0.0));
                const double w1 = 0.5 * (qb + copysign(disc, qb));
                const double e1 = w1 / qa, e2 = w1 != 0.0 ? qc / w1 : e1;
                if (e1 > Dj && e1 < Dj1) eta = e1;
                else if (e2 > Dj && e2 < Dj1) eta = e2;
            }
        } else {
            const double sj = rho * dpsi * Dj * Dj, c = f - sj / Dj;
            eta = c != 0.0 ? Dj + sj / c : 0.5 * (hi - t);
        }
        double tn = t + eta;
        if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
        const double step = fabs(tn - t);
        t = tn;
        if (step <= 2.220446049250313e-16 * fabs(t) || hi - lo <= 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)))
            break;
    }
    if (lane == 0) {
        tau[j] = t;
        org[j] = o;
    }
}

// ---------------------------------------------------------------------------
// merge step 3: z recomputed from the roots, then the eigenvectors of D + rho z z^T
// ---------------------------------------------------------------------------
// a warp per entry, the lanes multiply every 32nd factor (one thread per entry: 2.2 ms at n = 7810, a
// chain of divisions)
__global__ void __launch_bounds__(256) dc_zhat_kernel(const DcMerge *__restrict__ mg, const int *__restrict__ scal,
                                                      double *ws, int *iws)
{
    const int mi = blockIdx.y;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2;
    const int K = scal[DC_NS * mi];
    const int lane = threadIdx.x & 31, i = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (i >= K) return;
    double *V = ws + M.off_v;
    const double *dd = V, *zz = V + k, *tau = V + 5 * (long)k;
    double *zh = V + 6 * (long)k;
    const int *org = iws + M.off_i + 4 * (long)k;
    const double di = dd[i];
    // (d_i - lambda_i) prod_{j != i} (d_i - lambda_j) / (d_i - d_j)   (< 0)
    double p = lane == 0 ? (di - dd[org[i]]) - tau[i] : 1.0;
#pragma unroll 4
    for (int j = lane; j < K; j += 32) {
        const double f = ((di - dd[org[j]]) - tau[j]) / (di - dd[j]);
        if (j != i) p *= f;
    }
    for (int o = 16; o > 0; o >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, o);
    if (lane == 0) zh[i] = copysign(sqrt(fmax(-p, 0.0)), zz[i]);
}

// U(pos[i], j) = zh_i / (d_i - lambda_j) / ||.||; one warp per column j
__global__ void dc_vec_kernel(const DcMerge *__restrict__ mg, const int *__restrict__ scal, double *ws, int *iws)
{
    const int mi = blockIdx.y;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2;
    const int K = scal[DC_NS * mi];
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (j >= K) return;
    double *V = ws + M.off_v;
    const double *dd = V, *tau = V + 5 * (long)k, *zh = V + 6 * (long)k;
    const int *pos = iws + M.off_i;
    const int *org = iws + M.off_i + 4 * (long)k;
    double *U = ws + M.off_u;
    const double dj = dd[org[j]], tj = tau[j];
    double ss = 0.0;
    for (int i = lane; i < K; i += 32) {
        const double u = zh[i] / ((dd[i] - dj) - tj);
        ss += u * u;
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const double inv = 1.0 / sqrt(ss);
    for (int i = lane; i < K; i += 32) {
        const double u = zh[i] / ((dd[i] - dj) - tj);
        U[pos[i] + (long)K * j] = u * inv;
    }
}

// ---------------------------------------------------------------------------
// merge step 4: ascending order of the merged eigenvalues, columns into Z
// ---------------------------------------------------------------------------
// colmap[c] = final column of merged column c (c < K: root c, c >= K: deflated Qg column c)
__global__ void __launch_bounds__(256) dc_rank_kernel(const DcMerge *__restrict__ mg, const int *__restrict__ scal,
                                                      double *ws, int *iws, double *w)
{
    const int mi = blockIdx.x;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2, s = M.s;
    const int K = scal[DC_NS * mi];
    double *V = ws + M.off_v;
    const double *dd = V, *dval = V + 2 * (long)k, *tau = V + 5 * (long)k;
    const int *org = iws + M.off_i + 4 * (long)k;
    int *colmap = iws + M.off_i + 5 * (long)k;
    const int nd = k - K;
    // roots ascending, deflated values ascending: merge by binary search (ties: roots first)
    for (int c = threadIdx.x; c < k; c += blockDim.x) {
        double v;
        int rk;
        if (c < K) {
            v = dd[org[c]] + tau[c];
            int lo = 0, hi = nd;          // deflated values < v
            while (lo < hi) { const int md = (lo + hi) >> 1; if (dval[md] < v) lo = md + 1; else hi = md; }
            rk = c + lo;
        } else {
            const int q = c - K;
            v = dval[q];
            int lo = 0, hi = K;           // roots <= v
            while (lo < hi) {
                const int md = (lo + hi) >> 1;
                if (dd[org[md]] + tau[md] <= v) lo = md + 1; else hi = md;
            }
            rk = q + lo;
        }
        colmap[c] = rk;
        w[s + rk] = v;
    }
}

// Z's columns of the roots: Qg U, the upper rows from the columns of types 1 and 2, the lower ones from
// types 2 and 3; every product of a level in one launch (blockIdx.z = 2 merge + half), written to its
// columns' places directly.  The sizes come from the device, so a level is queued without reading the
// deflation counts back.
__global__ void __launch_bounds__(dmma::Sq::NT) dc_gemm_kernel(const DcMerge *__restrict__ mg,
                                                               const int *__restrict__ scal, const double *ws,
                                                               const int *iws, double *Z, long ldz)
{
    extern __shared__ __align__(16) double smem[];
    using C = dmma::Sq;
    const int mi = blockIdx.z >> 1, half = blockIdx.z & 1;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2, rows = half ? M.k2 : M.k1;
    const int K = scal[DC_NS * mi], n1 = scal[DC_NS * mi + 1], n2 = scal[DC_NS * mi + 2];
    const int m0 = blockIdx.x * C::BM, n0 = blockIdx.y * C::BN;
    if (m0 >= rows || n0 >= K) return;
    const double *A = ws + M.off_g + (half ? M.k1 + (long)k * n1 : 0), *B = ws + M.off_u + (half ? n1 : 0);
    double acc[C::FM][C::FN][2];
    dmma::tile_mma<C, false, false>(acc, smem, A, k, B, K, rows, K, 0, half ? K - n1 : n1 + n2, m0, n0);
    const int *colmap = iws + M.off_i + 5 * (long)k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp % C::WM, wn = warp / C::WM, r = lane >> 2, q = lane & 3;
#pragma unroll
    for (int t = 0; t < C::FN; t++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int col = n0 + wn * C::TN + t * 8 + 2 * q + j;
            if (col >= K) continue;
            double *out = Z + M.s + (half ? M.k1 : 0) + ldz * (long)(M.s + colmap[col]);
#pragma unroll
            for (int s = 0; s < C::FM; s++) {
                const int row = m0 + wm * C::TM + s * 8 + r;
                if (row < rows) out[row] = acc[s][t][j];
            }
        }
}

// the deflated columns
__global__ void dc_copy_kernel(const DcMerge *__restrict__ mg, const int *__restrict__ scal, const double *ws,
                               const int *iws, double *Z, long ldz)
{
    const int mi = blockIdx.y;
    const DcMerge M = mg[mi];
    const int k = M.k1 + M.k2, s = M.s;
    const int K = scal[DC_NS * mi];
    const int *colmap = iws + M.off_i + 5 * (long)k;
    const double *Qg = ws + M.off_g;
    for (int c = K + blockIdx.x; c < k; c += gridDim.x) {
        const double *src = Qg + (long)k * c;
        double *dst = Z + s + ldz * (long)(s + colmap[c]);
        for (int r = threadIdx.x; r < k; r += blockDim.x) dst[r] = src[r];
    }
}

struct Node { int s, k1, k2; };

// ---------------------------------------------------------------------------
// eigenvalues alone: bisection on Sturm counts
// ---------------------------------------------------------------------------
// Gershgorin bounds of T / 2^q, widened to hold 0, 2^q above both: b[0] lower, b[1] upper, b[2] = 2^-q,
// b[3] = 2^q; NaN if an entry is not finite.
__global__ void __launch_bounds__(1024) sturm_bounds_kernel(int n, const double *__restrict__ d,
                                                            const double *__restrict__ e, double *b)
{
    __shared__ double red[32];
    double lo = 0.0, hi = 0.0, bad = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
        lo = fmax(lo, r - d[i]);
        hi = fmax(hi, d[i] + r);
        if (!isfinite(d[i]) || !isfinite(r)) bad = 1.0;
    }
    lo = blk_max(lo, red);
    hi = blk_max(hi, red);
    bad = blk_max(bad, red);
    if (threadIdx.x == 0) {
        const double l = -lo, h = hi, top = fmax(lo, hi);
        int q = 0;
        if (top > 0.0) frexp(top, &q);
        // a hair beyond the bounds: the counts at the ends are 0 and n
        const double slack = 4.0 * 2.220446049250313e-16 * n;
        b[0] = bad > 0.0 ? NAN : ldexp(l, -q) - slack;
        b[1] = bad > 0.0 ? NAN : ldexp(h, -q) + slack;
        b[2] = ldexp(1.0, -q);
        b[3] = ldexp(1.0, q);
    }
}

// L lanes per eigenvalue count the eigenvalues below L points of its interval at once, so a pass divides
// the interval by L + 1; PASSES take it below 2^-55 of the bounds.  The count is the number of sign changes
// of the leading minors, p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}, rescaled every fourth step: without the
// division of the ratios' form.  e^2 is taken as 2^-140 at least (a shift of the eigenvalues by 2^-70 at most),
// so four steps shrink a pair of minors by 2^-568 at most and grow it by 3^4.
// What bounds it: the FP64 and integer issue slots of a step.
// Measured (n = 2176): 0.58 ms; the ratios' form with 32 lanes 2.36 ms
constexpr int ST_T = 256, ST_CH = 256;
template <int L, int PASSES>
__global__ void __launch_bounds__(ST_T) sturm_kernel(int n, const double *__restrict__ d, const double *__restrict__ e,
                                                     const double *__restrict__ b, double *__restrict__ w)
{
    __shared__ double2 ch[ST_CH];                            // (d_i, e_{i-1}^2), scaled
    const int lane = threadIdx.x & 31, sub = lane % L, j = (blockIdx.x * ST_T + threadIdx.x) / L;
    const double sc = b[2];
    double lo = b[0], hi = b[1];
    for (int pass = 0; pass < PASSES; pass++) {
        const double x = lo + (hi - lo) * ((sub + 1) * (1.0 / (L + 1)));
        double p0 = 0.0, p1 = 1.0;
        int cnt = 0;
        for (int c0 = 0; c0 < n; c0 += ST_CH) {
            const int m = min(ST_CH, n - c0), m4 = (m + 3) & ~3;
            __syncthreads();
            for (int i = threadIdx.x; i < m4; i += ST_T) {
                const double f = c0 + i > 0 && i < m ? e[c0 + i - 1] * sc : 0.0;
                // beyond the end: minors that keep their sign (d above every x)
                ch[i] = i < m ? make_double2(d[c0 + i] * sc, fmax(f * f, 0x1p-140)) : make_double2(4.0, 0.0);
            }
            __syncthreads();
#pragma unroll 2
            for (int i = 0; i < m4; i += 4) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double2 v = ch[i + q];
                    const double p = fma(v.x - x, p1, -(v.y * p0));
                    cnt += (unsigned)(__double2hiint(p) ^ __double2hiint(p1)) >> 31;
                    p0 = p1;
                    p1 = p;
                }
                const int ex = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
                const double r = __hiloint2double(0x7fe00000 - ex, 0);
                p0 *= r;
                p1 *= r;
            }
        }
        const unsigned above = (__ballot_sync(0xffffffffu, cnt > j) >> (lane - sub)) & (L < 32 ? (1u << (L & 31)) - 1 : ~0u);
        const int f = above ? __ffs(above) - 1 : L;
        const double xl = __shfl_sync(0xffffffffu, x, lane - sub + (f > 0 ? f - 1 : 0));
        const double xh = __shfl_sync(0xffffffffu, x, lane - sub + (f < L ? f : L - 1));
        if (f > 0) lo = xl;
        if (f < L) hi = xh;
    }
    if (sub == 0 && j < n) w[j] = 0.5 * (lo + hi) * b[3];
}

// equal eigenvalues can come out a rounding out of order: running maxima
__global__ void __launch_bounds__(1024) sturm_order_kernel(int n, double *w)
{
    __shared__ double top[32];
    const int tid = threadIdx.x, per = (n + 1023) / 1024, i0 = min(n, tid * per), i1 = min(n, i0 + per);
    double m = -INFINITY;
    for (int i = i0; i < i1; i++) m = fmax(m, w[i]);
    double x = m;
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if ((tid & 31) >= o) x = fmax(x, y);
    }
    if ((tid & 31) == 31) top[tid >> 5] = x;
    double before = __shfl_up_sync(0xffffffffu, x, 1);
    if ((tid & 31) == 0) before = -INFINITY;
    __syncthreads();
    for (int q = 0; q < tid >> 5; q++) before = fmax(before, top[q]);
    for (int i = i0; i < i1; i++) {
        if (w[i] < before) w[i] = before;
        before = fmax(before, w[i]);
    }
}

}  // namespace

// the eigenvalues of T = tridiag(e, d, e), ascending, into w; work: 8 doubles
int tridiag_values(cudaStream_t st, int n, const double *d, const double *e, double *w, double *work)
{
    if (n < 1) return BSRG_OK;
    sturm_bounds_kernel<<<1, 1024, 0, st>>>(n, d, e, work);
    // fewer lanes per eigenvalue make fewer counts but longer chains, as long as the chains alone fill the SMs
    // (32 / 16 / 8 lanes: 104 / 108 / 135 us at n = 344, 549 / 431 / 537 at 1564, 1418 / 1194 / 997 at 2934,
    // 8045 / 5888 / 3968 at 7810)
    const auto grid = [&](int lanes) { return (unsigned)(((long)n * lanes + ST_T - 1) / ST_T); };
    if (n <= 512) sturm_kernel<32, 11><<<grid(32), ST_T, 0, st>>>(n, d, e, work, w);
    else if (n <= 2400) sturm_kernel<16, 14><<<grid(16), ST_T, 0, st>>>(n, d, e, work, w);
    else sturm_kernel<8, 18><<<grid(8), ST_T, 0, st>>>(n, d, e, work, w);
    sturm_order_kernel<<<1, 1024, 0, st>>>(n, w);
    return cuda_fail(cudaGetLastError(), "tridiagonal eigenvalues");
}

size_t dc_workspace_bytes(int n)
{
    // per level: sum over merges of 2k^2 + 8k doubles and 6k ints, at most 2n^2 + 8n doubles
    const size_t dbl = 2 * (size_t)n * n + 8 * (size_t)n + 64;
    const size_t ints = 6 * (size_t)n + 64;
    const size_t maxm = (size_t)n / (DC_LEAF / 2) + 8;
    // splits, leaf starts and sizes, merge descriptors, per-merge scalars, 256-byte alignment of 7 parts
    return dbl * 8 + ints * 4 + maxm * (3 * sizeof(int) + sizeof(DcMerge) + DC_NS * sizeof(int)) + 8 * 256 + 1024;
}

// T = tridiag(d, e) (device; d is overwritten by the torn diagonal), eigenvalues
// ascending into w, eigenvectors into Z (ldz).  ws: dc_workspace_bytes(n) device
// bytes; pinned: dc_pinned_bytes(n) bytes of pinned host staging.
size_t dc_pinned_bytes(int n)
{
    const size_t maxm = (size_t)n / (DC_LEAF / 2) + 8;
    return maxm * (3 * sizeof(int) + sizeof(DcMerge) + DC_NS * sizeof(int)) + 256;
}

// where the parts of the pinned staging lie
struct DcStaging {
    int *splits, *ls, *lk, *scal;
    DcMerge *mg;
};
static DcStaging dc_staging(int n, void *pinned)
{
    const size_t maxm = (size_t)n / (DC_LEAF / 2) + 8;
    DcStaging h;
    h.splits = (int *)pinned;
    h.ls = h.splits + maxm;
    h.lk = h.ls + maxm;
    h.mg = (DcMerge *)(((uintptr_t)(h.lk + maxm) + 15) & ~(uintptr_t)15);
    h.scal = (int *)(h.mg + maxm);
    return h;
}

double dc_gemm_flops(int n, void *pinned, int nmerge)
{
    const DcStaging h = dc_staging(n, pinned);
    double f = 0.0;
    for (int q = 0; q < nmerge; q++) {
        const double K = h.scal[DC_NS * q], n1 = h.scal[DC_NS * q + 1], n2 = h.scal[DC_NS * q + 2];
        f += 2.0 * K * (h.mg[q].k1 * (n1 + n2) + h.mg[q].k2 * (K - n1));
    }
    return f;
}

// The caller has made sure that no earlier copy still reads the staging, and leaves it alone until the
// stream is through with this call.  nmerge non-null: the counts come back too, for dc_gemm_flops.
int tridiag_dc(cudaStream_t st, int n, double *d, const double *e, double *w, double *Z, long ldz, void *ws_base,
               size_t ws_bytes, void *pinned, size_t pinned_bytes, int *nmerge, int *launches)
{
    if (nmerge) *nmerge = 0;
    if (launches) *launches = 0;
    if (n < 1) return BSRG_OK;
    int nlaunch = 0;
    if (n > DC_MAXK) { set_error("dstedc: n=%d above %d", n, DC_MAXK); return BSRG_ERR_ARG; }
    if (ws_bytes < dc_workspace_bytes(n) || pinned_bytes < dc_pinned_bytes(n)) {
        set_error("dstedc: workspace too small");
        return BSRG_ERR_NOMEM;
    }
    cudaError_t err;
    // ---- the tree (host): halves down to DC_LEAF rows ----
    std::vector<Node> leaves;                  // s, k1 = size
    std::vector<std::vector<Node>> merges;     // by depth
    std::vector<int> splits;
    struct Frame { int s, n, depth; };
    std::vector<Frame> stack{{0, n, 0}};
    while (!stack.empty()) {
        Frame f = stack.back();
        stack.pop_back();
        if (f.n <= DC_LEAF) { leaves.push_back({f.s, f.n, 0}); continue; }
        const int h = f.n / 2;
        if ((int)merges.size() <= f.depth) merges.resize(f.depth + 1);
        merges[f.depth].push_back({f.s, h, f.n - h});
        splits.push_back(f.s + h);
        stack.push_back({f.s, h, f.depth + 1});
        stack.push_back({f.s + h, f.n - h, f.depth + 1});
    }
    // ---- workspace layout ----
    char *base = (char *)ws_base;
    size_t off = 0;
    auto take = [&](size_t bytes) { off = (off + 255) & ~(size_t)255; char *p = base + off; off += bytes; return p; };
    const size_t maxm = (size_t)n / (DC_LEAF / 2) + 8;
    int *d_splits = (int *)take(sizeof(int) * maxm);
    int *d_ls = (int *)take(sizeof(int) * maxm), *d_lk = (int *)take(sizeof(int) * maxm);
    DcMerge *d_mg = (DcMerge *)take(sizeof(DcMerge) * maxm);
    int *d_scal = (int *)take(sizeof(int) * DC_NS * maxm);
    double *wsd = (double *)take(sizeof(double) * (2 * (size_t)n * n + 8 * (size_t)n + 64));
    int *wsi = (int *)take(sizeof(int) * (6 * (size_t)n + 64));
    if (off > ws_bytes || leaves.size() > maxm || splits.size() > maxm) {
        set_error("dstedc: workspace layout");
        return BSRG_ERR_NOMEM;
    }
    const DcStaging h = dc_staging(n, pinned);
    int *h_splits = h.splits, *h_ls = h.ls, *h_lk = h.lk, *h_scal = h.scal;
    DcMerge *h_mg = h.mg;
    for (size_t q = 0; q < splits.size(); q++) h_splits[q] = splits[q];
    for (size_t q = 0; q < leaves.size(); q++) { h_ls[q] = leaves[q].s; h_lk[q] = leaves[q].k1; }
    double *norm = wsd + 2 * (size_t)n * n + 8 * (size_t)n;          // after the merges' vectors
    if (!splits.empty()) {
        dc_norm_kernel<<<1, 1024, 0, st>>>(n, d, e, norm);
        if ((err = cudaMemcpyAsync(d_splits, h_splits, sizeof(int) * splits.size(), cudaMemcpyHostToDevice, st)) !=
            cudaSuccess)
            return cuda_fail(err, "dstedc upload");
        dc_tear_kernel<<<(unsigned)((splits.size() + 127) / 128), 128, 0, st>>>((int)splits.size(), d_splits, d, e);
    }
    if ((err = cudaMemcpyAsync(d_ls, h_ls, sizeof(int) * leaves.size(), cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (err = cudaMemcpyAsync(d_lk, h_lk, sizeof(int) * leaves.size(), cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return cuda_fail(err, "dstedc upload");
    dc_leaf_kernel<<<(unsigned)leaves.size(), 256, 0, st>>>(d_ls, d_lk, d, e, w, Z, ldz);
    if ((err = cudaGetLastError()) != cudaSuccess) return cuda_fail(err, "dstedc leaves");
    // ---- merges, deepest level first; the descriptors of all levels go up together ----
    int nmg = 0;
    std::vector<int> first(merges.size());
    for (int lv = (int)merges.size() - 1; lv >= 0; lv--) {
        long og = 0, ov = 0, oi = 0;
        first[lv] = nmg;
        for (const Node &N : merges[lv]) {
            DcMerge &M = h_mg[nmg++];
            const long k = N.k1 + N.k2;
            M.s = N.s; M.k1 = N.k1; M.k2 = N.k2; M.pad = 0;
            M.off_g = og; og += k * k;
            M.off_u = og; og += k * k;
            M.off_v = 2 * (long)n * n + ov; ov += 8 * k;
            M.off_i = oi; oi += 6 * k;
        }
    }
    if (nmg > 0 && (err = cudaMemcpyAsync(d_mg, h_mg, sizeof(DcMerge) * nmg, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return cuda_fail(err, "dstedc merge upload");
    const int gemm_smem = dmma::Smem<dmma::Sq, false, false>::BYTES;
    if ((err = smem_attr(dc_gemm_kernel, gemm_smem)) != cudaSuccess) return cuda_fail(err, "dstedc gemm smem");
    for (int lv = (int)merges.size() - 1; lv >= 0; lv--) {
        const std::vector<Node> &L = merges[lv];
        const int nm = (int)L.size();
        const DcMerge *mg = d_mg + first[lv];
        int *sc = d_scal + DC_NS * first[lv];
        int kmax = 0, hmax = 0;
        for (const Node &N : L) { kmax = std::max(kmax, N.k1 + N.k2); hmax = std::max(hmax, std::max(N.k1, N.k2)); }
        const int smem_prep = kmax * 21 + 64, smem_sec = 16 * kmax;
        if ((err = smem_attr(dc_prep_kernel, smem_prep)) != cudaSuccess ||
            (err = smem_attr(dc_secular_kernel, smem_sec)) != cudaSuccess)
            return cuda_fail(err, "dstedc smem");
        dc_prep_kernel<<<nm, 512, smem_prep, st>>>(mg, e, w, Z, ldz, wsd, wsi, sc, norm);
        const dim3 gg((unsigned)((kmax + 127) / 128), (unsigned)((kmax + 31) / 32), nm);
        dc_gather_kernel<<<gg, 128, 0, st>>>(mg, Z, ldz, wsd, wsi);
        dc_rotate_kernel<<<dim3((unsigned)((kmax + 127) / 128), nm), 128, 0, st>>>(mg, sc, wsd, wsi);
        dc_secular_kernel<<<dim3((unsigned)((kmax + SEC_WARPS - 1) / SEC_WARPS), nm), 32 * SEC_WARPS, smem_sec, st>>>(
            mg, sc, wsd, wsi, kmax);
        const dim3 gv((unsigned)((kmax + 7) / 8), nm);
        dc_zhat_kernel<<<gv, 256, 0, st>>>(mg, sc, wsd, wsi);
        dc_vec_kernel<<<gv, 256, 0, st>>>(mg, sc, wsd, wsi);
        dc_rank_kernel<<<nm, 256, 0, st>>>(mg, sc, wsd, wsi, w);
        const dim3 gm((unsigned)((hmax + dmma::Sq::BM - 1) / dmma::Sq::BM),
                      (unsigned)((kmax + dmma::Sq::BN - 1) / dmma::Sq::BN), (unsigned)(2 * nm));
        dc_gemm_kernel<<<gm, dmma::Sq::NT, gemm_smem, st>>>(mg, sc, wsd, wsi, Z, ldz);
        dc_copy_kernel<<<dim3((unsigned)std::min(kmax, 512), nm), 128, 0, st>>>(mg, sc, wsd, wsi, Z, ldz);
        if ((err = cudaGetLastError()) != cudaSuccess) return cuda_fail(err, "dstedc merge");
        nlaunch += 9;
    }
    // the counts, for the caller that waits for the stream anyway (dc_gemm_flops)
    if (nmerge && nmg > 0) {
        *nmerge = nmg;
        if ((err = cudaMemcpyAsync(h_scal, d_scal, sizeof(int) * DC_NS * nmg, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
            return cuda_fail(err, "dstedc counts");
    }
    if (launches) *launches = nlaunch + (splits.empty() ? 1 : 3);
    return BSRG_OK;
}

}  // namespace bsrg

using namespace bsrg;

extern "C" int bsrg_dstedc(bsrg_ctx *c, int n, const double *d, const double *e, double *w, double *Z, int ldz)
{
    if (!c || (n > 0 && (!d || !w || !Z || (n > 1 && !e)))) { set_error("dstedc: null argument"); return BSRG_ERR_ARG; }
    if (n < 0 || ldz < (n > 0 ? n : 1)) { set_error("dstedc: n=%d ldz=%d", n, ldz); return BSRG_ERR_ARG; }
    if (n == 0) return BSRG_OK;
    cudaSetDevice(c->device);
    const size_t need = dc_workspace_bytes(n) + sizeof(double) * (size_t)n + 1024;
    int rc = ctx_reserve(c, need);
    if (rc == BSRG_OK) rc = ctx_reserve_pinned(c, dc_pinned_bytes(n));
    if (rc != BSRG_OK) return rc;
    cudaStream_t s = c->stream;
    double *dt = (double *)c->ws;                        // torn copy of d
    char *rest = (char *)c->ws + (((size_t)n * sizeof(double) + 255) & ~(size_t)255);
    cudaError_t e1 = cudaEventSynchronize(c->ev_stage);   // the staging's last copies are through
    if (e1 != cudaSuccess) return cuda_fail(e1, "dstedc staging");
    e1 = cudaMemcpyAsync(dt, d, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
    if (e1 != cudaSuccess) return cuda_fail(e1, "dstedc copy");
    static const double zero = 0.0;
    rc = tridiag_dc(s, n, dt, n > 1 ? e : &zero, w, Z, ldz, rest, c->ws_bytes - (rest - (char *)c->ws), c->pinned,
                    c->pinned_bytes, nullptr, nullptr);
    if (rc != BSRG_OK) return rc;
    cudaEventRecord(c->ev_stage, s);
    return cuda_fail(cudaGetLastError(), "dstedc");
}
