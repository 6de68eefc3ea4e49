// The B-spline integral tables from the cell moments, in the reference's summation order:
//
//   mrk_cell, mmk_cell (mrk_cell.f90:2, mmk_cell.f90:2)  pairs 's','s'
//   mtk_cell           (mtk_cell.f90:2)                  pairs 'n','n'
//   mvk_cell, mwk_cell (mvk_cell.f90:2, mwk_cell.f90:2)  pairs 'n','s'
//   mnk_cell           (mnk_cell.f90:2)                  pairs 's','s', r2 < r1 only
//   mqk_cell           (mqk_cell.f90:2)                  pairs 'n','n', antisymmetric
//
// Element (i, j, ip, jp) sums, over the intervals jv of its electron-2 pair and iv of its electron-1
// pair, uA(iv) w2(jv) where iv < jv, w1(jv) uB(iv) where iv > jv, and the diagonal cell
// rkd(ii, jj, iv) where iv = jv; jv outer, iv inner, both ascending.  A pair of splines offset by
// ip has NI = ks - |offset| intervals.
//
// What bounds it: the adds.  Each element is one chain of up to NI NJ dependent, separately rounded
// multiplies and adds (ns^2 (ks (ks + 1) / 2)^2 of them in an R^k table: 14 us of the FP64 units at
// ks = 10, ns = 200), so it pays to leave nothing else in the loop:
// - the moments that the inner loop runs over lie in registers (the body is instantiated for their
//   number), those of the outer one are one shared-memory load per row of terms;
// - two elements' intervals overlap only where |i - j| < ks.  Outside this band a cell is a product
//   and its kind depends on the element alone; a warp has 32 consecutive i of one j there.  In the
//   band a warp has 32 consecutive i of one j - i, so that all its lanes reach the diagonal cell
//   at the same term.  The band's tiles come first in the grid: they take longest;
// - the moments staged for intervals outside the grid are zeros, whose products change no sum; only if
//   some moment is not finite (a high power at a small radius) the terms are tested one by one.
// Measured (ks = 10, ns = 200): R^k 188 -> 58 us; (ks = 8, ns = 150): T^k 154 -> 63, V^k 96 -> 37,
// N^k 41 -> 17 and Q^k 2278 -> 212 us, from one thread per element with every cell's kind tested and
// the moments read per term.  What is left above the adds is the per-row work of the short pairs
// (NI = 1..4) and instruction fetches: 34 M instructions, 9.5 M of them adds and multiplies.  Two
// chains per thread were no faster (72 us); three CTAs per SM beat two (70 us) and four (64 us).
// Compiled with --fmad=false: the results equal the reference's order bit for bit.
#include <algorithm>

#include "bsrg_internal.h"

namespace bsrg {
namespace {

constexpr int TI = 32, TJ = 64, NWARP = 8;   // tile: 32 i (lanes) x 64 j, or 32 i x the band's 2 ks - 1 j - i
constexpr int TQ = BSRG_MAXKS;
static_assert(TJ >= TI + 2 * (TQ - 1), "the band's columns fit the staged ones");

struct Side {                    // the pairs of one electron: moments a, b at [ii + np * iv]
    const double *a, *b;         // electron 1: uA, uB; electron 2: w1, w2
    int np;                      // pairs per interval
};
struct ExpandArgs {
    int ks, ns, nv, ldp;
    double fine;
    Side e1, e2;
    const double *rkd;           // rkd[ii + e1.np (jj + e2.np iv)]
    double *rkb;
};

// a pair stored in column p: its offset, the number of its intervals, and the place ih of its first
// spline in the first of them (one less in each next)
struct Pair {
    int off, count, ihmax;
    template <bool FULL> __device__ __forceinline__ static Pair of(int ks, int p)
    {
        Pair r;
        r.off = FULL ? p - (ks - 1) : p;
        r.count = r.off < 0 ? ks + r.off : ks - r.off;
        r.ihmax = r.off < 0 ? ks - 1 : ks - 1 - r.off;
        return r;
    }
    template <bool FULL> __device__ __forceinline__ int index(int ks, int q) const      // in its interval q
    {
        const int ih = ihmax - q;
        return FULL ? ih * ks + ih + off : ih * ks - ih * (ih - 1) / 2 + off;
    }
};

// moments of interval q of the pair whose first spline is first + x to s[q W + x], x < W, zero outside
// the grid; returns whether one of them is not finite
template <bool FULL, int W>
__device__ __forceinline__ bool stage(double *sa, double *sb, const Side &e, int ks, int nv, int first, const Pair &p)
{
    bool bad = false;
    for (int k = threadIdx.x; k < p.count * W; k += 32 * NWARP) {
        const int q = k / W, iv = first - p.ihmax + q + k % W;
        double x = 0.0, y = 0.0;
        if (iv >= 0 && iv < nv) {
            const size_t at = p.template index<FULL>(ks, q) + (size_t)e.np * iv;
            x = __ldg(e.a + at);
            y = __ldg(e.b + at);
            bad |= !isfinite(x) || !isfinite(y);
        }
        sa[k] = x;
        sb[k] = y;
    }
    return bad;
}

// acc + u[0] r + u[1] r ..., the terms lo <= q < hi alone if TEST
template <int N, bool TEST>
__device__ __forceinline__ double add_row(double acc, const double (&u)[N], double r, int lo, int hi)
{
#pragma unroll
    for (int q = 0; q < N; q++) {
        const double s = acc + u[q] * r;
        acc = (!TEST || (q >= lo && q < hi)) ? s : acc;
    }
    return acc;
}

// The elements of one (ip, jp) and one tile.  The inner loop has N terms: electron 1's intervals, or
// electron 2's for LOWER (iv outer, jv <= iv inner).
template <int N, bool FI, bool FJ, bool LOWER, bool TEST>
__device__ __forceinline__ void expand_body(const ExpandArgs &a, const double *uA, const double *uB, const double *w1,
                                            const double *w2, const Pair &pi, const Pair &pj, int i0, int j0, int ip,
                                            int jp, bool band)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ks = a.ks, nv = a.nv, ns = a.ns;
    const int i = i0 + lane, ilo = i - pi.ihmax;
    const int qlo = max(0, -ilo), qhi = min(pi.count, nv - ilo);
    double *out = a.rkb + i + (size_t)ns * ns * (ip + (size_t)a.ldp * jp);
    double ua[N], ub[N];
    if (!LOWER) {
#pragma unroll
        for (int q = 0; q < N; q++) {
            ua[q] = uA[q * TI + lane];
            ub[q] = uB[q * TI + lane];
        }
    }
    if (!band) {
        for (int jl = warp; jl < TJ; jl += NWARP) {
            const int j = j0 + jl, jlo = j - pj.ihmax;
            if (j >= ns) break;
            if (i0 > j - ks && i0 + TI - 1 < j + ks) continue;             // the warp is inside the band
            const int rlo = max(0, -jlo), rhi = min(pj.count, nv - jlo);
            double acc = 0.0;
            if (LOWER) {
                if (i0 + TI - 1 > j) {                                    // else every jv is above every iv
#pragma unroll
                    for (int r = 0; r < N; r++) ua[r] = w1[r * TJ + jl];
                    for (int q = 0; q < pi.count; q++) {
                        const double s = add_row<N, TEST>(acc, ua, uB[q * TI + lane], rlo, rhi);
                        acc = (!TEST || (q >= qlo && q < qhi)) ? s : acc;
                    }
                    if (i < j) acc = 0.0;
                }
            } else if (i0 + TI - 1 < j) {
                for (int r = rlo; r < rhi; r++) acc = add_row<N, TEST>(acc, ua, w2[r * TJ + jl], qlo, qhi);
            } else if (i0 > j) {
                for (int r = rlo; r < rhi; r++) acc = add_row<N, TEST>(acc, ub, w1[r * TJ + jl], qlo, qhi);
            } else {
                double u[N];
#pragma unroll
                for (int q = 0; q < N; q++) u[q] = i < j ? ua[q] : ub[q];
                const double *w = i < j ? w2 : w1;
                for (int r = rlo; r < rhi; r++) acc = add_row<N, TEST>(acc, u, w[r * TJ + jl], qlo, qhi);
            }
            if (i < ns && (i - j >= ks || j - i >= ks)) out[(size_t)ns * j] = acc * a.fine;
        }
        return;
    }
    for (int dd = warp; dd < 2 * ks - 1; dd += NWARP) {
        const int j = i + dd - (ks - 1), jl = lane + dd, jlo = j - pj.ihmax;   // the staged columns start at i0 - (ks - 1)
        const int rlo = max(0, -jlo), rhi = min(pj.count, nv - jlo);
        const int shift = dd - (ks - 1) - pj.ihmax + pi.ihmax;              // interval r of j is interval r + shift of i
        double acc = 0.0;
        if (!LOWER) {
            for (int r = 0; r < pj.count; r++) {
                const int d = r + shift;
                const double x1 = w1[r * TJ + jl], x2 = w2[r * TJ + jl];
                double diag = 0.0;
                if (d >= qlo && d < qhi && r >= rlo && r < rhi)
                    diag = __ldg(a.rkd + pi.template index<FI>(ks, d) +
                                 (size_t)a.e1.np * (pj.template index<FJ>(ks, r) + (size_t)a.e2.np * (jlo + r)));
                const bool in = r >= rlo && r < rhi;
#pragma unroll
                for (int q = 0; q < N; q++) {
                    double c;
                    if (q < d) c = ua[q] * x2;
                    else if (q > d) c = ub[q] * x1;
                    else c = diag;
                    const double s = acc + c;
                    acc = (!TEST || (in && q >= qlo && q < qhi)) ? s : acc;
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < N; r++) ua[r] = w1[r * TJ + jl];
            for (int q = 0; q < pi.count; q++) {
                const int d = q - shift;                                  // jv = iv at r = d
                const double x = uB[q * TI + lane];
                double diag = 0.0;
                if (d >= rlo && d < rhi && q >= qlo && q < qhi)
                    diag = __ldg(a.rkd + pi.template index<FI>(ks, q) +
                                 (size_t)a.e1.np * (pj.template index<FJ>(ks, d) + (size_t)a.e2.np * (ilo + q)));
                const bool in = q >= qlo && q < qhi;
#pragma unroll
                for (int r = 0; r < N; r++) {
                    if (r > d) continue;
                    const double c = r < d ? ua[r] * x : diag, s = acc + c;
                    acc = (!TEST || (in && r >= rlo && r < rhi)) ? s : acc;
                }
            }
        }
        if (i < ns && j >= 0 && j < ns) out[(size_t)ns * j] = acc * a.fine;
    }
}

// zeros in the columns past the table's
__device__ __forceinline__ void store_zero_tile(double *rkb, int ns, int ldp, int i0, int j0, int ip, int jp, bool band,
                                                double zero)
{
    const int i = i0 + (threadIdx.x & 31);
    if (band) return;
    for (int j = j0 + (threadIdx.x >> 5); j < min(ns, j0 + TJ); j += NWARP)
        if (i < ns) rkb[i + (size_t)ns * (j + (size_t)ns * (ip + (size_t)ldp * jp))] = zero;
}

template <bool FI, bool FJ, bool LOWER> __global__ void __launch_bounds__(32 * NWARP, 3) expand_kernel(ExpandArgs a)
{
    __shared__ double uA[TQ * TI], uB[TQ * TI], w1[TQ * TJ], w2[TQ * TJ];
    const int ip = blockIdx.z % a.ldp, jp = blockIdx.z / a.ldp, ks = a.ks;
    const bool band = blockIdx.y == 0;
    const int i0 = blockIdx.x * TI, j0 = band ? i0 - (ks - 1) : ((int)blockIdx.y - 1) * TJ;
    if (ip >= (FI ? 2 * ks - 1 : ks) || jp >= (FJ ? 2 * ks - 1 : ks)) {
        store_zero_tile(a.rkb, a.ns, a.ldp, i0, j0, ip, jp, band, 0.0 * a.fine);
        return;
    }
    const Pair pi = Pair::of<FI>(ks, ip), pj = Pair::of<FJ>(ks, jp);
    bool bad = stage<FI, TI>(uA, uB, a.e1, ks, a.nv, i0, pi);
    bad |= stage<FJ, TJ>(w1, w2, a.e2, ks, a.nv, j0, pj);
    const bool test = __syncthreads_or(bad);
    switch (LOWER ? pj.count : pi.count) {
#define BODY(N)                                                                                                  \
    case N:                                                                                                      \
        if (test) expand_body<N, FI, FJ, LOWER, true>(a, uA, uB, w1, w2, pi, pj, i0, j0, ip, jp, band);           \
        else expand_body<N, FI, FJ, LOWER, false>(a, uA, uB, w1, w2, pi, pj, i0, j0, ip, jp, band);               \
        break;
        BODY(1) BODY(2) BODY(3) BODY(4) BODY(5) BODY(6) BODY(7) BODY(8)
        BODY(9) BODY(10) BODY(11) BODY(12) BODY(13) BODY(14) BODY(15) BODY(16)
#undef BODY
    }
}

// mqk_cell adds every cell term to rkb(i, j, ip, jp) and subtracts it from rkb(j, i, jp, ip), jv outer.
// An element (i, j, ip, jp) so gets, per jv, its added block (iv over the intervals of (i, ip), if jv
// is one of (j, jp)'s) and its subtracted block (iv over (j, jp)'s, if jv is one of (i, ip)'s), in the
// order of the loops over (jh, jhp): the added block first if j < i, or j = i and jp < ip.  Outside
// the band the two ranges are apart and the lower one's blocks all come first.
struct QArgs {
    int ks, ns, nv, ldp;
    double fine;
    const double *r1, *r2, *r3, *r4, *rkd;      // (ks*ks, nv) each; rkd (ks*ks, ks*ks, nv)
    double *rkb;
    int z0;                                     // the launch's first pair of columns
};

// acc +- sum over the outer lo..hi-1 of x[outer] (row of inner terms y); the outer moments in registers,
// the inner ones read in order
template <int N, bool TEST>
__device__ __forceinline__ double sub_rows(double acc, const double (&x)[N], const double *y, int lo, int hi, int ylo,
                                           int yhi)
{
#pragma unroll
    for (int q = 0; q < N; q++) {
#pragma unroll 4
        for (int r = ylo; r < yhi; r++) {
            const double s = acc - y[r * TJ] * x[q];
            acc = (!TEST || (q >= lo && q < hi)) ? s : acc;
        }
    }
    return acc;
}

template <int N, bool TEST>
__device__ __forceinline__ void qk_body(const QArgs &a, const double (*I)[TQ * TI], const double (*J)[TQ * TJ],
                                        const Pair &pi, const Pair &pj, int i0, int j0, int ip, int jp, bool band)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ks = a.ks, nv = a.nv, ns = a.ns, jk = ks * ks;
    const int i = i0 + lane, ilo = i - pi.ihmax, qlo = max(0, -ilo), qhi = min(N, nv - ilo);
    double *out = a.rkb + i + (size_t)ns * ns * (ip + (size_t)a.ldp * jp);
    if (!band) {
        for (int jl = warp; jl < TJ; jl += NWARP) {
            const int j = j0 + jl, jlo = j - pj.ihmax;
            if (j >= ns) break;
            if (i0 > j - ks && i0 + TI - 1 < j + ks) continue;
            const int rlo = max(0, -jlo), rhi = min(pj.count, nv - jlo);
            double acc = 0.0, x[N];
            if (i < j) {                                    // jv of (i, ip) first: iv of (j, jp) above it
#pragma unroll
                for (int q = 0; q < N; q++) x[q] = I[0][q * TI + lane];
                acc = sub_rows<N, TEST>(acc, x, J[3] + jl, qlo, qhi, rlo, rhi);
#pragma unroll
                for (int q = 0; q < N; q++) x[q] = I[2][q * TI + lane];
                for (int r = rlo; r < rhi; r++) acc = add_row<N, TEST>(acc, x, J[1][r * TJ + jl], qlo, qhi);
            } else {
#pragma unroll
                for (int q = 0; q < N; q++) x[q] = I[3][q * TI + lane];
                for (int r = rlo; r < rhi; r++) acc = add_row<N, TEST>(acc, x, J[0][r * TJ + jl], qlo, qhi);
#pragma unroll
                for (int q = 0; q < N; q++) x[q] = I[1][q * TI + lane];
                acc = sub_rows<N, TEST>(acc, x, J[2] + jl, qlo, qhi, rlo, rhi);
            }
            if (i < ns && (i - j >= ks || j - i >= ks)) out[(size_t)ns * j] = acc * a.fine;
        }
        return;
    }
    // the band: the lanes share j - i, and with it which block comes first and where iv reaches jv
    for (int dd = warp; dd < 2 * ks - 1; dd += NWARP) {
        const int D = dd - (ks - 1), j = i + D, jl = lane + dd, jlo = j - pj.ihmax;
        const int rlo = max(0, -jlo), rhi = min(pj.count, nv - jlo);
        const int shift = D - pj.ihmax + pi.ihmax;          // interval r of j is interval r + shift of i
        const bool self = D == 0 && ip == jp, add_first = D < 0 || (D == 0 && jp < ip);
        double acc = 0.0;
        for (int q = min(0, shift); q < max(N, pj.count + shift); q++) {        // jv = ilo + q = jlo + r
            const int r = q - shift, jv = ilo + q;
            const bool okA = r >= 0 && r < pj.count, okS = q >= 0 && q < N;
            const bool vA = okA && r >= rlo && r < rhi, vS = okS && q >= qlo && q < qhi;
            for (int pass = 0; pass < 2; pass++) {
                if ((pass == 0) == add_first || self) {
                    if (!okA || (self && pass)) continue;
                    const double x1 = J[0][r * TJ + jl], x2 = J[1][r * TJ + jl];
                    const size_t at = (size_t)jk * (pj.template index<true>(ks, r) + (size_t)jk * max(jv, 0));
                    for (int p = 0; p < N; p++) {           // iv = ilo + p
                        const bool v = vA && p >= qlo && p < qhi;
                        double c;
                        if (p < q) c = I[2][p * TI + lane] * x2;
                        else if (p > q) c = x1 * I[3][p * TI + lane];
                        else c = v ? __ldg(a.rkd + pi.template index<true>(ks, p) + at) : 0.0;
                        double s = acc + c;
                        if (self) s = s - c;
                        acc = (!TEST || v) ? s : acc;
                    }
                } else {
                    if (!okS) continue;
                    const double x1 = I[0][q * TI + lane], x2 = I[1][q * TI + lane];
                    const size_t at = (size_t)jk * (pi.template index<true>(ks, q) + (size_t)jk * max(jv, 0));
                    for (int p = 0; p < pj.count; p++) {    // iv = jlo + p
                        const bool v = vS && p >= rlo && p < rhi;
                        double c;
                        if (p < r) c = J[2][p * TJ + jl] * x2;
                        else if (p > r) c = x1 * J[3][p * TJ + jl];
                        else c = v ? __ldg(a.rkd + pj.template index<true>(ks, p) + at) : 0.0;
                        const double s = acc - c;
                        acc = (!TEST || v) ? s : acc;
                    }
                }
            }
        }
        if (i < ns && j >= 0 && j < ns) out[(size_t)ns * j] = acc * a.fine;
    }
}

__global__ void __launch_bounds__(32 * NWARP) qk_expand_kernel(QArgs a)
{
    extern __shared__ double qsm[];                         // r1, r2, r3, r4 of the i pairs, then of the j pairs
    double (*I)[TQ * TI] = (double (*)[TQ * TI])qsm, (*J)[TQ * TJ] = (double (*)[TQ * TJ])(qsm + 4 * TQ * TI);
    const int z = a.z0 + (int)blockIdx.z, ip = z % a.ldp, jp = z / a.ldp, ks = a.ks;
    const bool band = blockIdx.y == 0;
    const int i0 = blockIdx.x * TI, j0 = band ? i0 - (ks - 1) : ((int)blockIdx.y - 1) * TJ;
    if (ip >= 2 * ks - 1 || jp >= 2 * ks - 1) {
        store_zero_tile(a.rkb, a.ns, a.ldp, i0, j0, ip, jp, band, 0.0 * a.fine);
        return;
    }
    const Pair pi = Pair::of<true>(ks, ip), pj = Pair::of<true>(ks, jp);
    const Side s12{a.r1, a.r2, ks * ks}, s34{a.r3, a.r4, ks * ks};
    bool bad = stage<true, TI>(I[0], I[1], s12, ks, a.nv, i0, pi);
    bad |= stage<true, TI>(I[2], I[3], s34, ks, a.nv, i0, pi);
    bad |= stage<true, TJ>(J[0], J[1], s12, ks, a.nv, j0, pj);
    bad |= stage<true, TJ>(J[2], J[3], s34, ks, a.nv, j0, pj);
    const bool test = __syncthreads_or(bad);
    switch (pi.count) {
#define BODY(N)                                                                       \
    case N:                                                                           \
        if (test) qk_body<N, true>(a, I, J, pi, pj, i0, j0, ip, jp, band);             \
        else qk_body<N, false>(a, I, J, pi, pj, i0, j0, ip, jp, band);                 \
        break;
        BODY(1) BODY(2) BODY(3) BODY(4) BODY(5) BODY(6) BODY(7) BODY(8)
        BODY(9) BODY(10) BODY(11) BODY(12) BODY(13) BODY(14) BODY(15) BODY(16)
#undef BODY
    }
}

dim3 tiles(const bsrg_basis *b, int ldp)
{
    return dim3((b->ns + TI - 1) / TI, (b->ns + TJ - 1) / TJ + 1, ldp * ldp);
}

}  // namespace

int launch_mrk_cell_scaled(const bsrg_basis *b, const double *rkd1, const double *rkd2, const double *rkd,
                           double fine, double *rkb, int ldp, cudaStream_t s)
{
    const int ik = ik_of(b->ks);
    const ExpandArgs a{b->ks, b->ns, b->nv, ldp, fine, {rkd1, rkd2, ik}, {rkd1, rkd2, ik}, rkd, rkb};
    expand_kernel<false, false, false><<<tiles(b, ldp), 32 * NWARP, 0, s>>>(a);
    return cuda_fail(cudaGetLastError(), "mrk_cell");
}

int launch_mrk_cell(const bsrg_basis *b, const double *rkd1, const double *rkd2, const double *rkd,
                    double *rkb, int ldp, cudaStream_t s)
{
    return launch_mrk_cell_scaled(b, rkd1, rkd2, rkd, 1.0, rkb, ldp, s);
}

int launch_mnk_cell(const bsrg_basis *b, const double *rkd1, const double *rkd2, const double *rkd, double fine,
                    double *rkb, int ldp, cudaStream_t s)
{
    const int ik = ik_of(b->ks);
    const ExpandArgs a{b->ks, b->ns, b->nv, ldp, fine, {rkd1, rkd2, ik}, {rkd1, rkd2, ik}, rkd, rkb};
    expand_kernel<false, false, true><<<tiles(b, ldp), 32 * NWARP, 0, s>>>(a);
    return cuda_fail(cudaGetLastError(), "mnk_cell");
}

int launch_mtk_cell(const bsrg_basis *b, int k, const double *rkd1, const double *rkd2, const double *rkd,
                    double fine, double *rkb, int ldp, cudaStream_t s)
{
    const int jk = b->ks * b->ks;
    const ExpandArgs a{b->ks, b->ns, b->nv, ldp, fine / (k + k + 1), {rkd1, rkd2, jk}, {rkd1, rkd2, jk}, rkd, rkb};
    expand_kernel<true, true, false><<<tiles(b, ldp), 32 * NWARP, 0, s>>>(a);
    return cuda_fail(cudaGetLastError(), "mtk_cell");
}

int launch_mvk_cell(const bsrg_basis *b, const double *rkd1, const double *rkd2, const double *rkd3,
                    const double *rkd4, const double *rkd, double fine, double *rkb, int ldp, cudaStream_t s)
{
    const ExpandArgs a{b->ks, b->ns, b->nv, ldp, fine, {rkd3, rkd4, b->ks * b->ks}, {rkd1, rkd2, ik_of(b->ks)}, rkd,
                       rkb};
    expand_kernel<true, false, false><<<tiles(b, ldp), 32 * NWARP, 0, s>>>(a);
    return cuda_fail(cudaGetLastError(), "mvk_cell");
}

int launch_mqk_cell(const bsrg_basis *b, const double *rkd1, const double *rkd2, const double *rkd3,
                    const double *rkd4, const double *rkd, double fine, double *rkb, int ldp, cudaStream_t s)
{
    QArgs a{b->ks, b->ns, b->nv, ldp, fine, rkd1, rkd2, rkd3, rkd4, rkd, rkb, 0};
    const int shm = 4 * TQ * (TI + TJ) * (int)sizeof(double);
    cudaError_t e = smem_attr(qk_expand_kernel, shm);
    if (e != cudaSuccess) return cuda_fail(e, "mqk_cell smem");
    // a grid's z ends at 65535: more pairs of columns (ldp > 255) take more launches
    dim3 grd = tiles(b, ldp);
    for (const int pairs = (int)grd.z; a.z0 < pairs; a.z0 += 65535) {
        grd.z = (unsigned)std::min(65535, pairs - a.z0);
        qk_expand_kernel<<<grd, 32 * NWARP, shm, s>>>(a);
    }
    return cuda_fail(cudaGetLastError(), "mqk_cell");
}

}  // namespace bsrg
