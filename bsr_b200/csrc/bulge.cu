// Band -> tridiagonal by bulge chasing (stage 2 of the two-stage eigensolver).
//
// Band storage: A(r, c), r >= c, r - c < 2NB, at AB[(r - c) + 2NB c] (the NB rows
// below the band hold the bulges).  Sweep j annihilates column j below the
// subdiagonal and chases the bulge: step (j, i) has the window rows
// r0 = j + 1 + i NB .. r1 - 1, r1 = min(r0 + NB, n), and one reflector H_i, made from
// the column x_i (column j for i = 0, else the first column of the block B_{i-1}).
// With D_i the diagonal block of the window and B_i the NB rows below it, the sweep
// does, for every i,
//     D_i <- H_i D_i H_i        B_i <- H_{i+1} (B_i H_i).
// A later sweep's step i reads only elements of D_i, D_{i+1}, B_i and B_{i+1} of this one (rows
// and columns shifted by one), and the elements below them are zeros that no sweep has touched.
//
// Sweeps run concurrently, one CTA each.  Every element is stored as a pair (value, number of
// sweeps that have written it) in one 16-byte access, so a sweep loads its blocks straight from
// the band and looks at the counts: there is no flag between the sweeps, and no fence.  Each
// element of a sweep's blocks is read once and written once by that sweep, after its count
// showed the previous sweep's write, so no write can overtake a read.
#include <algorithm>

#include "bsrg_internal.h"
#include "syevd2.h"

namespace bsrg {
namespace {

constexpr int XR = 8;               // ring of columns x_i
constexpr int BR = 4;               // rings of staged blocks B_i and D_i
constexpr int LB = 4, LDW = 4;      // warps that load B_i and D_i, NB / LB and NB / LDW columns each
constexpr int LD = NB + 1;
constexpr int BULGE_NT = 32 * (3 + LB + LDW);

struct BulgeArgs {
    ulonglong2 *AB;                 // (bits of the value, sweeps that have written it)
    int n;
    double *V2, *tau2;
    int S;
    int *err;
    unsigned *ticket;               // the next sweep
};

struct BulgeSmem {
    double x[XR][NB];
    double qs[NB];                  // kappa_{i+1} B^T u_{i+1}
    double us[NB], ws[NB];          // u_i and w of the D update
    double beta[XR], binv[XR];      // binv = 1 / beta, 0 when H_i is the identity
    double B[BR][NB][LD], D[BR][NB][LD];
    double Bt[NB][LD];              // B_i H_i
    int bready[LB], dready[LDW];    // steps staged, per loading warp
    int vready, doneB, doneD;       // steps whose reflector is known, whose blocks are stored
    int quit, sweep;
};

__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("{ .reg .b128 q; ld.relaxed.gpu.global.b128 q, [%2]; mov.b128 {%0, %1}, q; }"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void st_pair(ulonglong2 *p, double x, unsigned long long count)
{
    asm volatile("{ .reg .b128 q; mov.b128 q, {%1, %2}; st.relaxed.gpu.global.b128 [%0], q; }" ::"l"(p),
                 "l"((unsigned long long)__double_as_longlong(x)), "l"(count));
}

// A bounded wait: step() is called once a poll and returns false when the wait is to be given up
// (WAIT_NS has passed, which sets the error flag, or another warp or CTA has given up).
struct Patience {
    int *quit, *err;
    int spin = 0;
    unsigned long long t0 = 0;
    __device__ Patience(int *q, int *e) : quit(q), err(e) {}
    __device__ __forceinline__ bool step(int every)
    {
        if (*(volatile int *)quit) return false;
        if (++spin < every) return true;
        spin = 0;
        const unsigned long long t = gtime();
        if (t0 == 0) t0 = t;
        if (t - t0 > WAIT_NS) atomicExch(err, 2);
        if (*(volatile int *)err) {
            *(volatile int *)quit = 1;
            return false;
        }
        return true;
    }
};

// Wait until every one of N flags is >= need (one warp; the result is the same on every lane).
template <int N> __device__ __forceinline__ bool wait_flags(const int *flag, int need, int *quit, int *err)
{
    auto there = [&] {
        int v = ((volatile const int *)flag)[0];
#pragma unroll
        for (int q = 1; q < N; q++) v = min(v, ((volatile const int *)flag)[q]);
        return v >= need;
    };
    bool ok = true;
    if (!there()) {
        Patience pat(quit, err);
        while (!there())
            if (!pat.step(1024)) { ok = false; break; }
    }
    ok = __all_sync(0xffffffffu, ok);
    __threadfence_block();
    return ok;
}

// Loads the K pairs p[c * (LDAB - 1)], c < K, of this lane, all in flight at once (0 where need(c) is
// false), again until each has been written by `count` sweeps.  `any` is some address of the band.
template <int K, class Need>
__device__ __forceinline__ bool load_pairs(const ulonglong2 *p, const ulonglong2 *any, Need need,
                                           unsigned long long count, double (&x)[K], int *quit, int *err)
{
    Patience pat(quit, err);
    for (;;) {
        ulonglong2 v[K];
        bool there = true;
#pragma unroll
        for (int c = 0; c < K; c++) v[c] = ld_pair(need(c) ? p + c * (LDAB - 1) : any);
#pragma unroll
        for (int c = 0; c < K; c++) {
            x[c] = need(c) ? __longlong_as_double((long long)v[c].x) : 0.0;
            there &= (v[c].y >= count) | !need(c);
        }
        if (__all_sync(0xffffffffu, there)) return true;
        if (!__all_sync(0xffffffffu, pat.step(64))) return false;
    }
}

// What bounds it: the dependency chain.  Sweep j+1 follows sweep j at a distance of a few steps, so
// the run takes about n times that distance, whatever the arithmetic's rate.
// - Inside a sweep the chain is x_i -> x_{i+1}, and H_i x_i = beta e_1 gives x_{i+1} = B_i H_i e_1
//   = B_i x_i / beta: one product and one reciprocal square root, with neither the reflector's
//   scaling nor any update of B_i on the way.  Warp 0 does only that, and stores beta_i, the one
//   element of B_{i-1} that the next sweep would otherwise wait a step longer for.
// - The updates use the unscaled u = x - beta e_1, H = I - kappa u u^T, kappa = 1 / (beta (beta -
//   alpha)), on a warp each for B and D: B_i H_i is formed while x_{i+1} is still being made, and what
//   remains after it is one product and one rank-1 update.
// - Between two sweeps nothing but the data itself travels (the counts above).  With a flag per step,
//   the writer's fence (0.5 us), the reader's poll and fence (1 us) and its loads (1 us) followed one
//   another, and sweeps started 6.8 us apart.
// - A block is loaded by four warps, eight columns each: one warp's 32 16-byte loads took 2 us, and
//   sweeps started 6.2 us apart; with four warps a block and a warp for each update, 3.7 us.  More
//   update warps, in turns, made every warp slower (four each: 5.2 us): the rate of the shared-memory
//   and load units is what the loading warps' looks and the updates share.
// Measured (CUDA events) at n = 470, 1713, 4400, 7810: 3.0, 12.4, 33.1, 63.3 ms with the reflector,
// the right update and the reductions on the chain and a flag per step; 1.5, 6.0, 15.8, 29.1 ms so, as a cooperative
// launch with its sweeps dealt out in advance; 1.7, 6.5, 17.0, 31.4 ms with the sweeps taken by ticket from an ordinary
// launch.  A solve by itself loses those 8 % for the sake of solves side by side: a cooperative launch waits until
// all its SMs are free at once (eight symmetries on four streams: 121 ms, 145 where the calls met, against 116).
// Sweeps in flight from sweep j on: a sweep takes 2.0 us a step and follows its predecessor by 3.7 to 4 us.  More
// CTAs than that would only look for work, and keep SMs from other streams (n = 4000: 14.6 ms with steps / 1.5
// and steps / 2 CTAs, 14.9 ms with steps and steps / 2.5).
__host__ __device__ inline int sweeps_in_flight(int n, int j) { return sweep_steps(n, j) / 2 + 4; }

__global__ void __launch_bounds__(BULGE_NT, 1) bulge_kernel(BulgeArgs a)
{
    extern __shared__ __align__(16) unsigned char bulge_sm[];
    BulgeSmem &s = *(BulgeSmem *)bulge_sm;
    const int t = threadIdx.x & 31, w = threadIdx.x >> 5, n = a.n;
    ulonglong2 *AB = a.AB;
    auto at = [&](int r, int c) -> ulonglong2 * { return AB + (r - c) + (long)LDAB * c; };
    for (;;) {
        // Sweeps are taken in order, so a sweep's predecessor is done or with a CTA that is running: no wait
        // needs a CTA that is not.  The sweeps get shorter: a CTA that the rest cannot keep busy gives its SM back.
        if (threadIdx.x == 0) {
            const int next = (int)min(*(volatile unsigned *)a.ticket, (unsigned)n);
            s.sweep = next >= n - 2 || (int)blockIdx.x >= sweeps_in_flight(n, next) ? n : (int)atomicAdd(a.ticket, 1u);
        }
        __syncthreads();
        const int j = s.sweep;
        if (j >= n - 2) return;
        const int nst = sweep_steps(n, j);
        const unsigned long long before = (unsigned long long)j, after = before + 1;
        if (threadIdx.x == 0) {
            s.vready = 0;
            s.quit = 0;
            for (int m = 0; m < LB; m++) s.bready[m] = 0;
            for (int m = 0; m < LDW; m++) s.dready[m] = 0;
            s.doneB = s.doneD = 0;
        }
        __syncthreads();
        if (w == 0) {
            // ---- the chain x_i -> x_{i+1} ----
            const int L0 = min(NB, n - (j + 1));
            double x0[1];
            if (load_pairs<1>(at(j + 1 + t, j), at(j, j), [&](int) { return t < L0; }, before, x0,
                              &s.quit, a.err)) {
                s.x[0][t] = x0[0];
                __syncwarp();
                for (int i = 0; i < nst; i++) {
                    const double2 *x2 = (const double2 *)s.x[i % XR];
                    double2 xv[NB / 2];
                    double g0 = 0.0, g1 = 0.0, g2 = 0.0, g3 = 0.0;
#pragma unroll
                    for (int c = 0; c < NB / 2; c += 2) {
                        xv[c] = x2[c];
                        xv[c + 1] = x2[c + 1];
                        if (c > 0) g0 = fma(xv[c].x, xv[c].x, g0);
                        g1 = fma(xv[c].y, xv[c].y, g1);
                        g2 = fma(xv[c + 1].x, xv[c + 1].x, g2);
                        g3 = fma(xv[c + 1].y, xv[c + 1].y, g3);
                    }
                    const double sig = (g0 + g1) + (g2 + g3), alpha = xv[0].x;
                    const double nn = fma(alpha, alpha, sig);
                    double beta = alpha, binv = 0.0;
                    if (sig != 0.0 && nn >= SMALL_SQ) {
                        binv = -copysign(rsqrt(nn), alpha);
                        beta = nn * binv;
                    }
                    if (t == 0) {
                        s.beta[i % XR] = beta;
                        s.binv[i % XR] = binv;
                        __threadfence_block();
                        *(volatile int *)&s.vready = i + 1;
                        st_pair(i == 0 ? at(j + 1, j) : at(j + 1 + i * NB, j + 1 + (i - 1) * NB), beta, after);
                    }
                    if (i + 1 == nst) break;
                    if (!wait_flags<LB>(s.bready, i + 1, &s.quit, a.err)) break;
                    double y0 = 0.0, y1 = 0.0, y2 = 0.0, y3 = 0.0, b0 = 0.0;
                    const double *Br = s.B[i % BR][t];
#pragma unroll
                    for (int c = 0; c < NB / 2; c += 2) {
                        const double e0 = Br[2 * c], e1 = Br[2 * c + 1], e2 = Br[2 * c + 2], e3 = Br[2 * c + 3];
                        if (c == 0) b0 = e0;
                        y0 = fma(e0, xv[c].x, y0);
                        y1 = fma(e1, xv[c].y, y1);
                        y2 = fma(e2, xv[c + 1].x, y2);
                        y3 = fma(e3, xv[c + 1].y, y3);
                    }
                    const double xn = binv == 0.0 ? b0 : ((y0 + y1) + (y2 + y3)) * binv;
                    // the entry of x_{i+1} last held x_{i+1-XR}, which steps i-XR and i+1-XR read
                    while (min(*(volatile int *)&s.doneB, *(volatile int *)&s.doneD) < i + 2 - XR)
                        if (*(volatile int *)&s.quit) break;
                    s.x[(i + 1) % XR][t] = xn;
                    __threadfence_block();
                    __syncwarp();
                }
            }
        } else if (w <= LB) {
            // ---- load the blocks B_i, NB / LB columns per warp ----
            constexpr int K = NB / LB;
            const int m = w - 1, cb = m * K;
            for (int i = 0; i < nst; i++) {
                const int r0 = j + 1 + i * NB, r1 = min(r0 + NB, n), L = r1 - r0, nb2 = min(NB, n - r1);
                double x[K];
                // the last row's elements left of the last column are zeros no sweep has reached
                if (!load_pairs<K>(at(r1 + t, r0 + cb), at(r0, r0),
                                   [&](int c) { return t < nb2 && cb + c < L && (t < NB - 1 || cb + c == NB - 1); },
                                   before, x, &s.quit, a.err))
                    break;
                if (!wait_flags<1>(&s.doneB, i + 1 - BR, &s.quit, a.err)) break;
#pragma unroll
                for (int c = 0; c < K; c++) s.B[i % BR][t][cb + c] = x[c];
                __threadfence_block();
                __syncwarp();
                if (t == 0) *(volatile int *)&s.bready[m] = i + 1;
            }
        } else if (w <= LB + LDW) {
            // ---- load the diagonal blocks, NB / LDW columns per warp, and mirror them ----
            constexpr int K = NB / LDW;
            const int m = w - 1 - LB, cb = m * K;
            for (int i = 0; i < nst; i++) {
                const int r0 = j + 1 + i * NB, L = min(NB, n - r0);
                double x[K];
                if (!load_pairs<K>(at(r0 + t, r0 + cb), at(r0, r0), [&](int c) { return t < L && cb + c <= t; }, before,
                                   x, &s.quit, a.err))
                    break;
                if (!wait_flags<1>(&s.doneD, i + 1 - BR, &s.quit, a.err)) break;
#pragma unroll
                for (int c = 0; c < K; c++)
                    if (cb + c <= t) {
                        s.D[i % BR][t][cb + c] = x[c];
                        s.D[i % BR][cb + c][t] = x[c];
                    }
                __threadfence_block();
                __syncwarp();
                if (t == 0) *(volatile int *)&s.dready[m] = i + 1;
            }
        } else if (w == 1 + LB + LDW) {
            // ---- B_i <- H_{i+1} B_i H_i ----
            double *qs = s.qs;
            double (*Bt)[LD] = s.Bt;
            for (int i = 0; i < nst; i++) {
                const int r0 = j + 1 + i * NB, r1 = min(r0 + NB, n), L = r1 - r0, nb2 = min(NB, n - r1);
                const bool last = i + 1 == nst;
                if (!wait_flags<LB>(s.bready, i + 1, &s.quit, a.err)) break;
                double Br[NB];
#pragma unroll
                for (int c = 0; c < NB; c++) Br[c] = s.B[i % BR][t][c];
                if (!wait_flags<1>(&s.vready, i + 1, &s.quit, a.err)) break;
                {
                    const double2 *x2 = (const double2 *)s.x[i % XR];
                    const double beta = s.beta[i % XR], binv = s.binv[i % XR], u0 = x2[0].x - beta;
                    const double kap = binv == 0.0 ? 0.0 : -binv / u0;
                    double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
#pragma unroll
                    for (int c = 0; c < NB / 2; c += 2) {
                        const double2 u = x2[c], v = x2[c + 1];
                        p0 = fma(Br[2 * c], c == 0 ? u0 : u.x, p0);
                        p1 = fma(Br[2 * c + 1], u.y, p1);
                        p2 = fma(Br[2 * c + 2], v.x, p2);
                        p3 = fma(Br[2 * c + 3], v.y, p3);
                    }
                    const double pa = -kap * ((p0 + p1) + (p2 + p3));
#pragma unroll
                    for (int c = 0; c < NB / 2; c++) {
                        const double2 u = x2[c];
                        Br[2 * c] = fma(pa, c == 0 ? u0 : u.x, Br[2 * c]);
                        Br[2 * c + 1] = fma(pa, u.y, Br[2 * c + 1]);
                    }
                }
                if (!last) {
                    __syncwarp();                           // the warp's last reads of Bt and qs are over
#pragma unroll
                    for (int c = 0; c < NB; c++) Bt[t][c] = Br[c];
                    __syncwarp();
                    if (!wait_flags<1>(&s.vready, i + 2, &s.quit, a.err)) break;
                    const double2 *x2 = (const double2 *)s.x[(i + 1) % XR];
                    const double beta = s.beta[(i + 1) % XR], binv = s.binv[(i + 1) % XR], u0 = x2[0].x - beta;
                    double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0;
#pragma unroll
                    for (int r = 0; r < NB / 2; r += 2) {
                        const double2 u = x2[r], v = x2[r + 1];
                        q0 = fma(Bt[2 * r][t], r == 0 ? u0 : u.x, q0);
                        q1 = fma(Bt[2 * r + 1][t], u.y, q1);
                        q2 = fma(Bt[2 * r + 2][t], v.x, q2);
                        q3 = fma(Bt[2 * r + 3][t], v.y, q3);
                    }
                    const double kap = binv == 0.0 ? 0.0 : -binv / u0;
                    qs[t] = kap * ((q0 + q1) + (q2 + q3));
                    const double ut = t == 0 ? -u0 : -s.x[(i + 1) % XR][t];
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < NB; c += 2) {
                        const double2 qa = *(const double2 *)(qs + c);
                        Br[c] = fma(ut, qa.x, Br[c]);
                        Br[c + 1] = fma(ut, qa.y, Br[c + 1]);
                    }
                    Br[0] = 0.0;                            // column 0 is beta_{i+1} e_1, its head stored by warp 0
                }
                if (t < nb2) {
#pragma unroll
                    for (int c = 0; c < NB; c++)
                        if (c < L && (c > 0 || t > 0 || last)) st_pair(at(r1 + t, r0 + c), Br[c], after);
                }
                __syncwarp();
                if (t == 0) *(volatile int *)&s.doneB = i + 1;
            }
        } else {
            // ---- D_i <- H_i D_i H_i, and the reflector to its place ----
            double *us = s.us, *ws = s.ws;
            for (int i = 0; i < nst; i++) {
                const int r0 = j + 1 + i * NB, r1 = min(r0 + NB, n), L = r1 - r0;
                if (!wait_flags<LDW>(s.dready, i + 1, &s.quit, a.err)) break;
                double Dr[NB];
#pragma unroll
                for (int c = 0; c < NB; c++) Dr[c] = s.D[i % BR][t][c];
                if (!wait_flags<1>(&s.vready, i + 1, &s.quit, a.err)) break;
                const double alpha = s.x[i % XR][0], beta = s.beta[i % XR], binv = s.binv[i % XR], u0 = alpha - beta;
                const double u = t == 0 ? u0 : s.x[i % XR][t];
                __syncwarp();                               // the warp's last reads of us and ws are over
                us[t] = u;
                __syncwarp();
                double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
#pragma unroll
                for (int c = 0; c < NB; c += 4) {
                    const double2 ua = *(const double2 *)(us + c), ub = *(const double2 *)(us + c + 2);
                    p0 = fma(Dr[c], ua.x, p0);
                    p1 = fma(Dr[c + 1], ua.y, p1);
                    p2 = fma(Dr[c + 2], ub.x, p2);
                    p3 = fma(Dr[c + 3], ub.y, p3);
                }
                const double kap = binv == 0.0 ? 0.0 : -binv / u0;
                const double p = t < L ? kap * ((p0 + p1) + (p2 + p3)) : 0.0;
                double up = u * p;
                for (int o = 16; o > 0; o >>= 1) up += __shfl_xor_sync(0xffffffffu, up, o);
                const double wv = p - 0.5 * kap * up * u;
                ws[t] = wv;
                __syncwarp();
#pragma unroll
                for (int c = 0; c < NB; c += 2) {
                    const double2 ua = *(const double2 *)(us + c), wa = *(const double2 *)(ws + c);
                    Dr[c] -= u * wa.x + wv * ua.x;
                    Dr[c + 1] -= u * wa.y + wv * ua.y;
                }
                if (t < L) {
#pragma unroll
                    for (int c = 0; c < NB; c++)
                        if (c <= t) st_pair(at(r0 + t, r0 + c), Dr[c], after);
                }
                // a last row that no window of this sweep reaches is passed on as it is
                if (i + 1 == nst && r1 == n - 1) {
                    double corner[1];
                    if (!load_pairs<1>(at(n - 1, n - 1), at(n - 1, n - 1), [&](int) { return true; }, before, corner,
                                       &s.quit, a.err))
                        break;
                    if (t == 0) st_pair(at(n - 1, n - 1), corner[0], after);
                }
                const double scale = binv == 0.0 ? 0.0 : 1.0 / u0;
                if (a.V2) a.V2[((long)j * a.S + i) * NB + t] = t == 0 ? 1.0 : (t < L ? u * scale : 0.0);
                if (t == 0 && a.V2) a.tau2[(long)j * a.S + i] = binv == 0.0 ? 0.0 : 1.0 - alpha * binv;
                __syncwarp();
                if (t == 0) *(volatile int *)&s.doneD = i + 1;
            }
        }
        // (in this CTA's shared memory, so that its threads agree; a CTA that has not waited in vain finds the flag in
        // its next wait)
        __syncthreads();
        if (*(volatile int *)&s.quit) return;
    }
}

// (value, 0) pairs of the band AB(d, c) = A(c + d, c), d <= NB, and zeros below it
__global__ void band_extract_kernel(int n, const double *__restrict__ A, long lda, ulonglong2 *AB)
{
    const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (idx >= (long)n * LDAB) return;
    const int d = (int)(idx % LDAB), c = (int)(idx / LDAB);
    const double x = (d <= NB && c + d < n) ? A[(c + d) + lda * (long)c] : 0.0;
    AB[idx] = make_ulonglong2((unsigned long long)__double_as_longlong(x), 0ull);
}

// d(c) = A(c, c), e(c) = A(c+1, c)
__global__ void tridiag_extract_kernel(int n, const ulonglong2 *__restrict__ AB, double *d, double *e)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    d[c] = __longlong_as_double((long long)AB[(long)LDAB * c].x);
    if (c + 1 < n) e[c] = __longlong_as_double((long long)AB[1 + (long)LDAB * c].x);
}

}  // namespace

int band_extract(int n, const double *A, long lda, double *AB, cudaStream_t st)
{
    band_extract_kernel<<<(unsigned)(((long)n * LDAB + 255) / 256), 256, 0, st>>>(n, A, lda, (ulonglong2 *)AB);
    return cuda_fail(cudaGetLastError(), "dsyevd band");
}

int bulge_chase(int n, double *AB, double *d, double *e, double *V2, double *tau2, int S, int *err, unsigned *ticket,
                int nsm, cudaStream_t st)
{
    cudaError_t rc;
    if (n > 2) {
        rc = smem_attr(bulge_kernel, sizeof(BulgeSmem));
        if (rc != cudaSuccess) return cuda_fail(rc, "dsyevd bulge chasing smem");
        // an ordinary launch: it starts with the SMs that other streams leave
        const int ctas = std::max(1, std::min(n - 2, std::min(nsm, sweeps_in_flight(n, 0))));
        BulgeArgs a{(ulonglong2 *)AB, n, V2, tau2, S, err, ticket};
        bulge_kernel<<<ctas, BULGE_NT, sizeof(BulgeSmem), st>>>(a);
        if ((rc = cudaGetLastError()) != cudaSuccess) return cuda_fail(rc, "dsyevd bulge chasing");
    }
    tridiag_extract_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, (const ulonglong2 *)AB, d, e);
    return cuda_fail(cudaGetLastError(), "dsyevd tridiagonal");
}

}  // namespace bsrg
