// Dense -> band (stage 1 of the two-stage eigensolver): per panel of NB columns a Householder QR of the
// rows below the band, A22 <- (I - V T V^T)^T A22 (I - V T V^T) as FP64 tensor-core products
//     X = A22 V,  W = X T,  Y = W - 1/2 V (T^T V^T W),  A22 -= V Y^T + Y V^T
// (the last as one product of inner size 2 NB over the [V | Y | V] buffer).  The next panel's columns are
// updated first and the next panel is factorised on a second stream beside the rest of the update.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "ctx.h"
#include "dgemm.h"
#include "dmma.cuh"
#include "syevd2.h"

namespace bsrg {
namespace {

constexpr int PQ_ROWS = 512;        // panel rows held in shared memory per CTA of the grid-barrier form
constexpr int PQ_NT = 256;

// Grid barrier (all CTAs co-resident: cooperative launch).  bar[0] arrivals,
// bar[1] generation.  A wait longer than WAIT_NS sets *err and every CTA leaves.
__device__ bool grid_sync(unsigned *bar, int *err, unsigned nblocks)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *vgen = bar + 1;
        const unsigned my = *vgen;
        __threadfence();
        if (atomicAdd(bar, 1u) == nblocks - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            const unsigned long long t0 = gtime();
            while (*vgen == my) {
                if (*(volatile int *)err) break;
                if (gtime() - t0 > WAIT_NS) { atomicExch(err, 1); break; }
            }
        }
        __threadfence();
    }
    return __syncthreads_or(*(volatile int *)err) == 0;      // the whole CTA goes on, or none of it
}

// ---------------------------------------------------------------------------
// stage 1: panel QR
// ---------------------------------------------------------------------------
struct PanelArgs {
    double *P;          // panel (m x NB), leading dimension ldp: rows j+NB.., columns j..j+NB-1 of A
    long ldp;
    int m, rpc;         // rows, rows per CTA
    double *V;          // [V | Y | V] buffer (ld m): V written to columns 0..NB-1 and 2NB..3NB-1
    double *Vs;         // the saved V of this panel for the back-transformation (ld m), or null
    double *T;          // NB x NB (ld NB), upper triangular
    double *Ts;         // saved copy of T
    double *part;       // per CTA, per column parity: NB dots + NB pivot-row values
    double *gram;       // per CTA: NB x NB Gram partial
    unsigned *bar;
    int *err;
};

// Householder QR of the panel, LAPACK's dgeqrf/dlarfg conventions:
// H_c = I - tau_c v_c v_c^T, v_c(c) = 1, P = H_0 ... H_{NB-1} [R; 0].  This form, one grid barrier per
// column, is for devices or contexts that cannot place a 16-CTA cluster.
__global__ void __launch_bounds__(PQ_NT) panel_qr_kernel(PanelArgs a)
{
    extern __shared__ __align__(16) double ps[];       // rpc x (NB + 1)
    __shared__ double tot[NB], piv[NB], wv[NB], tau_s[NB];
    __shared__ double sc_tau, sc_scale, sc_beta;
    const int cta = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int m = a.m, r0 = cta * a.rpc, nr = max(0, min(a.rpc, m - r0));
    constexpr int LD = NB + 1;
    for (int q = tid; q < nr * NB; q += PQ_NT) {
        const int r = q % nr, c = q / nr;
        ps[r * LD + c] = a.P[(r0 + r) + a.ldp * (long)c];
    }
    const int kb = min(m, NB);
    __syncthreads();
    for (int c = 0; c < kb; c++) {
        double *buf = a.part + ((long)cta * 2 + (c & 1)) * 2 * NB;
        // partial dots over my rows below the pivot: g_k = sum P(r, c) P(r, k), k >= c
        for (int k = c + warp; k < NB; k += PQ_NT / 32) {
            double s = 0.0;
            for (int r = lane; r < nr; r += 32)
                if (r0 + r > c) s += ps[r * LD + c] * ps[r * LD + k];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) buf[k] = s;
        }
        if (cta == 0)
            for (int k = c + tid; k < NB; k += PQ_NT) buf[NB + k] = ps[c * LD + k];
        __threadfence();
        if (!grid_sync(a.bar, a.err, G)) return;
        for (int k = c + tid; k < NB; k += PQ_NT) {
            double s = 0.0;
            for (int q = 0; q < G; q++) s += __ldcg(a.part + ((long)q * 2 + (c & 1)) * 2 * NB + k);
            tot[k] = s;
            piv[k] = __ldcg(a.part + (c & 1) * 2 * NB + NB + k);
        }
        __syncthreads();
        if (tid == 0) {
            const double alpha = piv[c], sigma = tot[c];
            const double nn = alpha * alpha + sigma;
            if (sigma == 0.0 || nn < SMALL_SQ) { sc_tau = 0.0; sc_scale = 0.0; sc_beta = alpha; }
            else {
                const double beta = -copysign(sqrt(nn), alpha);
                sc_tau = (beta - alpha) / beta;
                sc_scale = 1.0 / (alpha - beta);
                sc_beta = beta;
            }
            tau_s[c] = sc_tau;
        }
        __syncthreads();
        const double tau = sc_tau, scale = sc_scale;
        for (int k = c + 1 + tid; k < NB; k += PQ_NT) wv[k] = piv[k] + scale * tot[k];   // v^T P(:, k)
        __syncthreads();
        // P(:, k) -= tau v w_k, k > c: rows below the pivot, then the pivot row (CTA 0)
        for (int q = tid; q < nr * (NB - c - 1); q += PQ_NT) {
            const int r = q % nr, k = c + 1 + q / nr;
            if (r0 + r > c) ps[r * LD + k] -= tau * scale * ps[r * LD + c] * wv[k];
        }
        if (cta == 0)
            for (int k = c + 1 + tid; k < NB; k += PQ_NT) ps[c * LD + k] -= tau * wv[k];
        __syncthreads();
        for (int r = tid; r < nr; r += PQ_NT)
            if (r0 + r > c) ps[r * LD + c] *= scale;        // v below the pivot
        if (cta == 0 && tid == 0) ps[c * LD + c] = sc_beta;
        __syncthreads();
    }
    // Gram of V (unit diagonal, zero above), partial over my rows
    double *gp = a.gram + (long)cta * NB * NB;
    for (int q = tid; q < NB * NB; q += PQ_NT) {
        const int i = q % NB, j = q / NB;
        double s = 0.0;
        if (i <= j && j < kb)
            for (int r = 0; r < nr; r++) {
                const int gr = r0 + r;
                const double vi = gr > i ? ps[r * LD + i] : (gr == i ? 1.0 : 0.0);
                const double vj = gr > j ? ps[r * LD + j] : (gr == j ? 1.0 : 0.0);
                s += vi * vj;
            }
        gp[q] = s;
    }
    // V out (unit diagonal, zeros above; columns beyond kb are zero) and the band form of the panel
    for (int q = tid; q < nr * NB; q += PQ_NT) {
        const int r = q % nr, c = q / nr, gr = r0 + r;
        const double v = c < kb ? (gr > c ? ps[r * LD + c] : (gr == c ? 1.0 : 0.0)) : 0.0;
        a.V[gr + (long)m * c] = v;
        a.V[gr + (long)m * (2 * NB + c)] = v;
        if (a.Vs) a.Vs[gr + (long)m * c] = v;
        a.P[gr + a.ldp * (long)c] = gr <= c ? ps[r * LD + c] : 0.0;
    }
    __threadfence();
    if (!grid_sync(a.bar, a.err, G)) return;
    if (cta != 0) return;
    // T from the Gram matrix: T(c,c) = tau_c, T(0:c, c) = -tau_c T(0:c, 0:c) G(0:c, c)
    double *Gs = ps;                      // reuse: NB x NB
    for (int q = tid; q < NB * NB; q += PQ_NT) {
        double s = 0.0;
        for (int g = 0; g < G; g++) s += __ldcg(a.gram + (long)g * NB * NB + q);
        Gs[q] = s;
    }
    __shared__ double Tt[NB][NB + 1];
    for (int q = tid; q < NB * NB; q += PQ_NT) Tt[q % NB][q / NB] = 0.0;
    __syncthreads();
    for (int c = 0; c < kb; c++) {
        if (tid < c) {
            double s = 0.0;
            for (int l = tid; l < c; l++) s += Tt[tid][l] * Gs[l + NB * c];
            wv[tid] = s;
        }
        __syncthreads();
        if (tid < c) Tt[tid][c] = -tau_s[c] * wv[tid];
        if (tid == 0) Tt[c][c] = tau_s[c];
        __syncthreads();
    }
    for (int q = tid; q < NB * NB; q += PQ_NT) {
        a.T[q] = Tt[q % NB][q / NB];
        if (a.Ts) a.Ts[q] = Tt[q % NB][q / NB];
    }
}

// The factorisation on one thread-block cluster.
//
// What bounds it: latency.  A column needs the panel's sums before the next can start, so a panel is 32
// dependent reductions over up to 16 CTAs however fast the arithmetic is.  Columns go in blocks of eight:
// inside a block a thread has its two rows' eight values in registers, a column's reduction carries at most
// eight sums (one cluster barrier; every CTA writes its sums into all the others' shared memory and adds
// the sixteen itself), and only after a block are the columns to its right updated, I - V8 T8^T V8^T with
// V8^T P on the tensor cores.  The same product gives the Gram blocks of T.
// Measured (CUDA events, average of the panels of a reduction): n = 7810 238 us, n = 1713 207 us with all 32
// columns' sums reduced at every column, five CTA barriers a column and T formed a column at a time at the
// end; 80 us at n = 1713 so.  The rows per CTA matter little (96 to 320: the same within 2 %).
constexpr int PC_NT = 320, PC_ROWS = 2 * PC_NT, PC_MAXG = 16, PC_W = PC_NT / 32;
constexpr int KB = 8;                // columns of a block
constexpr int PLD = NB + 1;

struct PanelSmem {
    double col[2][PC_MAXG + 1][KB];   // per column parity: every CTA's sums, then the pivot row
    double wsum[PC_W][KB], piv[KB];
    double Mw[PC_W][KB * NB];         // per warp: V8^T P over its rows
    double Rs[KB * NB + 2 * PC_MAXG]; // the entries this CTA sums, from every CTA
    double M[KB * NB];                // V8^T P over all rows
    double T8[KB][KB + 1], tau[NB];
    double Z[NB][KB];                 // T8^T V8^T P, by column of P
    double R[NB][PLD];                // CTA 0: the triangle
    double G[NB][PLD], T[NB][PLD];    // V^T V above the diagonal, T
    double ps[1];                     // rows x PLD
};
constexpr size_t panel_smem(int rpc) { return sizeof(PanelSmem) + sizeof(double) * (size_t)(rpc + 4) * PLD; }

__device__ __forceinline__ double shfl_xor_add(double v, int o) { return v + __shfl_xor_sync(0xffffffffu, v, o); }

__global__ void __launch_bounds__(PC_NT) panel_qr_cluster_kernel(PanelArgs a)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char panel_sm[];
    PanelSmem &s = *(PanelSmem *)panel_sm;
    const int cta = (int)cl.block_rank(), G = (int)cl.num_blocks(), tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int m = a.m, r0 = cta * a.rpc, nr = max(0, min(a.rpc, m - r0)), kb = min(m, NB);
    double *ps = s.ps;
    for (int c = warp; c < NB; c += PC_W) {
        for (int r = lane; r < nr; r += 32) ps[r * PLD + c] = a.P[(r0 + r) + a.ldp * (long)c];
        if (lane < 4) ps[(nr + lane) * PLD + c] = 0.0;      // the tensor-core product's rows past the end
    }
    for (int q = tid; q < NB * PLD; q += PC_NT) (&s.T[0][0])[q] = 0.0;
    if (tid < NB) s.tau[tid] = 0.0;
    const int row[2] = {tid, tid + PC_NT};
    const int vper = (KB * NB + G - 1) / G;                 // entries of V8^T P a CTA sums for all
    __syncthreads();
    for (int cb = 0; cb < NB; cb += KB) {
        double x[2][KB];
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int k = 0; k < KB; k++) x[q][k] = row[q] < nr ? ps[row[q] * PLD + cb + k] : 0.0;
#pragma unroll
        for (int j = 0; j < KB; j++) {
            const int c = cb + j;
            if (c < kb) {
                double (*buf)[KB] = s.col[j & 1];
                // this CTA's sums g_k = sum_{r > c} P(r, c) P(r, k), k = cb .. cb + 7
                double g[KB];
#pragma unroll
                for (int k = 0; k < KB; k++) {
                    const double z0 = r0 + row[0] > c ? x[0][j] : 0.0, z1 = r0 + row[1] > c ? x[1][j] : 0.0;
                    g[k] = fma(z0, x[0][k], z1 * x[1][k]);
                }
                // eight sums over 32 lanes: halves exchanged until a lane has one of them
                double g4[4], g2[2], g1;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double keep = lane & 16 ? g[k + 4] : g[k], send = lane & 16 ? g[k] : g[k + 4];
                    g4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
                }
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const double keep = lane & 8 ? g4[k + 2] : g4[k], send = lane & 8 ? g4[k] : g4[k + 2];
                    g2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
                }
                {
                    const double keep = lane & 4 ? g2[1] : g2[0], send = lane & 4 ? g2[0] : g2[1];
                    g1 = keep + __shfl_xor_sync(0xffffffffu, send, 4);
                }
                g1 = shfl_xor_add(g1, 2);
                g1 = shfl_xor_add(g1, 1);
                if ((lane & 3) == 0) s.wsum[warp][(lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1)] = g1;
                if (cta == 0 && tid == c) {
#pragma unroll
                    for (int k = 0; k < KB; k++) s.piv[k] = x[0][k];
                }
                __syncthreads();
                if (warp == 0) {
                    const int k = lane & 7, q = lane >> 3;
                    double v = s.wsum[q][k] + s.wsum[q + 4][k];
                    if (q + 8 < PC_W) v += s.wsum[q + 8][k];
                    v = shfl_xor_add(v, 8);
                    v = shfl_xor_add(v, 16);
                    for (int d = q; d < G; d += 4) *cl.map_shared_rank(&buf[cta][k], d) = v;
                    if (cta == 0) {                           // and the pivot row
                        const double pv = s.piv[k];
                        for (int d = q; d < G; d += 4) *cl.map_shared_rank(&buf[PC_MAXG][k], d) = pv;
                    }
                }
                cl.sync();
                double tot = 0.0;
                {
                    const int k = lane & 7, q = lane >> 3;
                    for (int d = q; d < G; d += 4) tot += buf[d][k];
                    tot = shfl_xor_add(tot, 8);
                    tot = shfl_xor_add(tot, 16);
                }
                const double piv = buf[PC_MAXG][lane & 7];
                const double sigma = __shfl_sync(0xffffffffu, tot, j), alpha = __shfl_sync(0xffffffffu, piv, j);
                const double nn = alpha * alpha + sigma;
                double tau = 0.0, scale = 0.0, beta = alpha;
                if (sigma != 0.0 && nn >= SMALL_SQ) {
                    beta = -copysign(sqrt(nn), alpha);
                    tau = (beta - alpha) / beta;
                    scale = 1.0 / (alpha - beta);
                }
                const double tw = tau * (piv + scale * tot);          // tau v^T P(:, k), lane k
                double v[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int gr = r0 + row[q];
                    v[q] = gr > c ? x[q][j] * scale : (gr == c ? 1.0 : 0.0);
                }
#pragma unroll
                for (int k = j + 1; k < KB; k++) {
                    const double w = __shfl_sync(0xffffffffu, tw, k);
                    x[0][k] = fma(-v[0], w, x[0][k]);
                    x[1][k] = fma(-v[1], w, x[1][k]);
                }
                if (cta == 0 && tid <= c) s.R[tid][c] = tid < c ? x[0][j] : beta;
                x[0][j] = row[0] < nr ? v[0] : 0.0;
                x[1][j] = row[1] < nr ? v[1] : 0.0;
                if (tid == 0) s.tau[c] = tau;
            } else {                                          // no row left below the diagonal
                if (cta == 0 && tid < NB && tid < nr) s.R[tid][c] = x[0][j];
                x[0][j] = x[1][j] = 0.0;
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (row[q] < nr)
#pragma unroll
                for (int k = 0; k < KB; k++) ps[row[q] * PLD + cb + k] = x[q][k];
        __syncthreads();
        // ---- M = V8^T P, all columns: those of earlier blocks and this one hold V ----
        {
            const int r = lane >> 2, c4 = lane & 3;
            double acc[4][2];
#pragma unroll
            for (int nt = 0; nt < 4; nt++) acc[nt][0] = acc[nt][1] = 0.0;
            for (int ks = warp; ks < (nr + 3) / 4; ks += PC_W) {
                const double *pr = ps + (4 * ks + c4) * PLD;
                const double af = pr[cb + r];
#pragma unroll
                for (int nt = 0; nt < 4; nt++) dmma::mma884(acc[nt][0], acc[nt][1], af, pr[8 * nt + r]);
            }
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
                s.Mw[warp][r * NB + 8 * nt + 2 * c4] = acc[nt][0];
                s.Mw[warp][r * NB + 8 * nt + 2 * c4 + 1] = acc[nt][1];
            }
        }
        __syncthreads();
        if (tid < KB * NB) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < PC_W; q++) v += s.Mw[q][tid];
            *cl.map_shared_rank(&s.Rs[cta * vper + tid % vper], tid / vper) = v;
        }
        cl.sync();
        for (int q = tid; q < vper * G; q += PC_NT) {
            const int e = q % vper, d = q / vper;             // the sum of entry e to CTA d
            if (cta * vper + e < KB * NB) {
                double v = 0.0;
                for (int g = 0; g < G; g++) v += s.Rs[g * vper + e];
                *cl.map_shared_rank(&s.M[cta * vper + e], d) = v;
            }
        }
        cl.sync();
        // ---- T8, one column after another, and Z = T8^T M ----
        if (warp == 0) {
            const int i = lane & 7;
            double trow[KB];                                  // row i of T8
#pragma unroll
            for (int j = 0; j < KB; j++) {
                double t = 0.0;
#pragma unroll
                for (int l = 0; l < j; l++) t = fma(trow[l], s.M[l * NB + cb + j], t);   // T8(i, l) G(l, j), l >= i
                const double tj = s.tau[cb + j];
                trow[j] = i < j ? -tj * t : (i == j ? tj : 0.0);
            }
            if (lane < KB)
#pragma unroll
                for (int j = 0; j < KB; j++) s.T8[i][j] = trow[j];
        }
        if (cta == 0) {
            // kept for the whole T: V^T V against the earlier columns
            for (int q = tid; q < KB * NB; q += PC_NT) {
                const int i = q / NB, l = q % NB;
                if (l < cb) s.G[l][cb + i] = s.M[q];
            }
        }
        __syncthreads();
        if (cta == 0 && tid < KB * KB) s.T[cb + tid / KB][cb + tid % KB] = s.T8[tid / KB][tid % KB];
        if (cb + KB < NB) {
            if (tid < KB * NB) {
                const int i = tid % KB, k = tid / KB;
                double z = 0.0;
#pragma unroll
                for (int l = 0; l < KB; l++) z = fma(l <= i ? s.T8[l][i] : 0.0, s.M[l * NB + k], z);
                s.Z[k][i] = z;
            }
            __syncthreads();
            // ---- the columns to the right ----
            for (int k = cb + KB; k < NB; k++) {
                const double2 *z2 = (const double2 *)s.Z[k];
                const double2 za = z2[0], zb = z2[1], zc = z2[2], zd = z2[3];
#pragma unroll
                for (int q = 0; q < 2; q++)
                    if (row[q] < nr) {
                        double p0 = ps[row[q] * PLD + k], p1 = 0.0;
                        p0 = fma(-x[q][0], za.x, p0);
                        p1 = fma(-x[q][1], za.y, p1);
                        p0 = fma(-x[q][2], zb.x, p0);
                        p1 = fma(-x[q][3], zb.y, p1);
                        p0 = fma(-x[q][4], zc.x, p0);
                        p1 = fma(-x[q][5], zc.y, p1);
                        p0 = fma(-x[q][6], zd.x, p0);
                        p1 = fma(-x[q][7], zd.y, p1);
                        ps[row[q] * PLD + k] = p0 + p1;
                    }
            }
            __syncthreads();
        }
    }
    // V out; the triangle to the panel's place (what is below it there is never read again)
    for (int c = warp; c < NB; c += PC_W)
        for (int r = lane; r < nr; r += 32) {
            const double v = ps[r * PLD + c];
            a.V[(r0 + r) + (long)m * c] = v;
            a.V[(r0 + r) + (long)m * (2 * NB + c)] = v;
            if (a.Vs) a.Vs[(r0 + r) + (long)m * c] = v;
        }
    if (cta == 0) {
        for (int q = tid; q < NB * NB; q += PC_NT) {
            const int r = q % NB, c = q / NB;
            if (r < m && r <= c) a.P[r + a.ldp * (long)c] = s.R[r][c];
        }
        // T(0:cb, block) = -T(0:cb, 0:cb) (G(0:cb, block) T8), block after block
        double *tmp = s.Mw[0];
        for (int cb = KB; cb < NB; cb += KB) {
            __syncthreads();
            for (int q = tid; q < cb * KB; q += PC_NT) {
                const int r = q / KB, j = q % KB;
                double v = 0.0;
                for (int l = 0; l <= j; l++) v = fma(s.G[r][cb + l], s.T[cb + l][cb + j], v);
                tmp[q] = v;
            }
            __syncthreads();
            for (int q = tid; q < cb * KB; q += PC_NT) {
                const int r = q / KB, j = q % KB;
                double v = 0.0;
                for (int l = r; l < cb; l++) v = fma(s.T[r][l], tmp[l * KB + j], v);
                s.T[r][cb + j] = -v;
            }
        }
        __syncthreads();
        for (int q = tid; q < NB * NB; q += PC_NT) {
            a.T[q] = s.T[q % NB][q / NB];
            if (a.Ts) a.Ts[q] = s.T[q % NB][q / NB];
        }
    }
    cl.sync();                                              // no CTA leaves while another may still write to it
}

// W = X T (X the sum of S split-K partials, each m x NB), and V^T W over this CTA's 128 rows; the last CTA to
// finish adds those in order and forms M2 = 1/2 T^T V^T W at Mp + gridDim.x NB^2 for ypass2_kernel.  A warp
// has eight rows of W and one 8 x 8 block of V^T W, both on the tensor cores.
// Measured (average over the panels, n = 1713; both passes): 39 us with 128-thread CTAs and one thread per row or
// per entry, 23 us so, which includes adding the split-K partials (2.3 us as a launch of its own).
constexpr int YP_NT = 512, YLD = NB + 4;
struct YpassSmem {
    double X[128][YLD], V[128][YLD], T[NB][YLD], M[NB][YLD];
    unsigned ticket;
};

__global__ void __launch_bounds__(YP_NT) ypass1_kernel(int m, const double *__restrict__ X, int S,
                                                       const double *__restrict__ V, const double *__restrict__ T,
                                                       double *W, double *Mp, unsigned *tick)
{
    extern __shared__ __align__(16) unsigned char yp_sm[];
    YpassSmem &s = *(YpassSmem *)yp_sm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    const int r0 = blockIdx.x * 128;
    for (int q = tid; q < 128 * NB; q += YP_NT) {
        const int rr = q & 127, k = q >> 7, gr = r0 + rr;
        double x = 0.0, v = 0.0;
        if (gr < m) {
            for (int p = 0; p < S; p++) x += X[gr + (long)m * (k + NB * p)];
            v = V[gr + (long)m * k];
        }
        s.X[rr][k] = x;
        s.V[rr][k] = v;
    }
    for (int q = tid; q < NB * NB; q += YP_NT) s.T[q % NB][q / NB] = T[q];
    __syncthreads();
    {
        double acc[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; nt++) acc[nt][0] = acc[nt][1] = 0.0;
#pragma unroll
        for (int ks = 0; ks < NB / 4; ks++) {
            const double af = s.X[8 * warp + r][4 * ks + c];
#pragma unroll
            for (int nt = 0; nt < 4; nt++) dmma::mma884(acc[nt][0], acc[nt][1], af, s.T[4 * ks + c][8 * nt + r]);
        }
        __syncwarp();                                       // a warp's rows of X are its own: W takes their place
#pragma unroll
        for (int nt = 0; nt < 4; nt++)
#pragma unroll
            for (int j = 0; j < 2; j++) s.X[8 * warp + r][8 * nt + 2 * c + j] = acc[nt][j];
    }
    __syncthreads();
    for (int q = tid; q < 128 * NB; q += YP_NT) {
        const int rr = q & 127, k = q >> 7;
        if (r0 + rr < m) W[r0 + rr + (long)m * k] = s.X[rr][k];
    }
    {
        const int mt = warp & 3, nt = warp >> 2;
        double a0 = 0.0, a1 = 0.0;
#pragma unroll 8
        for (int ks = 0; ks < 32; ks++)
            dmma::mma884(a0, a1, s.V[4 * ks + c][8 * mt + r], s.X[4 * ks + c][8 * nt + r]);
        double *out = Mp + (long)blockIdx.x * NB * NB + (8 * mt + r) + NB * (8 * nt + 2 * c);
        out[0] = a0;
        out[NB] = a1;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s.ticket = atomicAdd(tick, 1u);
    __syncthreads();
    if (s.ticket != gridDim.x - 1) return;
    __threadfence();
    for (int q = tid; q < NB * NB; q += YP_NT) {
        double v = 0.0;
#pragma unroll 8
        for (int ch = 0; ch < (int)gridDim.x; ch++) v += __ldcg(Mp + (long)ch * NB * NB + q);
        s.M[q % NB][q / NB] = v;
    }
    __syncthreads();
    double *M2 = Mp + (long)gridDim.x * NB * NB;
    for (int q = tid; q < NB * NB; q += YP_NT) {
        const int i = q % NB, j = q / NB;
        double v = 0.0;
        for (int l = 0; l <= i; l++) v = fma(s.T[l][i], s.M[l][j], v);     // T upper
        M2[q] = 0.5 * v;                                             // column-major M2(i, j)
    }
    if (tid == 0) *tick = 0u;
}

// Y = W - V M2, in W's place
__global__ void __launch_bounds__(YP_NT) ypass2_kernel(int m, const double *__restrict__ V, const double *__restrict__ M2g,
                                                       double *Y)
{
    extern __shared__ __align__(16) unsigned char yp_sm[];
    YpassSmem &s = *(YpassSmem *)yp_sm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    const int r0 = blockIdx.x * 128;
    for (int q = tid; q < 128 * NB; q += YP_NT) {
        const int rr = q & 127, k = q >> 7, gr = r0 + rr;
        s.X[rr][k] = gr < m ? Y[gr + (long)m * k] : 0.0;
        s.V[rr][k] = gr < m ? -V[gr + (long)m * k] : 0.0;
    }
    for (int q = tid; q < NB * NB; q += YP_NT) s.M[q % NB][q / NB] = M2g[q];
    __syncthreads();
    double acc[4][2];
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
        for (int j = 0; j < 2; j++) acc[nt][j] = s.X[8 * warp + r][8 * nt + 2 * c + j];
#pragma unroll
    for (int ks = 0; ks < NB / 4; ks++) {
        const double af = s.V[8 * warp + r][4 * ks + c];
#pragma unroll
        for (int nt = 0; nt < 4; nt++) dmma::mma884(acc[nt][0], acc[nt][1], af, s.M[4 * ks + c][8 * nt + r]);
    }
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
        for (int j = 0; j < 2; j++) s.X[8 * warp + r][8 * nt + 2 * c + j] = acc[nt][j];
    __syncthreads();
    for (int q = tid; q < 128 * NB; q += YP_NT) {
        const int rr = q & 127, k = q >> 7;
        if (r0 + rr < m) Y[r0 + rr + (long)m * k] = s.X[rr][k];
    }
}

}  // namespace

constexpr int PANEL_ROWS = 160;

int sy2sb_panels(int n)
{ return n > NB ? (n - 1) / NB : 0; }   // panels j = 0, NB, ... with j + NB < n

// Saved panels for the back-transformation: V of panel p (m_p x NB, ld m_p) at Vsave + voff(p),
// T of panel p at Tsave + p NB^2.
size_t sy2sb_vsave_doubles(int n)
{
    size_t t = 0;
    for (int j = 0; j + NB < n; j += NB) t += (size_t)(n - j - NB) * NB;
    return t + 64;
}

// Can the device hold the cluster form of the panel factorisation (16 CTAs with their shared memory)?  Asked
// once per device: the two calls wait until other threads' copies to pageable memory are done.
static cudaError_t panel_cluster_fits(bool *ok)
{
    static std::mutex mu;
    static std::map<int, bool> fits;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    const auto known = fits.find(dev);
    if (known != fits.end()) {
        *ok = known->second;
        return cudaSuccess;
    }
    const size_t smem_c = panel_smem(PC_ROWS);
    int nclusters = 0;
    if (cudaFuncSetAttribute(panel_qr_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess &&
        smem_attr(panel_qr_cluster_kernel, smem_c) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(PC_MAXG);
        cfg.blockDim = dim3(PC_NT);
        cfg.dynamicSmemBytes = smem_c;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = PC_MAXG;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&nclusters, panel_qr_cluster_kernel, &cfg) != cudaSuccess) nclusters = 0;
    }
    cudaGetLastError();
    *ok = fits[dev] = nclusters >= 1;
    return cudaSuccess;
}

int sy2sb(cudaStream_t st, int n, double *A, long lda, double *Vsave, double *Tsave, const Sy2sbWork &w)
{
    cudaError_t e;
    const int smem = PQ_ROWS * (NB + 1) * (int)sizeof(double);
    if ((e = smem_attr(panel_qr_kernel, smem)) != cudaSuccess ||
        (e = smem_attr(ypass1_kernel, sizeof(YpassSmem))) != cudaSuccess ||
        (e = smem_attr(ypass2_kernel, sizeof(YpassSmem))) != cudaSuccess)
        return cuda_fail(e, "sy2sb smem");
    bool use_cluster = false;
    if ((e = panel_cluster_fits(&use_cluster)) != cudaSuccess) return cuda_fail(e, "sy2sb device");
    // factorise panel p (columns j = p NB ..) on stream sq; its V goes to the [V | Y | V] buffer of p's parity
    auto factor_panel = [&](int p, size_t voff, cudaStream_t sq) -> int {
        const int j = p * NB, m = n - j - NB;
        int G = (m + PQ_ROWS - 1) / PQ_ROWS;
        G = std::max(1, std::min(G, std::max(1, m / NB)));      // CTA 0 holds the NB pivot rows
        const int rpc = (m + G - 1) / G;
        if (rpc > PQ_ROWS) { set_error("sy2sb: panel of %d rows does not fit", m); return BSRG_ERR_ARG; }
        PanelArgs a;
        a.P = A + (j + NB) + lda * (long)j;
        a.ldp = lda;
        a.m = m;
        a.rpc = rpc;
        a.V = (p & 1) && w.aux ? w.VYV2 : w.VYV;
        a.Vs = Vsave ? Vsave + voff : nullptr;
        a.T = w.T;
        a.Ts = Tsave ? Tsave + (size_t)p * NB * NB : nullptr;
        a.part = w.part;
        a.gram = w.gram;
        a.bar = w.bar;
        a.err = w.err;
        // CTAs of the cluster: PANEL_ROWS rows each while there are enough for all sixteen
        const int Gc = std::max((m + PC_ROWS - 1) / PC_ROWS, std::min(PC_MAXG, (m + PANEL_ROWS - 1) / PANEL_ROWS));
        if (use_cluster && Gc <= PC_MAXG) {
            a.rpc = std::max(NB, (m + Gc - 1) / Gc);       // CTA 0 has every pivot row
            const size_t smem_c = panel_smem(a.rpc);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)Gc);
            cfg.blockDim = dim3(PC_NT);
            cfg.dynamicSmemBytes = smem_c;
            cfg.stream = sq;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)Gc;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if ((e = cudaLaunchKernelEx(&cfg, panel_qr_cluster_kernel, a)) != cudaSuccess)
                return cuda_fail(e, "sy2sb panel (cluster)");
        } else {
            void *args[] = {&a};
            if ((e = cudaLaunchCooperativeKernel((const void *)panel_qr_kernel, G, PQ_NT, args, smem, sq)) !=
                cudaSuccess)
                return cuda_fail(e, "sy2sb panel");
        }
        return BSRG_OK;
    };
    size_t voff = 0;
    int rc = n > NB ? factor_panel(0, 0, st) : BSRG_OK;
    if (rc != BSRG_OK) return rc;
    bool qr_on_aux = false;                       // the current panel was factorised on the aux stream
    int p = 0;
    for (int j = 0; j + NB < n; j += NB, p++) {
        const int m = n - j - NB;
        double *VYV = (p & 1) && w.aux ? w.VYV2 : w.VYV;
        double *A22 = A + (j + NB) + lda * (long)(j + NB);
        double *Vp = VYV, *Yp = VYV + (long)m * NB;
        const size_t voff_next = voff + (size_t)m * NB;
        const bool has_next = j + 2 * NB < n;
        if (qr_on_aux && (e = cudaStreamWaitEvent(st, w.ev_c2, 0)) != cudaSuccess)
            return cuda_fail(e, "sy2sb look-ahead wait");
        // X = A22 V with A22 read from its lower triangle (only the lower triangle is updated)
        DgemmBatch gx{};
        gx.m = m; gx.n = NB; gx.k = m;
        gx.A = A22; gx.lda = lda; gx.B = Vp; gx.ldb = m; gx.C = w.X; gx.ldc = m;
        gx.alpha = 1.0; gx.beta = 0.0; gx.syma = 1;
        int S = 1;
        rc = dgemm_partial(gx, st, w.X, w.gemm_ws, w.gemm_ws_doubles, &S);
        if (rc != BSRG_OK) return rc;
        const int nch = (m + 127) / 128;
        ypass1_kernel<<<nch, YP_NT, sizeof(YpassSmem), st>>>(m, S > 1 ? w.gemm_ws : w.X, S, Vp, w.T, Yp, w.Mp, w.ticket);
        ypass2_kernel<<<nch, YP_NT, sizeof(YpassSmem), st>>>(m, Vp, w.Mp + (size_t)nch * NB * NB, Yp);
        // A22 -= [V Y] [Y V]^T, the tiles that reach the lower triangle
        if (!w.aux || m <= NB) {
            DgemmBatch gu{};
            gu.m = m; gu.n = m; gu.k = 2 * NB;
            gu.A = VYV; gu.lda = m; gu.B = Yp; gu.ldb = m; gu.C = A22; gu.ldc = lda;
            gu.alpha = -1.0; gu.beta = 1.0; gu.lowc = 1;
            rc = dgemm_ws(false, true, gu, 1, st, nullptr, 0);
            if (rc == BSRG_OK && has_next) rc = factor_panel(p + 1, voff_next, st);
            if (rc != BSRG_OK) return rc;
            qr_on_aux = false;
        } else {
            // look-ahead: the next panel's NB columns first; the next panel is then factorised on the
            // high-priority aux stream while the rest of the trailing matrix is updated here, so the
            // panel's few CTAs are placed before the update's fill the machine
            DgemmBatch g1{};
            g1.m = m; g1.n = NB; g1.k = 2 * NB;
            g1.A = VYV; g1.lda = m; g1.B = Yp; g1.ldb = m; g1.C = A22; g1.ldc = lda;
            g1.alpha = -1.0; g1.beta = 1.0;
            rc = dgemm_ws(false, true, g1, 1, st, nullptr, 0);
            if (rc != BSRG_OK) return rc;
            qr_on_aux = false;
            if (has_next) {
                if ((e = cudaEventRecord(w.ev_y, st)) != cudaSuccess ||
                    (e = cudaStreamWaitEvent(w.aux, w.ev_y, 0)) != cudaSuccess)
                    return cuda_fail(e, "sy2sb look-ahead");
                rc = factor_panel(p + 1, voff_next, w.aux);
                if (rc != BSRG_OK) return rc;
                if ((e = cudaEventRecord(w.ev_c2, w.aux)) != cudaSuccess) return cuda_fail(e, "sy2sb look-ahead");
                qr_on_aux = true;
            }
            const int m2 = m - NB;
            DgemmBatch g2{};
            g2.m = m2; g2.n = m2; g2.k = 2 * NB;
            g2.A = VYV + NB; g2.lda = m; g2.B = Yp + NB; g2.ldb = m; g2.C = A22 + NB + lda * (long)NB; g2.ldc = lda;
            g2.alpha = -1.0; g2.beta = 1.0; g2.lowc = 1;
            rc = dgemm_ws(false, true, g2, 1, st, nullptr, 0);
            if (rc != BSRG_OK) return rc;
        }
        voff = voff_next;
    }
    if (qr_on_aux && (e = cudaStreamWaitEvent(st, w.ev_c2, 0)) != cudaSuccess)
        return cuda_fail(e, "sy2sb look-ahead join");
    return cuda_fail(cudaGetLastError(), "sy2sb");
}

}  // namespace bsrg
