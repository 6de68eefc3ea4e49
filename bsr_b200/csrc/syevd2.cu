// Dense symmetric eigensolver for sm_100a: two-stage reduction to tridiagonal
// form, divide and conquer, back-transformation.
//
// The reference's DSYEV (LAP_DSYEV, src/libs/ZCOM/LAPACK_calls.f90:54-76,
// called from diag_hd.f90:312) reduces A = Q T Q^T one column at a time
// (DSYTRD: every column reads the whole trailing matrix, a latency-bound
// matrix-vector product per column on a GPU) and diagonalises T.  Here the
// reduction goes through a band matrix, as in LAPACK's two-stage DSYTRD_2STAGE:
//
//   1. dense -> band (bandwidth NB): per panel of NB columns a Householder QR
//      (one cooperative kernel, the panel in shared memory of a few CTAs, one
//      grid barrier per column), then the two-sided update of the trailing
//      matrix A22 <- (I - V T V^T)^T A22 (I - V T V^T) as FP64 tensor-core
//      GEMMs: X = A22 V, Y = X T - 1/2 V (T^T V^T X T), A22 -= V Y^T + Y V^T
//      (one GEMM of inner size 2 NB over the [V | Y | V] buffer);
//   2. band -> tridiagonal: bulge chasing (sweeps of Householder reflectors of
//      length NB, each annihilating one column and chasing the bulge down the
//      band), one persistent cooperative kernel (bulge.cu);
//   3. tridiagonal eigenpairs by divide and conquer (tridiag_dc.cu);
//   4. back-transformation: the stage-2 reflectors (in blocks of NB sweeps) and
//      the stage-1 panels (compact WY, GEMMs), applied to the eigenvectors.
#include <algorithm>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "ctx.h"
#include "dgemm.h"
#include "syevd2.h"

namespace bsrg {
namespace {

// ---------------------------------------------------------------------------
// back-transformation of the stage-1 panels, Q1_GROUP panels at a time
// ---------------------------------------------------------------------------
constexpr int Q1_GROUP = 8;
constexpr int Q1W = Q1_GROUP * NB;     // columns of a merged block reflector
constexpr int Q1H = 4 * NB;            // the unit of q1_tmerge_kernel: four panels

struct Q1Panels {
    const double *V[Q1_GROUP];   // V of each panel (m_q x NB, ld m_q), null past the last panel
    int m[Q1_GROUP];
};

// Vg (m0 x Q1W, ld m0): panel q's V shifted down by q NB rows, zeros above
__global__ void q1_gather_kernel(int m0, Q1Panels P, double *Vg)
{
    const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (idx >= (long)m0 * Q1W) return;
    const int r = (int)(idx % m0), c = (int)(idx / m0), q = c / NB, cc = c % NB;
    double v = 0.0;
    if (P.V[q] && r >= q * NB) v = P.V[q][(r - q * NB) + (long)P.m[q] * cc];
    Vg[idx] = v;
}

// The same T from the panels' own T factors (T1) and the Gram blocks, merging pairs as
// Q_a Q_b = I - [V_a V_b] [[T_a, -T_a G_ab T_b], [0, T_b]] [V_a V_b]^T (the block form of the
// recurrence above): two 32 x 32 merges, then one of the 64-column halves; small products in
// shared memory instead of 128 dependent column steps.
constexpr int Q1M_SMEM = (Q1H * (Q1H + 1) + 64 * 65) * (int)sizeof(double);

// T of the merged reflector of four consecutive panels (q0 .. q0+3 of the group): G and the
// output block T are Q1H x Q1H with leading dimension Q1W
__global__ void __launch_bounds__(Q1H) q1_tmerge_kernel(const double *__restrict__ G, Q1Panels P, int q0,
                                                        const double *__restrict__ T1, int p0, double *Tg)
{
    extern __shared__ __align__(16) double q1m_sm[];
    double (*Ts)[Q1H + 1] = (double (*)[Q1H + 1])q1m_sm;               // Ts[r][c]
    double (*W)[65] = (double (*)[65])(q1m_sm + Q1H * (Q1H + 1));
    const int t = threadIdx.x;
    for (int c = 0; c < Q1H; c++) Ts[t][c] = 0.0;
    __syncthreads();
    for (int q = 0; q < 4; q++) {
        if (!P.V[q0 + q]) continue;
        const double *Tp = T1 + (size_t)(p0 + q0 + q) * NB * NB;        // column-major NB x NB
        for (int e = t; e < NB * NB; e += Q1H) Ts[q * NB + e % NB][q * NB + e / NB] = Tp[e];
    }
    __syncthreads();
    // merges: width w = NB (pairs 0|1, 2|3), then 2 NB (halves)
    for (int w = NB; w < Q1H; w *= 2) {
        for (int a0 = 0; a0 < Q1H; a0 += 2 * w) {
            const int b0 = a0 + w;
            for (int e = t; e < w * w; e += Q1H) {
                const int r = e % w, c = e / w;
                double sacc = 0.0;
                for (int k = 0; k <= c; k++) sacc += __ldg(G + (a0 + r) + (long)Q1W * (b0 + k)) * Ts[b0 + k][b0 + c];
                W[r][c] = sacc;
            }
            __syncthreads();
            for (int e = t; e < w * w; e += Q1H) {
                const int r = e % w, c = e / w;
                double sacc = 0.0;
                for (int k = r; k < w; k++) sacc += Ts[a0 + r][a0 + k] * W[k][c];
                Ts[a0 + r][b0 + c] = -sacc;
            }
            __syncthreads();
        }
    }
    for (int c = 0; c < Q1H; c++) Tg[t + (long)Q1W * c] = Ts[t][c];
}

}  // namespace

}  // namespace bsrg

namespace bsrg {

int symmetrize_lower(int n, const double *A, long lda, double *F, long ldf, cudaStream_t s);   // refine.cu

// Workspace of dense_syevd in doubles (everything but the output Z)
// The workspace carve-up of syevd2_impl, as offsets (doubles, 32-aligned); the size
// function and the solver use this one layout.
struct Syevd2Layout {
    size_t Wk, AB, V1, T1, V2, tau2, Tq, dv, ev, VYV, X, T, Mp, part, gram, flags, W1, W2, Vg, Gq, Tg,
        gemm_ws, dcw, total;
};

static Syevd2Layout syevd2_layout(int n)
{
    Syevd2Layout L{};
    const size_t nn = (size_t)n * n;
    const size_t S = (size_t)sweep_steps(n, 0) + 1;
    size_t off = 0;
    auto take = [&](size_t cnt) { off = (off + 31) & ~(size_t)31; size_t p = off; off += cnt; return p; };
    // the fragments of Q2 take the place of the reduction's working copy and of the divide and conquer's
    // workspace, which are through by then
    L.Wk = L.Tq = take(nn);
    L.dcw = take(dc_workspace_bytes(n) / 8 + 8);
    off = std::max(off, L.Tq + q2_fragment_doubles(n));
    L.AB = take((size_t)2 * LDAB * n);
    L.V1 = take(sy2sb_vsave_doubles(n));
    L.T1 = take((size_t)(sy2sb_panels(n) + 1) * NB * NB);
    L.V2 = take((size_t)n * S * NB);
    L.tau2 = take((size_t)n * S);
    L.dv = take(n);
    L.ev = take(n + 1);
    L.VYV = take((size_t)n * 6 * NB);               // two [V | Y | V] buffers
    L.X = take((size_t)n * NB);
    L.T = take(NB * NB);
    L.Mp = take(((size_t)n / 128 + 2) * NB * NB);
    L.part = take((size_t)(n / NB + 8) * 4 * NB);
    L.gram = take((size_t)(n / NB + 8) * NB * NB);
    L.flags = take(8);
    L.W1 = take((size_t)Q1W * n);
    L.W2 = take(std::max((size_t)Q1W * n, (size_t)(Q1W / 2) * (Q1W / 2)));   // also the T merges' temporary
    L.Vg = take((size_t)Q1W * n);
    L.Gq = take((size_t)Q1W * Q1W);
    L.Tg = take((size_t)Q1W * Q1W);
    L.gemm_ws = take(8 * (size_t)Q1W * n);
    L.total = off + 64;
    return L;
}

size_t syevd2_workspace_doubles(int n) { return syevd2_layout(n).total; }

// Eigenvalues (ascending, w) and eigenvectors (Z, ldz) of the symmetric A (lower
// triangle referenced).  Z may be A itself.  ws: syevd2_workspace_doubles(n).
// tri_d / tri_e non-null: stop after the reduction and copy the tridiagonal (d: n, e: n-1) there
static int syevd2_impl(bsrg_ctx *c, int n, const double *A, long lda, double *w, double *Z, long ldz, double *ws,
                       size_t ws_doubles, void *pinned, size_t pinned_bytes, int *launches, double *tri_d,
                       double *tri_e)
{
    int nl = 0;
    if (n < 1) return BSRG_OK;
    cudaStream_t st = c->stream;
    cudaError_t e;
    if (ws_doubles < syevd2_workspace_doubles(n)) { set_error("dsyevd: workspace too small"); return BSRG_ERR_NOMEM; }
    if (n > 10240) { set_error("dsyevd: n=%d above 10240", n); return BSRG_ERR_ARG; }
    const int S = sweep_steps(n, 0) + 1;
    const Syevd2Layout L = syevd2_layout(n);
    double *Wk = ws + L.Wk, *AB = ws + L.AB, *V1 = ws + L.V1, *T1 = ws + L.T1;
    double *V2 = ws + L.V2, *tau2 = ws + L.tau2, *Tq = ws + L.Tq;
    double *dv = ws + L.dv, *ev = ws + L.ev;
    Sy2sbWork sw;
    sw.VYV = ws + L.VYV;
    sw.VYV2 = sw.VYV + (size_t)n * 3 * NB;
    sw.aux = getenv("BSRG_NO_LOOKAHEAD") ? nullptr : c->aux_stream;
    sw.ev_y = c->aux_ev[0];
    sw.ev_c2 = c->aux_ev[1];
    sw.X = ws + L.X;
    sw.T = ws + L.T;
    sw.Mp = ws + L.Mp;
    sw.part = ws + L.part;
    sw.gram = ws + L.gram;
    int *flags = (int *)(ws + L.flags);            // bar[2], err, err2
    sw.bar = (unsigned *)flags;
    sw.err = flags + 2;
    sw.ticket = (unsigned *)(flags + 4);
    double *W1 = ws + L.W1, *W2 = ws + L.W2;
    double *Vg = ws + L.Vg, *Gq = ws + L.Gq, *Tg = ws + L.Tg;
    sw.gemm_ws_doubles = 8 * (size_t)Q1W * n;
    sw.gemm_ws = ws + L.gemm_ws;
    double *dcw = ws + L.dcw;
    if ((e = cudaMemsetAsync(flags, 0, 8 * sizeof(int), st)) != cudaSuccess)
        return cuda_fail(e, "dsyevd init");
    const int np = sy2sb_panels(n);
    double fl_band = 0.0, fl_chase = 0.0, fl_q2 = 0.0, fl_q1 = 0.0, fl_dc = 0.0;
    for (int j = 0; j + NB < n; j += NB) {
        const double m = n - j - NB;
        // X (2 m^2 NB), the lower-triangle tiles of the rank-2NB update (~2 m^2 NB), QR and Y passes
        fl_band += 4.0 * m * m * NB + 6.0 * m * NB * NB + 4.0 * m * NB * NB;
        fl_q1 += 4.0 * (m + 1.5 * NB) * n * NB + 2.0 * Q1W * NB * n + 2.0 * Q1W * NB * m;  // per panel share of a group
    }
    // 1. full symmetric working copy, dense -> band
    stage_begin(c, 9);
    int rc = symmetrize_lower(n, A, lda, Wk, n, st);
    if (rc == BSRG_OK) rc = sy2sb(st, n, Wk, n, V1, T1, sw);
    if (rc != BSRG_OK) return rc;
    rc = band_extract(n, Wk, n, AB, st);
    if (rc != BSRG_OK) return rc;
    stage_end(c, 9, 2 + np * 6);
    c->stage_flops[9] += fl_band;
    stage_begin(c, 10);
    // 2. band -> tridiagonal
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
    rc = bulge_chase(n, AB, dv, ev, V2, tau2, S, sw.err, nsm, st);
    if (rc != BSRG_OK) return rc;
    fl_chase = 4.0 * NB * (3.0 * NB) * (double)n * n / (2.0 * NB);      // whole windows, n^2 / (2 NB) steps
    stage_end(c, 10, 2);
    c->stage_flops[10] += fl_chase;
    if (tri_d) {
        int hf = 0;
        if ((e = cudaMemcpyAsync(tri_d, dv, sizeof(double) * n, cudaMemcpyDeviceToDevice, st)) != cudaSuccess ||
            (n > 1 && (e = cudaMemcpyAsync(tri_e, ev, sizeof(double) * (n - 1), cudaMemcpyDeviceToDevice, st)) !=
                          cudaSuccess) ||
            (e = cudaMemcpyAsync(&hf, flags + 2, sizeof(int), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess)
            return cuda_fail(e, "dsytrd_2stage");
        if (hf != 0) {
            set_error("dsytrd_2stage: a device-side wait timed out (%s)", hf == 2 ? "bulge chasing" : "panel barrier");
            return BSRG_ERR_CUDA;
        }
        return BSRG_OK;
    }
    // 3. tridiagonal eigenpairs into Z
    stage_begin(c, 11);
    int ndc = 0, nmerge = 0;
    rc = tridiag_dc(st, n, dv, ev, w, Z, ldz, dcw, dc_workspace_bytes(n), pinned, pinned_bytes, &nmerge, &ndc);
    if (rc != BSRG_OK) return rc;
    stage_end(c, 11, ndc);
    // 4. back-transformation: Q2 then Q1
    stage_begin(c, 12);
    rc = q2_apply(n, V2, tau2, S, Tq, Z, ldz, sw.err, nsm, st);
    if (rc != BSRG_OK) return rc;
    fl_q2 = q2_flops(n);
    stage_end(c, 12, n > 2 ? 2 : 0);
    c->stage_flops[12] += fl_q2;
    stage_begin(c, 13);
    {
        std::vector<size_t> voff;
        size_t vo = 0;
        for (int j = 0; j + NB < n; j += NB) { voff.push_back(vo); vo += (size_t)(n - j - NB) * NB; }
        const int ngrp = (np + Q1_GROUP - 1) / Q1_GROUP;
        for (int gq = ngrp - 1; gq >= 0; gq--) {
            const int p0 = gq * Q1_GROUP, r0 = p0 * NB + NB, m0 = n - r0;
            Q1Panels P{};
            for (int q = 0; q < Q1_GROUP; q++) {
                const int p = p0 + q;
                P.V[q] = p < np ? V1 + voff[p] : nullptr;
                P.m[q] = p < np ? n - p * NB - NB : 0;
            }
            q1_gather_kernel<<<(unsigned)(((long)m0 * Q1W + 255) / 256), 256, 0, st>>>(m0, P, Vg);
            rc = dgemm(true, false, Q1W, Q1W, m0, 1.0, Vg, m0, Vg, m0, 0.0, Gq, Q1W, st, sw.gemm_ws,
                       sw.gemm_ws_doubles);
            if (rc != BSRG_OK) return rc;
            // T of the merged 256-column reflector: each 128-column half by pairwise merges of its
            // panels' T (q1_tmerge_kernel), then the off-diagonal block -T_a G_ab T_b by two GEMMs
            if ((e = smem_attr(q1_tmerge_kernel, Q1M_SMEM)) != cudaSuccess)
                return cuda_fail(e, "dsyevd Q1 smem");
            if ((e = cudaMemsetAsync(Tg, 0, sizeof(double) * Q1W * Q1W, st)) != cudaSuccess)
                return cuda_fail(e, "dsyevd Q1 T");
            for (int hq = 0; hq < Q1_GROUP / 4; hq++) {
                const long o = (long)hq * Q1H * (Q1W + 1);
                q1_tmerge_kernel<<<1, Q1H, Q1M_SMEM, st>>>(Gq + o, P, 4 * hq, T1, p0, Tg + o);
            }
            for (int w = Q1H; w < Q1W; w *= 2)
                for (int a0 = 0; a0 < Q1W; a0 += 2 * w) {
                    const int b0 = a0 + w;
                    // Wq = G(a, b) T_b (w x w), then T(a, b) = -T_a Wq
                    rc = dgemm(false, false, w, w, w, 1.0, Gq + a0 + (long)Q1W * b0, Q1W, Tg + b0 + (long)Q1W * b0,
                               Q1W, 0.0, W2, w, st);
                    if (rc == BSRG_OK)
                        rc = dgemm(false, false, w, w, w, -1.0, Tg + a0 + (long)Q1W * a0, Q1W, W2, w, 0.0,
                                   Tg + a0 + (long)Q1W * b0, Q1W, st);
                    if (rc != BSRG_OK) return rc;
                }
            double *Zs = Z + r0;
            rc = dgemm(true, false, Q1W, n, m0, 1.0, Vg, m0, Zs, ldz, 0.0, W1, Q1W, st, sw.gemm_ws,
                       sw.gemm_ws_doubles);
            if (rc == BSRG_OK) rc = dgemm(false, false, Q1W, n, Q1W, 1.0, Tg, Q1W, W1, Q1W, 0.0, W2, Q1W, st);
            if (rc == BSRG_OK) rc = dgemm(false, false, m0, n, Q1W, -1.0, Vg, m0, W2, Q1W, 1.0, Zs, ldz, st);
            if (rc != BSRG_OK) return rc;
        }
    }
    stage_end(c, 13, 10 * ((np + Q1_GROUP - 1) / Q1_GROUP));
    c->stage_flops[13] += fl_q1;
    // device-side waits report through the flags
    int hflag[2] = {0, 0};
    if ((e = cudaMemcpyAsync(hflag, flags + 2, sizeof(int) * 2, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(e, "dsyevd");
    fl_dc = dc_gemm_flops(n, pinned, nmerge);
    c->stage_flops[11] += fl_dc;
    c->stage_flops[6] += fl_band + fl_chase + fl_dc + fl_q2 + fl_q1;
    if (hflag[0] != 0) {
        set_error("dsyevd: a device-side wait timed out (%s)",
                  hflag[0] == 2 ? "bulge chasing" : hflag[0] == 3 ? "back-transformation wavefront" : "panel barrier");
        return BSRG_ERR_CUDA;
    }
    // kernels of this library per call
    nl = 2 + np * 6 + 2 + ndc + (n > 2 ? 2 : 0) + 3 * np;
    if (launches) *launches = nl;
    return BSRG_OK;
}

int dense_syevd(bsrg_ctx *c, int n, const double *A, long lda, double *w, double *Z, long ldz, double *ws,
                size_t ws_doubles, void *pinned, size_t pinned_bytes, int *launches)
{
    return syevd2_impl(c, n, A, lda, w, Z, ldz, ws, ws_doubles, pinned, pinned_bytes, launches, nullptr, nullptr);
}

}  // namespace bsrg

using namespace bsrg;

extern "C" int bsrg_dsytrd_2stage(bsrg_ctx *c, int n, const double *A, int lda, double *d, double *e)
{
    if (!c || (n > 0 && (!A || !d || (n > 1 && !e)))) { set_error("dsytrd_2stage: null argument"); return BSRG_ERR_ARG; }
    if (n < 0 || lda < (n > 0 ? n : 1)) { set_error("dsytrd_2stage: n=%d lda=%d", n, lda); return BSRG_ERR_ARG; }
    if (n == 0) return BSRG_OK;
    cudaSetDevice(c->device);
    int rc = ctx_reserve(c, syevd2_workspace_doubles(n) * sizeof(double) + 1024);
    if (rc != BSRG_OK) return rc;
    rc = syevd2_impl(c, n, A, lda, nullptr, nullptr, n, (double *)c->ws, c->ws_bytes / sizeof(double), nullptr, 0,
                     nullptr, d, e);
    cudaEventRecord(c->ev_stage, c->stream);
    return rc;
}

extern "C" int bsrg_dsyevd(bsrg_ctx *c, int n, const double *A, int lda, double *w, double *Z, int ldz)
{
    if (!c || (n > 0 && (!A || !w || !Z))) { set_error("dsyevd: null argument"); return BSRG_ERR_ARG; }
    if (n < 0 || lda < (n > 0 ? n : 1) || ldz < (n > 0 ? n : 1)) {
        set_error("dsyevd: n=%d lda=%d ldz=%d", n, lda, ldz);
        return BSRG_ERR_ARG;
    }
    if (n == 0) return BSRG_OK;
    cudaSetDevice(c->device);
    int rc = ctx_reserve(c, syevd2_workspace_doubles(n) * sizeof(double) + 1024);
    if (rc == BSRG_OK) rc = ctx_reserve_pinned(c, dc_pinned_bytes(n));
    if (rc != BSRG_OK) return rc;
    cudaError_t e = cudaEventSynchronize(c->ev_stage);     // the staging's last copies are through
    if (e != cudaSuccess) return cuda_fail(e, "dsyevd staging");
    rc = dense_syevd(c, n, A, lda, w, Z, ldz, (double *)c->ws, c->ws_bytes / sizeof(double), c->pinned,
                     c->pinned_bytes, nullptr);
    cudaEventRecord(c->ev_stage, c->stream);
    return rc;
}
