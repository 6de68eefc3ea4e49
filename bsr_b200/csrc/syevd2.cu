// Dense symmetric eigensolver for sm_100a: two-stage reduction to tridiagonal
// form, divide and conquer, back-transformation.
//
// The reference's DSYEV (LAP_DSYEV, src/libs/ZCOM/LAPACK_calls.f90:54-76,
// called from diag_hd.f90:312) reduces A = Q T Q^T one column at a time
// (DSYTRD: every column reads the whole trailing matrix, a latency-bound
// matrix-vector product per column on a GPU) and diagonalises T.  Here the
// reduction goes through a band matrix, as in LAPACK's two-stage DSYTRD_2STAGE:
//
//   1. dense -> band of width NB (band_reduce.cu): per panel of NB columns a Householder QR, on one cluster of
//      16 CTAs with the panel in shared memory and one cluster barrier per column (a cooperative kernel with a grid
//      barrier where no such cluster can be placed), then the two-sided update of the trailing matrix as FP64
//      tensor-core GEMMs; a panel is factorised on a second stream beside the update it does not need;
//   2. band -> tridiagonal (bulge.cu): bulge chasing (sweeps of Householder reflectors of length NB, each annihilating
//      one column and chasing the bulge down the band), a CTA per sweep, the sweeps taken by ticket from an ordinary
//      launch;
//   3. tridiagonal eigenpairs by divide and conquer, or the eigenvalues alone by bisection (tridiag_dc.cu);
//   4. back-transformation: the stage-2 reflectors in blocks of NB sweeps (q2_apply.cu), then the stage-1 panels
//      merged eight at a time (compact WY, GEMMs), their T factors made on the second stream beside step 2.
#include <algorithm>
#include <cmath>
#include <vector>

#include "aux_join.h"
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

// T of the merged reflector of four consecutive panels (q0 .. q0+3 of the group) from the panels' own T factors
// (T1) and the Gram blocks G = V^T V, merging pairs as
// Q_a Q_b = I - [V_a V_b] [[T_a, -T_a G_ab T_b], [0, T_b]] [V_a V_b]^T:
// two 32 x 32 merges, then one of the 64-column halves; small products in shared memory instead of the 128 dependent
// column steps of T(0:c, c) = -tau_c T(0:c, 0:c) G(0:c, c).  G and the output block T are Q1H x Q1H with leading
// dimension Q1W.
constexpr int Q1M_SMEM = (Q1H * (Q1H + 1) + 64 * 65) * (int)sizeof(double);

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

// ---------------------------------------------------------------------------
// the working copy, its scale, and what a non-finite entry gives
// ---------------------------------------------------------------------------
// A matrix whose largest entry lies outside 2^-150 .. 2^150 is solved scaled by a power of two (exact both ways),
// one with a NaN or an infinity as zeros with NaN results, so that no later kernel meets one.  Inside that range no
// sum of squares overflows, nor does 2 / |u|^2 times an entry (bulge.cu) for any column whose sum of squares is
// SMALL_SQ = 2^-700 at least.  Columns below that are dropped: their entries, under 2^-350, are less than 2^-199
// of the largest, while a reflector made from squares near the smallest number would not be orthogonal.
// One more pass over the triangle: 9 us at n = 2176, 53 at 7810.
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;

// max |A(i,j)|, i >= j, as bits (which order as the values do; a NaN is above infinity)
__global__ void __launch_bounds__(256) amax_kernel(int n, const double *__restrict__ A, long lda,
                                                   unsigned long long *amax)
{
    unsigned long long m = 0;
    for (int j = blockIdx.x; j < n; j += gridDim.x) {
        const double *col = A + (long)lda * j;
        for (int i = j + threadIdx.x; i < n; i += 256)
            m = max(m, (unsigned long long)__double_as_longlong(col[i]) & 0x7fffffffffffffffull);
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(amax, m);
}

// the exponent of the power of two that the matrix is divided by
__device__ __forceinline__ int scale_exp(unsigned long long bits)
{
    if (bits == 0 || bits >= kInfBits) return 0;
    int q;
    frexp(__longlong_as_double((long long)bits), &q);
    return q < -150 || q > 150 ? q : 0;
}

// F = the symmetric matrix of A's lower triangle, scaled; 32 x 32 tiles
__global__ void __launch_bounds__(256) work_copy_kernel(int n, const double *__restrict__ A, long lda,
                                                        double *__restrict__ F, const unsigned long long *amax)
{
    __shared__ double tile[32][33];
    const int bi = blockIdx.x, bj = blockIdx.y, tx = threadIdx.x, ty = threadIdx.y;
    if (bi < bj) return;
    const bool bad = *amax >= kInfBits;
    const int q2 = scale_exp(*amax);
    for (int q = ty; q < 32; q += 8) {
        const int i = bi * 32 + tx, j = bj * 32 + q;
        double v = 0.0;
        if (i < n && j < n && !bad) v = i >= j ? A[i + (long)lda * j] : A[j + (long)lda * i];
        if (q2) v = scalbn(v, -q2);
        tile[q][tx] = v;
        if (i < n && j < n) F[i + (long)n * j] = v;
    }
    __syncthreads();
    if (bi == bj) return;
    for (int q = ty; q < 32; q += 8) {
        const int i = bj * 32 + tx, j = bi * 32 + q;
        if (i < n && j < n) F[i + (long)n * j] = tile[tx][q];
    }
}

// x (nx values) and y (ny) back to the matrix's scale; for a non-finite matrix these and Z are NaN
__global__ void __launch_bounds__(256) work_finish_kernel(long nx, double *x, long ny, double *y, int n, double *Z,
                                                          long ldz, const unsigned long long *amax)
{
    const bool bad = *amax >= kInfBits;
    const int q2 = scale_exp(*amax);
    if (!bad && q2 == 0) return;
    const long t0 = blockIdx.x * 256L + threadIdx.x, step = gridDim.x * 256L;
    for (long i = t0; i < nx; i += step) x[i] = bad ? NAN : scalbn(x[i], q2);
    for (long i = t0; i < ny; i += step) y[i] = bad ? NAN : scalbn(y[i], q2);
    if (bad && Z)
        for (long i = t0; i < (long)n * n; i += step) Z[i % n + ldz * (i / n)] = NAN;
}

// The workspace carve-up of syevd2_impl, as offsets (doubles, 32-aligned); the size
// function and the solver use this one layout.
struct Syevd2Layout {
    size_t Wk, AB, V1, T1, V2, tau2, Tq, dv, ev, VYV, X, T, Mp, part, gram, flags, W1, W2, Vg, Gq, Tg,
        gemm_ws, gemm_doubles, dcw, total;
};

static int q1_groups(int n) { return (sy2sb_panels(n) + Q1_GROUP - 1) / Q1_GROUP; }

// vectors false: what the reduction and the eigenvalues need (no reflectors are kept)
static Syevd2Layout syevd2_layout(int n, bool vectors)
{
    Syevd2Layout L{};
    const size_t nn = (size_t)n * n;
    const size_t S = (size_t)sweep_steps(n, 0) + 1;
    size_t off = 0;
    auto take = [&](size_t cnt) { off = (off + 31) & ~(size_t)31; size_t p = off; off += cnt; return p; };
    L.Wk = take(nn);
    if (vectors) {
        // the fragments of Q2 take the place of the reduction's working copy and of the divide and
        // conquer's workspace, which are through by then
        L.Tq = L.Wk;
        L.dcw = take(dc_workspace_bytes(n) / 8 + 8);
        off = std::max(off, L.Tq + q2_fragment_doubles(n));
        L.V1 = take(sy2sb_vsave_doubles(n));
        L.T1 = take((size_t)(sy2sb_panels(n) + 1) * NB * NB);
        L.V2 = take((size_t)n * S * NB);
        L.tau2 = take((size_t)n * S);
        L.W1 = take((size_t)Q1W * n);
        L.W2 = take(std::max((size_t)Q1W * n, (size_t)(Q1W / 2) * (Q1W / 2)));   // also the T merges' temporary
        L.Vg = take((size_t)Q1W * n);
        L.Gq = take((size_t)Q1W * Q1W);
        L.Tg = take((size_t)q1_groups(n) * Q1W * Q1W);
    }
    L.AB = take((size_t)2 * LDAB * n);
    L.dv = take(n);
    L.ev = take(n + 8);
    L.VYV = take((size_t)n * 6 * NB);               // two [V | Y | V] buffers
    L.X = take((size_t)n * NB);
    L.T = take(NB * NB);
    L.Mp = take(((size_t)n / 128 + 2) * NB * NB);
    L.part = take((size_t)(n / NB + 8) * 4 * NB);
    L.gram = take((size_t)(n / NB + 8) * NB * NB);
    L.flags = take(8);
    // split-K partials: of X (16 slices of n x NB), with vectors also of the group products
    L.gemm_doubles = vectors ? 8 * (size_t)Q1W * n : 16 * (size_t)NB * n;
    L.gemm_ws = take(L.gemm_doubles);
    L.total = off + 64;
    return L;
}

// workspace of dense_syevd in doubles (everything but the output Z)
size_t syevd2_workspace_doubles(int n, bool vectors) { return syevd2_layout(n, vectors).total; }

// the panels of group gq, their V in V1
static Q1Panels q1_panels(int n, int gq, const double *V1)
{
    Q1Panels P{};
    const int np = sy2sb_panels(n);
    size_t off = 0;
    for (int p = 0; p < (gq + 1) * Q1_GROUP; p++) {
        const int q = p - gq * Q1_GROUP, m = n - p * NB - NB;
        if (q >= 0) {
            P.V[q] = p < np ? V1 + off : nullptr;
            P.m[q] = p < np ? m : 0;
        }
        if (p < np) off += (size_t)m * NB;
    }
    return P;
}

// T of every group's merged 256-column reflector: each 128-column half by pairwise merges of its panels' T
// (q1_tmerge_kernel), then the off-diagonal block -T_a G_ab T_b by two GEMMs.  They need the reduction's V and T
// only, and a CTA or a few each: on the second stream they pass beside the chase, which leaves SMs over
// (the stage, n = 1713: 2.30 -> 0.71 ms, n = 7810: 40.3 -> 32.7; the chase takes as long as before).
static int q1_tfactors(int n, const double *V1, const double *T1, double *Vg, double *Gq, double *W2, double *Tg,
                       double *gemm_ws, size_t gemm_ws_doubles, cudaStream_t st)
{
    cudaError_t e;
    const int ngrp = q1_groups(n);
    if ((e = smem_attr(q1_tmerge_kernel, Q1M_SMEM)) != cudaSuccess) return cuda_fail(e, "dsyevd Q1 smem");
    if ((e = cudaMemsetAsync(Tg, 0, sizeof(double) * Q1W * Q1W * ngrp, st)) != cudaSuccess)
        return cuda_fail(e, "dsyevd Q1 T");
    for (int gq = 0; gq < ngrp; gq++) {
        const int p0 = gq * Q1_GROUP, m0 = n - p0 * NB - NB;
        const Q1Panels P = q1_panels(n, gq, V1);
        double *T = Tg + (size_t)gq * Q1W * Q1W;
        q1_gather_kernel<<<(unsigned)(((long)m0 * Q1W + 255) / 256), 256, 0, st>>>(m0, P, Vg);
        int rc = dgemm(true, false, Q1W, Q1W, m0, 1.0, Vg, m0, Vg, m0, 0.0, Gq, Q1W, st, gemm_ws, gemm_ws_doubles);
        for (int hq = 0; hq < Q1_GROUP / 4 && rc == BSRG_OK; hq++) {
            const long o = (long)hq * Q1H * (Q1W + 1);
            q1_tmerge_kernel<<<1, Q1H, Q1M_SMEM, st>>>(Gq + o, P, 4 * hq, T1, p0, T + o);
            rc = cuda_fail(cudaGetLastError(), "dsyevd Q1 T");
        }
        for (int w = Q1H; w < Q1W && rc == BSRG_OK; w *= 2)
            for (int a0 = 0; a0 < Q1W && rc == BSRG_OK; a0 += 2 * w) {
                const int b0 = a0 + w;
                // Wq = G(a, b) T_b (w x w), then T(a, b) = -T_a Wq
                rc = dgemm(false, false, w, w, w, 1.0, Gq + a0 + (long)Q1W * b0, Q1W, T + b0 + (long)Q1W * b0, Q1W,
                           0.0, W2, w, st);
                if (rc == BSRG_OK)
                    rc = dgemm(false, false, w, w, w, -1.0, T + a0 + (long)Q1W * a0, Q1W, W2, w, 0.0,
                               T + a0 + (long)Q1W * b0, Q1W, st);
            }
        if (rc != BSRG_OK) return rc;
    }
    return BSRG_OK;
}

// wait for the stream; device-side waits that ran out report through flags[2], a non-finite matrix
// gives *info = 1 (the results are NaN)
static int syevd2_status(bsrg_ctx *c, const char *who, const int *flags, int *info)
{
    int h[10];
    cudaError_t e;
    if ((e = ctx_read(c, h, flags, sizeof(h))) != cudaSuccess) return cuda_fail(e, who);
    if (h[2] != 0) {
        set_error("%s: a device-side wait timed out (%s)", who,
                  h[2] == 2 ? "bulge chasing" : h[2] == 3 ? "back-transformation wavefront" : "panel barrier");
        return BSRG_ERR_CUDA;
    }
    if (info) *info = (((unsigned long long)(unsigned)h[9] << 32) | (unsigned)h[8]) >= kInfBits ? 1 : 0;
    return BSRG_OK;
}

// Eigenvalues (ascending, w) and eigenvectors (Z, ldz; null: none) of the symmetric A (lower
// triangle referenced).  Z may be A itself.  ws: syevd2_workspace_doubles(n, Z != null).
// tri_d / tri_e non-null: stop after the reduction and copy the tridiagonal (d: n, e: n-1) there
static int syevd2_impl(bsrg_ctx *c, int n, const double *A, long lda, double *w, double *Z, long ldz, double *ws,
                       size_t ws_doubles, void *pinned, size_t pinned_bytes, int *launches, double *tri_d,
                       double *tri_e, int *info)
{
    int nl = 0;
    if (n < 1) return BSRG_OK;
    cudaStream_t st = c->stream;
    cudaError_t e;
    const bool vectors = Z != nullptr;
    if (ws_doubles < syevd2_workspace_doubles(n, vectors)) { set_error("dsyevd: workspace too small"); return BSRG_ERR_NOMEM; }
    if (n > 10240) { set_error("dsyevd: n=%d above 10240", n); return BSRG_ERR_ARG; }
    const int S = sweep_steps(n, 0) + 1;
    const Syevd2Layout L = syevd2_layout(n, vectors);
    double *Wk = ws + L.Wk, *AB = ws + L.AB, *V1 = vectors ? ws + L.V1 : nullptr, *T1 = vectors ? ws + L.T1 : nullptr;
    double *V2 = vectors ? ws + L.V2 : nullptr, *tau2 = ws + L.tau2, *Tq = ws + L.Tq;
    double *dv = ws + L.dv, *ev = ws + L.ev;
    Sy2sbWork sw;
    sw.VYV = ws + L.VYV;
    sw.VYV2 = sw.VYV + (size_t)n * 3 * NB;
    sw.aux = getenv("BSRG_NO_LOOKAHEAD") ? nullptr : c->aux_stream;
    sw.ev_y = c->aux_ev[0];
    sw.ev_c2 = c->aux_ev[1];
    AuxJoin join(sw.aux, st, sw.ev_c2);
    sw.X = ws + L.X;
    sw.T = ws + L.T;
    sw.Mp = ws + L.Mp;
    sw.part = ws + L.part;
    sw.gram = ws + L.gram;
    int *flags = (int *)(ws + L.flags);            // bar[2], err, err2, two tickets; from flags + 8: amax
    unsigned long long *amax = (unsigned long long *)(flags + 8);
    sw.bar = (unsigned *)flags;
    sw.err = flags + 2;
    sw.ticket = (unsigned *)(flags + 4);
    double *W1 = ws + L.W1, *W2 = ws + L.W2;
    double *Vg = ws + L.Vg, *Gq = ws + L.Gq, *Tg = ws + L.Tg;
    sw.gemm_ws_doubles = L.gemm_doubles;
    sw.gemm_ws = ws + L.gemm_ws;
    double *dcw = ws + L.dcw;
    if ((e = cudaMemsetAsync(flags, 0, 8 * sizeof(double), st)) != cudaSuccess)
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
    amax_kernel<<<(unsigned)std::min(n, 148 * 8), 256, 0, st>>>(n, A, lda, amax);
    {
        const unsigned nt = (unsigned)((n + 31) / 32);
        work_copy_kernel<<<dim3(nt, nt), dim3(32, 8), 0, st>>>(n, A, lda, Wk, amax);
    }
    int rc = cuda_fail(cudaGetLastError(), "dsyevd working copy");
    if (rc == BSRG_OK) rc = sy2sb(st, n, Wk, n, V1, T1, sw);
    if (rc != BSRG_OK) return rc;
    rc = band_extract(n, Wk, n, AB, st);
    if (rc != BSRG_OK) return rc;
    stage_end(c, 9, 2 + np * 6);
    c->stage_flops[9] += fl_band;
    if (vectors && np > 0) {
        cudaStream_t sq = sw.aux ? sw.aux : st;
        if (sw.aux && ((e = cudaEventRecord(sw.ev_y, st)) != cudaSuccess ||
                       (e = cudaStreamWaitEvent(sw.aux, sw.ev_y, 0)) != cudaSuccess))
            return cuda_fail(e, "dsyevd Q1 T");
        rc = q1_tfactors(n, V1, T1, Vg, Gq, W2, Tg, sw.gemm_ws, sw.gemm_ws_doubles, sq);
        if (rc != BSRG_OK) return rc;
        if (sw.aux && (e = cudaEventRecord(sw.ev_c2, sw.aux)) != cudaSuccess) return cuda_fail(e, "dsyevd Q1 T");
    }
    stage_begin(c, 10);
    // 2. band -> tridiagonal
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
    rc = bulge_chase(n, AB, dv, ev, V2, tau2, S, sw.err, (unsigned *)(flags + 5), nsm, st);
    if (rc != BSRG_OK) return rc;
    fl_chase = 4.0 * NB * (3.0 * NB) * (double)n * n / (2.0 * NB);      // whole windows, n^2 / (2 NB) steps
    stage_end(c, 10, 2);
    c->stage_flops[10] += fl_chase;
    if (!vectors) {
        // the tridiagonal, or its eigenvalues
        if (tri_d) {
            if ((e = cudaMemcpyAsync(tri_d, dv, sizeof(double) * n, cudaMemcpyDeviceToDevice, st)) != cudaSuccess ||
                (n > 1 && (e = cudaMemcpyAsync(tri_e, ev, sizeof(double) * (n - 1), cudaMemcpyDeviceToDevice, st)) !=
                              cudaSuccess))
                return cuda_fail(e, "dsytrd_2stage");
            work_finish_kernel<<<8, 256, 0, st>>>(n, tri_d, n - 1, tri_e, n, nullptr, 0, amax);
        } else {
            stage_begin(c, 11);
            rc = tridiag_values(st, n, dv, ev, w, ev + n);
            stage_end(c, 11, 3);
            if (rc != BSRG_OK) return rc;
            work_finish_kernel<<<8, 256, 0, st>>>(n, w, 0, nullptr, n, nullptr, 0, amax);
            c->stage_flops[6] += fl_band + fl_chase;
            if (launches) *launches = 3 + np * 6 + 6;
        }
        join.done();                                // the reduction has joined the second stream
        return syevd2_status(c, tri_d ? "dsytrd_2stage" : "dsyevd", flags, info);
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
    if (sw.aux && np > 0 && (e = cudaStreamWaitEvent(st, sw.ev_c2, 0)) != cudaSuccess) return cuda_fail(e, "dsyevd Q1 T");
    join.done();
    {
        for (int gq = q1_groups(n) - 1; gq >= 0; gq--) {
            const int p0 = gq * Q1_GROUP, r0 = p0 * NB + NB, m0 = n - r0;
            const Q1Panels P = q1_panels(n, gq, V1);
            q1_gather_kernel<<<(unsigned)(((long)m0 * Q1W + 255) / 256), 256, 0, st>>>(m0, P, Vg);
            const double *Tq1 = Tg + (size_t)gq * Q1W * Q1W;
            double *Zs = Z + r0;
            rc = dgemm(true, false, Q1W, n, m0, 1.0, Vg, m0, Zs, ldz, 0.0, W1, Q1W, st, sw.gemm_ws,
                       sw.gemm_ws_doubles);
            if (rc == BSRG_OK) rc = dgemm(false, false, Q1W, n, Q1W, 1.0, Tq1, Q1W, W1, Q1W, 0.0, W2, Q1W, st);
            if (rc == BSRG_OK) rc = dgemm(false, false, m0, n, Q1W, -1.0, Vg, m0, W2, Q1W, 1.0, Zs, ldz, st);
            if (rc != BSRG_OK) return rc;
        }
    }
    stage_end(c, 13, 10 * q1_groups(n));
    c->stage_flops[13] += fl_q1;
    work_finish_kernel<<<148, 256, 0, st>>>(n, w, 0, nullptr, n, Z, ldz, amax);
    rc = syevd2_status(c, "dsyevd", flags, info);
    if (rc != BSRG_OK) return rc;
    fl_dc = dc_gemm_flops(n, pinned, nmerge);
    c->stage_flops[11] += fl_dc;
    c->stage_flops[6] += fl_band + fl_chase + fl_dc + fl_q2 + fl_q1;
    // kernels of this library per call
    nl = 4 + np * 6 + 2 + ndc + (n > 2 ? 2 : 0) + 3 * np;
    if (launches) *launches = nl;
    return BSRG_OK;
}

int dense_syevd(bsrg_ctx *c, int n, const double *A, long lda, double *w, double *Z, long ldz, double *ws,
                size_t ws_doubles, void *pinned, size_t pinned_bytes, int *launches, int *info)
{
    return syevd2_impl(c, n, A, lda, w, Z, ldz, ws, ws_doubles, pinned, pinned_bytes, launches, nullptr, nullptr,
                       info);
}

}  // namespace bsrg

using namespace bsrg;

extern "C" int bsrg_dsytrd_2stage(bsrg_ctx *c, int n, const double *A, int lda, double *d, double *e)
{
    if (!c || (n > 0 && (!A || !d || (n > 1 && !e)))) { set_error("dsytrd_2stage: null argument"); return BSRG_ERR_ARG; }
    if (n < 0 || lda < (n > 0 ? n : 1)) { set_error("dsytrd_2stage: n=%d lda=%d", n, lda); return BSRG_ERR_ARG; }
    if (n == 0) return BSRG_OK;
    cudaSetDevice(c->device);
    int rc = ctx_reserve(c, syevd2_workspace_doubles(n, false) * sizeof(double) + 1024);
    if (rc != BSRG_OK) return rc;
    rc = syevd2_impl(c, n, A, lda, nullptr, nullptr, n, (double *)c->ws, c->ws_bytes / sizeof(double), nullptr, 0,
                     nullptr, d, e, nullptr);
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
                     c->pinned_bytes, nullptr, nullptr);
    cudaEventRecord(c->ev_stage, c->stream);
    return rc;
}
