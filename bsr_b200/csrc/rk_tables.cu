// B-spline basis tables and R^k cell tables on the GPU.
//
// Replaces, for the reference's B-spline library (src/libs/BS):
//   initvb  (define_spline.f90:67)  -> basis_points_kernel
//   mdb1/mdb2/mrm (define_spline.f90:184,214, mrm.f90:2) -> band_kernel
//   moments/moment (moments.f90:2,76) -> moment_blocks
//   rk_triang/rk_pdiag (rk_moments.f90:56,105) -> rk_diag_cell
//   mrk_cell (mrk_cell.f90:2) and the Breit-Pauli tables: rk_expand.cu
//
// This file is compiled with --fmad=false: every sum is accumulated in the
// reference's order with separately rounded multiplies and adds, so the tables
// equal the Fortran restatement's bit for bit.
#include "bsrg_internal.h"

namespace bsrg {

// de Boor's bsplvb/bsplvd (vbsplvd.f90:3,170) for one point.  left is the
// 0-based knot index with t[left] <= x <= t[left+1].  db[j + k*m] = m-th
// derivative of the j-th of the k B-splines nonzero on that interval.
struct BvbState {
    int j;
    double deltal[BSRG_MAXKS + 1], deltar[BSRG_MAXKS + 1];
};

__device__ static void bsplvb_dev(const double *t, int jhigh, int index, double x, int left,
                                           double *biatx, BvbState &st)
{
    if (index == 1) {
        st.j = 1;
        biatx[0] = 1.0;
        if (st.j >= jhigh) return;
    }
    for (;;) {
        int j = st.j, jp1 = j + 1;
        st.deltar[j - 1] = t[left + j] - x;
        st.deltal[j - 1] = x - t[left + 1 - j];
        double saved = 0.0;
        for (int i = 1; i <= j; i++) {
            double term = biatx[i - 1] / (st.deltar[i - 1] + st.deltal[jp1 - i - 1]);
            biatx[i - 1] = saved + st.deltar[i - 1] * term;
            saved = st.deltal[jp1 - i - 1] * term;
        }
        biatx[jp1 - 1] = saved;
        st.j = jp1;
        if (st.j >= jhigh) break;
    }
}

__device__ static void bsplvd_dev(const double *t, int k, double x, int left, int nderiv, double *db)
{
    BvbState st;
    int mhigh = nderiv < k ? nderiv : k;
    if (mhigh < 1) mhigh = 1;
    int kp1 = k + 1;
    bsplvb_dev(t, kp1 - mhigh, 1, x, left, db, st);
    if (mhigh == 1) return;
    int ideriv = mhigh;
    for (int m = 2; m <= mhigh; m++) {
        int jp1mid = 1;
        for (int j = ideriv; j <= k; j++) {
            db[(j - 1) + k * (ideriv - 1)] = db[jp1mid - 1];
            jp1mid++;
        }
        ideriv--;
        bsplvb_dev(t, kp1 - ideriv, 2, x, left, db, st);
    }
    double a[BSRG_MAXKS * BSRG_MAXKS];
#define A(i, j) a[((i) - 1) + k * ((j) - 1)]
    int jlow = 1;
    for (int i = 1; i <= k; i++) {
        for (int j = jlow; j <= k; j++) A(j, i) = 0.0;
        jlow = i;
        A(i, i) = 1.0;
    }
    for (int m = 2; m <= mhigh; m++) {
        int kp1mm = kp1 - m;
        double fk = (double)kp1mm;
        int il = left, i = k;
        for (int ld = 1; ld <= kp1mm; ld++) {
            double factor = fk / (t[il + kp1mm] - t[il]);
            for (int j = 1; j <= i; j++) A(i, j) = (A(i, j) - A(i - 1, j)) * factor;
            il--;
            i--;
        }
        for (int ii = 1; ii <= k; ii++) {
            double sum = 0.0;
            int jl = ii > m ? ii : m;
            for (int j = jl; j <= k; j++) sum = sum + A(j, ii) * db[(j - 1) + k * (m - 1)];
            db[(ii - 1) + k * (m - 1)] = sum;
        }
    }
#undef A
}

// values of the ks B-splines at x (nderiv = 1): bsplvb_dev's steps with its arrays in registers (the
// divisions of one order are independent and overlap; through local memory they followed one another)
__device__ static void bspl_values(const double *t, int k, double x, int left, double *v)
{
    double b[BSRG_MAXKS], dl[BSRG_MAXKS], dr[BSRG_MAXKS];
    b[0] = 1.0;
#pragma unroll
    for (int j = 1; j < BSRG_MAXKS; j++) {
        if (j >= k) break;
        dr[j - 1] = t[left + j] - x;
        dl[j - 1] = x - t[left + 1 - j];
        double saved = 0.0;
#pragma unroll
        for (int i = 1; i <= j; i++) {
            const double term = b[i - 1] / (dr[i - 1] + dl[j - i]);
            b[i - 1] = saved + dr[i - 1] * term;
            saved = dl[j - i] * term;
        }
        b[j] = saved;
    }
#pragma unroll
    for (int j = 0; j < BSRG_MAXKS; j++)
        if (j < k) v[j] = b[j];
}

// ---------------------------------------------------------------------------
// initvb: one thread per (interval, Gauss point); thread nv*ks does the last knot.
// ---------------------------------------------------------------------------
struct GaussRule { double x[BSRG_MAXKS], w[BSRG_MAXKS]; };

__global__ void basis_points_kernel(int ks, int ns, int nv, const double *__restrict__ t, GaussRule g,
                                    double *gr, double *grm, double *grw, double *bsp, double *bsq,
                                    double *bspd)
{
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    double db[BSRG_MAXKS * 3];
    size_t ld = (size_t)(nv + 1);
    if (tid < nv * ks) {
        int iv = tid % nv, m = tid / nv;
        double tl = t[iv + ks - 1], tr = t[iv + ks];
        double x = (tr - tl) * g.x[m] + tl;
        double xm = 1.0 / x;
        gr[iv + (size_t)nv * m] = x;
        grm[iv + (size_t)nv * m] = xm;
        grw[iv + (size_t)nv * m] = (tr - tl) * g.w[m];
        bsplvd_dev(t, ks, x, iv + ks - 1, 3, db);
        for (int ith = 0; ith < ks; ith++) {
            size_t o = iv + ld * (m + (size_t)ks * ith);
            double v = db[ith], d1 = db[ith + ks], d2 = db[ith + 2 * ks];
            bsp[o] = v;
            bspd[o] = d1;
            bspd[o + ld * ks * ks] = d2;
            bsq[o] = d1 - xm * v;
        }
    } else if (tid == nv * ks) {
        double x = t[ns];
        bsplvd_dev(t, ks, x, ns - 1, 3, db);
        for (int ith = 0; ith < ks; ith++) {
            size_t o = nv + ld * (0 + (size_t)ks * ith);
            double v = db[ith], d1 = db[ith + ks], d2 = db[ith + 2 * ks];
            bsp[o] = v;
            bspd[o] = d1;
            bspd[o + ld * ks * ks] = d2;
            bsq[o] = d1 - v / x;
        }
    }
}

// ---------------------------------------------------------------------------
// Band operator matrices in lower-column storage, one thread per (irow, jcol):
//   kind 0: <B_i|r^mm|B_j> (mrm.f90), kind 1: <B_i|B'_j> (mdb1), kind 2: <B_i|B''_j> (mdb2).
// The reference accumulates over ith = 1..ks (outer loop) for a fixed element.
// ---------------------------------------------------------------------------
__device__ static double rpow_dev(double g, int p)
{
    double r = g;
    for (int q = 1; q < p; q++) r = r * g;
    return r;
}

__global__ void band_kernel(int ks, int ns, int nv, int kind, int mm, const double *__restrict__ gr,
                            const double *__restrict__ grm, const double *__restrict__ grw,
                            const double *__restrict__ bsp, const double *__restrict__ bspd, double *out)
{
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= ns * ks) return;
    int irow = tid % ns, jcol = tid / ns;
    size_t ld = (size_t)(nv + 1);
    double acc = 0.0;
    for (int ith = 0; ith < ks; ith++) {
        int iv = irow - ith;
        int jth = jcol + ith - (ks - 1);
        if (iv < 0 || iv >= nv || jth < 0 || jth > ith) continue;
        double s = 0.0;
        for (int m = 0; m < ks; m++) {
            double w = grw[iv + (size_t)nv * m];
            double bi = bsp[iv + ld * (m + (size_t)ks * ith)];
            double wb = w * bi, v;
            if (kind == 0) {
                double bj = bsp[iv + ld * (m + (size_t)ks * jth)];
                if (mm == 0) v = wb * bj;
                else if (mm == -1) v = wb * grm[iv + (size_t)nv * m] * bj;
                else if (mm <= -2) v = wb * rpow_dev(grm[iv + (size_t)nv * m], -mm) * bj;
                else if (mm == 1) v = wb * gr[iv + (size_t)nv * m] * bj;
                else v = wb * rpow_dev(gr[iv + (size_t)nv * m], mm) * bj;
            } else {
                double dj = bspd[iv + ld * (m + (size_t)ks * (jth + (size_t)ks * (kind - 1)))];
                v = wb * dj;
            }
            s = s + v;
        }
        acc = acc + s;
    }
    if (kind == 2 && tid == 0) {
        // db2(1,1) holds <B_{ns-1}|B''_{ns}> over the last interval (define_spline.f90:238)
        int iv = nv - 1;
        double s = 0.0;
        for (int m = 0; m < ks; m++)
            s = s + grw[iv + (size_t)nv * m] * bsp[iv + ld * (m + (size_t)ks * (ks - 2))] *
                        bspd[iv + ld * (m + (size_t)ks * ((ks - 1) + (size_t)ks * 1))];
        acc = acc + s;
    }
    out[irow + (size_t)ns * jcol] = acc;
}

// ---------------------------------------------------------------------------
// moments (moments.f90:2,76): rkm(ii, iv), one thread each.
// With me > 0 the geometric region repeats the reference's scaling chain
// rkm(:,iv) = rkm(:,iv-1)*hp starting from the last directly computed cell.
// ---------------------------------------------------------------------------
// One moment array of a launch: rkm(ii, iv), ii over the ks(ks+1)/2 pairs i <= j or (full) over all ks*ks
// pairs with B_j or (deriv) the derivative operator's bsq_j as the second spline; combine: the moments of
// W^k and Q^k (wk_moments.f90:44-52), 2 m(k) + c m2 or (minus) 2 m(k) - c m2 with m2 the moment k2 of B_j.
struct MomentJob {
    double *out;
    int full, deriv, k;
    double hp;
    int combine, minus, k2;
    double hp2, c;
};
constexpr int MAX_JOBS = 4;
struct MomentJobs {
    int n;
    MomentJob j[MAX_JOBS];
};
struct CellGrid {                // what every kernel of the cell moments reads
    int ks, nv, ml, me;
    const double *t, *gr, *grm, *grw, *bsp, *bsq, *bspd;
};

__device__ static double moment_value(const CellGrid &b, int iv_out, int k, double hp, int i, int j, const double *second)
{
    const int iv1 = iv_out + 1;                            // 1-based
    const int s0 = b.ml + b.ks, s1 = b.ml + b.me - b.ks + 2;  // scaled range (1-based), empty when me == 0
    const bool scaled = b.me != 0 && iv1 >= s0 && iv1 <= s1;
    const int iv = scaled ? s0 - 2 : iv_out;
    const size_t ld = (size_t)(b.nv + 1);
    double v = 0.0;
    for (int m = 0; m < b.ks; m++) {
        double gw = b.grw[iv + (size_t)b.nv * m];
        if (k > 0) gw = gw * rpow_dev(b.gr[iv + (size_t)b.nv * m], k);
        if (k < 0) gw = gw * rpow_dev(b.grm[iv + (size_t)b.nv * m], -k);
        const double bj = second[iv + ld * (m + (size_t)b.ks * j)] * gw;
        v = v + b.bsp[iv + ld * (m + (size_t)b.ks * i)] * bj;
    }
    if (scaled)
        for (int q = s0; q <= iv1; q++) v = v * hp;
    return v;
}

// the moment arrays of a launch, one element a thread; block 0 is the first after the diagonal cells'
__device__ static void moment_blocks(const CellGrid &b, const MomentJobs &jobs, int block)
{
    long e = (long)block * blockDim.x + threadIdx.x;
    for (int q = 0; q < jobs.n; q++) {
        const MomentJob &w = jobs.j[q];
        const int np = w.full ? b.ks * b.ks : b.ks * (b.ks + 1) / 2;
        const long size = (long)np * b.nv;
        if (e >= size) { e -= size; continue; }
        const int ii = (int)(e % np), iv = (int)(e / np);
        int i, j;
        if (w.full) { i = ii / b.ks; j = ii % b.ks; }
        else {
            int rem = ii;
            i = 0;
            while (rem >= b.ks - i) { rem -= b.ks - i; i++; }
            j = i + rem;
        }
        double v = moment_value(b, iv, w.k, w.hp, i, j, w.deriv ? b.bsq : b.bsp);
        if (w.combine) {
            const double m2 = moment_value(b, iv, w.k2, w.hp2, i, j, b.bsp);
            v = w.minus ? 2 * v - w.c * m2 : 2 * v + w.c * m2;
        }
        w.out[e] = v;
        return;
    }
}

// ---------------------------------------------------------------------------
// One interval's slice of the basis in shared memory: [m][i] values, bsq and derivatives, [m] 1/r and weights.
struct CellSlice {
    double b[BSRG_MAXKS * BSRG_MAXKS], q[BSRG_MAXKS * BSRG_MAXKS], d[BSRG_MAXKS * BSRG_MAXKS];
    double grm[BSRG_MAXKS], grw[BSRG_MAXKS];
};
__device__ static void load_slice(const CellGrid &b, int iv, bool ops, CellSlice &s)
{
    const size_t ld = (size_t)(b.nv + 1);
    const int ks = b.ks;
    for (int e = threadIdx.x; e < ks * ks; e += blockDim.x) {
        const size_t at = iv + ld * (e / ks + (size_t)ks * (e % ks));      // e = m ks + i
        s.b[e] = b.bsp[at];
        if (ops) {
            s.q[e] = b.bsq[at];
            s.d[e] = b.bspd[at];
        }
    }
    for (int m = threadIdx.x; m < ks; m += blockDim.x) {
        s.grm[m] = b.grm[iv + (size_t)b.nv * m];
        s.grw[m] = b.grw[iv + (size_t)b.nv * m];
    }
}

// rk_triang (rk_moments.f90:105): one CTA per diagonal cell.  With me > 0 the
// cells of the geometric region repeat rk_pdiag's chain rkd(iv) = rkd(iv-1)*(1+h).
// ---------------------------------------------------------------------------
__device__ static void rk_diag_cell(const CellGrid &b, double hscale, int k, const GaussRule &g, double *rkd, int iv_out)
{
    const int ks = b.ks, nv = b.nv, ml = b.ml, me = b.me;
    const double *t = b.t, *gr = b.gr;
    __shared__ CellSlice sl;
    extern __shared__ double sm[];
    const int ik = ks * (ks + 1) / 2;
    double *bt = sm;                          // [m][i][j] : ks*ks*ks  B-spline values at inner points
    double *wx = bt + ks * ks * ks;           // [m][i]   : weights * x^k at inner points
    double *INT = wx + ks * ks;               // [m][jj]  : ks*ik
    double *a = INT + ks * ik;                // [jj][ii] : ik*ik  (column-major a(ii,jj))
    double *BI = a + ik * ik;                 // [ii][m]  : ik*ks  bsp(i)*bsp(ip)*grw*grm^(k+1)
    int iv1 = iv_out + 1;
    int s0 = ml + ks, s1 = ml + me - ks + 2;
    int nscale = 0, iv = iv_out;
    if (me != 0 && iv1 >= s0 && iv1 <= s1) { iv = s0 - 2; nscale = iv1 - s0 + 1; }
    int left = iv + ks - 1;
    double xbase = t[left];
    load_slice(b, iv, false, sl);
    // inner points: for each outer Gauss point m, ks points on [t_left, gr(iv,m)]
    for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) {
        int m = q / ks, i = q % ks;
        double span = gr[iv + (size_t)nv * m] - xbase;
        double x = span * g.x[i] + xbase;
        double v[BSRG_MAXKS];
        bspl_values(t, ks, x, left, v);
        for (int j = 0; j < ks; j++) bt[(m * ks + i) * ks + j] = v[j];
        double w = span * g.w[i];
        double xk;
        if (k > 1) xk = w * rpow_dev(x, k);
        else if (k == 1) xk = w * x;
        else xk = w;
        wx[m * ks + i] = xk;
    }
    __syncthreads();
    // INT(j,jp,m) = SUM_i (wx_i * bt(i,j)) * bt(i,jp)
    for (int q = threadIdx.x; q < ks * ik; q += blockDim.x) {
        int m = q / ik, jj = q % ik;
        int j = 0, rem = jj;
        while (rem >= ks - j) { rem -= ks - j; j++; }
        int jp = j + rem;
        double s = 0.0;
        for (int i = 0; i < ks; i++) {
            double tmp = wx[m * ks + i] * bt[(m * ks + i) * ks + j];
            s = s + tmp * bt[(m * ks + i) * ks + jp];
        }
        INT[m * ik + jj] = s;
    }
    __syncthreads();
    // bi(ii,m) = bsp(i)*bsp(ip)*grw*grm^(k+1), once per cell
    for (int q = threadIdx.x; q < ik * ks; q += blockDim.x) {
        int ii = q / ks, m = q % ks;
        int i = 0, rem = ii;
        while (rem >= ks - i) { rem -= ks - i; i++; }
        int ip = i + rem;
        double g2;
        if (k != 0) g2 = sl.grw[m] * rpow_dev(sl.grm[m], k + 1);
        else g2 = sl.grw[m] * sl.grm[m];
        BI[q] = sl.b[m * ks + i] * sl.b[m * ks + ip] * g2;
    }
    __syncthreads();
    // a(ii,jj) = SUM_m bi(ii,m) * INT(jj,m)
    for (int q = threadIdx.x; q < ik * ik; q += blockDim.x) {
        int ii = q % ik, jj = q / ik;
        const double *bi = BI + ii * ks;
        double s = 0.0;
        for (int m = 0; m < ks; m++) s = s + bi[m] * INT[m * ik + jj];
        a[ii + ik * jj] = s;
    }
    __syncthreads();
    double *out = rkd + (size_t)ik * ik * iv_out;
    for (int q = threadIdx.x; q < ik * ik; q += blockDim.x) {
        int r = q % ik, c = q / ik;
        double v = a[r + ik * c] + a[c + ik * r];
        for (int n = 0; n < nscale; n++) v = v * hscale;
        out[r + (size_t)ik * c] = v;
    }
}

// ---------------------------------------------------------------------------
// Breit-Pauli N^k tables.  nk_triang (nk_moments.f90:105): the diagonal cell of
// r2 < r1 only (inner weight r2^k, k >= -1; outer r1^-(k+3) folded into the
// inner integral), not symmetrised; nk_pdiag's scaling law divides by (1+h).
// ---------------------------------------------------------------------------
__device__ static double ipow_dev(double x, int k)
{
    if (k == 0) return 1.0;
    double p = x;
    const int a = k > 0 ? k : -k;
    for (int q = 1; q < a; q++) p = p * x;
    return k > 0 ? p : 1.0 / p;
}

__device__ static void nk_diag_cell(const CellGrid &b, double hscale, int k, int sym, const GaussRule &g, double *rkd,
                                    int iv_out)
{
    const int ks = b.ks, nv = b.nv, ml = b.ml, me = b.me;
    const double *t = b.t, *gr = b.gr;
    __shared__ CellSlice sl;
    extern __shared__ double sm[];
    const int ik = ks * (ks + 1) / 2;
    double *bt = sm;                          // [m][i][j] : B-spline values at the inner points
    double *wx = bt + ks * ks * ks;           // [m][i]   : inner weights * x^k
    double *INT = wx + ks * ks;               // [m][jj]
    double *a = INT + ks * ik;                // [jj][ii] (sym only): a(ii,jj) before a + a^T
    int iv1 = iv_out + 1;
    int s0 = ml + ks, s1 = ml + me - ks + 2;
    int nscale = 0, iv = iv_out;
    if (me != 0 && iv1 >= s0 && iv1 <= s1) { iv = s0 - 2; nscale = iv1 - s0 + 1; }
    int left = iv + ks - 1;
    double xbase = t[left];
    load_slice(b, iv, false, sl);
    for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) {
        int m = q / ks, i = q % ks;
        double span = gr[iv + (size_t)nv * m] - xbase;
        double x = span * g.x[i] + xbase;
        double v[BSRG_MAXKS];
        bspl_values(t, ks, x, left, v);
        for (int j = 0; j < ks; j++) bt[(m * ks + i) * ks + j] = v[j];
        wx[m * ks + i] = span * g.w[i] * ipow_dev(x, k);
    }
    __syncthreads();
    // INT(j,jp,m) = (SUM_i (wx_i bt(i,j)) bt(i,jp)) * grw(m) grm(m)^(k+3)
    for (int q = threadIdx.x; q < ks * ik; q += blockDim.x) {
        int m = q / ik, jj = q % ik;
        int j = 0, rem = jj;
        while (rem >= ks - j) { rem -= ks - j; j++; }
        int jp = j + rem;
        double s = 0.0;
        for (int i = 0; i < ks; i++) {
            double tmp = wx[m * ks + i] * bt[(m * ks + i) * ks + j];
            s = s + tmp * bt[(m * ks + i) * ks + jp];
        }
        const double c = sl.grw[m] * ipow_dev(sl.grm[m], k + 3);
        INT[m * ik + jj] = s * c;
    }
    __syncthreads();
    double *out = rkd + (size_t)ik * ik * iv_out;
    for (int q = threadIdx.x; q < ik * ik; q += blockDim.x) {
        int ii = q % ik, jj = q / ik;
        int i = 0, rem = ii;
        while (rem >= ks - i) { rem -= ks - i; i++; }
        int ip = i + rem;
        double s = 0.0;
        for (int m = 0; m < ks; m++) {
            double g3 = sl.b[m * ks + i] * sl.b[m * ks + ip];
            s = s + g3 * INT[m * ik + jj];
        }
        if (sym) {
            a[ii + ik * jj] = s;
        } else {
            for (int n = 0; n < nscale; n++) s = s / hscale;
            out[ii + (size_t)ik * jj] = s;
        }
    }
    if (!sym) return;
    // mk_triang (mk_moments.f90:96): the cell returned as a + transpose(a)
    __syncthreads();
    for (int q = threadIdx.x; q < ik * ik; q += blockDim.x) {
        int r = q % ik, c = q / ik;
        double v = a[r + ik * c] + a[c + ik * r];
        for (int n = 0; n < nscale; n++) v = v / hscale;
        out[r + (size_t)ik * c] = v;
    }
}

// ---------------------------------------------------------------------------
// Breit-Pauli T^k (tk_moments.f90).
// ---------------------------------------------------------------------------
// tk_triang (tk_moments.f90:101): inner integral of B_j (dB_jp/dr - B_jp/r) r^k
// up to each outer Gauss point, outer weights bsq grw grm^(k+1), a + a^T.
__device__ static void tk_diag_cell(const CellGrid &b, double hscale, int k, const GaussRule &g, double *rkd, int iv_out)
{
    const int ks = b.ks, nv = b.nv, ml = b.ml, me = b.me;
    const double *t = b.t, *gr = b.gr;
    __shared__ CellSlice sl;
    extern __shared__ double sm[];
    const int jk = ks * ks;
    double *bt = sm;                          // [m][i][j] values
    double *bd = bt + ks * ks * ks;           // [m][i][j] derivative - value/x
    double *wx = bd + ks * ks * ks;           // [m][i]
    double *INT = wx + ks * ks;               // [m][j][jp]
    double *bq = INT + ks * ks * ks;          // [m][ip]
    double *a = bq + ks * ks;                 // a(ii,jj), column-major jk x jk
    const int iv1 = iv_out + 1;
    const int s0 = ml + ks, s1 = ml + me - ks + 2;
    int nscale = 0, iv = iv_out;
    if (me != 0 && iv1 >= s0 && iv1 <= s1) { iv = s0 - 2; nscale = iv1 - s0 + 1; }
    const int left = iv + ks - 1;
    const double xbase = t[left];
    load_slice(b, iv, true, sl);
    for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) {
        const int m = q / ks, i = q % ks;
        const double span = gr[iv + (size_t)nv * m] - xbase;
        const double x = span * g.x[i] + xbase;
        double db[2 * BSRG_MAXKS];
        bsplvd_dev(t, ks, x, left, 2, db);
        for (int j = 0; j < ks; j++) {
            bt[(m * ks + i) * ks + j] = db[j];
            bd[(m * ks + i) * ks + j] = db[j + ks] - db[j] / x;
        }
        wx[m * ks + i] = ipow_dev(x, k) * (span * g.w[i]);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) {
        const int m = q / ks, ip = q % ks;
        const double g2 = sl.grw[m] * ipow_dev(sl.grm[m], k + 1);
        bq[m * ks + ip] = sl.q[m * ks + ip] * g2;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < ks * jk; q += blockDim.x) {
        const int m = q / jk, j = (q % jk) / ks, jp = q % ks;
        double s = 0.0;
        for (int i = 0; i < ks; i++) {
            const double tmp = wx[m * ks + i] * bt[(m * ks + i) * ks + j];
            s = s + tmp * bd[(m * ks + i) * ks + jp];
        }
        INT[(m * ks + j) * ks + jp] = s;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < jk * jk; q += blockDim.x) {
        const int ii = q % jk, jj = q / jk;
        const int i = ii / ks, ip = ii % ks, j = jj / ks, jp = jj % ks;
        double s = 0.0;
        for (int m = 0; m < ks; m++) {
            const double g3 = sl.b[m * ks + i] * bq[m * ks + ip];
            s = s + g3 * INT[(m * ks + j) * ks + jp];
        }
        a[ii + jk * jj] = s;
    }
    __syncthreads();
    double *out = rkd + (size_t)jk * jk * iv_out;
    for (int q = threadIdx.x; q < jk * jk; q += blockDim.x) {
        const int r = q % jk, c = q / jk;
        double v = a[r + jk * c] + a[c + jk * r];
        for (int n = 0; n < nscale; n++) v = v / hscale;
        out[r + (size_t)jk * c] = v;
    }
}

// ---------------------------------------------------------------------------
// Breit-Pauli V^k (vk_moments.f90, mvk_cell.f90).  vk_triang (:131): two inner
// integrals, I1(i,ip) of B_i (dB_ip/dr - B_ip/r) r^k with outer grm^(k+2), and
// I2(j,jp) of B_j B_jp r^(k+1) with outer grm^(k+3); rkd(ii = (i,ip) all pairs,
// jj = (j <= jp)) = sum bsp_j bsp_jp I1 + sum bsp_i bsq_ip I2.
// ---------------------------------------------------------------------------
__device__ static void vk_diag_cell(const CellGrid &b, double hscale, int k, int mode, const GaussRule &g, double *rkd,
                                    int iv_out)
{
    const int ks = b.ks, nv = b.nv, ml = b.ml, me = b.me;
    const double *t = b.t, *gr = b.gr;
    __shared__ CellSlice sl;
    extern __shared__ double sm[];
    const int jk = ks * ks, ik = ks * (ks + 1) / 2;
    double *bt = sm;                          // [m][q][j] values
    double *bd = bt + ks * ks * ks;           // [m][q][j] derivative - value/x
    double *w1 = bd + ks * ks * ks;           // [m][q] span w x^k
    double *w2 = w1 + ks * ks;                // [m][q] span w x^(k+1)
    double *I1 = w2 + ks * ks;                // [m][i][ip]
    double *I2 = I1 + ks * ks * ks;           // [m][j][jp]
    const int iv1 = iv_out + 1;
    const int s0 = ml + ks, s1 = ml + me - ks + 2;
    int nscale = 0, iv = iv_out;
    if (me != 0 && iv1 >= s0 && iv1 <= s1) { iv = s0 - 2; nscale = iv1 - s0 + 1; }
    const int left = iv + ks - 1;
    const double xbase = t[left];
    load_slice(b, iv, true, sl);
    for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) {
        const int m = q / ks, i = q % ks;
        const double span = gr[iv + (size_t)nv * m] - xbase;
        const double x = span * g.x[i] + xbase;
        double db[2 * BSRG_MAXKS];
        bsplvd_dev(t, ks, x, left, 2, db);
        for (int j = 0; j < ks; j++) {
            bt[(m * ks + i) * ks + j] = db[j];
            // V^k: dB/dr - B/r; W^k (wk_triang, wk_moments.f90:167): 2 dB/dr + k B/r
            bd[(m * ks + i) * ks + j] = mode ? 2 * db[j + ks] + (double)k * db[j] / x : db[j + ks] - db[j] / x;
        }
        const double w = span * g.w[i] * ipow_dev(x, k);
        w1[m * ks + i] = w;
        w2[m * ks + i] = w * x;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < ks * jk; q += blockDim.x) {
        const int m = q / jk, a = (q % jk) / ks, b = q % ks;
        const double gm = sl.grm[m], gwm = sl.grw[m];
        double s = 0.0, u = 0.0;
        for (int i = 0; i < ks; i++) {
            const double x1 = w1[m * ks + i] * bt[(m * ks + i) * ks + a];
            s = s + x1 * bd[(m * ks + i) * ks + b];
            const double x2 = w2[m * ks + i] * bt[(m * ks + i) * ks + a];
            u = u + x2 * bt[(m * ks + i) * ks + b];
        }
        I1[(m * ks + a) * ks + b] = s * (ipow_dev(gm, k + 2) * gwm);
        I2[(m * ks + a) * ks + b] = u * (ipow_dev(gm, k + 3) * gwm);
    }
    __syncthreads();
    // V^k, W^k: jj over the ik pairs j <= jp; Q^k (mode 2, qk_triang): over all ks*ks pairs
    const int njj = mode == 2 ? jk : ik;
    double *out = rkd + (size_t)jk * njj * iv_out;
    for (int q = threadIdx.x; q < jk * njj; q += blockDim.x) {
        const int ii = q % jk, jj = q / jk;
        const int i = ii / ks, ip = ii % ks;
        int j, jp;
        if (mode == 2) {
            j = jj / ks;
            jp = jj % ks;
        } else {
            j = 0;
            int rem = jj;
            while (rem >= ks - j) { rem -= ks - j; j++; }
            jp = j + rem;
        }
        double s1 = 0.0, s2 = 0.0;
        for (int m = 0; m < ks; m++) {
            const double g3 = sl.b[m * ks + j] * sl.b[m * ks + jp];
            s1 = s1 + g3 * I1[(m * ks + i) * ks + ip];
        }
        for (int m = 0; m < ks; m++) {
            // V^k: bsq; W^k (wk_moments.f90:218): 2 dB/dr - (k+3) B/r from the basis tables
            const double op = mode ? 2 * sl.d[m * ks + ip] -
                                         (double)(k + 3) * sl.grm[m] * sl.b[m * ks + ip]
                                   : sl.q[m * ks + ip];
            const double g3 = sl.b[m * ks + i] * op;
            s2 = s2 + g3 * I2[(m * ks + j) * ks + jp];
        }
        double v = s1 + s2;
        for (int n = 0; n < nscale; n++) v = v / hscale;
        out[ii + (size_t)jk * jj] = v;
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static GaussRule rule_of(const bsrg_basis *b)
{
    GaussRule g;
    for (int i = 0; i < BSRG_MAXKS; i++) { g.x[i] = i < b->ks ? b->gx[i] : 0.0; g.w[i] = i < b->ks ? b->gw[i] : 0.0; }
    return g;
}

int launch_basis_tables(bsrg_basis *b, cudaStream_t s)
{
    int n = b->nv * b->ks + 1;
    basis_points_kernel<<<(n + 127) / 128, 128, 0, s>>>(b->ks, b->ns, b->nv, b->t, rule_of(b), b->gr, b->grm,
                                                         b->grw, b->bsp, b->bsq, b->bspd);
    int nb = b->ns * b->ks, bl = (nb + 127) / 128;
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 1, 0, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->db1);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 2, 0, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->db2);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, 0, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->sb);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, 1, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->r1);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, -1, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->rm1);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, -2, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->rm2);
    band_kernel<<<bl, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, -3, b->gr, b->grm, b->grw, b->bsp, b->bspd, b->rm3);
    return cuda_fail(cudaGetLastError(), "basis tables");
}

int launch_mrm(const bsrg_basis *b, int mm, double *rm, cudaStream_t s)
{
    int nb = b->ns * b->ks;
    band_kernel<<<(nb + 127) / 128, 128, 0, s>>>(b->ks, b->ns, b->nv, 0, mm, b->gr, b->grm, b->grw, b->bsp,
                                                 b->bspd, rm);
    return cuda_fail(cudaGetLastError(), "mrm");
}

static double ipow_host(double q, int k)
{
    double hp = 1.0;
    if (k >= 0) { for (int i = 0; i < k; i++) hp *= q; }
    else { double p = 1.0; for (int i = 0; i < -k; i++) p *= q; hp = 1.0 / p; }
    return hp;
}

static CellGrid grid_of(const bsrg_basis *b)
{
    return CellGrid{b->ks, b->nv, b->ml, b->me, b->t, b->gr, b->grm, b->grw, b->bsp, b->bsq, b->bspd};
}

// The moments and the diagonal cells of one multipole in one launch: blocks 0 .. ncell-1 a diagonal cell
// each, the others the moment arrays.  They are a few microseconds of latency each and independent: 35.5 us
// as three launches at ks = 10, ns = 200 (23.8 at ks = 8, ns = 60), 20.4 (11.3) in one.  Two CTAs per
// SM keep the 191 cells of a 200-spline grid in one wave (one CTA of 512 threads: 27 us).
constexpr int CELL_NT = 384;
enum { CELL_RK, CELL_NK, CELL_TK, CELL_VK };
template <int KIND>
__global__ void __launch_bounds__(CELL_NT, 2) cells_kernel(CellGrid b, MomentJobs jobs, int ncell, double hscale, int k, int mode,
                                                    GaussRule g, double *rkd)
{
    if ((int)blockIdx.x >= ncell) { moment_blocks(b, jobs, blockIdx.x - ncell); return; }
    if (KIND == CELL_RK) rk_diag_cell(b, hscale, k, g, rkd, blockIdx.x);
    if (KIND == CELL_NK) nk_diag_cell(b, hscale, k, mode, g, rkd, blockIdx.x);
    if (KIND == CELL_TK) tk_diag_cell(b, hscale, k, g, rkd, blockIdx.x);
    if (KIND == CELL_VK) vk_diag_cell(b, hscale, k, mode, g, rkd, blockIdx.x);
}

template <int KIND>
static int launch_cells(const bsrg_basis *b, const MomentJobs &jobs, int k, int mode, double *rkd, size_t shm,
                        const char *what, cudaStream_t s)
{
    long elems = 0;
    for (int q = 0; q < jobs.n; q++)
        elems += (long)(jobs.j[q].full ? b->ks * b->ks : ik_of(b->ks)) * b->nv;
    const int ncell = rkd ? b->nv : 0;
    const long blocks = ncell + (elems + CELL_NT - 1) / CELL_NT;
    if (blocks == 0) return BSRG_OK;
    if (!rkd) shm = 0;
    if (shm + sizeof(CellSlice) > 48 * 1024) {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (shm + sizeof(CellSlice) > (size_t)optin) {
            set_error("%s: a diagonal cell of ks=%d needs %zu bytes of shared memory (device limit %d)", what, b->ks, shm + sizeof(CellSlice),
                      optin);
            return BSRG_ERR_ARG;
        }
        cudaError_t e = smem_attr(cells_kernel<KIND>, shm);
        if (e != cudaSuccess) return cuda_fail(e, what);
    }
    cells_kernel<KIND><<<(unsigned)blocks, CELL_NT, shm, s>>>(grid_of(b), jobs, ncell, b->h + 1.0, k, mode, rule_of(b), rkd);
    return cuda_fail(cudaGetLastError(), what);
}

static void add_job(MomentJobs &jobs, double *out, int full, int deriv, int k, double hp)
{
    if (!out) return;
    MomentJob w{};
    w.out = out; w.full = full; w.deriv = deriv; w.k = k; w.hp = hp;
    jobs.j[jobs.n++] = w;
}

int launch_rk_moments(const bsrg_basis *b, int k, double *rkd1, double *rkd2, double *rkd, cudaStream_t s)
{
    const int ks = b->ks, ik = ik_of(ks);
    const double q = 1.0 + b->h;
    MomentJobs jobs{};
    add_job(jobs, rkd1, 0, 0, k, ipow_host(q, k) * q);
    add_job(jobs, rkd2, 0, 0, -(k + 1), ipow_host(q, -(k + 1)) * q);
    const size_t shm = sizeof(double) * ((size_t)ks * ks * ks + ks * ks + 2 * (size_t)ks * ik + (size_t)ik * ik);
    return launch_cells<CELL_RK>(b, jobs, k, 0, rkd, shm, "rk_moments", s);
}

// N^k (sym = 0) or M^k (sym = 1) moments: the same moments, M^k symmetrises the diagonal cells
int launch_nkmk_moments(const bsrg_basis *b, int k, int sym, double *rkd1, double *rkd2, double *rkd,
                        cudaStream_t s)
{
    const int ks = b->ks, ik = ik_of(ks);
    const double q = 1.0 + b->h;
    MomentJobs jobs{};
    add_job(jobs, rkd1, 0, 0, k, ipow_host(q, k) * q);
    add_job(jobs, rkd2, 0, 0, -(k + 3), ipow_host(q, -(k + 3)) * q);
    const size_t shm = sizeof(double) * ((size_t)ks * ks * ks + ks * ks + (size_t)ks * ik + (sym ? (size_t)ik * ik : 0));
    return launch_cells<CELL_NK>(b, jobs, k, sym, rkd, shm, sym ? "mk_moments" : "nk_moments", s);
}

int launch_tk_moments(const bsrg_basis *b, int k, double *rkd1, double *rkd2, double *rkd, cudaStream_t s)
{
    const int ks = b->ks, jk = ks * ks;
    const double q = 1.0 + b->h;
    // dir 'd': the scaling law of the moments carries no extra (1+h) (moments.f90)
    MomentJobs jobs{};
    add_job(jobs, rkd1, 1, 1, k, ipow_host(q, k));
    add_job(jobs, rkd2, 1, 1, -(k + 1), ipow_host(q, -(k + 1)));
    const size_t shm = sizeof(double) * (3 * (size_t)ks * ks * ks + 2 * (size_t)ks * ks + (size_t)jk * jk);
    return launch_cells<CELL_TK>(b, jobs, k, 0, rkd, shm, "tk_moments", s);
}

// mode 0: V^k (vk_moments.f90); mode 1: W^k (wk_moments.f90); mode 2: Q^k (qk_moments.f90: rkd1, rkd2 over
// all ks*ks pairs)
int launch_vw_moments(const bsrg_basis *b, int k, int mode, double *rkd1, double *rkd2, double *rkd3, double *rkd4,
                      double *rkd, cudaStream_t s)
{
    const int ks = b->ks;
    const double q = 1.0 + b->h;
    MomentJobs jobs{};
    add_job(jobs, rkd1, mode == 2, 0, k + 1, ipow_host(q, k + 1) * q);
    add_job(jobs, rkd2, mode == 2, 0, -(k + 2), ipow_host(q, -(k + 2)) * q);
    add_job(jobs, rkd3, 1, 1, k, ipow_host(q, k));
    if (rkd3 && mode) {
        MomentJob &w = jobs.j[jobs.n - 1];
        w.combine = 1; w.minus = 0; w.k2 = k - 1; w.hp2 = ipow_host(q, k - 1) * q; w.c = (double)(k + 2);
    }
    add_job(jobs, rkd4, 1, 1, -(k + 3), ipow_host(q, -(k + 3)));
    if (rkd4 && mode) {
        MomentJob &w = jobs.j[jobs.n - 1];
        w.combine = 1; w.minus = 1; w.k2 = -(k + 4); w.hp2 = ipow_host(q, -(k + 4)) * q; w.c = (double)(k + 1);
    }
    const size_t shm = sizeof(double) * (4 * (size_t)ks * ks * ks + 2 * (size_t)ks * ks);
    return launch_cells<CELL_VK>(b, jobs, k, mode, rkd, shm, mode == 2 ? "qk_moments" : mode ? "wk_moments" : "vk_moments",
                                 s);
}

}  // namespace bsrg
