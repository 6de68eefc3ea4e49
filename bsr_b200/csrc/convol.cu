// density, convol and SUM_AmB of the reference's B-spline library on the GPU.
//
//   density (density.f90:2)  -> density_kernel
//   convol  (convol.f90:2)   -> direct_convol_kernel (icase 1,2), exchange_convol_kernel (icase 3,4)
//   SUM_AmB (sum_amb.f90:2)  -> sum_amb_kernel
//
// convol's exchange cases scatter each rkb element into up to four places of
// the result.  Here every output element gathers its contributions instead,
// which needs no atomics and is deterministic: with R(x,x',y,y') the R^k
// integral of the electron-1 pair (x,x') and electron-2 pair (y,y'),
//   icase 3:  a(x , y') = sum_{x',y} R(x,x',y,y') d(x',y)
//   icase 4:  a(x', y ) = sum_{x,y'} R(x,x',y,y') d(x,y')
// where R is read from rkb through the storage map of each electron: 's'
// (symmetric, rkb(min, ., |x-x'|+1, .)) or 'n' (rkb(x, ., x'-x+ks, .)).
// The direct cases (a band result) and SUM_AmB keep the reference's summation order.  Compiled with --fmad=false.
#include "bsrg_internal.h"

namespace bsrg {

__global__ void density_kernel(int ns, int ks, double *d, const double *__restrict__ p1,
                               const double *__restrict__ p2, char type)
{
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (type == 's') {
        if (tid >= ns * ks) return;
        int i = tid % ns, j = tid / ns;
        double v = 0.0;
        if (j == 0) v = p1[i] * p2[i];
        else if (i < ns - j) v = p1[i] * p2[i + j] + p1[i + j] * p2[i];
        d[i + (size_t)ns * j] = v;
    } else if (type == 'n') {
        int k2 = 2 * ks - 1;
        if (tid >= ns * k2) return;
        int i = tid % ns, j = tid / ns;          // 0-based row, column (column j+1 in Fortran)
        int jj = i + j + 1 - ks;                 // partner index i + (j+1) - ks (0-based)
        double v = 0.0;
        if (jj >= 0 && jj < ns) v = p1[i] * p2[jj];
        d[i + (size_t)ns * j] = v;
    } else {
        if (tid >= ns * ns) return;
        int i = tid % ns, j = tid / ns;
        d[i + (size_t)ns * j] = p1[i] * p2[j];
    }
}

// band geometry: column c (0-based) of a band of storage 's' holds rows
// 0..ns-1-c; of storage 'n' holds rows max(0,ks-1-c)..min(ns-1, ns-1+ks-1-c)
__device__ __forceinline__ void band_rows(char sym, int ns, int ks, int c, int &lo, int &hi)
{
    if (sym == 's') { lo = 0; hi = ns - 1 - c; }
    else {
        lo = ks - 1 - c; if (lo < 0) lo = 0;
        hi = ns - 1 + ks - 1 - c; if (hi > ns - 1) hi = ns - 1;
    }
}

// icase 1: a(o,op) over band(sym_i) = sum over band(sym_j) (jp outer, j inner) d(j,jp) rkb(o,j,op,jp)
// icase 2: a(o,op) over band(sym_j) = sum over band(sym_i) (ip outer, i inner) d(i,ip) rkb(i,o,ip,op)
//
// What bounds it: each output is one chain of ns (ks or 2 ks - 1) dependent, separately rounded adds, and
// with a thread that loads, multiplies and adds, each add waits for its loads.  A CTA has DC_O outputs of
// one column; its other warps form the products of the next DC_Q terms in shared memory while warp 0 adds
// the last ones, a lane per output.  Terms outside the band are staged as zeros, which change no sum.
// Measured at ks = 10, ns = 200, 's', 's': 132 -> 29 us
constexpr int DC_O = 16, DC_Q = 128, DC_NT = 256;

__global__ void __launch_bounds__(DC_NT) direct_convol_kernel(int ns, int ks, int ldp, int icase, char si, char sj,
                                                              double *a, const double *__restrict__ d,
                                                              const double *__restrict__ rkb)
{
    __shared__ double prod[2][DC_Q][DC_O + 1];
    const char so = icase == 1 ? si : sj;      // output band storage
    const char sc = icase == 1 ? sj : si;      // contracted band storage
    const int ncc = sc == 's' ? ks : 2 * ks - 1, o0 = blockIdx.x * DC_O, op = blockIdx.y;
    const int total = ncc * ns, tiles = (total + DC_Q - 1) / DC_Q;
    const size_t nn = (size_t)ns * ns;
    auto fill = [&](int tile, int t0, int nt) {
        double (*p)[DC_O + 1] = prod[tile & 1];
        constexpr int PER = (DC_Q * DC_O + DC_NT - 33) / (DC_NT - 32);
        double x[PER], y[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int e = t0 + u * nt;
            const int q = icase == 1 ? e / DC_O : e % DC_Q, ol = icase == 1 ? e % DC_O : e / DC_Q, o = o0 + ol;
            const int s = tile * DC_Q + q, cp = s / ns, c = s - cp * ns;
            x[u] = y[u] = 0.0;
            if (e < DC_Q * DC_O && s < total && o < ns) {
                int lo, hi;
                band_rows(sc, ns, ks, cp, lo, hi);
                if (c >= lo && c <= hi) {
                    x[u] = d[s];
                    y[u] = rkb[icase == 1 ? o + (size_t)ns * c + nn * (op + (size_t)ldp * cp)
                                          : c + (size_t)ns * o + nn * (cp + (size_t)ldp * op)];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int e = t0 + u * nt;
            if (e < DC_Q * DC_O)
                p[icase == 1 ? e / DC_O : e % DC_Q][icase == 1 ? e % DC_O : e / DC_Q] = x[u] * y[u];
        }
    };
    const int tid = threadIdx.x;
    if (tid >= 32) fill(0, tid - 32, DC_NT - 32);
    __syncthreads();
    double c = 0.0;
    for (int t = 0; t < tiles; t++) {
        if (tid >= 32) {
            if (t + 1 < tiles) fill(t + 1, tid - 32, DC_NT - 32);
        } else if (tid < DC_O) {
#pragma unroll 16
            for (int q = 0; q < DC_Q; q++) c = c + prod[t & 1][q][tid];
        }
        __syncthreads();
    }
    if (tid < DC_O && o0 + tid < ns) {
        int lo, hi;
        band_rows(so, ns, ks, op, lo, hi);
        if (o0 + tid >= lo && o0 + tid <= hi) a[o0 + tid + (size_t)ns * op] = c;   // the others stay untouched
    }
}

// map an electron pair (x, x') to (stored row, stored column index) of rkb;
// returns false if the pair has no entry.
__device__ __forceinline__ bool pair_map(char sym, int ns, int ks, int x, int xp, int &row, int &col)
{
    int dx = xp - x;
    if (dx <= -ks || dx >= ks || x < 0 || xp < 0 || x >= ns || xp >= ns) return false;
    if (sym == 's') { row = dx >= 0 ? x : xp; col = dx >= 0 ? dx : -dx; }
    else { row = x; col = dx + ks - 1; }
    return true;
}

// A CTA has 32 rows u of one column v, each warp the offsets e = warp, warp + XC_E, ... of the first
// electron; the warps' sums are added in a fixed order.  A row of 2 ks - 1 offsets f is one
// batch of loads (a thread per output, which waited for each pair of loads, took 108 us at ks = 10,
// ns = 200; this takes 41).
constexpr int XC_E = 8;

__global__ void __launch_bounds__(32 * XC_E) exchange_convol_kernel(int ns, int ks, int ldp, int icase, char si, char sj,
                                                                    double *a, const double *__restrict__ d,
                                                                    const double *__restrict__ rkb)
{
    __shared__ double part[XC_E][32];
    const int u = blockIdx.x * 32 + threadIdx.x, v = blockIdx.y, w = threadIdx.y;     // output a(u, v)
    const size_t nn = (size_t)ns * ns;
    double c = 0.0;
    for (int e = w - (ks - 1); e <= ks - 1; e += XC_E) {
        // icase 3: a(x,y') <- d(x',y) with x = u, y' = v; icase 4: a(x',y) <- d(x,y') with x' = u, y = v
        const int x = icase == 3 ? u : u + e, xp = icase == 3 ? u + e : u;
        int r1, c1;
        if (!pair_map(si, ns, ks, x, xp, r1, c1)) continue;
        const int xd = icase == 3 ? xp : x;
        const double *rk = rkb + r1 + nn * c1;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 10
        for (int f = -(ks - 1); f <= ks - 1; f += 2) {
            double rv[2], dv[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int y = icase == 3 ? v + f + q : v, yp = icase == 3 ? v : v + f + q, yd = v + f + q;
                int r2 = 0, c2 = 0;
                const bool ok = f + q <= ks - 1 && pair_map(sj, ns, ks, y, yp, r2, c2);
                rv[q] = ok ? __ldg(rk + (size_t)ns * r2 + nn * ((size_t)ldp * c2)) : 0.0;
                dv[q] = ok ? __ldg(d + xd + (size_t)ns * yd) : 0.0;
            }
            s0 = s0 + rv[0] * dv[0];
            s1 = s1 + rv[1] * dv[1];
        }
        c = c + (s0 + s1);
    }
    part[w][threadIdx.x] = c;
    __syncthreads();
    if (w == 0 && u < ns) {
        for (int q = 1; q < XC_E; q++) c = c + part[q][threadIdx.x];
        a[u + (size_t)ns * v] = c;
    }
}

// SUM(a*b) over the storage mode, one ordered chain of adds: 'x' row by row, the bands column by
// column.  The other warps form the products of the next SA_CHUNK terms in shared memory while one
// thread adds the last ones; terms outside a band are staged as zeros, which change no sum.
// Measured at ks = 10, ns = 200: 'x' (40000 terms) 1280 -> 200 us, ten cycles an add; 's' 66 -> 12 us
constexpr int SA_CHUNK = 2048, SA_NT = 512;

__global__ void __launch_bounds__(SA_NT) sum_amb_kernel(int ns, int ks, const double *__restrict__ a,
                                                        const double *__restrict__ b, char sym, double *out)
{
    __shared__ __align__(16) double prod[2][SA_CHUNK];
    const long total = (long)ns * (sym == 'x' ? ns : sym == 'n' ? 2 * ks - 1 : ks);
    const int chunks = (int)((total + SA_CHUNK - 1) / SA_CHUNK), tid = threadIdx.x;
    auto fill = [&](int chunk) {
        constexpr int NT = SA_NT - 32, PER = (SA_CHUNK + NT - 1) / NT;
        double x[PER], y[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int e = tid - 32 + u * NT;
            const long s = (long)chunk * SA_CHUNK + e;
            x[u] = y[u] = 0.0;
            if (e < SA_CHUNK && s < total) {
                const int g = (int)(s / ns), k = (int)(s - (long)g * ns);
                bool in = true;
                if (sym == 's') in = k < ns - g;
                else if (sym == 'l') in = k >= ks - 1 - g;
                else if (sym == 'n') in = k >= ks - 1 - g && k < ns + ks - 1 - g;
                const size_t at = sym == 'x' ? g + (size_t)ns * k : (size_t)s;
                if (in) { x[u] = a[at]; y[u] = b[at]; }
            }
        }
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int e = tid - 32 + u * NT;
            if (e < SA_CHUNK) prod[chunk & 1][e] = x[u] * y[u];
        }
    };
    if (tid >= 32) fill(0);
    __syncthreads();
    double x = 0.0;
    for (int c = 0; c < chunks; c++) {
        if (tid >= 32) {
            if (c + 1 < chunks) fill(c + 1);
        } else if (tid == 0) {
            const double2 *p = (const double2 *)prod[c & 1];
            const int n2 = (int)(min((long)SA_CHUNK, total - (long)c * SA_CHUNK) + 1) / 2;
#pragma unroll 16
            for (int q = 0; q < n2; q++) {
                const double2 v = p[q];
                x = x + v.x;
                x = x + v.y;
            }
        }
        __syncthreads();
    }
    if (tid == 0) *out = x;
}

int launch_density(int ns, int ks, double *d, const double *p1, const double *p2, char type, cudaStream_t s)
{
    int n = type == 's' ? ns * ks : (type == 'n' ? ns * (2 * ks - 1) : ns * ns);
    density_kernel<<<(n + 127) / 128, 128, 0, s>>>(ns, ks, d, p1, p2, type);
    return cuda_fail(cudaGetLastError(), "density");
}

int launch_convol(int ns, int ks, double *a, const double *d, const double *rkb, int ldp, int icase, char si,
                  char sj, cudaStream_t s)
{
    if (icase == 1 || icase == 2) {
        const char so = icase == 1 ? si : sj;
        const dim3 grd((ns + DC_O - 1) / DC_O, so == 's' ? ks : 2 * ks - 1);
        direct_convol_kernel<<<grd, DC_NT, 0, s>>>(ns, ks, ldp, icase, si, sj, a, d, rkb);
    } else {
        exchange_convol_kernel<<<dim3((ns + 31) / 32, ns), dim3(32, XC_E), 0, s>>>(ns, ks, ldp, icase, si, sj, a, d, rkb);
    }
    return cuda_fail(cudaGetLastError(), "convol");
}

int launch_sum_amb(int ns, int ks, const double *a, const double *b, char sym, double *out, cudaStream_t s)
{
    sum_amb_kernel<<<1, SA_NT, 0, s>>>(ns, ks, a, b, sym, out);
    return cuda_fail(cudaGetLastError(), "sum_amb");
}

// bav (bav.f90:2): y = B v ('s'; 'n' with side 'r') or y = v B ('n', side 'l').  One thread
// per output, the terms added in the order the reference's scatter loops reach that output
// (for 's': within each diagonal ip the transposed term b(x-ip+1, ip) v(x-ip+1) comes first).
__global__ void bav_kernel(int ns, int ks, const double *__restrict__ b, const double *__restrict__ v, double *y,
                           char type, char side)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;   // 0-based output index
    if (x >= ns) return;
    double acc;
    if (type == 's') {
        acc = b[x] * v[x];
        for (int ip = 2; ip <= ks; ip++) {
            const int i1 = x - ip + 1;            // row i whose j = i + ip - 1 is x
            if (i1 >= 0) acc = acc + b[i1 + (size_t)ns * (ip - 1)] * v[i1];
            if (x <= ns - ip) acc = acc + b[x + (size_t)ns * (ip - 1)] * v[x + ip - 1];
        }
    } else {
        acc = 0.0;
        for (int ip = 1; ip <= ks + ks - 1; ip++) {
            const int imin = max(1, 1 + ks - ip), imax = min(ns, ns + ks - ip);
            if (side == 'r') {
                const int i = x + 1, j = i + ip - ks;
                if (i >= imin && i <= imax) acc = acc + b[(i - 1) + (size_t)ns * (ip - 1)] * v[j - 1];
            } else {
                const int i = x + 1 - ip + ks;     // j = i + ip - ks = x + 1
                if (i >= imin && i <= imax) acc = acc + b[(i - 1) + (size_t)ns * (ip - 1)] * v[i - 1];
            }
        }
    }
    y[x] = acc;
}

// bvmv (bvmv.f90:2): <x, A y> for a band array, in the reference's summation order
// (one thread: the sum is a single ordered accumulation of O(n k) terms)
__device__ double bvmv_dev(int n, int k, const double *ar, char type, const double *x, const double *y)
{
    double s = 0.0;
    if (type != 'g') {
        for (int jp = 1; jp <= k - 1; jp++)
            for (int i = k + 1 - jp; i <= n; i++) {
                const int j = i + jp - k;
                s = s + ar[(i - 1) + (size_t)n * (jp - 1)] * (x[i - 1] * y[j - 1] + x[j - 1] * y[i - 1]);
            }
        if (type == 'a') s = s + x[n - 2] * y[n - 1] * (ar[0] - ar[(n - 1) + (size_t)n * (k - 2)]);
    } else {
        for (int jp = 1; jp <= k - 1; jp++)
            for (int i = k - jp + 1; i <= n; i++) {
                const int j = i + jp - k, kp = 2 * k - jp;
                s = s + ar[(i - 1) + (size_t)n * (jp - 1)] * x[i - 1] * y[j - 1];
                s = s + ar[(j - 1) + (size_t)n * (kp - 1)] * x[j - 1] * y[i - 1];
            }
    }
    double c = 0.0;
    for (int i = 1; i <= n; i++) c = c + ar[(i - 1) + (size_t)n * (k - 1)] * x[i - 1] * y[i - 1];
    return s + c;
}

__global__ void bvmv_kernel(int n, int k, const double *ar, char type, const double *x, const double *y, double *out)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) *out = bvmv_dev(n, k, ar, type, x, y);
}

int launch_bav(int ns, int ks, const double *b, const double *v, double *y, char type, char side, cudaStream_t s)
{
    bav_kernel<<<(ns + 127) / 128, 128, 0, s>>>(ns, ks, b, v, y, type, side);
    return cuda_fail(cudaGetLastError(), "bav");
}

int launch_bvmv(int n, int k, const double *ar, char type, const double *x, const double *y, double *out,
                cudaStream_t s)
{
    bvmv_kernel<<<1, 32, 0, s>>>(n, k, ar, type, x, y, out);
    return cuda_fail(cudaGetLastError(), "bvmv");
}

}  // namespace bsrg
