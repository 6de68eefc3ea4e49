// Shared by the parts of the two-stage symmetric eigensolver (syevd2.cu, bulge.cu).
#pragma once
#include <cuda_runtime.h>

namespace bsrg {

constexpr int NB = 32;              // bandwidth of the intermediate band matrix
constexpr int LDAB = 2 * NB;        // rows of the band storage: the band and room for the bulges
// A column whose sum of squares lies below this counts as zero in the reductions (see amax_kernel in syevd2.cu)
constexpr double SMALL_SQ = 0x1p-700;
constexpr unsigned long long WAIT_NS = 2000000000ull;   // bound of every device-side wait (2 s)

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// reflectors of sweep j of the bulge chasing
__host__ __device__ __forceinline__ int sweep_steps(int n, int j) { return j <= n - 3 ? (n - 3 - j) / NB + 1 : 0; }

// stage 1 (band_reduce.cu): the lower triangle of A to a band of width NB in place.  The panels' V go to
// Vsave one after another (panel p: m_p x NB, m_p = n - (p + 1) NB, ld m_p), their T to Tsave + p NB^2 (both null:
// not kept).
struct Sy2sbWork {
    double *VYV;       // m x 3NB
    double *VYV2;      // the second [V | Y | V] buffer (panels alternate while the look-ahead runs)
    cudaStream_t aux;  // the look-ahead's second stream (null: one stream)
    cudaEvent_t ev_y, ev_c2;
    double *X;         // m x NB
    double *T;         // NB x NB
    double *Mp;        // chunks x NB x NB
    double *part;      // PQ CTAs x 4NB
    double *gram;      // PQ CTAs x NB x NB
    unsigned *bar;     // 2
    unsigned *ticket;  // ypass1's last-CTA counter (zero between panels)
    int *err;
    double *gemm_ws;   // split-K workspace
    size_t gemm_ws_doubles;
};

int sy2sb_panels(int n);
size_t sy2sb_vsave_doubles(int n);
int sy2sb(cudaStream_t st, int n, double *A, long lda, double *Vsave, double *Tsave, const Sy2sbWork &w);

// stage 2 (bulge.cu).  band_extract: the band of A (its NB subdiagonals) into AB, 2 LDAB n doubles;
// bulge_chase: AB to tridiagonal form, d (n) and e (n-1), one kernel; ticket: zero.  Reflector i of
// sweep j goes to V2[((long)j S + i) NB ..] and tau2[(long)j S + i] unless V2 is null.  *err (zero on entry) is set to
// 2 if a wait runs out.
int band_extract(int n, const double *A, long lda, double *AB, cudaStream_t s);
int bulge_chase(int n, double *AB, double *d, double *e, double *V2, double *tau2, int S, int *err, unsigned *ticket, int nsm,
                cudaStream_t s);

// back-transformation of stage 2 (q2_apply.cu): Z <- Q2 Z for the n columns of Z.  frag:
// q2_fragment_doubles(n), 16-byte aligned.  *err is set to 3 if a wait runs out.
size_t q2_fragment_doubles(int n);
double q2_flops(int n);
int q2_apply(int n, const double *V2, const double *tau2, int S, double *frag, double *Z, long ldz, int *err, int nsm,
             cudaStream_t st);

}  // namespace bsrg
