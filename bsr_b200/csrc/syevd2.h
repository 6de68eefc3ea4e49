// Shared by the parts of the two-stage symmetric eigensolver (syevd2.cu, bulge.cu).
#pragma once
#include <cuda_runtime.h>

namespace bsrg {

constexpr int NB = 32;              // bandwidth of the intermediate band matrix
constexpr int LDAB = 2 * NB;        // rows of the band storage: the band and room for the bulges
constexpr unsigned long long WAIT_NS = 2000000000ull;   // bound of every device-side wait (2 s)

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// reflectors of sweep j of the bulge chasing
__host__ __device__ __forceinline__ int sweep_steps(int n, int j) { return j <= n - 3 ? (n - 3 - j) / NB + 1 : 0; }

// stage 2 (bulge.cu).  band_extract: the band of A (its NB subdiagonals) into AB, 2 LDAB n doubles;
// bulge_chase: AB to tridiagonal form, d (n) and e (n-1), one cooperative kernel.  Reflector i of
// sweep j goes to V2[((long)j S + i) NB ..] and tau2[(long)j S + i].  *err (zero on entry) is set to
// 2 if a wait runs out.
int band_extract(int n, const double *A, long lda, double *AB, cudaStream_t s);
int bulge_chase(int n, double *AB, double *d, double *e, double *V2, double *tau2, int S, int *err, int nsm,
                cudaStream_t s);

}  // namespace bsrg
