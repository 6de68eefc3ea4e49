// FP64 tensor-core GEMM core for sm_100a: mma.sync.aligned.m8n8k4 f64 (DMMA).
//
// FP64 has no tcgen05 kind, so the FP64 tensor pipe is reached through the
// warp-level m8n8k4 f64 MMA.  A CTA computes a BM x BN tile of
// C = op(A) op(B) with WM x WN warps, each warp a (BM/WM) x (BN/WN) sub-tile of
// 8 x 8 MMA tiles.  K advances in steps of 16 through a 3-stage cp.async
// pipeline; every operand tile is staged in shared memory in the orientation
// its global layout gives (no transposes), with a padding of 4 doubles so that
// the fragment loads of each half-warp hit 16 distinct 8-byte bank slots.
// Shapes: 64 x 64 (4 warps, 32 x 32 each, three to four CTAs per SM) for square work, 128 x 32 and
// 32 x 128 (4 warps, 32 x 32 each) for the panel products of the eigensolver.  Several small
// CTAs fill one another's barriers, prologues and epilogues, and leave a shorter last wave: at
// 7810^3, 2000 x 820 x 2000 and 1700^3 a 128 x 128 tile of 8 warps took 28.5, 0.272 and 0.464 ms, the
// 64 x 64 one 27.2, 0.217 and 0.301 (34.6, 0.346 and 0.590 with the slices' copies issued together
// after the barrier); cuBLAS measures 35.5 TFLOP/s where this is at 35.0.
//
// Fragment layouts of m8n8k4 f64 (row.col): A 8x4 -- lane holds A[lane>>2][lane&3];
// B 4x8 -- lane holds B[lane&3][lane>>2]; C 8x8 -- lane holds C[lane>>2][2(lane&3)+{0,1}].
//
// All matrices are column-major (Fortran).  op(A) is M x K: A (lda >= M) when
// TA is false, A^T of a K x M array when TA is true; likewise op(B) is K x N.
#pragma once
#include <cuda_runtime.h>

namespace bsrg {
namespace dmma {

constexpr int BK = 16, STAGES = 3, PAD = 4;

template <int BM_, int BN_, int WM_, int WN_> struct Cfg {
    static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_;
    static constexpr int NT = 32 * WM * WN;
    static constexpr int TM = BM / WM, TN = BN / WN;     // warp tile
    static constexpr int FM = TM / 8, FN = TN / 8;       // MMA tiles per warp
    static_assert(TM % 8 == 0 && TN % 8 == 0, "warp tile of whole 8x8 MMA tiles");
    static_assert((BM * BK) % NT == 0 && (BN * BK) % NT == 0, "whole loads per thread");
};
using Sq = Cfg<64, 64, 2, 2>;     // 128 threads
using Tall = Cfg<128, 32, 4, 1>;  // 128 threads
using Wide = Cfg<32, 128, 1, 4>;  // 128 threads

template <class C, bool TA> struct ALayout {
    // !TA: As[k][m] (m contiguous), TA: As[m][k] (k contiguous)
    static constexpr int ELEMS = TA ? C::BM * (BK + PAD) : BK * (C::BM + PAD);
};
template <class C, bool TB> struct BLayout {
    // !TB: Bs[n][k] (k contiguous), TB: Bs[k][n] (n contiguous)
    static constexpr int ELEMS = TB ? BK * (C::BN + PAD) : C::BN * (BK + PAD);
};
template <class C, bool TA, bool TB, bool SYMA = false> struct Smem {
    static constexpr int STAGE = ALayout<C, TA>::ELEMS + BLayout<C, TB>::ELEMS;
    static constexpr int BYTES = SYMA ? STAGES * 8 * (ALayout<C, true>::ELEMS + BLayout<C, TB>::ELEMS) : STAGES * STAGE * 8;
};

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem, bool valid)
{
    unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    int bytes = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void mma884(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// One operand's share of the staging of a BK slice by a thread: N copies, spread over the slice's four
// MMA steps.  CONTIG elements of the tile are contiguous in memory (m for a column-major A, k for A^T),
// and a thread's copies differ only along the other index, so a copy costs one pointer addition.
// Outside the matrix and outside [k0, kend) zeros are staged.
template <int TILE, bool KFAST, int NT> struct Stager {
    static constexpr int N = TILE * BK / NT;
    static constexpr int STEP = KFAST ? NT / BK : NT / TILE;        // tile (or k) indices between two copies
    static_assert(KFAST ? NT % BK == 0 : NT % TILE == 0, "a thread keeps its contiguous index");
    static_assert(N % 4 == 0, "whole copies per MMA step");
    static constexpr int LD = KFAST ? BK + PAD : TILE + PAD;
    const double *p, *base;
    long ld, stride;
    int kl, left, dst;               // first k of this thread in the slice; tile indices it may read (from its first)
    __device__ __forceinline__ Stager(const double *A, long ld_, int size, int t0, int kbeg, int tid)
    {
        const int tl = KFAST ? tid / BK : tid % TILE;
        kl = KFAST ? tid % BK : tid / TILE;
        left = size - t0 - tl;
        base = A;
        ld = ld_;
        stride = STEP * ld;
        p = A + (KFAST ? (kbeg + kl) + (long)(t0 + tl) * ld : (t0 + tl) + (long)(kbeg + kl) * ld);
        dst = KFAST ? tl * LD + kl : kl * LD + tl;
    }
    // copies q N / 4 .. of the slice with krem k indices left
    __device__ __forceinline__ void part(double *s, int q, int krem) const
    {
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const int c = q * (N / 4) + i;
            const bool v = KFAST ? (kl < krem && c * STEP < left) : (left > 0 && kl + c * STEP < krem);
            cp_async8(s + dst + c * STEP * LD, v ? p + c * stride : base, v);
        }
    }
    __device__ __forceinline__ void advance() { p += KFAST ? BK : BK * ld; }
};

// The same for the diagonal tiles of a square symmetric A of which only the lower triangle is stored (tile_mma
// takes the others as they are or transposed): element (m, k) is read from (max, min).
template <int TILE, int NT> struct SymStager {
    static constexpr int N = TILE * BK / NT, LD = TILE + PAD;
    const double *base;
    long ld;
    int size, t0, k0, tid;
    __device__ __forceinline__ SymStager(const double *A, long ld_, int size_, int t0_, int kbeg, int tid_)
        : base(A), ld(ld_), size(size_), t0(t0_), k0(kbeg), tid(tid_)
    {
    }
    __device__ __forceinline__ void part(double *s, int q, int krem) const
    {
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const int idx = tid + (q * (N / 4) + i) * NT;
            const int tl = idx % TILE, kl = idx / TILE;
            const int gm = t0 + tl, gk = k0 + kl;
            const bool v = gm < size && kl < krem;
            cp_async8(s + kl * LD + tl, v ? (gm >= gk ? base + gm + (long)gk * ld : base + gk + (long)gm * ld) : base, v);
        }
    }
    __device__ __forceinline__ void advance() { k0 += BK; }
};
template <class C, bool TA, bool SYMA> struct AStager { using T = Stager<C::BM, TA, C::NT>; };
template <class C, bool TA> struct AStager<C, TA, true> { using T = SymStager<C::BM, C::NT>; };

// acc[s][t][j]: row m0 + wm*TM + s*8 + (lane>>2), column n0 + wn*TN + t*8 + 2*(lane&3) + j,
// summed over k in [kbeg, kend).  The copies of the slice after next are issued a quarter at a time
// between the MMA steps (issued together after the barrier they left the tensor pipe idle: both warps of a
// scheduler were in them at once), and a step's fragments are read while the last one's MMAs run.
template <class C, bool TA, bool TB, bool SYMA = false>
__device__ __forceinline__ void tile_mma_add(double (&acc)[C::FM][C::FN][2], double *smem, const double *A, long lda,
                                         const double *B, long ldb, int M, int N, int kbeg, int kend, int m0, int n0)
{
    constexpr int SA = ALayout<C, TA>::ELEMS, STG = Smem<C, TA, TB>::STAGE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp % C::WM, wn = warp / C::WM;
    const int r = lane >> 2, c = lane & 3;
    if (kend <= kbeg) return;
    const int ktiles = (kend - kbeg + BK - 1) / BK;
    typename AStager<C, TA, SYMA>::T la(A, lda, M, m0, kbeg, threadIdx.x);
    Stager<C::BN, !TB, C::NT> lb(B, ldb, N, n0, kbeg, threadIdx.x);
    int krem = kend - kbeg;
#pragma unroll
    for (int st = 0; st < STAGES - 1; st++) {
        if (st < ktiles) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                la.part(smem + st * STG, q, krem);
                lb.part(smem + st * STG + SA, q, krem);
            }
            la.advance();
            lb.advance();
            krem -= BK;
        }
        cp_async_commit();
    }
    double af[2][C::FM], bf[2][C::FN];
    auto fragments = [&](int slice, int kk) {
        const double *sA = smem + (slice % STAGES) * STG, *sB = sA + SA;
#pragma unroll
        for (int s = 0; s < C::FM; s++) {
            const int ml = wm * C::TM + s * 8 + r, kl = kk * 4 + c;
            af[kk & 1][s] = TA ? sA[ml * (BK + PAD) + kl] : sA[kl * (C::BM + PAD) + ml];
        }
#pragma unroll
        for (int t = 0; t < C::FN; t++) {
            const int nl = wn * C::TN + t * 8 + r, kl = kk * 4 + c;
            bf[kk & 1][t] = TB ? sB[kl * (C::BN + PAD) + nl] : sB[nl * (BK + PAD) + kl];
        }
    };
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    fragments(0, 0);
    for (int kt = 0; kt < ktiles; kt++) {
        const int nk = kt + STAGES - 1;
        double *next = smem + (nk % STAGES) * STG;
#pragma unroll
        for (int kk = 0; kk < BK / 4; kk++) {
            if (kk + 1 < BK / 4) fragments(kt, kk + 1);
            else {
                // every warp has read the last of this slice: the next one's first fragments before the
                // last MMAs of this one, so that the barrier is passed with MMAs still to issue
                cp_async_wait<STAGES - 3>();
                __syncthreads();
                fragments(kt + 1, 0);
            }
            if (nk < ktiles) {
                la.part(next, kk, krem);
                lb.part(next + SA, kk, krem);
            }
#pragma unroll
            for (int s = 0; s < C::FM; s++)
#pragma unroll
                for (int t = 0; t < C::FN; t++) mma884(acc[s][t][0], acc[s][t][1], af[kk & 1][s], bf[kk & 1][t]);
        }
        la.advance();
        lb.advance();
        krem -= BK;
        cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();
}

template <class C, bool TA, bool TB, bool SYMA = false>
__device__ __forceinline__ void tile_mma(double (&acc)[C::FM][C::FN][2], double *smem, const double *A, long lda,
                                         const double *B, long ldb, int M, int N, int kbeg, int kend, int m0, int n0)
{
#pragma unroll
    for (int s = 0; s < C::FM; s++)
#pragma unroll
        for (int t = 0; t < C::FN; t++) acc[s][t][0] = acc[s][t][1] = 0.0;
    if (!SYMA) {
        tile_mma_add<C, TA, TB>(acc, smem, A, lda, B, ldb, M, N, kbeg, kend, m0, n0);
    } else {
        // left of the diagonal tile A as it is stored, below it A^T: only the tile itself picks its
        // triangle element by element
        const int d0 = m0, d1 = m0 + C::BM;
        tile_mma_add<C, false, TB>(acc, smem, A, lda, B, ldb, M, N, kbeg, min(kend, d0), m0, n0);
        tile_mma_add<C, false, TB, true>(acc, smem, A, lda, B, ldb, M, N, max(kbeg, d0), min(kend, d1), m0, n0);
        tile_mma_add<C, true, TB>(acc, smem, A, lda, B, ldb, M, N, max(kbeg, d1), kend, m0, n0);
    }
}

}  // namespace dmma
}  // namespace bsrg
