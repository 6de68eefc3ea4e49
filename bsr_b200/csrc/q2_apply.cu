// Back-transformation of the bulge chasing's reflectors (stage 2 of the two-stage eigensolver): Z <- Q2 Z.
//
// Block (g, i): the step-i reflectors of sweeps j = g NB + q, q < NB, as one compact WY factor
// I - V T V^T = H_{gNB} H_{gNB+1} ... (V's column q occupies rows q .. q + NB - 1 of the block's window of 2 NB
// rows, which starts at row (g + i) NB + 1).  Applied to Z: groups g descending, within a group blocks i
// ascending, each block's reflectors in the product order above -- the order of creation reversed up
// to commuting (disjoint) pairs.  With K = (n - 3) / NB + 1 blocks in group 0, group g has K - g, and
// chunk c, rows c NB + 1 .. (c + 1) NB, is touched by groups g <= c: every group runs through chunks g .. K.
#include <algorithm>

#include "bsrg_internal.h"
#include "dmma.cuh"
#include "syevd2.h"

namespace bsrg {
namespace {

constexpr int NF_A = 20, NF_B = 26;                          // fragment pairs of V and of V T per block
constexpr int FRAG_A = NF_A * 32, FRAG_B = NF_B * 32;        // in double2
constexpr int Q2_GMAX = 4;                                   // groups in flight in a CTA
constexpr int Q2_P = 4;                                      // warps (parts of the strip) per group
constexpr int Q2_BUF = 2;                                    // blocks of fragments per group
constexpr int Q2_TMAX = 7;                                   // 8-column tiles of a strip (shared memory)

// first fragment pair of V T for row tile rt: pairs t = max(0, rt - 4) .. 3
__host__ __device__ constexpr int fragb_at(int rt) { return rt <= 4 ? 4 * rt : rt == 5 ? 20 : rt == 6 ? 23 : 25; }
__host__ __device__ constexpr int fragb_t0(int rt) { return rt <= 4 ? 0 : rt - 4; }

__host__ __device__ __forceinline__ int q2_blocks0(int n) { return (n - 3) / NB + 1; }          // K
__host__ __device__ __forceinline__ size_t q2_block_at(int K, int g) { return (size_t)g * K - (size_t)g * (g - 1) / 2; }

// The fragments of every block, in the order and lane layout q2_apply_kernel reads them (see there):
//   pair (t, i) of V, i < 5:  V(8 (t + i) + 2 c + e, 8 t + r), e = 0, 1
//   pair (rt, t) of -V T:    -(V T)(8 rt + r, 8 t + 2 c + e)
// with lane = 4 r + c.  One CTA per block.
__global__ void __launch_bounds__(128) q2_fragment_kernel(int n, int S, const double *__restrict__ V2,
                                                          const double *__restrict__ tau2, double2 *__restrict__ F)
{
    // G = V^T V is through when U = -V T is formed in its place
    __shared__ double V[2 * NB][NB + 1], U[2 * NB][NB + 1], T[NB][NB + 1], tau[NB];
    double (*G)[NB + 1] = U;
    const int g = blockIdx.y, i = blockIdx.x, tid = threadIdx.x, K = q2_blocks0(n);
    if (i >= K - g) return;
    for (int e = tid; e < 2 * NB * (NB + 1); e += 128) (&V[0][0])[e] = 0.0;
    __syncthreads();
    for (int e = tid; e < NB * NB; e += 128) {
        const int q = e / NB, t = e % NB, j = g * NB + q;
        const bool in = j < n - 2 && i < sweep_steps(n, j);
        if (in) V[t + q][q] = V2[((long)j * S + i) * NB + t];
        if (t == 0) tau[q] = in ? tau2[(long)j * S + i] : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < NB * NB; e += 128) {
        const int a = e / NB, b = e % NB;
        double s = 0.0;
        if (a < b)
            for (int r = b; r < a + NB; r++) s = fma(V[r][a], V[r][b], s);
        G[a][b] = s;
        T[a][b] = 0.0;
    }
    __syncthreads();
    if (tid < NB) {
        // T(:, c) = -tau_c T(:, 0:c) G(0:c, c), T(c, c) = tau_c; row tid
        for (int c = 0; c < NB; c++) {
            double s0 = 0.0, s1 = 0.0;
            int l = tid;
            for (; l + 1 < c; l += 2) {
                s0 = fma(T[tid][l], G[l][c], s0);
                s1 = fma(T[tid][l + 1], G[l + 1][c], s1);
            }
            if (l < c) s0 = fma(T[tid][l], G[l][c], s0);
            T[tid][c] = tid < c ? -tau[c] * (s0 + s1) : (tid == c ? tau[c] : 0.0);
        }
    }
    __syncthreads();
    for (int e = tid; e < 2 * NB * NB; e += 128) {
        const int r = e / NB, q = e % NB;
        double s = 0.0;
        for (int l = max(0, r - NB + 1); l <= min(q, r); l++) s = fma(V[r][l], T[l][q], s);
        U[r][q] = -s;
    }
    __syncthreads();
    double2 *out = F + (q2_block_at(K, g) + i) * (FRAG_A + FRAG_B);
    for (int e = tid; e < FRAG_A; e += 128) {
        const int p = e >> 5, lane = e & 31, r = lane >> 2, c = lane & 3, t = p / 5, rt = t + p % 5;
        out[e] = rt < 8 ? make_double2(V[8 * rt + 2 * c][8 * t + r], V[8 * rt + 2 * c + 1][8 * t + r])
                        : make_double2(0.0, 0.0);
    }
    for (int e = tid; e < FRAG_B; e += 128) {
        const int p = e >> 5, lane = e & 31, r = lane >> 2, c = lane & 3;
        const int rt = p < 20 ? p / 4 : p < 23 ? 5 : p < 25 ? 6 : 7, t = fragb_t0(rt) + p - fragb_at(rt);
        out[FRAG_A + e] = make_double2(U[8 * rt + r][8 * t + 2 * c], U[8 * rt + r][8 * t + 2 * c + 1]);
    }
}

// ---- the application ----
//
// What bounds it: the FP64 tensor pipe, if nothing else is let in its way.  The products are taken on Z^T:
// the accumulator layout of an 8 x 8 tile (column 4 r + c's row: rows 2 c, 2 c + 1 of the tile) is then
// also the layout of an A operand whose k index c stands for those two rows, so a warp's window of Z,
// and W^T between the two products, never leave its registers; V and -V T come as B operands in
// fragment order, prepared once per block by q2_fragment_kernel.  T is multiplied into V there: 92 MMAs per
// block and eight columns against 100 for V^T Z, T W and V W, and one product less in the chain.
//
// A CTA has a strip of columns and G groups in flight, four warps each (one or two 8-column tiles a warp); slot p works one chunk of 32 rows behind slot p - 1 and takes its finished chunks through a link
// of two chunks in shared memory, a register image per lane.  Slot 0 copies chunks of Z ahead
// asynchronously, the last slot stores them, and slot 0 goes on to the next G groups as soon as the
// chunks it needs are stored: Z crosses HBM once per G groups.  The fragments of the block after next
// come by bulk copies issued by whichever of the slot's warps is the last to finish with the buffer.  (Four
// groups with two warps each and one buffer: 63.9 ms at n = 7810, the loads were not early enough.)
// The strip's width is T tiles, the warps with one tile less on another scheduler in each slot.  A slot's
// block takes about 1390 T cycles, but never less than 4400 (T = 2: a take, two products and a pass that
// depend on one another), so T minimises waves times max(T, 3.2); at T = 2, where the chain and not the
// tensor pipe is the limit and the links are small, G = 4, else 3.
// Measured (n = 7810, 5800, 4400, 1713): 102.7, 58.7, 17.5, 2.9 ms with V, T and Z in shared memory, three
// products and a barrier of two warps between them; 50.8, 22.0, 9.9, 1.07 ms so (27 TFLOP/s executed at 7810).
struct Q2Shared {
    unsigned long long full[Q2_GMAX][2][Q2_BUF];    // mbarriers: slot, operand (V, V T), buffer
    int used[Q2_GMAX][2][Q2_BUF];                   // warps of the slot that have finished with it
    int made[Q2_GMAX][Q2_P];                        // chunks a slot's part has passed on: round (K + 2) + k + 1
    int taken[Q2_GMAX][Q2_P];                       // chunks it has taken from the slot before it
    int dead;
};

struct Q2Args {
    int n, ncol, K, rounds;
    const double2 *F;
    double *Z;
    long ldz;
    int *err;
};

__device__ __forceinline__ unsigned saddr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(saddr(dst)),
                 "l"(src), "r"(bytes), "r"(saddr(bar))
                 : "memory");
}

// bounded waits: once one has run out, dead is set and the others return at once
__device__ __forceinline__ bool over_time(Q2Shared &s, unsigned long long &t0, int *err)
{
    const unsigned long long t = gtime();
    if (t0 == 0) t0 = t;
    if (t - t0 > WAIT_NS) {
        atomicExch(err, 3);
        *(volatile int *)&s.dead = 1;
    }
    return *(volatile int *)&s.dead != 0;
}
__device__ __forceinline__ bool is_full(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(saddr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ void wait_full(Q2Shared &s, unsigned long long *bar, unsigned parity, int *err)
{
    unsigned long long t0 = 0;
    while (!is_full(bar, parity))
        if (over_time(s, t0, err)) break;
    __syncwarp();
}
__device__ __forceinline__ void wait_count(Q2Shared &s, const int *flag, int need, int *err)
{
    unsigned long long t0 = 0;
    int spin = 0;
    while (*(volatile const int *)flag < need)
        if ((++spin & 1023) == 0 && over_time(s, t0, err)) break;
    __syncwarp();
    __threadfence_block();
}

// block i of group g, counted on into the slot's next groups
template <int G>
__device__ __forceinline__ void load_part(const Q2Args &a, Q2Shared &s, double2 *fa, int slot, int g, int i, int part,
                                          int buf)
{
    while (g >= 0 && i >= a.K - g) {
        i -= a.K - g;
        g -= G;
    }
    if (g < 0) return;
    const int at = part ? FRAG_A : 0;
    bulk_load(fa + (size_t)buf * (FRAG_A + FRAG_B) + at, a.F + (q2_block_at(a.K, g) + i) * (FRAG_A + FRAG_B) + at,
              (part ? FRAG_B : FRAG_A) * 16u, &s.full[slot][part][buf]);
}

// a slot's blocks on 8 MT columns
template <int MT, int G>
__device__ __forceinline__ void q2_warp(const Q2Args &a, Q2Shared &s, double2 *frags, double2 *links, int slot, int half,
                                        int parts, int c0)
{
    constexpr int NBUF = Q2_BUF;
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    constexpr int CHUNK = MT * 4 * 32;                       // pairs of a chunk of this warp's columns
    double2 *in = links + (size_t)(slot * 2) * CHUNK, *out = in + 2 * CHUNK;
    double2 *fa = frags + (size_t)slot * NBUF * (FRAG_A + FRAG_B);
    const int period = a.K + 2;
    // tile (mt, nt) of chunk k: rows row(k, nt), + 1 of column 8 mt + r
    auto row = [&](int k, int nt) { return k * NB + 1 + 8 * nt + 2 * c; };
    bool col[MT];
    double *zp[MT];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        col[mt] = c0 + 8 * mt + r < a.ncol;
        zp[mt] = a.Z + a.ldz * (long)(col[mt] ? c0 + 8 * mt + r : 0);
    }
    double z[MT][8][2], w[MT][4][2];
    int seq = 0;                                             // blocks of this slot so far
    for (int round = 0; round < a.rounds; round++) {
        const int g = a.K - 1 - round * G - slot;
        if (g < 0) break;
        const int nblk = a.K - g;
        const bool last = slot == G - 1 || g == 0;
        // a chunk of Z as the round before left it
        auto fetch = [&](int k) {
            if (round > 0) wait_count(s, &s.made[G - 1][half], (round - 1) * period + k + 1, a.err);
            double2 *dst = in + (k & 1) * CHUNK + lane;
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int nt = 0; nt < 4; nt++) {
                    const int rw = row(k, nt);
                    double *d = (double *)(dst + (mt * 4 + nt) * 32);
                    const bool v0 = col[mt] && rw < a.n, v1 = col[mt] && rw + 1 < a.n;
                    dmma::cp_async8(d, zp[mt] + (v0 ? rw : 0), v0);
                    dmma::cp_async8(d + 1, zp[mt] + (v1 ? rw + 1 : 0), v1);
                }
            dmma::cp_async_commit();
        };
        // chunk k into the lower half of the window
        auto take = [&](int k) {
            if (slot == 0) {
                if (k == g + 1) fetch(k);
                if (k < a.K) {
                    fetch(k + 1);
                    dmma::cp_async_wait<1>();
                } else {
                    dmma::cp_async_wait<0>();
                }
            } else {
                wait_count(s, &s.made[slot - 1][half], round * period + k + 1, a.err);
            }
            const double2 *src = in + (k & 1) * CHUNK + lane;
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int nt = 0; nt < 4; nt++) {
                    const double2 v = src[(mt * 4 + nt) * 32];
                    z[mt][nt + 4][0] = v.x;
                    z[mt][nt + 4][1] = v.y;
                }
            if (slot > 0) {
                __threadfence_block();
                __syncwarp();
                if (lane == 0) *(volatile int *)&s.taken[slot][half] = round * period + k + 1;
            }
        };
        // the upper half of the window, chunk k, to the next slot or back to Z
        auto pass = [&](int k) {
            if (last) {
#pragma unroll
                for (int mt = 0; mt < MT; mt++)
#pragma unroll
                    for (int nt = 0; nt < 4; nt++) {
                        const int rw = row(k, nt);
                        if (col[mt] && rw < a.n) zp[mt][rw] = z[mt][nt][0];
                        if (col[mt] && rw + 1 < a.n) zp[mt][rw + 1] = z[mt][nt][1];
                    }
            } else {
                // the link's place held chunk k - 2, or the end of the last round
                const int need = k - 2 >= g ? round * period + k - 1 : round > 0 ? (round - 1) * period + a.K + 1 : 0;
                wait_count(s, &s.taken[slot + 1][half], need, a.err);
                double2 *dst = out + (k & 1) * CHUNK + lane;
#pragma unroll
                for (int mt = 0; mt < MT; mt++)
#pragma unroll
                    for (int nt = 0; nt < 4; nt++) dst[(mt * 4 + nt) * 32] = make_double2(z[mt][nt][0], z[mt][nt][1]);
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) *(volatile int *)&s.made[slot][half] = round * period + k + 1;
        };
        auto shift = [&] {
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int nt = 0; nt < 4; nt++) {
                    z[mt][nt][0] = z[mt][nt + 4][0];
                    z[mt][nt][1] = z[mt][nt + 4][1];
                }
        };
        // this warp is through with an operand of block i: the last one loads that of the block NBUF on
        auto release = [&](int i, int part, int buf) {
            __threadfence_block();
            __syncwarp();
            if (lane == 0 && atomicAdd(&s.used[slot][part][buf], 1) % parts == parts - 1) {
                __threadfence_block();
                load_part<G>(a, s, fa, slot, g, i + NBUF, part, buf);
            }
        };
        // chunk g: no group before this one has touched it
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
                const int rw = row(g, nt);
                z[mt][nt + 4][0] = col[mt] && rw < a.n ? __ldcg(zp[mt] + rw) : 0.0;
                z[mt][nt + 4][1] = col[mt] && rw + 1 < a.n ? __ldcg(zp[mt] + rw + 1) : 0.0;
            }
        for (int i = 0; i < nblk; i++, seq++) {
            const int buf = seq % NBUF;
            const unsigned parity = (seq / NBUF) & 1;
            shift();
            take(g + i + 1);
            const double2 *va = fa + (size_t)buf * (FRAG_A + FRAG_B) + lane, *vb = va + FRAG_A;
            // ---- W^T = Z^T V ----
            wait_full(s, &s.full[slot][0][buf], parity, a.err);
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int t = 0; t < 4; t++) w[mt][t][0] = w[mt][t][1] = 0.0;
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
                double2 f[4];
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (nt >= t && nt <= t + 4) f[t] = va[(t * 5 + nt - t) * 32];
#pragma unroll
                for (int e = 0; e < 2; e++)
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (nt >= t && nt <= t + 4)
#pragma unroll
                            for (int mt = 0; mt < MT; mt++)
                                dmma::mma884(w[mt][t][0], w[mt][t][1], z[mt][nt][e], e ? f[t].y : f[t].x);
            }
            release(i, 0, buf);
            // ---- Z^T -= W^T (V T)^T ----
            wait_full(s, &s.full[slot][1][buf], parity, a.err);
#pragma unroll
            for (int rh = 0; rh < 8; rh += 4)
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    double2 f[4];
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (t >= fragb_t0(rh + q)) f[q] = vb[(fragb_at(rh + q) + t - fragb_t0(rh + q)) * 32];
#pragma unroll
                    for (int e = 0; e < 2; e++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (t >= fragb_t0(rh + q))
#pragma unroll
                                for (int mt = 0; mt < MT; mt++)
                                    dmma::mma884(z[mt][rh + q][0], z[mt][rh + q][1], w[mt][t][e], e ? f[q].y : f[q].x);
                }
            release(i, 1, buf);
            pass(g + i);
        }
        shift();
        pass(a.K);
    }
}

constexpr int q2_smem(int G, int T) { return 512 + 16 * (G * Q2_BUF * (FRAG_A + FRAG_B) + 2 * G * 4 * 32 * T); }

template <int G> __global__ void __launch_bounds__(32 * Q2_P * G, 1) q2_apply_kernel(Q2Args a, int T)
{
    extern __shared__ __align__(128) unsigned char q2_sm[];
    static_assert(sizeof(Q2Shared) <= 512, "the head of the shared memory");
    Q2Shared &s = *(Q2Shared *)q2_sm;
    double2 *frags = (double2 *)(q2_sm + 512), *links = frags + G * Q2_BUF * (FRAG_A + FRAG_B);
    const int tid = threadIdx.x, w = tid >> 5;
    if (tid < (int)(sizeof(Q2Shared) / 4)) ((int *)&s)[tid] = 0;
    __syncthreads();
    if (tid == 0) {
        for (int q = 0; q < Q2_GMAX * 2 * Q2_BUF; q++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&s.full[0][0][0] + q)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int p = 0; p < G; p++)
            for (int q = 0; q < Q2_BUF; q++)
                for (int part = 0; part < 2; part++)
                    load_part<G>(a, s, frags + (size_t)p * Q2_BUF * (FRAG_A + FRAG_B), p, a.K - 1 - p, q, part, q);
    }
    __syncthreads();
    // part p of the strip has T / 4 tiles, one more for p < T mod 4
    const int slot = w / Q2_P, part = (w + slot) % Q2_P;
    const int base = T / Q2_P, more = T % Q2_P, mine = base + (part < more), first = part * base + min(part, more);
    const int parts = min(T, Q2_P), c0 = 8 * ((int)blockIdx.x * T + first);
    double2 *mylinks = links + 2 * G * 4 * 32 * first;
    if (mine == 1) q2_warp<1, G>(a, s, frags, mylinks, slot, part, parts, c0);
    else if (mine == 2) q2_warp<2, G>(a, s, frags, mylinks, slot, part, parts, c0);
    __syncthreads();
    if (*(volatile int *)&s.dead) {
        // a wait ran out: let the copies in flight land (or the limit pass) before the CTA goes
        const unsigned long long t0 = gtime();
        while (gtime() - t0 < 1000000ull) {}
    }
}

}  // namespace

size_t q2_fragment_doubles(int n)
{
    if (n <= 2) return 64;
    const size_t K = (size_t)q2_blocks0(n);
    return K * (K + 1) / 2 * (FRAG_A + FRAG_B) * 2 + 64;
}

double q2_flops(int n)
{
    if (n <= 2) return 0.0;
    const double K = q2_blocks0(n);
    return K * (K + 1) / 2 * 2 * (NF_A + NF_B) * 512.0 * ((n + 7) / 8);
}

int q2_apply(int n, const double *V2, const double *tau2, int S, double *frag, double *Z, long ldz, int *err, int nsm,
             cudaStream_t st)
{
    if (n <= 2) return BSRG_OK;
    const int K = q2_blocks0(n);
    q2_fragment_kernel<<<dim3((unsigned)K, (unsigned)K), 128, 0, st>>>(n, S, V2, tau2, (double2 *)frag);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "dsyevd Q2 fragments");
    const int tiles = (n + 7) / 8;
    int T = 2;
    double cost = 1e30;
    for (int t = 2; t <= Q2_TMAX; t++) {
        const int strips = (tiles + t - 1) / t;
        const double c = (strips + nsm - 1) / nsm * std::max((double)t, 3.2);
        if (c < cost) { cost = c; T = t; }
    }
    static_assert(Q2_TMAX <= 2 * Q2_P && q2_smem(3, Q2_TMAX) <= 227 * 1024 && q2_smem(4, 2) <= 227 * 1024,
                  "a strip fits");
    const unsigned strips = (unsigned)((tiles + T - 1) / T);
    const int G = T == 2 ? 4 : 3, smem = q2_smem(G, T);
    const Q2Args a{n, n, K, (K + G - 1) / G, (const double2 *)frag, Z, ldz, err};
    e = G == 4 ? smem_attr(q2_apply_kernel<4>, smem) : smem_attr(q2_apply_kernel<3>, smem);
    if (e != cudaSuccess) return cuda_fail(e, "dsyevd Q2 smem");
    if (G == 4) q2_apply_kernel<4><<<strips, 32 * Q2_P * 4, smem, st>>>(a, T);
    else q2_apply_kernel<3><<<strips, 32 * Q2_P * 3, smem, st>>>(a, T);
    return cuda_fail(cudaGetLastError(), "dsyevd Q2");
}

}  // namespace bsrg
