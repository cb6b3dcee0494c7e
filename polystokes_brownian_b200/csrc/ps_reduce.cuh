// ps_reduce.cuh -- segmented per-replica reductions shared by the Krylov
// solvers: a block covers a contiguous range of one replica's vector, and the
// blocks' sums are added in fixed order, so results never depend on block
// scheduling or on other replicas.  Two ways to the total: every block of the next
// kernel adds them (rep_total), or the replica's last block to arrive does, by an
// atomic counter (finish_block).
#pragma once
#include "ps_kernels.h"

namespace ps {

constexpr int RB_THREADS = 256;
constexpr int RB_EPT = 4;                       // elements per thread
constexpr int RB_SPAN = RB_THREADS * RB_EPT;    // elements per block

// Block-level sum of NV values; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sh)[NV])
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        double t = v[q];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) sh[wid][q] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            double t = 0;
            for (int w = 0; w < RB_THREADS / 32; w++) t += sh[w][q];
            v[q] = t;
        }
    }
}

// Writes this block's partials and returns true in thread 0 of the last block
// of its replica; that thread then holds the replica totals in tot[].
template <int NV>
__device__ __forceinline__ bool finish_block(const RedTable &T, const RBlk &b, int bid, double (&v)[NV], double (&tot)[NV])
{
    __shared__ bool last;
    if (threadIdx.x == 0) {
        for (int q = 0; q < NV; q++) T.d_part[4 * bid + q] = v[q];
        __threadfence();
        int t = atomicAdd(&T.d_counter[b.rep], 1);
        last = (t == T.d_count[b.rep] - 1);
    }
    __syncthreads();
    if (!last) return false;
    if (threadIdx.x == 0) {
        __threadfence();
        int f = T.d_first[b.rep], c = T.d_count[b.rep];
        for (int q = 0; q < NV; q++) tot[q] = 0.0;
        for (int k = 0; k < c; k++)
            for (int q = 0; q < NV; q++) tot[q] += ((volatile double *)T.d_part)[4 * (f + k) + q];
        T.d_counter[b.rep] = 0;
        return true;
    }
    return false;
}

// Total of a replica's nb block sums, the same in every thread of the block and in a fixed
// order (of nb and the block's width, at most RB_THREADS).  Every block of a kernel adds its
// replica's sums itself: no counters, no fences, no last block.
__device__ __forceinline__ double rep_total(const double *__restrict__ part, int nb)
{
    __shared__ double ws[RB_THREADS / 32];
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) t += part[b];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    __syncthreads();                       // an earlier total has been read
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = t;
    __syncthreads();
    t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += ws[w];
    return t;
}

// MINRES scalars after an iteration, from its r.z total bb (Paige & Saunders; PETSc's test):
// the pending w/x update, the next beta, convergence
__device__ __forceinline__ void minres_advance(MinresScal &m, double bb, int maxit)
{
    m.it += 1;
    m.oldb = m.beta;
    m.pending = 0;
    if (bb < 0) { m.done = 1; m.reason = -8; return; }
    m.beta = sqrt(bb);
    const double oldeps = m.epsln;
    const double delta = m.cs * m.dbar + m.sn * m.alfa;
    const double gbar = m.sn * m.dbar - m.cs * m.alfa;
    m.epsln = m.sn * m.beta;
    m.dbar = -m.cs * m.beta;
    double gamma = sqrt(gbar * gbar + m.beta * m.beta);
    if (gamma < 2.2250738585072014e-308) gamma = 2.2250738585072014e-308;
    m.cs = gbar / gamma;
    m.sn = m.beta / gamma;
    const double phi = m.cs * m.phibar;
    m.phibar = m.sn * m.phibar;
    m.up_oldeps = oldeps; m.up_delta = delta; m.up_ginv = 1.0 / gamma; m.up_phi = phi;
    m.pending = 1;
    m.np = m.np * fabs(m.sn);
    if (m.np <= m.ttol) { m.done = 1; m.reason = 2; }
    else if (m.beta == 0.0) { m.done = 1; m.reason = 3; }
    else if (m.it >= maxit) { m.done = 1; m.reason = -3; }
    m.sinv = m.beta != 0.0 ? 1.0 / m.beta : 0.0;
}

// First half of a MINRES iteration for one entry per thread: index q of the saddle vectors (act:
// the entry exists), Az its product; B, the block of the saddle table.  Writes Av over it.
// Returns at once for a replica that was done, carrying its scalars on.
__device__ __forceinline__ void mr_alpha(const RedTable &T, const RBlk &B, int n, long q, bool act, double Az,
                                         const MrAlpha &A, double *__restrict__ Av)
{
    __shared__ MinresScal sm;
    __shared__ double sh[RB_THREADS / 32][1];
    const int first = T.d_first[B.rep];
    const bool lead = blockIdx.y == 0 && (int)blockIdx.x == first && threadIdx.x == 0;
    // everything that does not wait for the scalars is asked for ahead of them
    double z = 0.0, v = 0.0, w1 = 0.0, w2 = 0.0, xq = 0.0, rm = 0.0;
    if (act) {
        z = A.z[q];
        if (A.k > 1) { v = A.v[q]; w1 = A.w1[q]; w2 = A.w2[q]; xq = A.x[q]; rm = A.rkm1[q]; }
    }
    const double bb = A.k > 1 ? rep_total(A.pb + RB_EPT * first, (n + RB_THREADS - 1) / RB_THREADS) : 0.0;
    if (threadIdx.x == 0) {
        MinresScal m = A.st0[B.rep];
        if (A.k > 1) minres_advance(m, bb, A.maxit);
        sm = m;
        if (lead) {
            if (m.done) atomicSub(A.nactive, 1);
            m.pending = 0;                                 // applied below
            A.st1[B.rep] = m;
        }
    }
    __syncthreads();
    double s[1] = {0.0};
    if (act) {
        if (sm.pending) {
            const double wn = (v - sm.up_oldeps * w1 - sm.up_delta * w2) * sm.up_ginv;
            A.wnew[q] = wn;
            A.x[q] = xq + sm.up_phi * wn;
        }
        if (!sm.done) {
            const double vq = z * sm.sinv;
            double a = Az * sm.sinv;
            if (A.k >= 2) a -= (sm.beta / sm.oldb) * rm;
            A.v[q] = vq;
            Av[q] = a;
            s[0] = vq * a;
        }
    }
    if (sm.done) return;
    block_sum<1>(s, sh);
    if (threadIdx.x == 0) A.pa[RB_EPT * blockIdx.x + blockIdx.y] = s[0];
}

// sums of sixteen values over the warp by halving exchanges (16 double shuffles): the lane
// ends with the total of value idx (each total in two lanes)
__device__ __forceinline__ double warp_sum16(double (&v)[16], int lane, int &idx)
{
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int c = 0; c < h; c++) {
            const double send = up ? v[c] : v[c + h], keep = up ? v[c + h] : v[c];
            v[c] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    idx = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// sums of 32 values over the warp; the lane ends with the total of value `lane`
__device__ __forceinline__ double warp_sum32(double (&v)[32], int lane)
{
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int c = 0; c < h; c++) {
            const double send = up ? v[c] : v[c + h], keep = up ? v[c + h] : v[c];
            v[c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    return v[0];
}

// Entry k (one per thread, when act) of the first LZ_REG of the vectors V_0..V_j, zero beyond: asked
// for at a kernel's start, all at once, so that subtraction and dots find them in registers.
constexpr int LZ_REG = 32;
__device__ __forceinline__ void lz_load(const double *__restrict__ V, long ldv, long k, bool act, int j, double (&v)[LZ_REG])
{
#pragma unroll
    for (int i = 0; i < LZ_REG; i++) v[i] = act && i <= j ? V[(long)i * ldv + k] : 0.0;
}

// A block's dots of its entries (one per thread: value q at index k, when act; v from lz_load) with the
// Lanczos vectors V_0..V_j, into out[0..j]; RB_THREADS threads, every one of which takes part.
__device__ __forceinline__ void lz_block_dots(const double (&v)[LZ_REG], const double *__restrict__ V, long ldv, long k,
                                              bool act, double q, int j, double *__restrict__ out)
{
    __shared__ double sh[RB_THREADS / 32][LZ_KMAX];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (j < 16) {
        double p[16];
#pragma unroll
        for (int c = 0; c < 16; c++) p[c] = v[c] * q;
        int idx;
        const double t = warp_sum16(p, lane, idx);
        if (!(lane & 1)) sh[wid][idx] = t;
    } else {
        double p[LZ_REG];
#pragma unroll
        for (int c = 0; c < LZ_REG; c++) p[c] = v[c] * q;
        sh[wid][lane] = warp_sum32(p, lane);
    }
    for (int i0 = LZ_REG; i0 <= j; i0 += 16) {
        double p[16];
#pragma unroll
        for (int c = 0; c < 16; c++) p[c] = (act && i0 + c <= j) ? V[(long)(i0 + c) * ldv + k] * q : 0.0;
        int idx;
        const double t = warp_sum16(p, lane, idx);
        if (!(lane & 1) && i0 + idx <= j) sh[wid][i0 + idx] = t;
    }
    __syncthreads();
    if (threadIdx.x <= j) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < RB_THREADS / 32; w++) t += sh[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
}

// The same from memory, sixteen vectors at a time: the combine of an apply forms q late and has many
// blocks in flight, where 32 entries held since its start cost more blocks than they save waits (64
// replicas 15.7 against 17.6 us a launch, 1024 beads 5.1 against 4.6).
__device__ __forceinline__ void lz_block_dots(const double *__restrict__ V, long ldv, long k, bool act, double q, int j,
                                              double *__restrict__ out)
{
    __shared__ double sh[RB_THREADS / 32][LZ_KMAX];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int i0 = 0; i0 <= j; i0 += 16) {
        double v[16];
#pragma unroll
        for (int c = 0; c < 16; c++) v[c] = (act && i0 + c <= j) ? V[(long)(i0 + c) * ldv + k] * q : 0.0;
        int idx;
        const double t = warp_sum16(v, lane, idx);
        if (!(lane & 1) && i0 + idx <= j) sh[wid][i0 + idx] = t;
    }
    __syncthreads();
    if (threadIdx.x <= j) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < RB_THREADS / 32; w++) t += sh[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
}

}  // namespace ps
