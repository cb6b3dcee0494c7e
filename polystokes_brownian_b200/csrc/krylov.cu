// krylov.cu -- batched preconditioned MINRES (KSPSolve stand-in) and the
// Lanczos square root M^{1/2} z, with device-side per-replica scalars and
// convergence flags.
//
// MINRES follows the preconditioned Paige & Saunders (1975) recurrences with
// PETSc KSPMINRES semantics (src/ksp/ksp/impls/minres of PETSc 3.22+; called
// from src/vel.cpp:41-43 of the reference with PCJACOBI fix-diagonal,
// src/init.cpp:217-241): convergence when ||B r0||_2 * prod|s_k| <= rtol * ref,
// ref = ||B r0|| for a zero guess and ||B b|| for a nonzero guess.
//
// Reductions are segmented per replica: each block covers a contiguous range of one
// replica and leaves its sum in memory, and every block of the next kernel adds its
// replica's sums itself in fixed order (rep_total, lz_total), so the result never depends
// on other replicas or on block scheduling.  A solve's start, single dots and the ordered
// sweeps of the square root (k_lz_ord_*) instead leave the totals to the replica's last
// block to arrive (finish_block).
#include <cmath>
#include <cstdio>
#include <vector>
#include <cooperative_groups.h>
#include "ps_internal.h"
#include "ps_kernels.h"
#include "ps_reduce.cuh"

namespace ps {

// layout 0: saddle vectors, 1: mobility (top) vectors, 2: velocity vectors
int build_red_table(Engine &E, RedTable &T, int layout)
{
    std::vector<RBlk> blk;
    std::vector<int> first(E.R), cnt(E.R);
    for (int r = 0; r < E.R; r++) {
        const Seg &s = E.segs[r];
        int n = layout == 1 ? s.nm3nc11 : (layout == 2 ? s.nm3nc6 : s.n);
        int off = layout == 1 ? s.top_off : (layout == 2 ? s.vel_off : s.vec_off);
        first[r] = (int)blk.size();
        int nb = (n + RB_SPAN - 1) / RB_SPAN;
        if (nb == 0) nb = 1;
        for (int b = 0; b < nb; b++) {
            int st = b * RB_SPAN, len = std::min(RB_SPAN, n - st);
            if (len < 0) len = 0;
            blk.push_back({r, off + st, len});
        }
        cnt[r] = nb;
    }
    T.nblk = (int)blk.size();
    // where blocks are many, none beyond the longest one's length (4000 replicas of 3 beads: an apply 22 us for 30)
    T.nsub = RB_EPT;
    if (T.nblk > 4 * 148) {
        T.nsub = 1;
        for (const RBlk &b : blk) T.nsub = std::max(T.nsub, (b.len + RB_THREADS - 1) / RB_THREADS);
    }
    PS_CK(cudaMalloc(&T.d_blk, sizeof(RBlk) * T.nblk));
    PS_CK(cudaMalloc(&T.d_first, sizeof(int) * E.R));
    PS_CK(cudaMalloc(&T.d_count, sizeof(int) * E.R));
    PS_CK(cudaMalloc(&T.d_counter, sizeof(int) * E.R));
    PS_CK(cudaMalloc(&T.d_part, sizeof(double) * 4 * T.nblk));
    PS_CK(cudaMemcpy(T.d_blk, blk.data(), sizeof(RBlk) * T.nblk, cudaMemcpyHostToDevice));
    PS_CK(cudaMemcpy(T.d_first, first.data(), sizeof(int) * E.R, cudaMemcpyHostToDevice));
    PS_CK(cudaMemcpy(T.d_count, cnt.data(), sizeof(int) * E.R, cudaMemcpyHostToDevice));
    PS_CK(cudaMemset(T.d_counter, 0, sizeof(int) * E.R));
    return PS_OK;
}

void free_red_table(RedTable &T)
{
    cudaFree(T.d_blk); cudaFree(T.d_first); cudaFree(T.d_count); cudaFree(T.d_counter); cudaFree(T.d_part);
    T = RedTable();
}

// ---------------------------------------------------------------------------
// generic segmented dot: out[rep] = a.b
__global__ void k_seg_dot(RedTable T, const double *__restrict__ a, const double *__restrict__ b, double *out)
{
    pdl_enter();
    __shared__ double sh[RB_THREADS / 32][1];
    const RBlk B = T.d_blk[blockIdx.x];
    double v[1] = {0.0};
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) v[0] += a[B.start + e] * b[B.start + e];
    block_sum<1>(v, sh);
    double tot[1];
    if (finish_block<1>(T, B, blockIdx.x, v, tot)) out[B.rep] = tot[0];
}

void seg_dot(Engine &E, RedTable &T, const double *a, const double *b, double *out, cudaStream_t st)
{
    ps_launch(k_seg_dot, T.nblk, RB_THREADS, 0, st, T, a, b, out);
}

// ---------------------------------------------------------------------------
// MINRES
__global__ void k_mr_init(RedTable T, const Seg *segs, const double *__restrict__ b, const double *__restrict__ Ax,
                          const double *__restrict__ D, double *__restrict__ r, double *__restrict__ z,
                          double *__restrict__ x, MinresScal *mr, int warm, double rtol, int maxit,
                          double *__restrict__ v, double *__restrict__ w0, double *__restrict__ w1,
                          double *__restrict__ w2)
{
    pdl_enter();
    __shared__ double sh[RB_THREADS / 32][3];
    const RBlk B = T.d_blk[blockIdx.x];
    double s[3] = {0.0, 0.0, 0.0};
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) {
        long k = B.start + e;
        double bk = b[k], rk, dk = D[k];
        if (warm) rk = bk - Ax[k];
        else { rk = bk; x[k] = 0.0; }
        double zk = rk / dk;
        r[k] = rk; z[k] = zk;
        v[k] = 0.0; w0[k] = 0.0; w1[k] = 0.0; w2[k] = 0.0;
        s[0] += zk * zk;
        s[1] += rk * zk;
        double bz = bk / dk;
        s[2] += bz * bz;
    }
    block_sum<3>(s, sh);
    double tot[3];
    if (finish_block<3>(T, B, blockIdx.x, s, tot)) {
        MinresScal m = {};
        double np0 = sqrt(tot[0]);
        double ref = warm ? sqrt(tot[2]) : np0;
        double ttol = rtol * ref;
        if (ttol < 1e-50) ttol = 1e-50;
        m.np = np0; m.ttol = ttol; m.it = 0; m.pending = 0;
        (void)maxit;
        if (tot[1] < 0) { m.done = 1; m.reason = -8; }
        else if (np0 <= ttol || tot[1] == 0.0) { m.done = 1; m.reason = 2; }
        else {
            m.done = 0; m.reason = 0;
            m.beta = sqrt(tot[1]); m.oldb = 0; m.dbar = 0; m.epsln = 0; m.phibar = m.beta;
            m.cs = -1; m.sn = 0; m.sinv = 1.0 / m.beta;
        }
        mr[B.rep] = m;
    }
}

// An iteration's vector work, one entry per thread (sub-blocks of RB_THREADS entries): the
// combine of the apply goes on with mr_alpha (ps_reduce.cuh), k_mr_beta follows.  The
// scalars between them are recomputed by every block from the sub-block sums of the kernel
// before (rep_total), so no kernel ends in a last block that sums and runs the recurrence
// while the chip waits.  mr_alpha closes iteration k - 1 (its scalars, the w and x update) and
// opens iteration k: v = z / beta, Av = A z / beta - (beta / oldb) r_{k-1}, sums of
// alfa = v.Av.  k_mr_beta: r_{k+1} = Av - (alfa / beta) r_k, z = r_{k+1} / D, sums of r.z.  The
// scalars of iteration k live in st[k & 1]: a kernel reads one and its replica's first block
// writes the other.
//
// Bound: latency (a dependent launch with an L2 round trip takes some 4 us).  516 beads, one
// iteration: 21.5 us with a launch for each half and last-block sums, 16.5 us without
// them, 14.9 us with the first half in the combine, 14.2 us with the vectors' loads ahead of
// the totals.
__global__ void k_mr_beta(RedTable T, const Seg *__restrict__ segs, double *__restrict__ Av, const double *__restrict__ rk,
                          const double *__restrict__ D, double *__restrict__ z, MinresScal *__restrict__ st,
                          const double *__restrict__ pa, double *__restrict__ pb)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const int e = blockIdx.y * RB_THREADS + threadIdx.x;
    if (blockIdx.y * RB_THREADS >= B.len || st[B.rep].done) return;
    __shared__ double sh[RB_THREADS / 32][1];
    const int first = T.d_first[B.rep];
    const bool act = e < B.len;
    const long q = (long)B.start + e;
    // asked for ahead of the total
    const double av = act ? Av[q] : 0.0, r = act ? rk[q] : 0.0, d = act ? D[q] : 1.0, bt = st[B.rep].beta;
    const double alfa = rep_total(pa + RB_EPT * first, (segs[B.rep].n + RB_THREADS - 1) / RB_THREADS);
    if (blockIdx.y == 0 && (int)blockIdx.x == first && threadIdx.x == 0) st[B.rep].alfa = alfa;
    double s[1] = {0.0};
    if (act) {
        const double a = av - (alfa / bt) * r;
        const double zq = a / d;
        Av[q] = a;
        z[q] = zq;
        s[0] = a * zq;
    }
    block_sum<1>(s, sh);
    if (threadIdx.x == 0) pb[RB_EPT * blockIdx.x + blockIdx.y] = s[0];
}

int minres_solve(Engine &E, const double *b, double *x, const ps_ksp_opts *o, ps_ksp_result *res, cudaStream_t st)
{
    ps_ksp_opts opt = {1e-6, 10000, 0, 8, PS_SOLVE_MINRES};
    if (o) opt = *o;
    if (opt.check_every <= 0) opt.check_every = 8;
    if (opt.maxit <= 0) opt.maxit = 10000;
    RedTable &T = E.red;
    int rc = diag_saddle(E, E.d_D, st);
    if (rc) return rc;
    const double *Ax = nullptr;
    if (opt.warm) {
        apply_operator(E, 0, x, E.d_Rr[2], false, st);
        Ax = E.d_Rr[2];
    }
    // r_1 in slot 1 (slot k % 3 holds r_k); scalars in d_mr[(k & 1) R ..]
    ps_launch(k_mr_init, T.nblk, RB_THREADS, 0, st, T, E.d_segs, b, Ax, E.d_D, E.d_Rr[1], E.d_z, x, E.d_mr, opt.warm,
            opt.rtol, opt.maxit, E.d_v, E.d_W[0], E.d_W[1], E.d_W[2]);
    PS_CK(cudaGetLastError());
    // count active replicas
    std::vector<MinresScal> hm(E.R);
    PS_CK(cudaMemcpyAsync(hm.data(), E.d_mr, sizeof(MinresScal) * E.R, cudaMemcpyDeviceToHost, st));
    PS_CK(cudaStreamSynchronize(st));
    int nact = 0;
    for (auto &m : hm) nact += !m.done;
    *E.h_nactive = nact;
    PS_CK(cudaMemcpyAsync(E.d_nactive, E.h_nactive, sizeof(int), cudaMemcpyHostToDevice, st));
    double *pa = E.d_mrp, *pb = pa + (long)RB_EPT * T.nblk;
    const dim3 sub((unsigned)T.nblk, (unsigned)T.nsub);
    MinresScal *last = E.d_mr;
    // the apply of iteration k closes iteration k - 1, so the check stands between the apply and
    // k_mr_beta, and a solve that converged at k - 1 has spent one apply of iteration k
    for (int k = 1, next = opt.check_every + 1; nact > 0; k++) {
        double *Av = E.d_Rr[(k + 1) % 3];
        const double *rk = E.d_Rr[k % 3];
        const double *rkm1 = E.d_Rr[(k + 2) % 3];
        // iteration k - 1's update writes w_{k-1} into slot (k-1)%3; w_{k-3} and w_{k-2} are in the others
        double *wnew = E.d_W[(k + 2) % 3];
        const double *w1 = E.d_W[(k + 0) % 3], *w2 = E.d_W[(k + 1) % 3];
        MinresScal *s0 = E.d_mr + (long)E.R * ((k - 1) & 1), *s1 = E.d_mr + (long)E.R * (k & 1);
        const MrAlpha al = {E.d_z, rkm1, w1, w2, pb, E.d_v, wnew, x, pa, s0, s1, E.d_nactive, k, opt.maxit};
        apply_operator(E, 0, E.d_z, Av, E.precision == PS_PREC_MIXED, st, &s0[0].done, (int)sizeof(MinresScal), false,
                       nullptr, &al);
        last = s1;
        if (k == next || k > opt.maxit) {
            PS_CK(cudaMemcpyAsync(E.h_nactive, E.d_nactive, sizeof(int), cudaMemcpyDeviceToHost, st));
            PS_CK(cudaStreamSynchronize(st));
            nact = *E.h_nactive;
            if (k > opt.maxit) break;
            // long solves are looked at less often: a missed stop costs launches of blocks that leave at
            // once (about 8 us an iteration), a look some 15 us
            next += std::max(opt.check_every, std::min(k / 4, 4 * opt.check_every));
        }
        if (nact > 0)
            ps_launch(k_mr_beta, sub, RB_THREADS, 0, st, T, E.d_segs, Av, rk, E.d_D, E.d_z, s1, pa, pb);
    }
    PS_CK(cudaMemcpyAsync(hm.data(), last, sizeof(MinresScal) * E.R, cudaMemcpyDeviceToHost, st));
    PS_CK(cudaStreamSynchronize(st));
    PS_CK(cudaGetLastError());
    int worst = 1000, itmax = 0;
    long itsum = 0;
    double rmax = 0;
    for (auto &m : hm) {
        int reason = m.done ? m.reason : -3;
        if (reason < worst) worst = reason;
        itmax = std::max(itmax, m.it);
        itsum += m.it;
        rmax = std::max(rmax, m.np);
    }
    if (res) { res->reason = worst; res->iters_max = itmax; res->iters_sum = itsum; res->rnorm_max = rmax; }
    return worst;
}


// ---------------------------------------------------------------------------
// Lanczos square root w = M^{1/2} z on the mobility vectors (top layout), full
// two-pass Gram-Schmidt reorthogonalisation, projected spectrum floored at 0
// (the policy of schur_sqrt_lanczos, slip_vel.cpp:351-477, applied to the full
// grand mobility instead of SLEPc MFN/FNSQRT, slip_vel.cpp:27-49).
// done after j vectors lives in done[j & 1]: the launches of vector j read it there and the
// orthogonalisation's last one writes done[(j + 1) & 1], so that all threads of a launch see one value.
struct LzScal {
    double b0;
    int m, nneg, done[2];
};

// Reorthogonalisation of one Lanczos vector, q = M V_j against V_0..V_j: two
// passes of classical Gram-Schmidt.  One thread owns one entry of the replica's
// vector, in sub-blocks of 256 entries (a quarter of a reduction-table block).
// The combine that forms q also forms the first pass's dots (k_combine), then
// k_lz_sub_dots subtracts and forms the second pass's dots and the norm, and
// k_lz_sub_scale subtracts, tests for breakdown and scales.  Each
// kernel leaves its sub-blocks' sums in memory, and every block of the next one
// adds its replica's sums itself, in a fixed order that depends on the vector's
// length alone -- no counters and no fences, and a replica's noise does not depend
// on its batch.  Replicas whose far field may be indefinite (Seg::indef) take
// k_lz_orth_cluster or the k_lz_ord_* sweeps, and the QL check, instead.
//
// Bound: latency and L2 (the basis is read twice from L2 and once from L1 per
// vector, k_lz_sub_dots reading its slices twice).  With 1024 entries per block of
// 256 threads, or one cluster of eight blocks per replica, too few loads were in
// flight: a vector with its apply took 42 us at 1024 beads (23 this way), 72 us at the
// 4097-bead brush (49 this way), and the sweeps of 64 replicas, 62000 beads, 100 us
// (44 this way).  Taking the norm with the second dots instead of in a launch of its
// own is 2 us of these; holding the thread's entries of the first 32 vectors in registers, asked
// for before the totals are added, 2 us more (k_lz_sub_dots 5.5 -> 4.4 us at 1024 beads).
constexpr int LZ_SUB = RB_THREADS;                    // entries of a sub-block
static_assert(RB_SPAN == RB_EPT * LZ_SUB, "RB_EPT sub-blocks per table block");

// the replica's total of the sub-block sums part[][i], i <= j, into h[] (shared, zero beyond j); NORM: that
// of npart[] into h[LZ_KMAX].  The replica's first table block and length come from the caller.
template <bool NORM>
__device__ __forceinline__ void lz_total(int first_blk, int n, const double *__restrict__ part,
                                         const double *__restrict__ npart, int j, double *__restrict__ h)
{
    __shared__ double sh4[RB_THREADS / LZ_KMAX][LZ_KMAX];
    constexpr int G = RB_THREADS / LZ_KMAX;
    const int i = threadIdx.x % LZ_KMAX, g = threadIdx.x / LZ_KMAX;
    const int nb = (n + LZ_SUB - 1) / LZ_SUB;
    const long first = (long)RB_EPT * first_blk;
    const double *p = part + first * LZ_KMAX + i;
    double t = 0.0, n2 = 0.0;
    const bool norm = NORM && threadIdx.x >= RB_THREADS - 32;      // the warp whose dots come last
    if (norm)
        for (int b = threadIdx.x & 31; b < nb; b += 32) n2 += npart[first + b];
    if (i <= j) {
#pragma unroll 4
        for (int b = g; b < nb; b += G) t += p[(long)b * LZ_KMAX];
    }
    sh4[g][i] = t;
    if (norm) {
        for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
        if (threadIdx.x == RB_THREADS - 1) h[LZ_KMAX] = n2;
    }
    __syncthreads();
    if (threadIdx.x < LZ_KMAX) {
        double v = 0.0;
        for (int c = 0; c < G; c++) v += sh4[c][threadIdx.x];
        h[threadIdx.x] = v;
    }
    __syncthreads();
}

// q -= sum_i h_i V_i for this thread's entry (v from lz_load), in four interleaved sums
__device__ __forceinline__ double lz_subtract(const double (&v)[LZ_REG], const double *__restrict__ V, long ldv, long k,
                                              bool act, double q, int j, const double *__restrict__ h)
{
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < LZ_REG; i += 8)
        if (i <= j) {
#pragma unroll
            for (int c = 0; c < 8; c++) t[c & 3] += h[i + c] * v[i + c];
        }
    if (act)
        for (int i = LZ_REG; i <= j; i += 8)
#pragma unroll
            for (int c = 0; c < 8; c++)
                if (i + c <= j) t[c & 3] += h[i + c] * V[(long)(i + c) * ldv + k];
    return q - ((t[0] + t[1]) + (t[2] + t[3]));
}

__global__ void k_lz_sub_dots(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ V, long ldv,
                              double *__restrict__ q, int j, const LzScal *__restrict__ lz,
                              const double *__restrict__ part1, double *__restrict__ alpha, double *__restrict__ part2,
                              double *__restrict__ npart)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const int e = blockIdx.y * LZ_SUB + threadIdx.x;
    if (blockIdx.y * LZ_SUB >= B.len) return;
    const int first = T.d_first[B.rep];
    const bool act = e < B.len;
    const long k = (long)B.start + e;
    double vr[LZ_REG], v = act ? q[k] : 0.0;
    lz_load(V, ldv, k, act, j, vr);
    if (lz[B.rep].done[j & 1] || segs[B.rep].indef) return;
    __shared__ double h[LZ_KMAX], wn[RB_THREADS / 32];
    lz_total<false>(first, segs[B.rep].nm3nc11, part1, nullptr, j, h);
    v = lz_subtract(vr, V, ldv, k, act, v, j, h);
    if (act) q[k] = v;
    if (threadIdx.x == 0 && blockIdx.y == 0 && (int)blockIdx.x == first) alpha[(long)LZ_KMAX * B.rep + j] = h[j];
    double n2 = v * v;
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    if ((threadIdx.x & 31) == 0) wn[threadIdx.x >> 5] = n2;
    lz_block_dots(vr, V, ldv, k, act, v, j, part2 + (long)LZ_KMAX * (RB_EPT * blockIdx.x + blockIdx.y));   // a barrier inside
    if (threadIdx.x == RB_THREADS - 1) {
        n2 = 0.0;
        for (int w = 0; w < RB_THREADS / 32; w++) n2 += wn[w];
        npart[RB_EPT * blockIdx.x + blockIdx.y] = n2;
    }
}

// Second subtraction, beta_j = ||q||, V_{j+1} = q / beta_j, m = j + 1; an invariant subspace stops
// the replica.  The norm after the subtraction is that before it less the dots' squares (the
// basis is orthonormal), so no further sum over the replica, and no further launch, is needed: the
// dots of a second pass are rounding residues of the first, and only at a breakdown not far
// smaller than q.
__global__ void k_lz_sub_scale(RedTable T, const Seg *__restrict__ segs, double *__restrict__ V, long ldv,
                               const double *__restrict__ q, int j, int kmax, LzScal *__restrict__ lz,
                               const double *__restrict__ part2, const double *__restrict__ npart,
                               double *__restrict__ alpha, double *__restrict__ betad)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const int e = blockIdx.y * LZ_SUB + threadIdx.x;
    if (blockIdx.y * LZ_SUB >= B.len) return;
    const int first = T.d_first[B.rep];
    const bool act = e < B.len;
    const long k = (long)B.start + e;
    double vr[LZ_REG];
    const double qk = act ? q[k] : 0.0;
    lz_load(V, ldv, k, act, j, vr);
    const bool lead = threadIdx.x == 0 && blockIdx.y == 0 && (int)blockIdx.x == first;
    const int done = lz[B.rep].done[j & 1], indef = segs[B.rep].indef;
    if (done || indef) {
        if (lead && !indef) lz[B.rep].done[(j + 1) & 1] = done;
        return;
    }
    __shared__ double h[LZ_KMAX + 1];
    lz_total<true>(first, segs[B.rep].nm3nc11, part2, npart, j, h);
    double h2[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = 0; i <= j; i += 4)
#pragma unroll
        for (int c = 0; c < 4; c++) h2[c] += h[i + c] * h[i + c];      // zero beyond j
    // a norm that is not a number stays one (fmax would make it 0, which reads as a breakdown)
    const double n2 = h[LZ_KMAX] - ((h2[0] + h2[1]) + (h2[2] + h2[3])), bj = sqrt(n2 < 0.0 ? 0.0 : n2);
    const bool broken = bj <= 1e-12 * lz[B.rep].b0;
    if (!broken && j + 1 < kmax && act)
        V[(long)(j + 1) * ldv + k] = lz_subtract(vr, V, ldv, k, act, qk, j, h) * (bj > 0 ? 1.0 / bj : 0.0);
    if (lead) {
        alpha[(long)LZ_KMAX * B.rep + j] += h[j];
        lz[B.rep].m = j + 1;
        lz[B.rep].done[(j + 1) & 1] = broken ? 2 : 0;      // 2: finalise with m = j + 1
        if (!broken && j + 1 < kmax) betad[(long)LZ_KMAX * B.rep + j] = bj;
    }
}

__global__ void k_lz_init(RedTable T, const Seg *__restrict__ segs, double *__restrict__ V,
                          const double *__restrict__ z, LzScal *__restrict__ lz, const double *__restrict__ nrm2)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    // shell replicas take the block-Cholesky noise path instead
    const bool skip = !segs[B.rep].mm_HI;
    double b0 = sqrt(nrm2[B.rep]);
    double inv = b0 > 0 ? 1.0 / b0 : 0.0;
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) V[B.start + e] = z[B.start + e] * inv;
    if (threadIdx.x == 0 && (B.start == T.d_blk[T.d_first[B.rep]].start)) {
        lz[B.rep].b0 = skip ? 0.0 : b0; lz[B.rep].m = 0; lz[B.rep].done[0] = (b0 == 0.0 || skip); lz[B.rep].nneg = 0;
    }
}

// Implicit QL (symmetric tridiagonal, Wilkinson shift) on one warp.  Lane 0
// runs each QL iteration's scalar recurrence on the shared d, e and records
// the iteration's rotations (c, s) in rot; then every lane applies them, in the
// recurrence's order, to its own rows of Z.  A row sees the same rotations in
// the same order as when each rotation is applied to all rows at once, so Z is
// the same, without a warp barrier per rotation.  rot holds 2 n doubles;
// n <= 64 (two rows of Z per lane).  The warp's lanes search for the split
// point together.  Every lane of the warp takes part.
__device__ void warp_tql(double *d, double *e, double *Z, double *rot, int n)
{
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < n * n; k += 32) Z[k] = (k / n == k % n) ? 1.0 : 0.0;
    __syncwarp();
    for (int l = 0; l < n; l++) {
        int iter = 0;
        while (true) {
            // the first m >= l with a negligible e[m] (n - 1 if none), tested 32 at a time
            int m = n - 1, iend = l;
            for (int m0 = l; m0 < n - 1; m0 += 32) {
                const int mm = m0 + lane;
                bool hit = false;
                if (mm < n - 1) {
                    const double dd = fabs(d[mm]) + fabs(d[mm + 1]);
                    hit = fabs(e[mm]) <= 1e-16 * dd;
                }
                const unsigned b = __ballot_sync(0xffffffffu, hit);
                if (b) { m = m0 + __ffs(b) - 1; break; }
            }
            const bool go = (m != l) && (iter < 60);
            if (lane == 0) {
                if (go) {
                    double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
                    double r = hypot(g, 1.0);
                    g = d[m] - d[l] + e[l] / (g + copysign(r, g));
                    double s = 1, c = 1, p = 0;
                    bool brk = false;
                    for (int i = m - 1; i >= l; i--) {
                        const double ei = e[i], di = d[i], di1 = d[i + 1];
                        double f = s * ei, b = c * ei;
                        // rotation from one reciprocal square root (the chain of dependent
                        // divisions is this loop's latency; f, g are O(|T|), far from overflow)
                        const double r2 = f * f + g * g, ri = r2 > 0.0 ? rsqrt(r2) : 0.0;
                        const double rr = r2 * ri;
                        if (rr == 0.0) {
                            e[i + 1] = rr; d[i + 1] = di1 - p; e[m] = 0.0;
                            brk = true;
                            iend = i + 1;
                            break;
                        }
                        s = f * ri; c = g * ri;
                        g = di1 - p;
                        r = (di - g) * s + 2.0 * c * b;
                        p = s * r;
                        e[i + 1] = rr; d[i + 1] = g + p;
                        g = c * r - b;
                        rot[2 * i] = c; rot[2 * i + 1] = s;
                    }
                    if (!brk) { d[l] -= p; e[l] = g; e[m] = 0.0; }
                }
            }
            iter++;
            iend = __shfl_sync(0xffffffffu, iend, 0);
            if (!go) break;
            __syncwarp();                       // rot, d, e written by lane 0 are visible
            // rows lane and lane + 32 (n <= 64) advance together, each in the order i = m-1 .. iend
            const int k0 = lane, k1 = lane + 32;
            if (k0 < n) {
                double *Z0 = Z + k0 * n, *Z1 = Z + (k1 < n ? k1 : k0) * n;
                const bool two = k1 < n;
                for (int i = m - 1; i >= iend; i--) {
                    const double c = rot[2 * i], sn = rot[2 * i + 1];
                    const double f0 = Z0[i + 1], g0 = Z0[i];
                    double f1 = 0.0, g1 = 0.0;
                    if (two) { f1 = Z1[i + 1]; g1 = Z1[i]; }
                    Z0[i + 1] = sn * g0 + c * f0;
                    Z0[i] = c * g0 - sn * f0;
                    if (two) {
                        Z1[i + 1] = sn * g1 + c * f1;
                        Z1[i] = c * g1 - sn * f1;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// The eigenpairs of T_m (diagonal d, off-diagonal e, n <= LZ_KMAX) by one block:
// eigenvalues by Sturm counts, all at once, eigenvectors from twisted
// factorisations, one per pair of threads (Dhillon & Parlett, Linear Algebra
// Appl. 387 (2004) 1).  d gets the eigenvalues, column j of Z the unit vector of
// eigenvalue j.  Vectors of close eigenvalues come out orthogonal to rounding
// over their gap only; the caller makes up for that to first order, and where
// U U^T e1 misses e1 by more than 1e-10 (nearly equal eigenvalues) or the input
// is not finite, false is returned and the caller falls back on the QL iteration.
//
// Bound: latency.  The QL recurrence is one chain of about 0.8 n^2 rotations of
// some 100 ns; here a chain is n multiply-adds per bisection step and n divisions
// per factorisation.  m = 40: 230 us by QL, 36 us by this.
constexpr int LZE_THREADS = 512;
constexpr int LZE_TEAM = LZE_THREADS / LZ_KMAX;    // threads per eigenvalue
// doubles of shared memory: d, e, scaled copies, multipliers and vectors
constexpr int LZE_SMEM = 6 * LZ_KMAX + 3 * LZ_KMAX * (LZ_KMAX + 1);

// eigenvalues below x of the tridiagonal matrix with diagonal a and squared
// off-diagonal b2: sign changes of the characteristic polynomials of its leading
// blocks (Givens), rescaled every eight steps.  |a - x| <= 2 by the caller's scaling.
__device__ __forceinline__ int sturm_below(const double *__restrict__ a, const double *__restrict__ b2, int n, double x)
{
    double p0 = 1.0, p1 = a[0] - x;
    bool neg = p1 < 0.0 || p1 == 0.0;          // a zero counts with the sign opposite to its predecessor
    int cnt = neg;
    for (int i = 1; i < n; i++) {
        const double p2 = fma(a[i] - x, p1, -(b2[i - 1] * p0));
        const bool ng = p2 < 0.0 || (p2 == 0.0 && !neg);
        cnt += ng != neg;
        neg = ng;
        p0 = p1;
        p1 = p2;
        if ((i & 7) == 0) {
            const double m = fmax(fabs(p0), fabs(p1));
            if (m < 1e-100) { p0 *= 1e100; p1 *= 1e100; }
        }
    }
    return cnt;
}

__device__ bool block_tridiag_eig(double *d, const double *e, double *a, double *b, double *b2, double *Z, double *Lf,
                                  double *Lb, int n)
{
    constexpr int LD = LZ_KMAX + 1;
    __shared__ double sc[2];
    const int tid = threadIdx.x, lane = tid & 31;
    // shift and scale so that Gershgorin's discs fill [-1, 1]
    if (tid < 32) {
        double lo = 1e300, hi = -1e300;
        bool fin = true;
        for (int i = lane; i < n; i += 32) {
            const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
            lo = fmin(lo, d[i] - r);
            hi = fmax(hi, d[i] + r);
            fin = fin && isfinite(d[i]) && isfinite(r);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        fin = __all_sync(0xffffffffu, fin);
        if (lane == 0) {
            const double h = 0.5 * (hi - lo);
            sc[0] = 0.5 * (hi + lo);
            sc[1] = fin && h > 0.0 && isfinite(h) ? h : 0.0;
        }
    }
    __syncthreads();
    const double mid = sc[0], half = sc[1];
    if (half == 0.0) return false;
    for (int i = tid; i < n; i += LZE_THREADS) {
        a[i] = (d[i] - mid) / half;
        const double bi = i < n - 1 ? e[i] / half : 0.0;
        b[i] = bi;
        b2[i] = bi * bi;
    }
    __syncthreads();
    // eigenvalue k of team k: the bracket shrinks by LZE_TEAM + 1 per round
    const int k = tid / LZE_TEAM, t = tid % LZE_TEAM;
    const int kk = k < n ? k : n - 1;                      // idle teams mirror the last (whole warps stay together)
    double lo = -1.0 - 1e-12, hi = 1.0 + 1e-12;
    const unsigned sh = lane & ~(LZE_TEAM - 1);
    for (int round = 0; round < 17; round++) {             // 9^17 > 2^53
        const double w = (hi - lo) * (1.0 / (LZE_TEAM + 1));
        const double x = lo + (t + 1) * w;
        const bool above = sturm_below(a, b2, n, x) > kk;  // eigenvalue kk lies below x
        const unsigned m = (__ballot_sync(0xffffffffu, above) >> sh) & ((1u << LZE_TEAM) - 1);
        const int f = m ? __ffs(m) - 1 : LZE_TEAM;         // the first point above it
        const double l2 = lo + f * w;
        hi = f < LZE_TEAM ? lo + (f + 1) * w : hi;
        lo = f > 0 ? l2 : lo;
    }
    const double th = 0.5 * (lo + hi);
    // twisted factorisation of T - theta: thread 0 of the team from the top, thread 1 from the bottom
    const double tiny = 1e-18;
    if (k < n && t == 0) {
        double p = a[0] - th;
        for (int i = 0; i < n; i++) {
            if (fabs(p) < tiny) p = p < 0.0 ? -tiny : tiny;
            Lf[i * LD + k] = p;
            if (i + 1 < n) p = (a[i + 1] - th) - b2[i] / p;
        }
    } else if (k < n && t == 1) {
        double p = a[n - 1] - th;
        for (int i = n - 1; i >= 0; i--) {
            if (fabs(p) < tiny) p = p < 0.0 ? -tiny : tiny;
            Lb[i * LD + k] = p;
            if (i > 0) p = (a[i - 1] - th) - b2[i - 1] / p;
        }
    }
    __syncwarp();
    if (k < n && t < 2) {
        // the twist where the pivot is smallest; each thread takes its side of it
        int kt = 0;
        double g = 1e300;
        for (int i = 0; i < n; i++) {
            const double v = fabs(Lf[i * LD + k] + Lb[i * LD + k] - (a[i] - th));
            if (v < g) { g = v; kt = i; }
        }
        double z = 1.0, nz = t == 0 ? 1.0 : 0.0;
        if (t == 0) {
            Z[kt * LD + k] = 1.0;
            for (int i = kt - 1; i >= 0; i--) {
                z *= -b[i] / Lf[i * LD + k];
                Z[i * LD + k] = z;
                nz += z * z;
            }
        } else {
            for (int i = kt + 1; i < n; i++) {
                z *= -b[i - 1] / Lb[i * LD + k];
                Z[i * LD + k] = z;
                nz += z * z;
            }
        }
        const unsigned two = 3u << sh;
        nz += __shfl_xor_sync(two, nz, 1);
        __syncwarp(two);
        const double rn = rsqrt(nz);
        for (int i = t == 0 ? 0 : kt + 1; i < (t == 0 ? kt + 1 : n); i++) Z[i * LD + k] *= rn;
        if (t == 0) d[k] = fma(th, half, mid);
    }
    __syncthreads();
    return true;
}

// y = Z x or Z^T x, a team per entry (n <= LZ_KMAX entries, leading dimension ld), scaled
// and added: y_k = ca c_k + cb sum; every thread of the block takes part
__device__ __forceinline__ void team_matvec(const double *__restrict__ Z, int ld, bool trans, const double *__restrict__ x,
                                            int n, double ca, const double *__restrict__ c, double cb,
                                            double *__restrict__ y)
{
    const int k = threadIdx.x / LZE_TEAM, t = threadIdx.x % LZE_TEAM;
    double v = 0.0;
    if (k < n)
        for (int j = t; j < n; j += LZE_TEAM) v += (trans ? Z[j * ld + k] : Z[k * ld + j]) * x[j];
    for (int o = LZE_TEAM / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (k < n && t == 0) y[k] = ca * c[k] + cb * v;
    __syncthreads();
}

// A check's outcome for one replica, written by the speculative checks.
struct LzSpec {
    int conv;      // converged at m
    int m;
    int fin;       // converged, or already done when the check started
    int pad;
};

// one block per replica: eig of T_m, g = b0 U sqrt(max(theta,0)) U^T e1,
// convergence ||g - g_prev|| <= tol ||g|| (the Lanczos basis is orthonormal).
// final_ = 1: the final estimate, on the replica's own m when it is done, into lz.
// final_ = 0: a speculative check beside the next basis vectors: it reads the
// snapshot `snap` of lz taken when it was launched (the vectors that follow
// move lz on) and writes its outcome into spec; the host applies it later
// (k_lz_spec_apply).  g_prev is the previous check's g in both cases.
__global__ void __launch_bounds__(LZE_THREADS)
k_lz_check(int R, const Seg *__restrict__ segs, LzScal *__restrict__ lz, const LzScal *__restrict__ snap, LzSpec *__restrict__ spec,
           const double *__restrict__ alpha, const double *__restrict__ betad, double *__restrict__ gbuf,
           int m, int cur, double tol, int final_)
{
    pdl_enter();
    extern __shared__ double sm[];
    __shared__ double red[2][2];
    __shared__ int rneg[2];
    const int r = blockIdx.x;
    if (segs[r].indef) return;
    const LzScal L = final_ ? lz[r] : snap[r];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int done = L.done[cur];
    if (!final_ && done) {
        if (tid == 0) spec[r] = LzSpec{0, L.m, 1, 0};
        return;
    }
    const int mr = done ? L.m : m;
    if (mr <= 0) {
        if (!final_ && tid == 0) spec[r] = LzSpec{0, 0, 0, 0};
        return;
    }
    double *d = sm, *e = d + LZ_KMAX, *a = e + LZ_KMAX, *b = a + LZ_KMAX, *b2 = b + LZ_KMAX, *v = b2 + LZ_KMAX;
    double *Z = v + LZ_KMAX, *Lf = Z + LZ_KMAX * (LZ_KMAX + 1), *Lb = Lf + LZ_KMAX * (LZ_KMAX + 1);
    auto load = [&]() {
        for (int i = tid; i < mr; i += LZE_THREADS) {
            d[i] = alpha[(long)LZ_KMAX * r + i];
            e[i] = (i < mr - 1) ? betad[(long)LZ_KMAX * r + i] : 0.0;
        }
        __syncthreads();
    };
    load();
    int ld = LZ_KMAX + 1;
    // v = U^T e1 and a = U v, which is e1 when the vectors are orthonormal
    bool ok = block_tridiag_eig(d, e, a, b, b2, Z, Lf, Lb, mr);
    if (ok) {
        for (int j = tid; j < mr; j += LZE_THREADS) v[j] = Z[j];
        __syncthreads();
        team_matvec(Z, ld, false, v, mr, 0.0, v, 1.0, a);
        bool miss = false;
        for (int i = tid; i < mr; i += LZE_THREADS) miss = miss || !(fabs(a[i] - (i == 0)) <= 1e-10);
        ok = !__syncthreads_or(miss);
    }
    if (!ok) {
        load();
        ld = mr;
        if (wid == 0) {
            warp_tql(d, e, Z, Lf, mr);
            __syncwarp();
            for (int j = lane; j < mr; j += 32) { v[j] = Z[j]; a[j] = j == 0; }
        }
        __syncthreads();
    }
    // f(T) e1 with U (U^T U)^(-1/2) in place of U, to first order in U^T U - I:
    // w = f (3 v - U^T U v) / 2, then U (3 w - U^T U w) / 2
    team_matvec(Z, ld, true, a, mr, 1.5, v, -0.5, b);
    for (int j = tid; j < mr; j += LZE_THREADS) b[j] *= d[j] < 0.0 ? 0.0 : sqrt(d[j]);   // a NaN stays one
    __syncthreads();
    team_matvec(Z, ld, false, b, mr, 0.0, b, 1.0, a);
    team_matvec(Z, ld, true, a, mr, 1.5, b, -0.5, b2);
    team_matvec(Z, ld, false, b2, mr, 0.0, b2, L.b0, a);
    double *g = gbuf + (long)(LZ_KMAX + 1) * r;   // g[0..m-1] of the previous check
    if (tid < LZ_KMAX) {
        const int i = tid;
        const double gi = i < mr ? a[i] : 0.0, old = g[i];
        double diff2 = (gi - old) * (gi - old), nrm2 = gi * gi;
        int nneg = i < mr && d[i] < 0.0;
        if (i < mr) g[i] = gi;
        for (int o = 16; o > 0; o >>= 1) {
            diff2 += __shfl_down_sync(0xffffffffu, diff2, o);
            nrm2 += __shfl_down_sync(0xffffffffu, nrm2, o);
            nneg += __shfl_down_sync(0xffffffffu, nneg, o);
        }
        if (lane == 0) { red[wid][0] = diff2; red[wid][1] = nrm2; rneg[wid] = nneg; }
    }
    __syncthreads();
    if (tid == 0) {
        const int conv = sqrt(red[0][0] + red[1][0]) <= tol * sqrt(red[0][1] + red[1][1]);
        if (final_) {
            lz[r].nneg = rneg[0] + rneg[1];
            if (!done) {
                lz[r].m = mr;
                lz[r].done[cur] = 1;
            }
        } else {
            spec[r] = LzSpec{conv, mr, conv, 0};
        }
    }
}

// k_lz_check for the replicas reps[] that keep their order, one warp per replica: QL, g summed
// eigenvalue by eigenvalue.  eig of T_m, g = b0 U sqrt(max(theta,0)) U^T e1,
// convergence ||g - g_prev|| <= tol ||g|| (the Lanczos basis is orthonormal).
// final_ = 1: the final estimate, on the replica's own m when it is done, into lz.
// final_ = 0: a speculative check beside the next basis vectors: it reads the
// snapshot `snap` of lz taken when it was launched (the vectors that follow
// move lz on) and writes its outcome into spec; the host applies it later
// (k_lz_spec_apply).  g_prev is the previous check's g in both cases.
__global__ void k_lz_check_ql(const int *__restrict__ reps, LzScal *__restrict__ lz, const LzScal *__restrict__ snap, LzSpec *__restrict__ spec,
                           const double *__restrict__ alpha, const double *__restrict__ betad, double *__restrict__ gbuf,
                           int m, int cur, double tol, int final_)
{
    pdl_enter();
    extern __shared__ double sm[];
    const int r = reps[blockIdx.x];
    const LzScal L = final_ ? lz[r] : snap[r];
    const int lane = threadIdx.x;
    const int done = L.done[cur];
    if (!final_ && done) {
        if (lane == 0) spec[r] = LzSpec{0, L.m, 1, 0};
        return;
    }
    int mr = done ? L.m : m;
    if (mr <= 0) {
        if (!final_ && lane == 0) spec[r] = LzSpec{0, 0, 0, 0};
        return;
    }
    double *d = sm, *e = sm + LZ_KMAX, *Z = sm + 2 * LZ_KMAX, *rot = Z + LZ_KMAX * LZ_KMAX;
    for (int i = lane; i < mr; i += 32) {
        d[i] = alpha[(long)LZ_KMAX * r + i];
        e[i] = (i < mr - 1) ? betad[(long)LZ_KMAX * r + i] : 0.0;
    }
    __syncwarp();
    warp_tql(d, e, Z, rot, mr);
    __syncwarp();
    double *g = gbuf + (long)(LZ_KMAX + 1) * r;   // g[0..m-1], g[LZ_KMAX] = |g|^2 of previous
    double diff2 = 0, nrm2 = 0;
    int nneg = 0;
    for (int i = lane; i < LZ_KMAX; i += 32) {
        double gi = 0;
        if (i < mr) {
            for (int j = 0; j < mr; j++) {
                double th = d[j];
                double sq = th < 0.0 ? 0.0 : sqrt(th);      // a NaN stays one
                gi += Z[i * mr + j] * sq * Z[0 * mr + j];
            }
            gi *= L.b0;
        }
        double old = g[i];
        diff2 += (gi - old) * (gi - old);
        nrm2 += gi * gi;
        if (i < mr) g[i] = gi;
    }
    for (int j = lane; j < mr; j += 32) nneg += d[j] < 0.0;
    for (int o = 16; o > 0; o >>= 1) {
        diff2 += __shfl_down_sync(0xffffffffu, diff2, o);
        nrm2 += __shfl_down_sync(0xffffffffu, nrm2, o);
        nneg += __shfl_down_sync(0xffffffffu, nneg, o);
    }
    if (lane == 0) {
        const int conv = sqrt(diff2) <= tol * sqrt(nrm2);
        if (final_) {
            lz[r].nneg = nneg;
            if (!done) {
                lz[r].m = mr;
                lz[r].done[cur] = 1;
            }
        } else {
            spec[r] = LzSpec{conv, mr, conv, 0};
        }
    }
}

// a speculative check's outcome, applied in stream order after the vectors that
// ran beside it: a replica that had converged at m stops there (done, m), as if
// the check had held the vectors back; the vectors it took meanwhile are unused
__global__ void k_lz_spec_apply(int R, LzScal *__restrict__ lz, const LzSpec *__restrict__ spec, int cur)
{
    pdl_enter();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    if (spec[r].conv) { lz[r].done[cur] = 1; lz[r].m = spec[r].m; }
}

// w = V g (top layout)
__global__ void k_lz_combine(RedTable T, const double *__restrict__ V, long ldv, const LzScal *__restrict__ lz,
                             const double *__restrict__ gbuf, double *__restrict__ w)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const int m = lz[B.rep].m;
    const double *g = gbuf + (long)(LZ_KMAX + 1) * B.rep;
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) {
        double acc = 0;
        for (int i = 0; i < m; i++) acc += g[i] * V[(long)i * ldv + B.start + e];
        w[B.start + e] = (lz[B.rep].b0 == 0.0) ? 0.0 : acc;
    }
}

// Orthogonalisation of the replicas that keep the summation order of the reduction table's blocks
// (Seg::indef).  Their far field may be indefinite: about one in ten of the saddle solves that
// their noise drives is close to singular, takes hundreds to thousands of iterations and returns,
// within rtol, whatever the rounding before it selects, so another order of these sums moves
// positions by 1e-9 to 1e-6.  A replica's vector is cut into the table's RB_SPAN blocks, RB_THREADS
// threads form a block's partials, and every sum over blocks runs in block order: both passes of the
// reorthogonalisation (dots against V_0..V_j, then q -= V h), the norm, the breakdown test and the
// next basis vector.  Two forms with the same bits:
//   k_lz_orth_cluster   one launch, a cluster of LZC_CTAS blocks per replica, cluster barriers between the phases,
//                       the cross-block sums read through distributed shared memory and the entries of q held in
//                       registers throughout (1024 colloids 27 us a launch, 30 with q read and written per pass)
//   k_lz_ord_*          four launches over the table
// The clusters are taken while all of a batch's are resident at once, and for replicas of one table block per
// half-block.  Roots of 40 vectors by clusters and by the table, ms, reference pair scalars: 60 beads, 8
// replicas 1.95 and 2.20, 28 replicas 2.35 and 2.38, 36 replicas 2.99 and 2.49, 256 replicas 9.65 and 3.00; 500
// beads, 8 replicas 2.46 and 2.74, 28 replicas 3.26 and 3.24, 36 replicas 3.99 and 3.43, 128 replicas 9.66 and
// 6.11; suspensions, one of 1024 colloids (11 table blocks) 2.62 and 2.92, 28 of 300 4.03 and 3.95; one of 2048
// colloids (22 blocks, two one after the other in some clusters' blocks) 5.6 and 4.7.
constexpr int LZC_CTAS = 8, LZC_HALVES = 2, LZC_THREADS = RB_THREADS * LZC_HALVES;
constexpr int LZC_VB = LZC_CTAS * LZC_HALVES;         // table blocks of a cluster
constexpr int LZC_MAX_REPS = 28;

void lz_ordered_list(Engine &E, std::vector<int> &reps)
{
    bool fit = true;
    for (int r = 0; r < E.R; r++)
        if (E.segs[r].indef) {
            reps.push_back(r);
            fit = fit && E.segs[r].nm3nc11 <= LZC_VB * RB_SPAN;
        }
    E.n_lz_ord = (int)reps.size();
    E.lz_cluster = fit && E.n_lz_ord <= LZC_MAX_REPS;
}

// Partial dots of q (held by the block's threads in qv) against V_0..V_j, one block of the
// table; the last block of the replica sums the partials in block order into h[].
__device__ __forceinline__ void lz_ord_block_dots(const RedTable &T, const RBlk &B, const double *__restrict__ V, long ldv,
                                                  const double (&qv)[RB_EPT], int j, double *__restrict__ part,
                                                  double *__restrict__ h)
{
    __shared__ double sh[RB_THREADS / 32][LZ_KMAX];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // eight basis vectors per pass keep 8 x RB_EPT loads in flight.  Each dot is
    // summed in element order and reduced by the same shuffle tree as one at a time.
    for (int i0 = 0; i0 <= j; i0 += 8) {
        double v[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            v[c] = 0.0;
            if (i0 + c <= j) {
                const double *Vi = V + (long)(i0 + c) * ldv + B.start;
#pragma unroll
                for (int k = 0; k < RB_EPT; k++) {
                    const int e = threadIdx.x + k * RB_THREADS;
                    if (e < B.len) v[c] += Vi[e] * qv[k];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 8; c++) {
            double t = v[c];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0 && i0 + c <= j) sh[wid][i0 + c] = t;
        }
    }
    __syncthreads();
    if (threadIdx.x <= j) {
        double t = 0;
        for (int w = 0; w < RB_THREADS / 32; w++) t += sh[w][threadIdx.x];
        part[(long)LZ_KMAX * RB_EPT * blockIdx.x + threadIdx.x] = t;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = atomicAdd(&T.d_counter[B.rep], 1);
        last = (t == T.d_count[B.rep] - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int f = T.d_first[B.rep], c = T.d_count[B.rep];
    if (threadIdx.x <= j) {
        double t = 0;
        for (int k = 0; k < c; k++) t += ((volatile double *)part)[(long)LZ_KMAX * RB_EPT * (f + k) + threadIdx.x];
        h[(long)LZ_KMAX * B.rep + threadIdx.x] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) T.d_counter[B.rep] = 0;
}

// a table block's entries (thread t of RB_THREADS holds t, t + RB_THREADS, ..) less sum_i h_i V_i, in the
// order i = 0..j per entry; V: the block's part of V_0
__device__ __forceinline__ void lz_ord_subtract(const double *__restrict__ V, long ldv, int len, int t, int j,
                                                const double *__restrict__ h, double (&acc)[RB_EPT])
{
#pragma unroll 4
    for (int i = 0; i <= j; i++) {
        const double hi = h[i];
        const double *Vi = V + (long)i * ldv;
#pragma unroll
        for (int k = 0; k < RB_EPT; k++) {
            const int e = t + k * RB_THREADS;
            if (e < len) acc[k] -= hi * Vi[e];
        }
    }
}

// the thread's part of q.q, entry by entry onto zero (a sum of the four squares alone may be contracted otherwise)
__device__ __forceinline__ double lz_ord_square(int len, int t, const double (&v)[RB_EPT])
{
    double x = 0.0;
#pragma unroll
    for (int k = 0; k < RB_EPT; k++)
        if (t + k * RB_THREADS < len) x += v[k] * v[k];
    return x;
}

// a table block's entries into registers, zero beyond its length, and back
__device__ __forceinline__ void lz_ord_load(const double *__restrict__ q, int len, int t, double (&v)[RB_EPT])
{
#pragma unroll
    for (int k = 0; k < RB_EPT; k++) {
        const int e = t + k * RB_THREADS;
        v[k] = e < len ? q[e] : 0.0;
    }
}
__device__ __forceinline__ void lz_ord_store(double *__restrict__ q, int len, int t, const double (&v)[RB_EPT], double f)
{
#pragma unroll
    for (int k = 0; k < RB_EPT; k++) {
        const int e = t + k * RB_THREADS;
        if (e < len) q[e] = v[k] * f;
    }
}

// h = V_0..V_j dotted with q (first pass of the Gram-Schmidt step)
__global__ void k_lz_ord_dots(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ V, long ldv,
                              const double *__restrict__ q, int j, const LzScal *__restrict__ lz, double *__restrict__ part,
                              double *__restrict__ h)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    if (lz[B.rep].done[j & 1] || !segs[B.rep].indef) return;
    double qv[RB_EPT];
    lz_ord_load(q + B.start, B.len, threadIdx.x, qv);
    lz_ord_block_dots(T, B, V, ldv, qv, j, part, h);
}

// the first pass's subtraction and the second pass's dots in one sweep: alpha_j = h_j, h2 = V_0..V_j
// dotted with the new q, which the block still holds in registers
__global__ void k_lz_ord_sub_dots(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ V, long ldv,
                                  double *__restrict__ q, int j, const LzScal *__restrict__ lz,
                                  const double *__restrict__ h, double *__restrict__ alpha, double *__restrict__ part,
                                  double *__restrict__ h2)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    if (lz[B.rep].done[j & 1] || !segs[B.rep].indef) return;
    const double *hr = h + (long)LZ_KMAX * B.rep;
    double acc[RB_EPT];
    lz_ord_load(q + B.start, B.len, threadIdx.x, acc);
    lz_ord_subtract(V + B.start, ldv, B.len, threadIdx.x, j, hr, acc);
    lz_ord_store(q + B.start, B.len, threadIdx.x, acc, 1.0);
    if (threadIdx.x == 0 && (int)blockIdx.x == T.d_first[B.rep]) alpha[(long)LZ_KMAX * B.rep + j] = 0.0 + hr[j];
    lz_ord_block_dots(T, B, V, ldv, acc, j, part, h2);
}

// the second pass's subtraction, the norm and the breakdown test in one sweep: alpha_j += h2_j, nrm2 = q.q
// summed as the segmented dot sums it; the replica's last block records m = j + 1 and stops the
// replica on an invariant subspace
__global__ void k_lz_ord_sub_norm(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ V, long ldv,
                                  double *__restrict__ q, int j, LzScal *__restrict__ lz, const double *__restrict__ h2,
                                  double *__restrict__ alpha, double *__restrict__ nrm2)
{
    pdl_enter();
    __shared__ double sh[RB_THREADS / 32][1];
    const RBlk B = T.d_blk[blockIdx.x];
    if (!segs[B.rep].indef) return;
    const bool lead = threadIdx.x == 0 && (int)blockIdx.x == T.d_first[B.rep];
    const int done = lz[B.rep].done[j & 1];
    if (done) {
        if (lead) lz[B.rep].done[(j + 1) & 1] = done;
        return;
    }
    const double *hr = h2 + (long)LZ_KMAX * B.rep;
    double acc[RB_EPT];
    lz_ord_load(q + B.start, B.len, threadIdx.x, acc);
    lz_ord_subtract(V + B.start, ldv, B.len, threadIdx.x, j, hr, acc);
    lz_ord_store(q + B.start, B.len, threadIdx.x, acc, 1.0);
    if (lead) alpha[(long)LZ_KMAX * B.rep + j] = alpha[(long)LZ_KMAX * B.rep + j] + hr[j];
    double v[1] = {lz_ord_square(B.len, threadIdx.x, acc)};
    block_sum<1>(v, sh);
    double tot[1];
    if (finish_block<1>(T, B, blockIdx.x, v, tot)) {
        nrm2[B.rep] = tot[0];
        lz[B.rep].m = j + 1;
        lz[B.rep].done[(j + 1) & 1] = sqrt(tot[0]) <= 1e-12 * lz[B.rep].b0 ? 2 : 0;   // 2: finalise with m = j + 1
    }
}

// V_{j+1} = q / ||q||; beta_j = ||q||  (norm from nrm2[rep])
__global__ void k_lz_ord_next(RedTable T, const Seg *__restrict__ segs, double *__restrict__ V, long ldv,
                              const double *__restrict__ q, int j, const LzScal *__restrict__ lz,
                              const double *__restrict__ nrm2, double *__restrict__ betad)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    if (lz[B.rep].done[(j + 1) & 1] || !segs[B.rep].indef) return;
    const double bj = sqrt(nrm2[B.rep]);
    const double inv = bj > 0 ? 1.0 / bj : 0.0;
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) V[(long)(j + 1) * ldv + B.start + e] = q[B.start + e] * inv;
    if (threadIdx.x == 0 && (int)blockIdx.x == T.d_first[B.rep]) betad[(long)LZ_KMAX * B.rep + j] = bj;
}

namespace cgr = cooperative_groups;

__global__ void __cluster_dims__(LZC_CTAS, 1, 1) __launch_bounds__(LZC_THREADS)
k_lz_orth_cluster(const Seg *__restrict__ segs, const int *__restrict__ reps, double *__restrict__ V, long ldv,
                  const double *__restrict__ q, int j, int kmax, LzScal *__restrict__ lz, double *__restrict__ alpha,
                  double *__restrict__ betad)
{
    pdl_enter();
    cgr::cluster_group cl = cgr::this_cluster();
    const int rank = (int)cl.block_rank();
    const int r = reps[blockIdx.x / LZC_CTAS];
    const int half = threadIdx.x / RB_THREADS, t = threadIdx.x % RB_THREADS;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int HW = RB_THREADS / 32;                   // warps per half
    __shared__ double part[2][LZC_HALVES][LZ_KMAX];       // per pass: the table block's partial dots
    __shared__ double npart[LZC_HALVES];                  // ... and partial norms
    __shared__ double sh[LZC_THREADS / 32][8];
    __shared__ double hsh[LZ_KMAX];
    const Seg &s = segs[r];
    const int done = lz[r].done[j & 1];
    if (done) {                                 // the whole cluster
        if (rank == 0 && threadIdx.x == 0) lz[r].done[(j + 1) & 1] = done;
        return;
    }
    const int n = s.nm3nc11, nb = (n + RB_SPAN - 1) / RB_SPAN;
    const int rb = rank * LZC_HALVES + half;              // this half's table block
    const int len = rb < nb ? min(RB_SPAN, n - rb * RB_SPAN) : 0;
    const long st = (long)s.top_off + (long)rb * RB_SPAN;
    double alpha_j = 0.0, qv[RB_EPT];
    lz_ord_load(q + st, len, t, qv);
    for (int pass = 0; pass < 2; pass++) {
        for (int i0 = 0; i0 <= j; i0 += 8) {
            double v[8];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                v[c] = 0.0;
                if (i0 + c <= j) {
                    const double *Vi = V + (long)(i0 + c) * ldv + st;
#pragma unroll
                    for (int k = 0; k < RB_EPT; k++) {
                        const int e = t + k * RB_THREADS;
                        if (e < len) v[c] += Vi[e] * qv[k];
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < 8; c++) {
                double x = v[c];
                for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
                if (lane == 0) sh[wid][c] = x;
            }
            __syncthreads();
            if (t < 8 && i0 + t <= j) {
                double x = 0.0;
                for (int w = 0; w < HW; w++) x += sh[half * HW + w][t];
                part[pass][half][i0 + t] = x;
            }
            __syncthreads();
        }
        cl.sync();
        for (int i = threadIdx.x; i <= j; i += LZC_THREADS) {   // h_i over the table blocks in block order
            double h = 0.0;
            for (int b = 0; b < nb; b++)
                h += cl.map_shared_rank(&part[pass][b % LZC_HALVES][0], b / LZC_HALVES)[i];
            hsh[i] = h;
        }
        __syncthreads();
        lz_ord_subtract(V + st, ldv, len, t, j, hsh, qv);
        alpha_j += hsh[j];
        __syncthreads();
    }
    {                                                          // the block's norm, as seg_dot sums it
        double x = lz_ord_square(len, t, qv);
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[wid][0] = x;
        __syncthreads();
        if (t == 0) {
            double y = 0.0;
            for (int w = 0; w < HW; w++) y += sh[half * HW + w][0];
            npart[half] = y;
        }
    }
    cl.sync();
    double nrm2 = 0.0;
    for (int b = 0; b < nb; b++) nrm2 += cl.map_shared_rank(&npart[b % LZC_HALVES], b / LZC_HALVES)[0];
    cl.sync();                                  // no block leaves while others read its shared memory
    const double bj = sqrt(nrm2);
    const bool broken = bj <= 1e-12 * lz[r].b0;
    if (rank == 0 && threadIdx.x == 0) {
        alpha[(long)LZ_KMAX * r + j] = alpha_j;
        lz[r].m = j + 1;
        lz[r].done[(j + 1) & 1] = broken ? 2 : 0;   // 2, an invariant subspace: finalise with m = j + 1
        if (!broken && j + 1 < kmax) betad[(long)LZ_KMAX * r + j] = bj;
    }
    if (!broken && j + 1 < kmax) lz_ord_store(V + (long)(j + 1) * ldv + st, len, t, qv, bj > 0 ? 1.0 / bj : 0.0);
}

int lanczos_sqrt(Engine &E, const double *z, double *w, const ps_sqrt_opts *o, ps_sqrt_result *res, cudaStream_t st)
{
    int kmax = o && o->kmax > 0 ? o->kmax : 40;
    double tol = o && o->tol > 0 ? o->tol : 1e-6;
    if (kmax > LZ_KMAX) kmax = LZ_KMAX;
    RedTable &T = E.red_top;
    long ldv = E.ntop;
    double *V = E.d_lzV, *q = E.d_lzq;
    LzScal *lz = (LzScal *)E.d_lzs;
    double *alpha = E.d_lzT;                                // [R][LZ_KMAX]
    double *betad = alpha + (long)LZ_KMAX * E.R;            // [R][LZ_KMAX]
    double *gbuf = betad + (long)LZ_KMAX * E.R;             // [R][LZ_KMAX+1]
    double *nrm2 = gbuf + (long)(LZ_KMAX + 1) * E.R;        // [R]
    // sub-block sums of the reorthogonalisation: both passes' dots, the norm
    double *part1 = E.d_lzp, *part2 = part1 + (long)LZ_KMAX * RB_EPT * T.nblk;
    double *npart = part2 + (long)LZ_KMAX * RB_EPT * T.nblk;
    seg_dot(E, T, z, z, nrm2, st);
    ps_launch(k_lz_init, T.nblk, RB_THREADS, 0, st, T, E.d_segs, V, z, lz, nrm2);
    PS_CK(cudaMemsetAsync(gbuf, 0, sizeof(double) * (LZ_KMAX + 1) * E.R, st));
    const int check = 8;   // convergence test every 8 vectors; the cap is handled after the loop
    const bool any_free = E.n_lz_ord < E.R;
    double *h = nrm2 + E.R, *h2 = h + (long)LZ_KMAX * E.R;  // [R][LZ_KMAX]: both passes' dots of the ordered replicas
    const size_t smem = sizeof(double) * LZE_SMEM, smem_ql = sizeof(double) * (4 * LZ_KMAX + LZ_KMAX * LZ_KMAX);
    PS_CK(cudaFuncSetAttribute(k_lz_check, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    std::vector<LzScal> hl(E.R);
    LzScal *snap = lz + E.R;                                 // the scalars when a check was launched
    LzSpec *spec = (LzSpec *)(snap + E.R);                   // the checks' outcomes
    LzSpec *hspec = (LzSpec *)E.h_spec;
    bool pending = false;
    int j = 0, cur = 0;                                      // cur: where done stands, the number of vectors & 1
    for (j = 0; j < kmax; j++) {
        cur = (j + 1) & 1;
        const LzDots dots = {V, ldv, j, part1};
        apply_operator(E, 1, V + (long)j * ldv, q, E.precision == PS_PREC_MIXED, st, &lz[0].done[j & 1],
                       (int)sizeof(LzScal), false, any_free ? &dots : nullptr);
        const dim3 sub((unsigned)T.nblk, (unsigned)T.nsub);
        if (E.n_lz_ord && E.lz_cluster)
            ps_launch(k_lz_orth_cluster, E.n_lz_ord * LZC_CTAS, LZC_THREADS, 0, st, E.d_segs, E.d_lz_ord, V, ldv, q, j, kmax,
                    lz, alpha, betad);
        else if (E.n_lz_ord) {
            // the ordered replicas' blocks leave their part of part2 to these sums
            ps_launch(k_lz_ord_dots, T.nblk, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, lz, part2, h);
            ps_launch(k_lz_ord_sub_dots, T.nblk, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, lz, h, alpha, part2, h2);
            ps_launch(k_lz_ord_sub_norm, T.nblk, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, lz, h2, alpha, nrm2);
            if (j + 1 < kmax)
                ps_launch(k_lz_ord_next, T.nblk, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, lz, nrm2, betad);
        }
        if (any_free) {
            ps_launch(k_lz_sub_dots, sub, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, lz, part1, alpha, part2, npart);
            ps_launch(k_lz_sub_scale, sub, RB_THREADS, 0, st, T, E.d_segs, V, ldv, q, j, kmax, lz, part2, npart, alpha,
                    betad);
        }
        if ((j + 1) % check == 0 && j + 1 < kmax) {
            if (pending) {
                // the previous check (normally finished long before): apply its outcomes
                PS_CK(cudaEventSynchronize(E.ev_chk));
                pending = false;
                ps_launch(k_lz_spec_apply, (E.R + 127) / 128, 128, 0, st, E.R, lz, spec, cur);
                bool all = true;
                for (int r = 0; r < E.R; r++) all &= hspec[r].fin != 0;
                if (all) break;
            }
            // check at m = j + 1 beside the next vectors, on a snapshot of the scalars
            PS_CK(cudaMemcpyAsync(snap, lz, sizeof(LzScal) * E.R, cudaMemcpyDeviceToDevice, st));
            PS_CK(cudaEventRecord(E.ev_fork2, st));
            PS_CK(cudaStreamWaitEvent(E.side2, E.ev_fork2, 0));
            if (any_free)
                ps_launch(k_lz_check, E.R, LZE_THREADS, smem, E.side2, E.R, E.d_segs, lz, snap, spec, alpha, betad, gbuf,
                        j + 1, cur, tol, 0);
            if (E.n_lz_ord)
                ps_launch(k_lz_check_ql, E.n_lz_ord, 32, smem_ql, E.side2, E.d_lz_ord, lz, snap, spec, alpha, betad, gbuf, j + 1,
                        cur, tol, 0);
            PS_CK(cudaMemcpyAsync(hspec, spec, sizeof(LzSpec) * E.R, cudaMemcpyDeviceToHost, E.side2));
            PS_CK(cudaEventRecord(E.ev_chk, E.side2));
            pending = true;
        }
    }
    if (pending) {
        // the last check's outcomes, and its g, ahead of the final estimate
        PS_CK(cudaStreamWaitEvent(st, E.ev_chk, 0));
        ps_launch(k_lz_spec_apply, (E.R + 127) / 128, 128, 0, st, E.R, lz, spec, cur);
    }
    // final estimate: replicas at the cap, replicas stopped by breakdown, and the converged ones on their own m
    if (any_free)
        ps_launch(k_lz_check, E.R, LZE_THREADS, smem, st, E.R, E.d_segs, lz, snap, spec, alpha, betad, gbuf,
                std::min(j + 1, kmax), cur, tol, 1);
    if (E.n_lz_ord)
        ps_launch(k_lz_check_ql, E.n_lz_ord, 32, smem_ql, st, E.d_lz_ord, lz, snap, spec, alpha, betad, gbuf,
                std::min(j + 1, kmax), cur, tol, 1);
    ps_launch(k_lz_combine, T.nblk, RB_THREADS, 0, st, T, V, ldv, lz, gbuf, w);
    PS_CK(cudaMemcpyAsync(hl.data(), lz, sizeof(LzScal) * E.R, cudaMemcpyDeviceToHost, st));
    PS_CK(cudaStreamSynchronize(st));
    PS_CK(cudaGetLastError());
    if (res) {
        res->iters_max = 0; res->nneg = 0;
        for (auto &l : hl) { res->iters_max = std::max(res->iters_max, l.m); res->nneg += l.nneg; }
    }
    return PS_OK;
}

// ---------------------------------------------------------------------------
// Schur Lanczos noise of the shell (arrowhead) path above the dense Schur limit,
// schur_sqrt_lanczos (slip_vel.cpp:351-477): sqrt(S) xi_c with
// S q = Mcc q - beta Mcm (Mcm^T q) applied matrix-free through two mobility
// applies per vector ([0; q] gives Mcm^T q in the monomer rows and Mcc q in the
// colloid rows; [Mcm^T q; 0] gives Mcm Mcm^T q in the colloid rows), at most
// min(40, nc11) vectors, two-pass reorthogonalisation against the whole basis,
// stop on an invariant subspace (||w|| <= 1e-12 ||xi_c||) or the cap, then the
// square root of the projected tridiagonal with negative eigenvalues floored at
// 0.  One block per such replica for the short vectors (length nc11).
struct SlScal {
    double b0;
    int m, done, nneg, pad;
};
constexpr int SL_THREADS = 256;

// sum over the block in a fixed order (thread-strided partials, shuffle tree, warp order)
__device__ double sl_block_sum(double v)
{
    __shared__ double ws[SL_THREADS / 32];
    __shared__ double tot;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) ws[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < SL_THREADS / 32; w++) t += ws[w];
        tot = t;
    }
    __syncthreads();
    double r = tot;
    __syncthreads();
    return r;
}

__device__ double sl_dot(const double *a, const double *b, int n)
{
    double acc = 0;
    for (int i = threadIdx.x; i < n; i += SL_THREADS) acc += a[i] * b[i];
    return sl_block_sum(acc);
}

// V_0 = xi_c / ||xi_c||
__global__ void k_sl_init(const Seg *__restrict__ segs, const int *__restrict__ reps, const double *__restrict__ fb,
                          double *__restrict__ V, SlScal *__restrict__ sc, int *__restrict__ skip)
{
    pdl_enter();
    const int slot = blockIdx.x, r = reps[slot];
    const Seg &s = segs[r];
    const int n = s.nc11;
    const double *b = fb + s.top_off + s.nm3;
    const double b0 = sqrt(sl_dot(b, b, n));
    double *V0 = V + s.sl_off;
    const double inv = b0 > 0 ? 1.0 / b0 : 0.0;
    for (int i = threadIdx.x; i < n; i += SL_THREADS) V0[i] = b[i] * inv;
    if (threadIdx.x == 0) {
        sc[slot].b0 = b0; sc[slot].m = 0; sc[slot].nneg = 0; sc[slot].done = (b0 == 0.0);
        skip[r] = (b0 == 0.0);
    }
}

// u = [0 ; V_j] (stage 0) or u = [y_m ; 0] (stage 1) on the Lanczos replicas, 0 elsewhere
__global__ void k_sl_load(long ntop, const int *__restrict__ top_offs, int R, const Seg *__restrict__ segs,
                          const double *__restrict__ V, const SlScal *__restrict__ sc, int j, int stage,
                          const double *__restrict__ y, double *__restrict__ u)
{
    pdl_enter();
    long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ntop) return;
    int lo = 0, hi = R;
    while (hi - lo > 1) { int mid = (lo + hi) >> 1; if (top_offs[mid] <= k) lo = mid; else hi = mid; }
    const Seg &s = segs[lo];
    const int i = (int)(k - s.top_off);
    double v = 0.0;
    if (s.sl_slot >= 0 && !sc[s.sl_slot].done) {
        if (stage == 0) { if (i >= s.nm3) v = V[s.sl_off + (long)j * s.nc11 + (i - s.nm3)]; }
        else if (i < s.nm3) v = y[k];
    }
    u[k] = v;
}

// one Lanczos vector: w = S V_j - beta_{j-1} V_{j-1}, alpha_j, two reorthogonalisation passes,
// beta_j and V_{j+1} (row j+1 of the basis holds w while it is formed)
__global__ void k_sl_iter(const Seg *__restrict__ segs, const int *__restrict__ reps, double *__restrict__ V,
                          double *__restrict__ ab, SlScal *__restrict__ sc, int *__restrict__ skip,
                          const double *__restrict__ y, const double *__restrict__ y2, int j)
{
    pdl_enter();
    const int slot = blockIdx.x, r = reps[slot];
    if (sc[slot].done) return;
    const Seg &s = segs[r];
    const int n = s.nc11;
    double *Vb = V + s.sl_off;
    double *w = Vb + (long)(j + 1) * n;
    double *alpha = ab + (long)2 * SL_KMAX * slot, *betad = alpha + SL_KMAX;
    const double *yc = y + s.top_off + s.nm3, *y2c = y2 + s.top_off + s.nm3;
    for (int i = threadIdx.x; i < n; i += SL_THREADS) {
        double v = yc[i] - s.beta * y2c[i];
        if (j > 0) v -= betad[j - 1] * Vb[(long)(j - 1) * n + i];
        w[i] = v;
    }
    __syncthreads();
    const double *Vj = Vb + (long)j * n;
    const double aj = sl_dot(Vj, w, n);
    for (int i = threadIdx.x; i < n; i += SL_THREADS) w[i] -= aj * Vj[i];
    __syncthreads();
    for (int pass = 0; pass < 2; pass++)
        for (int l = 0; l <= j; l++) {
            const double *Vl = Vb + (long)l * n;
            const double h = sl_dot(Vl, w, n);
            for (int i = threadIdx.x; i < n; i += SL_THREADS) w[i] -= h * Vl[i];
            __syncthreads();
        }
    const double bj = sqrt(sl_dot(w, w, n));
    const int kmax = n < SL_KMAX ? n : SL_KMAX;
    const bool stop = (bj <= 1e-12 * sc[slot].b0) || (j == kmax - 1);
    if (!stop) {
        const double inv = 1.0 / bj;
        for (int i = threadIdx.x; i < n; i += SL_THREADS) w[i] *= inv;
    }
    if (threadIdx.x == 0) {
        alpha[j] = aj;
        sc[slot].m = j + 1;
        if (stop) { sc[slot].done = 1; skip[r] = 1; }
        else betad[j] = bj;
    }
}

// W_m = sqrt(beta_inv) xi_m; W_c = sqrt(beta) (Mcm xi_m) + b0 V U sqrt(max(theta, 0)) U^T e1
__global__ void k_sl_finish(const Seg *__restrict__ segs, const int *__restrict__ reps, const double *__restrict__ V,
                            const double *__restrict__ ab, SlScal *__restrict__ sc, const double *__restrict__ fb,
                            const double *__restrict__ ymcm, double *__restrict__ W)
{
    pdl_enter();
    __shared__ double d[SL_KMAX], e[SL_KMAX], Z[SL_KMAX * SL_KMAX], g[SL_KMAX], rot[2 * SL_KMAX];
    const int slot = blockIdx.x, r = reps[slot];
    const Seg &s = segs[r];
    const int n = s.nc11, m = sc[slot].m;
    const double b0 = sc[slot].b0;
    for (int i = threadIdx.x; i < s.nm3; i += blockDim.x) W[s.top_off + i] = sqrt(s.beta_inv) * fb[s.top_off + i];
    const double *alpha = ab + (long)2 * SL_KMAX * slot, *betad = alpha + SL_KMAX;
    if (m > 0 && threadIdx.x < 32) {
        for (int i = threadIdx.x; i < m; i += 32) { d[i] = alpha[i]; e[i] = (i < m - 1) ? betad[i] : 0.0; }
        __syncwarp();
        warp_tql(d, e, Z, rot, m);
        __syncwarp();
        int nneg = 0;
        for (int i = threadIdx.x; i < m; i += 32) {
            double gi = 0;
            for (int c = 0; c < m; c++) gi += Z[i * m + c] * (d[c] > 0 ? sqrt(d[c]) : 0.0) * Z[c];
            g[i] = b0 * gi;
            nneg += d[i] < 0.0;
        }
        for (int o = 16; o > 0; o >>= 1) nneg += __shfl_down_sync(0xffffffffu, nneg, o);
        if (threadIdx.x == 0) sc[slot].nneg = nneg;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double acc = sqrt(s.beta) * ymcm[s.top_off + s.nm3 + i];
        for (int c = 0; c < m; c++) acc += g[c] * V[s.sl_off + (long)c * n + i];
        W[s.top_off + s.nm3 + i] = acc;
    }
}

int schur_lanczos_noise(Engine &E, const double *fb, const double *ymcm, double *W, int *nneg, cudaStream_t st)
{
    if (!E.n_sl_reps) return PS_OK;
    SlScal *sc = (SlScal *)E.d_sl_sc;
    const int ns = E.n_sl_reps;
    int kmax = 0;
    for (auto &s : E.segs)
        if (s.sl_slot >= 0) kmax = std::max(kmax, std::min(s.nc11, SL_KMAX));
    ps_launch(k_sl_init, ns, SL_THREADS, 0, st, E.d_segs, E.d_sl_reps, fb, E.d_slV, sc, E.d_sl_skip);
    const int thr = 256;
    const unsigned gb = (unsigned)((E.ntop + thr - 1) / thr);
    for (int j = 0; j < kmax; j++) {
        ps_launch(k_sl_load, gb, thr, 0, st, E.ntop, E.d_top_offs, E.R, E.d_segs, E.d_slV, sc, j, 0,
                nullptr, E.d_sl_u);
        apply_operator(E, 1, E.d_sl_u, E.d_sl_y, false, st, E.d_sl_skip, (int)sizeof(int));
        ps_launch(k_sl_load, gb, thr, 0, st, E.ntop, E.d_top_offs, E.R, E.d_segs, E.d_slV, sc, j, 1,
                E.d_sl_y, E.d_sl_u);
        apply_operator(E, 1, E.d_sl_u, E.d_sl_y2, false, st, E.d_sl_skip, (int)sizeof(int));
        ps_launch(k_sl_iter, ns, SL_THREADS, 0, st, E.d_segs, E.d_sl_reps, E.d_slV, E.d_slT, sc,
                E.d_sl_skip, E.d_sl_y, E.d_sl_y2, j);
    }
    ps_launch(k_sl_finish, ns, SL_THREADS, 0, st, E.d_segs, E.d_sl_reps, E.d_slV, E.d_slT, sc, fb, ymcm, W);
    // the operator applies of the next noise draw start from the Lanczos set again
    std::vector<int> skip(E.R, 1);
    for (auto &s : E.segs)
        if (s.sl_slot >= 0) skip[&s - &E.segs[0]] = 0;
    PS_CK(cudaMemcpyAsync(E.d_sl_skip, skip.data(), sizeof(int) * E.R, cudaMemcpyHostToDevice, st));
    std::vector<SlScal> hs(ns);
    PS_CK(cudaMemcpyAsync(hs.data(), sc, sizeof(SlScal) * ns, cudaMemcpyDeviceToHost, st));
    PS_CK(cudaStreamSynchronize(st));
    PS_CK(cudaGetLastError());
    if (nneg) { *nneg = 0; for (auto &h : hs) *nneg += h.nneg; }
    return PS_OK;
}
}  // namespace ps
