// solve.cu -- structured saddle solves (PS_SOLVE_STRUCTURED).
//
// The saddle system of the reference (arrays.cpp:349-408, matfree_A.cpp:38-80)
//     [ M    B    ] [F]   [b_top]        B = [-I_{nm3nc6} ; 0]
//     [ B^T  -R   ] [U] = [b_bot]        R = R_lub (0 without lubrication)
// splits F = [F_t ; F_S] (forces/torques of every bead, then colloid stresslets).
//
// Without lubrication it is solved exactly by block elimination:
//     F_t = -b_bot                          (constraint rows)
//     M_SS F_S = b_S - M_St F_t             (dense nc5 x nc5 colloid-stresslet solve)
//     U = (M F)_t - b_t                     (velocity rows)
// which costs two operator applies instead of a Krylov iteration.  The solution
// is the same one MINRES converges to (it is the unique solution of the system).
//
// With lubrication the constraint rows couple U to the forces through R_lub;
// the system is solved in pair space by preconditioned CG (pair_solve below),
// with the same exact elimination of the stresslets and velocities around it.
//
// Replicas with more than 12 colloids (M_SS not solved densely) keep the
// stresslets as CG unknowns in the same solve.  Replicas whose CG breaks down
// because M is not positive definite (the reference's own monomer pair scalars
// make it indefinite) take the result as the warm start of a MINRES polish.
#include <cmath>
#include <curand_kernel.h>
#include <vector>
#include "ps_internal.h"
#include "ps_kernels.h"
#include "ps_reduce.cuh"
#include "lub_dev.cuh"

namespace ps {

constexpr int SS_MAX = 64;   // dense stresslet block limit (nc5 <= 64: up to 12 colloids)

__device__ __forceinline__ int rep_at(const int *__restrict__ offs, int R, long k)
{
    int lo = 0, hi = R;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (offs[mid] <= k) lo = mid; else hi = mid;
    }
    return lo;
}

// x = [F_t = -b_bot ; F_S = 0 ; U = 0]
__global__ void k_struct_init(long nvec, const int *__restrict__ vec_offs, int R, const Seg *__restrict__ segs,
                              const double *__restrict__ b, double *__restrict__ x)
{
    pdl_enter();
    long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nvec) return;
    int r = rep_at(vec_offs, R, k);
    const Seg &s = segs[r];
    int i = (int)(k - s.vec_off);
    x[k] = (i < s.nm3nc6) ? -b[s.vec_off + s.nm3nc11 + i] : 0.0;
}

// entry (i, j) of M_SS: self + colloid pair stresslet blocks + the Schur
// correction of the shell path
__device__ double ss_entry(const Seg &s, const double *__restrict__ pos_x, const double *__restrict__ delta, int i, int j)
{
    double v = 0.0;
    int ci = i / 5, pi = i % 5, cj = j / 5, pj = j % 5;
    if (ci == cj) {
        if (pi == pj) v = 1.8;
        else if ((pi == 0 && pj == 4) || (pi == 4 && pj == 0)) v = 0.9;
    } else {
        bool lo = ci < cj;
        long bl = (long)s.bead_off + s.Nm + (lo ? ci : cj), bh = (long)s.bead_off + s.Nm + (lo ? cj : ci);
        double dx = pos_x[3 * bl] - pos_x[3 * bh], dy = pos_x[3 * bl + 1] - pos_x[3 * bh + 1];
        double dz = pos_x[3 * bl + 2] - pos_x[3 * bh + 2];
        double r2 = dx * dx + dy * dy + dz * dz, ri = rsqrt(r2);
        double e[3] = {dx * ri, dy * ri, dz * ri};
        double ri3 = ri * ri * ri, ri5 = ri3 * ri * ri;
        double Mm[25];
        mm_flat<double>(e, -4.5 * ri3 + 10.8 * ri5, 2.25 * ri3 - 7.2 * ri5, 1.8 * ri5, Mm);
        // row of the lower colloid uses Mm, row of the upper one Mm^T (mob.cpp:1129-1143)
        v = lo ? Mm[pi * 5 + pj] : Mm[pj * 5 + pi];
    }
    if (s.shell_schur) v += delta[s.schur_off + (long)(s.nc6 + i) * s.nc11 + (s.nc6 + j)];
    return v;
}

// One block per replica with colloids: assemble M_SS, solve M_SS F_S = b_S - y_S by Gauss-Jordan
// elimination with partial pivoting (the pivots' sizes compared to 2^-20).
//
// Bound: latency.  Rows stay in place, every warp finds the pivot row itself from the
// column's leading words, and each step takes every other row's column out, so a step has
// one barrier and no back substitution follows: 11.1 -> 6.4 us with two colloids (n = 10),
// 6.2 -> 3.8 us with one, against a pivot search and a back substitution on one thread.
__global__ void k_struct_ss(const Seg *__restrict__ segs, const int *__restrict__ reps, const double *__restrict__ pos_x,
                            const double *__restrict__ delta, const double *__restrict__ b,
                            const double *__restrict__ y, double *__restrict__ x)
{
    pdl_enter();
    __shared__ double A[SS_MAX][SS_MAX + 1];
    __shared__ int prow[SS_MAX];
    const int r = reps[blockIdx.x];
    const Seg &s = segs[r];
    const int n = s.nc5, lane = threadIdx.x & 31;
    const int i0 = threadIdx.x / (n + 1), j0 = threadIdx.x % (n + 1), di = blockDim.x / (n + 1), dj = blockDim.x % (n + 1);
    for (int i = i0, j = j0; i < n;) {
        A[i][j] = (j == n) ? b[s.vec_off + s.nm3nc6 + i] - y[s.vec_off + s.nm3nc6 + i] : ss_entry(s, pos_x, delta, i, j);
        i += di; j += dj;
        if (j > n) { j -= n + 1; i++; }
    }
    bool used[SS_MAX / 32] = {};                  // of rows lane, lane + 32, ..
    for (int k = 0; k < n; k++) {
        __syncthreads();
        unsigned key[SS_MAX / 32], best = 0;
#pragma unroll
        for (int c = 0; c < SS_MAX / 32; c++) {
            const int i = 32 * c + lane;
            key[c] = i < n && !used[c] ? 1u + (unsigned)(__double2hiint(A[i][k]) & 0x7fffffff) : 0u;
            best = max(best, key[c]);
        }
        best = __reduce_max_sync(0xffffffffu, best);
        int p = -1;
#pragma unroll
        for (int c = 0; c < SS_MAX / 32; c++) {
            const unsigned hit = __ballot_sync(0xffffffffu, key[c] == best);
            if (p < 0 && hit) {
                p = 32 * c + __ffs(hit) - 1;
                used[c] = used[c] || lane == __ffs(hit) - 1;
            }
        }
        if (threadIdx.x == 0) prow[k] = p;
        const double inv = 1.0 / A[p][k];
        for (int i = i0, j = j0; i < n;) {
            if (j > k && i != p) A[i][j] -= A[i][k] * inv * A[p][j];
            i += di; j += dj;
            if (j > n) { j -= n + 1; i++; }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) x[s.vec_off + s.nm3nc6 + k] = A[prow[k]][n] / A[prow[k]][k];
}

// U = (M F)_t - b_t
__global__ void k_struct_u(long nvec, const int *__restrict__ vec_offs, int R, const Seg *__restrict__ segs,
                           const double *__restrict__ b, const double *__restrict__ y, double *__restrict__ x)
{
    pdl_enter();
    long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nvec) return;
    int r = rep_at(vec_offs, R, k);
    const Seg &s = segs[r];
    int i = (int)(k - s.vec_off);
    if (i >= s.nm3nc11) {
        int j = i - s.nm3nc11;
        x[k] = y[s.vec_off + j] - b[s.vec_off + j];
    }
}

// ---------------------------------------------------------------------------
// lubricated resistance-form PCG

// inverse of M_SS per replica (LU with partial pivoting in shared memory, then
// one column of the inverse per thread); stored row-major at ssinv + s.ss_off
__global__ void k_ss_inverse(const Seg *__restrict__ segs, const int *__restrict__ reps, const double *__restrict__ pos_x,
                             const double *__restrict__ delta, double *__restrict__ ssinv)
{
    pdl_enter();
    __shared__ double A[SS_MAX][SS_MAX + 1];
    __shared__ int perm[SS_MAX];
    __shared__ int piv;
    const Seg &s = segs[reps[blockIdx.x]];
    const int n = s.nc5;
    for (int t = threadIdx.x; t < n * n; t += blockDim.x) A[t / n][t % n] = ss_entry(s, pos_x, delta, t / n, t % n);
    for (int t = threadIdx.x; t < n; t += blockDim.x) perm[t] = t;
    __syncthreads();
    for (int k = 0; k < n; k++) {
        if (threadIdx.x == 0) {
            int p = k;
            double best = fabs(A[k][k]);
            for (int i = k + 1; i < n; i++)
                if (fabs(A[i][k]) > best) { best = fabs(A[i][k]); p = i; }
            piv = p;
            if (p != k) { int t = perm[k]; perm[k] = perm[p]; perm[p] = t; }
        }
        __syncthreads();
        if (piv != k)
            for (int j = threadIdx.x; j < n; j += blockDim.x) { double t = A[k][j]; A[k][j] = A[piv][j]; A[piv][j] = t; }
        __syncthreads();
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) A[i][k] /= A[k][k];
        __syncthreads();
        for (int t = threadIdx.x; t < (n - k - 1) * (n - k - 1); t += blockDim.x) {
            int i = k + 1 + t / (n - k - 1), j = k + 1 + t % (n - k - 1);
            A[i][j] -= A[i][k] * A[k][j];
        }
        __syncthreads();
    }
    // column c of the inverse: solve L U x = P e_c
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        double xv[SS_MAX];
        for (int i = 0; i < n; i++) {
            double v = (perm[i] == c) ? 1.0 : 0.0;
            for (int j = 0; j < i; j++) v -= A[i][j] * xv[j];
            xv[i] = v;
        }
        for (int i = n - 1; i >= 0; i--) {
            double v = xv[i];
            for (int j = i + 1; j < n; j++) v -= A[i][j] * xv[j];
            xv[i] = v / A[i][i];
        }
        for (int i = 0; i < n; i++) ssinv[s.ss_off + (long)i * n + c] = xv[i];
    }
}

// out_S = M_SS^{-1} (ca a_S + cb b_S), one block per replica with a dense
// stresslet block; layouts: 0 saddle vector, 1 mobility vector
__global__ void k_ss_apply(const Seg *__restrict__ segs, const int *__restrict__ reps, const double *__restrict__ ssinv,
                           const double *__restrict__ a, int la, double ca, const double *__restrict__ b, int lb,
                           double cb, double *__restrict__ out, int lo, const char *__restrict__ done, int dstride)
{
    pdl_enter();
    __shared__ double in[SS_MAX];
    const int r = reps[blockIdx.x];
    if (done && *(const int *)(done + (long)r * dstride)) return;
    const Seg &s = segs[r];
    const int n = s.nc5;
    const long oa = (la == 0 ? s.vec_off : s.top_off) + s.nm3nc6, ob = (lb == 0 ? s.vec_off : s.top_off) + s.nm3nc6;
    const long oo = (lo == 0 ? s.vec_off : s.top_off) + s.nm3nc6;
    for (int i = threadIdx.x; i < n; i += blockDim.x) in[i] = ca * a[oa + i] + (b ? cb * b[ob + i] : 0.0);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double *row = ssinv + s.ss_off + (long)i * n;
        double v = 0.0;
        for (int j = 0; j < n; j++) v += row[j] * in[j];
        out[oo + i] = v;
    }
}

// reference norm ||D^{-1} b|| over the saddle vector; initial scalars; all R replicas active
__global__ void k_pcg_start(RedTable T, const double *__restrict__ b, const double *__restrict__ D, PcgScal *pc,
                            double rtol, int R, int *__restrict__ nactive)
{
    pdl_enter();
    __shared__ double sh[RB_THREADS / 32][1];
    const RBlk B = T.d_blk[blockIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 0) *nactive = R;
    double v[1] = {0.0};
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) {
        double t = b[B.start + e] / D[B.start + e];
        v[0] += t * t;
    }
    block_sum<1>(v, sh);
    double tot[1];
    if (finish_block<1>(T, B, blockIdx.x, v, tot)) {
        PcgScal p = {};
        p.tol = rtol * sqrt(tot[0]);
        pc[B.rep] = p;
    }
}

// ---------------------------------------------------------------------------
// Lubricated solve in pair space.  With R = L L^T, L = [B_p K_p^{1/2}] over the
// near pairs p (K_p the 12x12 pair block, B_p its velocity DOFs), the force
// unknowns are F_t = -b_bot + L y, and y solves the SPD system
//     (I + L^T Mr L) y = L^T (g + Mr b_bot),
// of dimension 12 per pair (from (I + R Mr) F_t = R g - b_bot: F_t + b_bot lies
// in the range of R; no term of the right-hand side carries the pair stiffness,
// so the FP32 far field is not amplified by it).  CG is preconditioned
// block-diagonally with (I + K_p^{1/2} M_pp K_p^{1/2})^{-1}, M_pp the pair's own
// two-body FT mobility (self + pair blocks of the far field): the stiff squeeze
// and shear modes of each near pair are resolved by its block, the far-field
// coupling by CG.  After the solve U = Mr F_t - g exactly, so the saddle
// residual is [0 ; 0 ; L r_y]: CG stops on ||D^{-1} L r_y|| <= rtol ||D^{-1} b||,
// the MINRES test of the same system.
//
// Replicas with more than 12 colloids (no dense M_SS inverse) keep the
// stresslets as unknowns beside y: with F_t = -b_bot + L y the system in (y, F_S)
//     [ I + L^T M_tt L   L^T M_tS ] [ y  ]   [ L^T (b_tt + M_tt b_bot) ]
//     [ M_St L           M_SS     ] [F_S ] = [ b_S + M_St b_bot        ]
// is SPD too (J + P^T M P with P = diag(L, I)); each iteration costs one plain M
// apply, the stresslet part is preconditioned by the inverse self block, and the
// saddle residual is [0 ; r_S ; L r_y].  This covers colloid suspensions of any
// size, with or without lubrication.
//
// Pair vectors hold 12 entries per canonical pair q (monomer pairs use the
// first 6).

constexpr int PS_THREADS = 64;

// per-replica done flag at done + r * stride (CG or MINRES scalars); null: none done
__device__ __forceinline__ bool rep_done(const char *done, int stride, int r)
{
    return done && *(const int *)(done + (long)r * stride);
}

// shared-memory scratch of one warp for one colloid pair
struct PsWarpSmem {
    double K[144], Q[144], S[144], M[144];
};

// One colloid pair (lo, hi) by one warp: S = K^{1/2} of the R_lub pair block in
// closed form (colloid_pair_sqrt_coeffs), M = two-body FT far-field mobility
// (symmetrised), P = (I + S M S)^{-1} by Cholesky, identity if not positive
// definite.  Every matrix-product entry sums over k in ascending order.
__device__ void ps_setup_colloid_pair(const Seg &s, long lo, long hi, const double *__restrict__ x,
                                      const double *__restrict__ tab, int nrow, double *__restrict__ So,
                                      double *__restrict__ Po, PsWarpSmem &w, int lane)
{
    double *K = w.K, *Q = w.Q, *S = w.S, *M = w.M;
    for (int t = lane; t < 144; t += 32) { S[t] = 0.0; M[t] = 0.0; }
    __syncwarp();
    {
        double d[3], f[10], kc[10], g[10];
        lub_pair_geom(s, x, tab, nrow, lo, hi, 1.0, d, f);
        lub_pair_coeffs(f, 1.0, kc);
        colloid_pair_sqrt_coeffs(kc, g);
        if (lane < 9) pair_block_entries(d, g, false, lane / 3, lane % 3, S);
    }
    if (lane < 12) {
        // the partner's (F, T) column -> this bead's (U, W) rows, e = (x_lo - x_hi)/r as in the BB kernel
        const double dx = x[3 * lo] - x[3 * hi], dy = x[3 * lo + 1] - x[3 * hi + 1], dz = x[3 * lo + 2] - x[3 * hi + 2];
        const double r2 = dx * dx + dy * dy + dz * dz, rinv = 1.0 / sqrt(r2), r = r2 * rinv;
        const double e[3] = {dx * rinv, dy * rinv, dz * rinv};
        M[lane * 12 + lane] = lane < 6 ? 1.0 : 0.75;
        const bool is_lo = lane < 6;
        const int c = lane % 6;
        const int rowU = is_lo ? 0 : 3, rowW = is_lo ? 6 : 9, colF = is_lo ? 3 : 0, colT = is_lo ? 9 : 6;
        double in[11], out[11];
        for (int k = 0; k < 11; k++) { in[k] = 0.0; out[k] = 0.0; }
        in[c] = 1.0;
        bb_apply<double>(e, r, rinv, is_lo, in, out);
        const int col = c < 3 ? colF + c : colT + (c - 3);
        for (int a = 0; a < 3; a++) { M[(rowU + a) * 12 + col] = out[a]; M[(rowW + a) * 12 + col] = out[3 + a]; }
    }
    __syncwarp();
    for (int t = lane; t < 144; t += 32) {
        const int a = t / 12, c = t % 12;
        if (c > a) {
            const double v = 0.5 * (M[a * 12 + c] + M[c * 12 + a]);
            M[a * 12 + c] = v; M[c * 12 + a] = v;
        }
    }
    __syncwarp();
    for (int t = lane; t < 144; t += 32) {          // K <- M S
        const int a = t / 12, c = t % 12;
        double v = 0.0;
        for (int k = 0; k < 12; k++) v += M[a * 12 + k] * S[k * 12 + c];
        K[t] = v;
    }
    __syncwarp();
    for (int t = lane; t < 144; t += 32) {          // Q <- I + S M S
        const int a = t / 12, c = t % 12;
        double v = (a == c) ? 1.0 : 0.0;
        for (int k = 0; k < 12; k++) v += S[a * 12 + k] * K[k * 12 + c];
        Q[t] = v;
    }
    __syncwarp();
    bool ok = true;
    for (int j = 0; j < 12; j++) {                  // Cholesky Q = C C^T in place (lower)
        double dj = Q[j * 12 + j];
        for (int k = 0; k < j; k++) dj -= Q[j * 12 + k] * Q[j * 12 + k];
        if (!(dj > 0)) { ok = false; break; }
        dj = sqrt(dj);
        const int i = j + 1 + lane;
        double v = 0.0;
        if (i < 12) {
            v = Q[i * 12 + j];
            for (int k = 0; k < j; k++) v -= Q[i * 12 + k] * Q[j * 12 + k];
        }
        __syncwarp();
        if (lane == 0) Q[j * 12 + j] = dj;
        if (i < 12) Q[i * 12 + j] = v / dj;
        __syncwarp();
    }
    for (int t = lane; t < 144; t += 32) So[t] = S[t];
    if (!ok) {
        for (int t = lane; t < 144; t += 32) Po[t] = (t / 12 == t % 12) ? 1.0 : 0.0;
        __syncwarp();
        return;
    }
    if (lane < 12) {                                // P = Q^{-1}, column `lane`
        const int c = lane;
        double v[12];
        for (int i = 0; i < 12; i++) {
            double t = (i == c) ? 1.0 : 0.0;
            for (int k = 0; k < i; k++) t -= Q[i * 12 + k] * v[k];
            v[i] = t / Q[i * 12 + i];
        }
        for (int i = 11; i >= 0; i--) {
            double t = v[i];
            for (int k = i + 1; k < 12; k++) t -= Q[k * 12 + i] * v[k];
            v[i] = t / Q[i * 12 + i];
        }
        for (int i = 0; i < 12; i++) Po[i * 12 + c] = v[i];
    }
    __syncwarp();
}

// per pair: S = K^{1/2} and P = (I + S M_pp S)^{-1} (identity if not positive
// definite); each pair owns a 144-double slot in S and in P.  Monomer pairs: one
// thread each, closed form, compact 6 x 6 blocks (row stride 6).  Colloid pairs:
// one warp per colloid in the blocks past the pair blocks, taking the canonical
// pairs for which it is the lower bead (ps_setup_colloid_pair), 12 x 12 blocks.
// Where every bead is a colloid (warp_pairs), one warp per pair instead (1024
// colloids: 105 -> 22 us).
__global__ void __launch_bounds__(PS_THREADS)
k_ps_setup(long npair, const int2 *__restrict__ pairs, const int *__restrict__ bead_offs, int R,
           const Seg *__restrict__ segs, const double *__restrict__ x, const double *__restrict__ chain,
           const double *__restrict__ tab, int nrow, long ncoll, const int *__restrict__ coll_rep,
           const int *__restrict__ cptr, double *__restrict__ Sout, double *__restrict__ Pout, int warp_pairs)
{
    pdl_enter();
    __shared__ PsWarpSmem wsm[PS_THREADS / 32];
    const long nbp = warp_pairs ? 0 : (npair + blockDim.x - 1) / blockDim.x;
    if (blockIdx.x >= nbp) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const long c = (long)(blockIdx.x - nbp) * (blockDim.x >> 5) + wid;   // pair or colloid of this warp
        if (c >= (warp_pairs ? npair : ncoll)) return;
        const Seg &s = segs[warp_pairs ? rep_of_b(bead_offs, R, pairs[c].x) : coll_rep[c]];
        const long b = warp_pairs ? (long)pairs[c].x : s.bead_off + s.Nm + (c - s.coll_off);
        const long q0 = warp_pairs ? c : cptr[b], q1 = warp_pairs ? c + 1 : cptr[b + 1];
        for (long q = q0; q < q1; q++)
            ps_setup_colloid_pair(s, b, pairs[q].y, x, tab, nrow, Sout + 144L * q, Pout + 144L * q, wsm[wid], lane);
        return;
    }
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npair) return;
    const long lo = pairs[q].x, hi = pairs[q].y;
    const Seg &s = segs[rep_of_b(bead_offs, R, lo)];
    if ((lo - s.bead_off) >= s.Nm) return;            // colloid pair: its lower colloid's warp
    double *So = Sout + 144 * q, *Po = Pout + 144 * q;
    // closed form: S and the mobility share the modes of the pair block
    double d[3], lam[4], sq[4], pm[4];
    mono_pair_modes(s, x, tab, nrow, lo, hi, d, lam);
    double xs = 0.0, ys = 0.0;
    if (s.mm_HI && !(s.chain_HI && chain[lo] == chain[hi])) {
        double dx = x[3 * lo] - x[3 * hi], dy = x[3 * lo + 1] - x[3 * hi + 1], dz = x[3 * lo + 2] - x[3 * hi + 2];
        const double r = ref_pair_dist(dx, dy, dz), rinv = 1.0 / r;
        if (s.aa_mode == PS_AA_RPY) aa_scalars_rpy<double>(r, rinv, 2.0 * s.beta, xs, ys);
        else aa_scalars<double>(r, rinv, 2.0 * s.beta, xs, ys);
    }
    const double mob[4] = {s.beta_inv + xs, s.beta_inv + ys, s.beta_inv - xs, s.beta_inv - ys};
    for (int k = 0; k < 4; k++) {
        double l = lam[k] > 0 ? lam[k] : 0.0;
        sq[k] = sqrt(l);
        double t = 1.0 + l * mob[k];
        pm[k] = t > 0 ? 1.0 / t : 1.0;
    }
    // compact 6 x 6 blocks (row stride 6) at the start of the pair's slot
    mono_pair_matrix(d, sq, So, 6);
    mono_pair_matrix(d, pm, Po, 6);
}

static void launch_ps_setup(Engine &E, cudaStream_t st)
{
    const long npair = E.lub_npairs;
    const long nbp = (npair + PS_THREADS - 1) / PS_THREADS, nbc = (E.ncoll + PS_THREADS / 32 - 1) / (PS_THREADS / 32);
    const bool warp_pairs = E.ntot == E.ncoll;
    ps_launch(k_ps_setup, (unsigned)(warp_pairs ? (npair + PS_THREADS / 32 - 1) / (PS_THREADS / 32) : nbp + nbc), PS_THREADS, 0, st,
            npair, E.d_lub_pairs, E.d_bead_offs, E.R, E.d_segs, E.d_x, E.d_chain, E.d_lubtab, E.lub_nrow, E.ncoll,
            E.d_coll_rep, E.d_lubc_ptr, E.d_pS, E.d_pP, warp_pairs ? 1 : 0);
}

// ---------------------------------------------------------------------------
// Work split of the pair space.  A replica of Np beads has a fixed number of blocks
// (PairBlk, built with the context: 32 beads each, 2 where it has only colloids, whose
// near pairs are many and 12 x 12, and never more than 512); block b takes the b-th share of the replica's
// canonical pairs, of its beads and of its colloids, whatever the lists of the staging
// hold.  Blocks never mix replicas, each leaves one sum per dot, and the blocks of the
// next kernel add their replica's sums themselves (rep_total) and run the scalar
// recurrence on them: no counters, no fences, no separate reductions, and an order that
// depends on the replica alone.
//
// Bound: latency (a dependent launch with an L2 round trip, 3 to 4 us each).  A CG
// iteration of a lubricated replica took 7 launches beside the applies; 4 this way: the
// direction, L^T, the update, and one gather for L z and for the residual test's L r
// (u = L p is kept by its own recurrence L p = L z + beta L p).  Lubricated steps: 980
// beads 5.50 -> 5.25 ms, 64 replicas of 62000 beads 22.8 -> 19.8 ms.
constexpr int PB_THREADS = 128;
constexpr int LT_LANES = 16;                 // lanes per pair: lane a owns entry a of the pair vectors

struct PairTab {
    const PairBlk *blk;
    const int2 *pairs;
    const int *cptr;                         // canonical pairs by lower bead
    const Seg *segs;
};

// share b of n items
__device__ __forceinline__ int share(int n, int b, int G) { return (int)((long)n * b / G); }

// canonical pairs [lo, hi) of a block
__device__ __forceinline__ void pair_share(const PairTab &T, const PairBlk &B, const Seg &s, long &lo, long &hi)
{
    const int q0 = T.cptr[s.bead_off], n = T.cptr[s.bead_off + s.Np] - q0;
    lo = q0 + share(n, B.b, B.G);
    hi = q0 + share(n, B.b + 1, B.G);
}

__device__ __forceinline__ double pb_sum(double v)
{
    __shared__ double ws[PB_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < PB_THREADS / 32; w++) t += ws[w];
    return t;
}

// z_a = (P_q r)_a for lane a of a pair's team (r_c held by lane c); rows and
// columns past nd (6 for monomer pairs) add nothing, columns in ascending order
__device__ __forceinline__ double pm_matvec(const double *__restrict__ Pq, int a, int nd, double ra, unsigned team)
{
    double z = 0.0;
#pragma unroll
    for (int c = 0; c < 12; c++) {
        const double rc = __shfl_sync(team, ra, c, LT_LANES);
        if (a < nd && c < nd) z += Pq[a * nd + c] * rc;
    }
    return z;
}

// entry a of S_q (y + y2 (+ addv)) gathered at the pair's DOFs: lane a gathers entry a and
// forms row a (the L^T of an apply's output)
__device__ __forceinline__ double lt_row(const Seg &s, long lo, long hi, int a, int nd, unsigned team,
                                         const double *__restrict__ Sq, const double *__restrict__ y,
                                         const double *__restrict__ y2, const double *__restrict__ addv)
{
    double za = 0.0;
    if (a < nd) {
        const long bd = (a % 6) < 3 ? lo : hi;
        int tb, wb;
        vel_dofs(s, (int)(bd - s.bead_off), tb, wb);
        const int d = (a < 6 ? tb : wb) + a % 3;
        za = y[s.top_off + d] + (s.ss_off >= 0 ? y2[s.top_off + d] : 0.0) + (addv ? addv[s.vel_off + d] : 0.0);
    }
    return pm_matvec(Sq, a, nd, za, team);
}

// The loop over a block's pairs, a team of LT_LANES lanes per pair: for every lane of the team,
// w = load(q, lo, hi, nd, a, team), what a kernel can fetch and form before it knows the
// replica's scalars, then work(w, q, nd, a, team).  The first pair's load runs ahead of mid(),
// which adds the sums and runs the recurrence, so that their round trips overlap.
template <class L, class M, class W>
__device__ __forceinline__ void for_pairs(const PairTab &T, const PairBlk &B, const Seg &s, L load, M mid, W work)
{
    long q0, q1;
    pair_share(T, B, s, q0, q1);
    const int a = threadIdx.x % LT_LANES;
    const unsigned team = 0xffffu << (threadIdx.x & 16);
    long q = q0 + threadIdx.x / LT_LANES;
    int nd = 12;
    auto get = [&]() {
        const int2 p = T.pairs[q];
        nd = (p.x - s.bead_off) < s.Nm ? 6 : 12;                     // monomer pairs: 6 x 6 blocks
        return load(q, (long)p.x, (long)p.y, nd, a, team);
    };
    decltype(load(0L, 0L, 0L, 0, 0, 0u)) w{};
    if (q < q1) w = get();
    if (!mid()) return;
    while (q < q1) {
        work(w, q, nd, a, team);
        q += PB_THREADS / LT_LANES;
        if (q < q1) w = get();
    }
}

template <class F>
__device__ __forceinline__ void for_pairs(const PairTab &T, const PairBlk &B, const Seg &s, F f)
{
    for_pairs(T, B, s, [](long, long lo, long hi, int, int, unsigned) { return longlong2{lo, hi}; }, []() { return true; },
              [&](longlong2 p, long q, int nd, int a, unsigned team) { f(q, p.x, p.y, nd, a, team); });
}

// row a of a pair's block
struct Row12 { double v[12]; };
__device__ __forceinline__ Row12 block_row(const double *__restrict__ P, int a, int nd)
{
    Row12 r;
#pragma unroll
    for (int c = 0; c < 12; c++) r.v[c] = a < nd && c < nd ? P[a * nd + c] : 0.0;
    return r;
}
__device__ __forceinline__ double row_dot(const Row12 &r, double x, unsigned team)
{
    double z = 0.0;
#pragma unroll
    for (int c = 0; c < 12; c++) z += r.v[c] * __shfl_sync(team, x, c, LT_LANES);
    return z;
}

// (L y)_d = sum over the bead's near pairs of the rows of S_q y_q that belong to it, for two
// vectors at once (y1 may be null): a monomer's three rows by three lanes of a quad, pairs
// in ascending partner order; a colloid's six rows by two groups of six lanes of sixteen,
// the pairs of its list added in the order of a warp with a lane per pair and a butterfly over
// the lanes (16, 8, 4, 2, 1).  f(dof, (L y0)_d, (L y1)_d) once per row.
template <class F>
__device__ __forceinline__ void for_gather(const PairBlk &B, const Seg &s, const int *__restrict__ sptr,
                                           const int *__restrict__ snbr, const int *__restrict__ cidx,
                                           const double *__restrict__ S, const double *__restrict__ y0,
                                           const double *__restrict__ y1, F f)
{
    const int i0 = share(s.Np, B.b, B.G), i1 = share(s.Np, B.b + 1, B.G);
    // the rows of pairs t0, t0 + step, ... of bead b's list, added up in order
    auto rows = [&](long b, int row, int nd, int t0, int step, double &v0, double &v1) {
        for (int t = sptr[b] + t0; t < sptr[b + 1]; t += step) {
            const int q = cidx[t];
            if (q < 0) continue;                            // not in the canonical list (lists disagree)
            const double *r = S + 144L * q + (6 * (row / 3) + (b < (long)snbr[t] ? 0 : 3) + row % 3) * nd;
            double a = 0.0, c = 0.0;
#pragma unroll
            for (int k = 0; k < 12; k++)
                if (k < nd) {
                    const double sk = r[k];
                    a += sk * y0[12L * q + k];
                    if (y1) c += sk * y1[12L * q + k];
                }
            v0 += a;
            v1 += c;
        }
    };
    const int row4 = threadIdx.x & 3;
    for (int i = i0 + (threadIdx.x >> 2); i < min(i1, s.Nm); i += PB_THREADS / 4) {
        double v0 = 0.0, v1 = 0.0;
        if (row4 < 3) {
            rows((long)s.bead_off + i, row4, 6, 0, 1, v0, v1);
            f(3 * i + row4, v0, v1);
        }
    }
    const int l = threadIdx.x & 15, grp = l / 6, row6 = l % 6;
    const unsigned team = 0xffffu << (threadIdx.x & 16);
    for (int i = max(i0, s.Nm) + (threadIdx.x >> 4); i < i1; i += PB_THREADS / 16) {
        const long b = (long)s.bead_off + i;
        const int t0 = sptr[b], n = sptr[b + 1] - t0;
        // leaf p of the tree: the pairs p, p + 32, ... of the list, in order
        double v0 = 0.0, v1 = 0.0;
        if (n <= 8) {
            // leaves 0..7: ((0 + 4) + (2 + 6)) + ((1 + 5) + (3 + 7)); group 0 takes the even ones
            double x0[4] = {0, 0, 0, 0}, x1[4] = {0, 0, 0, 0};
            if (grp < 2)
                for (int k = 0; k < 4; k++)
                    if (2 * k + grp < n) rows(b, row6, 12, 2 * k + grp, 32, x0[k], x1[k]);
            v0 = (x0[0] + x0[2]) + (x0[1] + x0[3]);
            v1 = (x1[0] + x1[2]) + (x1[1] + x1[3]);
        } else if (grp < 2) {
            // the tree by levels, even leaves in group 0, odd ones in group 1
            auto leaf = [&](int p, double &a0, double &a1) { a0 = 0.0; a1 = 0.0; if (p < n) rows(b, row6, 12, p, 32, a0, a1); };
            for (int h = 0; h < 2; h++) {             // bit 1 of the leaf
                double y0 = 0.0, y1 = 0.0;
                for (int f = 0; f < 2; f++) {         // bit 2
                    double z0 = 0.0, z1 = 0.0;
                    for (int e = 0; e < 2; e++) {     // bit 3; bit 4 inside
                        const int p = grp + 2 * h + 4 * f + 8 * e;
                        double a0, a1, c0, c1;
                        leaf(p, a0, a1);
                        leaf(p + 16, c0, c1);
                        a0 += c0; a1 += c1;
                        if (e == 0) { z0 = a0; z1 = a1; } else { z0 += a0; z1 += a1; }
                    }
                    if (f == 0) { y0 = z0; y1 = z1; } else { y0 += z0; y1 += z1; }
                }
                if (h == 0) { v0 = y0; v1 = y1; } else { v0 += y0; v1 += y1; }
            }
        }
        v0 += __shfl_sync(team, v0, l + 6, 16);
        v1 += __shfl_sync(team, v1, l + 6, 16);
        if (grp == 0) {
            int tb, wb;
            vel_dofs(s, i, tb, wb);
            f((row6 < 3 ? tb : wb) + row6 % 3, v0, v1);
        }
    }
}

// u_t = L y (+ add); optionally also into the force rows of a saddle vector
__global__ void __launch_bounds__(PB_THREADS)
k_ps_L(PairTab T, const int *__restrict__ sptr, const int *__restrict__ snbr, const int *__restrict__ cidx,
       const double *__restrict__ S, const double *__restrict__ y, const double *__restrict__ add,
       double *__restrict__ u, double *__restrict__ vel, double *__restrict__ x, const char *__restrict__ done,
       int dstride)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    if (rep_done(done, dstride, B.rep)) return;
    const Seg &s = T.segs[B.rep];
    for_gather(B, s, sptr, snbr, cidx, S, y, nullptr, [&](int d, double v, double) {
        if (add) v += add[s.vel_off + d];
        if (u) u[s.top_off + d] = v;
        if (vel) vel[s.vel_off + d] = v;
        if (x) x[s.vec_off + d] = v;
    });
}

// ---------------------------------------------------------------------------
// pair-space CG.  The scalars of iteration k live in st[k & 1].
struct PcgVec { double *y, *r, *z, *p, *Ap, *Lz, *Lp; };

// r = L^T (g + M b_bot) (y, y2: the apply to b_bot), z = P r, y = 0; sums of r.z
__global__ void __launch_bounds__(PB_THREADS)
k_pc_init(PairTab T, const double *__restrict__ S, const double *__restrict__ P, const double *__restrict__ y,
          const double *__restrict__ y2, const double *__restrict__ g, PcgVec V, double *__restrict__ prz)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    const Seg &s = T.segs[B.rep];
    double dot = 0.0;
    for_pairs(T, B, s, [&](long q, long lo, long hi, int nd, int a, unsigned team) {
        const double ra = lt_row(s, lo, hi, a, nd, team, S + 144 * q, y, y2, g);
        const double za = pm_matvec(P + 144 * q, a, nd, ra, team);
        if (a < nd) {
            const long e = 12 * q + a;
            V.y[e] = 0.0; V.r[e] = ra; V.z[e] = za;
            dot += ra * za;
        }
    });
    dot = pb_sum(dot);
    if (threadIdx.x == 0) prz[blockIdx.x] = dot;
}

// L z for the next direction, and the residual test ||D^{-1} L r||^2
__global__ void __launch_bounds__(PB_THREADS)
k_pc_gather(PairTab T, const int *__restrict__ sptr, const int *__restrict__ snbr, const int *__restrict__ cidx,
            const double *__restrict__ S, PcgVec V, const double *__restrict__ D, const PcgScal *__restrict__ st,
            double *__restrict__ perr)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    if (st[B.rep].done || st[B.rep].stop) return;
    const Seg &s = T.segs[B.rep];
    double err = 0.0;
    for_gather(B, s, sptr, snbr, cidx, S, V.z, V.r, [&](int d, double lz, double lr) {
        V.Lz[s.vel_off + d] = lz;
        const double t = lr / D[s.vec_off + s.nm3nc11 + d];
        err += t * t;
    });
    err = pb_sum(err);
    if (threadIdx.x == 0) perr[blockIdx.x] = err;
}

// closes an iteration (k > 0) or the start (k = 0): the residual test, beta; then p = z + beta p,
// u = L p = L z + beta L p
__global__ void __launch_bounds__(PB_THREADS)
k_pc_dir(PairTab T, const PcgScal *__restrict__ st0, PcgScal *__restrict__ st1, const double *__restrict__ prz,
         const double *__restrict__ perr, PcgVec V, double *__restrict__ u, int k, int maxit, int *nactive)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    __shared__ PcgScal sm;
    if (st0[B.rep].done) {
        if (B.b == 0 && threadIdx.x == 0) st1[B.rep] = st0[B.rep];
        return;
    }
    if (st0[B.rep].stop) {                                 // the update before met non-positive curvature
        if (B.b == 0 && threadIdx.x == 0) {
            PcgScal p = st0[B.rep];
            p.done = 1;
            p.reason = -8;
            st1[B.rep] = p;
            atomicSub(nactive, 1);
        }
        return;
    }
    const double rz = rep_total(prz + B.first, B.G), err2 = rep_total(perr + B.first, B.G);
    if (threadIdx.x == 0) {
        PcgScal p = st0[B.rep];
        p.err = sqrt(err2);
        if (k > 0) p.it++;
        if (p.err <= p.tol) { p.done = 1; p.reason = 2; }
        else if (rz <= 0.0) { p.done = 1; p.reason = -8; }
        else if (p.it >= maxit) { p.done = 1; p.reason = -3; }
        else {
            p.beta = k == 0 ? 0.0 : rz / p.rz;
            p.rz = rz;
        }
        if (B.b == 0) {
            if (p.done) atomicSub(nactive, 1);
            st1[B.rep] = p;
        }
        sm = p;
    }
    __syncthreads();
    if (sm.done) return;
    const double beta = sm.beta;
    const Seg &s = T.segs[B.rep];
    for_pairs(T, B, s, [&](long q, long, long, int nd, int a, unsigned) {
        const long e = 12 * q + a;
        if (a < nd) V.p[e] = k == 0 ? V.z[e] : V.z[e] + beta * V.p[e];
    });
    auto dof = [&](int d) {
        const long v = (long)s.vel_off + d;
        const double t = k == 0 ? V.Lz[v] : V.Lz[v] + beta * V.Lp[v];
        V.Lp[v] = t;
        u[s.top_off + d] = t;
    };
    const int i0 = share(s.Np, B.b, B.G), i1 = share(s.Np, B.b + 1, B.G), c0 = max(i0 - s.Nm, 0), c1 = i1 - s.Nm;
    for (int d = 3 * i0 + threadIdx.x; d < 3 * i1; d += PB_THREADS) dof(d);
    for (int d = 3 * c0 + threadIdx.x; d < 3 * c1; d += PB_THREADS) dof(s.nm3nc3 + d);
}

// Ap = p + L^T (M L p); sums of p.Ap
__global__ void __launch_bounds__(PB_THREADS)
k_pc_apply(PairTab T, const double *__restrict__ S, const double *__restrict__ y, const double *__restrict__ y2, PcgVec V,
           const PcgScal *__restrict__ st, double *__restrict__ pap)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    if (st[B.rep].done) return;
    const Seg &s = T.segs[B.rep];
    double dot = 0.0;
    for_pairs(T, B, s, [&](long q, long lo, long hi, int nd, int a, unsigned team) {
        const double v = lt_row(s, lo, hi, a, nd, team, S + 144 * q, y, y2, nullptr);
        if (a < nd) {
            const double pa = V.p[12 * q + a], w = v + pa;
            V.Ap[12 * q + a] = w;
            dot += pa * w;
        }
    });
    dot = pb_sum(dot);
    if (threadIdx.x == 0) pap[blockIdx.x] = dot;
}

// y += alpha p ; r -= alpha Ap ; z = P r ; sums of r.z.  A direction of non-positive curvature stops the
// replica: its first block notes it, which no block of this launch reads, and k_pc_dir makes it done.
__global__ void __launch_bounds__(PB_THREADS)
k_pc_update(PairTab T, const double *__restrict__ P, PcgVec V, PcgScal *__restrict__ st, const double *__restrict__ pap,
            double *__restrict__ prz)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    if (st[B.rep].done) return;
    const Seg &s = T.segs[B.rep];
    struct In { double y, p, r, Ap; Row12 P; };
    double dot = 0.0, alpha = 0.0;
    bool stop = false;
    for_pairs(T, B, s,
        [&](long q, long, long, int nd, int a, unsigned) {
            const long e = 12 * q + a;
            In w{};
            if (a < nd) { w.y = V.y[e]; w.p = V.p[e]; w.r = V.r[e]; w.Ap = V.Ap[e]; }
            w.P = block_row(P + 144 * q, a, nd);
            return w;
        },
        [&]() {
            const double pAp = rep_total(pap + B.first, B.G);
            stop = pAp <= 0.0;
            if (stop && B.b == 0 && threadIdx.x == 0) st[B.rep].stop = 1;
            if (!stop) alpha = st[B.rep].rz / pAp;
            return !stop;
        },
        [&](const In &w, long q, int nd, int a, unsigned team) {
            const long e = 12 * q + a;
            const double ra = w.r - alpha * w.Ap, za = row_dot(w.P, ra, team);
            if (a < nd) {
                V.y[e] = w.y + alpha * w.p;
                V.r[e] = ra;
                V.z[e] = za;
                dot += ra * za;
            }
        });
    if (stop) return;
    dot = pb_sum(dot);
    if (threadIdx.x == 0) prz[blockIdx.x] = dot;
}

// g = b_tt - (M [0 ; M_SS^{-1} b_S])_t, c = -b_bot (velocity layout), u_t = b_bot
__global__ void k_ps_rhs(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ b,
                         const double *__restrict__ y2, double *__restrict__ g, double *__restrict__ c,
                         double *__restrict__ u)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const Seg &s = segs[B.rep];
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) {
        const long k = (long)B.start + e;
        const int j = (int)(k - s.vel_off);
        const double v = b[s.vec_off + s.nm3nc11 + j];
        g[k] = b[s.vec_off + j] - (s.ss_off >= 0 ? y2[s.top_off + j] : 0.0);
        c[k] = -v;
        u[s.top_off + j] = v;
    }
}

// U = (y + y2)_t - g into the saddle solution
__global__ void k_ps_fin(RedTable T, const Seg *__restrict__ segs, const double *__restrict__ y,
                         const double *__restrict__ y2, const double *__restrict__ g, double *__restrict__ x)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const Seg &s = segs[B.rep];
    for (int e = threadIdx.x; e < B.len; e += RB_THREADS) {
        long k = B.start + e;
        int j = (int)(k - s.vel_off);
        double v = y[s.top_off + j] + (s.ss_off >= 0 ? y2[s.top_off + j] : 0.0) - g[k];
        x[s.vec_off + s.nm3nc11 + j] = v;
    }
}

// F_S of the joint replicas (colloids beyond the dense stresslet limit) into u and the solution
__global__ void k_ps_S(long ncoll, const int *__restrict__ coll_rep, const Seg *__restrict__ segs,
                       const double *__restrict__ yS, double *__restrict__ u, double *__restrict__ x)
{
    pdl_enter();
    const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncoll) return;
    const Seg &s = segs[coll_rep[c]];
    if (s.ss_off >= 0) return;
    const long o = s.nm3nc6 + 5 * (c - s.coll_off);
    for (int k = 0; k < 5; k++) {
        const double v = yS[s.top_off + o + k];
        u[s.top_off + o + k] = v;
        x[s.vec_off + o + k] = v;
    }
}

// Mr applied to the force rows held in E.d_pu (stresslet part zero):
// d_py = M [u ; 0], d_pu2 = [0 ; -M_SS^{-1} (d_py)_S], d_py2 = M d_pu2
static void mr_apply(Engine &E, bool fp32, const void *dn, int ds, cudaStream_t st)
{
    apply_operator(E, 1, E.d_pu, E.d_py, fp32, st, dn, ds);
    if (E.n_ss_reps) {
        ps_launch(k_ss_apply, E.n_ss_reps, 64, 0, st, E.d_segs, E.d_ss_reps, E.d_ssinv, E.d_py, 1, -1.0,
                nullptr, 1, 0.0, E.d_pu2, 1, (const char *)dn, ds);
        apply_operator(E, 1, E.d_pu2, E.d_py2, fp32, st, dn, ds, true);
    }
}

// ---------------------------------------------------------------------------
// Pair-space MINRES, for replica sets whose far-field mobility may be
// indefinite (colloid pairs near contact: the far-field FTS mobility is not
// positive definite there; the reference's own monomer pair scalars).  The
// operator and preconditioner are those of the CG above; the recurrences are
// Paige & Saunders' preconditioned MINRES as in krylov.cu, with PETSc's test on
// the preconditioned residual estimate (np * prod |s_k| <= rtol * np_0).
// Vectors live in the two storages of the pair space: 12 entries per pair, and
// the stresslet entries of the joint replicas' colloids (mobility layout).
struct PMVec { double *pair; double *s; };
struct PMArgs {
    PMVec R0, R1, R2;          // r_k, r_{k+1} (first Av), r_{k-1}
    PMVec W0, W1, W2;          // w_{k-3}, w_{k-2}, w_{k-1} (formed by iteration k)
    PMVec v, z, x;
    const double *b, *g;       // right-hand side, g of the velocity rows
    const double *y;           // the apply's output (mobility layout; its S part is y_S)
    const double *y2;          // the dense stresslet block's share of the output (replicas with one)
    const double *S;           // pair square-root blocks (L = [B_q S_q])
    double *u;                 // the apply's input (mobility layout): its S part gets z_S
    const double *P;           // pair preconditioner blocks
    double *da, *db, *dn;      // v.Av, r.z, z.z (start): one number per pair, then one per bead
    long npair;
};

// A replica's total of the dots d (per canonical pair, then per bead from d + npair on), the same
// in every thread: thread t takes pairs t, t + 128, ... into eight sums joined in pairs, then the
// beads likewise, then a shuffle tree and the warps in order.  Every block adds all of its
// replica's numbers, 4500 for 1024 colloids, rather than one number per block, because this
// order is part of the answer where the system is close to singular.
__device__ __forceinline__ double strided_sum(const double *__restrict__ x, long lo, long hi)
{
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long q = lo + threadIdx.x; q < hi; q += 8 * PB_THREADS) {
        double t[8];
#pragma unroll
        for (int u = 0; u < 8; u++) t[u] = q + u * PB_THREADS < hi ? x[q + u * PB_THREADS] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; u++) acc[u] += t[u];
    }
    return ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
}

__device__ __forceinline__ double pm_total(const PairTab &T, const Seg &s, const double *__restrict__ d, long npair)
{
    __shared__ double ws[PB_THREADS / 32];
    const int q0 = T.cptr[s.bead_off], q1 = T.cptr[s.bead_off + s.Np];
    // only a joint replica's colloids have numbers of their own
    const double *db = d + npair;
    double v = strided_sum(d, q0, q1) + (s.Nc > 0 && s.ss_off < 0 ? strided_sum(db, s.bead_off, (long)s.bead_off + s.Np) : 0.0);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < PB_THREADS / 32; w++) t += ws[w];
    return t;
}

// a pair's dot over its team, stored by lane 0
__device__ __forceinline__ void pair_dot(double v, unsigned team, int a, double *__restrict__ out)
{
#pragma unroll
    for (int o = LT_LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(team, v, o, LT_LANES);
    if (a == 0) *out = v;
}

__device__ __forceinline__ void s_precond(const double r[5], double z[5])
{
    const double det = 1.8 * 1.8 - 0.9 * 0.9;
    z[0] = (1.8 * r[0] - 0.9 * r[4]) / det;
    z[4] = (1.8 * r[4] - 0.9 * r[0]) / det;
    for (int k = 1; k < 4; k++) z[k] = r[k] / 1.8;
}

// the loop over a block's share of a joint replica's colloids, one thread each: f(first entry of
// the colloid's stresslet in mobility layout, in the saddle vector, its bead)
template <class F>
__device__ __forceinline__ void for_stresslets(const PairBlk &B, const Seg &s, F f)
{
    if (s.Nc == 0 || s.ss_off >= 0) return;
    for (int c = share(s.Nc, B.b, B.G) + threadIdx.x; c < share(s.Nc, B.b + 1, B.G); c += PB_THREADS)
        f((long)s.top_off + s.nm3nc6 + 5 * c, (long)s.vec_off + s.nm3nc6 + 5 * c, (long)s.bead_off + s.Nm + c);
}

// rhs into r_1 (pairs L^T (g + Mr b_bot), stresslets b_S + (M b_bot)_S), z = P r, zeros; sums
// of r.z and z.z
__global__ void __launch_bounds__(PB_THREADS) k_pm_init(PairTab T, PMArgs A)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    const Seg &s = T.segs[B.rep];
    for_pairs(T, B, s, [&](long q, long lo, long hi, int nd, int a, unsigned team) {
        const double ra = lt_row(s, lo, hi, a, nd, team, A.S + 144 * q, A.y, A.y2, A.g);
        const double za = pm_matvec(A.P + 144 * q, a, nd, ra, team);
        if (a < nd) {
            const long e = 12 * q + a;
            A.R1.pair[e] = ra; A.z.pair[e] = za;
            A.x.pair[e] = 0.0; A.v.pair[e] = 0.0;
            A.W0.pair[e] = 0.0; A.W1.pair[e] = 0.0; A.W2.pair[e] = 0.0;
        }
        pair_dot(ra * za, team, a, A.db + q);
        pair_dot(za * za, team, a, A.dn + q);
    });
    for_stresslets(B, s, [&](long t, long v, long bead) {
        double r[5], z[5], rz = 0.0, zz = 0.0;
        for (int a = 0; a < 5; a++) r[a] = A.b[v + a] + A.y[t + a];
        s_precond(r, z);
        for (int a = 0; a < 5; a++) {
            A.R1.s[t + a] = r[a]; A.z.s[t + a] = z[a];
            A.x.s[t + a] = 0.0; A.v.s[t + a] = 0.0;
            A.W0.s[t + a] = 0.0; A.W1.s[t + a] = 0.0; A.W2.s[t + a] = 0.0;
            rz += r[a] * z[a];
            zz += z[a] * z[a];
            A.u[t + a] = z[a];
        }
        A.db[A.npair + bead] = rz;
        A.dn[A.npair + bead] = zz;
    });
}

// closes iteration k - 1 (or the start): scalars, pending w and x update; opens iteration k:
// v = z / beta, Av = (z + L^T (y + y2)) / beta - (beta / oldb) r_{k-1} in pair rows, y_S / beta - ... in
// stresslet rows; sums of v.Av
__global__ void __launch_bounds__(PB_THREADS)
k_pm_alpha(PairTab T, PMArgs A, const MinresScal *__restrict__ st0, MinresScal *__restrict__ st1, int k, int maxit,
           double rtol, int *nactive)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    __shared__ MinresScal sm;
    if (st0[B.rep].done) {
        if (B.b == 0 && threadIdx.x == 0) st1[B.rep] = st0[B.rep];
        return;
    }
    const Seg &s = T.segs[B.rep];
    const MinresScal &m = sm;
    double c1 = 0.0;
    // entry t of one storage (pick), its inputs w: z, v, w_{k-3}, w_{k-2}, x, r_{k-1}; az: the row of A z;
    // adds v Av to dot
    struct In { double az, z, v, w0, w1, x, r; };
    auto fetch = [&](auto pick, long t, double az) {
        return In{az, pick(A.z)[t], pick(A.v)[t], pick(A.W0)[t], pick(A.W1)[t], pick(A.x)[t], k >= 2 ? pick(A.R2)[t] : 0.0};
    };
    auto entry = [&](auto pick, long t, const In &w, double &dot) {
        if (m.pending) {
            const double wn = (w.v - m.up_oldeps * w.w0 - m.up_delta * w.w1) * m.up_ginv;
            pick(A.W2)[t] = wn;
            pick(A.x)[t] = w.x + m.up_phi * wn;
        }
        if (!m.done) {
            const double v = w.z * m.sinv;
            double x = m.sinv * w.az;
            if (k >= 2) x -= c1 * w.r;
            pick(A.v)[t] = v;
            pick(A.R1)[t] = x;
            dot += v * x;
        }
    };
    auto pair = [](const PMVec &p) { return p.pair; };
    auto strs = [](const PMVec &p) { return p.s; };
    for_pairs(T, B, s,
        [&](long q, long lo, long hi, int nd, int a, unsigned team) {
            const double sy = lt_row(s, lo, hi, a, nd, team, A.S + 144 * q, A.y, A.y2, nullptr);
            In w{};
            if (a < nd) { w = fetch(pair, 12 * q + a, 0.0); w.az = sy + w.z; }
            return w;
        },
        [&]() {
            const double bb = pm_total(T, s, A.db, A.npair), zz = k == 1 ? pm_total(T, s, A.dn, A.npair) : 0.0;
            if (threadIdx.x == 0) {
                MinresScal n = st0[B.rep];
                if (k == 1) {
                    n = MinresScal{};
                    n.np = sqrt(zz);
                    n.ttol = fmax(rtol * n.np, 1e-50);
                    if (bb < 0) { n.done = 1; n.reason = -8; }
                    else if (n.np <= n.ttol || bb == 0.0) { n.done = 1; n.reason = 2; }
                    else { n.beta = sqrt(bb); n.phibar = n.beta; n.cs = -1; n.sn = 0; n.sinv = 1.0 / n.beta; }
                } else
                    minres_advance(n, bb, maxit);
                sm = n;
                if (B.b == 0) {
                    if (n.done) atomicSub(nactive, 1);
                    n.pending = 0;                         // applied below
                    st1[B.rep] = n;
                }
            }
            __syncthreads();
            c1 = k >= 2 && !m.done ? m.beta / m.oldb : 0.0;
            return true;
        },
        [&](const In &w, long q, int nd, int a, unsigned team) {
            double dot = 0.0;
            if (a < nd) entry(pair, 12 * q + a, w, dot);
            if (!m.done) pair_dot(dot, team, a, A.da + q);
        });
    for_stresslets(B, s, [&](long t, long, long bead) {
        double dot = 0.0;
        for (int a = 0; a < 5; a++) entry(strs, t + a, fetch(strs, t + a, A.y[t + a]), dot);
        if (!m.done) A.da[A.npair + bead] = dot;
    });
}

// r_{k+1} = Av - (alfa / beta) r_k, z = P r (z_S into the apply's input); sums of r.z
__global__ void __launch_bounds__(PB_THREADS) k_pm_beta(PairTab T, PMArgs A, MinresScal *__restrict__ st)
{
    pdl_enter();
    const PairBlk B = T.blk[blockIdx.x];
    if (st[B.rep].done) return;
    const Seg &s = T.segs[B.rep];
    const PMVec Rn = A.R1, Rk = A.R0;
    struct In { double r, k; Row12 P; };
    double c2 = 0.0;
    for_pairs(T, B, s,
        [&](long q, long, long, int nd, int a, unsigned) {
            In w{};
            if (a < nd) { w.r = Rn.pair[12 * q + a]; w.k = Rk.pair[12 * q + a]; }
            w.P = block_row(A.P + 144 * q, a, nd);
            return w;
        },
        [&]() {
            const double alfa = pm_total(T, s, A.da, A.npair);
            if (B.b == 0 && threadIdx.x == 0) st[B.rep].alfa = alfa;
            c2 = alfa / st[B.rep].beta;
            return true;
        },
        [&](const In &w, long q, int nd, int a, unsigned team) {
            const long e = 12 * q + a;
            const double ra = a < nd ? w.r - c2 * w.k : 0.0, za = row_dot(w.P, ra, team);
            if (a < nd) {
                Rn.pair[e] = ra;
                A.z.pair[e] = za;
            }
            pair_dot(ra * za, team, a, A.db + q);
        });
    for_stresslets(B, s, [&](long t, long, long bead) {
        double r[5], z[5], dot = 0.0;
        for (int a = 0; a < 5; a++) { r[a] = Rn.s[t + a] - c2 * Rk.s[t + a]; Rn.s[t + a] = r[a]; }
        s_precond(r, z);
        for (int a = 0; a < 5; a++) {
            A.z.s[t + a] = z[a];
            dot += r[a] * z[a];
            A.u[t + a] = z[a];
        }
        A.db[A.npair + bead] = dot;
    });
}

static int grow(double *&p, long n)
{
    cudaFree(p);
    p = nullptr;
    PS_CK(cudaMalloc(&p, sizeof(double) * n));
    return PS_OK;
}

static int ensure_pair_space(Engine &E)
{
    const long need = std::max<long>(E.lub_npairs, 1);
    if (need <= E.pair_cap) return PS_OK;
    E.ps_setup_valid = false;
    E.pair_cap = 0;
    const long cap = need * 3 / 2 + 256;
    int rc;
    if ((rc = grow(E.d_pS, 144 * cap)) || (rc = grow(E.d_pP, 144 * cap))) return rc;
    for (auto &p : E.d_py_)
        if ((rc = grow(p, 12 * cap))) return rc;
    E.pair_cap = cap;
    return PS_OK;
}

// the pair-space MINRES vectors, for the contexts that come to use them
static int ensure_pm_space(Engine &E, cudaStream_t st)
{
    if (E.pm_cap == E.pair_cap) return PS_OK;
    E.pm_cap = 0;
    int rc;
    for (auto &p : E.d_pmp)
        if ((rc = grow(p, 12 * E.pair_cap))) return rc;
    if ((rc = grow(E.d_pmd, 3 * (E.pair_cap + E.ntot)))) return rc;
    // beads without stresslet unknowns never write theirs; on the solve's stream, which alone orders it
    // before the kernels that write the others'
    PS_CK(cudaMemsetAsync(E.d_pmd, 0, sizeof(double) * 3 * (E.pair_cap + E.ntot), st));
    E.pm_cap = E.pair_cap;
    return PS_OK;
}

static PairTab pair_tab(const Engine &E) { return {E.d_pblk, E.d_lub_pairs, E.d_lubc_ptr, E.d_segs}; }

static void launch_ps_L(Engine &E, const double *y, const double *add, double *u, double *vel, double *x,
                        const char *done, int dstride, cudaStream_t st)
{
    ps_launch(k_ps_L, (unsigned)E.n_pblk, PB_THREADS, 0, st, pair_tab(E), E.d_lub_ptr, E.d_lub_nbr, E.d_lub_cidx, E.d_pS, y,
            add, u, vel, x, done, dstride);
}

// iterations of a pair-space solver are looked at by the host every check_every of them, long
// solves less often (a missed stop costs launches of blocks that leave at once)
static int next_check(int k, int check_every) { return k + std::max(check_every, std::min(k / 4, 4 * check_every)); }

// MINRES iterations of the pair-space system; the setup (pair blocks, g, the
// u_t = b_bot apply input) has run.  Returns the solution's pair and stresslet
// storages in *ysol / *ssol.
static int pair_minres(Engine &E, const double *b, const double *g, int maxit, double rtol, int check_every, bool fp32,
                       cudaStream_t st, double **ysol, double **ssol, MinresScal **scal)
{
    const int ds = (int)sizeof(MinresScal);
    const unsigned nb = (unsigned)E.n_pblk;
    const PairTab T = pair_tab(E);
    int rc = ensure_pm_space(E, st);
    if (rc) return rc;
    PMArgs A;
    // r_k lives in slot k % 3, w_k in slot 3 + k % 3
    auto slots = [&](int k) {
        PMVec *r[3] = {&A.R0, &A.R1, &A.R2}, *w[3] = {&A.W0, &A.W1, &A.W2};
        for (int j = 0; j < 3; j++) {
            const int i = (k + j) % 3;
            *r[j] = {E.d_pmp[i], E.d_pms[i]};
            *w[j] = {E.d_pmp[3 + i], E.d_pms[3 + i]};
        }
    };
    slots(0);
    A.v = {E.d_pmp[6], E.d_pms[6]};
    A.z = {E.d_pmp[7], E.d_pms[7]};
    A.x = {E.d_pmp[8], E.d_pms[8]};
    A.b = b;
    A.g = g;
    A.y = E.d_py;
    A.y2 = E.d_py2;
    A.S = E.d_pS;
    A.u = E.d_pu;
    A.P = E.d_pP;
    const long nd = E.pair_cap + E.ntot;
    A.da = E.d_pmd; A.db = A.da + nd; A.dn = A.db + nd;
    A.npair = E.pair_cap;
    PS_CK(cudaMemsetAsync(E.d_pmr, 0, sizeof(MinresScal) * 2 * E.R, st));
    mr_apply(E, fp32, nullptr, 0, st);
    ps_launch(k_pm_init, nb, PB_THREADS, 0, st, T, A);
    int nact = E.R;
    MinresScal *last = E.d_pmr;
    for (int k = 1, next = check_every + 1; nact > 0; k++) {
        MinresScal *s0 = E.d_pmr + (long)E.R * ((k - 1) & 1), *s1 = E.d_pmr + (long)E.R * (k & 1);
        const char *dn = (const char *)&s0[0].done;
        slots(k);
        // A z: u = [L z_y ; z_S] (z_S already in u), apply; k_pm_alpha forms z_y + L^T (...)_t itself
        if (k <= maxit) {
            launch_ps_L(E, A.z.pair, nullptr, E.d_pu, nullptr, nullptr, dn, ds, st);
            mr_apply(E, fp32, dn, ds, st);
        }
        ps_launch(k_pm_alpha, nb, PB_THREADS, 0, st, T, A, s0, s1, k, maxit, rtol, E.d_nactive);
        last = s1;
        if (k == next || k > maxit) {
            PS_CK(cudaMemcpyAsync(E.h_nactive, E.d_nactive, sizeof(int), cudaMemcpyDeviceToHost, st));
            PS_CK(cudaStreamSynchronize(st));
            nact = *E.h_nactive;
            if (k > maxit) break;
            next = next_check(k, check_every);
        }
        if (nact > 0) ps_launch(k_pm_beta, nb, PB_THREADS, 0, st, T, A, s1);
    }
    PS_CK(cudaGetLastError());
    *ysol = A.x.pair;
    *ssol = A.x.s;
    *scal = last;
    return PS_OK;
}

static int pair_cg(Engine &E, const double *g, int maxit, int check_every, bool fp32, cudaStream_t st, const PcgVec &V,
                   PcgScal **scal)
{
    const int ds = (int)sizeof(PcgScal);
    const unsigned nb = (unsigned)E.n_pblk;
    const PairTab T = pair_tab(E);
    double *pap = E.d_pbp, *prz = pap + E.n_pblk, *perr = prz + E.n_pblk;
    // rhs = L^T (g + Mr b_bot)
    mr_apply(E, fp32, nullptr, 0, st);
    ps_launch(k_pc_init, nb, PB_THREADS, 0, st, T, E.d_pS, E.d_pP, E.d_py, E.d_py2, g, V, prz);
    PcgScal *s1 = E.d_pcg;
    int nact = E.R;
    for (int k = 0, next = 0;; k++) {
        // residual test of iteration k - 1 (or of the start), next direction
        PcgScal *s0 = s1;
        s1 = E.d_pcg + (long)E.R * ((k + 1) & 1);
        ps_launch(k_pc_gather, nb, PB_THREADS, 0, st, T, E.d_lub_ptr, E.d_lub_nbr, E.d_lub_cidx, E.d_pS, V, E.d_D, s0, perr);
        ps_launch(k_pc_dir, nb, PB_THREADS, 0, st, T, s0, s1, prz, perr, V, E.d_pu, k, maxit, E.d_nactive);
        if (k == next || k >= maxit) {
            PS_CK(cudaMemcpyAsync(E.h_nactive, E.d_nactive, sizeof(int), cudaMemcpyDeviceToHost, st));
            PS_CK(cudaStreamSynchronize(st));
            nact = *E.h_nactive;
            if (nact <= 0 || k >= maxit) break;
            next = next_check(k, check_every);
        }
        const char *dn = (const char *)&s1[0].done;
        mr_apply(E, fp32, dn, ds, st);
        ps_launch(k_pc_apply, nb, PB_THREADS, 0, st, T, E.d_pS, E.d_py, E.d_py2, V, s1, pap);
        ps_launch(k_pc_update, nb, PB_THREADS, 0, st, T, E.d_pP, V, s1, pap, prz);
    }
    PS_CK(cudaGetLastError());
    *scal = s1;
    return PS_OK;
}

static int pair_solve(Engine &E, const double *b, double *x, const ps_ksp_opts *o, ps_ksp_result *res,
                      cudaStream_t st, bool minres)
{
    RedTable &TV = E.red_vel;
    const bool fp32 = E.precision == PS_PREC_MIXED;
    // CG converges in tens of iterations on positive definite far fields; a cap
    // hands the rare indefinite case to MINRES early
    const int maxit = minres ? (o->maxit > 0 ? o->maxit : 10000) : std::min(o->maxit > 0 ? o->maxit : 10000, 1000);
    const int check_every = o->check_every > 0 ? o->check_every : 8;
    const long npair = E.lub_npairs;
    int rc = diag_saddle(E, E.d_D, st);
    if (rc) return rc;
    if ((rc = ensure_pair_space(E))) return rc;
    double *cvel = E.d_pV, *g = E.d_pg;
    // replicas beyond the dense stresslet limit keep their stresslets as unknowns: their part of
    // the apply's input starts at zero (elsewhere it is never written)
    if (E.n_ss_polish) PS_CK(cudaMemsetAsync(E.d_pu, 0, sizeof(double) * E.ntop, st));
    ps_launch(k_pcg_start, E.red.nblk, RB_THREADS, 0, st, E.red, b, E.d_D, E.d_pcg, o->rtol, E.R, E.d_nactive);
    // the pair blocks depend on the staged positions and the table only: solves
    // that share a staging (the deterministic and the noise solve) set them up once
    if (npair && !E.ps_setup_valid) {
        launch_ps_setup(E, st);
        E.ps_setup_valid = true;
    }
    if (E.n_ss_reps) {
        ps_launch(k_ss_inverse, E.n_ss_reps, 64, 0, st, E.d_segs, E.d_ss_reps, E.d_x, E.d_delta, E.d_ssinv);
        // g: u2 = [0 ; M_SS^{-1} b_S]
        ps_launch(k_ss_apply, E.n_ss_reps, 64, 0, st, E.d_segs, E.d_ss_reps, E.d_ssinv, b, 0, 1.0, nullptr,
                0, 0.0, E.d_pu2, 1, nullptr, 0);
        apply_operator(E, 1, E.d_pu2, E.d_py2, fp32, st, nullptr, 0, true);
    }
    ps_launch(k_ps_rhs, TV.nblk, RB_THREADS, 0, st, TV, E.d_segs, b, E.d_py2, g, cvel, E.d_pu);
    PS_CK(cudaGetLastError());
    double *yv = E.d_py_[0], *yS = nullptr;
    PcgScal *cs = nullptr;
    MinresScal *ms = nullptr;
    if (minres) {
        if ((rc = pair_minres(E, b, g, maxit, o->rtol, check_every, fp32, st, &yv, &yS, &ms))) return rc;
    } else {
        const PcgVec V = {E.d_py_[0], E.d_py_[1], E.d_py_[2], E.d_py_[3], E.d_py_[4], E.d_pz, E.d_pp};
        if ((rc = pair_cg(E, g, maxit, check_every, fp32, st, V, &cs))) return rc;
    }
    // F_t = -b_bot + L y (into u_t and the force rows), then U = Mr F_t - g, F_S
    launch_ps_L(E, yv, cvel, E.d_pu, nullptr, x, nullptr, 0, st);
    if (E.n_ss_polish)
        ps_launch(k_ps_S, (unsigned)((E.ncoll + 127) / 128), 128, 0, st, E.ncoll, E.d_coll_rep, E.d_segs, yS, E.d_pu, x);
    mr_apply(E, fp32, nullptr, 0, st);
    ps_launch(k_ps_fin, TV.nblk, RB_THREADS, 0, st, TV, E.d_segs, E.d_py, E.d_py2, g, x);
    if (E.n_ss_reps)
        ps_launch(k_ss_apply, E.n_ss_reps, 64, 0, st, E.d_segs, E.d_ss_reps, E.d_ssinv, b, 0, 1.0, E.d_py,
                1, -1.0, x, 0, nullptr, 0);
    PS_CK(cudaGetLastError());
    int worst = 1000, itmax = 0;
    long itsum = 0;
    double emax = 0;
    auto add = [&](int done, int reason, int it, double err) {
        worst = std::min(worst, done ? reason : -3);
        itmax = std::max(itmax, it);
        itsum += it;
        emax = std::max(emax, err);
    };
    if (minres) {
        std::vector<MinresScal> hm(E.R);
        PS_CK(cudaMemcpyAsync(hm.data(), ms, sizeof(MinresScal) * E.R, cudaMemcpyDeviceToHost, st));
        PS_CK(cudaStreamSynchronize(st));
        for (auto &m : hm) add(m.done, m.reason, m.it, m.np);
    } else {
        std::vector<PcgScal> hp(E.R);
        PS_CK(cudaMemcpyAsync(hp.data(), cs, sizeof(PcgScal) * E.R, cudaMemcpyDeviceToHost, st));
        PS_CK(cudaStreamSynchronize(st));
        for (auto &p : hp) add(p.done, p.reason, p.it, p.err);
    }
    if (worst == 1000) worst = 2;
    if (res) { res->reason = worst; res->iters_max = itmax; res->iters_sum = itsum; res->rnorm_max = emax; }
    return PS_OK;
}

int structured_solve(Engine &E, const double *b, double *x, const ps_ksp_opts *o, ps_ksp_result *res,
                     cudaStream_t st)
{
    if (E.any_lub || E.n_ss_polish) {
        ps_ksp_result r0 = {2, 0, 0, 0.0};
        int rc = pair_solve(E, b, x, o, &r0, st, E.any_indef);
        if (rc) return rc;
        if (r0.reason < 0 && !E.any_indef) {      // CG met an indefinite far field: MINRES on the same system
            ps_ksp_result r2 = {2, 0, 0, 0.0};
            if ((rc = pair_solve(E, b, x, o, &r2, st, true))) return rc;
            r2.iters_max += r0.iters_max;
            r2.iters_sum += r0.iters_sum;
            r0 = r2;
        }
        // replicas whose CG broke down (an indefinite far-field mobility: the
        // reference's own pair scalars) finish with MINRES from the CG iterate
        if (r0.reason < 0) {
            ps_ksp_opts po = *o;
            po.warm = 1;
            po.method = PS_SOLVE_MINRES;
            ps_ksp_result r1;
            rc = minres_solve(E, b, x, &po, &r1, st);
            if (rc == PS_ERR_CUDA) return rc;
            r0.reason = r1.reason;
            r0.iters_max = std::max(r0.iters_max, r1.iters_max);
            r0.iters_sum += r1.iters_sum;
            r0.rnorm_max = std::max(r0.rnorm_max, r1.rnorm_max);
        }
        if (res) *res = r0;
        return r0.reason;
    }
    const int thr = 256;
    unsigned nb = (unsigned)((E.nvec + thr - 1) / thr);
    double *y = E.d_Rr[0];
    bool fp32 = E.precision == PS_PREC_MIXED;
    ps_launch(k_struct_init, nb, thr, 0, st, E.nvec, E.d_vec_offs, E.R, E.d_segs, b, x);
    if (E.n_ss_reps) {
        apply_operator(E, 0, x, y, fp32, st);   // y_top = M [F_t ; 0]
        ps_launch(k_struct_ss, E.n_ss_reps, 256, 0, st, E.d_segs, E.d_ss_reps, E.d_x, E.d_delta, b, y, x);
    }
    apply_operator(E, 0, x, y, fp32, st);       // y_top = M F
    ps_launch(k_struct_u, nb, thr, 0, st, E.nvec, E.d_vec_offs, E.R, E.d_segs, b, y, x);
    PS_CK(cudaGetLastError());
    if (res) *res = {2, 0, 0, 0.0};
    return 2;
}

// ---------------------------------------------------------------------------
// Brownian lubrication force, rhs_bot += -sqrt(2 kT / dt) sum_p B_p R_p^{1/2} z_p.
// Each canonical pair q owns 12 normals z_q (monomer pairs use the first 6):
// injected (z + 12 q) or drawn from the replica's Philox stream with
// subsequence q - (first canonical pair of the replica).  R_p^{1/2} is the
// symmetric square root that the pair-space setup stores as the pair's S block,
// so the force is the L-gather of the pair-space solve applied to z (one
// evaluation per pair; the staging's setup is shared with the solve after it).
__global__ void k_lub_z(long npair, const int2 *__restrict__ pairs, const int *__restrict__ bead_offs, int R,
                        const Seg *__restrict__ segs, const int *__restrict__ cptr, const uint64_t *__restrict__ rseed,
                        const uint64_t *__restrict__ rstep, double *__restrict__ z)
{
    pdl_enter();
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npair) return;
    const int r = rep_of_b(bead_offs, R, pairs[q].x);
    curandStatePhilox4_32_10_t stt;
    curand_init(rseed[r], (unsigned long long)(q - cptr[segs[r].bead_off]), (3ull * rstep[r] + 2) * 4ull, &stt);
    for (int k = 0; k < 12; k++) z[12 * q + k] = curand_normal_double(&stt);
}

__global__ void k_lub_noise_add(long nvel, const int *__restrict__ vel_offs, int R, const Seg *__restrict__ segs,
                                const double *__restrict__ v, double *__restrict__ rhs)
{
    pdl_enter();
    const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nvel) return;
    const Seg &s = segs[rep_at(vel_offs, R, k)];
    rhs[(long)s.vec_off + s.nm3nc11 + (k - s.vel_off)] += -sqrt(2.0 * s.kT / s.dt) * v[k];
}

int lub_noise(Engine &E, const double *z, double *rhs, cudaStream_t st)
{
    const long npair = E.lub_npairs;
    if (npair <= 0) return PS_OK;
    int rc;
    if ((rc = ensure_pair_space(E))) return rc;
    const unsigned nbp = (unsigned)((npair + PS_THREADS - 1) / PS_THREADS);
    if (!E.ps_setup_valid) {
        launch_ps_setup(E, st);
        E.ps_setup_valid = true;
    }
    if (!z) {
        const long nz = 12 * npair;
        if (nz > E.zlub_cap) {
            cudaFree(E.d_zlub);
            E.zlub_cap = nz * 3 / 2 + 1024;
            PS_CK(cudaMalloc(&E.d_zlub, sizeof(double) * E.zlub_cap));
        }
        ps_launch(k_lub_z, nbp, PS_THREADS, 0, st, npair, E.d_lub_pairs, E.d_bead_offs, E.R, E.d_segs,
                E.d_lubc_ptr, E.d_rseed, E.d_rstep, E.d_zlub);
        z = E.d_zlub;
    }
    launch_ps_L(E, z, nullptr, nullptr, E.d_tmp_vel, nullptr, nullptr, 0, st);
    const int thr = 256;
    ps_launch(k_lub_noise_add, (unsigned)((E.nvel + thr - 1) / thr), thr, 0, st,
            E.nvel, E.d_vel_offs, E.R, E.d_segs, E.d_tmp_vel, rhs);
    PS_CK(cudaGetLastError());
    return PS_OK;
}

}  // namespace ps
