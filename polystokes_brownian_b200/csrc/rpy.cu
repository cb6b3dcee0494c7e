// rpy.cu -- matrix-free grand-mobility and saddle-operator apply.
//
// y = M u over every replica of the batch, with M the grand mobility that the
// reference assembles densely into A's top-left block (mm_HI, mob.cpp:843-1160)
// or applies as the arrowhead shell (matfree_A.cpp:38-80).  Pair tensors are
// recomputed on the fly from the positions (O(N) memory).  Monomer pairs are
// taken once each, tile pair by tile pair, and applied to both beads (below);
// colloid rows sweep column chunks staged in shared memory.  Tiles and chunks
// of a replica depend on its own size only, and their partial sums are added in
// fixed order by k_combine, so results are deterministic and bit-identical
// whatever else shares the batch.
#include <algorithm>
#include "ps_internal.h"
#include "ps_kernels.h"
#include "ps_reduce.cuh"

namespace ps {

// Single-precision image of a positive double in [2^-126, 2^128) by exponent re-bias and
// mantissa truncation (relative error below 2^-23), with integer operations only, so the
// FP64 pipe is left to the arithmetic; seed_as_double widens a positive normal float exactly.
__device__ __forceinline__ float trunc_to_float(double a)
{
    const int hi = __double2hiint(a), lo = __double2loint(a);
    return __int_as_float(((hi - (896 << 20)) << 3) | (int)((unsigned)lo >> 29));
}
__device__ __forceinline__ double seed_as_double(float f)
{
    const int b = __float_as_int(f);
    return __hiloint2double((b >> 3) + (896 << 20), b << 29);
}

__device__ __forceinline__ double rsqrt_seeded(double a, float af)
{
    const double y = seed_as_double(rsqrtf(af));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double rsqrt_seeded(double a) { return rsqrt_seeded(a, trunc_to_float(a)); }

// ---------------------------------------------------------------------------
// AB/BA: a tile of 128 monomers x the colloids of the replica.  Monomer outputs
// go to part_m (no chunking: Nc is small whenever Nm > 0); each colloid's output
// from this tile's monomers is block-reduced into part_ba (one 11-vector per
// (monomer tile, colloid)).  The blocks are applied in contracted form as for
// colloid pairs (bb_apply): with S^ the stresslet as a symmetric traceless
// matrix, v = S^ e and kg = xg + 2 yg,
//   monomer: T F_c + yb e x T_c + 2 yg v - kg (e.v) e
//   colloid: T^T F_m, yb F_m x e, flat(yg (e F_m^T + F_m e^T) - kg (e.F_m) e e^T),
// T = x e e^T + y (1 - e e^T) in RPY mode; in reference mode the replica's stale
// 3x3 block tab (row-major mob_a[a][b]), nothing on the shell path.
constexpr int AB_TILE = 128, AB_WARPS = AB_TILE / 32;

// sums of eleven values over the warp by halving exchanges; the lane ends with value idx
template <class T>
__device__ __forceinline__ T warp_sum11(const T (&c)[11], int lane, int &idx)
{
    T v[8];
    const bool up = lane & 16;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const T hi = k < 3 ? c[8 + k] : T(0);
        v[k] = (up ? hi : c[k]) + __shfl_xor_sync(0xffffffffu, up ? c[k] : hi, 16);
    }
#pragma unroll
    for (int h = 4, o = 8; h >= 1; h >>= 1, o >>= 1) {
        const bool u = lane & o;
#pragma unroll
        for (int k = 0; k < h; k++) v[k] = (u ? v[k + h] : v[k]) + __shfl_xor_sync(0xffffffffu, u ? v[k] : v[k + h], o);
    }
    idx = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <class T>
__device__ __forceinline__ void ab_block(const Seg &sg, int rep, int mt, const typename V4<T>::t *__restrict__ pos,
                                         const float4 *__restrict__ plo, const double *__restrict__ u, int uoff,
                                         const double *__restrict__ tab, double *__restrict__ part_m,
                                         double *__restrict__ part_ba, T (*red)[AB_WARPS][12])
{
    typedef typename V4<T>::t P4;
    constexpr bool F32 = sizeof(T) == 4;
    const int Nm = sg.Nm, Nc = sg.Nc, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = AB_TILE * mt + threadIdx.x;
    const bool active = threadIdx.x < AB_TILE && i < Nm;
    const long bi = (long)sg.bead_off + (active ? i : AB_TILE * mt);
    const P4 pm = pos[bi];
    T f[3], om[3] = {0, 0, 0};
    for (int a = 0; a < 3; a++) f[a] = active ? (T)u[uoff + 3 * i + a] : T(0);
    const int mode = sg.ab_mode;
    const bool rpy = mode == PS_AB_RPY || mode == PS_AB_RPY_REG, stale = !rpy && sg.mm_HI;
    const T beta2 = T(sg.beta * sg.beta);
    for (int cc = 0; cc < Nc; cc++) {
        if (wid < AB_WARPS) {
            const P4 pc = pos[sg.bead_off + Nm + cc];
            T F[3], Q[3], S[5];
            for (int a = 0; a < 3; a++) {
                F[a] = (T)u[uoff + sg.nm3 + 3 * cc + a];
                Q[a] = (T)u[uoff + sg.nm3 + sg.nc3 + 3 * cc + a];
            }
            for (int q = 0; q < 5; q++) S[q] = (T)u[uoff + sg.nm3nc6 + 5 * cc + q];
            T dx = pm.x - pc.x, dy = pm.y - pc.y, dz = pm.z - pc.z;
            if constexpr (F32) {
                const float4 lm = plo[bi], lc = plo[sg.bead_off + Nm + cc];
                dx += lm.x - lc.x; dy += lm.y - lc.y; dz += lm.z - lc.z;
            }
            const T r2 = dx * dx + dy * dy + dz * dz, rinv = rsqrt_t<T>(r2);
            const T e0 = dx * rinv, e1 = dy * rinv, e2 = dz * rinv;
            T yb, xg, yg;
            ab_scalars<T>(rinv, beta2, yb, xg, yg);
            T c[11];
            if (rpy) {
                T xa, ya;
                ab_trans_scalars<T>(r2 * rinv, rinv, T(sg.beta), mode == PS_AB_RPY_REG, xa, ya, yb);
                const T tF = (xa - ya) * (e0 * F[0] + e1 * F[1] + e2 * F[2]);
                const T tf = (xa - ya) * (e0 * f[0] + e1 * f[1] + e2 * f[2]);
                om[0] += ya * F[0] + tF * e0; om[1] += ya * F[1] + tF * e1; om[2] += ya * F[2] + tF * e2;
                c[0] = ya * f[0] + tf * e0; c[1] = ya * f[1] + tf * e1; c[2] = ya * f[2] + tf * e2;
            } else {
                for (int a = 0; a < 3; a++) c[a] = T(0);
                if (stale)
                    for (int a = 0; a < 3; a++)
                        for (int b = 0; b < 3; b++) {
                            const T t = (T)tab[9 * rep + 3 * a + b];
                            om[a] += t * F[b];
                            c[b] += t * f[a];
                        }
            }
            const T kg = xg + T(2) * yg;
            const T v0 = S[0] * e0 + S[1] * e1 + S[2] * e2, v1 = S[1] * e0 + S[4] * e1 + S[3] * e2;
            const T v2 = S[2] * e0 + S[3] * e1 - (S[0] + S[4]) * e2;
            const T ks = kg * (e0 * v0 + e1 * v1 + e2 * v2);
            om[0] += yb * (e1 * Q[2] - e2 * Q[1]) + T(2) * yg * v0 - ks * e0;
            om[1] += yb * (e2 * Q[0] - e0 * Q[2]) + T(2) * yg * v1 - ks * e1;
            om[2] += yb * (e0 * Q[1] - e1 * Q[0]) + T(2) * yg * v2 - ks * e2;
            c[3] = yb * (f[1] * e2 - f[2] * e1);
            c[4] = yb * (f[2] * e0 - f[0] * e2);
            c[5] = yb * (f[0] * e1 - f[1] * e0);
            const T kf = kg * (e0 * f[0] + e1 * f[1] + e2 * f[2]);
            const T w0 = T(2) * yg * f[0] - kf * e0, w1 = T(2) * yg * f[1] - kf * e1, w2 = T(2) * yg * f[2] - kf * e2;
            const T z22 = e2 * w2;                 // Z = (e w^T + w e^T) / 2
            c[6] = e0 * w0 - z22;
            c[7] = e0 * w1 + e1 * w0;
            c[8] = e0 * w2 + e2 * w0;
            c[9] = e1 * w2 + e2 * w1;
            c[10] = e1 * w1 - z22;
            if (!active)
                for (int q = 0; q < 11; q++) c[q] = T(0);
            int idx;
            const T t = warp_sum11<T>(c, lane, idx);
            if (!(lane & 1) && idx < 11) red[cc & 1][wid][idx] = t;
        }
        __syncthreads();                           // two buffers: the next colloid's sums do not overtake these
        if (threadIdx.x < 11) {
            T v = 0;
            for (int w = 0; w < AB_WARPS; w++) v += red[cc & 1][w][threadIdx.x];
            part_ba[((long)sg.ba_off + (long)mt * Nc + cc) * 11 + threadIdx.x] = (double)v;
        }
    }
    if (active) {
        double *o = part_m + sg.top_off + 3 * i;
        for (int a = 0; a < 3; a++) o[a] = (double)om[a];
    }
}

// ---------------------------------------------------------------------------
// BB: colloid rows x colloid columns (FTS, 11 -> 11), FP64.  A block takes BB_ROWS
// rows of one column chunk, one row per lane; warp h of SPLIT takes the chunk's
// columns h, h + SPLIT, ... (every lane the same column: shared-memory broadcasts),
// and the warps' sums are joined in warp order in shared memory.
//
// Bound: the chain of a pair's dependent FP64 operations; small blocks spread a suspension
// over all SMs.  Against blocks of 128 rows, one launch: 300
// colloids 17.0 -> 9.2 us, 512 17.8 -> 9.6, 1600 51.1 -> 37.9.
// The order of the sums (columns in a chunk by group, groups, chunks) and the arithmetic of a pair are
// part of the answer: the solves of a suspension whose far field is close to singular return, within
// rtol, whatever their rounding selects.  (A pair action of 140 operations for 190 and chunks of 32
// columns gave 14.9 us at 1024 colloids, and positions off by 1e-6 in one step of ten.)
constexpr int BB_ROWS = BB_TILE, BB_CT = 64;
struct BbSmem { double4 sp[BB_CT]; double su[BB_CT * 11]; };

template <int ROWS, int SPLIT>
__device__ __forceinline__ void bb_block(const Seg &sg, int rt, int c, const double4 *__restrict__ pos,
                                         const double *__restrict__ u, int uoff, double *__restrict__ part,
                                         long part_stride, BbSmem &sm, double (*sred)[11][ROWS])
{
    const int row = threadIdx.x % ROWS, grp = threadIdx.x / ROWS;
    const int Nc = sg.Nc, Nm = sg.Nm;
    const int j0 = (int)((long)Nc * c / sg.nch_bb), j1 = (int)((long)Nc * (c + 1) / sg.nch_bb);
    const int i = ROWS * rt + row;
    const bool active = i < Nc;
    const double4 pi = pos[sg.bead_off + Nm + (active ? i : ROWS * rt)];
    double out[11];   // accumulated over the chunk's column tiles in column order
    for (int q = 0; q < 11; q++) out[q] = 0.0;
    for (int jt = j0; jt < j1; jt += BB_CT) {
        const int nj = min(BB_CT, j1 - jt);
        __syncthreads();
        for (int t = threadIdx.x; t < nj * 11; t += blockDim.x) {
            int k = t / 11, q = t - 11 * k, j = jt + k;
            int idx = q < 3 ? sg.nm3 + 3 * j + q : (q < 6 ? sg.nm3 + sg.nc3 + 3 * j + (q - 3) : sg.nm3nc6 + 5 * j + (q - 6));
            sm.su[t] = u[uoff + idx];
        }
        for (int t = threadIdx.x; t < nj; t += blockDim.x) sm.sp[t] = pos[sg.bead_off + Nm + jt + t];
        __syncthreads();
        for (int k = grp; k < nj; k += SPLIT) {
            const int j = jt + k;
            if (j == i) continue;
            const double4 pj = sm.sp[k];
            const bool lo = i < j;
            double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            if (!lo) { dx = -dx; dy = -dy; dz = -dz; }
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double rinv = rsqrt(r2);
            const double e[3] = {dx * rinv, dy * rinv, dz * rinv};
            bb_apply<double>(e, r2 * rinv, rinv, lo, sm.su + 11 * k, out);
        }
    }
    if constexpr (SPLIT > 1) {
        if (grp > 0)
            for (int q = 0; q < 11; q++) sred[grp - 1][q][row] = out[q];
        __syncthreads();
    }
    if (grp == 0 && active) {
        for (int g = 0; g < SPLIT - 1; g++)
            for (int q = 0; q < 11; q++) out[q] += sred[g][q][row];
        double *o = part + (long)c * part_stride + sg.top_off;
        for (int a = 0; a < 3; a++) {
            o[sg.nm3 + 3 * i + a] = out[a];
            o[sg.nm3 + sg.nc3 + 3 * i + a] = out[3 + a];
        }
        for (int q = 0; q < 5; q++) o[sg.nm3nc6 + 5 * i + q] = out[6 + q];
    }
}

// Colloid pairs of the replicas without monomers (suspensions); those beside
// monomers ride in the monomer kernels' launches.
constexpr int BB_SPLIT = 4;
template <int ROWS>
__global__ void __launch_bounds__(ROWS * BB_SPLIT)
k_rpy_bb(const Seg *__restrict__ segs, const Tile *__restrict__ tiles, const double4 *__restrict__ pos,
         const double *__restrict__ u, int in_top, double *__restrict__ part, long part_stride,
         const char *__restrict__ done, int done_stride)
{
    pdl_enter();
    const Tile tl = tiles[blockIdx.x];
    if (done && *(const int *)(done + (long)tl.rep * done_stride)) return;
    __shared__ BbSmem sm;
    __shared__ double sred[BB_SPLIT - 1][11][ROWS];
    const Seg &sg = segs[tl.rep];
    if ((int)blockIdx.y >= sg.nch_bb) return;
    bb_block<ROWS, BB_SPLIT>(sg, tl.mtile, blockIdx.y, pos, u, in_top ? sg.top_off : sg.vec_off, part, part_stride, sm, sred);
}

// The partial sums of one apply, as the far-field kernels write them.
struct FarOut { double *aa, *ab, *ba, *bb; const double *tab; long bb_stride; };

// ---------------------------------------------------------------------------
// Monomer-monomer far field (AA), each unordered pair once.  The pair block is
// symmetric, so one evaluation of the geometry serves U_i += M_ij u_j and
// U_j += M_ij u_i: 32 FMA-pipe operations per unordered pair against 2 x 22 when
// every row sweeps every column.  The monomers of a replica are cut into tiles of
// S beads (aa_tile_edge, a function of Nm alone) and a block takes one tile pair
// (I, J), I <= J; a diagonal tile (I = J) sweeps its ordered pairs row by row.
//
// A warp takes cells of 64 rows x 64 columns (FP32, two columns per packed lane
// pair) or 64 rows x 32 columns (FP64).  Lane l owns rows l and l + 32 in
// registers and walks the cell's columns on the rotation (l + s) mod 32, s the
// step, so the 32 lanes always hold 32 different columns: a row's sums stay in
// its lane, and a column's sums travel with the column, one lane per step, by
// shuffle -- no atomics, and both sides are summed in a fixed order.  A block's
// warps split the tile pair into row groups and column groups, and for the
// smallest edge into bands of steps, so that a replica of a few hundred beads
// still spreads over the chip; their sums join in shared memory in FP64 in warp
// order.  The block writes rows I into partial slot J and rows J into slot I, so
// slot c of a row holds its sum over the columns of tile c, and k_combine adds
// the slots in order.
//
// Bound: the FMA pipe (64 % busy at 16384 beads in FP32, the FP64 pipe 68 % in
// FP64); what is left is fixed-latency waits at 16 warps per SM (124 and 128
// registers; 96 registers and 20 warps measured slower, 215 against 198 us).
// Against a sweep of all ordered pairs (two rows per thread, 256-column chunks),
// one launch, FP32 / FP64: 516 beads 21.8 -> 4.8 us / 47.0 -> 5.1 us, 4096 beads
// 32.5 -> 19.4 / 70.6 -> 33.8, 16384 beads 229 -> 198 / 530 -> 420; error against
// 64-bit sums 1.8e-7 -> 1.1e-7, 1.6e-7 -> 1.4e-7 and 2.2e-7 -> 1.9e-7 in FP32.
constexpr float AAC_PAD = 1e18f;       // padding columns sit at +AAC_PAD, padding rows at -AAC_PAD, with u = 0

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

__device__ __forceinline__ void aa_near_lane(bool n, float r2, float ri, float ri2, float nx0, float nx1, float ny0,
                                             float ny1, float &yv, float &g)
{
    if (n) {
        const float r = r2 * ri, x = nx0 + nx1 * r;
        yv = ny0 + ny1 * r;
        g = (x - yv) * ri2;
    }
}

// AA in FP32 with packed FP32x2 arithmetic (sm_100 FFMA2/FADD2/FMUL2): rows A
// and B of a lane as broadcast pairs (loop-invariant), two columns per step in
// the packed lanes, four unordered pairs per step.  Shared columns are stored
// pairwise, so the loads deliver every operand pair as it is consumed: sXY
// (-x_j, -x_j+1, -y_j, -y_j+1), sZU (-z_j, -z_j+1, u0_j, u0_j+1), sUU (u1_j,
// u1_j+1, u2_j, u2_j+1); sLA (lo x_j, x_j+1, lo y_j, y_j+1) and sLB (lo z_j,
// z_j+1, chain_j, chain_j+1) are read inside the exact radius or by CHECK tiles.
//
// Positions are hi + lo floats.  Separations start as d = hi_i - hi_j, whose
// error is at most 2^-23 X for a replica whose coordinates stay below X in
// magnitude; within the replica's exact radius (r <= max(2.1 beta, X / 16), so
// the hi-only relative error stays below 2^-19 where it is used) the warp adds
// the low parts, d = (hi_i - hi_j) + (lo_i - lo_j), the same rounding as a full
// hi + lo difference.  Self pairs and skipped same-chain pairs get rinv = 0,
// which zeroes their contribution without a branch; the near-overlap form
// (r <= 2 beta) lies inside the exact radius.  Far form in factored scalars:
// y = ri (c + d ri^2), (x - y)/r^2 = ri^3 (a + b ri^2), a = c0 - c2, b = c1 - c3,
// c = c2, d = c3; the near form (r^2 <= (2 beta)^2) overwrites both.
struct AaRowsF {
    float2 ax, ay, az, bx, by, bz;     // positions of rows A and B, broadcast
    float2 au[3], bu[3];               // inputs of rows A and B, broadcast
    float wA, wB;                      // chain ids
    int iA, iB, gA, gB;                // replica-local and global bead indices
};

template <bool SYM, bool CHECK, bool REF>
__device__ __forceinline__ void aa_f2_cell(const float4 *__restrict__ sXY, const float4 *__restrict__ sZU,
                                           const float4 *__restrict__ sUU, const float4 *__restrict__ sLA,
                                           const float4 *__restrict__ sLB, int jc, int s0, int ns, bool chain_hi,
                                           const AaRowsF &R, const float4 *__restrict__ plo, float2 fa, float2 fb,
                                           float2 fc, float2 fd, const Seg &sg, float te2,
                                           const double4 *__restrict__ p64, float2 (&t)[6], float2 (&c)[3])
{
    const int lane = threadIdx.x & 31;
    int k = (lane + s0) & 31;
#pragma unroll 1
    for (int s = 0; s < ns; s++) {
        const float4 XY = sXY[k], ZU = sZU[k], UU = sUU[k];
        float2 dA[3], dB[3];
        dA[0] = __fadd2_rn(R.ax, make_float2(XY.x, XY.y)); dA[1] = __fadd2_rn(R.ay, make_float2(XY.z, XY.w));
        dA[2] = __fadd2_rn(R.az, make_float2(ZU.x, ZU.y));
        dB[0] = __fadd2_rn(R.bx, make_float2(XY.x, XY.y)); dB[1] = __fadd2_rn(R.by, make_float2(XY.z, XY.w));
        dB[2] = __fadd2_rn(R.bz, make_float2(ZU.x, ZU.y));
        float2 r2A = __ffma2_rn(dA[2], dA[2], __ffma2_rn(dA[1], dA[1], __fmul2_rn(dA[0], dA[0])));
        float2 r2B = __ffma2_rn(dB[2], dB[2], __ffma2_rn(dB[1], dB[1], __fmul2_rn(dB[0], dB[0])));
        bool eA0 = false, eA1 = false, eB0 = false, eB1 = false;
        if constexpr (CHECK) {
            const int j = jc + 2 * k;
            const float4 LB = sLB[k];
            eA0 = (j == R.iA) || (chain_hi && R.wA == LB.z);
            eA1 = (j + 1 == R.iA) || (chain_hi && R.wA == LB.w);
            eB0 = (j == R.iB) || (chain_hi && R.wB == LB.z);
            eB1 = (j + 1 == R.iB) || (chain_hi && R.wB == LB.w);
        }
        const bool inner = __any_sync(0xffffffffu, fminf(fminf(r2A.x, r2A.y), fminf(r2B.x, r2B.y)) <= te2);
        if (inner) {
            const float4 LA = sLA[k], LB = sLB[k], RA = __ldg(plo + R.gA), RB = __ldg(plo + R.gB);
            const float2 cx = make_float2(-LA.x, -LA.y), cy = make_float2(-LA.z, -LA.w), cz = make_float2(-LB.x, -LB.y);
            dA[0] = __fadd2_rn(dA[0], __fadd2_rn(f2(RA.x), cx)); dA[1] = __fadd2_rn(dA[1], __fadd2_rn(f2(RA.y), cy));
            dA[2] = __fadd2_rn(dA[2], __fadd2_rn(f2(RA.z), cz));
            dB[0] = __fadd2_rn(dB[0], __fadd2_rn(f2(RB.x), cx)); dB[1] = __fadd2_rn(dB[1], __fadd2_rn(f2(RB.y), cy));
            dB[2] = __fadd2_rn(dB[2], __fadd2_rn(f2(RB.z), cz));
            r2A = __ffma2_rn(dA[2], dA[2], __ffma2_rn(dA[1], dA[1], __fmul2_rn(dA[0], dA[0])));
            r2B = __ffma2_rn(dB[2], dB[2], __ffma2_rn(dB[1], dB[1], __fmul2_rn(dB[0], dB[0])));
        }
        const float2 riA = make_float2(eA0 ? 0.f : rsqrtf(r2A.x), eA1 ? 0.f : rsqrtf(r2A.y));
        const float2 riB = make_float2(eB0 ? 0.f : rsqrtf(r2B.x), eB1 ? 0.f : rsqrtf(r2B.y));
        const float2 ri2A = __fmul2_rn(riA, riA), ri2B = __fmul2_rn(riB, riB);
        float2 yA = __fmul2_rn(__ffma2_rn(fd, ri2A, fc), riA), yB = __fmul2_rn(__ffma2_rn(fd, ri2B, fc), riB);
        float2 gA = __fmul2_rn(__ffma2_rn(fb, ri2A, fa), __fmul2_rn(ri2A, riA));
        float2 gB = __fmul2_rn(__ffma2_rn(fb, ri2B, fa), __fmul2_rn(ri2B, riB));
        if (inner) {
            const float tb2 = (float)(4.0 * sg.beta * sg.beta);
            const float nx0 = sg.aa_c[4], nx1 = sg.aa_c[5], ny0 = sg.aa_c[6], ny1 = sg.aa_c[7];
            bool nA0 = !eA0 && r2A.x <= tb2, nA1 = !eA1 && r2A.y <= tb2, nB0 = !eB0 && r2B.x <= tb2,
                 nB1 = !eB1 && r2B.y <= tb2;
            if constexpr (REF) {
                // the reference's scalars jump at 2 beta (chain bonds often sit there): within a
                // band of the FP32 test its own FP64 distance decides (RPY is continuous there)
                const double tb = 2.0 * sg.beta;
                const int j = jc + 2 * k;
                auto decide = [&](bool e, float r2, int bi, int jj, bool &n) {
                    if (e || fabsf(r2 - tb2) > 1e-5f * tb2) return;
                    const double4 P = p64[bi], Q = p64[sg.bead_off + jj];
                    n = !(ref_pair_dist(P.x - Q.x, P.y - Q.y, P.z - Q.z) > tb);
                };
                decide(eA0, r2A.x, R.gA, j, nA0); decide(eA1, r2A.y, R.gA, j + 1, nA1);
                decide(eB0, r2B.x, R.gB, j, nB0); decide(eB1, r2B.y, R.gB, j + 1, nB1);
            }
            aa_near_lane(nA0, r2A.x, riA.x, ri2A.x, nx0, nx1, ny0, ny1, yA.x, gA.x);
            aa_near_lane(nA1, r2A.y, riA.y, ri2A.y, nx0, nx1, ny0, ny1, yA.y, gA.y);
            aa_near_lane(nB0, r2B.x, riB.x, ri2B.x, nx0, nx1, ny0, ny1, yB.x, gB.x);
            aa_near_lane(nB1, r2B.y, riB.y, ri2B.y, nx0, nx1, ny0, ny1, yB.y, gB.y);
        }
        // rows: mob_a u_j = y u_j + (x - y)(d.u_j) d / r^2
        const float2 u0 = make_float2(ZU.z, ZU.w), u1 = make_float2(UU.x, UU.y), u2 = make_float2(UU.z, UU.w);
        const float2 hA = __fmul2_rn(gA, __ffma2_rn(dA[2], u2, __ffma2_rn(dA[1], u1, __fmul2_rn(dA[0], u0))));
        const float2 hB = __fmul2_rn(gB, __ffma2_rn(dB[2], u2, __ffma2_rn(dB[1], u1, __fmul2_rn(dB[0], u0))));
        t[0] = __ffma2_rn(hA, dA[0], __ffma2_rn(yA, u0, t[0]));
        t[1] = __ffma2_rn(hA, dA[1], __ffma2_rn(yA, u1, t[1]));
        t[2] = __ffma2_rn(hA, dA[2], __ffma2_rn(yA, u2, t[2]));
        t[3] = __ffma2_rn(hB, dB[0], __ffma2_rn(yB, u0, t[3]));
        t[4] = __ffma2_rn(hB, dB[1], __ffma2_rn(yB, u1, t[4]));
        t[5] = __ffma2_rn(hB, dB[2], __ffma2_rn(yB, u2, t[5]));
        if constexpr (SYM) {
            // columns: the same block applied to the rows' inputs
            const float2 kA = __fmul2_rn(gA, __ffma2_rn(dA[2], R.au[2], __ffma2_rn(dA[1], R.au[1], __fmul2_rn(dA[0], R.au[0]))));
            const float2 kB = __fmul2_rn(gB, __ffma2_rn(dB[2], R.bu[2], __ffma2_rn(dB[1], R.bu[1], __fmul2_rn(dB[0], R.bu[0]))));
#pragma unroll
            for (int a = 0; a < 3; a++) {
                c[a] = __ffma2_rn(kB, dB[a], __ffma2_rn(yB, R.bu[a], __ffma2_rn(kA, dA[a], __ffma2_rn(yA, R.au[a], c[a]))));
                // hand the column's sums to the lane that takes it next
                c[a].x = __shfl_sync(0xffffffffu, c[a].x, lane + 1);
                c[a].y = __shfl_sync(0xffffffffu, c[a].y, lane + 1);
            }
        }
        k = (k + 1) & 31;
    }
}

// columns [j0, j0 + S) of a tile as aa_f2_cell reads them, padding beyond the replica, by nt threads
template <int P>
__device__ __forceinline__ void aa_load_columns_f(const Seg &sg, int Nm, const float4 *__restrict__ pos,
                                                  const float4 *__restrict__ plo, const double *__restrict__ u, int uoff,
                                                  int j0, int S, int tid, int nt, float4 (&cols)[5][P])
{
    for (int p = tid; p < S / 2; p += nt) {
        float4 A[2], B[2];
        float v[2][3];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + 2 * p + h;
            if (j < Nm) {
                A[h] = pos[sg.bead_off + j]; B[h] = plo[sg.bead_off + j];
                for (int a = 0; a < 3; a++) v[h][a] = (float)u[uoff + 3 * j + a];
            } else {
                A[h] = make_float4(AAC_PAD, AAC_PAD, AAC_PAD, __int_as_float(0x7fc00000));
                B[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                v[h][0] = v[h][1] = v[h][2] = 0.f;
            }
        }
        cols[0][p] = make_float4(-A[0].x, -A[1].x, -A[0].y, -A[1].y);
        cols[1][p] = make_float4(-A[0].z, -A[1].z, v[0][0], v[1][0]);
        cols[2][p] = make_float4(v[0][1], v[1][1], v[0][2], v[1][2]);
        cols[3][p] = make_float4(B[0].x, B[1].x, B[0].y, B[1].y);
        cols[4][p] = make_float4(B[0].z, B[1].z, A[0].w, A[1].w);
    }
}

// rows R.iA and R.iB (padding beyond the replica; i0: a bead of the replica)
__device__ __forceinline__ void aa_load_rows_f(const Seg &sg, int Nm, const float4 *__restrict__ pos, const double *__restrict__ u,
                                               int uoff, int i0, AaRowsF &R)
{
    const bool actA = R.iA < Nm, actB = R.iB < Nm;
    R.gA = sg.bead_off + (actA ? R.iA : i0); R.gB = sg.bead_off + (actB ? R.iB : i0);
    {
        const float nan = __int_as_float(0x7fc00000);
        const float4 pad = make_float4(-AAC_PAD, -AAC_PAD, -AAC_PAD, nan);
        const float4 PA = actA ? pos[R.gA] : pad, PB = actB ? pos[R.gB] : pad;
        R.ax = f2(PA.x); R.ay = f2(PA.y); R.az = f2(PA.z); R.bx = f2(PB.x); R.by = f2(PB.y); R.bz = f2(PB.z);
        R.wA = PA.w; R.wB = PB.w;
        for (int a = 0; a < 3; a++) {
            R.au[a] = f2(actA ? (float)u[uoff + 3 * R.iA + a] : 0.f);
            R.bu[a] = f2(actB ? (float)u[uoff + 3 * R.iB + a] : 0.f);
        }
    }
}

constexpr int AAF_THREADS = 128;

template <bool REF>
__global__ void __launch_bounds__(AAF_THREADS, 4)
k_rpy_aa_f2(const Seg *__restrict__ segs, const AaTile *__restrict__ tiles, const float4 *__restrict__ pos,
            const float4 *__restrict__ plo, const float *__restrict__ aa_te2, const double4 *__restrict__ p64,
            const double *__restrict__ u, int in_top, FarOut O, const char *__restrict__ done, int done_stride)
{
    pdl_enter();
    const AaTile tl = tiles[blockIdx.x];
    if (done && *(const int *)(done + (long)tl.rep * done_stride)) return;
    const Seg &sg = segs[tl.rep];
    // one instance per pair-scalar family: the reference's scalars take the FP64 branch decision
    if ((sg.aa_mode == PS_AA_REFERENCE) != REF) return;
    __shared__ union {
        struct {
            float4 cols[5][AA_TILE_MAX / 2];               // sXY, sZU, sUU, sLA, sLB
            float col[3 * 4 * AA_TILE_MAX];                // column sums per row group or band
            double row[3 * AA_TILE_MAX];                   // row sums per column group or band (3 S slots in all)
        } aa;
        float red[2][AB_WARPS][12];
        struct { BbSmem t; double sred[AAF_THREADS / BB_ROWS - 1][11][BB_ROWS]; } bb;
    } sm;
    if (tl.S == FAR_AB) {
        ab_block<float>(sg, tl.rep, tl.I, pos, plo, u, in_top ? sg.top_off : sg.vec_off, O.tab, O.ab, O.ba, sm.red);
        return;
    }
    if (tl.S == FAR_BB) {
        bb_block<BB_ROWS, AAF_THREADS / BB_ROWS>(sg, tl.I, tl.J, p64, u, in_top ? sg.top_off : sg.vec_off, O.bb, O.bb_stride,
                                        sm.bb.t, sm.bb.sred);
        return;
    }
    float4 (&sCols)[5][AA_TILE_MAX / 2] = sm.aa.cols;
    float *sCol = sm.aa.col;
    double *sRow = sm.aa.row;
    const int Nm = sg.Nm, S = tl.S, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = tl.I * S, j0 = tl.J * S;
    const int uoff = in_top ? sg.top_off : sg.vec_off;
    aa_load_columns_f(sg, Nm, pos, plo, u, uoff, j0, S, tid, AAF_THREADS, sCols);
    // the warp's share: edge 64, one cell in four bands of 8 steps; 128, 2 x 2 cells; 256, one
    // row group of four cells each
    const int rg = S == 64 ? 0 : (S == 128 ? w >> 1 : w);
    const int cg0 = S == 128 ? w & 1 : 0, ncg = S == 256 ? 4 : 1;
    const int s0 = S == 64 ? 8 * w : 0, ns = S == 64 ? 8 : 32;
    const int rslot = S == 64 ? w : (S == 128 ? w & 1 : 0), nrslot = S == 64 ? 4 : (S == 128 ? 2 : 1);
    const int cslot = S == 64 ? w : rg, ncslot = S == 128 ? 2 : 4;
    AaRowsF R;
    R.iA = i0 + 64 * rg + lane; R.iB = R.iA + 32;
    aa_load_rows_f(sg, Nm, pos, u, uoff, i0, R);
    const bool chain_hi = sg.chain_HI != 0, diag = tl.I == tl.J;
    const float2 fa = f2(sg.aa_c[0] - sg.aa_c[2]), fb = f2(sg.aa_c[1] - sg.aa_c[3]);
    const float2 fc = f2(sg.aa_c[2]), fd = f2(sg.aa_c[3]);
    const float te2 = aa_te2[tl.rep];
    double *rs = sRow + 3 * (rslot * S + 64 * rg + lane);  // this thread's own row sums (rows A, then B)
#pragma unroll
    for (int a = 0; a < 3; a++) { rs[a] = 0.0; rs[96 + a] = 0.0; }
    __syncthreads();
    for (int cg = cg0; cg < cg0 + ncg; cg++) {
        float2 t[6] = {f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f)}, c[3] = {f2(0.f), f2(0.f), f2(0.f)};
        const int o = 32 * cg, jc = j0 + 64 * cg;
        if (diag)
            aa_f2_cell<false, true, REF>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sCols[3] + o, sCols[4] + o, jc, s0,
                                         ns, chain_hi, R, plo, fa, fb, fc, fd, sg, te2, p64, t, c);
        else if (chain_hi)
            aa_f2_cell<true, true, REF>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sCols[3] + o, sCols[4] + o, jc, s0, ns,
                                        true, R, plo, fa, fb, fc, fd, sg, te2, p64, t, c);
        else
            aa_f2_cell<true, false, REF>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sCols[3] + o, sCols[4] + o, jc, s0,
                                         ns, false, R, plo, fa, fb, fc, fd, sg, te2, p64, t, c);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            rs[a] += (double)(t[a].x + t[a].y);
            rs[96 + a] += (double)(t[3 + a].x + t[3 + a].y);
        }
        if (!diag) {
            float *o3 = sCol + 3 * (cslot * S + 64 * cg + 2 * ((lane + s0 + ns) & 31));
#pragma unroll
            for (int a = 0; a < 3; a++) { o3[a] = c[a].x; o3[3 + a] = c[a].y; }
        }
    }
    __syncthreads();
    double *oI = O.aa + sg.paa_off + (long)tl.J * sg.nm3 + 3 * i0, *oJ = O.aa + sg.paa_off + (long)tl.I * sg.nm3 + 3 * j0;
    for (int e = tid; e < 3 * S; e += AAF_THREADS) {
        if (3 * i0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < nrslot; q++) v += sRow[3 * S * q + e];
            oI[e] = v;
        }
        if (!diag && 3 * j0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < ncslot; q++) v += (double)sCol[3 * S * q + e];
            oJ[e] = v;
        }
    }
}

// AA in FP64: rows l and l + 32 of a 64-row cell in a lane's registers, one
// column per lane and step.  Reciprocal square root: a single-precision seed (the
// float image taken with integer operations) refined by the second-order
// term of the binomial series (1 - e)^(-1/2) = 1 + e/2 + 3 e^2 / 8 + O(e^3),
// e = 1 - a y0^2 (Householder's iteration of order 2 for f(y) = y^-2 - a): from
// a seed accurate to 2^-22 the truncation is below 2^-64, so the result is
// within a couple of ulp of the correctly rounded value (checked against CUDA's
// rsqrt by ps_rsqrt_check).  Self pairs and skipped same-chain pairs get
// ri = 0, which zeroes their contribution; the near form (r <= 2 beta) is taken
// under a warp vote.  Far form in factored scalars: y = ri (c + d ri^2),
// (x - y) / r^2 = ri^3 (a + b ri^2), a = c0 - c2, b = c1 - c3, c = c2, d = c3.

struct AaScalD { double ca, cb, cc, cd, tb, n0, n1, n2, n3; float tb2f; };

template <bool SYM, bool CHECK>
__device__ __forceinline__ void aa_d2_cell(const double2 *__restrict__ sXY, const double2 *__restrict__ sZU,
                                           const double2 *__restrict__ sUU, const double *__restrict__ sW, int jc, int s0,
                                           int ns, int iA, int iB, bool chain_hi, const double4 &PA, const double4 &PB,
                                           const double (&uA)[3], const double (&uB)[3], const AaScalD &K,
                                           double (&t)[6], double (&c)[3])
{
    const int lane = threadIdx.x & 31;
    int k = (lane + s0) & 31;
#pragma unroll 1
    for (int s = 0; s < ns; s++) {
        const double2 XY = sXY[k], ZU = sZU[k], UU = sUU[k];
        const double ax = PA.x - XY.x, ay = PA.y - XY.y, az = PA.z - ZU.x;
        const double bx = PB.x - XY.x, by = PB.y - XY.y, bz = PB.z - ZU.x;
        const double r2A = fma(az, az, fma(ay, ay, ax * ax));
        const double r2B = fma(bz, bz, fma(by, by, bx * bx));
        bool sA = false, sB = false;
        if constexpr (CHECK) {
            const int j = jc + k;
            sA = (j == iA) || (chain_hi && PA.w == sW[k]);
            sB = (j == iB) || (chain_hi && PB.w == sW[k]);
        }
        const float fA = trunc_to_float(r2A), fB = trunc_to_float(r2B);
        const double riA = sA ? 0.0 : rsqrt_seeded(r2A, fA), riB = sB ? 0.0 : rsqrt_seeded(r2B, fB);
        const double qA = riA * riA, qB = riB * riB;
        double yA = riA * fma(K.cd, qA, K.cc), yB = riB * fma(K.cd, qB, K.cc);
        double gA = (qA * riA) * fma(K.cb, qA, K.ca), gB = (qB * riB) * fma(K.cb, qB, K.ca);
        // candidates for the near form (a single-precision test with a 1e-6 margin, off the FP64
        // pipe); the reference's own distance decides within the band
        const bool nA = !sA && fA <= K.tb2f, nB = !sB && fB <= K.tb2f;
        if (__any_sync(0xffffffffu, nA || nB)) {
            if (nA) {
                const double r = ref_pair_dist(ax, ay, az);
                if (!(r > K.tb)) { const double ri = 1.0 / r, x = fma(K.n1, r, K.n0); yA = fma(K.n3, r, K.n2); gA = (x - yA) * ri * ri; }
            }
            if (nB) {
                const double r = ref_pair_dist(bx, by, bz);
                if (!(r > K.tb)) { const double ri = 1.0 / r, x = fma(K.n1, r, K.n0); yB = fma(K.n3, r, K.n2); gB = (x - yB) * ri * ri; }
            }
        }
        const double hA = gA * fma(az, UU.y, fma(ay, UU.x, ax * ZU.y));
        const double hB = gB * fma(bz, UU.y, fma(by, UU.x, bx * ZU.y));
        t[0] = fma(hA, ax, fma(yA, ZU.y, t[0]));
        t[1] = fma(hA, ay, fma(yA, UU.x, t[1]));
        t[2] = fma(hA, az, fma(yA, UU.y, t[2]));
        t[3] = fma(hB, bx, fma(yB, ZU.y, t[3]));
        t[4] = fma(hB, by, fma(yB, UU.x, t[4]));
        t[5] = fma(hB, bz, fma(yB, UU.y, t[5]));
        if constexpr (SYM) {
            const double kA = gA * fma(az, uA[2], fma(ay, uA[1], ax * uA[0]));
            const double kB = gB * fma(bz, uB[2], fma(by, uB[1], bx * uB[0]));
            c[0] = fma(kB, bx, fma(yB, uB[0], fma(kA, ax, fma(yA, uA[0], c[0]))));
            c[1] = fma(kB, by, fma(yB, uB[1], fma(kA, ay, fma(yA, uA[1], c[1]))));
            c[2] = fma(kB, bz, fma(yB, uB[2], fma(kA, az, fma(yA, uA[2], c[2]))));
#pragma unroll
            for (int a = 0; a < 3; a++) c[a] = __shfl_sync(0xffffffffu, c[a], lane + 1);
        }
        k = (k + 1) & 31;
    }
}

__device__ __forceinline__ AaScalD aa_scal_d(const Seg &sg)
{
    AaScalD K;
    double c0, c1, c2, c3;
    if (sg.aa_mode == PS_AA_RPY) {
        const double b = sg.beta, b2 = b * b;
        c0 = 1.5; c1 = -b2; c2 = 0.75; c3 = 0.5 * b2;
        K.n0 = 1.0 / b; K.n1 = -0.1875 / b2; K.n2 = 1.0 / b; K.n3 = -0.28125 / b2;
    } else {
        c0 = 0.375; c1 = -2.0; c2 = 0.75; c3 = -0.5;
        K.n0 = -1.0; K.n1 = 0.375; K.n2 = 1.0; K.n3 = -0.28125;
    }
    K.tb = 2.0 * sg.beta; K.ca = c0 - c2; K.cb = c1 - c3; K.cc = c2; K.cd = c3;
    K.tb2f = (float)(K.tb * K.tb * (1.0 + 1e-6));
    return K;
}

// columns [j0, j0 + S) of a tile as aa_d2_cell reads them, padding beyond the replica, by nt threads
template <int P>
__device__ __forceinline__ void aa_load_columns_d(const Seg &sg, int Nm, const double4 *__restrict__ pos,
                                                  const double *__restrict__ u, int uoff, int j0, int S, int tid, int nt,
                                                  double2 (&cols)[3][P], double *__restrict__ w)
{
    for (int p = tid; p < S; p += nt) {
        const int j = j0 + p;
        if (j < Nm) {
            const double4 P = pos[sg.bead_off + j];
            const double *v = u + uoff + 3 * j;
            cols[0][p] = make_double2(P.x, P.y);
            cols[1][p] = make_double2(P.z, v[0]);
            cols[2][p] = make_double2(v[1], v[2]);
            w[p] = P.w;
        } else {
            cols[0][p] = make_double2(AAC_PAD, AAC_PAD);
            cols[1][p] = make_double2(AAC_PAD, 0.0);
            cols[2][p] = make_double2(0.0, 0.0);
            w[p] = __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}

// rows iA and iB (padding beyond the replica)
__device__ __forceinline__ void aa_load_rows_d(const Seg &sg, int Nm, const double4 *__restrict__ pos, const double *__restrict__ u,
                                               int uoff, int iA, int iB, double4 &PA, double4 &PB, double (&uA)[3],
                                               double (&uB)[3])
{
    const bool actA = iA < Nm, actB = iB < Nm;
    const double4 pad = make_double4(-AAC_PAD, -AAC_PAD, -AAC_PAD, __longlong_as_double(0x7ff8000000000000ll));
    PA = actA ? pos[sg.bead_off + iA] : pad; PB = actB ? pos[sg.bead_off + iB] : pad;
    for (int a = 0; a < 3; a++) {
        uA[a] = actA ? u[uoff + 3 * iA + a] : 0.0;
        uB[a] = actB ? u[uoff + 3 * iB + a] : 0.0;
    }
}

constexpr int AAD_THREADS = 256;

__global__ void __launch_bounds__(AAD_THREADS, 2)
k_rpy_aa_d2(const Seg *__restrict__ segs, const AaTile *__restrict__ tiles, const double4 *__restrict__ pos,
            const double *__restrict__ u, int in_top, FarOut O, const char *__restrict__ done, int done_stride)
{
    pdl_enter();
    const AaTile tl = tiles[blockIdx.x];
    if (done && *(const int *)(done + (long)tl.rep * done_stride)) return;
    __shared__ union {
        struct {
            double2 cols[3][AA_TILE_MAX];                  // x, y | z, u0 | u1, u2; then the row sums in the same space
            double w[AA_TILE_MAX], col[3 * 4 * AA_TILE_MAX];   // chain ids; column sums per row group or band
        } aa;
        double red[2][AB_WARPS][12];
        struct { BbSmem t; double sred[AAD_THREADS / BB_ROWS - 1][11][BB_ROWS]; } bb;
    } sm;
    const Seg &sg = segs[tl.rep];
    if (tl.S == FAR_AB) {
        ab_block<double>(sg, tl.rep, tl.I, pos, nullptr, u, in_top ? sg.top_off : sg.vec_off, O.tab, O.ab, O.ba, sm.red);
        return;
    }
    if (tl.S == FAR_BB) {
        bb_block<BB_ROWS, AAD_THREADS / BB_ROWS>(sg, tl.I, tl.J, pos, u, in_top ? sg.top_off : sg.vec_off, O.bb, O.bb_stride,
                                            sm.bb.t, sm.bb.sred);
        return;
    }
    double2 (&sCols)[3][AA_TILE_MAX] = sm.aa.cols;
    double *sW = sm.aa.w, *sCol = sm.aa.col;
    double *sRow = reinterpret_cast<double *>(sCols);      // row sums per column group or band: 1536 doubles
    static_assert(sizeof(sm.aa.cols) >= 1536 * sizeof(double), "row sums alias the columns");
    const int Nm = sg.Nm, S = tl.S, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = tl.I * S, j0 = tl.J * S;
    const int uoff = in_top ? sg.top_off : sg.vec_off;
    aa_load_columns_d(sg, Nm, pos, u, uoff, j0, S, tid, AAD_THREADS, sCols, sW);
    // the warp's share: edge 64, one 64 x 32 cell per column group in four bands of 8 steps;
    // 128, 2 x 4 cells; 256, a row group's four cells of one half of the columns
    const int rg = S == 64 ? 0 : (S == 128 ? w >> 2 : w >> 1);
    const int cg0 = S == 64 ? w & 1 : (S == 128 ? w & 3 : 4 * (w & 1)), ncg = S == 256 ? 4 : 1;
    const int s0 = S == 64 ? 8 * (w >> 1) : 0, ns = S == 64 ? 8 : 32;
    const int rslot = S == 64 ? w : (S == 128 ? w & 3 : w & 1), nrslot = S == 64 ? 8 : (S == 128 ? 4 : 2);
    const int cslot = S == 64 ? w >> 1 : rg, ncslot = S == 128 ? 2 : 4;
    const int iA = i0 + 64 * rg + lane, iB = iA + 32;
    double4 PA, PB;
    double uA[3], uB[3];
    aa_load_rows_d(sg, Nm, pos, u, uoff, iA, iB, PA, PB, uA, uB);
    const bool chain_hi = sg.chain_HI != 0, diag = tl.I == tl.J;
    const AaScalD K = aa_scal_d(sg);
    __syncthreads();
    double racc[6] = {0, 0, 0, 0, 0, 0};
    for (int cg = cg0; cg < cg0 + ncg; cg++) {
        double c[3] = {0, 0, 0};
        const int o = 32 * cg, jc = j0 + o;
        if (diag)
            aa_d2_cell<false, true>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, s0, ns, iA, iB, chain_hi, PA,
                                    PB, uA, uB, K, racc, c);
        else if (chain_hi)
            aa_d2_cell<true, true>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, s0, ns, iA, iB, true, PA, PB,
                                   uA, uB, K, racc, c);
        else
            aa_d2_cell<true, false>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, s0, ns, iA, iB, false, PA, PB,
                                    uA, uB, K, racc, c);
        if (!diag) {
            double *o3 = sCol + 3 * (cslot * S + o + ((lane + s0 + ns) & 31));
#pragma unroll
            for (int a = 0; a < 3; a++) o3[a] = c[a];
        }
    }
    __syncthreads();                                       // the columns have been read
    {
        double *o3 = sRow + 3 * (rslot * S + 64 * rg + lane);
#pragma unroll
        for (int a = 0; a < 3; a++) { o3[a] = racc[a]; o3[96 + a] = racc[3 + a]; }
    }
    __syncthreads();
    double *oI = O.aa + sg.paa_off + (long)tl.J * sg.nm3 + 3 * i0, *oJ = O.aa + sg.paa_off + (long)tl.I * sg.nm3 + 3 * j0;
    for (int e = tid; e < 3 * S; e += AAD_THREADS) {
        if (3 * i0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < nrslot; q++) v += sRow[3 * S * q + e];
            oI[e] = v;
        }
        if (!diag && 3 * j0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < ncslot; q++) v += sCol[3 * S * q + e];
            oJ[e] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Tile pairs of edge 64 by two warps each, for launches of many: the bands that the block kernels give to a
// warp each are taken one after the other, and the same sums are joined in the same order, so the
// slots hold the same bits.  A block of all bands spreads a lone replica; where the tile pairs fill the
// chip many times over, its barriers, its idle warps and the steps that meet padding only are what a
// launch takes.  Padding adds exact zeros, so cells of padding columns and, in a diagonal cell, steps
// without a pair are left out.
//
// Taken for contexts whose tile pairs are all of edge 64 and more than AAN_MIN_TILES (two and one waves of the
// block kernels in FP64 and FP32), or, where monomer-colloid and colloid blocks then need a launch of
// their own, than AAN_MIN_WITH_PRE (four waves) unless every replica has a few beads only.  One apply, block
// -> two warps, us, FP64 / FP32: 1000 replicas of 3 beads 22.7 -> 8.1 / 14.5 -> 8.0, of 65 beads 57.3 ->
// 30.7 / 33.7 -> 27.5, 100 of 1000 beads 240 -> 185 / 124 -> 104; 30 of 200 beads (300 tile pairs) 12.1 ->
// 16.3 / 10.0 -> 12.2; with probes, 128 replicas of 64 to 700 beads (2000 tile pairs) 46.4 -> 42.4 / 28.0 ->
// 29.2, 48 of them 22.4 -> 26.9 / 15.8 -> 19.4.
constexpr int AAN_THREADS = 64, AAN_BLOCKS = 8;
constexpr int AAN_MIN_TILES = 4 * 148, AAN_MIN_WITH_PRE[2] = {8 * 148, 16 * 148};      // FP64, FP32

// [s0, s1) and [s2, s0 + 8): the steps of a diagonal band that meet a pair, where rows sit in lanes below nr and
// lane l holds column (l + s) mod 32, one of nc
__device__ __forceinline__ void aa_band_steps(int s0, int nr, int nc, int &s1, int &s2)
{
    s1 = min(s0 + 8, max(s0, nc));
    s2 = min(s0 + 8, max(s1, 33 - nr));
}

__global__ void __launch_bounds__(AAN_THREADS, AAN_BLOCKS)
k_rpy_aa_dn(const Seg *__restrict__ segs, const AaTile *__restrict__ tiles, const double4 *__restrict__ pos,
            const double *__restrict__ u, int in_top, double *__restrict__ paa, const char *__restrict__ done, int done_stride)
{
    pdl_enter();
    __shared__ double2 sCols[3][64];
    __shared__ double sW[64], sRow[8 * 192], sCol[4 * 192];
    const AaTile tl = tiles[blockIdx.x];
    if (done && *(const int *)(done + (long)tl.rep * done_stride)) return;
    const Seg &sg = segs[tl.rep];
    const int Nm = sg.Nm, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = 64 * tl.I, j0 = 64 * tl.J, uoff = in_top ? sg.top_off : sg.vec_off;
    aa_load_columns_d(sg, Nm, pos, u, uoff, j0, 64, tid, AAN_THREADS, sCols, sW);
    const int iA = i0 + lane, iB = iA + 32;
    double4 PA, PB;
    double uA[3], uB[3];
    aa_load_rows_d(sg, Nm, pos, u, uoff, iA, iB, PA, PB, uA, uB);
    const bool chain_hi = sg.chain_HI != 0, diag = tl.I == tl.J;
    const AaScalD K = aa_scal_d(sg);
    __syncthreads();
    for (int q = 4 * w; q < 4 * w + 4; q++) {              // band q / 2 of column group q mod 2
        const int b = q >> 1, s0 = 8 * b, o = 32 * (q & 1), jc = j0 + o;
        double t[6] = {0, 0, 0, 0, 0, 0}, c[3] = {0, 0, 0};
        if (jc >= Nm) ;
        else if (diag) {
            int s1, s2;
            aa_band_steps(s0, Nm - i0, Nm - jc, s1, s2);
            for (int h = 0; h < 2; h++)
                aa_d2_cell<false, true>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, h ? s2 : s0,
                                        h ? s0 + 8 - s2 : s1 - s0, iA, iB, chain_hi, PA, PB, uA, uB, K, t, c);
        } else if (chain_hi)
            aa_d2_cell<true, true>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, s0, 8, iA, iB, true, PA, PB, uA, uB,
                                   K, t, c);
        else
            aa_d2_cell<true, false>(sCols[0] + o, sCols[1] + o, sCols[2] + o, sW + o, jc, s0, 8, iA, iB, false, PA, PB, uA, uB,
                                    K, t, c);
        double *r = sRow + 192 * q + 3 * lane, *o3 = sCol + 192 * b + 3 * (o + ((lane + s0 + 8) & 31));
        for (int a = 0; a < 3; a++) { r[a] = t[a]; r[96 + a] = t[3 + a]; o3[a] = c[a]; }
    }
    __syncthreads();
    double *oI = paa + sg.paa_off + (long)tl.J * sg.nm3 + 3 * i0, *oJ = paa + sg.paa_off + (long)tl.I * sg.nm3 + 3 * j0;
    for (int e = tid; e < 192; e += AAN_THREADS) {
        if (3 * i0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < 8; q++) v += sRow[192 * q + e];
            oI[e] = v;
        }
        if (!diag && 3 * j0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < 4; q++) v += sCol[192 * q + e];
            oJ[e] = v;
        }
    }
}

template <bool REF>
__global__ void __launch_bounds__(AAN_THREADS, AAN_BLOCKS)
k_rpy_aa_fn(const Seg *__restrict__ segs, const AaTile *__restrict__ tiles, const float4 *__restrict__ pos,
            const float4 *__restrict__ plo, const float *__restrict__ aa_te2, const double4 *__restrict__ p64,
            const double *__restrict__ u, int in_top, double *__restrict__ paa, const char *__restrict__ done, int done_stride)
{
    pdl_enter();
    __shared__ float4 sCols[5][32];
    __shared__ double sRow[4 * 192];
    __shared__ float sCol[4 * 192];
    const AaTile tl = tiles[blockIdx.x];
    if (done && *(const int *)(done + (long)tl.rep * done_stride)) return;
    const Seg &sg = segs[tl.rep];
    if ((sg.aa_mode == PS_AA_REFERENCE) != REF) return;
    const int Nm = sg.Nm, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = 64 * tl.I, j0 = 64 * tl.J, uoff = in_top ? sg.top_off : sg.vec_off;
    aa_load_columns_f(sg, Nm, pos, plo, u, uoff, j0, 64, tid, AAN_THREADS, sCols);
    AaRowsF R;
    R.iA = i0 + lane; R.iB = R.iA + 32;
    aa_load_rows_f(sg, Nm, pos, u, uoff, i0, R);
    const bool chain_hi = sg.chain_HI != 0, diag = tl.I == tl.J;
    const float2 fa = f2(sg.aa_c[0] - sg.aa_c[2]), fb = f2(sg.aa_c[1] - sg.aa_c[3]);
    const float2 fc = f2(sg.aa_c[2]), fd = f2(sg.aa_c[3]);
    const float te2 = aa_te2[tl.rep];
    __syncthreads();
    for (int b = 2 * w; b < 2 * w + 2; b++) {
        const int s0 = 8 * b;
        float2 t[6] = {f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f)}, c[3] = {f2(0.f), f2(0.f), f2(0.f)};
        if (diag) {
            int s1, s2;
            aa_band_steps(s0, Nm - i0, (Nm - j0 + 1) / 2, s1, s2);
            for (int h = 0; h < 2; h++)
                aa_f2_cell<false, true, REF>(sCols[0], sCols[1], sCols[2], sCols[3], sCols[4], j0, h ? s2 : s0,
                                             h ? s0 + 8 - s2 : s1 - s0, chain_hi, R, plo, fa, fb, fc, fd, sg, te2, p64, t, c);
        } else if (chain_hi)
            aa_f2_cell<true, true, REF>(sCols[0], sCols[1], sCols[2], sCols[3], sCols[4], j0, s0, 8, true, R, plo, fa, fb, fc,
                                        fd, sg, te2, p64, t, c);
        else
            aa_f2_cell<true, false, REF>(sCols[0], sCols[1], sCols[2], sCols[3], sCols[4], j0, s0, 8, false, R, plo, fa, fb, fc,
                                         fd, sg, te2, p64, t, c);
        double *r = sRow + 192 * b + 3 * lane;
        for (int a = 0; a < 3; a++) { r[a] = (double)(t[a].x + t[a].y); r[96 + a] = (double)(t[3 + a].x + t[3 + a].y); }
        float *o3 = sCol + 192 * b + 6 * ((lane + s0 + 8) & 31);
        for (int a = 0; a < 3; a++) { o3[a] = c[a].x; o3[3 + a] = c[a].y; }
    }
    __syncthreads();
    double *oI = paa + sg.paa_off + (long)tl.J * sg.nm3 + 3 * i0, *oJ = paa + sg.paa_off + (long)tl.I * sg.nm3 + 3 * j0;
    for (int e = tid; e < 192; e += AAN_THREADS) {
        if (3 * i0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < 4; q++) v += sRow[192 * q + e];
            oI[e] = v;
        }
        if (!diag && 3 * j0 + e < sg.nm3) {
            double v = 0.0;
            for (int q = 0; q < 4; q++) v += (double)sCol[192 * q + e];
            oJ[e] = v;
        }
    }
}

// max |own - CUDA| / ulp(CUDA) of the reciprocal square root over a[0..n)
__global__ void k_rsqrt_check(long n, const double *__restrict__ a, unsigned long long *__restrict__ worst)
{
    pdl_enter();
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double ref = rsqrt(a[i]), own = rsqrt_seeded(a[i]);
    long long d = __double_as_longlong(own) - __double_as_longlong(ref);
    atomicMax(worst, (unsigned long long)(d < 0 ? -d : d));
}

// ---------------------------------------------------------------------------
// Combine: self terms + pair partials (fixed order) + constraint blocks.
// mode 0: saddle   y = [[M, B], [B^T, -R_lub]] x   (vectors in saddle layout)
// mode 1: mobility y_top = M u                      (vectors in top layout)

// v + the n partial sums p[0], p[stride], ... in order, eight loads in flight
__device__ __forceinline__ double add_slots(double v, const double *__restrict__ p, int n, long stride)
{
    for (int c = 0; c < n; c += 8) {
        double t[8];
#pragma unroll
        for (int k = 0; k < 8; k++) t[k] = c + k < n ? p[(c + k) * stride] : 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) v += t[k];
    }
    return v;
}

// what a combine goes on with
enum { CB_PLAIN, CB_DOTS, CB_MINRES };
struct NoTail {};

// entry k (index i within the replica) of the product
__device__ __forceinline__ double combine_entry(const Seg &sg, int mode, int i, int xo, const double *__restrict__ x,
                                                const double *__restrict__ partAA, int with_aa,
                                                const double *__restrict__ partAB, const double *__restrict__ partBB,
                                                const double *__restrict__ partBA, const double *__restrict__ delta,
                                                const double *__restrict__ lub_y, long part_stride)
{
    double v = 0.0;
    if (i < sg.nm3nc11) {
        if (i < sg.nm3) {
            v = sg.beta_inv * x[xo + i];
            if (with_aa) {
                v = add_slots(v, partAA + sg.paa_off + i, sg.aa_nt, sg.nm3);      // one slot per column tile
            }
            if (sg.Nc > 0) v += partAB[sg.top_off + i];
        } else {
            int j = i - sg.nm3;          // colloid-local DOF in [0, nc11)
            int cidx, q;                 // colloid index, component
            double self;
            if (j < sg.nc3) { cidx = j / 3; q = j % 3; self = x[xo + i]; }
            else if (j < sg.nc6) { cidx = (j - sg.nc3) / 3; q = 3 + (j - sg.nc3) % 3; self = 0.75 * x[xo + i]; }
            else {
                cidx = (j - sg.nc6) / 5; q = 6 + (j - sg.nc6) % 5;
                int sb = xo + sg.nm3nc6 + 5 * cidx, p = q - 6;
                self = 1.8 * x[sb + p];
                if (p == 0) self += 0.9 * x[sb + 4];
                if (p == 4) self += 0.9 * x[sb + 0];
            }
            v = self;
            if (sg.Nc >= 2) {
                v = add_slots(v, partBB + sg.top_off + i, sg.nch_bb, part_stride);
            }
            if (sg.Nm > 0)
                for (int t = 0; t < sg.n_mtiles; t++) v += partBA[((long)sg.ba_off + (long)t * sg.Nc + cidx) * 11 + q];
            if (sg.shell_schur) {
                const double *D = delta + sg.schur_off + (long)j * sg.nc11;
                double acc = 0.0;
                for (int b = 0; b < sg.nc11; b++) acc += D[b] * x[xo + sg.nm3 + b];
                v += acc;
            }
        }
        if (mode == 0 && i < sg.nm3nc6) v -= x[xo + sg.nm3nc11 + i];
    } else {
        int j = i - sg.nm3nc11;
        v = -x[xo + j];
        if (sg.lub_on && lub_y) v -= lub_y[sg.vel_off + j];
    }
    return v;
}

// A block of the grid per entry of the replica-aligned block table of the output layout (saddle vectors for
// mode 0, mobility vectors for mode 1) and sub-block of it (blockIdx.y), an output per thread: the
// replica is known without a search, a converged replica's blocks leave at once, and a single
// replica's partial sums are read by as many threads as it has outputs.
template <int TAIL, class X>
__global__ void k_combine(const Seg *__restrict__ segs, RedTable T, int mode, const double *__restrict__ x,
                          const double *__restrict__ partAA, int with_aa,
                          const double *__restrict__ partAB, const double *__restrict__ partBB,
                          const double *__restrict__ partBA, const double *__restrict__ delta,
                          const double *__restrict__ lub_y, long part_stride, double *__restrict__ y,
                          const char *__restrict__ done, int done_stride, X tail)
{
    pdl_enter();
    const RBlk B = T.d_blk[blockIdx.x];
    const int r = B.rep;
    if (done && *(const int *)(done + (long)r * done_stride)) {         // converged replica: skip
        if constexpr (TAIL == CB_MINRES)
            if (blockIdx.y == 0 && (int)blockIdx.x == T.d_first[r] && threadIdx.x == 0) tail.st1[r] = tail.st0[r];
        return;
    }
    const Seg &sg = segs[r];
    const int xo = mode == 0 ? sg.vec_off : sg.top_off;
    // one entry per thread
    const int e = blockIdx.y * RB_THREADS + threadIdx.x;
    const long k = (long)B.start + e;
    double out = 0.0;
    if (e < B.len) {
        out = combine_entry(sg, mode, (int)(k - xo), xo, x, partAA, with_aa, partAB, partBB, partBA, delta, lub_y, part_stride);
        if constexpr (TAIL != CB_MINRES) y[k] = out;
    }
    if (blockIdx.y * RB_THREADS >= B.len) return;
    if constexpr (TAIL == CB_DOTS)
        lz_block_dots(tail.V, tail.ldv, k, e < B.len, out, tail.j,
                      tail.part + (long)LZ_KMAX * (RB_EPT * blockIdx.x + blockIdx.y));
    if constexpr (TAIL == CB_MINRES) mr_alpha(T, B, sg.n, k, e < B.len, out, tail, y);
}

// ---------------------------------------------------------------------------
// host launchers
// Far-field blocks of the replicas with monomers: monomer-colloid and colloid-colloid
// blocks first (E.n_far_pre of them), then the monomer tile pairs, in one launch per
// pair-scalar family (in launches of their own on a side stream, the first two kinds cost 6 us of
// fork and join on an apply of 12 us).  Colloid-colloid FTS blocks stay FP64 in the mixed
// form: near contact the far-field FTS mobility is ill-conditioned and FP32 blocks leave a
// 1.2e-6 velocity error on a suspension at gap 0.01 (FP64: tracks rtol); they are cheap
// wherever monomers carry the O(N^2) work.
static void launch_far(Engine &E, const double *u, int in_top, bool fp32, int first, int n, cudaStream_t st,
                       const char *done, int dstride)
{
    if (n <= 0) return;
    const FarOut O = {E.d_partAA, E.d_partAB, E.d_partBA, E.d_partBB, E.d_tab, E.part_stride};
    const AaTile *tiles = E.d_aa_tiles + first;
    if (!fp32) {
        ps_launch(k_rpy_aa_d2, n, AAD_THREADS, 0, st, E.d_segs, tiles, E.d_pos64, u, in_top, O, done, dstride);
        return;
    }
    if (E.any_aa_rpy)
        ps_launch(k_rpy_aa_f2<false>, n, AAF_THREADS, 0, st, E.d_segs, tiles, E.d_pos32, E.d_pos32lo, E.d_aa_te2, E.d_pos64,
                u, in_top, O, done, dstride);
    if (E.any_aa_ref)
        ps_launch(k_rpy_aa_f2<true>, n, AAF_THREADS, 0, st, E.d_segs, tiles, E.d_pos32, E.d_pos32lo, E.d_aa_te2, E.d_pos64,
                u, in_top, O, done, dstride);
}

// the monomer tile pairs where k_rpy_aa_dn and k_rpy_aa_fn take them all (set_aa_chunking)
static void launch_far_narrow(Engine &E, const double *u, int in_top, bool fp32, cudaStream_t st, const char *done, int dstride)
{
    const int n = E.n_aa_tiles;
    if (!n || !E.aa_narrow[fp32]) return;
    const AaTile *tiles = E.d_aa_tiles + E.n_far_pre;
    if (!fp32) {
        ps_launch(k_rpy_aa_dn, n, AAN_THREADS, 0, st, E.d_segs, tiles, E.d_pos64, u, in_top, E.d_partAA, done, dstride);
        return;
    }
    if (E.any_aa_rpy)
        ps_launch(k_rpy_aa_fn<false>, n, AAN_THREADS, 0, st, E.d_segs, tiles, E.d_pos32, E.d_pos32lo, E.d_aa_te2, E.d_pos64, u,
                in_top, E.d_partAA, done, dstride);
    if (E.any_aa_ref)
        ps_launch(k_rpy_aa_fn<true>, n, AAN_THREADS, 0, st, E.d_segs, tiles, E.d_pos32, E.d_pos32lo, E.d_aa_te2, E.d_pos64, u,
                in_top, E.d_partAA, done, dstride);
}

static void launch_bb(Engine &E, const double *u, int in_top, cudaStream_t st, const char *done, int dstride)
{
    if (!E.n_bb_tiles) return;
    const dim3 grid(E.n_bb_tiles, E.nch_bb);
    if (E.bb_wide)
        ps_launch(k_rpy_bb<BB_WIDE>, grid, BB_WIDE * BB_SPLIT, 0, st, E.d_segs, E.d_bb_tiles, E.d_pos64, u, in_top, E.d_partBB,
                E.part_stride, done, dstride);
    else
        ps_launch(k_rpy_bb<BB_ROWS>, grid, BB_ROWS * BB_SPLIT, 0, st, E.d_segs, E.d_bb_tiles, E.d_pos64, u, in_top, E.d_partBB,
                E.part_stride, done, dstride);
}

void apply_operator(Engine &E, int mode, const double *x, double *y, bool fp32, cudaStream_t st,
                    const void *done, int done_stride, bool skip_aa, const LzDots *dots, const MrAlpha *mr)
{
    int in_top = mode == 1;
    const char *dn = (const char *)done;
    launch_far(E, x, in_top, fp32, 0, E.n_far_pre + (skip_aa || E.aa_narrow[fp32] ? 0 : E.n_aa_tiles), st, dn, done_stride);
    if (!skip_aa) launch_far_narrow(E, x, in_top, fp32, st, dn, done_stride);
    launch_bb(E, x, in_top, st, dn, done_stride);
    const double *lub_y = nullptr;
    if (mode == 0 && E.any_lub) {
        lub_apply(E, x, E.d_luby, st);
        lub_y = E.d_luby;
    }
    const RedTable &T = mode == 0 ? E.red : E.red_top;
    const dim3 grid((unsigned)T.nblk, (unsigned)T.nsub);
    const int with_aa = skip_aa ? 0 : 1;
    if (dots)
        ps_launch(k_combine<CB_DOTS, LzDots>, grid, RB_THREADS, 0, st, E.d_segs, T, mode, x, E.d_partAA, with_aa, E.d_partAB, E.d_partBB,
                E.d_partBA, E.d_delta, lub_y, E.part_stride, y, dn, done_stride, *dots);
    else if (mr)
        ps_launch(k_combine<CB_MINRES, MrAlpha>, grid, RB_THREADS, 0, st, E.d_segs, T, mode, x, E.d_partAA, with_aa, E.d_partAB, E.d_partBB,
                E.d_partBA, E.d_delta, lub_y, E.part_stride, y, dn, done_stride, *mr);
    else
        ps_launch(k_combine<CB_PLAIN, NoTail>, grid, RB_THREADS, 0, st, E.d_segs, T, mode, x, E.d_partAA, with_aa, E.d_partAB, E.d_partBB,
                E.d_partBA, E.d_delta, lub_y, E.part_stride, y, dn, done_stride, NoTail{});
}

int g_aa_chunk_cols = AA_TILE_MAX;

static int capped_edge(const Seg &s, int cols) { return std::min(aa_tile_edge(s.Nm), std::max(cols, AA_TILE_MIN)); }

bool same_aa_chunking(const Engine &E, int a, int b)
{
    return std::all_of(E.segs.begin(), E.segs.end(), [&](const Seg &s) {
        return !s.mm_HI || s.Nm < 2 || capped_edge(s, a) == capped_edge(s, b);
    });
}

// tiles of the monomer far field for a widest edge of `cols`: per-replica edges and
// partial slots, the list of tile pairs (large tiles first) and the partial buffer
int set_aa_chunking(Engine &E, int cols)
{
    std::vector<AaTile> pre, tiles;
    long off = 0;
    for (int r = 0; r < E.R; r++) {
        Seg &s = E.segs[r];
        const bool on = s.mm_HI && s.Nm >= 2;
        const int S = capped_edge(s, cols);
        s.aa_nt = on ? (s.Nm + S - 1) / S : 0;
        s.paa_off = off;
        off += (long)s.aa_nt * s.nm3;
        for (int i = 0; i < s.aa_nt; i++)
            for (int j = i; j < s.aa_nt; j++) tiles.push_back({r, i, j, S});
        if (s.Nm > 0) {
            if (s.Nc > 0)
                for (int t = 0; t < s.n_mtiles; t++) pre.push_back({r, t, 0, FAR_AB});
            if (s.Nc >= 2)
                for (int t = 0; t * BB_ROWS < s.Nc; t++)
                    for (int c = 0; c < s.nch_bb; c++) pre.push_back({r, t, c, FAR_BB});
        }
    }
    std::stable_sort(tiles.begin(), tiles.end(), [](const AaTile &a, const AaTile &b) { return a.S > b.S; });
    E.n_aa_tiles = (int)tiles.size();
    E.n_far_pre = (int)pre.size();
    const bool narrow = std::all_of(tiles.begin(), tiles.end(), [](const AaTile &t) { return t.S == AA_TILE_MIN; });
    const bool tiny = std::all_of(E.segs.begin(), E.segs.end(), [](const Seg &s) { return s.Nm <= 32; });
    for (int f = 0; f < 2; f++)
        E.aa_narrow[f] = narrow && E.n_aa_tiles > (pre.empty() || tiny ? AAN_MIN_TILES : AAN_MIN_WITH_PRE[f]);
    tiles.insert(tiles.begin(), pre.begin(), pre.end());
    PS_CK(cudaDeviceSynchronize());
    cudaFree(E.d_partAA);
    cudaFree(E.d_aa_tiles);
    E.d_partAA = nullptr;
    E.d_aa_tiles = nullptr;
    if (cudaMalloc(&E.d_partAA, sizeof(double) * std::max<long>(off, 1)) != cudaSuccess ||
        cudaMalloc(&E.d_aa_tiles, sizeof(AaTile) * std::max<size_t>(tiles.size(), 1)) != cudaSuccess) {
        set_error(std::string("monomer far-field partial sums: ") + cudaGetErrorString(cudaGetLastError()));
        return PS_ERR_NOMEM;
    }
    if (!tiles.empty())
        PS_CK(cudaMemcpy(E.d_aa_tiles, tiles.data(), sizeof(AaTile) * tiles.size(), cudaMemcpyHostToDevice));
    PS_CK(cudaMemcpy(E.d_segs, E.segs.data(), sizeof(Seg) * E.segs.size(), cudaMemcpyHostToDevice));
    PS_CK(cudaDeviceSynchronize());      // a copy from pageable memory may return ahead of its transfer
    return PS_OK;
}

// ---------------------------------------------------------------------------
// diagnostics: average duration (CUDA events on `st`) of one far-field kernel
// which: 0 monomer pairs, 1 monomer-colloid pairs and the colloid pairs beside monomers, 2 colloid pairs of
// replicas without monomers, 3 whole mobility apply
int time_pairs(Engine &E, int which, int reps, const double *u, double *ms, cudaStream_t st)
{
    bool fp32 = E.precision == PS_PREC_MIXED;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    auto launch = [&]() {
        if (which == 0) {
            if (!E.aa_narrow[fp32]) launch_far(E, u, 1, fp32, E.n_far_pre, E.n_aa_tiles, st, nullptr, 0);
            launch_far_narrow(E, u, 1, fp32, st, nullptr, 0);
        } else if (which == 1) {
            launch_far(E, u, 1, fp32, 0, E.n_far_pre, st, nullptr, 0);
        } else if (which == 2) {
            launch_bb(E, u, 1, st, nullptr, 0);
        } else if (which == 3) {
            apply_operator(E, 1, u, E.d_tmp_top2, fp32, st);
        }
    };
    launch();   // warm
    cudaEventRecord(a, st);
    for (int k = 0; k < reps; k++) launch();
    cudaEventRecord(b, st);
    cudaEventSynchronize(b);
    float t = 0;
    cudaEventElapsedTime(&t, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    *ms = reps > 0 ? (double)t / reps : 0.0;
    PS_CK(cudaGetLastError());
    return PS_OK;
}

// largest distance in ulp between rsqrt_seeded and CUDA's rsqrt over a device array
int rsqrt_check(const double *a, long n, unsigned long long *max_ulp, cudaStream_t st)
{
    unsigned long long *d = nullptr;
    PS_CK(cudaMallocAsync(&d, sizeof(unsigned long long), st));
    PS_CK(cudaMemsetAsync(d, 0, sizeof(unsigned long long), st));
    if (n > 0) ps_launch(k_rsqrt_check, (unsigned)((n + 255) / 256), 256, 0, st, n, a, d);
    PS_CK(cudaMemcpyAsync(max_ulp, d, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    PS_CK(cudaFreeAsync(d, st));
    PS_CK(cudaStreamSynchronize(st));
    return PS_OK;
}

// measured FMA throughput: 8 independent FMA chains per thread, all SMs busy
template <class T>
__global__ void k_fma(T *out, int iters, T seed)
{
    pdl_enter();
    T a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = seed + T(k) * T(1e-3) + T(threadIdx.x) * T(1e-7);
    const T m = T(0.999999), c = T(1e-7);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = a[k] * m + c;
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k];
    if (s == T(-12345)) out[0] = s;
}

// the same with packed FP32x2 FMAs (FFMA2): 8 independent float2 chains per thread
__global__ void k_fma2(float *out, int iters, float seed)
{
    pdl_enter();
    float2 a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = make_float2(seed + k * 1e-3f + threadIdx.x * 1e-7f, seed - k * 1e-3f);
    const float2 m = make_float2(0.999999f, 0.999999f), c = make_float2(1e-7f, 1e-7f);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = __ffma2_rn(a[k], m, c);
    }
    float s = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k].x + a[k].y;
    if (s == -12345.f) out[0] = s;
}

int fma_peak(int fp64, double *tflops, cudaStream_t st)
{
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    void *buf = nullptr;
    PS_CK(cudaMalloc(&buf, 64));
    const int thr = 256, blocks = nsm * 8, iters = 1 << 14;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    // FP32: the larger of the scalar and the packed (FFMA2) throughput
    double best_tf = 0;
    for (int form = 0; form < (fp64 ? 1 : 2); form++) {
        float best = 1e30f;
        for (int rep = 0; rep < 4; rep++) {
            cudaEventRecord(a, st);
            if (fp64) ::ps_launch_count++, k_fma<double><<<blocks, thr, 0, st>>>((double *)buf, iters, 1.0);
            else if (form == 0) ::ps_launch_count++, k_fma<float><<<blocks, thr, 0, st>>>((float *)buf, iters, 1.0f);
            else ::ps_launch_count++, k_fma2<<<blocks, thr, 0, st>>>((float *)buf, iters / 2, 1.0f);
            cudaEventRecord(b, st);
            cudaEventSynchronize(b);
            float t = 0;
            cudaEventElapsedTime(&t, a, b);
            if (rep > 0) best = std::min(best, t);
        }
        // both forms: 8 chains x iters FMA per thread (packed: iters / 2 steps of 2 lanes)
        double flops = 2.0 * 8.0 * (double)iters * thr * blocks;
        best_tf = std::max(best_tf, flops / (best * 1e-3) / 1e12);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(buf);
    *tflops = best_tf;
    PS_CK(cudaGetLastError());
    return PS_OK;
}
}  // namespace ps
