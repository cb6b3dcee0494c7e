// ps_reduce.cuh -- segmented per-replica reductions shared by the Krylov
// solvers: a block covers a contiguous range of one replica's vector; the last
// block of a replica to arrive (atomic counter) sums the partials in fixed
// order, so results never depend on block scheduling or on other replicas.
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

// A block's dots of its entries (one per thread: value q at index k, when act) with the
// Lanczos vectors V_0..V_j, into out[0..j]; RB_THREADS threads, every one of which takes part.
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
