// Device helpers shared by the persistent kernels: bounded grid barrier and
// deterministic reductions.
#pragma once

#include "fg_internal.h"

namespace fg {

// ---------------------------------------------------------------------------------
// small helpers

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier for cooperative (co-resident) launches: one arrival (release) per block on a
// counter that only grows, then a wait (acquire) until the last block's arrival is counted. That is
// two trips to L2 where there was one for each of a generation read, the arrival, its reset and
// release, the wait and a read of the error flag by every thread (solve of 7.7k tets, 18 barriers,
// 127 -> 108 us; of the 1.2M-tet film in FP64 0.48 -> 0.46 ms). The wait is bounded: a block that saw no
// progress for 2 s takes the round back (the counter returns to the round's begin, marked expired)
// and returns false. It can do so only while an arrival is missing, and a marked round never
// completes: a block that arrives late, or still waits, returns false too. So every block passes a
// round or none does, each leaves the kernel at the same barrier, and no launch can hang the GPU.
__device__ inline bool grid_sync(GridBar *gb) {
    if (gridDim.x == 1) {  // a single block meets itself
        __syncthreads();
        return true;
    }
    int ok = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        constexpr unsigned long long EXPIRED = 1ull << 63;
        unsigned long long ticket, seen;
        asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(ticket) : "l"(&gb->count) : "memory");
        const unsigned long long part = ticket >> 32 ? ticket % gridDim.x : (unsigned)ticket % gridDim.x;
        const unsigned long long begin = ticket - part, last = begin + gridDim.x;  // of the round
        if (ticket & EXPIRED) ok = 0;
        else if (ticket + 1 != last) {
            // the timer is read every 32 polls (reading it before the first cost 0.1 us per barrier)
            unsigned long long t0 = 0;
            for (int k = 1; ok; k++) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(&gb->count) : "memory");
                if ((seen & ~EXPIRED) >= last) break;  // also where a later round has expired
                if (seen & EXPIRED) ok = 0;
                else if (k % 32 == 0) {
                    const unsigned long long t = gtimer();
                    if (t0 == 0) t0 = t;
                    else if (t - t0 > 2000000000ull && atomicCAS(&gb->count, seen, EXPIRED | begin) == seen) ok = 0;
                }
            }
        }
    }
    return __syncthreads_and(ok);
}

// Deterministic block reduction of NV sums into partial[k*G + blockIdx.x].
template <int NV>
__device__ __forceinline__ void block_store(double (&val)[NV], double *partial, int G) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
        for (int o = 16; o > 0; o >>= 1) val[k] += __shfl_down_sync(0xffffffffu, val[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[k][warp] = val[k];
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double x = lane < nw ? sh[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) partial[k * G + blockIdx.x] = x;
        }
    }
    __syncthreads();
}

// The same from FP32 per-thread sums: the warp stage adds in FP32, the block and grid
// stages in FP64. GB300's FP64 pipe runs at 1/64 of the FP32 rate, so converting and
// accumulating every element in FP64 would bound an FP32 Krylov body on that pipe.
template <int NV>
__device__ __forceinline__ void block_store_f(float (&val)[NV], double *partial, int G) {
    __shared__ double shf[NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
        for (int o = 16; o > 0; o >>= 1) val[k] += __shfl_down_sync(0xffffffffu, val[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) shf[k][warp] = (double)val[k];
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double x = lane < nw ? shf[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) partial[k * G + blockIdx.x] = x;
        }
    }
    __syncthreads();
}

// Scalar FP64 work (divisions, square roots of the Krylov recurrences) evaluated once per
// block by thread 0 and handed to every thread, instead of 256 copies on the 1/64-rate FP64
// pipe. Every thread of the block must make the call.
template <typename F>
__device__ __forceinline__ double block_once(F f) {
    __shared__ double v;
    if (threadIdx.x == 0) v = f();
    __syncthreads();
    const double r = v;
    __syncthreads();
    return r;
}

// Every block sums the G partials of each of the NV slots in the same fixed order.
template <int NV>
__device__ __forceinline__ void grid_sum(const double *partial, int G, double (&out)[NV]) {
    __shared__ double res[NV];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double x = 0.0;
            for (int b = lane; b < G; b += 32) x += *(volatile const double *)&partial[k * G + b];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) res[k] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) out[k] = res[k];
    __syncthreads();
}

// The sums of blocks [b0, b1) and NX scalars that f forms from them (f(sums, x), by one thread: a
// division or square root in every thread would queue on the 1/64-rate FP64 pipe), for every
// thread of the block.
template <int NV, int NX, typename F>
__device__ __forceinline__ void sum_scalars(const double *partial, int G, int b0, int b1, double (&out)[NV],
                                            double (&x)[NX], F f) {
    __shared__ double res[NV + NX];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        double s[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double v = 0.0;
            for (int b = b0 + lane; b < b1; b += 32) v += *(volatile const double *)&partial[k * G + b];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            s[k] = v;
        }
        if (lane == 0) {
            double y[NX];
            f(s, y);
#pragma unroll
            for (int k = 0; k < NV; k++) res[k] = s[k];
#pragma unroll
            for (int k = 0; k < NX; k++) res[NV + k] = y[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) out[k] = res[k];
#pragma unroll
    for (int k = 0; k < NX; k++) x[k] = res[NV + k];
    __syncthreads();
}

// Sum of the partials of blocks [b0, b1) only (one sample of a batch), same fixed order.
template <int NV>
__device__ __forceinline__ void range_sum(const double *partial, int G, int b0, int b1, double (&out)[NV]) {
    __shared__ double res[NV];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double x = 0.0;
            for (int b = b0 + lane; b < b1; b += 32) x += *(volatile const double *)&partial[k * G + b];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) res[k] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) out[k] = res[k];
    __syncthreads();
}

__device__ __forceinline__ double dmax_reduce_block(double v) {
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        v = lane < nw ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    }
    __syncthreads();
    return v;
}


template <typename T>
__device__ __forceinline__ void tangent(int i, const T *ep, const T *eq, T xp, T xq, T *W) {
    W[3 * i] = xp * ep[3 * i] + xq * eq[3 * i];
    W[3 * i + 1] = xp * ep[3 * i + 1] + xq * eq[3 * i + 1];
    W[3 * i + 2] = xp * ep[3 * i + 2] + xq * eq[3 * i + 2];
}

// (K x)_i for node i from the tangent vectors W of x: the 2x2 block row of node i in the
// factorised form (c0 S W projected on (eq_i, ep_i) plus the diagonal block). W is written
// by other blocks of the persistent kernels, so it is read through L2 (ld.cg).
template <typename T>
__device__ __forceinline__ void apply_row(int i, const int *__restrict__ Sptr, const int *__restrict__ Scol,
                                          const T *__restrict__ Sval, const T *W, const T *ep, const T *eq,
                                          const T *A, const T *Dl, T c0, T xp, T xq, T &y0, T &y1) {
    T a0 = 0, a1 = 0, a2 = 0;
    const int k1 = Sptr[i + 1];
    for (int k = Sptr[i]; k < k1; k++) {
        const int j = Scol[k];
        const T s = Sval[k];
        a0 += s * __ldcg(W + 3 * j);
        a1 += s * __ldcg(W + 3 * j + 1);
        a2 += s * __ldcg(W + 3 * j + 2);
    }
    const T q0 = eq[3 * i], q1 = eq[3 * i + 1], q2 = eq[3 * i + 2];
    const T e0 = ep[3 * i], e1 = ep[3 * i + 1], e2 = ep[3 * i + 2];
    const T ai = A[i], di = Dl[i];
    y0 = c0 * (q0 * a0 + q1 * a1 + q2 * a2) + ai * xp + di * xq;
    y1 = c0 * (e0 * a0 + e1 * a1 + e2 * a2) + di * xp - ai * xq;
}

// apply_row for a group of LPR consecutive lanes sharing row i (LPR = 1: thread per row):
// the lanes split the row's neighbour list and add their partial sums with shuffles, so a
// row's column indices and values are read by adjacent lanes. Every lane of the warp must
// call it (valid = false for lanes without a row); all lanes of the group get y0, y1.
template <typename T, int LPR>
__device__ __forceinline__ void apply_row_g(bool valid, int i, int sub, const int *__restrict__ Sptr,
                                            const int *__restrict__ Scol, const T *__restrict__ Sval, const T *W,
                                            const T *ep, const T *eq, const T *A, const T *Dl, T c0, T xp, T xq,
                                            T &y0, T &y1) {
    if constexpr (LPR == 1) {
        if (valid) apply_row<T>(i, Sptr, Scol, Sval, W, ep, eq, A, Dl, c0, xp, xq, y0, y1);
        return;
    }
    T a0 = 0, a1 = 0, a2 = 0;
    if (valid) {
        const int k1 = Sptr[i + 1];
        for (int k = Sptr[i] + sub; k < k1; k += LPR) {
            const int j = Scol[k];
            const T s = Sval[k];
            a0 += s * __ldcg(W + 3 * j);
            a1 += s * __ldcg(W + 3 * j + 1);
            a2 += s * __ldcg(W + 3 * j + 2);
        }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    if (valid) {
        const T q0 = eq[3 * i], q1 = eq[3 * i + 1], q2 = eq[3 * i + 2];
        const T e0 = ep[3 * i], e1 = ep[3 * i + 1], e2 = ep[3 * i + 2];
        const T ai = A[i], di = Dl[i];
        y0 = c0 * (q0 * a0 + q1 * a1 + q2 * a2) + ai * xp + di * xq;
        y1 = c0 * (e0 * a0 + e1 * a1 + e2 * a2) + di * xp - ai * xq;
    }
}

}  // namespace fg
