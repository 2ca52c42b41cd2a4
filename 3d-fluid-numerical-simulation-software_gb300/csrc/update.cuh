// What the kernels that set a level's conserved variables share: primitive variables
// (source/PrimitiveVars.cpp:7-28), detection of out-of-range cells and their repair
// (source/Limit_FlowVars.cpp:8-118) by the last block of a solve, so that neither takes a launch of its own.
#pragma once
#include "gbt_common.cuh"
#include "kernels.hpp"

namespace gbt {

// primitive variables from the conserved ones
template <typename T>
__device__ __forceinline__ void prim_from_cons(const Phys &P, const double c[5], T q[6])
{
    if constexpr (sizeof(T) == 4) {
        // mixed form: primitives are stored in FP32, so they are formed in FP32 from the FP64 Q
        // (conversions by integer operations: the same roundings as the conversion instructions)
        const float d = f64_to_f32_rn(c[0]), rd = 1.0f / d;
        const float u = f64_to_f32_rn(c[1]) * rd, v = f64_to_f32_rn(c[2]) * rd, w = f64_to_f32_rn(c[3]) * rd;
        const float V2 = u * u + v * v + w * w;
        const float pr = ((float)P.gamma - 1.0f) * (f64_to_f32_rn(c[4]) - d * V2 * 0.5f);
        q[PD] = d; q[PU] = u; q[PV] = v; q[PW] = w; q[PP] = pr; q[PT] = pr * rd / (float)P.rgas;
    } else {
        // one FP64 division by the density, products with its reciprocal (within rounding)
        const double d = c[0], rd = 1.0 / d, u = c[1] * rd, v = c[2] * rd, w = c[3] * rd;
        const double V2 = u * u + v * v + w * w;
        const double pr = (P.gamma - 1.0) * (c[4] - d * V2 * 0.5);
        q[PD] = (T)d; q[PU] = (T)u; q[PV] = (T)v; q[PW] = (T)w; q[PP] = (T)pr; q[PT] = (T)(pr * rd / P.rgas);
    }
}

template <typename T>
__device__ __forceinline__ bool out_of_range(const T q[6])
{
    const T dmin = (T)(double)1.0E-6f, dmax = (T)1000, pmin = (T)(double)1.0E-6f, pmax = (T)1000, vmax = (T)1000;
    return q[PD] < dmin || q[PD] > dmax || q[PP] < pmin || q[PP] > pmax || q[PU] > vmax || q[PV] > vmax || q[PW] > vmax;
}

// whether this block is the last of its group to get here (all threads call it; what the group's blocks
// wrote before is then visible: the barrier orders the block's writes before the fence of its first thread).
// The counter is put back to zero for the next launch.
__device__ __forceinline__ bool last_block(unsigned *count, unsigned blocks)
{
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(count, 1u) == blocks - 1;
        if (last) { *count = 0; __threadfence(); }
    }
    __syncthreads();
    return last;
}

// The reference repairs limited cells one after another in i, j, k order, each from the mean of
// its in-range neighbours as they are at that moment, so a repaired cell can feed a later one.
// Rare; one thread per solve replays that order over the (sorted) list of flagged cells. When
// the list overflowed, the thread scans every cell instead.
template <typename T>
__device__ __noinline__ void limit_cells(const Batch &B, const Phys &P, const Flow<T> &W, int level, int s, int *bad_list, int bad_cap, int n)
{
    const Lvl L = B.lv[s];
    const int nI = L.IM - 1, nJ = L.JM - 1, nK = L.KM - 1;
    int *lst = bad_list + (long long)s * bad_cap;
    const bool full = n > bad_cap;
    if (!full) {
        for (int a = 1; a < n; a++) {                 // insertion sort: lists are short
            int v = lst[a], b = a - 1;
            while (b >= 0 && lst[b] > v) { lst[b + 1] = lst[b]; b--; }
            lst[b + 1] = v;
        }
    }
    const long long total = (long long)nI * nJ * nK;
    const long long m = full ? total : n;
    for (long long e = 0; e < m; e++) {
        const long long lin = full ? e : lst[e];
        const int i = 1 + (int)(lin / ((long long)nJ * nK)), j = 1 + (int)((lin / nK) % nJ), k = 1 + (int)(lin % nK);
        const long long p = ix(L, i, j, k);
        T q[6];
        for (int c = 0; c < 6; c++) q[c] = W.pv[c][p];
        if (!out_of_range(q)) continue;
        double d = 0, u = 0, v = 0, w = 0, pr = 0;
        int kn = 0, i1 = 0, j1 = 0, k1 = 0;
        for (int ia = -1; ia <= 1; ia++)
            for (int ja = -1; ja <= 1; ja++)
                for (int ka = -1; ka <= 1; ka++) {
                    k1 = k + ka; j1 = j + ja; i1 = i + ia;
                    if (i1 > 0 && i1 < L.IM && j1 > 0 && j1 < L.JM && k1 > 0 && k1 < L.KM) {
                        const long long r = ix(L, i1, j1, k1);
                        T qq[6];
                        for (int c = 0; c < 6; c++) qq[c] = W.pv[c][r];
                        if (!out_of_range(qq)) {
                            d += qq[PD]; u += qq[PU]; v += qq[PV]; w += qq[PW]; pr += qq[PP]; kn++;
                        }
                    }
                }
        if (kn == 0) {
            // last visited neighbour (i+1, j+1, k+1), clipped to the admissible range
            const long long r = ix(L, i1, j1, k1);
            d = W.pv[PD][r]; u = W.pv[PU][r]; v = W.pv[PV][r]; w = W.pv[PW][r]; pr = W.pv[PP][r];
            const double lo = (double)1.0E-6f;
            if (d < lo) d = lo;
            if (d > 1000.0) d = 1000.0;
            if (pr < lo) pr = lo;
            if (pr > 1000.0) pr = 1000.0;
            if (fabs(u) > 1000.0) u = u < 0 ? -1000.0 : 1000.0;
            if (fabs(v) > 1000.0) v = v < 0 ? -1000.0 : 1000.0;
            if (fabs(w) > 1000.0) w = w < 0 ? -1000.0 : 1000.0;
        } else {
            const double sn1 = (double)(1.0f / (float)kn);
            d *= sn1; u *= sn1; v *= sn1; w *= sn1; pr *= sn1;
        }
        W.pv[PD][p] = (T)d; W.pv[PU][p] = (T)u; W.pv[PV][p] = (T)v; W.pv[PW][p] = (T)w; W.pv[PP][p] = (T)pr;
        W.pv[PT][p] = (T)(pr / d / P.rgas);
        W.cv[0][p] = d; W.cv[1][p] = d * u; W.cv[2][p] = d * v; W.cv[3][p] = d * w;
        W.cv[4][p] = pr / (P.gamma - 1.0) + d * (u * u + v * v + w * w) / 2.0;
    }
    B.st[s].flag_low_dt[level] = 10;
    atomicOr(&B.st[s].status, GBT_STATUS_LIMITER | (full ? GBT_STATUS_LIMITER_OVF : 0));
    B.st[s].limiter_hits += n;
}

// Limiter of a kernel whose blocks cover a solve's cells: every thread calls limit_flag for its cell, then every
// thread of the block limit_done, with the number of blocks that cover the solve. The last of them repairs
// the flagged cells. (The list's length and the counter are zero between launches.)
template <typename T>
__device__ __forceinline__ void limit_flag(const Phys &P, const LimitLists &q, const Lvl &L, int s, int i, int j, int k, const T v[6])
{
    if (!P.limiter || !out_of_range(v)) return;
    const int n = atomicAdd(&q.count[s], 1);
    if (n < q.cap) q.list[(long long)s * q.cap + n] = (int)(((long long)(i - 1) * (L.JM - 1) + (j - 1)) * (L.KM - 1) + (k - 1));
}
template <typename T>
__device__ __forceinline__ void limit_done(const Batch &B, const Phys &P, const Flow<T> &W, int level, const LimitLists &q, int s, unsigned blocks)
{
    if (!P.limiter || !last_block(q.done + s, blocks) || threadIdx.x != 0) return;
    const int n = q.count[s];
    if (n == 0) { atomicAnd(&B.st[s].status, ~GBT_STATUS_LIMITER); return; }
    q.count[s] = 0;
    limit_cells<T>(B, P, W, level, s, q.list, q.cap, n);
}
// blocks of 256 threads that cover the cells of a solve
__device__ __forceinline__ unsigned cell_blocks(const Lvl &L) { return ((unsigned)((L.IM - 1) * (L.JM - 1) * (L.KM - 1)) + 255u) / 256u; }

}  // namespace gbt
