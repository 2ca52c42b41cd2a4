// Primitive variables (source/PrimitiveVars.cpp:7-28) and the limiter (source/Limit_FlowVars.cpp:8-118) by
// themselves, the residual norm (source/ComputeAllBlockVars.cpp:318-372), the inlet and outlet integrals
// (source/Ouput.cpp:9-107,282-300) and the CFL ramp.
#include "gbt_common.cuh"
#include "kernels.hpp"
#include "flux.cuh"
#include "update.cuh"

namespace gbt {

// primitive variables of a level (PRIM), out-of-range cells repaired (LIM)
template <typename T, bool PRIM, bool LIM>
__global__ void __launch_bounds__(256) k_primitive(Batch B, Phys P, Flow<T> W, int level, LimitLists q)
{
    const int s = blockIdx.y;
    const Lvl L = B.lv[s];
    const unsigned blocks = cell_blocks(L);
    if (blockIdx.x >= blocks) return;
    int i, j, k;
    if (box_index(L.IM - 1, L.JM - 1, L.KM - 1, i, j, k)) {
        const long long p = ix(L, i, j, k);
        T v[6];
        if constexpr (PRIM) {
            double c[5];
#pragma unroll
            for (int n = 0; n < 5; n++) c[n] = W.cv[n][p];
            prim_from_cons<T>(P, c, v);
#pragma unroll
            for (int n = 0; n < 6; n++) W.pv[n][p] = v[n];
        } else {
#pragma unroll
            for (int n = 0; n < 6; n++) v[n] = W.pv[n][p];
        }
        if constexpr (LIM) limit_flag<T>(P, q, L, s, i, j, k, v);
    }
    if constexpr (LIM) limit_done<T>(B, P, W, level, q, s, blocks);
}

template <typename T>
void launch_primitive(const LaunchCtx &ctx, const Phys &P, Flow<T> W)
{
    k_primitive<T, true, false><<<ctx.grid_cells(256), 256, 0, ctx.stream>>>(ctx.batch, P, W, 0, {});
}

template <typename T>
void launch_limiter(const LaunchCtx &ctx, const Phys &P, Flow<T> W, int level, const LimitLists &q)
{
    if (P.limiter) k_primitive<T, false, true><<<ctx.grid_cells(256), 256, 0, ctx.stream>>>(ctx.batch, P, W, level, q);
}

// ---- residual norm: sum |(Q_old - Q)/Q_old| * Vol / V_total, FP64, in a fixed order: each thread four or
// more cells, the threads of a block, the blocks of a case (its last block to arrive sums them for every
// slot). Bound by its FP64 instructions: 45 per cell in the FP64 form (25 us for the 129x49x49 passage),
// 5 in the mixed form, whose reductions counted more. With 304 blocks for every slot, each reduced by 25
// shuffled additions per warp, and the blocks' sums added up by five threads of a second kernel it took 62
// and 46 us, and 195 us for 32 solves of 25x25x65 nodes; now 33, 20 and 48.
constexpr int kNormThreads = 256, kNormCells = 4 * kNormThreads;
__device__ __forceinline__ int norm_blocks(const Lvl &L, int most)
{
    const int n = ((L.IM - 1) * (L.JM - 1) * (L.KM - 1) + kNormCells - 1) / kNormCells;
    return n < most ? n : most;
}

// the iteration's row of the history, by the case's first slot
__device__ __forceinline__ void history_row(const SolveState *state, const SolveConst &sc, const HistorySink &hist)
{
    const volatile SolveState &st = state[sc.lead];
    const int row = st.iter - *hist.base;
    if (row < 0 || row >= hist.rows) return;
    double *r = hist.out + ((long long)row * hist.ncase + sc.cix) * 12;
    r[0] = st.iter;
    for (int c = 0; c < 5; c++) r[1 + c] = st.res[c];
    r[6] = st.m_in; r[7] = st.m_out; r[8] = st.pr; r[9] = st.eff; r[10] = st.m_ratio;
    r[11] = st.cfl;
}
// one of the six values' groups a row waits for (five components of the norm, the integrals) is in the state
__device__ __forceinline__ void history_arrive(const SolveState *state, const SolveConst &sc, const HistorySink &hist)
{
    __threadfence();
    if (atomicAdd(hist.both + sc.lead, 1u) != 5u) return;
    hist.both[sc.lead] = 0;
    __threadfence();
    history_row(state, sc, hist);
}

template <typename T>
__global__ void __launch_bounds__(kNormThreads) k_norm(Batch B, Geo G, Flow<T> W, double *partials, int nblk, const double *totalvol,
                                                       unsigned *count, HistorySink hist)
{
    const int s = blockIdx.y;
    const Lvl L = B.lv[s];
    const int nb = norm_blocks(L, nblk);
    if ((int)blockIdx.x >= nb) return;
    const int nI = L.IM - 1, nJ = L.JM - 1, nK = L.KM - 1;
    const unsigned n = (unsigned)nI * (unsigned)nJ * (unsigned)nK;
    double acc[5] = {0, 0, 0, 0, 0};
    for (unsigned t = blockIdx.x * kNormThreads + threadIdx.x; t < n; t += (unsigned)nb * kNormThreads) {
        const unsigned q = t / (unsigned)nK, r = q / (unsigned)nJ;
        const int k = (int)(t - q * (unsigned)nK) + 1, j = (int)(q - r * (unsigned)nJ) + 1, i = (int)r + 1;
        const long long p = ix(L, i, j, k);
        const double vol = G.vol[p];
        double o[5], c[5];
#pragma unroll
        for (int m = 0; m < 5; m++) { o[m] = W.cvold[m][p]; c[m] = W.cv[m][p]; }
#pragma unroll
        for (int m = 0; m < 5; m++) acc[m] += rel_change_t<T>(o[m], c[m]) * vol;
    }
    __shared__ double sh[5][kNormThreads];
#pragma unroll
    for (int m = 0; m < 5; m++) sh[m][threadIdx.x] = acc[m];
    __syncthreads();
    const int m = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto warp_sum = [](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        return v;
    };
    if (m < 5) {                                  // one warp per component
        double v = 0;
        for (int e = lane; e < kNormThreads; e += 32) v += sh[m][e];
        v = warp_sum(v);
        if (lane == 0) partials[((long long)s * nblk + blockIdx.x) * 5 + m] = v;
    }
    const SolveConst &sc = B.sc[s];
    unsigned blocks = 0;
    for (int q = sc.lead; q < sc.lead + sc.nblk; q++) blocks += (unsigned)norm_blocks(B.lv[q], nblk);
    if (!last_block(count + sc.lead, blocks) || m >= 5) return;
    // the norm of the case: the sums of its slots over the case's volume (every slot keeps it)
    double v = 0;
    for (int q = sc.lead; q < sc.lead + sc.nblk; q++) {
        const int nq = norm_blocks(B.lv[q], nblk);
        for (int e = lane; e < nq; e += 32) v += __ldcg(&partials[((long long)q * nblk + e) * 5 + m]);
    }
    v = warp_sum(v);
    if (lane != 0) return;
    for (int q = sc.lead; q < sc.lead + sc.nblk; q++) {
        const double w = v / totalvol[q];
        B.st[q].res[m] = w;
        if (m == 0 && !isfinite(w)) atomicOr(&B.st[q].status, GBT_STATUS_NAN);
    }
    if (hist.both) history_arrive(B.st, sc, hist);
}

template <typename T>
void launch_res_norm(const LaunchCtx &ctx, const Geo &G, Flow<T> W, const double *totalvol, double *partials, int nblk, unsigned *count,
                     const HistorySink &hist)
{
    const Batch &B = ctx.batch;
    ctx.mark("res_norm", 1, 1);
    // (the product of a batch's largest extents, which need not be one slot's, may take more than 32 bits)
    const long long most = ((long long)(ctx.maxIM - 1) * (ctx.maxJM - 1) * (ctx.maxKM - 1) + kNormCells - 1) / kNormCells;
    k_norm<T><<<dim3((unsigned)(most < nblk ? most : nblk), B.nsolve), kNormThreads, 0, ctx.stream>>>(B, G, W, partials, nblk, totalvol, count, hist);
    ctx.mark("res_norm", 0, 1);
}

// ---- inlet/outlet integrals (source/Ouput.cpp:9-107,282-300)
// Partial sums over one section (inlet or outlet k face): mass flow, sum Pt^((g-1)/g) * m and sum Tt * m;
// grid (kIntegralBlocks, solves, 2 sections). With Pt = p fac^(g/(g-1)) the power is p^((g-1)/g) fac, one
// FP64 power per point instead of two, and Ma^2 needs no roots. The last block of a solve adds its
// blocks' sums up in their order and forms the reported values, a lane per section where they are powers.
// Bound by the latency of the FP64 chains: 48 us per evaluation of the 129x49x49 passage as two kernels
// with two powers per point, sums and powers of a solve on one thread; 27 with a third power in a row at the end,
// 25 now.
template <typename T>
__global__ void __launch_bounds__(128) k_integrals(Batch B, Phys P, Geo G, Flow<T> W, const DevInOut *inl, const DevInOut *outl,
                                                   double *part, unsigned *count, HistorySink hist)
{
    const int s = blockIdx.y, sec = blockIdx.z;
    // the section's block: the case's Inlet[1] / Outlet[1] may lie in any of its blocks
    const DevInOut &sp = sec == 0 ? inl[s] : outl[s];
    const Lvl L = B.lv[sp.solve];
    const int K = sp.ks;
    const int nI = L.IM - 1, nJ = L.JM - 1;
    const double g = P.gamma, g1 = g - 1.0, R = P.rgas;
    double m = 0, pm = 0, tm = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nI * nJ; t += kIntegralBlocks * blockDim.x) {
        const int i = 1 + t / nJ, j = 1 + t % nJ;
        const long long p = ix(L, i, j, K), q = ix(L, i, j, K - 1);
        const double d = 0.5 * ((double)W.pv[PD][p] + (double)W.pv[PD][q]);
        const double u = 0.5 * ((double)W.pv[PU][p] + (double)W.pv[PU][q]);
        const double v = 0.5 * ((double)W.pv[PV][p] + (double)W.pv[PV][q]);
        const double w = 0.5 * ((double)W.pv[PW][p] + (double)W.pv[PW][q]);
        const double mc = d * (u * G.S[2][0][p] + v * G.S[2][1][p] + w * G.S[2][2][p]);
        const double tf = 0.5 * ((double)W.pv[PT][p] + (double)W.pv[PT][q]);
        // (no speed of sound, and no total state, at a negative temperature)
        const double c2 = g * R * tf, Ma2 = c2 < 0.0 ? nan("") : (u * u + v * v + w * w) / fabs(c2);
        const double fac = 1.0 + g1 / 2.0 * Ma2;
        m += mc;
        pm += pow((double)W.pv[PP][p], g1 / g) * fac * mc;
        tm += (double)W.pv[PT][p] * fac * mc;
    }
    __shared__ double sh[3][4];
    double v3[3] = {m, pm, tm};
    for (int c = 0; c < 3; c++) {
        double v = v3[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sh[c][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += sh[threadIdx.x][w];
        part[(((long long)s * 2 + sec) * kIntegralBlocks + blockIdx.x) * 3 + threadIdx.x] = v;
    }
    if (!last_block(count + s, 2 * kIntegralBlocks) || threadIdx.x >= 32) return;
    // lanes 0..2: the inlet's sums, 3..5: the outlet's
    const int lane = threadIdx.x;
    double sum = 0;
    if (lane < 6) {
        double v[kIntegralBlocks];
#pragma unroll
        for (int b = 0; b < kIntegralBlocks; b++) v[b] = __ldcg(&part[(((long long)s * 2 + lane / 3) * kIntegralBlocks + b) * 3 + lane % 3]);
#pragma unroll
        for (int b = 0; b < kIntegralBlocks; b++) sum += v[b];
    }
    double a[3], b[3];
    for (int c = 0; c < 3; c++) {
        a[c] = __shfl_sync(0xffffffffu, sum, c);
        b[c] = __shfl_sync(0xffffffffu, sum, 3 + c);
    }
    // blade count of the inlet's and of the outlet's block (source/Ouput.cpp:288,294)
    const double mi = a[0] * P.dens_ref * P.vel_ref * B.sc[inl[s].solve].nblade;
    const double mo = b[0] * P.dens_ref * P.vel_ref * B.sc[outl[s].solve].nblade;
    const double fa = a[1] / a[0], fb = b[1] / b[0];
    const double pt = pow(lane == 0 ? fa : fb, g / g1) * P.dens_ref * P.vel_ref * P.vel_ref;
    const double pti = __shfl_sync(0xffffffffu, pt, 0), pto = __shfl_sync(0xffffffffu, pt, 1);
    const double tti = a[2] / a[0] * P.temp_ref, tto = b[2] / b[0] * P.temp_ref;
    const double PR = pto / pti;
    // (PR^((g-1)/g) is the quotient of the two bases, or PR where that is infinite or not a number)
    const double Ladk = g / g1 * R * tti * ((isfinite(PR) ? fb / fa : PR) - 1.0);
    const double Lk = g / g1 * R * tti * (tto / tti - 1.0);
    if (lane != 0) return;
    SolveState &st = B.st[s];
    st.m_in = mi; st.m_out = mo; st.pr = PR; st.eff = Ladk / Lk;
    st.m_ratio = fabs((mi - mo) / mi);
    if (!isfinite(mi) || !isfinite(mo)) atomicOr(&st.status, GBT_STATUS_NAN);
    const SolveConst &sc = B.sc[s];
    if (sc.lead != s) return;
    if (hist.both) history_arrive(B.st, sc, hist);
    else history_row(B.st, sc, hist);
}

template <typename T>
void launch_integrals(const LaunchCtx &ctx, const Phys &P, const Geo &G, Flow<T> W, const BcTables &bc, const HistorySink &hist)
{
    // first inlet and first outlet patch of every solve (the reference reports Inlet[1], Outlet[1])
    const Batch &B = ctx.batch;
    k_integrals<T><<<dim3(kIntegralBlocks, B.nsolve, 2), 128, 0, ctx.stream>>>(B, P, G, W, bc.inlet_first, bc.outlet_first,
                                                                               bc.integ_part, bc.integ_count, hist);
}

// CFL ramp of the driver (source/Solver.cpp:49-60): x1.2 whenever the density residual falls
// below a threshold that then drops tenfold; capped at 10
__global__ void k_cfl_ramp(Batch B, int iter)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= B.nsolve || iter <= 1) return;
    SolveState &st = B.st[s];
    if (st.res[0] <= st.cfl_res) {
        st.cfl = st.cfl * (double)1.2f;
        st.cfl_res = st.cfl_res / 10.0;
    }
    if (st.cfl > 10.0) st.cfl = 10.0;
}
void launch_cfl_ramp(const LaunchCtx &ctx, int iter)
{
    k_cfl_ramp<<<(ctx.batch.nsolve + 127) / 128, 128, 0, ctx.stream>>>(ctx.batch, iter);
}

#define GBT_INST(T)                                                                                                   \
    template void launch_primitive<T>(const LaunchCtx &, const Phys &, Flow<T>);                                       \
    template void launch_limiter<T>(const LaunchCtx &, const Phys &, Flow<T>, int, const LimitLists &);                 \
    template void launch_res_norm<T>(const LaunchCtx &, const Geo &, Flow<T>, const double *, double *, int, unsigned *, const HistorySink &);          \
    template void launch_integrals<T>(const LaunchCtx &, const Phys &, const Geo &, Flow<T>, const BcTables &, const HistorySink &);
GBT_INST(double)
GBT_INST(float)

}  // namespace gbt
