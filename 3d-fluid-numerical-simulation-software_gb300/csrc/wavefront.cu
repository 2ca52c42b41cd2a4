// LU-SGS sweeps (source/LU_SGS_Marching.cpp:10-291) as one launch per direction over every solve of the
// batch. The forward sweep's cell (i, j, k) needs the terms of (i-1, j, k), (i, j-1, k), (i, j, k-1); the
// backward sweep is its mirror image.
//
// What bounds it is the chain of i + j + k planes, not the arithmetic or the bytes. A block owns a tile of 4 x 8 grid
// columns (i, j; 2 x 8 in FP64) and marches it along k skewed: at step t the column (a, b) of the tile is at
// k = t - a - b, so that the terms it needs from inside the tile are the ones its neighbours formed one step
// earlier, and a step costs the block one barrier. Tiles run side by side on as many SMs as there are,
// each a few steps behind the two it reads from. The 224 planes of the 129x49x49 passage take 314 us in FP64, where a
// step of 1.4 us hides the way of a term from tile to tile. In FP32 a step takes 0.3 us, and of the 120 us of a
// sweep the planes are 67: the rest is some 3 us for each of 17 crossings (term to the outgoing warp, to L2, to
// the incoming warp that polls for it, to the tile). With a launch per plane a plane took 1.8 us in FP32, 3.4 in FP64.
//
// What a step costs is the number of instructions one warp issues (a lone warp of a sub-partition issues
// one every three to four cycles, and an FP64 instruction holds its sub-partition for some 70): with a
// lane per cell a step took 337 instructions and 1.3k cycles in FP32. So four lanes share a cell (eight in
// FP64, 22 FP64 instructions a step where four lanes took 38; 26 with three terms to a lane, 0.193 and 0.177 ms
// a sweep of the 65x33x33 duct), four warps a step, and everything that is not the cell's arithmetic is
// done by two further warps of the block:
//   a cell's lanes     receive a component each (FP32: and the fifth); lanes 0..2 form V_n of a direction each, and
//                      lane 3 the pressure with the same instructions; the fifteen terms are formed by
//                      direction on lanes 0..2 (FP64: two to a lane of eight, or one to a lane of sixteen
//                      in narrow tiles, where there is an SM for each of them)
//   the incoming warp  reads the terms that cross into the tile and puts them beside the tile's own
//   the outgoing warp  sends the terms that leave it and fetches the inputs of later steps
//
// Between tiles a term travels as 16-byte packets in global memory, written and read by single 128-bit
// relaxed accesses: values and a tag that names the sweep, so a reader that sees the tag has the values,
// and neither side needs a fence. The reader asks kAhead steps before a packet is needed and asks again
// while the tag is old. Every slot is written once per sweep and the next sweep has another tag. Tiles are
// handed out by a counter in an order in which a tile follows the two it reads from, so the ones that are
// waited for are always running. Every wait is bounded: a warp whose wait runs out reports it in the
// solve's status and goes on without waiting.
//
// Every input of a step lies in one block of memory ([step][values][cells]) and comes through a ring in
// shared memory by bulk copies. k_wave_gather writes the blocks with everything a cell can form without
// its neighbours: the right-hand side, its terms' coefficients and, in FP64, its old fluxes (in FP32 they
// are formed in the sweep: the bytes cost more there). k_wave_update turns dQ back into box order and
// applies it.
//
// A cell sends one term per direction d (the reference's A and V terms of a neighbour, :95-150, 293-419),
//   w_d = h_d (F_d(Q + dQ) - F_d(Q)) +- c_d dQ      (+ forward, - backward)
//   h_d = (|S_d| / 2) / alpha, c_d = (relax lambda_c,d / 2 + lambda_v,d) / alpha, alpha the receiver's diagonal,
// and a cell receives
//   forward:  dQ = -R / alpha + (w_I + w_J + w_K)
//   backward: dQ = dQ* - (w_I + w_J + w_K).
// The Spalart-Allmaras variable's sweep (:76-258) has the same shape and follows the mean flow's of the
// same direction. Products, sums and fused operations are written out and keep the order that the
// plane-by-plane sweeps had, so that a solve's trajectory keeps its bits: runs that cross the switches of
// the turbulence model and the limiter amplify the last one.
#include "gbt_common.cuh"
#include "kernels.hpp"
#include "flux.cuh"
#include "update.cuh"
#include "ring_feed.hpp"
#include <type_traits>

namespace gbt {

namespace {

// columns of a tile in i and j, lanes of a cell: 128 lanes a step in both precisions. N = 1 is the form for grids of
// which every tile has an SM: in FP64 narrow tiles of 2 x 4 columns with sixteen lanes a cell, one term to
// a lane (18 FP64 instructions a step instead of 22); in FP32 a step's inputs are read, and the old
// fluxes formed, during the step before, where they fill the gaps of its chain (cycle of the 129x49x49
// passage 0.672 and 0.660 ms; 12 solves on three meshes, whose SMs have several tiles to fill them with,
// 3.844 and 3.867).
template <typename T> constexpr int kPA = sizeof(T) == 4 ? 4 : 2;
template <typename T, int N> constexpr int kPB = N && sizeof(T) == 8 ? 4 : 8;
template <typename T, int N> constexpr int kCells = kPA<T> * kPB<T, N>;
template <typename T, int N> constexpr int kLanes = 128 / kCells<T, N>;
constexpr int kGroup = 2, kStages = 3;          // steps of a stage of the input ring, stages
constexpr int kSlots = kGroup * kStages;        // steps whose terms are kept: the outgoing warp fetches a stage
                                                // after it has sent the steps that used it, so a step's terms
                                                // are never overwritten before they are sent
constexpr int kAhead = 2;                       // steps that the incoming warp asks ahead: with one, the answer takes
                                                // longer than a step; asked earlier, it is more often too early and
                                                // costs a second round (137, 146, 154, 186 us a forward sweep of the
                                                // 129x49x49 passage in FP32 with 2, 3, 4, 8)
constexpr unsigned kWaitLimit = 1u << 21;       // polls of a wait before it gives up: 8 s on a barrier (a poll of one that
                                                // does not complete takes 4 us), some 2 s on a packet
constexpr int kSteps32 = 16;                    // steps of a block of the FP32 gather kernel
template <typename T, int N> constexpr int kSteps = 256 / kCells<T, N>;                   // of the kernels with a thread per cell

// bytes of a step's blocks, packets of an edge cell and of a step
//   FP32: geo {n_d, V_entrainment,d} at 3 cell + d; flow {h_d, c_d} at 3 cell + d of the forward sweep, {rho, m},
//         {rho E, p, 1/rho, 0} per cell, {h_d, c_d} of the backward sweep (a sweep copies its own end and the
//         middle); packets {w_1, w_2, w_3, tag}, {w_4, w_5, 0, tag}
//   FP64: geo {n_1, n_2}, {n_3, V_entrainment} at 3 cell + d; flow {h_d, c_d} of the forward sweep, f_1, .., f_5
//         at 3 cell + d, Q_1..Q_4, Q_5 per cell, {h_d, c_d} of the backward sweep; packets {w_c, tag}
//   dq:   component q at 4 cell + q, the fifth per cell: the right-hand side, then dQ
//   the variable's sweep: flow V_d, ev V_old,d, |S_d|, relax lambda_c,d, lambda_v,d at 3 cell + d, ev, alpha per cell;
//         dq one value per cell; packets {A term, V term, 0, tag} in FP32, one {value, tag} each in FP64
enum Kind { MEAN, VAR };
template <typename T, Kind K, int N = 0> struct Lay {
    static constexpr int PA = kPA<T>, PB = kPB<T, N>, NC = kCells<T, N>;
    static constexpr int B = sizeof(T), CA = K == VAR ? 2 : 4, CB = K == VAR ? 0 : 1, NV = CA + CB;   // values of a term
    static constexpr int geo = K == VAR ? 0 : 12 * NC * B;
    static constexpr int ends = K == MEAN ? 6 * NC * B : 0;                  // of the flow block, one sweep's own
    static constexpr int flow = K == VAR ? 17 * NC * B : 2 * ends + (B == 4 ? 8 : 20) * NC * B;
    static constexpr int dq = (K == VAR ? 1 : NV) * NC * B;
    static constexpr int pp = B == 4 ? (K == VAR ? 1 : 2) : NV, pkt = pp * (PA + PB);
    // shared memory: the ring of inputs, the terms of the last steps (halo cells included), barriers
    static constexpr int flow_in = flow - ends, step = geo + flow_in + dq, ring = kSlots * step;
    static constexpr int IA = 0, IB = IA + CA * (PA + 1) * PB * B, JA = IB + CB * (PA + 1) * PB * B, JB = JA + CA * PA * (PB + 1) * B,
                         KA = JB + CB * PA * (PB + 1) * B, KB = KA + CA * NC * B, slot = KB + CB * NC * B;
    static constexpr int bars = ring + kSlots * slot, smem = bars + 8 * (kStages + 2 * kSlots);
    static_assert(slot % 16 == 0 && JA % 16 == 0 && KA % 16 == 0 && geo % 16 == 0 && flow_in % 16 == 0 && ends % 16 == 0 && dq % 16 == 0,
                  "alignment");
};

__device__ __forceinline__ void packet_store(uint4 *p, unsigned long long lo, unsigned long long hi)
{
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo), "l"(hi)
                 : "memory");
}
__device__ __forceinline__ void packet_load(const uint4 *p, unsigned long long &lo, unsigned long long &hi)
{
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}" : "=l"(lo), "=l"(hi) : "l"(p)
                 : "memory");
}
__device__ __forceinline__ unsigned long long pack2(float a, float b)
{
    return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo_f(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_f(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

__device__ __forceinline__ void bar_init(unsigned bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// false once a wait has run out; nothing is waited for after that
__device__ __forceinline__ void bar_wait(unsigned bar, unsigned parity, bool &ok)
{
    if (!ok || bar_try(bar, parity)) return;
    for (unsigned n = 0; n < kWaitLimit; n++)
        if (bar_try(bar, parity)) return;
    ok = false;
}
// the same for a whole warp whose lanes vote later on: a wait that runs out on one of them has run out on all. (Votes of
// all lanes in every poll instead, met or not, cost the 129x49x49 passage 1.5% in FP64; this costs nothing.)
__device__ __forceinline__ void bar_wait_warp(unsigned bar, unsigned parity, bool &ok)
{
    bar_wait(bar, parity, ok);
    ok = __all_sync(0xffffffffu, ok) != 0;
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const char *src, unsigned bytes, unsigned bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar) : "memory");
}

// where a tile is and whom it exchanges with
struct Where {
    WaveSolve S;
    int slot, PI, PJ;
    long long step0;                            // its first step
    bool has_i, has_j, next_i, next_j;          // tiles it reads from and sends to
    long long from_i, from_j;                   // first step of the ones it reads from
};
template <int DIR>
__device__ __forceinline__ Where tile_of(const WaveTables &V, unsigned ticket)
{
    Where w;
    const int2 it = V.item[DIR > 0 ? ticket : V.n_item - 1 - ticket];
    w.slot = it.x;
    w.S = V.solve[it.x];
    w.PI = it.y / w.S.nPJ;
    w.PJ = it.y - w.PI * w.S.nPJ;
    w.step0 = w.S.step0 + (long long)(w.PI * w.S.nPJ + w.PJ) * w.S.T;
    w.has_i = DIR > 0 ? w.PI > 0 : w.PI < w.S.nPI - 1;
    w.next_i = DIR > 0 ? w.PI < w.S.nPI - 1 : w.PI > 0;
    w.has_j = DIR > 0 ? w.PJ > 0 : w.PJ < w.S.nPJ - 1;
    w.next_j = DIR > 0 ? w.PJ < w.S.nPJ - 1 : w.PJ > 0;
    w.from_i = w.step0 - (long long)DIR * w.S.nPJ * w.S.T;
    w.from_j = w.step0 - (long long)DIR * w.S.T;
    return w;
}

// byte offsets in a slot of the first and the second group of a term's components: halo cells sit before the
// first column (row) in the forward sweep and after the last one in the backward sweep
template <class L> __device__ __forceinline__ int off_ia(int row, int b) { return L::IA + L::CA * (row * L::PB + b) * L::B; }
template <class L> __device__ __forceinline__ int off_ib(int row, int b) { return L::IB + L::CB * (row * L::PB + b) * L::B; }
template <class L> __device__ __forceinline__ int off_ja(int a, int col) { return L::JA + L::CA * (a * (L::PB + 1) + col) * L::B; }
template <class L> __device__ __forceinline__ int off_jb(int a, int col) { return L::JB + L::CB * (a * (L::PB + 1) + col) * L::B; }

// a step's cell on its quad of lanes: what it receives -> dQ -> what it sends. in: the step's inputs;
// rd: the slot of the last step, wr: this step's
template <typename T, int DIR, Kind K, int N> struct CellStep;

template <int DIR, int FORM> struct CellStep<float, DIR, MEAN, FORM> {
    using L = Lay<float, MEAN, FORM>;
    static __device__ __forceinline__ float dot(float a0, float a1, float a2, float b0, float b1, float b2)
    {
        return __fmaf_rn(a2, b2, __fmaf_rn(a0, b0, __fmul_rn(a1, b1)));
    }
    static constexpr int NC = L::NC;
    struct Pre { float4 N, o, x; float2 hc; float rq, r4, f0, f1, f2, f3, f4; };
    static __device__ __forceinline__ Pre pre(const char *in, int cell, int q)
    {
        const int e = 3 * cell + (q < 3 ? q : 0);
        const float4 N = ((const float4 *)in)[e];
        const char *own = in + L::geo + (DIR > 0 ? 0 : L::flow_in - L::ends), *mid = in + L::geo + (DIR > 0 ? L::ends : 0);
        const float2 hc = ((const float2 *)own)[e];
        const float4 o = ((const float4 *)mid)[cell], x = ((const float4 *)mid)[NC + cell];       // x: rho E, p, 1/rho
        const float *fq = (const float *)(in + L::geo + L::flow_in);
        const float rq = fq[4 * cell + q], r4 = fq[4 * NC + cell];
        // the old flux of this lane's direction
        const float vo = dot(__fmul_rn(o.y, x.z), __fmul_rn(o.z, x.z), __fmul_rn(o.w, x.z), N.x, N.y, N.z), dv = __fadd_rn(vo, -N.w);
        const float f0 = __fmul_rn(o.x, dv), f1 = __fmaf_rn(o.y, dv, __fmul_rn(x.y, N.x)), f2 = __fmaf_rn(o.z, dv, __fmul_rn(x.y, N.y)),
                    f3 = __fmaf_rn(o.w, dv, __fmul_rn(x.y, N.z)), f4 = __fmaf_rn(x.y, N.w, __fmul_rn(__fadd_rn(x.x, x.y), dv));
        return {N, o, x, hc, rq, r4, f0, f1, f2, f3, f4};
    }
    static __device__ __forceinline__ void run(const Pre &p, const char *rd, char *wr, int cell, int q, const int r_off[4], int w_off,
                                               int w_off4, bool active, float gm1, char *dq_out)
    {
        const float4 N = p.N, o = p.o, x = p.x;
        const float2 hc = p.hc;
        const float rq = p.rq, r4 = p.r4, f0 = p.f0, f1 = p.f1, f2 = p.f2, f3 = p.f3, f4 = p.f4;
        // received
        const float sq = __fadd_rn(__fadd_rn(((const float *)(rd + r_off[0]))[q], ((const float *)(rd + r_off[2]))[q]),
                                   ((const float *)(rd + L::KA))[4 * cell + q]);
        const float s4 = __fadd_rn(__fadd_rn(((const float *)(rd + r_off[1]))[0], ((const float *)(rd + r_off[3]))[0]),
                                   ((const float *)(rd + L::KB))[L::CB * cell]);
        float dqq = DIR > 0 ? __fadd_rn(rq, sq) : __fadd_rn(rq, -sq), dq4 = DIR > 0 ? __fadd_rn(r4, s4) : __fadd_rn(r4, -s4);
        if (!active) dqq = dq4 = 0.0f;
        const unsigned quad = (threadIdx.x & 31) & ~3u;
        const float d0 = __shfl_sync(0xffffffffu, dqq, quad), d1 = __shfl_sync(0xffffffffu, dqq, quad + 1),
                    d2 = __shfl_sync(0xffffffffu, dqq, quad + 2), d3 = __shfl_sync(0xffffffffu, dqq, quad + 3);
        const float nd = __fadd_rn(o.x, d0), nx = __fadd_rn(o.y, d1), ny = __fadd_rn(o.z, d2), nz = __fadd_rn(o.w, d3),
                    ne = __fadd_rn(x.x, dq4);
        // lanes 0..2: V_n - ve; lane 3: p = (gamma - 1)(rho E - |m|^2 / (2 rho))
        const float inv = frcp<float>(nd);
        const float mm = dot(nx, ny, nz, q < 3 ? N.x : nx, q < 3 ? N.y : ny, q < 3 ? N.z : nz);
        const float dn = q < 3 ? __fmaf_rn(mm, inv, -N.w) : __fmul_rn(gm1, __fmaf_rn(-0.5f, __fmul_rn(mm, inv), ne));
        const float pn = __shfl_sync(0xffffffffu, dn, quad + 3);
        auto term = [&](float dF, float d) { return __fmaf_rn(hc.x, dF, DIR > 0 ? __fmul_rn(hc.y, d) : -__fmul_rn(hc.y, d)); };
        const float4 s = make_float4(term(__fmaf_rn(nd, dn, -f0), d0), term(__fmaf_rn(nx, dn, __fmaf_rn(pn, N.x, -f1)), d1),
                                     term(__fmaf_rn(ny, dn, __fmaf_rn(pn, N.y, -f2)), d2),
                                     term(__fmaf_rn(nz, dn, __fmaf_rn(pn, N.z, -f3)), d3));
        const float t4 = term(__fmaf_rn(__fadd_rn(ne, pn), dn, __fmaf_rn(pn, N.w, -f4)), dq4);
        if (q < 3) {
            *(float4 *)(wr + w_off) = s;
            *(float *)(wr + w_off4) = t4;
        }
        float *out = (float *)dq_out;
        out[4 * cell + q] = dqq;
        if (q == 0) out[4 * NC + cell] = dq4;
    }
};

template <int DIR, int N> struct CellStep<double, DIR, MEAN, N> {
    using L = Lay<double, MEAN, N>;
    static constexpr int lanes = kLanes<double, N>;
    static constexpr int NC = L::NC;
    struct Pre { double2 g0, g1, ha, hb; double fa, fb, o, r, ka, kb; };
    static __device__ __forceinline__ Pre pre(const char *in, int cell, int q)
    {
        const int d = q & 3, c = q < 4 ? q : 4, e = 3 * cell + (d < 3 ? d : 0);     // direction, component received
        const bool low = q < 4;
        const int t0 = min(q, 14), d0 = t0 / 5, c0 = t0 % 5, t1 = min(q + 8, 14), d1 = t1 / 5, c1 = t1 % 5;   // the terms
        const double2 *g = (const double2 *)in + e;
        const char *own = in + L::geo + (DIR > 0 ? 0 : L::flow_in - L::ends), *mid = in + L::geo + (DIR > 0 ? L::ends : 0);
        const double *oc = (const double *)mid + 15 * NC + (low ? 4 * cell + c : 4 * NC + cell),
                     *rc = (const double *)(in + L::geo + L::flow_in) + (low ? 4 * cell + c : 4 * NC + cell);
        const double2 g0 = g[0], g1 = g[3 * NC], ha = ((const double2 *)own)[3 * cell + d0];
        auto coef = [&](int dir, int cc) { return ((const double *)in)[(cc > 2 ? 6 * NC : 0) + 2 * (3 * cell + dir) + ((cc - 1) & 1)]; };
        const double fa = ((const double *)mid)[3 * (NC * c0 + cell) + d0], o = *oc, r = *rc, ka = coef(d0, c0);
        double2 hb = make_double2(0.0, 0.0);
        double fb = 0.0, kb = 0.0;
        if (lanes == 8) { hb = ((const double2 *)own)[3 * cell + d1]; fb = ((const double *)mid)[3 * (NC * c1 + cell) + d1]; kb = coef(d1, c1); }
        return {g0, g1, ha, hb, fa, fb, o, r, ka, kb};
    }
    static __device__ __forceinline__ void run(const Pre &p, const char *rd, char *wr, int cell, int q, const int r_off[4], int w_off,
                                               int w_off4, bool active, double gm1, char *dq_out)
    {
        const int d = q & 3, c = q < 4 ? q : 4, t0 = min(q, 14), d0 = t0 / 5, c0 = t0 % 5, t1 = min(q + 8, 14), d1 = t1 / 5, c1 = t1 % 5;
        const bool low = q < 4;
        const double2 g0 = p.g0, g1 = p.g1, ha = p.ha, hb = p.hb;
        const double fa = p.fa, fb = p.fb, o = p.o, r = p.r, ka = p.ka, kb = p.kb;
        // received
        const double s = __dadd_rn(__dadd_rn(*(const double *)(rd + r_off[0]), *(const double *)(rd + r_off[1])), *(const double *)(rd + r_off[2]));
        const double x = __dadd_rn(r, DIR > 0 ? s : -s), dq = active ? x : 0.0, nq = __dadd_rn(o, dq);
        const unsigned first = (threadIdx.x & 31) & ~(unsigned)(lanes - 1);
        auto from = [&](double v, int lane) { return __shfl_sync(0xffffffffu, v, first + lane); };
        const double n0 = from(nq, 0), n1 = from(nq, 1), n2 = from(nq, 2), n3 = from(nq, 3), n4 = from(nq, 4);
        const double va = from(dq, c0), na = from(nq, c0);
        const double inv = rcp_nr(n0);
        // lanes 0..2 of a half: V_n - ve; lane 3: p = (gamma - 1)(rho E - |m|^2 / (2 rho))
        const double mm = fma(n3, d < 3 ? g1.x : n3, fma(n1, d < 3 ? g0.x : n1, __dmul_rn(n2, d < 3 ? g0.y : n2)));
        const double dn = fma(mm, inv, d < 3 ? -g1.y : -0.0);
        const double pn = from(__dmul_rn(gm1, fma(-0.5, dn, n4)), 3), ep = __dadd_rn(n4, pn);
        auto term = [&](double n, double dv, double y, double v, const double2 &h) {
            const double w = __dmul_rn(h.y, v);
            return fma(h.x, fma(n, dv, y), DIR > 0 ? w : -w);
        };
        const double ya = fma(pn, ka, -fa), ta = term(c0 < 4 ? na : ep, from(dn, d0), c0 > 0 ? ya : -fa, va, ha);
        if (q < 15) *(double *)(wr + w_off) = ta;
        if constexpr (lanes == 8) {
            const double vb = from(dq, c1), nb = from(nq, c1), yb = fma(pn, kb, -fb);
            const double tb = term(c1 < 4 ? nb : ep, from(dn, d1), c1 > 0 ? yb : -fb, vb, hb);
            if (q < 7) *(double *)(wr + w_off4) = tb;
        }
        if (q < 5) ((double *)dq_out)[low ? 4 * cell + c : 4 * NC + cell] = dq;
    }
};

// the variable's sweep: A terms of the three directions, then V terms, then the division
template <typename T, int DIR, int N> struct CellStep<T, DIR, VAR, N> {
    using L = Lay<T, VAR, N>;
    static constexpr int NC = L::NC;
    static __device__ __forceinline__ T add(T a, T b) { if constexpr (sizeof(T) == 4) return __fadd_rn(a, b); else return __dadd_rn(a, b); }
    static __device__ __forceinline__ T mul(T a, T b) { if constexpr (sizeof(T) == 4) return __fmul_rn(a, b); else return __dmul_rn(a, b); }
    struct Pre { T vn, eb, sd, rl, lv, ev, alpha, r; };
    static __device__ __forceinline__ Pre pre(const char *in, int cell, int q)
    {
        const T *f = (const T *)in, *v = f + 3 * cell + (q < 3 ? q : 0);
        return {v[0], v[3 * NC], v[6 * NC], v[9 * NC], v[12 * NC], f[15 * NC + cell], f[16 * NC + cell], ((const T *)(in + L::flow_in))[cell]};
    }
    static __device__ __forceinline__ void run(const Pre &p, const char *rd, char *wr, int cell, int q, const int r_off[4], int w_off,
                                               int, bool active, T, char *dq_out)
    {
        const T vn = p.vn, eb = p.eb, sd = p.sd, rl = p.rl, lv = p.lv, ev = p.ev, alpha = p.alpha, r = p.r;
        const T *i = (const T *)(rd + r_off[0]), *j = (const T *)(rd + r_off[2]), *k = (const T *)(rd + L::KA) + 2 * cell;
        T t = DIR > 0 ? r : mul(alpha, r);
        t = DIR > 0 ? add(add(add(t, i[0]), j[0]), k[0]) : add(add(add(t, -i[0]), -j[0]), -k[0]);
        t = add(add(add(t, i[1]), j[1]), k[1]);
        const T d = active ? t / alpha : (T)0;
        const T dF = fma(add(ev, d), vn, -eb), x = mul(rl, d);
        if (q < 3) {
            ((T *)(wr + w_off))[0] = (T)0.5 * fma(dF, sd, DIR > 0 ? x : -x);
            ((T *)(wr + w_off))[1] = mul(lv, d);
        }
        if (q == 0) ((T *)dq_out)[cell] = d;
    }
};

template <typename T, int DIR, Kind K, int N>
__global__ void __launch_bounds__(192, sizeof(T) == 4 ? 4 : 2) k_wave(Batch B, WaveTables V, T gm1)
{
    using L = Lay<T, K, N>;
    constexpr int PA = L::PA, PB = L::PB, NC = L::NC;
    extern __shared__ __align__(128) char smem[];
    __shared__ unsigned s_take[2];
    const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
    const unsigned full = base + L::bars, edge = full + 8 * kStages, done = edge + 8 * kSlots;
    char *terms = smem + L::ring;
    if (threadIdx.x == 0) {
        s_take[0] = atomicAdd(&V.ctl->ticket[DIR > 0 ? 0 : 1], 1u);
        s_take[1] = 2u * V.ctl->epoch + (DIR > 0 ? 0u : 1u);
        for (int s = 0; s < kStages + 2 * kSlots; s++) bar_init(full + 8 * s);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for (int e = threadIdx.x; e < kSlots * L::slot / 16; e += blockDim.x) ((uint4 *)terms)[e] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const unsigned tag = s_take[1];
    const Where w = tile_of<DIR>(V, s_take[0]);
    const int T_ = w.S.T, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool edges = w.has_i || w.has_j;
    bool ok = true;
    if (warp < 4) {
        const int cell = threadIdx.x / kLanes<T, N>, q = threadIdx.x % kLanes<T, N>, a = cell / PB, b = cell % PB;
        const bool column = w.PI * PA + a < w.S.nI && w.PJ * PB + b < w.S.nJ;
        // (a step is called done only by a thread whose waits have all been met: its inputs have landed then)
        constexpr int F = DIR > 0 ? 1 : 0;          // forward: halo first
        // terms read: FP64, component q (or the fifth) of the three directions; otherwise both groups of I and J
        int r_off[4] = {off_ia<L>(a + 1 - F, b), off_ib<L>(a + 1 - F, b), off_ja<L>(a, b + 1 - F), off_jb<L>(a, b + 1 - F)};
        if (sizeof(T) == 8 && K == MEAN) {
            const bool low = q < 4;
            r_off[0] = low ? r_off[0] + 8 * q : r_off[1];
            r_off[1] = low ? r_off[2] + 8 * q : r_off[3];
            r_off[2] = low ? L::KA + 8 * (4 * cell + q) : L::KB + 8 * cell;
        }
        auto to_a = [&](int dir) { return dir == 0 ? off_ia<L>(a + F, b) : dir == 1 ? off_ja<L>(a, b + F) : L::KA + L::CA * cell * L::B; };
        auto to_b = [&](int dir) { return dir == 0 ? off_ib<L>(a + F, b) : dir == 1 ? off_jb<L>(a, b + F) : L::KB + L::CB * cell * L::B; };
        int w_off = to_a(q), w_off4 = to_b(q);
        if (sizeof(T) == 8 && K == MEAN) {             // terms written: q and q + 8 of the fifteen
            auto to = [&](int t) { return t % 5 < 4 ? to_a(t / 5) + 8 * (t % 5) : to_b(t / 5); };
            w_off = to(min(q, 14));
            w_off4 = to(min(q + 8, 14));
        }
        char *dq = V.dq + (w.step0 + (DIR > 0 ? 0 : T_ - 1)) * L::dq;
        int k = (DIR > 0 ? 0 : T_ - 1) - a - b;
        unsigned ph = 0;
        int slot = 0, stage = 0;
        const char *rd = terms + (kSlots - 1) * L::slot;
        using Step = CellStep<T, DIR, K, N>;
        if constexpr (sizeof(T) == 4 && K == MEAN && N) {
            auto input = [&](int st, int n) {            // (a stage holds its steps in order of t; the last one may hold fewer)
                const int u = n % kGroup, cnt = min(kGroup, T_ - (n - u));
                return smem + st * kGroup * L::step + (DIR > 0 ? u : cnt - 1 - u) * L::step;
            };
            bar_wait(full, 0, ok);
            typename Step::Pre now = Step::pre(input(0, 0), cell, q);
            for (int n = 0; n < T_; n++) {
                // the stage of the next step, and its phase
                const bool turn = (n + 1) % kGroup == 0;
                int next = stage;
                unsigned next_ph = ph;
                if (turn && ++next == kStages) { next = 0; next_ph ^= 1; }
                if (turn && n + 1 < T_) bar_wait(full + 8 * next, next_ph, ok);
                if (edges) bar_wait(edge + 8 * slot, ph, ok);
                const typename Step::Pre then = Step::pre(input(next, min(n + 1, T_ - 1)), cell, q);
                char *wr = terms + slot * L::slot;
                Step::run(now, rd, wr, cell, q, r_off, w_off, w_off4, column && (unsigned)k < (unsigned)w.S.nK, gm1, dq);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (threadIdx.x == 0 && ok) bar_arrive(done + 8 * slot);
                now = then;
                rd = wr;
                k += DIR;
                dq += DIR * L::dq;
                if (++slot == kSlots) slot = 0;
                stage = next;
                ph = next_ph;
            }
        } else {
            for (int n = 0; n < T_; n += kGroup) {
                bar_wait(full + 8 * stage, ph, ok);
                const char *in = smem + stage * kGroup * L::step;
                // (a stage holds its steps in order of t; the last one may hold fewer)
                const int cnt = min(kGroup, T_ - n);
#pragma unroll
                for (int u = 0; u < kGroup; u++) {
                    if (u >= cnt) break;
                    if (edges) bar_wait(edge + 8 * slot, ph, ok);
                    char *wr = terms + slot * L::slot;
                    Step::run(Step::pre(in + (DIR > 0 ? u : cnt - 1 - u) * L::step, cell, q), rd, wr, cell, q, r_off, w_off, w_off4,
                              column && (unsigned)k < (unsigned)w.S.nK, gm1, dq);
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (threadIdx.x == 0 && ok) bar_arrive(done + 8 * slot);
                    rd = wr;
                    k += DIR;
                    dq += DIR * L::dq;
                    slot++;
                }
                if (++stage == kStages) { stage = slot = 0; ph ^= 1; }
            }
        }
    } else if (warp == 4) {
        if (!edges) return;
        // packet p of a step's incoming ones: edge cell p / pp, part p % pp
        constexpr int RND = (L::pkt + 31) / 32;
        const uint4 *src[RND];
        int koff[RND], to[RND];
        bool mine[RND];
#pragma unroll
        for (int r = 0; r < RND; r++) {
            const int p = lane + 32 * r, e = p / L::pp, h = p % L::pp;
            const bool is_i = e < PB;
            const int a = is_i ? (DIR > 0 ? 0 : PA - 1) : e - PB, b = is_i ? e : (DIR > 0 ? 0 : PB - 1);
            mine[r] = p < L::pkt && (is_i ? w.has_i : w.has_j) && w.PI * PA + a < w.S.nI && w.PJ * PB + b < w.S.nJ;
            koff[r] = a + b;
            // the sender's edge column is PA - 1 (PB - 1) steps later in k
            const long long s0 = is_i ? w.from_i + DIR * (PA - 1) : w.from_j + DIR * (PB - 1);
            src[r] = V.pkt + s0 * L::pkt + p;
            const int row = DIR > 0 ? 0 : PA, col = DIR > 0 ? 0 : PB;
            const int oa = is_i ? off_ia<L>(row, b) : off_ja<L>(a, col), ob = is_i ? off_ib<L>(row, b) : off_jb<L>(a, col);
            if (L::B == 4) to[r] = h == 0 ? oa : ob;
            else to[r] = h < 4 ? oa + 8 * h : ob + 8 * (h - 4);
        }
        auto wants = [&](int r, int n) {
            const int k = (DIR > 0 ? n : T_ - 1 - n) - koff[r];
            return mine[r] && n < T_ && k >= 0 && k < w.S.nK;
        };
        unsigned long long lo[kAhead][RND], hi[kAhead][RND];
        auto ask = [&](int r, int n, unsigned long long &l, unsigned long long &h) {
            packet_load(src[r] + (long long)(DIR > 0 ? n : T_ - 1 - n) * L::pkt, l, h);
        };
        auto fresh = [&](unsigned long long h) { return (sizeof(T) == 4 ? (unsigned)(h >> 32) : (unsigned)h) == tag; };
#pragma unroll
        for (int u = 0; u < kAhead; u++)
#pragma unroll
            for (int r = 0; r < RND; r++) {
                lo[u][r] = hi[u][r] = 0;
                if (wants(r, u)) ask(r, u, lo[u][r], hi[u][r]);
            }
        int slot = 0;
        unsigned ph = 0;
        for (int n0 = 0; n0 < T_; n0 += kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                const int n = n0 + u;
                if (n >= T_) break;
                // the slot's halo cells are free once the step that read them last is done
                if (n >= kSlots) bar_wait_warp(done + 8 * slot, ph ^ 1, ok);
                for (unsigned polls = 0; ok; polls++) {
                    bool late = false;
#pragma unroll
                    for (int r = 0; r < RND; r++) late = late || (wants(r, n) && !fresh(hi[u][r]));
                    if (!__any_sync(0xffffffffu, late)) break;
                    if (polls > kWaitLimit) { ok = false; break; }
#pragma unroll
                    for (int r = 0; r < RND; r++)
                        if (wants(r, n) && !fresh(hi[u][r])) ask(r, n, lo[u][r], hi[u][r]);
                }
                // beside the terms of the last step
                char *s = terms + (slot == 0 ? kSlots - 1 : slot - 1) * L::slot;
#pragma unroll
                for (int r = 0; r < RND; r++)
                    if (wants(r, n)) {
                        if constexpr (L::pp == 1) *(float2 *)(s + to[r]) = make_float2(lo_f(lo[u][r]), hi_f(lo[u][r]));
                        else if constexpr (L::B == 4) {
                            float *d = (float *)(s + to[r]);
                            if (lane & 1) d[0] = hi_f(lo[u][r]);
                            else { d[0] = lo_f(lo[u][r]); d[1] = hi_f(lo[u][r]); d[2] = lo_f(hi[u][r]); }
                        } else *(double *)(s + to[r]) = __longlong_as_double((long long)lo[u][r]);
                    }
                if constexpr (L::B == 4 && K == MEAN) {
                    // the fourth component travels with the second packet
                    const unsigned w3 = __shfl_down_sync(0xffffffffu, (unsigned)lo[u][0], 1);
                    if ((lane & 1) == 0 && wants(0, n)) ((float *)(s + to[0]))[3] = __uint_as_float(w3);
                }
                __syncwarp();
                if (lane == 0) bar_arrive(edge + 8 * slot);
#pragma unroll
                for (int r = 0; r < RND; r++)
                    if (wants(r, n + kAhead)) ask(r, n + kAhead, lo[u][r], hi[u][r]);
                if (++slot == kSlots) { slot = 0; ph ^= 1; }
            }
        }
    } else {
        // inputs of a group of steps into its stage, on lane 0
        RingFeed<kStages> feed{(T_ + kGroup - 1) / kGroup};
        auto fetch = [&](int g, int stage) {
            const int n = g * kGroup, cnt = min(kGroup, T_ - n);
            const long long t = w.step0 + (DIR > 0 ? n : T_ - n - cnt);
            const unsigned bar = full + 8 * stage, d = base + stage * kGroup * L::step;
            bar_expect(bar, cnt * L::step);
            for (int u = 0; u < cnt; u++) {
                const unsigned x = d + u * L::step;
                if (L::geo) bulk_copy(x, V.geo + (t + u) * L::geo, L::geo, bar);
                bulk_copy(x + L::geo, V.flow + (t + u) * L::flow + (DIR > 0 ? 0 : L::ends), L::flow_in, bar);
                bulk_copy(x + L::geo + L::flow_in, V.dq + (t + u) * L::dq, L::dq, bar);
            }
        };
        if (lane == 0)
            for (int s = 0; s < kStages; s++) feed.next(ok, fetch);
        constexpr int RND = (L::pkt + 31) / 32;
        int from[RND];
        bool mine[RND];
#pragma unroll
        for (int r = 0; r < RND; r++) {
            const int p = lane + 32 * r, e = p / L::pp, h = p % L::pp;
            const bool is_i = e < PB;
            constexpr int F = DIR > 0 ? 1 : 0;
            const int a = is_i ? (DIR > 0 ? PA - 1 : 0) : e - PB, b = is_i ? e : (DIR > 0 ? PB - 1 : 0);
            mine[r] = p < L::pkt && (is_i ? w.next_i : w.next_j);
            const int oa = is_i ? off_ia<L>(a + F, b) : off_ja<L>(a, b + F), ob = is_i ? off_ib<L>(a + F, b) : off_jb<L>(a, b + F);
            if (L::B == 4) from[r] = h == 0 ? oa : ob;
            else from[r] = h < 4 ? oa + 8 * h : ob + 8 * (h - 4);
        }
        uint4 *dst = V.pkt + (w.step0 + (DIR > 0 ? 0 : T_ - 1)) * L::pkt + lane;
        int slot = 0;
        unsigned ph = 0;
        for (int n = 0; n < T_; n++) {
            bar_wait(done + 8 * slot, ph, ok);
            const char *s = terms + slot * L::slot;
            const unsigned long long tg = (unsigned long long)tag << 32;
            if constexpr (L::pp == 1) {
                if (mine[0]) {
                    const float2 v = *(const float2 *)(s + from[0]);
                    packet_store(dst, pack2(v.x, v.y), tg);
                }
            } else if constexpr (L::B == 4) {
                float x = 0, y = 0, z = 0, w3 = 0;
                if (mine[0]) {
                    if (lane & 1) y = *(const float *)(s + from[0]);
                    else { const float4 v = *(const float4 *)(s + from[0]); x = v.x; y = v.y; z = v.z; w3 = v.w; }
                }
                const float up = __shfl_up_sync(0xffffffffu, w3, 1);
                if (lane & 1) x = up;
                if (mine[0]) packet_store(dst, pack2(x, y), __float_as_uint(z) | tg);
            } else {
#pragma unroll
                for (int r = 0; r < RND; r++)
                    if (mine[r]) packet_store(dst + 32 * r, (unsigned long long)__double_as_longlong(*(const double *)(s + from[r])), tag);
            }
            dst += DIR * L::pkt;
            __syncwarp();
            if ((n + 1) % kGroup == 0 && lane == 0) feed.next(ok, fetch);
            if (++slot == kSlots) { slot = 0; ph ^= 1; }
        }
        // no copy is in flight when the block ends, also where a wait ran out
        if (lane == 0) {
            bool last = true;
            feed.drain([&](int stage, unsigned parity) { bar_wait(full + 8 * stage, parity, last); });
            ok = ok && last;
        }
    }
    if (!ok) atomicOr(&B.st[w.slot].status, GBT_STATUS_WAIT_TIMEOUT);
}

// ---- into step order: everything a cell contributes without its neighbours. Cells outside the solve's
// box get zeros and a density of one, with which every term they form is zero.
struct Chunk { bool live; WaveSolve S; int PI, PJ, t0, nt; long long step; };
__device__ __forceinline__ Chunk chunk_of(const WaveTables &V, int steps)
{
    Chunk c;
    c.S = V.solve[blockIdx.y];
    const int nc = (c.S.T + steps - 1) / steps, p = (int)blockIdx.x / nc;
    c.live = p < c.S.nPI * c.S.nPJ;
    c.PI = p / c.S.nPJ;
    c.PJ = p - c.PI * c.S.nPJ;
    c.t0 = ((int)blockIdx.x - p * nc) * steps;
    c.nt = min(steps, c.S.T - c.t0);
    c.step = c.S.step0 + (long long)p * c.S.T + c.t0;
    return c;
}
__device__ __forceinline__ void next_sweep(const WaveTables &V)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        V.ctl->epoch += 1;
        V.ctl->ticket[0] = V.ctl->ticket[1] = 0;
    }
}

// FP32: a block takes 16 steps of a tile, one thread per cell: a half-warp reads 16 consecutive k of a column
// (each column its own 16, shifted by a + b), and the block writes its steps as contiguous pieces through
// shared memory. Bound by the latency of its loads, some 30 per cell: with 32 steps and four cells per
// thread one after another it took 43 us on the 129x49x49 passage and 168 us per cycle on 32 solves of
// 25x25x65 nodes, one cell per thread 15 and 64 (40 for the bytes of the latter).
__global__ void __launch_bounds__(kCells<float, 0> * kSteps32) k_wave_gather32(Batch B, PhysW<float> P, Flow<float> W, WaveTables V)
{
    using L = Lay<float, MEAN>;
    constexpr int PA = L::PA, PB = L::PB, NC = L::NC;
    constexpr int NF = L::flow / 16, ND = L::dq / 16, stride = NF + ND + 1;      // quads per step, and in shared memory
    extern __shared__ __align__(128) char smem[];
    float4 *tile = (float4 *)smem;
    next_sweep(V);
    const Chunk c = chunk_of(V, kSteps32);
    if (!c.live) return;
    const Lvl Lv = B.lv[blockIdx.y];
    const int cell = threadIdx.x / kSteps32, st = threadIdx.x % kSteps32, a = cell / PB, b = cell % PB;
    const int i = c.PI * PA + a + 1, j = c.PJ * PB + b + 1, k = c.t0 + st - a - b + 1;
    float4 o = {1.0f, 0, 0, 0}, x = {0, 0, 1.0f, 0}, r = {0, 0, 0, 0};
    float2 hc[2][3] = {};
    float r4 = 0.0f;
    if (i <= c.S.nI && j <= c.S.nJ && k >= 1 && k <= c.S.nK) {
        const long long p = ix(Lv, i, j, k);
        const long long sn[3] = {(long long)Lv.NJ * Lv.NK, Lv.NK, 1};
        const double q0 = W.cv[0][p], q1 = W.cv[1][p], q2 = W.cv[2][p], q3 = W.cv[3][p], q4 = W.cv[4][p];
        const float *area = (const float *)V.area + (c.step + st) * (3 * NC) + 3 * cell;
        const float inva = W.dinv[p];
        float lc[3], lv[3], ar[3], up[3], dn[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lc[d] = W.lamc[d][p]; lv[d] = W.lamv[d][p]; ar[d] = area[d];
            // what the cell's term is scaled with is the diagonal of the cell that receives it (one that
            // lies outside the box has none and receives nothing)
            up[d] = W.dinv[p + sn[d]]; dn[d] = W.dinv[p - sn[d]];
        }
        const float s0 = W.res[0][p], s1 = W.res[1][p], s2 = W.res[2][p], s3 = W.res[3][p], s4 = W.res[4][p];
        x.y = W.pv[PP][p];
        o = make_float4(f64_to_f32_rn(q0), f64_to_f32_rn(q1), f64_to_f32_rn(q2), f64_to_f32_rn(q3));
        x.x = f64_to_f32_rn(q4);
        x.z = 1.0f / o.x;
        r = make_float4(__fmul_rn(-s0, inva), __fmul_rn(-s1, inva), __fmul_rn(-s2, inva), __fmul_rn(-s3, inva));
        r4 = __fmul_rn(-s4, inva);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const float h = 0.5f * ar[d], q = __fmaf_rn(0.5f, __fmul_rn(P.relax, lc[d]), lv[d]);
            hc[0][d] = make_float2(__fmul_rn(h, up[d]), __fmul_rn(q, up[d]));
            hc[1][d] = make_float2(__fmul_rn(h, dn[d]), __fmul_rn(q, dn[d]));
        }
    }
    char *t = smem + st * stride * 16;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        ((float2 *)t)[3 * cell + d] = hc[0][d];
        ((float2 *)(t + L::flow - L::ends))[3 * cell + d] = hc[1][d];
    }
    ((float4 *)(t + L::ends))[cell] = o;
    ((float4 *)(t + L::ends))[NC + cell] = x;
    ((float4 *)(t + L::flow))[cell] = r;
    ((float *)(t + L::flow))[4 * NC + cell] = r4;
    __syncthreads();
    float4 *df = (float4 *)(V.flow + c.step * L::flow), *dd = (float4 *)(V.dq + c.step * L::dq);
    for (int e = threadIdx.x; e < c.nt * NF; e += NC * kSteps32) df[e] = tile[(e / NF) * stride + e % NF];
    for (int e = threadIdx.x; e < c.nt * ND; e += NC * kSteps32) dd[e] = tile[(e / ND) * stride + NF + e % ND];
}

// FP64: one thread per cell and step, 16 steps per block (a line of a column's row serves them from L1). Bound by its FP64 instructions, some 75 per cell.
template <int N>
__global__ void __launch_bounds__(256) k_wave_gather64(Batch B, PhysW<double> P, Flow<double> W, WaveTables V)
{
    using L = Lay<double, MEAN, N>;
    constexpr int PA = L::PA, PB = L::PB, NC = L::NC;
    next_sweep(V);
    const Chunk c = chunk_of(V, kSteps<double, N>);
    const int cell = threadIdx.x % NC, st = threadIdx.x / NC, a = cell / PB, b = cell % PB;
    if (!c.live || st >= c.nt) return;
    const Lvl Lv = B.lv[blockIdx.y];
    const int i = c.PI * PA + a + 1, j = c.PJ * PB + b + 1, k = c.t0 + st - a - b + 1;
    char *blk = V.flow + (c.step + st) * L::flow;
    double2 *fw = (double2 *)blk + 3 * cell, *bw = (double2 *)(blk + L::flow - L::ends) + 3 * cell;
    double *f = (double *)(blk + L::ends) + 3 * cell, *oq = (double *)(blk + L::ends) + 15 * NC;
    double *rq = (double *)(V.dq + (c.step + st) * L::dq);
    if (i > c.S.nI || j > c.S.nJ || k < 1 || k > c.S.nK) {
        // (the rest of such a cell's block stays zero)
        oq[4 * cell] = 1.0;
        return;
    }
    const long long p = ix(Lv, i, j, k);
    const long long sn[3] = {(long long)Lv.NJ * Lv.NK, Lv.NK, 1};
    double o[5];
#pragma unroll
    for (int n = 0; n < 5; n++) o[n] = W.cv[n][p];
    const double po = W.pv[PP][p], inva = W.dinv[p], oinv = rcp_nr(o[0]);
    const double u = __dmul_rn(o[1], oinv), v = __dmul_rn(o[2], oinv), w = __dmul_rn(o[3], oinv), ep = __dadd_rn(o[4], po);
    const double2 *geo = (const double2 *)(V.geo + (c.step + st) * L::geo) + 3 * cell;
    const double *area = (const double *)V.area + (c.step + st) * (3 * NC) + 3 * cell;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double2 g0 = geo[d], g1 = geo[3 * NC + d];
        const double dv = __dadd_rn(fma(w, g1.x, fma(u, g0.x, __dmul_rn(v, g0.y))), -g1.y);
        f[d] = __dmul_rn(o[0], dv);
        f[3 * NC + d] = fma(po, g0.x, __dmul_rn(o[1], dv));
        f[6 * NC + d] = fma(po, g0.y, __dmul_rn(o[2], dv));
        f[9 * NC + d] = fma(po, g1.x, __dmul_rn(o[3], dv));
        f[12 * NC + d] = fma(po, g1.y, __dmul_rn(ep, dv));
        // what the cell's term is scaled with is the diagonal of the cell that receives it (one that lies
        // outside the box has none and receives nothing)
        const double h = 0.5 * area[d], q = fma(0.5, __dmul_rn(P.relax, W.lamc[d][p]), W.lamv[d][p]);
        const double up = W.dinv[p + sn[d]], dn = W.dinv[p - sn[d]];
        fw[d] = make_double2(__dmul_rn(h, up), __dmul_rn(q, up));
        bw[d] = make_double2(__dmul_rn(h, dn), __dmul_rn(q, dn));
    }
    double2 *o2 = (double2 *)(oq + 4 * cell), *r2 = (double2 *)(rq + 4 * cell);
    o2[0] = make_double2(o[0], o[1]);
    o2[1] = make_double2(o[2], o[3]);
    oq[4 * NC + cell] = o[4];
    r2[0] = make_double2(__dmul_rn(-W.res[0][p], inva), __dmul_rn(-W.res[1][p], inva));
    r2[1] = make_double2(__dmul_rn(-W.res[2][p], inva), __dmul_rn(-W.res[3][p], inva));
    rq[4 * NC + cell] = __dmul_rn(-W.res[4][p], inva);
}

// inputs of the variable's sweep of one direction, from the mean flow's dQ of that direction: everything
// that does not depend on the variable's own update
template <typename T, int DIR, int N>
__global__ void __launch_bounds__(256) k_wave_var(Batch B, PhysW<T> P, Geo G, Flow<T> W, WaveTables V, WaveTables VV)
{
    using L = Lay<T, VAR, N>;
    constexpr int PA = L::PA, PB = L::PB, NC = L::NC;
    next_sweep(VV);
    const Chunk c = chunk_of(V, kSteps<T, N>);
    const int cell = threadIdx.x % NC, st = threadIdx.x / NC, a = cell / PB, b = cell % PB;
    if (!c.live || st >= c.nt) return;
    const Lvl Lv = B.lv[blockIdx.y];
    const int i = c.PI * PA + a + 1, j = c.PJ * PB + b + 1, k = c.t0 + st - a - b + 1;
    T *f = (T *)(VV.flow + (c.step + st) * L::flow), *fd = f + 3 * cell;
    if (i > c.S.nI || j > c.S.nJ || k < 1 || k > c.S.nK) {
        f[16 * NC + cell] = (T)1;              // (a diagonal of one and zeros: no term, no update)
        return;
    }
    const long long p = ix(Lv, i, j, k);
    const T *dq = (const T *)(V.dq + (c.step + st) * Lay<T, MEAN, N>::dq) + 4 * cell;
    const double o0 = W.cv[0][p], o1 = W.cv[1][p], o2 = W.cv[2][p], o3 = W.cv[3][p];
    auto next = [&](double o, T q) { return to_work<T>(o + to_f64<T>(q)); };
    const T dn0 = next(o0, dq[0]), dn1 = next(o1, dq[1]), dn2 = next(o2, dq[2]), dn3 = next(o3, dq[3]);
    const T evo = to_work<T>(W.ev[p]);
    // the normals and areas as the mean flow's sweep has them
    const T *geo = (const T *)(V.geo + (c.step + st) * Lay<T, MEAN, N>::geo), *area = (const T *)V.area + (c.step + st) * (3 * Lay<T, MEAN, N>::NC) + 3 * cell;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int g = 3 * cell + d;
        const T nx = geo[sizeof(T) == 4 ? 4 * g : 2 * g], ny = geo[sizeof(T) == 4 ? 4 * g + 1 : 2 * g + 1],
                nz = geo[sizeof(T) == 4 ? 4 * g + 2 : 6 * NC + 2 * g];
        fd[d] = dn1 / dn0 * nx + dn2 / dn0 * ny + dn3 / dn0 * nz;
        if (DIR > 0) {
            const T q0 = to_work<T>(o0), Vold = to_work<T>(o1) / q0 * nx + to_work<T>(o2) / q0 * ny + to_work<T>(o3) / q0 * nz;
            fd[3 * NC + d] = evo * Vold;
            fd[6 * NC + d] = area[d];
            fd[9 * NC + d] = P.relax * W.lamc[d][p];
            fd[12 * NC + d] = W.lamv[d][p];
        }
    }
    if (DIR > 0) {
        const T lc = W.lamc[0][p] + W.lamc[1][p] + W.lamc[2][p];
        const T lv = W.lamv[0][p] + W.lamv[1][p] + W.lamv[2][p];
        f[15 * NC + cell] = evo;
        f[16 * NC + cell] = to_work<T>(G.vol[p]) / W.dt[p] + P.relax * lc + (T)3 * lv;
        ((T *)(VV.dq + (c.step + st) * L::dq))[cell] = -W.res_ev[p];
    }
}

// geometry of the steps (once per level): the mean normal, entrainment speed and area of each direction
template <typename T, int N>
__global__ void __launch_bounds__(256) k_wave_geometry(Batch B, Geo G, WaveTables V)
{
    constexpr int PA = kPA<T>, PB = kPB<T, N>, NC = kCells<T, N>;
    const WaveSolve S = V.solve[blockIdx.y];
    const Lvl Lv = B.lv[blockIdx.y];
    const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned st = e / NC;
    const int cell = (int)(e % NC);
    if (st >= (unsigned)(S.nPI * S.nPJ * S.T)) return;
    const int p = (int)(st / (unsigned)S.T), t = (int)(st - (unsigned)p * S.T), a = cell / PB, b = cell % PB;
    const int i = (p / S.nPJ) * PA + a + 1, j = (p % S.nPJ) * PB + b + 1, k = t - a - b + 1;
    if (i > S.nI || j > S.nJ || k < 1 || k > S.nK) return;            // (the pool is zeroed)
    const long long x = ix(Lv, i, j, k);
    char *o = V.geo + (S.step0 + st) * Lay<T, MEAN, N>::geo;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const T n0 = (T)G.cn[d][0][x], n1 = (T)G.cn[d][1][x], n2 = (T)G.cn[d][2][x], ve = (T)G.cve[d][x];
        if constexpr (sizeof(T) == 4) ((float4 *)o)[3 * cell + d] = make_float4(n0, n1, n2, ve);
        else {
            ((double2 *)o)[3 * cell + d] = make_double2(n0, n1);
            ((double2 *)o)[3 * NC + 3 * cell + d] = make_double2(n2, ve);
        }
        ((T *)V.area)[(S.step0 + st) * (3 * NC) + 3 * cell + d] = (T)G.cs[d][x];
    }
}

// ---- dQ back into box order and applied: Q_old = Q, Q += dQ (FP64 in both precision forms), primitive
// variables, limiter. A block takes the 32 k of every column of a tile that share a line of the box (the
// rows' padded index a multiple of 32 on), which lie in up to 42 steps. Bound by HBM (184 bytes a cell in
// the mixed form) on large batches: 12 solves on three meshes 0.255 ms per cycle as two launches, scatter
// and update, 0.214 as one; with runs of 16 or 32 k that start anywhere, 0.352 and 0.285.
constexpr int kRun = 32;
__host__ __device__ inline int runs_of(int nK) { return (nK + PAD) / kRun + 1; }
template <typename T, int N>
__global__ void __launch_bounds__(256) k_wave_update(Batch B, Phys P, Flow<T> W, WaveTables V, int level, LimitLists q)
{
    using L = Lay<T, MEAN, N>;
    constexpr int PA = L::PA, PB = L::PB, NC = L::NC, R = NC * kRun / 256, NW = L::dq / 16, stride = NW + 1, ST = kRun + PA + PB - 2;
    __shared__ float4 tile[ST * stride];
    const int s = blockIdx.y;
    const WaveSolve S = V.solve[s];
    const int nr = runs_of(S.nK), p = (int)blockIdx.x / nr, k0 = ((int)blockIdx.x - p * nr) * kRun - PAD;
    if (p >= S.nPI * S.nPJ) return;
    const int PI = p / S.nPJ, PJ = p - PI * S.nPJ;
    const Lvl Lv = B.lv[s];
    // cells (a, b, k) of the run, at step k - 1 + a + b
    const int kk = k0 + (int)threadIdx.x % kRun, c0 = (int)threadIdx.x / kRun;
    bool in[R];
    long long at[R];
    double o[R][5];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int cell = c0 + r * (256 / kRun), i = PI * PA + cell / PB + 1, j = PJ * PB + cell % PB + 1;
        in[r] = i <= S.nI && j <= S.nJ && kk >= 1 && kk <= S.nK;
        at[r] = ix(Lv, i, j, kk);
#pragma unroll
        for (int n = 0; n < 5; n++) o[r][n] = in[r] ? W.cv[n][at[r]] : 0.0;
    }
    const int t0 = max(0, k0 - 1), t1 = min(S.T, k0 - 1 + ST);
    const float4 *src = (const float4 *)(V.dq + (S.step0 + (long long)p * S.T + t0) * L::dq);
    for (int e = threadIdx.x; e < (t1 - t0) * NW; e += 256) tile[(e / NW) * stride + e % NW] = src[e];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (!in[r]) continue;
        const int cell = c0 + r * (256 / kRun), a = cell / PB, b = cell % PB;
        const T *d = (const T *)(tile + (kk - 1 + a + b - t0) * stride);
        double cv[5];
#pragma unroll
        for (int n = 0; n < 5; n++) {
            const T dq = n < 4 ? d[4 * cell + n] : d[4 * NC + cell];
            W.dq[n][at[r]] = dq;
            W.cvold[n][at[r]] = o[r][n];
            cv[n] = o[r][n] + to_f64<T>(dq);
            W.cv[n][at[r]] = cv[n];
        }
        T v[6];
        prim_from_cons<T>(P, cv, v);
#pragma unroll
        for (int n = 0; n < 6; n++) W.pv[n][at[r]] = v[n];
        limit_flag<T>(P, q, Lv, s, PI * PA + a + 1, PJ * PB + b + 1, kk, v);
    }
    limit_done<T>(B, P, W, level, q, s, (unsigned)(S.nPI * S.nPJ * nr));
}

template <typename T, int N>
__global__ void __launch_bounds__(256) k_wave_scatter_var(Batch B, Flow<T> W, WaveTables VV)
{
    constexpr int PA = kPA<T>, PB = kPB<T, N>, NC = kCells<T, N>;
    const Chunk c = chunk_of(VV, kSteps<T, N>);
    const int cell = threadIdx.x % NC, st = threadIdx.x / NC, a = cell / PB, b = cell % PB;
    if (!c.live || st >= c.nt) return;
    const int i = c.PI * PA + a + 1, j = c.PJ * PB + b + 1, k = c.t0 + st - a - b + 1;
    if (i > c.S.nI || j > c.S.nJ || k < 1 || k > c.S.nK) return;
    W.dq_ev[ix(B.lv[blockIdx.y], i, j, k)] = ((const T *)(VV.dq + (c.step + st) * Lay<T, VAR, N>::dq))[cell];
}

constexpr unsigned kGatherBytes = kSteps32 * (Lay<float, MEAN>::flow + Lay<float, MEAN>::dq + 16);

// Shared memory of a block of the march. FP64: no more than two blocks on an SM, whose FP64 pipes they share:
// further ones slow the tiles that the others wait for (forward sweep of four 129x49x49 passages 1110 us
// with four blocks, 903 with two, 1012 with one; of one 161x65x65 passage 751, 751, 709).
template <typename T, Kind K, int N> constexpr int kMarchShared = sizeof(T) == 8 && Lay<T, K, N>::smem < 100000 ? 100000 : Lay<T, K, N>::smem;

// (shared memory beyond the default limit has to be asked for, once per kernel and device)
template <typename T, Kind K, int N>
void allow_shared()
{
    cudaFuncSetAttribute(k_wave<T, 1, K, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMarchShared<T, K, N>);
    cudaFuncSetAttribute(k_wave<T, -1, K, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMarchShared<T, K, N>);
}

template <typename T, int DIR, Kind K, int N>
void march(const LaunchCtx &ctx, const WaveTables &V, T gm1)
{
    k_wave<T, DIR, K, N><<<V.n_item, 192, kMarchShared<T, K, N>, ctx.stream>>>(ctx.batch, V, gm1);
}

// f with the tiles' shape as a constant
template <typename T, typename F>
void with_shape(const WaveTables &V, F f)
{
    if (V.narrow) f(std::integral_constant<int, 1>{});
    else f(std::integral_constant<int, 0>{});
}

}  // namespace

void wave_patch(int fp64, int narrow, int &pa, int &pb)
{
    pa = fp64 ? kPA<double> : kPA<float>;
    pb = fp64 && narrow ? kPB<double, 1> : kPB<float, 0>;
}

void wave_bytes(int fp64, int narrow, int sa, WaveBytes &w)
{
    auto set = [&](auto mean, auto var) {
        using L = decltype(mean);
        using X = decltype(var);
        w = {L::geo, L::flow, L::dq, L::pkt * 16, 3 * L::NC * L::B, 0, 0, 0};
        if (sa) { w.var_flow = X::flow; w.var_dq = X::dq; w.var_pkt = X::pkt * 16; }
    };
    if (fp64 && narrow) set(Lay<double, MEAN, 1>{}, Lay<double, VAR, 1>{});
    else if (fp64) set(Lay<double, MEAN>{}, Lay<double, VAR>{});
    else set(Lay<float, MEAN>{}, Lay<float, VAR>{});
}

template <typename T>
void launch_wave_geometry(const LaunchCtx &ctx, const Geo &G, const WaveTables &V)
{
    if (sizeof(T) == 4) cudaFuncSetAttribute(k_wave_gather32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGatherBytes);
    with_shape<T>(V, [&](auto shape) {
        constexpr int N = decltype(shape)::value;
        allow_shared<T, MEAN, N>();
        allow_shared<T, VAR, N>();
        k_wave_geometry<T, N><<<ctx.grid_n(V.max_steps * kCells<T, N>, 256), 256, 0, ctx.stream>>>(ctx.batch, G, V);
    });
}

template <typename T, int N>
static void sweeps(const LaunchCtx &ctx, const Phys &PH, const PhysW<T> &P, const Geo &G, Flow<T> W, const WaveTables &V,
                         const WaveTables &VV, int level, const LimitLists &q)
{
    auto chunks = [&](int steps) { return dim3((unsigned)(V.max_tiles * ((V.max_T + steps - 1) / steps)), ctx.batch.nsolve); };
    ctx.mark("sweep_forward", 1, 2);
    if constexpr (sizeof(T) == 4) k_wave_gather32<<<chunks(kSteps32), kCells<float, 0> * kSteps32, kGatherBytes, ctx.stream>>>(ctx.batch, P, W, V);
    else k_wave_gather64<N><<<chunks(kSteps<T, N>), 256, 0, ctx.stream>>>(ctx.batch, P, W, V);
    march<T, 1, MEAN, N>(ctx, V, P.gm1);
    ctx.mark("sweep_forward", 0, 2);
    // The variable's sweep of a direction needs the mean flow's dQ of that direction and nothing of the other one,
    // nor of the update: its march, as the mean flow's bound by the chain of planes, runs beside them on the
    // second stream once its inputs are formed.
    LaunchCtx second = ctx;
    if (ctx.side) second.stream = ctx.side;
    auto beside = [&](auto launches) {
        if (ctx.side) {
            cudaEventRecord(ctx.fork, ctx.stream);
            cudaStreamWaitEvent(ctx.side, ctx.fork, 0);
        }
        launches();
        if (ctx.side) cudaEventRecord(ctx.join, ctx.side);
    };
    auto meet = [&] { if (ctx.side) cudaStreamWaitEvent(ctx.stream, ctx.join, 0); };
    if (W.ev) {
        ctx.mark("sa_sweeps", 1, 2);
        k_wave_var<T, 1, N><<<chunks(kSteps<T, N>), 256, 0, ctx.stream>>>(ctx.batch, P, G, W, V, VV);
        beside([&] { march<T, 1, VAR, N>(second, VV, (T)0); });
        ctx.mark("sa_sweeps", 0, 2);
    }
    ctx.mark("sweep_backward", 1, 1);
    march<T, -1, MEAN, N>(ctx, V, P.gm1);
    ctx.mark("sweep_backward", 0, 1);
    if (W.ev) {
        ctx.mark("sa_sweeps", 1, 3);
        meet();
        k_wave_var<T, -1, N><<<chunks(kSteps<T, N>), 256, 0, ctx.stream>>>(ctx.batch, P, G, W, V, VV);
        beside([&] {
            march<T, -1, VAR, N>(second, VV, (T)0);
            k_wave_scatter_var<T, N><<<chunks(kSteps<T, N>), 256, 0, second.stream>>>(ctx.batch, W, VV);
        });
        ctx.mark("sa_sweeps", 0, 3);
    }
    ctx.mark("update_limiter", 1, 1);
    k_wave_update<T, N><<<dim3((unsigned)(V.max_tiles * runs_of(ctx.maxKM - 1)), ctx.batch.nsolve), 256, 0, ctx.stream>>>(ctx.batch, PH, W, V, level, q);
    if (W.ev) {
        meet();
        // the variable's update and Limit_SA after the mean flow's (source/LU_SGS_Marching.cpp:275-277,
        // source/ComputeAllBlockVars.cpp:257-266); the limiter's list is reused
        launch_sa_update<T>(ctx, PH, W, q.list, q.cap, q.count);
        if (PH.limiter) {
            launch_sa_limit<T>(ctx, W, q.list, q.cap, q.count);
            cudaMemsetAsync(q.count, 0, sizeof(int) * ctx.batch.nsolve, ctx.stream);
        }
    }
    ctx.mark("update_limiter", 0, 1);
}

template <typename T>
void launch_lusgs_sweeps(const LaunchCtx &ctx, const Phys &PH, const PhysW<T> &P, const Geo &G, Flow<T> W, const WaveTables &V,
                         const WaveTables &VV, int level, const LimitLists &q)
{
    with_shape<T>(V, [&](auto shape) { sweeps<T, decltype(shape)::value>(ctx, PH, P, G, W, V, VV, level, q); });
}

#define GBT_WAVE_INST(T)                                                                                              \
    template void launch_wave_geometry<T>(const LaunchCtx &, const Geo &, const WaveTables &);                        \
    template void launch_lusgs_sweeps<T>(const LaunchCtx &, const Phys &, const PhysW<T> &, const Geo &, Flow<T>,     \
                                         const WaveTables &, const WaveTables &, int, const LimitLists &);
GBT_WAVE_INST(double)
GBT_WAVE_INST(float)

}  // namespace gbt
