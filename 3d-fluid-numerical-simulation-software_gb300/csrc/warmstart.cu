// Learned warm start (see warmstart.hpp): the network's kernels and its host side.
//
// The three products of training and inference run on the tcgen05 tensor cores with the
// accumulator in tensor memory (TMEM):
//   forward        Z[cells x N]   = H[cells x K] . W[N x K]^T        (+ bias, SiLU in the epilogue)
//   backward data  dH[cells x K]  = dZ[cells x N] . W[N x K]          (x SiLU'(Z) in the epilogue)
//   weight grad    dW[N x K]      = dZ^T . H  (the cells are the reduction dimension)
// Operands are staged in shared memory by TMA in the 128-byte swizzle (boxes of 64 columns, a row of 128
// bytes; operands of 16 columns and the activations of the fused inference in core matrices of 8 rows x
// 16 bytes, without swizzle), one elected thread issues
// tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = 128), tcgen05.commit arrives on an mbarrier
// that every thread waits on (bounded), and the epilogue reads the accumulator rows with
// tcgen05.ld (warp w owns TMEM lanes 32w..32w+31, i.e. rows 32w..32w+31 of the tile).
#include "warmstart.hpp"
#include "gbt_common.cuh"
#include "host_rows.hpp"
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <stdexcept>
#include <string>

namespace gbt {

typedef __nv_bfloat16 bf16;

#define WCK(x) check_cuda((x), #x)

// ---------------------------------------------------------------- tcgen05 / mbarrier primitives
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor (tcgen05 form, no swizzle): start address, byte distance between
// core matrices adjacent along K (lbo) and along M/N (sbo), all in 16-byte units; bits 46-47 = 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// the same for an operand in the 128-byte swizzle (bits 61-63 = 2; 1024-byte groups of eight 128-byte rows).
// K-major: sbo is the distance of groups adjacent along M/N, lbo is not read. MN-major (a row is 64 elements
// of M/N): lbo is the distance of blocks of 64 along M/N, sbo that of groups adjacent along K.
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return smem_desc(addr, lbo, sbo) | (2ull << 61);
}
// instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1),
// both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// some 17 s at most (a poll of a barrier that does not complete takes 4 us); a wait that runs out is reported through
// the error flag
constexpr int kMbarWaitLimit = 1 << 22;
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity)
{
    for (int t = 0; t < kMbarWaitLimit; t++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (t > 32) __nanosleep(64);
    }
    return false;
}
// the same for a whole warp, which goes on together: a wait that runs out on one of its lanes has run out on all
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity)) != 0;
}
// 32 TMEM lanes x 16 columns of 32 bits: thread t of the warp receives lane (base lane + t)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// the same for 32 columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------- operand staging
// 1 / (1 + 2^(-z log2 e)). The forms that flush subnormal numbers save the scaling around them and give the
// bits of __expf and __fdividef: a flushed power adds nothing to 1, and the quotient by more than 2^126 is 0
// in both. Inference of 262144 rows 188 us before, 168 now.
__device__ __forceinline__ float sigmoidf_(float z)
{
    float e, s;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.0f + e));
    return s;
}

constexpr int kChunk = 64;
constexpr int kEpiWarps = 16;                    // four per TMEM lane quadrant
constexpr int kEpiStage = 32 * 64;               // 32 rows x 32 BF16 columns per epilogue warp

__host__ __device__ inline int tmem_cols(int n) { int c = 32; while (c < n) c <<= 1; return c; }

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// ---------------------------------------------------------------- the row products, all layers fused
// The products of rows (cells) with the layers' matrices, D[128 x N] = A[128 x K] . B[N x K]^T per tile of 128
// rows and layer, a tile's activations kept on chip from layer to layer:
//   PASS_INFER     Y[rows x 16] = the whole network on X[rows x 64]; nothing but X and Y crosses HBM
//   PASS_FORWARD   the same, and Z = D + bias, H = SiLU(Z) of every hidden layer stored (BF16) for the gradients
//   PASS_BACKWARD  from dY[rows x 16]: dZ5 = (dY . W6) * SiLU'(Z5), ..., dZ1 = (dZ2 . W2) * SiLU'(Z1), stored (BF16)
// A CTA works on two tiles in turn, so that the tensor cores run a layer of one while the epilogue warps are
// on the other: each has a shared-memory buffer of activations (K-major core matrices: 8-column groups
// 2 KB apart, rows 16 B apart) and a TMEM accumulator. Persistent over the tiles:
//   warp 16: TMA producer. Loads a tile's input rows into its activation buffer once the last layer of the
//     buffer's previous tile has read it, and streams the weights, 64-column chunk by chunk in the
//     128-byte swizzle, layer by layer and tile by tile, through a ring (they stay in L2). Rows past M read
//     as zeros. (16 columns: boxes of 8, no swizzle.)
//   warp 17: MMA issuer. Per layer and tile: waits for the tile's epilogue of the layer before (its
//     outputs are this layer's inputs, and it has read the accumulator out), issues the layer's MMAs with A
//     from the activation buffer, commits the accumulator; after the last layer it frees the buffer.
//   warps 0-15: epilogue (warp w: TMEM lanes 32(w%4)..32(w%4)+31, the (w/4)-th quarter of the columns).
//     Bias and SiLU of the accumulator, or the product with SiLU', rounded to BF16, written over the
//     activation buffer, and stored; or bias and FP32 rows of Y (the output layer). Rows of 32 BF16 columns
//     go to and come from HBM through 2 KB of shared memory per warp, so that an access covers 8 rows x
//     64 bytes instead of 32 rows x 16.
// Inference and forward pass have the same MMA order and arithmetic, so the same bits in Y. Bound by the
// epilogue's MUFU operations (two an element, 16 a clock: 144 us for the inference of 262144 rows). Inference of
// 262144 rows with boxes of 8 columns (about one row of 16 bytes a clock) and one tile at a time 371 us,
// now 168 us. On 32768 rows a launch per layer took 90 us forward and 76 us backward, now 52 and 46.
enum { PASS_INFER, PASS_FORWARD, PASS_BACKWARD };
struct ChainArgs {
    long long M;
    const float *bias[kWsLayers];
    float *Y;
    bf16 *Z[kWsLayers - 1], *H[kWsLayers - 1], *dZ[kWsLayers - 1];
    int *err;
};
constexpr int kStageB = kWsHidden * kChunk * 2;
constexpr int kActs = 128 * kWsHidden * 2;                  // 64 KB of activations
__host__ __device__ constexpr int chain_stages(int pass) { return pass == PASS_INFER ? 3 : 2; }
__host__ __device__ constexpr int chain_smem(int pass)
{
    return chain_stages(pass) * kStageB + 2 * kActs + (pass == PASS_INFER ? 0 : kEpiWarps * kEpiStage) + 256;
}
__host__ __device__ constexpr int chain_layers(int pass) { return pass == PASS_BACKWARD ? kWsLayers - 1 : kWsLayers; }
__host__ __device__ constexpr int chain_n(int pass, int l) { return pass != PASS_BACKWARD && l == kWsLayers - 1 ? kWsOut : kWsHidden; }
__host__ __device__ constexpr int chain_k(int pass, int l) { return l > 0 ? kWsHidden : pass == PASS_BACKWARD ? kWsOut : kWsIn; }

// 32 rows x 32 BF16 columns (one row per lane in v) to rows row0.. of dst through the warp's 2 KB
__device__ __forceinline__ void store_rows32(unsigned char *st, int lane, const bf16 v[32], bf16 *dst, long long row0, long long M)
{
#pragma unroll
    for (int c = 0; c < 4; c++)
        *reinterpret_cast<uint4 *>(st + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = reinterpret_cast<const uint4 *>(v)[c];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int r = q * 8 + (lane >> 2), c = lane & 3;
        const uint4 w = *reinterpret_cast<const uint4 *>(st + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
        if (row0 + r < M) *reinterpret_cast<uint4 *>(dst + (row0 + r) * kWsHidden + c * 8) = w;
    }
    __syncwarp();
}

template <int PASS>
__global__ void __launch_bounds__(32 * (kEpiWarps + 2), 1) k_mlp_chain(
    const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tw0, const __grid_constant__ CUtensorMap tw1,
    const __grid_constant__ CUtensorMap tw2, const __grid_constant__ CUtensorMap tw3, const __grid_constant__ CUtensorMap tw4,
    const __grid_constant__ CUtensorMap tw5, const __grid_constant__ ChainArgs g)
{
    constexpr int kStages = chain_stages(PASS), NL = chain_layers(PASS), KX = chain_k(PASS, 0);
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char *ring = sm;                                           // weight chunks
    unsigned char *hbuf = sm + kStages * kStageB;                    // activations of two tiles
    unsigned char *epi = hbuf + 2 * kActs;                               // rows on their way, per epilogue warp
    uint64_t *bars = reinterpret_cast<uint64_t *>(epi + (PASS == PASS_INFER ? 0 : kEpiWarps * kEpiStage));
    // bars: full[], empty[]; of each tile x_full, h_free, acc_full, h_ready
    uint32_t *slot = reinterpret_cast<uint32_t *>(bars + 2 * kStages + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(kStages + s); };
    auto x_full = [&](int h) { return bar0 + 8u * (uint32_t)(2 * kStages + 4 * h); };
    auto h_free = [&](int h) { return x_full(h) + 8u; };
    auto acc_full = [&](int h) { return x_full(h) + 16u; };
    auto h_ready = [&](int h) { return x_full(h) + 24u; };
    if (warp == kEpiWarps) tmem_alloc(smem_u32(slot), 512);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int h = 0; h < 2; h++) {
            mbar_init(x_full(h), 1);
            mbar_init(h_free(h), 1);
            mbar_init(acc_full(h), 1);
            mbar_init(h_ready(h), kEpiWarps);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot;
    const long long tiles = (g.M + 127) / 128, step = 2 * (long long)gridDim.x;
    bool failed = false;
    // pair p of the CTA's tiles: blockIdx.x + 2 p gridDim.x and, where there is one, the tile gridDim.x further
    if (warp == kEpiWarps) {
        if (lane == 0) {
            long long it = 0, p = 0;
            int xs[2] = {0, 0};                                         // input loads issued
            for (long long t = blockIdx.x; t < tiles && !failed; t += step, p++) {
                const int nh = t + gridDim.x < tiles ? 2 : 1;
                for (int l = 0; l < NL && !failed; l++) {
                    const CUtensorMap *wm = l == 0 ? &tw0 : l == 1 ? &tw1 : l == 2 ? &tw2 : l == 3 ? &tw3 : l == 4 ? &tw4 : &tw5;
                    const int n = chain_n(PASS, l), k = chain_k(PASS, l), w = k < kChunk ? k : kChunk;
                    for (int h = 0; h < nh && !failed; h++) {
                        if (l == 0) {
                            if (!mbar_wait_bounded(h_free(h), (uint32_t)((p & 1) ^ 1))) { failed = true; break; }
                            mbar_expect_tx(x_full(h), (uint32_t)(KX / 8) * 128u * 16u);
                            const uint32_t hb = smem_u32(hbuf + (size_t)h * kActs);
                            for (int k8 = 0; k8 < KX / 8; k8++)
                                tma_load_2d(hb + (uint32_t)k8 * 2048u, &tmX, k8 * 8, (int)((t + h * (long long)gridDim.x) * 128), x_full(h));
                            xs[h]++;
                        }
                        for (int kc = 0; kc < k / w; kc++, it++) {
                            const int s = (int)(it % kStages);
                            if (!mbar_wait_bounded(empty(s), (uint32_t)(((it / kStages) & 1) ^ 1))) { failed = true; break; }
                            mbar_expect_tx(full(s), (uint32_t)(w * n) * 2u);
                            const uint32_t b_s = smem_u32(ring + (size_t)s * kStageB);
                            if (w == kChunk) tma_load_2d(b_s, wm, kc * kChunk, 0, full(s));
                            else
                                for (int k8 = 0; k8 < w / 8; k8++) tma_load_2d(b_s + (uint32_t)(k8 * n) * 16u, wm, k8 * 8, 0, full(s));
                        }
                    }
                }
            }
            // nothing of a tile that was given up on may still be on its way when the CTA ends
            if (failed) {
                for (int h = 0; h < 2; h++)
                    if (xs[h] > 0) mbar_wait_bounded(x_full(h), (uint32_t)((xs[h] - 1) & 1));
                for (long long q = it < kStages ? 0 : it - kStages; q < it; q++)
                    mbar_wait_bounded(full((int)(q % kStages)), (uint32_t)((q / kStages) & 1));
            }
        }
    } else if (warp == kEpiWarps + 1) {
        if (lane == 0) {
            long long it = 0, p = 0;
            uint32_t hu[2] = {0u, 0u};                                  // epilogues waited for
            for (long long t = blockIdx.x; t < tiles && !failed; t += step, p++) {
                const int nh = t + gridDim.x < tiles ? 2 : 1;
                for (int l = 0; l < NL && !failed; l++) {
                    const int n = chain_n(PASS, l), k = chain_k(PASS, l), w = k < kChunk ? k : kChunk;
                    const uint32_t idesc = idesc_bf16(128, n);
                    for (int h = 0; h < nh && !failed; h++) {
                        if (l == 0 && !mbar_wait_bounded(x_full(h), (uint32_t)(p & 1))) { failed = true; break; }
                        // the epilogue of the layer before has written this layer's inputs and read the accumulator
                        if (p > 0 || l > 0) {
                            if (!mbar_wait_bounded(h_ready(h), hu[h] & 1u)) { failed = true; break; }
                            hu[h]++;
                        }
                        tc_fence_after();
                        const uint32_t hb = smem_u32(hbuf + (size_t)h * kActs);
                        for (int kc = 0; kc < k / w; kc++, it++) {
                            const int s = (int)(it % kStages);
                            if (!mbar_wait_bounded(full(s), (uint32_t)((it / kStages) & 1))) { failed = true; break; }
                            tc_fence_after();
                            const uint32_t b_s = smem_u32(ring + (size_t)s * kStageB);
                            for (int ks = 0; ks < w / 16; ks++)
                                mma_bf16(tmem + (uint32_t)(h * 256),
                                         smem_desc(hb + (uint32_t)(kc * (kChunk / 16) + ks) * 2u * 2048u, 2048u, 128u),
                                         w == kChunk ? smem_desc_sw(b_s + (uint32_t)ks * 32u, 16u, 1024u)
                                                     : smem_desc(b_s + (uint32_t)(2 * ks * n) * 16u, (uint32_t)n * 16u, 128u),
                                         idesc, (kc > 0 || ks > 0) ? 1u : 0u);
                            mma_commit(empty(s));
                        }
                        if (failed) break;
                        mma_commit(acc_full(h));
                        if (l == NL - 1) mma_commit(h_free(h));
                    }
                }
            }
        }
    } else {
        uint32_t au[2] = {0u, 0u};                                     // accumulators waited for
        const int quad = warp & 3;
        unsigned char *st = epi + warp * kEpiStage;
        const int r = quad * 32 + lane;                                // the TMEM lane = row of the tile
        for (long long t = blockIdx.x; t < tiles && !failed; t += step) {
            const int nh = t + gridDim.x < tiles ? 2 : 1;
            for (int l = 0; l < NL && !failed; l++) {
                for (int h = 0; h < nh; h++) {
                    const long long row0 = (t + h * (long long)gridDim.x) * 128 + quad * 32;
                    const int cbeg = (warp >> 2) * (kWsHidden / 4);
                    uint4 zl[2][4];                          // Z of the warp's 64 columns, asked for before the wait
                    if constexpr (PASS == PASS_BACKWARD) {
                        const bf16 *Z = g.Z[NL - 1 - l] + cbeg + (lane & 3) * 8;
#pragma unroll
                        for (int c = 0; c < 2; c++)
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const long long zr = row0 + q * 8 + (lane >> 2);
                                zl[c][q] = zr < g.M ? *reinterpret_cast<const uint4 *>(Z + zr * kWsHidden + c * 32) : make_uint4(0u, 0u, 0u, 0u);
                            }
                    }
                    const bool ok = mbar_wait_warp(acc_full(h), au[h] & 1u);
                    au[h]++;
                    tc_fence_after();
                    if (!ok) { failed = true; break; }
                    const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(h * 256);
                    if (PASS == PASS_BACKWARD || l < NL - 1) {
                        const float *bias = g.bias[l];
                        unsigned char *hb = hbuf + (size_t)h * kActs + (size_t)r * 16;
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            const int c0 = cbeg + c * 32;
                            float v[32];
                            tmem_ld32(acc + (uint32_t)c0, v);
                            alignas(16) bf16 ho[32];
                            if constexpr (PASS == PASS_BACKWARD) {
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const int zr = q * 8 + (lane >> 2), zc = lane & 3;
                                    *reinterpret_cast<uint4 *>(st + zr * 64 + ((zc ^ ((zr >> 1) & 3)) << 4)) = zl[c][q];
                                }
                                __syncwarp();
                                alignas(16) bf16 zi[32];
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    reinterpret_cast<uint4 *>(zi)[q] = *reinterpret_cast<const uint4 *>(st + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4));
                                __syncwarp();
#pragma unroll
                                for (int i = 0; i < 32; i++) {
                                    const float z = __bfloat162float(zi[i]);
                                    const float sg = sigmoidf_(z);
                                    ho[i] = __float2bfloat16_rn(v[i] * (sg * (1.0f + z * (1.0f - sg))));
                                }
                                store_rows32(st, lane, ho, g.dZ[NL - 1 - l] + c0, row0, g.M);
                            } else {
                                alignas(16) bf16 zo[32];
#pragma unroll
                                for (int i = 0; i < 32; i += 4) {
                                    const float4 b = *reinterpret_cast<const float4 *>(bias + c0 + i);
                                    const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                                    for (int n = 0; n < 4; n++) {
                                        const float z = v[i + n] + bb[n];
                                        zo[i + n] = __float2bfloat16_rn(z);
                                        ho[i + n] = __float2bfloat16_rn(z * sigmoidf_(z));
                                    }
                                }
                                if constexpr (PASS == PASS_FORWARD) {
                                    store_rows32(st, lane, zo, g.Z[l] + c0, row0, g.M);
                                    store_rows32(st, lane, ho, g.H[l] + c0, row0, g.M);
                                }
                            }
                            if (l < NL - 1)
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    *reinterpret_cast<uint4 *>(hb + (size_t)(c0 / 8 + q) * 2048) = reinterpret_cast<uint4 *>(ho)[q];
                        }
                    } else if (warp < 4) {
                        const float *bias = g.bias[l];
                        float v[16];
                        tmem_ld16(acc, v);
                        const long long row = row0 + lane;
                        if (row < g.M) {
                            float4 *yp = reinterpret_cast<float4 *>(g.Y + row * kWsOut);
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                yp[i] = make_float4(v[4 * i] + bias[4 * i], v[4 * i + 1] + bias[4 * i + 1],
                                                    v[4 * i + 2] + bias[4 * i + 2], v[4 * i + 3] + bias[4 * i + 3]);
                        }
                    }
                    fence_proxy_async();                               // the activations, for the tensor cores
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(h_ready(h));
                }
            }
        }
    }
    if (failed) atomicOr(g.err, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kEpiWarps) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- the gradients
// Of layer l: part[(ay * gridDim.x + bx)][b][a] = sum over the CTA's cells of Xa[cell][128 ay + a] Xb[cell][b]
// (a < 128, b < Nb): the cells are the product's K, split over blockIdx.x; blockIdx.z is the layer, so that one
// launch covers the network. Both operands are MN-major: a TMA box of 64 features x 64 cells lands in the
// 128-byte swizzle as 64 rows of 128 bytes, 8 KB from the next 64 features. (Xb of 16 features: two boxes of
// 8, core matrices stacked along K.) Warp 4 loads (2-stage ring), warp 5 issues the MMAs into one
// accumulator, warps 0-3 write it out once the CTA's cells are done, in its own order (lanes along a,
// so that a store is one line); two CTAs per SM, so that one loads while the other writes.
// Bound by the loads from L2: with boxes of 8 features (3072 rows of 16 bytes a stage) and stores along b
// 190 us for the six layers of 32768 cells, now 41.
struct WgradArgs {
    CUtensorMap a[kWsLayers], b[kWsLayers];
    long long M; int Nb[kWsLayers]; long long chunk;
    float *part[kWsLayers];
    int *err;
};

constexpr int kWgCells = 64, kWgStages = 2;
constexpr int kWgStageA = 128 * kWgCells * 2, kWgStageB = 256 * kWgCells * 2;
constexpr int kWgSmem = kWgStages * (kWgStageA + kWgStageB) + 256;

__global__ void __launch_bounds__(192, 2) k_mlp_wgrad(const __grid_constant__ WgradArgs g)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char *ring = sm;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + kWgStages * (kWgStageA + kWgStageB));
    uint32_t *slot = reinterpret_cast<uint32_t *>(bars + 2 * kWgStages + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, layer = blockIdx.z, Nb = g.Nb[layer];
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(kWgStages + s); };
    const uint32_t accf = bar0 + 8u * (uint32_t)(2 * kWgStages);
    const uint32_t ncols = (uint32_t)tmem_cols(Nb);
    if (warp == 4) tmem_alloc(smem_u32(slot), ncols);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kWgStages; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(accf, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot;
    const long long c_begin = (long long)blockIdx.x * g.chunk;
    const long long c_end = c_begin + g.chunk < g.M ? c_begin + g.chunk : g.M;
    const int nch = c_end > c_begin ? (int)((c_end - c_begin + kWgCells - 1) / kWgCells) : 0;
    const int a0 = (int)blockIdx.y * 128;
    const bool sw = Nb >= 64;
    const int wb = sw ? 64 : 8;                              // features of a box of Xb
    bool failed = false;
    if (warp == 4) {
        if (lane == 0) {
            const uint32_t bytes = (uint32_t)(128 + Nb) * kWgCells * 2u;
            int it = 0;
            for (; it < nch; it++) {
                const int s = it % kWgStages;
                if (!mbar_wait_bounded(empty(s), (uint32_t)(((it / kWgStages) & 1) ^ 1))) { failed = true; break; }
                mbar_expect_tx(full(s), bytes);
                const uint32_t a_s = smem_u32(ring + (size_t)s * (kWgStageA + kWgStageB));
                const uint32_t b_s = a_s + kWgStageA;
                const int y = (int)(c_begin + (long long)it * kWgCells);
                for (int q = 0; q < 2; q++) tma_load_2d(a_s + (uint32_t)q * 8192u, &g.a[layer], a0 + q * 64, y, full(s));
                for (int q = 0; q < Nb / wb; q++) tma_load_2d(b_s + (uint32_t)(q * wb) * 128u, &g.b[layer], q * wb, y, full(s));
            }
            if (failed)                                       // no copy of its own may outlive the CTA
                for (int q = it < kWgStages ? 0 : it - kWgStages; q < it; q++)
                    mbar_wait_bounded(full(q % kWgStages), (uint32_t)((q / kWgStages) & 1));
        }
    } else if (warp == 5) {
        if (lane == 0 && nch > 0) {
            const uint32_t idesc = idesc_bf16(128, Nb) | (1u << 15) | (1u << 16);      // both MN-major
            for (int it = 0; it < nch && !failed; it++) {
                const int s = it % kWgStages;
                if (!mbar_wait_bounded(full(s), (uint32_t)((it / kWgStages) & 1))) { failed = true; break; }
                tc_fence_after();
                const uint32_t a_s = smem_u32(ring + (size_t)s * (kWgStageA + kWgStageB));
                const uint32_t b_s = a_s + kWgStageA;
                // 16 cells further: two groups of eight rows; without swizzle lbo = K step (128 B), sbo = MN step (1 KB)
                for (int ks = 0; ks < kWgCells / 16; ks++)
                    mma_bf16(tmem, smem_desc_sw(a_s + (uint32_t)ks * 2048u, 8192u, 1024u),
                             sw ? smem_desc_sw(b_s + (uint32_t)ks * 2048u, 8192u, 1024u) : smem_desc(b_s + (uint32_t)ks * 256u, 128u, 1024u),
                             idesc, (it > 0 || ks > 0) ? 1u : 0u);
                mma_commit(empty(s));
            }
            if (!failed) mma_commit(accf);
        }
    } else {
        float *out = g.part[layer] + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 128 * Nb + warp * 32 + lane;
        bool ok = true;
        if (nch > 0) {
            ok = mbar_wait_warp(accf, 0u);
            tc_fence_after();
        }
        if (!ok) failed = true;
        else
            for (int c0 = 0; c0 < Nb; c0 += 16) {
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int i = 0; i < 16; i++) out[(size_t)(c0 + i) * 128] = nch > 0 ? v[i] : 0.0f;
            }
    }
    if (failed) atomicOr(g.err, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 4) tmem_dealloc(tmem, ncols);
}

// column sums of the layers' X[M x W] (W <= 256; layer = blockIdx.y): per block the sum of its rows in their
// order, two columns a thread, 32 rows asked for at a time
struct ColsumArgs {
    const bf16 *X[kWsLayers];
    int W[kWsLayers];
    float *part[kWsLayers];
    long long M, rows;
};
__global__ void __launch_bounds__(128) k_colsum_partial(ColsumArgs g)
{
    const int W = g.W[blockIdx.y], c = 2 * threadIdx.x;
    if (c >= W) return;
    const bf16 *X = g.X[blockIdx.y] + c;
    const long long r0 = (long long)blockIdx.x * g.rows, r1 = r0 + g.rows < g.M ? r0 + g.rows : g.M;
    float s0 = 0.0f, s1 = 0.0f;
    long long r = r0;
    for (; r + 32 <= r1; r += 32) {
        __nv_bfloat162 x[32];
#pragma unroll
        for (int q = 0; q < 32; q++) x[q] = *reinterpret_cast<const __nv_bfloat162 *>(X + (r + q) * W);
#pragma unroll
        for (int q = 0; q < 32; q++) { s0 += __low2float(x[q]); s1 += __high2float(x[q]); }
    }
    for (; r < r1; r++) {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162 *>(X + r * W);
        s0 += __low2float(x);
        s1 += __high2float(x);
    }
    float *dst = g.part[blockIdx.y] + (size_t)blockIdx.x * W + c;
    dst[0] = s0;
    dst[1] = s1;
}

// ---------------------------------------------------------------- features, loss, optimiser
// normalisation constants: coord min[3], max[3] (axial z, radius, pitch angle); parameter
// mean[3], std[3]; target mean[6], std[6]
__device__ __forceinline__ void ws_features(const float *nrm, float z, float r, float th, const float *pr, bf16 *out)
{
    float c[3] = {z, r, th};
#pragma unroll
    for (int d = 0; d < 3; d++) c[d] = (c[d] - nrm[d]) / (nrm[3 + d] - nrm[d]);
    int o = 0;
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
        for (int f = 0; f < 8; f++) {
            float s, co;
            sincospif((float)(1 << f) * c[d], &s, &co);
            out[o++] = __float2bfloat16_rn(s);
            out[o++] = __float2bfloat16_rn(co);
        }
#pragma unroll
    for (int d = 0; d < 3; d++) out[o++] = __float2bfloat16_rn(c[d]);
#pragma unroll
    for (int q = 0; q < 3; q++) out[o++] = __float2bfloat16_rn((pr[q] - nrm[6 + q]) / nrm[9 + q]);
    for (; o < kWsIn; o++) out[o] = __float2bfloat16_rn(0.0f);
}

// training sample layout: z, r, theta, params[3], targets[6]
constexpr int kWsSample = 12;

__device__ __forceinline__ unsigned long long mix64(unsigned long long x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__global__ void k_ws_gather(const float *set, long long n_set, unsigned long long seed, long long M, const float *nrm,
                            bf16 *X0, float *T)
{
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const long long s = (long long)(mix64(seed ^ (unsigned long long)m * 0xD1B54A32D192ED03ull) % (unsigned long long)n_set);
    const float *p = set + s * kWsSample;
    alignas(16) bf16 f[kWsIn];
    ws_features(nrm, p[0], p[1], p[2], p + 3, f);
    uint4 *dst = reinterpret_cast<uint4 *>(X0 + m * kWsIn);
#pragma unroll
    for (int q = 0; q < kWsIn / 8; q++) dst[q] = reinterpret_cast<uint4 *>(f)[q];
#pragma unroll
    for (int o = 0; o < kWsOutUsed; o++) T[m * 8 + o] = (p[6 + o] - nrm[12 + o]) / nrm[18 + o];
    T[m * 8 + 6] = 0.0f;
    T[m * 8 + 7] = 0.0f;
}

// dY = 2 (y - t) / 6 on the six used outputs (the 1 / M of the mean is applied to the gradients);
// per block, the sum of squared errors
__global__ void __launch_bounds__(256) k_ws_loss(const float *Y, const float *T, long long M, bf16 *dY, float *part)
{
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float se = 0.0f;
    if (m < M) {
        alignas(16) bf16 d[kWsOut];
#pragma unroll
        for (int o = 0; o < kWsOut; o++) {
            float g = 0.0f;
            if (o < kWsOutUsed) {
                const float e = Y[m * kWsOut + o] - T[m * 8 + o];
                se += e * e;
                g = 2.0f * e / (float)kWsOutUsed;
            }
            d[o] = __float2bfloat16_rn(g);
        }
        reinterpret_cast<uint4 *>(dY + m * kWsOut)[0] = reinterpret_cast<uint4 *>(d)[0];
        reinterpret_cast<uint4 *>(dY + m * kWsOut)[1] = reinterpret_cast<uint4 *>(d)[1];
    }
    __shared__ float sh[256];
    sh[threadIdx.x] = se;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__device__ __forceinline__ void adam(float *p, float gi, float *m, float *v, float lr, float b1, float b2, float eps, float c1, float c2)
{
    const float mi = b1 * *m + (1.0f - b1) * gi, vi = b2 * *v + (1.0f - b2) * gi * gi;
    *m = mi;
    *v = vi;
    *p -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// The end of a step in one launch: every gradient as scale * the sum of its partial sums in their order, and
// ADAM: the optimiser step and the BF16 weights, as stored [N x K] and transposed [K x N]; else: the
// gradients to G. Blocks 0 .. nw-1 take 32 x 32 weights of a layer (partials read along a, parameters along
// their rows), the last six the biases of a layer. Bound by the partials (84 MB for 32768 cells on
// 152 SMs); as 19 launches with one load in flight a thread 150 us, now 25 us.
struct StepArgs {
    float *P, *G, *Mo, *Vo;
    long long w_off[kWsLayers], b_off[kWsLayers];
    const float *part[kWsLayers], *cpart[kWsLayers];
    bf16 *Wb[kWsLayers], *Wt[kWsLayers];
    int Nb[kWsLayers], trans[kWsLayers], W[kWsLayers], first[kWsLayers + 1];       // blocks of a layer
    int gx, nb;
    float scale, lr, b1, b2, eps, c1, c2;
};
template <bool ADAM>
__global__ void __launch_bounds__(256) k_ws_step(StepArgs g)
{
    const int nw = g.first[kWsLayers];
    if ((int)blockIdx.x >= nw) {
        const int l = (int)blockIdx.x - nw, W = g.W[l], c = threadIdx.x;
        if (c >= W) return;
        const float *q = g.cpart[l] + c;
        float s = 0.0f;
        int b = 0;
        for (; b + 32 <= g.nb; b += 32) {
            float x[32];
#pragma unroll
            for (int n = 0; n < 32; n++) x[n] = q[(size_t)(b + n) * W];
#pragma unroll
            for (int n = 0; n < 32; n++) s += x[n];
        }
        for (; b < g.nb; b++) s += q[(size_t)b * W];
        const long long i = g.b_off[l] + c;
        if constexpr (ADAM) adam(g.P + i, g.scale * s, g.Mo + i, g.Vo + i, g.lr, g.b1, g.b2, g.eps, g.c1, g.c2);
        else g.G[i] = g.scale * s;
        return;
    }
    __shared__ float tile[32][33];                         // [b][a]
    int l = 0;
    while ((int)blockIdx.x >= g.first[l + 1]) l++;
    const int Nb = g.Nb[l], tb = (Nb + 31) / 32, at = ((int)blockIdx.x - g.first[l]) / tb, bt = ((int)blockIdx.x - g.first[l]) - at * tb;
    const int a = at * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    const float *q = g.part[l] + (size_t)(a >> 7) * g.gx * 128 * Nb + (a & 127);
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    bool in[4];
#pragma unroll
    for (int n = 0; n < 4; n++) in[n] = bt * 32 + w + 8 * n < Nb;
    int bx = 0;
    for (; bx + 8 <= g.gx; bx += 8) {
        float x[8][4];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int n = 0; n < 4; n++) x[u][n] = in[n] ? q[((size_t)(bx + u) * Nb + bt * 32 + w + 8 * n) * 128] : 0.0f;
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int n = 0; n < 4; n++) s[n] += x[u][n];
    }
    for (; bx < g.gx; bx++)
#pragma unroll
        for (int n = 0; n < 4; n++) s[n] += in[n] ? q[((size_t)bx * Nb + bt * 32 + w + 8 * n) * 128] : 0.0f;
#pragma unroll
    for (int n = 0; n < 4; n++) tile[w + 8 * n][threadIdx.x & 31] = s[n];
    __syncthreads();
    // the layer's matrix is [a][b], or [b][a] where it is stored transposed
    const int Wa = kWsHidden, trans = g.trans[l], K = trans ? Wa : Nb, N = trans ? Nb : Wa;
#pragma unroll
    for (int n = 0; n < 4; n++) {
        const int f = threadIdx.x & 31, r = w + 8 * n;     // along a row of the matrix, row
        const int ai = at * 32 + (trans ? f : r), bi = bt * 32 + (trans ? r : f);
        if (bi >= Nb) continue;
        float &e = tile[trans ? r : f][trans ? f : r];
        const int row = trans ? bi : ai, col = trans ? ai : bi;
        const long long i = g.w_off[l] + (long long)row * K + col;
        if constexpr (ADAM) {
            adam(g.P + i, g.scale * e, g.Mo + i, g.Vo + i, g.lr, g.b1, g.b2, g.eps, g.c1, g.c2);
            e = g.P[i];
            g.Wb[l][(size_t)row * K + col] = __float2bfloat16_rn(e);
        } else g.G[i] = g.scale * e;
    }
    if constexpr (ADAM) {
        __syncthreads();
#pragma unroll
        for (int n = 0; n < 4; n++) {
            const int f = threadIdx.x & 31, r = w + 8 * n; // along a column of the matrix, column
            const int ai = at * 32 + (trans ? r : f), bi = bt * 32 + (trans ? f : r);
            if (bi >= Nb) continue;
            const int row = trans ? bi : ai, col = trans ? ai : bi;
            g.Wt[l][(size_t)col * N + row] = __float2bfloat16_rn(tile[trans ? f : r][trans ? r : f]);
        }
    }
}

// BF16 copies of a layer's weights, as stored [N x K] and transposed [K x N]
__global__ void k_ws_weights_bf16(const float *w, int N, int K, bf16 *wb, bf16 *wt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * K) return;
    const int n = t / K, k = t - n * K;
    const bf16 b = __float2bfloat16_rn(w[t]);
    wb[t] = b;
    wt[(size_t)k * N + n] = b;
}

// n values to BF16; V = 4 values a load (x 16-byte aligned), 4 loads in flight a thread. x may be the caller's
// host memory: 262144 rows of 64 read over the link to the CPU at 200 GB/s, 0.34 ms, where a copy to
// the device takes 0.50 ms and the conversion from there 0.04.
template <int V>
__global__ void __launch_bounds__(256) k_f32_to_bf16(const float *x, long long n, bf16 *y)
{
    const long long i0 = ((long long)blockIdx.x * 1024 + threadIdx.x) * V;
    float v[4][V];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const long long i = i0 + q * 256 * V;
        if (i + V <= n) {
            if constexpr (V == 4) {
                const float4 t = *reinterpret_cast<const float4 *>(x + i);
                v[q][0] = t.x; v[q][1] = t.y; v[q][2] = t.z; v[q][3] = t.w;
            } else v[q][0] = x[i];
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const long long i = i0 + q * 256 * V;
        if (i + V > n) continue;
        alignas(8) bf16 o[V];
#pragma unroll
        for (int u = 0; u < V; u++) o[u] = __float2bfloat16_rn(v[q][u]);
        if constexpr (V == 4) *reinterpret_cast<uint2 *>(y + i) = *reinterpret_cast<uint2 *>(o);
        else y[i] = o[0];
    }
}

// ---------------------------------------------------------------- cells of a solver's fine level
// cell t of the batch: slot by bisection of the prefix counts, then (i, j, k) with k fastest
__device__ __forceinline__ int ws_cell(const Lvl *lv, const long long *off, int nslot, long long t, long long &p)
{
    int lo = 0, hi = nslot - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const Lvl L = lv[lo];
    const long long q = t - off[lo];
    const int nk = L.KM - 1, nj = L.JM - 1;
    const int k = (int)(q % nk) + 1;
    const long long r = q / nk;
    const int j = (int)(r % nj) + 1, i = (int)(r / nj) + 1;
    p = ix(L, i, j, k);
    return lo;
}

struct CellsArgs {
    const Lvl *lv; const long long *off; int nslot;
    const int *slot_case; const float *params;           // per case
    const double *cc0, *cc1, *cc2;
    double *cv0, *cv1, *cv2, *cv3, *cv4;
    const void *mut; int fp32;
};

// training samples from the current fields of cells t0 .. t0+n
__global__ void k_ws_collect(CellsArgs a, long long t0, long long n, float *out)
{
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    long long p;
    const int s = ws_cell(a.lv, a.off, a.nslot, t0 + u, p);
    const double x = a.cc0[p], y = a.cc1[p], z = a.cc2[p];
    float *o = out + u * kWsSample;
    o[0] = (float)z;
    o[1] = (float)sqrt(x * x + y * y);
    o[2] = (float)atan2(y, x);
    const float *pr = a.params + (size_t)a.slot_case[s] * kWsParams;
    o[3] = pr[0]; o[4] = pr[1]; o[5] = pr[2];
    o[6] = (float)a.cv0[p]; o[7] = (float)a.cv1[p]; o[8] = (float)a.cv2[p]; o[9] = (float)a.cv3[p]; o[10] = (float)a.cv4[p];
    o[11] = a.fp32 ? ((const float *)a.mut)[p] : (float)((const double *)a.mut)[p];
}

__global__ void k_ws_cell_features(CellsArgs a, long long t0, long long n, const float *nrm, bf16 *X0)
{
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    long long p;
    const int s = ws_cell(a.lv, a.off, a.nslot, t0 + u, p);
    const double x = a.cc0[p], y = a.cc1[p], z = a.cc2[p];
    alignas(16) bf16 f[kWsIn];
    ws_features(nrm, (float)z, (float)sqrt(x * x + y * y), (float)atan2(y, x), a.params + (size_t)a.slot_case[s] * kWsParams, f);
    uint4 *dst = reinterpret_cast<uint4 *>(X0 + u * kWsIn);
#pragma unroll
    for (int q = 0; q < kWsIn / 8; q++) dst[q] = reinterpret_cast<uint4 *>(f)[q];
}

__global__ void k_ws_write_cv(CellsArgs a, long long t0, long long n, const float *nrm, const float *Y)
{
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    long long p;
    ws_cell(a.lv, a.off, a.nslot, t0 + u, p);
    const float *y = Y + u * kWsOut;
    double q[5];
#pragma unroll
    for (int c = 0; c < 5; c++) q[c] = (double)(y[c] * nrm[18 + c] + nrm[12 + c]);
    a.cv0[p] = q[0]; a.cv1[p] = q[1]; a.cv2[p] = q[2]; a.cv3[p] = q[3]; a.cv4[p] = q[4];
}

// per block: min, max, sum, sum of squares of each of the 12 sample columns
__global__ void __launch_bounds__(256) k_ws_stats(const float *set, long long n, double *part)
{
    double mn[kWsSample], mx[kWsSample], s1[kWsSample], s2[kWsSample];
    for (int c = 0; c < kWsSample; c++) { mn[c] = 1e300; mx[c] = -1e300; s1[c] = 0.0; s2[c] = 0.0; }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < kWsSample; c++) {
            const double v = set[i * kWsSample + c];
            mn[c] = fmin(mn[c], v); mx[c] = fmax(mx[c], v); s1[c] += v; s2[c] += v * v;
        }
    __shared__ double sh[256];
    for (int c = 0; c < kWsSample; c++)
        for (int kind = 0; kind < 4; kind++) {
            double v = kind == 0 ? mn[c] : kind == 1 ? mx[c] : kind == 2 ? s1[c] : s2[c];
            sh[threadIdx.x] = v;
            __syncthreads();
            for (int w = 128; w > 0; w >>= 1) {
                if ((int)threadIdx.x < w) {
                    const double o = sh[threadIdx.x + w];
                    sh[threadIdx.x] = kind == 0 ? fmin(sh[threadIdx.x], o) : kind == 1 ? fmax(sh[threadIdx.x], o) : sh[threadIdx.x] + o;
                }
                __syncthreads();
            }
            if (threadIdx.x == 0) part[((size_t)blockIdx.x * kWsSample + c) * 4 + kind] = sh[0];
            __syncthreads();
        }
}

// ---------------------------------------------------------------- host side
// 2D tensor map of a row-major BF16 matrix [rows x cols] (row stride ld elements) read in boxes
// of 64 columns (128 bytes, in the 128-byte swizzle) x box_rows rows, or of 8 without swizzle where it has
// fewer than 64 or wide is false; rows past the end read as zeros
static CUtensorMap tensor_map_rows(const bf16 *base, long long rows, int cols, long long ld, int box_rows, bool wide = true)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        WCK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q));
        if (!f || q != cudaDriverEntryPointSuccess) throw std::runtime_error("cuTensorMapEncodeTiled is not available");
        encode = (PFN_cuTensorMapEncodeTiled_v12000)f;
    }
    wide = wide && cols >= kChunk;
    if (((uintptr_t)base & 15) || ((ld * 2) & 15) || (cols & 7) || box_rows < 1 || box_rows > 256)
        throw std::runtime_error("tensor map: misaligned matrix or box");
    CUtensorMap m;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {wide ? (cuuint32_t)kChunk : 8u, (cuuint32_t)box_rows};
    const cuuint32_t es[2] = {1u, 1u};
    const CUresult r = encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)base, dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed");
    return m;
}

static const int kN[kWsLayers] = {kWsHidden, kWsHidden, kWsHidden, kWsHidden, kWsHidden, kWsOut};
static const int kK[kWsLayers] = {kWsIn, kWsHidden, kWsHidden, kWsHidden, kWsHidden, kWsHidden};

static size_t w_off(int l)
{
    size_t o = 0;
    for (int q = 0; q < l; q++) o += (size_t)kN[q] * kK[q] + kN[q];
    return o;
}
constexpr long long kPiece = 32768;              // rows of a piece of a call on host rows (a multiple of 128)
constexpr int kLossKept = 20;                    // steps whose loss train() averages
static size_t b_off(int l) { return w_off(l) + (size_t)kN[l] * kK[l]; }

struct WarmStart::Impl {
    cudaStream_t st = nullptr, st2 = nullptr, st3 = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr, caller = nullptr, asked[3] = {}, made[2] = {};
    int n_sm = 0;
    float *P = nullptr, *G = nullptr, *Mo = nullptr, *Vo = nullptr;
    bf16 *Wb[kWsLayers] = {}, *Wt[kWsLayers] = {};
    int *err = nullptr;
    float *nrm_d = nullptr;
    float nrm[kWsNorm] = {};
    bool have_norm = false;
    int adam_t = 0;
    // rows in and out for up to cap rows, activations, targets and gradients for up to tcap
    long long cap = 0, tcap = 0;
    bf16 *X0 = nullptr, *Z[5] = {}, *H[5] = {}, *dY = nullptr, *dZ[5] = {};
    float *F = nullptr;                              // host rows on their way, where the device cannot read them
    bool host_rows = false;
    float *Y = nullptr, *T = nullptr, *part = nullptr, *cpart = nullptr, *lpart = nullptr;
    size_t part_n = 0;
    // training set
    float *set = nullptr;
    long long set_cap = 0;
    unsigned long long rng = 0;

    static bf16 *abf(long long n) { bf16 *p; WCK(cudaMalloc(&p, sizeof(bf16) * n)); return p; }
    static float *af(long long n) { float *p; WCK(cudaMalloc(&p, sizeof(float) * n)); return p; }
    void ensure(long long M)
    {
        if (M <= cap) return;
        cudaFree(X0); cudaFree(Y);
        X0 = nullptr; Y = nullptr;
        cap = 0;
        const long long n = std::max(M, (long long)4096);
        X0 = abf(n * kWsIn);
        Y = af(n * kWsOut);
        cap = n;
    }
    void ensure_train(long long M)
    {
        ensure(M);
        if (M <= tcap) return;
        release_train();
        const long long n = std::max(M, (long long)4096);
        for (int l = 0; l < 5; l++) { Z[l] = abf(n * kWsHidden); H[l] = abf(n * kWsHidden); dZ[l] = abf(n * kWsHidden); }
        dY = abf(n * kWsOut);
        T = af(n * 8);
        lpart = af(kLossKept * ((n + 255) / 256));
        if (!cpart) cpart = af(kWsLayers * 512 * kWsHidden);
        tcap = n;
    }
    void release_train()
    {
        for (int l = 0; l < 5; l++) { cudaFree(Z[l]); cudaFree(H[l]); cudaFree(dZ[l]); Z[l] = H[l] = dZ[l] = nullptr; }
        cudaFree(dY); cudaFree(T); cudaFree(lpart);
        dY = nullptr; T = lpart = nullptr;
        tcap = 0;
    }
    void release_acts()
    {
        release_train();
        cudaFree(X0); cudaFree(Y);
        X0 = nullptr; Y = nullptr;
        cap = 0;
    }

    void refresh_bf16()
    {
        for (int l = 0; l < kWsLayers; l++)
            k_ws_weights_bf16<<<(kN[l] * kK[l] + 255) / 256, 256, 0, st>>>(P + w_off(l), kN[l], kK[l], Wb[l], Wt[l]);
    }

    // Whether the device is to read the rows at feat where they are: host memory, where it reaches that through the
    // host's page tables. Rows in device or managed memory, which the host cannot look at first, and rows that are not
    // aligned are copied.
    bool in_place(const float *feat) const
    {
        cudaPointerAttributes a{};
        WCK(cudaPointerGetAttributes(&a, feat));
        return rows_in_place(feat, host_rows, a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged);
    }
    // what the caller has under way on the default stream and the streams that it waits for, which may still
    // write the rows
    void after_caller(cudaStream_t q)
    {
        WCK(cudaEventRecord(caller, cudaStreamLegacy));
        WCK(cudaStreamWaitEvent(q, caller, 0));
    }

    // features of the caller's M rows from row r0 on into X0, on stream q
    void features(const float *feat, long long r0, long long M, bool direct, cudaStream_t q)
    {
        const float *x = feat + r0 * kWsIn;
        if (direct) read_every_page(x, sizeof(float) * (size_t)M * kWsIn);
        else {
            if (!F) F = af(kPiece * kWsIn);
            WCK(cudaMemcpyAsync(F, x, sizeof(float) * (size_t)M * kWsIn, cudaMemcpyHostToDevice, q));
            x = F;
        }
        const long long n = M * kWsIn;
        if (((uintptr_t)x & 15) == 0) k_f32_to_bf16<4><<<(unsigned)((n + 4095) / 4096), 256, 0, q>>>(x, n, X0 + r0 * kWsIn);
        else k_f32_to_bf16<1><<<(unsigned)((n + 1023) / 1024), 256, 0, q>>>(x, n, X0 + r0 * kWsIn);
        WCK(cudaGetLastError());
    }

    template <int PASS>
    void chain(long long M, long long r0 = 0)
    {
        if (M <= 0) return;
        ChainArgs g{};
        g.M = M; g.Y = Y + r0 * kWsOut; g.err = err;
        for (int l = 0; l < kWsLayers; l++) g.bias[l] = P + b_off(l);
        for (int l = 0; l < kWsLayers - 1; l++) { g.Z[l] = Z[l]; g.H[l] = H[l]; g.dZ[l] = dZ[l]; }
        const bool back = PASS == PASS_BACKWARD;
        const int kx = chain_k(PASS, 0);
        const CUtensorMap tx = tensor_map_rows(back ? dY : X0 + r0 * kWsIn, M, kx, kx, 128, false);
        CUtensorMap tw[kWsLayers] = {};
        for (int l = 0; l < chain_layers(PASS); l++)
            tw[l] = tensor_map_rows(back ? Wt[kWsLayers - 1 - l] : Wb[l], chain_n(PASS, l), chain_k(PASS, l), chain_k(PASS, l), chain_n(PASS, l));
        const int grid = (int)std::min<long long>((M + 127) / 128, n_sm);
        k_mlp_chain<PASS><<<grid, 32 * (kEpiWarps + 2), chain_smem(PASS), st>>>(tx, tw[0], tw[1], tw[2], tw[3], tw[4], tw[5], g);
        WCK(cudaGetLastError());
    }
    // rows r0 .. r0 + M - 1 of X0 -> Y (inference: no activations kept)
    void infer(long long M, long long r0 = 0) { chain<PASS_INFER>(M, r0); }
    // rows of X0 -> Y and the hidden activations, which training needs
    void forward(long long M) { chain<PASS_FORWARD>(M); }

    // from dY: every gradient (mean over the M rows) into G, or with adam the optimiser step
    void backward(long long M, const StepArgs *adam = nullptr)
    {
        chain<PASS_BACKWARD>(M);
        // dW[l] = dZ^T . inputs, with 256 rows on the a side: of the last layer the transposed, H5^T . dY
        const int gy = kWsHidden / 128;
        int gx = std::max(1, n_sm / gy);
        const long long chunk = ((M + gx - 1) / gx + 63) / 64 * 64;
        gx = (int)((M + chunk - 1) / chunk);
        const int nb = (int)std::min<long long>(std::max<long long>(1, (M + 255) / 256), 512);
        size_t need = 0;
        for (int l = 0; l < kWsLayers; l++) need += (size_t)gy * gx * 128 * (l == kWsLayers - 1 ? kWsOut : kK[l]);
        if (need > part_n) {
            cudaFree(part);
            part = nullptr;
            part_n = 0;
            part = af((long long)need);
            part_n = need;
        }
        WgradArgs w{};
        ColsumArgs c{};
        StepArgs t{};
        if (adam) t = *adam;
        w.M = c.M = M; w.chunk = chunk; w.err = err;
        c.rows = (M + nb - 1) / nb;
        t.P = P; t.G = G; t.Mo = Mo; t.Vo = Vo; t.gx = gx; t.nb = nb; t.scale = 1.0f / (float)M;
        float *at = part;
        for (int l = 0; l < kWsLayers; l++) {
            const bool last = l == kWsLayers - 1;
            const bf16 *in = l == 0 ? X0 : H[l - 1], *d = last ? dY : dZ[l];
            w.Nb[l] = t.Nb[l] = last ? kWsOut : kK[l];
            w.a[l] = tensor_map_rows(last ? in : d, M, kWsHidden, kWsHidden, kWgCells);
            w.b[l] = tensor_map_rows(last ? d : in, M, w.Nb[l], w.Nb[l], kWgCells);
            w.part[l] = at;
            t.part[l] = at;
            at += (size_t)gy * gx * 128 * w.Nb[l];
            c.X[l] = d; c.W[l] = t.W[l] = kN[l];
            c.part[l] = cpart + (size_t)l * 512 * kWsHidden;
            t.cpart[l] = c.part[l];
            t.w_off[l] = (long long)w_off(l); t.b_off[l] = (long long)b_off(l);
            t.Wb[l] = Wb[l]; t.Wt[l] = Wt[l]; t.trans[l] = last;
            t.first[l + 1] = t.first[l] + kWsHidden / 32 * ((t.Nb[l] + 31) / 32);
        }
        // the column sums need no shared memory, so they run beside the weight gradients
        WCK(cudaEventRecord(fork, st));
        WCK(cudaStreamWaitEvent(st2, fork, 0));
        k_colsum_partial<<<dim3(nb, kWsLayers), 128, 0, st2>>>(c);
        k_mlp_wgrad<<<dim3(gx, gy, kWsLayers), 192, kWgSmem, st>>>(w);
        WCK(cudaEventRecord(join, st2));
        WCK(cudaStreamWaitEvent(st, join, 0));
        if (adam) k_ws_step<true><<<t.first[kWsLayers] + kWsLayers, 256, 0, st>>>(t);
        else k_ws_step<false><<<t.first[kWsLayers] + kWsLayers, 256, 0, st>>>(t);
        WCK(cudaGetLastError());
    }

    // dY of the loss; its sums per block stay in slot (step % kLossKept) until losses() reads them
    void loss(long long M, int step) { k_ws_loss<<<loss_blocks(M), 256, 0, st>>>(Y, T, M, dY, lpart + (size_t)(step % kLossKept) * loss_blocks(M)); }
    static int loss_blocks(long long M) { return (int)((M + 255) / 256); }
    // the losses of steps first .. first + n - 1, n <= kLossKept
    std::vector<float> losses(long long M, int first, int n)
    {
        const int nb = loss_blocks(M);
        std::vector<float> h((size_t)kLossKept * nb), out;
        WCK(cudaMemcpyAsync(h.data(), lpart, sizeof(float) * h.size(), cudaMemcpyDeviceToHost, st));
        WCK(cudaStreamSynchronize(st));
        for (int q = first; q < first + n; q++) {
            double s = 0.0;
            for (int b = 0; b < nb; b++) s += h[(size_t)(q % kLossKept) * nb + b];
            out.push_back((float)(s / ((double)M * kWsOutUsed)));
        }
        return out;
    }
};

size_t WarmStart::n_params() { return w_off(kWsLayers); }

WarmStart::WarmStart(unsigned seed) : d(new Impl)
{
    int dev = 0;
    WCK(cudaGetDevice(&dev));
    WCK(cudaDeviceGetAttribute(&d->n_sm, cudaDevAttrMultiProcessorCount, dev));
    WCK(cudaStreamCreateWithFlags(&d->st, cudaStreamNonBlocking));
    WCK(cudaStreamCreateWithFlags(&d->st2, cudaStreamNonBlocking));
    int reach = 0, tables = 0;
    WCK(cudaDeviceGetAttribute(&reach, cudaDevAttrPageableMemoryAccess, dev));
    WCK(cudaDeviceGetAttribute(&tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev));
    d->host_rows = reach && tables;
    WCK(cudaEventCreateWithFlags(&d->fork, cudaEventDisableTiming));
    WCK(cudaEventCreateWithFlags(&d->join, cudaEventDisableTiming));
    WCK(cudaEventCreateWithFlags(&d->caller, cudaEventDisableTiming));
    WCK(cudaStreamCreateWithFlags(&d->st3, cudaStreamNonBlocking));
    for (auto &e : d->made) WCK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto &e : d->asked) WCK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    WCK(cudaFuncSetAttribute(k_mlp_chain<PASS_INFER>, cudaFuncAttributeMaxDynamicSharedMemorySize, chain_smem(PASS_INFER)));
    WCK(cudaFuncSetAttribute(k_mlp_chain<PASS_FORWARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, chain_smem(PASS_FORWARD)));
    WCK(cudaFuncSetAttribute(k_mlp_chain<PASS_BACKWARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, chain_smem(PASS_BACKWARD)));
    WCK(cudaFuncSetAttribute(k_mlp_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem));
    const size_t np = n_params();
    WCK(cudaMalloc(&d->P, sizeof(float) * np));
    WCK(cudaMalloc(&d->G, sizeof(float) * np));
    WCK(cudaMalloc(&d->Mo, sizeof(float) * np));
    WCK(cudaMalloc(&d->Vo, sizeof(float) * np));
    WCK(cudaMemset(d->G, 0, sizeof(float) * np));
    WCK(cudaMemset(d->Mo, 0, sizeof(float) * np));
    WCK(cudaMemset(d->Vo, 0, sizeof(float) * np));
    for (int l = 0; l < kWsLayers; l++) {
        WCK(cudaMalloc(&d->Wb[l], sizeof(bf16) * kN[l] * kK[l]));
        WCK(cudaMalloc(&d->Wt[l], sizeof(bf16) * kN[l] * kK[l]));
    }
    WCK(cudaMalloc(&d->err, sizeof(int)));
    WCK(cudaMemset(d->err, 0, sizeof(int)));
    WCK(cudaMalloc(&d->nrm_d, sizeof(float) * kWsNorm));
    // Glorot-uniform weights, zero biases; the padded outputs 6..15 stay zero (their gradient is zero)
    std::mt19937 rng(seed);
    std::vector<float> h(np, 0.0f);
    for (int l = 0; l < kWsLayers; l++) {
        const float a = std::sqrt(6.0f / (float)(kK[l] + kN[l]));
        std::uniform_real_distribution<float> u(-a, a);
        for (int n = 0; n < kN[l]; n++)
            for (int k = 0; k < kK[l]; k++) {
                const float v = u(rng);
                h[w_off(l) + (size_t)n * kK[l] + k] = (l == kWsLayers - 1 && n >= kWsOutUsed) ? 0.0f : v;
            }
    }
    WCK(cudaMemcpy(d->P, h.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    d->refresh_bf16();
    d->rng = ((unsigned long long)seed << 32) ^ 0x5DEECE66Dull;
    for (int q = 0; q < kWsNorm; q++) d->nrm[q] = (q >= 3 && q < 6) || q >= 9 ? 1.0f : 0.0f;
    WCK(cudaMemcpy(d->nrm_d, d->nrm, sizeof(d->nrm), cudaMemcpyHostToDevice));
    WCK(cudaStreamSynchronize(d->st));
}

WarmStart::~WarmStart()
{
    if (!d) return;
    cudaStreamSynchronize(d->st);
    d->release_acts();
    cudaFree(d->P); cudaFree(d->G); cudaFree(d->Mo); cudaFree(d->Vo);
    for (int l = 0; l < kWsLayers; l++) { cudaFree(d->Wb[l]); cudaFree(d->Wt[l]); }
    cudaFree(d->err); cudaFree(d->nrm_d); cudaFree(d->part); cudaFree(d->cpart); cudaFree(d->set); cudaFree(d->F);
    cudaStreamDestroy(d->st);
    cudaStreamSynchronize(d->st2);
    cudaStreamDestroy(d->st2);
    cudaEventDestroy(d->fork);
    cudaEventDestroy(d->join);
    cudaEventDestroy(d->caller);
    for (auto e : d->asked) cudaEventDestroy(e);
    for (auto e : d->made) cudaEventDestroy(e);
    cudaStreamDestroy(d->st3);
    delete d;
}

int WarmStart::error_flag()
{
    int e = 0;
    WCK(cudaMemcpy(&e, d->err, sizeof(int), cudaMemcpyDeviceToHost));
    return e;
}

static CellsArgs cells_args(const FineView &v, const long long *off, const int *slot_case, const float *params)
{
    CellsArgs a{};
    a.lv = v.lv_dev; a.off = off; a.nslot = v.nslot; a.slot_case = slot_case; a.params = params;
    a.cc0 = v.cc[0]; a.cc1 = v.cc[1]; a.cc2 = v.cc[2];
    a.cv0 = v.cv[0]; a.cv1 = v.cv[1]; a.cv2 = v.cv[2]; a.cv3 = v.cv[3]; a.cv4 = v.cv[4];
    a.mut = v.mut; a.fp32 = v.fp32 ? 1 : 0;
    return a;
}

// device tables of a solver's fine cells: prefix counts per slot, slot -> case, case parameters
struct CellTables {
    DevBuf mem;
    long long *off = nullptr;
    int *slot_case = nullptr;
    float *params = nullptr;
    long long total = 0;
    CellTables(SolverBase &s, const FineView &v, const float *params_h)
    {
        std::vector<long long> off_h(v.nslot + 1, 0);
        for (int q = 0; q < v.nslot; q++)
            off_h[q + 1] = off_h[q] + (long long)(v.lv[q].IM - 1) * (v.lv[q].JM - 1) * (v.lv[q].KM - 1);
        total = off_h[v.nslot];
        std::vector<int> sc(v.nslot, 0);
        for (int c = 0; c < s.ncase; c++)
            for (int b = 0; b < s.case_nblk[c]; b++) sc[s.case_first[c] + b] = c;
        mem.bytes = sizeof(long long) * off_h.size() + 256 + sizeof(int) * sc.size() + 256 + sizeof(float) * kWsParams * s.ncase + 256;
        WCK(cudaMalloc(&mem.p, mem.bytes));
        char *q = (char *)mem.p;
        off = (long long *)q; q += (sizeof(long long) * off_h.size() + 255) & ~(size_t)255;
        slot_case = (int *)q; q += (sizeof(int) * sc.size() + 255) & ~(size_t)255;
        params = (float *)q;
        WCK(cudaMemcpy(off, off_h.data(), sizeof(long long) * off_h.size(), cudaMemcpyHostToDevice));
        WCK(cudaMemcpy(slot_case, sc.data(), sizeof(int) * sc.size(), cudaMemcpyHostToDevice));
        WCK(cudaMemcpy(params, params_h, sizeof(float) * kWsParams * s.ncase, cudaMemcpyHostToDevice));
    }
};

void WarmStart::add_solves(SolverBase &s, const float *params)
{
    WCK(cudaStreamSynchronize(s.stream));
    FineView v = s.fine_view();
    CellTables t(s, v, params);
    if (n_set + t.total > d->set_cap) {
        long long cap = std::max(n_set + t.total, 2 * d->set_cap);
        float *p;
        WCK(cudaMalloc(&p, sizeof(float) * kWsSample * cap));
        if (d->set && n_set) WCK(cudaMemcpy(p, d->set, sizeof(float) * kWsSample * n_set, cudaMemcpyDeviceToDevice));
        cudaFree(d->set);
        d->set = p;
        d->set_cap = cap;
    }
    CellsArgs a = cells_args(v, t.off, t.slot_case, t.params);
    k_ws_collect<<<(unsigned)((t.total + 255) / 256), 256, 0, d->st>>>(a, 0, t.total, d->set + n_set * kWsSample);
    WCK(cudaGetLastError());
    WCK(cudaStreamSynchronize(d->st));
    n_set += t.total;
}

float WarmStart::train(int steps, int batch, float lr)
{
    if (n_set <= 0) throw std::runtime_error("the training set is empty");
    if (batch < 128) throw std::invalid_argument("batch below 128 samples");
    Impl &m = *d;
    if (!m.have_norm) {
        const int nb = 256;
        DevBuf pb;
        pb.bytes = sizeof(double) * nb * kWsSample * 4;
        WCK(cudaMalloc(&pb.p, pb.bytes));
        k_ws_stats<<<nb, 256, 0, m.st>>>(m.set, n_set, (double *)pb.p);
        std::vector<double> h(nb * kWsSample * 4);
        WCK(cudaMemcpyAsync(h.data(), pb.p, pb.bytes, cudaMemcpyDeviceToHost, m.st));
        WCK(cudaStreamSynchronize(m.st));
        double mn[kWsSample], mx[kWsSample], s1[kWsSample], s2[kWsSample];
        for (int c = 0; c < kWsSample; c++) { mn[c] = 1e300; mx[c] = -1e300; s1[c] = s2[c] = 0.0; }
        for (int b = 0; b < nb; b++)
            for (int c = 0; c < kWsSample; c++) {
                const double *q = &h[((size_t)b * kWsSample + c) * 4];
                mn[c] = std::min(mn[c], q[0]); mx[c] = std::max(mx[c], q[1]); s1[c] += q[2]; s2[c] += q[3];
            }
        const double N = (double)n_set;
        for (int c = 0; c < 3; c++) {
            m.nrm[c] = (float)mn[c];
            m.nrm[3 + c] = (float)(mx[c] - mn[c] > 1e-12 ? mx[c] : mn[c] + 1.0);
        }
        for (int c = 0; c < 3 + kWsOutUsed; c++) {
            const double mean = s1[3 + c] / N, var = std::max(0.0, s2[3 + c] / N - mean * mean);
            const double sd = std::sqrt(var) > 1e-6 * std::max(1.0, std::fabs(mean)) ? std::sqrt(var) : 1.0;
            if (c < 3) { m.nrm[6 + c] = (float)mean; m.nrm[9 + c] = (float)sd; }
            else { m.nrm[12 + c - 3] = (float)mean; m.nrm[18 + c - 3] = (float)sd; }
        }
        WCK(cudaMemcpy(m.nrm_d, m.nrm, sizeof(m.nrm), cudaMemcpyHostToDevice));
        m.have_norm = true;
    }
    m.ensure_train(batch);
    StepArgs adam{};
    adam.lr = lr; adam.b1 = 0.9f; adam.b2 = 0.999f; adam.eps = 1e-8f;
    for (int it = 0; it < steps; it++) {
        m.rng = m.rng * 6364136223846793005ull + 1442695040888963407ull;
        k_ws_gather<<<(batch + 63) / 64, 64, 0, m.st>>>(m.set, n_set, m.rng, batch, m.nrm_d, m.X0, m.T);
        m.forward(batch);
        m.loss(batch, it);
        m.adam_t++;
        adam.c1 = 1.0f - std::pow(0.9f, (float)m.adam_t);
        adam.c2 = 1.0f - std::pow(0.999f, (float)m.adam_t);
        m.backward(batch, &adam);
    }
    const int nacc = std::max(0, std::min(steps, kLossKept));
    double acc = 0.0;
    for (float l : m.losses(batch, steps - nacc, nacc)) acc += l;
    WCK(cudaStreamSynchronize(m.st));
    WCK(cudaGetLastError());
    if (error_flag()) throw std::runtime_error("a tensor-core wait of the warm-start network ran out");
    return nacc ? (float)(acc / nacc) : 0.0f;
}

void WarmStart::apply(SolverBase &s, const float *params, int *used, double *res_warm, double *res_uniform)
{
    if (!d->have_norm) throw std::runtime_error("the network has no normalisation constants (train or set_norm first)");
    Impl &m = *d;
    s.init_uniform();
    s.save_fine_state();
    s.fill_uniform_fine({});
    s.fine_primitive();
    std::vector<double> r_uni, r_warm;
    s.fine_residual(r_uni);
    FineView v = s.fine_view();
    CellTables t(s, v, params);
    CellsArgs a = cells_args(v, t.off, t.slot_case, t.params);
    const long long chunk = 1 << 19;
    m.ensure(std::min(chunk, std::max(t.total, 1LL)));
    for (long long t0 = 0; t0 < t.total; t0 += chunk) {
        const long long n = std::min(chunk, t.total - t0);
        k_ws_cell_features<<<(unsigned)((n + 255) / 256), 256, 0, m.st>>>(a, t0, n, m.nrm_d, m.X0);
        m.infer(n);
        k_ws_write_cv<<<(unsigned)((n + 255) / 256), 256, 0, m.st>>>(a, t0, n, m.nrm_d, m.Y);
    }
    WCK(cudaStreamSynchronize(m.st));
    WCK(cudaGetLastError());
    if (error_flag()) throw std::runtime_error("a tensor-core wait of the warm-start network ran out");
    s.fine_primitive();
    s.fine_residual(r_warm);
    std::vector<int> back;
    int n_used = 0;
    for (int c = 0; c < s.ncase; c++) {
        const bool ok = std::isfinite(r_warm[c]) && r_warm[c] < r_uni[c];
        used[c] = ok ? 1 : 0;
        n_used += ok;
        if (res_warm) res_warm[c] = r_warm[c];
        if (res_uniform) res_uniform[c] = r_uni[c];
        if (!ok)
            for (int b = 0; b < s.case_nblk[c]; b++) back.push_back(s.case_first[c] + b);
    }
    if (n_used == 0) {
        s.restore_fine_state(true);              // every case on the plain start-up, as init_uniform left it
        return;
    }
    s.restore_fine_state(false);
    if (!back.empty()) {
        s.fill_uniform_fine(back);
        s.fine_primitive();
    }
    WCK(cudaStreamSynchronize(s.stream));
    s.start_from_fine_state();
}

void WarmStart::get_params(float *out)
{
    WCK(cudaStreamSynchronize(d->st));
    WCK(cudaMemcpy(out, d->P, sizeof(float) * n_params(), cudaMemcpyDeviceToHost));
}
void WarmStart::set_params(const float *in)
{
    WCK(cudaStreamSynchronize(d->st));
    WCK(cudaMemcpy(d->P, in, sizeof(float) * n_params(), cudaMemcpyHostToDevice));
    d->refresh_bf16();
    WCK(cudaStreamSynchronize(d->st));
}
void WarmStart::get_norm(float *out) const { std::memcpy(out, d->nrm, sizeof(d->nrm)); }
void WarmStart::set_norm(const float *in)
{
    std::memcpy(d->nrm, in, sizeof(d->nrm));
    WCK(cudaMemcpy(d->nrm_d, d->nrm, sizeof(d->nrm), cudaMemcpyHostToDevice));
    d->have_norm = true;
}

void WarmStart::forward(const float *feat, int M, float *y)
{
    Impl &m = *d;
    m.ensure(M);
    // nothing of the call may outlive it, also where it ends in an error: the kernels read the caller's rows
    struct Done {
        Impl &m;
        ~Done() { cudaStreamSynchronize(m.st2); cudaStreamSynchronize(m.st); cudaStreamSynchronize(m.st3); }
    } done{m};
    // Piece by piece: features on st2 up to two pieces ahead of the network on st, the copy to the caller (which
    // the host waits for) a piece behind it on st3. A caller whose y lies in its features gets one copy at the end.
    const uintptr_t fa = (uintptr_t)feat, ya = (uintptr_t)y;
    const bool apart = ya + sizeof(float) * (size_t)M * kWsOut <= fa || fa + sizeof(float) * (size_t)M * kWsIn <= ya;
    const long long np = (M + kPiece - 1) / kPiece;
    auto rows = [&](long long p) { return std::min(kPiece, M - p * kPiece); };
    const bool direct = m.in_place(feat);
    auto ask = [&](long long p) {
        if (p >= np) return;
        m.features(feat, p * kPiece, rows(p), direct, m.st2);
        WCK(cudaEventRecord(m.asked[p % 3], m.st2));
    };
    m.after_caller(np == 1 ? m.st : m.st2);
    if (np == 1) m.features(feat, 0, M, direct, m.st);
    else for (long long p = 0; p < 2; p++) ask(p);
    auto give = [&](long long p) {
        const long long o = apart ? p * kPiece * kWsOut : 0, n = apart ? rows(p) : p == np - 1 ? M : 0;
        if (n <= 0) return;
        WCK(cudaStreamWaitEvent(m.st3, m.made[p % 2], 0));
        WCK(cudaMemcpyAsync(y + o, m.Y + o, sizeof(float) * (size_t)n * kWsOut, cudaMemcpyDeviceToHost, m.st3));
    };
    for (long long p = 0; p < np; p++) {
        if (np > 1) {
            ask(p + 2);
            WCK(cudaStreamWaitEvent(m.st, m.asked[p % 3], 0));
        }
        m.infer(rows(p), p * kPiece);
        WCK(cudaEventRecord(m.made[p % 2], m.st));
        if (p > 0) give(p - 1);
    }
    give(np - 1);
    WCK(cudaStreamSynchronize(m.st3));
    if (error_flag()) throw std::runtime_error("a tensor-core wait of the warm-start network ran out");
}

float WarmStart::forward_backward(const float *feat, const float *target, int M, float *grad)
{
    Impl &m = *d;
    m.ensure_train(M);
    std::vector<float> t8((size_t)M * 8, 0.0f);
    struct Done {
        Impl &m;
        ~Done() { cudaStreamSynchronize(m.st); }
    } done{m};                                            // the kernels read the caller's rows
    const bool direct = m.in_place(feat);
    m.after_caller(m.st);
    WCK(cudaEventSynchronize(m.caller));                  // (the targets are read on the host)
    for (long long r0 = 0; r0 < M; r0 += kPiece) m.features(feat, r0, std::min<long long>(kPiece, M - r0), direct, m.st);
    for (int r = 0; r < M; r++)
        for (int o = 0; o < kWsOutUsed; o++) t8[(size_t)r * 8 + o] = target[(size_t)r * kWsOutUsed + o];
    WCK(cudaMemcpyAsync(m.T, t8.data(), sizeof(float) * t8.size(), cudaMemcpyHostToDevice, m.st));
    m.forward(M);
    m.loss(M, 0);
    m.backward(M);
    const float l = m.losses(M, 0, 1)[0];
    WCK(cudaMemcpyAsync(grad, m.G, sizeof(float) * n_params(), cudaMemcpyDeviceToHost, m.st));
    WCK(cudaStreamSynchronize(m.st));
    if (error_flag()) throw std::runtime_error("a tensor-core wait of the warm-start network ran out");
    return l;
}

__global__ void k_ws_random_rows(long long M, unsigned long long seed, bf16 *X0, float *T)
{
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    for (int c = 0; c < kWsIn; c++) {
        const unsigned long long h = mix64(seed ^ ((unsigned long long)m * kWsIn + c));
        X0[m * kWsIn + c] = __float2bfloat16_rn((float)(h >> 40) * (2.0f / 16777216.0f) - 1.0f);
    }
    for (int o = 0; o < 8; o++) {
        const unsigned long long h = mix64(~seed ^ ((unsigned long long)m * 8 + o));
        T[m * 8 + o] = o < kWsOutUsed ? (float)(h >> 40) * (2.0f / 16777216.0f) - 1.0f : 0.0f;
    }
}

void WarmStart::benchmark(long long M, int iters, float *ms_forward, float *ms_step, float *ms_infer, double *max_diff)
{
    if (M < 128 || iters < 1) throw std::invalid_argument("benchmark: at least 128 rows and one iteration");
    Impl &m = *d;
    m.ensure_train(M);
    k_ws_random_rows<<<(unsigned)((M + 255) / 256), 256, 0, m.st>>>(M, 12345ull, m.X0, m.T);
    cudaEvent_t e0, e1;
    WCK(cudaEventCreate(&e0));
    WCK(cudaEventCreate(&e1));
    m.forward(M);                                        // warm-up
    WCK(cudaEventRecord(e0, m.st));
    for (int i = 0; i < iters; i++) m.forward(M);
    WCK(cudaEventRecord(e1, m.st));
    WCK(cudaEventSynchronize(e1));
    float t = 0.f;
    WCK(cudaEventElapsedTime(&t, e0, e1));
    *ms_forward = t / iters;
    // the fused inference: timed, and its outputs against the layer-by-layer pass's (the same bits)
    std::vector<float> y_layers((size_t)M * kWsOut), y_fused((size_t)M * kWsOut);
    WCK(cudaMemcpyAsync(y_layers.data(), m.Y, sizeof(float) * y_layers.size(), cudaMemcpyDeviceToHost, m.st));
    m.infer(M);                                          // warm-up
    WCK(cudaEventRecord(e0, m.st));
    for (int i = 0; i < iters; i++) m.infer(M);
    WCK(cudaEventRecord(e1, m.st));
    WCK(cudaEventSynchronize(e1));
    WCK(cudaEventElapsedTime(&t, e0, e1));
    if (ms_infer) *ms_infer = t / iters;
    WCK(cudaMemcpyAsync(y_fused.data(), m.Y, sizeof(float) * y_fused.size(), cudaMemcpyDeviceToHost, m.st));
    WCK(cudaStreamSynchronize(m.st));
    double dmax = 0.0;
    for (size_t q = 0; q < y_fused.size(); q++) {
        const double dq = std::fabs((double)y_fused[q] - (double)y_layers[q]);
        dmax = (dq > dmax || dq != dq) ? dq : dmax;
    }
    if (max_diff) *max_diff = dmax;
    WCK(cudaEventRecord(e0, m.st));
    for (int i = 0; i < iters; i++) {
        m.forward(M);
        m.loss(M, 0);
        m.backward(M);
    }
    WCK(cudaEventRecord(e1, m.st));
    WCK(cudaEventSynchronize(e1));
    WCK(cudaEventElapsedTime(&t, e0, e1));
    *ms_step = t / iters;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (error_flag()) throw std::runtime_error("a tensor-core wait of the warm-start network ran out");
}

}  // namespace gbt
