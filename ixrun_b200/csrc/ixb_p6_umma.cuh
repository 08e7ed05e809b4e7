// Small-M GEMM on the resident P6 layout for 9..64 activation rows (batched serving, speculative verification), in one pass
// over its bytes, on the 5th-generation tensor cores: the weights go from registers into tensor memory and are the A operand of
// tcgen05.mma there, beside the accumulators.
//
//   Y[t][n] = sum_k X[t][k] * bf16(code[n][k] * scale)        t < m_tok <= NTOK
//
//   CTA      = 128 weight rows (8 row tiles, the MMA's M) x a contiguous range of column blocks; K is split over the CTAs of a
//              cluster as far as it takes to fill the chip, and the splits' sums are added in pairs, pairs of pairs and so on
//              through distributed shared memory: no scratch, no second launch, reproducible.
//   stage    = two column blocks (128 k): the packed weights of 8 row tiles arrive by one three-dimensional TMA copy (eight
//              stages ahead), the activations [tokens rounded up to 16] by one two-dimensional copy per block (four stages,
//              rows of 128 bytes, 128-byte swizzle); the converted weights are 64 columns of tensor memory (four stages).
//   warps    0..23  converters, three per row tile, every third block each (a warp reaches the 32 lanes of tensor memory of its
//                   number modulo four: two row tiles): the GEMV's conversion; the block's outliers OR-ed over their
//                   placeholders (+0.0) from an image of the lanes' registers in shared memory; one tcgen05.st of 16
//                   registers, which are the words of the block's rows in column order (p6_elem)
//            24     feeds the tensor core: eight tcgen05.mma per stage (M = 128 rows, N = tokens, K = 16)
//            25,26  ask for activations and packed weights
//            epilogue: tcgen05.ld of the accumulators by warps 0..23, outputs (or a split's sums) from there
//
// What bounds it: the conversion's instructions (66 per 1024 weights and lane, about 130 with outliers and hand-over); the rows
// cost next to nothing (17408 x 5120: 25.5 us at 16 rows, 26.8 at 64; k_p6_rows beside it 26.9 and 48.9).  Without the conversion it
// takes 16.0 us, HBM alone would take 10.5.  How it came there, on that layer at 64 rows: mma.sync with the weights in registers
// (k_p6_rows) 48.6, bound by its rate of 540 TFLOP/s and a barrier per block; the weights through shared memory to tcgen05 59.7, by
// the hand-over; weights in tensor memory 35.3, by the chain of instructions of the one thread that issues the MMAs (hence uniform
// addresses, unrolled slots, two blocks per hand-over); activations by cp.async 39 to 52 (16-byte pieces of core matrices are half a
// sector each), by TMA 30.3; packed weights by TMA instead of registers, so that the loads of outliers and weights wait for nobody,
// 25.4 (by eight one-dimensional bulk copies a stage 27.5).  That chain of instructions still counts: the vote on the waits of
// a stage is the cheapest form of them (17408 x 5120 at 16 rows 25.5; without it 26.7, with the MMAs predicated on them 28.7).
//
// Every wait on an mbarrier is bounded, and no thread begins one that depends on the activations before the kernel ahead is
// complete: such a wait counts this CTA's own copies, conversions and MMAs only, however long that kernel takes.  A thread whose
// wait gave up asks for nothing more; the loaders then wait (bounded too) for the copies that they did ask for and every thread for
// the MMAs that were issued, so that nothing lands in memory that has got another use; the CTA's outputs become NaN, and the
// kernel carries on to its end, so tensor memory is always released.
#pragma once
#include <cuda.h>
#include "ixb_gemm_tc.cuh"
#include "ixb_p6.cuh"
#include "ixb_p6_rows.cuh"

namespace ixb {

constexpr int kPuTiles = 8;                              // row tiles per CTA
constexpr int kPuRows = kPuTiles * kTileRows;            // 128, the MMA's M
constexpr int kPuMaxRows = 64;
constexpr int kPuMaxSplits = 16;                         // CTAs of a cluster (above 8 by opt-in)
constexpr int kPuPhases = 3;                             // converter warps per row tile
constexpr int kPuConv = kPuTiles * kPuPhases;            // warps 0..23
constexpr int kPuMmaWarp = kPuConv;                      // 24
constexpr int kPuLoadWarp = kPuMmaWarp + 1;              // 25
constexpr int kPuWLoadWarp = kPuLoadWarp + 1;            // 26
constexpr int kPuWarps = kPuWLoadWarp + 1;
constexpr int kPuThreads = kPuWarps * 32;                // 864
constexpr uint32_t kPuWaitLimit = 1u << 20;               // polls
constexpr uint32_t kPuTmemCols = 512;                    // all of it: 256 columns of accumulators, 256 of weights
constexpr uint32_t kPuStages = 4;                        // of two column blocks: 64 columns of tensor memory each, and their activations
constexpr uint32_t kPuWStages = 2 * kPuStages;           // ... of packed weights in shared memory
constexpr uint32_t kPuWStage = kPuTiles * 2 * kP6BlockBytes;       // 12288 bytes
constexpr int kPuRedPitch = kPuRows + 4;                 // floats of one token in a split's sums
constexpr int32_t kPuEntries = 128;                      // outlier entries of its run that a converter warp stages

// Column block b adds into accumulator b % pu_accs: the tensor core cuts the low bits of what it adds to a large sum, so many
// short chains lose less than one long one.  They are joined in pairs for the same reason: 2-norm error of fp32 outputs against 64
// bits, one after the other / in pairs, 300 x 16384 (16 splits) 0.86e-7 / 0.65e-7, 2048 x 6144 with 16 rows 0.60e-7 / 0.55e-7.
__host__ __device__ __forceinline__ uint32_t pu_accs(uint32_t n_pad)
{
    const uint32_t n = 256u / n_pad;
    return n < 8u ? n : 8u;
}
template <int NTOK>
struct PuCfg {
    static constexpr uint32_t kXBlk = NTOK * kTileCols * 2;                        // one column block's activations: rows of 128 bytes
    static constexpr uint32_t kWOff = kPuStages * 2 * kXBlk;
    static constexpr uint32_t kImgOff = kWOff + kPuWStages * kPuWStage;
    static constexpr uint32_t kEntOff = kImgOff + kPuConv * 2048;
    static constexpr uint32_t kBarOff = kEntOff + kPuConv * kPuEntries * 4;
    static constexpr uint32_t kBars = 2 * kPuStages + 2 * kPuWStages + 1;
    static constexpr uint32_t kRed = NTOK * kPuRedPitch * 4;                       // a split's sums [token][128 rows], over the rest
    static constexpr uint32_t kSmem = kBarOff + kBars * 8 + 16 + 1024;             // (the stages start on 1024 bytes)
    static_assert(kXBlk % 1024 == 0 && kBarOff % 8 == 0 && kRed <= kBarOff && kSmem <= 227 * 1024, "alignment and size");
};

__device__ __forceinline__ uint32_t pu_idesc(uint32_t n_pad)       // kind::f16, bf16 x bf16 -> fp32, both K-major, M = 128
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n_pad >> 3) << 17) | ((uint32_t)(kPuRows >> 4) << 24);
}
__device__ __forceinline__ bool pu_wait(uint32_t mbar, uint32_t parity)
{
    for (uint32_t it = 0; it < kPuWaitLimit; ++it) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void pu_arrive(uint32_t mbar)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ uint32_t pu_elect()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(e));
    return e;
}
// by the elected lane of a converged warp: D[128 x N] (+)= A[128 x 16] (tensor memory) * B[N x 16]^T (shared memory)
__device__ __forceinline__ void pu_mma(uint32_t el, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(el) : "memory");
}
__device__ __forceinline__ void pu_commit(uint32_t el, uint32_t mbar)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar), "r"(el) : "memory");
}
// grid: row groups x splits, split index fastest; a cluster is one row group's splits
template <int NTOK>
__global__ void __launch_bounds__(kPuThreads, 1)
k_p6_umma(P6 p, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, uint32_t m_tok, const __nv_bfloat16 *__restrict__ bias, void *y, int y_f32,
          uint32_t splits)
{
    using CF = PuCfg<NTOK>;
    extern __shared__ __align__(1024) unsigned char pu_smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    unsigned char *pu_smem = pu_smem_raw + ((1024u - ((uint32_t)__cvta_generic_to_shared(pu_smem_raw) & 1023u)) & 1023u);
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(pu_smem);
    // barriers: packed weights there, activations there, weights converted, stage done, all done
    const uint32_t wfull0 = smem0 + CF::kBarOff, xfull0 = wfull0 + kPuWStages * 8u, full0 = xfull0 + kPuStages * 8u,
                   empty0 = full0 + kPuWStages * 8u, done_bar = empty0 + kPuStages * 8u;
    uint32_t *tmem_slot = (uint32_t *)(pu_smem + CF::kBarOff + CF::kBars * 8);
    volatile uint32_t *failed = tmem_slot + 1;

    const uint32_t group = blockIdx.x / splits, split = blockIdx.x - group * splits;
    const uint32_t KB = p.kb;
    const uint32_t kq = KB / splits, kr = KB - kq * splits;
    const uint32_t kb0 = p6_begin(split, kq, kr), nk = p6_begin(split + 1, kq, kr) - kb0;    // column blocks
    const uint32_t ns = (nk + 1u) / 2u;                                                       // stages
    const uint32_t n_pad = (m_tok + 15u) & ~15u;
    asm volatile("griddepcontrol.launch_dependents;");

    const uint32_t quarter = (uint32_t)warp & 3u, cidx = (uint32_t)warp;
    const uint32_t tile = 2u * quarter + (cidx >> 2 & 1u), phase = cidx >> 3;      // (of a converter)
    const uint32_t R = group * kPuTiles + tile;
    const bool conv = warp < kPuConv, have = conv && R < p.rt;                      // (warp uniform) no such tile: arrivals only
    const uint32_t b_first = (have ? R : 0u) * KB + kb0;
    const uint32_t img_s = smem0 + CF::kImgOff + cidx * 2048u, ent_s = smem0 + CF::kEntOff + cidx * kPuEntries * 4u;
    int32_t ent0 = 0;
    if (have) {
        // the run's first outlier entries, from the 16-byte boundary at or below the first one
        const int32_t ent1 = __ldg(p.blk_off + b_first + nk);
        ent0 = __ldg(p.blk_off + b_first) & ~3;
        if (ent0 + lane * 4 < ent1) p6_cp16(ent_s + lane * 16, p.esc + ent0 + lane * 4);
        cp_async_commit();
#pragma unroll
        for (int q = 0; q < 4; ++q)
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(img_s + (q * 32 + lane) * 16), "r"(0u) : "memory");
    }
    // packed weights of stage i, two blocks of eight row tiles in one copy (they do not depend on the kernel ahead; what lies
    // beyond the tensor arrives as zeros, and is not looked at)
    auto load_w = [&](uint32_t i) {
        const uint32_t s = i & (kPuWStages - 1u), bar = wfull0 + 8u * s;
        if (lane == 0) {
            asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(kPuWStage) : "memory");
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                         :: "r"(smem0 + CF::kWOff + s * kPuWStage), "l"(&wmap), "r"(0), "r"(kb0 + 2u * i), "r"(group * kPuTiles), "r"(bar) : "memory");
        }
        __syncwarp();
    };
    if (warp == kPuWLoadWarp) {
        if (lane == 0) {
            auto init = [&](uint32_t bar, uint32_t n, uint32_t count) {
                for (uint32_t i = 0; i < n; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8u * i), "r"(count) : "memory");
            };
            init(wfull0, kPuWStages, 1u);
            init(xfull0, kPuStages, 1u);
            init(full0, kPuWStages, 2u * kPuTiles);
            init(empty0, kPuStages, 1u);
            init(done_bar, 1u, 1u);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            *failed = 0u;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
        }
        __syncwarp();
        for (uint32_t i = 0; i < kPuWStages && i < ns; ++i) load_w(i);
    }
    if (warp == kPuMmaWarp) {
        const uint32_t slot_addr = (uint32_t)__cvta_generic_to_shared(tmem_slot);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(kPuTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0), tmem_a = tmem + 256u;
    bool ok = true;

    if (warp == kPuLoadWarp) {
        // ---- the activations of a stage (rows and columns beyond x arrive as zeros; rows of 128 bytes, their 16-byte pieces
        // swizzled) as soon as the stage four before it is done
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t i = 0;
        for (; i < ns; ++i) {
            const uint32_t s = i & (kPuStages - 1u), bar = xfull0 + 8u * s, n = min(2u, nk - 2u * i);
            ok = ok && pu_wait(empty0 + 8u * s, (i / kPuStages & 1u) ^ 1u);
            if (__any_sync(0xffffffffu, !ok)) break;
            if (lane == 0) {
                asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(n * n_pad * 128u) : "memory");
                for (uint32_t h = 0; h < n; ++h)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 :: "r"(smem0 + (2u * s + h) * CF::kXBlk), "l"(&xmap), "r"((kb0 + 2u * i + h) * kTileCols), "r"(0), "r"(bar) : "memory");
            }
            __syncwarp();
        }
        // the copies that may still be in flight (the tensor core's warp waits for them too, unless it gave up)
        bool landed = true;
        for (uint32_t j = i > kPuStages ? i - kPuStages : 0u; j < i; ++j)
            landed = pu_wait(xfull0 + 8u * (j & (kPuStages - 1u)), j / kPuStages & 1u) && landed;
        ok = ok && landed;
    } else if (warp == kPuWLoadWarp) {
        // ---- the packed weights of a stage as soon as those of the stage eight before it are converted (the barriers of converted
        // weights are as many as the slots of packed ones: a warp that runs behind by a whole round is never waited past)
        uint32_t i = 0;
        for (; i + kPuWStages < ns; ++i) {
            // (from the fifth stage on the converters wait for the tensor core, and that for activations)
            if (i == kPuStages) asm volatile("griddepcontrol.wait;" ::: "memory");
            ok = ok && pu_wait(full0 + 8u * (i & (kPuWStages - 1u)), i / kPuWStages & 1u);
            if (__any_sync(0xffffffffu, !ok)) break;
            load_w(i + kPuWStages);
        }
        bool landed = true;                                            // as above
        for (uint32_t j = i, end = min(ns, i + kPuWStages); j < end; ++j)
            landed = pu_wait(wfull0 + 8u * (j & (kPuWStages - 1u)), j / kPuWStages & 1u) && landed;
        ok = ok && landed;
    } else if (warp == kPuMmaWarp) {
        // ---- the warp that feeds the tensor core; its addresses and descriptors are uniform, slots unrolled, because a stage
        // takes as long as this warp's chain of instructions if that is long.  (Tokens m_tok .. n_pad - 1 of a stage are whatever
        // lies there: their sums are not looked at.)
        const uint32_t idesc = pu_idesc(n_pad), el = pu_elect(), accs = pu_accs(n_pad);
        uint32_t d = tmem;                                              // the accumulator of the next block
        const uint64_t dx0 = umma_desc(smem0, 16u, 1024u) | 2ull << 61;     // eight rows of 128 bytes, 128-byte swizzle
        asm volatile("griddepcontrol.wait;" ::: "memory");             // (a wait for activations is not one for the kernel ahead)
        for (uint32_t i0 = 0; i0 < ns && ok; i0 += kPuWStages) {
            const uint32_t par = i0 / kPuWStages & 1u;
#pragma unroll
            for (uint32_t ws = 0; ws < kPuWStages; ++ws) {
                const uint32_t st = ws % kPuStages;
                if (i0 + ws >= ns) break;
                ok = ok && pu_wait(xfull0 + 8u * st, ws / kPuStages & 1u);            // (two rounds of these to one of the weights')
                ok = ok && pu_wait(full0 + 8u * ws, par);
                ok = __all_sync(0xffffffffu, ok);                       // (also: no lane falls a phase behind the one that issues)
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (uint32_t h = 0; h < 2u; ++h) {
                    if (2u * (i0 + ws) + h >= nk) break;
                    const uint32_t blk = 2u * st + h, first = 2u * (i0 + ws) + h < accs ? 1u : 0u;
#pragma unroll
                    for (uint32_t k = 0; k < kTileCols / 16; ++k)
                        pu_mma(el, d, tmem_a + blk * 32u + 8u * k,
                               dx0 + ((blk * CF::kXBlk + 32u * k) >> 4), idesc, k ? 1u : 1u - first);
                    d = d + n_pad == tmem + accs * n_pad ? tmem : d + n_pad;
                }
                pu_commit(el, empty0 + 8u * st);
            }
        }
        pu_commit(el, done_bar);
    } else {
        // ---- converters: warp (tile, phase) converts the blocks phase, phase + 3, ... of its row tile
        uint32_t e2;
        const uint32_t s2 = p6_scale2(p.scale[(have ? R : 0u) * p.scale_stride]);
        asm volatile("mov.b32 %0, 0x43004300;" : "=r"(e2));
        const uint32_t dst = tmem_a + ((32u * quarter + 16u * (tile & 1u)) << 16);
        // lane l keeps blk_off[b_first + win + l] and the 32 offsets after the next 30 blocks
        uint32_t win = phase;
        auto offsets = [&](uint32_t b) { return have ? __ldg(p.blk_off + b_first + min(b + (uint32_t)lane, nk)) : 0; };
        int32_t off_l = offsets(win), off_n = offsets(win + 30u);
        cp_async_wait<0>();                                            // the staged entries
        __syncwarp();
        // (with an odd number of blocks the last stage's second half is arrivals only)
        for (uint32_t i = phase; i < 2u * ns; i += kPuPhases) {
            const uint32_t slot = i / 2u & (kPuStages - 1u), ws = i / 2u & (kPuWStages - 1u);
            const bool work = have && i < nk;                          // warp uniform
            uint32_t f[16];
            if (work) {
                if (i >= win + 30u) {                                  // (warp uniform)
                    win += 30u;
                    off_l = off_n;
                    off_n = offsets(win + 30u);
                }
                const int32_t lo = __shfl_sync(0xffffffffu, off_l, (int)(i - win)), hi = __shfl_sync(0xffffffffu, off_l, (int)(i + 1u - win));
                const int32_t at = lo + lane;
                const uint32_t src = smem0 + CF::kWOff + ws * kPuWStage + (2u * tile + (i & 1u)) * kP6BlockBytes;
                if (lo == hi) {                                        // warp uniform
                    ok = ok && pu_wait(wfull0 + 8u * ws, i / (2u * kPuWStages) & 1u);
                    const uint4 a = p6_lds128(src + lane * 16);
                    const uint2 a2 = p6_lds64(src + 512 + lane * 8);
                    const uint32_t w[6] = {a.x, a.y, a.z, a.w, a2.x, a2.y};
                    p6_unpack(w, e2, s2, f);
                } else {
                    // the block's outliers into an image of the lanes' registers in shared memory, and from there over their
                    // placeholders (+0.0)
                    auto put = [&](uint32_t where, uint32_t v) {
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(where), "h"((unsigned short)v) : "memory");
                    };
                    uint32_t where = 0;
                    if (at < hi) {
                        const uint32_t e = at < ent0 + kPuEntries ? p6_lds32(ent_s + (uint32_t)(at - ent0) * 4u) : __ldg(p.esc + at);
                        where = img_s + p6_image_at(e);
                        put(where, e >> 16);
                    }
                    for (int32_t j = at + 32; j < hi; j += 32) {       // rare: more than 32 in a block
                        const uint32_t e = __ldg(p.esc + j);
                        put(img_s + p6_image_at(e), e >> 16);
                    }
                    __syncwarp();
                    uint4 v[4];                                        // (requested before the wait for the weights)
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = p6_lds128(img_s + (q * 32 + lane) * 16);
                    ok = ok && pu_wait(wfull0 + 8u * ws, i / (2u * kPuWStages) & 1u);
                    const uint4 a = p6_lds128(src + lane * 16);
                    const uint2 a2 = p6_lds64(src + 512 + lane * 8);
                    const uint32_t w[6] = {a.x, a.y, a.z, a.w, a2.x, a2.y};
                    p6_unpack(w, e2, s2, f);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        f[4 * q] |= v[q].x;
                        f[4 * q + 1] |= v[q].y;
                        f[4 * q + 2] |= v[q].z;
                        f[4 * q + 3] |= v[q].w;
                    }
                    __syncwarp();
                    if (at < hi) put(where, 0);
                    for (int32_t j = at + 32; j < hi; j += 32) put(img_s + p6_image_at(__ldg(p.esc + j)), 0);
                }
            }
            // (the first wait for the tensor core, and so for activations)
            if (i >= 2u * kPuStages && i < 2u * kPuStages + kPuPhases) asm volatile("griddepcontrol.wait;" ::: "memory");
            ok = ok && pu_wait(empty0 + 8u * slot, (i / (2u * kPuStages) & 1u) ^ 1u);  // the slot's last reader (the tensor core) is done
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            __syncwarp();
            if (work) {                                                // register 4 j + 2 h + v: row g + 8 h of the tile, word 8 j + 2 t + v of the block's 32
                asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                             :: "r"(dst + (i & (2u * kPuStages - 1u)) * 32u), "r"(f[0]), "r"(f[2]), "r"(f[1]), "r"(f[3]), "r"(f[4]), "r"(f[6]), "r"(f[5]),
                                "r"(f[7]), "r"(f[8]), "r"(f[10]), "r"(f[9]), "r"(f[11]), "r"(f[12]), "r"(f[14]), "r"(f[13]), "r"(f[15]) : "memory");
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) pu_arrive(full0 + 8u * ws);
        }
    }
    __syncwarp();
    // (also: the kernels ahead may still read what y held)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    ok = pu_wait(done_bar, 0u) && ok;                                   // (the MMAs that were issued are done, whoever gave up)
    if (!ok) *failed = 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();                                                    // nobody uses the stages and the rings any more
    const bool bad = *failed != 0u;
    float *red = (float *)pu_smem;                                      // [token][kPuRedPitch]
    auto put = [&](uint32_t m, uint32_t r, float v) {
        const uint32_t row = group * kPuRows + r;
        if (row >= p.out_f) return;
        const size_t o = (size_t)m * p.out_f + row;
        if (y_f32) {
            ((float *)y)[o] = bias ? v + __bfloat162float(bias[row]) : v;
        } else {
            __nv_bfloat16 hv = __float2bfloat16_rn(v);
            if (bias) hv = __hadd(hv, bias[row]);
            ((__nv_bfloat16 *)y)[o] = hv;
        }
    };
    // warp: its quarter of the rows (lane = row), every sixth run of eight tokens
    const uint32_t r0 = 32u * quarter + (uint32_t)lane;
    for (uint32_t c0 = ((uint32_t)warp >> 2) * 8u; warp < kPuConv && c0 < m_tok; c0 += (kPuConv / 4) * 8u) {
        // the accumulators in pairs, pairs of pairs and so on (one without a block was never written: zero)
        const uint32_t accs = min(nk, pu_accs(n_pad));
        auto load = [&](uint32_t q, uint32_t (&r)[8]) {
            if (q < accs) {                                             // (uniform)
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                             : "r"(tmem + ((32u * quarter) << 16) + q * n_pad + c0) : "memory");
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) r[j] = 0u;
            }
        };
        float v[8], four[8];
#pragma unroll
        for (uint32_t q = 0; q < 8u; q += 2u) {
            if (q >= 4u && q >= accs) break;
            uint32_t a[8], b[8];
            load(q, a);
            load(q + 1u, b);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                asm volatile("" : "+r"(a[j]), "+r"(b[j]));              // (not before the wait)
                const float two = __uint_as_float(a[j]) + __uint_as_float(b[j]);
                if (q == 0u) v[j] = two;
                else if (q == 4u) four[j] = two;
                else if (q == 2u) v[j] += two;
                else four[j] += two;
            }
        }
        if (accs > 4u) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += four[j];
        }
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            if (bad) v[j] = __int_as_float(0x7fc00000);
            if (c0 + j >= m_tok) continue;
            if (splits == 1u) put(c0 + j, r0, v[j]);
            else red[(c0 + j) * kPuRedPitch + r0] = v[j];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (splits > 1u) {
        pr_cluster_sync();
        for (uint32_t i = split * (uint32_t)kPuThreads + tid; i < m_tok * kPuRows; i += splits * (uint32_t)kPuThreads) {
            const uint32_t m = i / kPuRows, r = i % kPuRows, a = smem0 + (m * kPuRedPitch + r) * 4u;
            // the splits in pairs, pairs of pairs and so on (uniform branches: most launches have two to six)
            auto quad = [&](uint32_t c) {
                const float v0 = pr_ld_cluster(a, c), v1 = c + 1u < splits ? pr_ld_cluster(a, c + 1u) : 0.f;
                if (c + 2u >= splits) return v0 + v1;
                const float v2 = pr_ld_cluster(a, c + 2u), v3 = c + 3u < splits ? pr_ld_cluster(a, c + 3u) : 0.f;
                return (v0 + v1) + (v2 + v3);
            };
            float v = quad(0u);
            if (splits > 4u) v += quad(4u);
            if (splits > 8u) {
                float w = quad(8u);
                if (splits > 12u) w += quad(12u);
                v += w;
            }
            put(m, r, v);
        }
        pr_cluster_sync();                             // no CTA leaves while another reads its sums
    } else {
        __syncthreads();
    }
    if (warp == kPuMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPuTmemCols) : "memory");
}

}  // namespace ixb
