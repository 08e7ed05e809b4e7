// Small-M GEMM on the resident P6 layout on mma.sync, for 9..24 activation rows of layers with several outliers per block (the
// other calls of 9..64 rows are k_p6_umma's, ixb_p6_umma.cuh).
//
//   Y[m][n] = sum_k X[m][k] * bf16(code[n][k] * scale)        m < m_rows <= 24
//
// The reference runs this case as decode -> bf16 weight in HBM -> dense matmul (ixrun/engine.py:171-173; structural
// precedent for a fused kernel: ixrun/tpab_gemm.py:34-94).  Here the weights become the A operands of mma.sync in
// registers, as in the GEMV (k_p6_mma).
//
// What bounds it: 6.05 bits of HBM per weight and four instructions per pair of weights for the conversion (six where the
// field is split), the same as the GEMV; on top of that one mma per 16 x 16 weights and eight rows, and a barrier of four warps
// per block: 17408 x 5120 with 16 rows 26.2 us.  Its steps have slack for a block's outliers, which k_p6_umma's converters lack
// (8 per block: 29.5 and 32.3 us).
//
// CTA  = 8 row tiles (128 weight rows) x a contiguous range of column blocks; K is split over the CTAs of a cluster as
//        far as it takes to fill the chip, and the splits' sums are added in rank order through distributed shared memory.
// warp = two row tiles (so that an activation operand read from shared memory serves two mmas) x one of PARTS contiguous
//        parts of the CTA's columns; a part is four warps that share the activations of its current column block.
// step = one column block of every part: its activations and the warps' own plane blocks and outlier entries arrive by
//        cp.async in STAGES slots; the four warps of a part meet at a named barrier once per step.
// The block's outliers are written into a zeroed image of the lanes' A registers and OR-ed over their placeholders
// (+0.0), so their cost does not grow with the rows.  Sums: fp32, parts in order, then splits in order: reproducible.
#pragma once
#include "ixb_p6.cuh"

namespace ixb {

constexpr int kPrMaxRows = 24;
constexpr int kPrTiles = 8;                              // row tiles per CTA
constexpr int kPrRows = kPrTiles * kTileRows;            // 128
constexpr uint32_t kPrXPitch = kTileCols * 2 + 32;       // bytes of one activation row in a stage: 8-byte reads without conflicts
constexpr int kPrRedPitch = kPrRows + 4;                 // floats of one token in the sums: conflict free from the C fragments

template <int NT, int PARTS, int STAGES>
struct PrSmem {
    static constexpr uint32_t kX = NT * 8 * kPrXPitch;                             // activations of one part's column block
    static constexpr uint32_t kBlk = 2 * (kP6BlockBytes + 128);                    // a warp's two blocks and 32 + 32 entries
    static constexpr uint32_t kWarps = PARTS * 4;
    static constexpr uint32_t kXOff = 0, kBlkOff = kXOff + STAGES * PARTS * kX;
    static constexpr uint32_t kImgOff = kBlkOff + STAGES * kWarps * kBlk;
    static constexpr uint32_t kRed = NT * 8 * kPrRedPitch * 4;                     // one part's sums (over the ring, at the end)
    static constexpr uint32_t kRing = kImgOff + kWarps * 2048;
    static constexpr uint32_t kBytes = kRing > PARTS * kRed ? kRing : PARTS * kRed;
    static_assert(kX % 16 == 0 && kBlk % 16 == 0 && kBytes <= 227 * 1024, "alignment and size");
};

__device__ __forceinline__ void pr_cp4_if(uint32_t dst, const void *src, bool on)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.ca.shared.global [%0], [%1], 4;\n\t}"
                 ::"r"(dst), "l"(src), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ float pr_ld_cluster(uint32_t addr, uint32_t rank)
{
    float v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
                 : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}
__device__ __forceinline__ void pr_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// grid: row groups x splits, split index fastest; a cluster is one row group's splits
template <int NT, int PARTS, int STAGES>
__global__ void __launch_bounds__(PARTS * 128, 1)
k_p6_rows(P6 p, const __nv_bfloat16 *__restrict__ x, uint32_t m_rows, const __nv_bfloat16 *__restrict__ bias, void *y,
          int y_f32, uint32_t splits)
{
    using SM = PrSmem<NT, PARTS, STAGES>;
    extern __shared__ __align__(128) unsigned char pr_smem[];
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(pr_smem);
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t part = (uint32_t)wid >> 2, pair = (uint32_t)wid & 3u;
    const uint32_t group = blockIdx.x / splits, split = blockIdx.x - group * splits;
    const uint32_t KB = p.kb;
    const uint32_t kq = KB / splits, kr = KB - kq * splits;
    const uint32_t kb0 = p6_begin(split, kq, kr), nk = p6_begin(split + 1, kq, kr) - kb0;
    const uint32_t pq = nk / PARTS, prm = nk - pq * PARTS;
    const uint32_t c0 = kb0 + p6_begin(part, pq, prm), steps = p6_begin(part + 1, pq, prm) - p6_begin(part, pq, prm);
    const uint32_t tile0 = group * kPrTiles + pair * 2u;               // this warp's row tiles tile0, tile0 + 1
    const bool have[2] = {tile0 < p.rt, tile0 + 1u < p.rt};            // warp uniform
    const uint32_t blk[2] = {(have[0] ? tile0 : 0u) * KB + c0, (have[1] ? tile0 + 1u : 0u) * KB + c0};

    asm volatile("griddepcontrol.launch_dependents;");
    // ---- outlier bookkeeping: lane l keeps blk_off[blk + win + l] of both tiles
    uint32_t win = 0;
    int32_t off_l[2];
    auto load_window = [&](uint32_t s) {
        win = s;
#pragma unroll
        for (int i = 0; i < 2; ++i) off_l[i] = __ldg(p.blk_off + blk[i] + min(s + (uint32_t)lane, steps));
    };
    load_window(0);
    auto slot_of = [&](uint32_t s) { return s % STAGES; };
    const uint32_t my_blk = smem0 + SM::kBlkOff + wid * SM::kBlk;      // + slot * kWarps * kBlk
    auto fetch_blocks = [&](uint32_t s) {                              // plane blocks and entries of step s < steps
        const uint32_t dst = my_blk + slot_of(s) * (SM::kWarps * SM::kBlk);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned char *src = p.plane + (size_t)(blk[i] + s) * kP6BlockBytes + lane * 16;
            const uint32_t d = dst + i * (kP6BlockBytes + 128);
            p6_cp16_if(d + lane * 16, src, have[i]);
            p6_cp16_if(d + lane * 16 + 512, src + 512, have[i] && lane < 16);
            const int32_t lo = __shfl_sync(0xffffffffu, off_l[i], (int)(s - win)), hi = __shfl_sync(0xffffffffu, off_l[i], (int)(s + 1u - win));
            pr_cp4_if(d + kP6BlockBytes + lane * 4, p.esc + lo + lane, have[i] && lo + lane < hi);
        }
    };
    const uint32_t xpart = smem0 + SM::kXOff + part * SM::kX;          // + slot * PARTS * kX
    auto fetch_x = [&](uint32_t s) {                                   // the part's four warps together
        const uint32_t dst = xpart + slot_of(s) * (PARTS * SM::kX);
        const uint32_t col = (c0 + s) * kTileCols;
        for (uint32_t c = tid & 127u; c < m_rows * 8u; c += 128u) {
            const uint32_t m = c >> 3, k8 = (c & 7u) * 8u;
            const uint32_t d = dst + m * kPrXPitch + k8 * 2u;
            if (col + k8 < p.in_f) p6_cp16(d, x + (size_t)m * p.in_f + col + k8);      // in_f % 8 == 0: whole pieces
            else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(d), "r"(0u) : "memory");
        }
    };
    // the weights of the first steps do not depend on the kernel ahead in the stream
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if ((uint32_t)s < steps) fetch_blocks(s);
    unsigned char *img = pr_smem + SM::kImgOff + wid * 2048;
#pragma unroll
    for (int q = 0; q < 4; ++q) ((uint4 *)img)[q * 32 + lane] = make_uint4(0, 0, 0, 0);
    const uint32_t img_s = (uint32_t)__cvta_generic_to_shared(img);
    uint32_t s2[2], e2;
    asm volatile("mov.b32 %0, 0x43004300;" : "=r"(e2));
#pragma unroll
    for (int i = 0; i < 2; ++i) s2[i] = p6_scale2(p.scale[(have[i] ? tile0 + i : 0u) * p.scale_stride]);
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if ((uint32_t)s < steps) fetch_x(s);
        cp_async_commit();                             // (the first group also holds all of the blocks above)
    }
    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[i][n][0] = acc[i][n][1] = acc[i][n][2] = acc[i][n][3] = 0.f;
    const uint32_t xl = (uint32_t)g * kPrXPitch + 8u * t;              // this lane's activations of row g, 4 of every 16: + 8 n rows
    for (uint32_t s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();                   // step s has landed for this thread ...
        asm volatile("bar.sync %0, 128;" ::"r"(part + 1u) : "memory");   // ... and for the part, which is done with step s - 1
        const uint32_t nxt = s + STAGES - 1;
        if (nxt < steps) {
            if (nxt + 1u >= win + 32u) load_window(s);                 // (holds steps s .. s + 31 then)
            fetch_blocks(nxt);
            fetch_x(nxt);
        }
        cp_async_commit();
        uint32_t f[2][16];
        const uint32_t src = my_blk + slot_of(s) * (SM::kWarps * SM::kBlk);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t d = src + i * (kP6BlockBytes + 128);
            const uint4 a = p6_lds128(d + lane * 16);
            const uint2 a2 = p6_lds64(d + 512 + lane * 8);
            const uint32_t w[6] = {a.x, a.y, a.z, a.w, a2.x, a2.y};
            p6_unpack(w, e2, s2[i], f[i]);
            const int32_t lo = __shfl_sync(0xffffffffu, off_l[i], (int)(s - win)), hi = __shfl_sync(0xffffffffu, off_l[i], (int)(s + 1u - win));
            if (!have[i] || lo == hi) continue;        // (warp uniform) no outliers in the block
            // the block's outliers into the image
            auto patch = [&](uint32_t where, uint32_t v) {
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(where), "h"((unsigned short)v) : "memory");
            };
            uint32_t where = 0;
            if (lo + lane < hi) {
                const uint32_t e = p6_lds32(d + kP6BlockBytes + lane * 4);
                where = img_s + p6_image_at(e);
                patch(where, e >> 16);
            }
            for (int32_t j = lo + 32 + lane; j < hi; j += 32) {        // rare: more than 32 in a block
                const uint32_t e = __ldg(p.esc + j);
                patch(img_s + p6_image_at(e), e >> 16);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = p6_lds128(img_s + (q * 32 + lane) * 16);
                f[i][4 * q] |= v.x;
                f[i][4 * q + 1] |= v.y;
                f[i][4 * q + 2] |= v.z;
                f[i][4 * q + 3] |= v.w;
            }
            __syncwarp();
            if (lo + lane < hi) patch(where, 0);
            for (int32_t j = lo + 32 + lane; j < hi; j += 32) patch(img_s + p6_image_at(__ldg(p.esc + j)), 0);
            __syncwarp();
        }
        const uint32_t xb = xpart + slot_of(s) * (PARTS * SM::kX) + xl;
        uint2 xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = p6_lds64(xb + 32u * j);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            uint2 yv[4];
            if (n + 1 < NT) {
#pragma unroll
                for (int j = 0; j < 4; ++j) yv[j] = p6_lds64(xb + (n + 1) * 8 * kPrXPitch + 32u * j);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    p6_mma(acc[i][n], f[i][4 * j], f[i][4 * j + 1], f[i][4 * j + 2], f[i][4 * j + 3], xv[j].x, xv[j].y);
            if (n + 1 < NT) {
#pragma unroll
                for (int j = 0; j < 4; ++j) xv[j] = yv[j];
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();                                   // the ring becomes the parts' sums [part][token][128 rows]
    float *red = (float *)pr_smem;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float *dst = red + (size_t)part * NT * 8 * kPrRedPitch + pair * 32 + i * 16 + g;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            dst[(n * 8 + 2 * t) * kPrRedPitch] = acc[i][n][0];
            dst[(n * 8 + 2 * t + 1) * kPrRedPitch] = acc[i][n][1];
            dst[(n * 8 + 2 * t) * kPrRedPitch + 8] = acc[i][n][2];
            dst[(n * 8 + 2 * t + 1) * kPrRedPitch + 8] = acc[i][n][3];
        }
    }
    __syncthreads();
    auto put = [&](uint32_t m, uint32_t r, float v) {
        const uint32_t row = group * kPrRows + r;
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
    const uint32_t n_out = m_rows * kPrRows;
    for (uint32_t i = tid; i < n_out; i += PARTS * 128u) {
        const uint32_t m = i / kPrRows, r = i % kPrRows;
        float v = red[m * kPrRedPitch + r];
#pragma unroll
        for (int q = 1; q < PARTS; ++q) v += red[((uint32_t)q * NT * 8 + m) * kPrRedPitch + r];
        if (splits == 1u) put(m, r, v);
        else red[m * kPrRedPitch + r] = v;             // (this thread is the only reader of the word it overwrites)
    }
    if (splits == 1u) return;
    pr_cluster_sync();
    for (uint32_t i = split * (PARTS * 128u) + tid; i < n_out; i += splits * (PARTS * 128u)) {
        const uint32_t m = i / kPrRows, r = i % kPrRows, a = smem0 + (m * kPrRedPitch + r) * 4u;
        float v = pr_ld_cluster(a, 0);
        for (uint32_t c = 1; c < splits; ++c) v += pr_ld_cluster(a, c);
        put(m, r, v);
    }
    pr_cluster_sync();                                 // no CTA leaves while another reads its sums
}

}  // namespace ixb
