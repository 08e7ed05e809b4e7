// GEMV on the resident P6 layout for 1..8 activation rows of layers with few blocks per warp (a decode step of a 1B-class model
// consists of them): what k_p6_mma (ixb_p6.cuh) does, arranged for the shortest chain behind the dependency wait.
//
//   Y[m][n] = sum_k X[m][k] * bf16(code[n][k] * scale)        m < m_rows <= 8
//
//   CTA   = a contiguous range of whole row tiles, so that nothing is joined across CTAs; 16 warps.
//   warp  = a contiguous part of K, the same one in every tile of the CTA: its activations are its own (no CTA barrier between
//           their arrival and the first product) and are fetched once for all tiles.
//   Ahead of griddepcontrol.wait: all of the warp's blocks (eight at most, which is what the kernel is taken for) are requested into
//   registers, two of them are already weights with their outliers OR-ed over the placeholders (+0.0) from an image of the lanes'
//   registers in shared memory.  Behind it: activations (cp.async), four mma.sync per block, partial tiles to shared memory, one barrier, sums of
//   the 16 parts by shuffles in a fixed tree, outputs.
//
// What bounds it: one chain of latencies: launch, activations from L2, two to eight blocks, the barrier, the sums, the stores.  In a
// graph with dependent launch, k_p6_mma and this kernel at 1 / 8 rows: 2048 x 2048 5.3 -> 2.9, 7.1 -> 4.2 us; 4096 x 2048 6.0 -> 4.1,
// 7.7 -> 5.4; 2048 x 6144 6.7 -> 5.0, 8.7 -> 6.7; 1024 x 3072 5.0 -> 2.1, 7.0 -> 3.5.  There, joining the parts of 24 warps through
// arrival counters took 1.75 us of the 5.3, the outliers' own pass 0.45 at one row and 1.5 at five, the CTA-wide staging of
// activations the rest.  With more blocks per warp, the rest requested one by one, it was the slower one: 10240 x 2048 (10 blocks) 7.6
// and 7.7 us, 9.1 and 10.0; 12288 x 2048 (12) 7.8 and 9.2.
#pragma once
#include "ixb_p6.cuh"

namespace ixb {

constexpr int kPsWarps = 16;
constexpr int kPsThreads = kPsWarps * 32;
constexpr int kPsReady = 2;                              // blocks converted ahead of the dependency wait
constexpr int kPsAhead = 6;                              // packed blocks in registers behind those
constexpr uint32_t kPsMaxBlocks = kPsReady + kPsAhead;   // blocks of a warp: all are requested at once, none later

struct PsPlan {
    uint32_t grid, tiles, slice;                         // CTAs; most tiles of a CTA; most column blocks of a warp
    uint32_t xpitch, smem;                               // bytes of an activation row of a warp's slice; all of shared memory
};
// floats of one warp's part of a tile
__host__ __device__ constexpr uint32_t ps_part(bool multi) { return multi ? 128u : 16u; }
__host__ __device__ constexpr uint32_t ps_xpitch(uint32_t slice) { return slice * 128u + 32u; }      // 8-byte reads of eight rows without conflicts

template <bool MULTI>
__global__ void __launch_bounds__(kPsThreads, 1)
k_p6_short(P6 p, const __nv_bfloat16 *__restrict__ x, uint32_t m_rows, const __nv_bfloat16 *__restrict__ bias, void *y, int y_f32,
           PsPlan plan, P6Push push)
{
    extern __shared__ __align__(128) unsigned char ps_smem[];
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t wid = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(ps_smem);
    const uint32_t img_s = smem0 + wid * 2048u, xs = smem0 + kPsWarps * 2048u + wid * m_rows * plan.xpitch;
    float *parts = (float *)(ps_smem + kPsWarps * 2048u + kPsWarps * m_rows * plan.xpitch);       // [tile][warp][ps_part]
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t KB = p.kb, tq = p.rt / plan.grid, tr = p.rt - tq * plan.grid;
    const uint32_t t0 = p6_begin(blockIdx.x, tq, tr), tiles = p6_begin(blockIdx.x + 1, tq, tr) - t0;
    const uint32_t kq = KB / kPsWarps, kr = KB - kq * kPsWarps;
    const uint32_t k0 = p6_begin(wid, kq, kr), nk = p6_begin(wid + 1, kq, kr) - k0;
    const uint32_t n = tiles * nk;                       // the warp's blocks, tile by tile
    // ---- the block to request next, and the one to convert next
    struct Blk { uint4 a; uint2 b; int32_t lo, hi; uint32_t e; };       // plane, outlier range, this lane's first outlier
    uint32_t ft = 0, fk = 0;
    auto fetch = [&](Blk &q) {
        if (ft >= tiles) return;                         // (warp uniform)
        const uint32_t b = (t0 + ft) * KB + k0 + fk;
        const unsigned char *src = p.plane + (size_t)b * kP6BlockBytes;
        q.a = __ldg((const uint4 *)src + lane);
        q.b = __ldg((const uint2 *)(src + 512) + lane);
        q.lo = __ldg(p.blk_off + b);
        q.hi = __ldg(p.blk_off + b + 1);
        if (++fk == nk) {
            fk = 0;
            ++ft;
        }
    };
    auto fetch_entry = [&](Blk &q) {                     // (once the range is there)
        if (q.lo + lane < q.hi) q.e = __ldg(p.esc + q.lo + lane);
    };
    Blk ready[kPsReady] = {}, ahead[kPsAhead] = {};
    if (nk) {
#pragma unroll
        for (int i = 0; i < kPsReady; ++i) fetch(ready[i]);
#pragma unroll
        for (int i = 0; i < kPsAhead; ++i) fetch(ahead[i]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(img_s + (q * 32 + lane) * 16), "r"(0u) : "memory");
    __syncwarp();
    uint32_t e2;
    asm volatile("mov.b32 %0, 0x43004300;" : "=r"(e2));
    auto convert = [&](const Blk &q, uint32_t s2, uint32_t (&f)[16]) {
        const uint32_t w[6] = {q.a.x, q.a.y, q.a.z, q.a.w, q.b.x, q.b.y};
        if (q.lo == q.hi) {                              // warp uniform
            p6_unpack(w, e2, s2, f);
            return;
        }
        auto put = [&](uint32_t where, uint32_t v) {
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(where), "h"((unsigned short)v) : "memory");
        };
        uint32_t where = 0;
        const bool mine = q.lo + lane < q.hi;
        if (mine) {
            where = img_s + p6_image_at(q.e);
            put(where, q.e >> 16);
        }
        for (int32_t j = q.lo + 32 + lane; j < q.hi; j += 32) {
            const uint32_t e = __ldg(p.esc + j);
            put(img_s + p6_image_at(e), e >> 16);
        }
        __syncwarp();
        p6_unpack(w, e2, s2, f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint4 v = p6_lds128(img_s + (k * 32 + lane) * 16);
            f[4 * k] |= v.x;
            f[4 * k + 1] |= v.y;
            f[4 * k + 2] |= v.z;
            f[4 * k + 3] |= v.w;
        }
        __syncwarp();
        if (mine) put(where, 0);
        for (int32_t j = q.lo + 32 + lane; j < q.hi; j += 32) put(img_s + p6_image_at(__ldg(p.esc + j)), 0);
        __syncwarp();
    };
    // the scale of a tile, one tile ahead
    uint32_t s_cur = p6_scale2(p.scale[t0 * p.scale_stride]);
    uint32_t s_next = p6_scale2(p.scale[min(t0 + 1u, p.rt - 1u) * p.scale_stride]);
    uint32_t fr[kPsReady][16];
#pragma unroll
    for (int i = 0; i < kPsReady; ++i) fetch_entry(ready[i]);
    fetch_entry(ahead[0]);
    fetch_entry(ahead[1]);
#pragma unroll
    for (int i = 0; i < kPsReady; ++i)
        if ((uint32_t)i < n) convert(ready[i], (uint32_t)i >= nk ? s_next : s_cur, fr[i]);      // (nk == 1: the second block is of the second tile)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t push_e = push.world ? __ldcg(push.epoch) + 1u : 0u;      // (see k_p6_mma)
    // ---- the slice's activations: 16-byte pieces, zeros behind the rows' ends (in_f % 8 == 0)
    for (uint32_t m = 0; m < m_rows; ++m)
        for (uint32_t c = lane; c < nk * 8u; c += 32u) {
            const uint32_t col = k0 * kTileCols + c * 8u, dst = xs + m * plan.xpitch + c * 16u;
            if (col < p.in_f) p6_cp16(dst, x + (size_t)m * p.in_f + col);
            else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
        }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    const uint32_t xl = xs + min((uint32_t)g, m_rows - 1u) * plan.xpitch + 8u * t;               // (rows beyond m_rows only feed unused columns)
    float c[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t tile = 0, k = 0;                            // of the next block
    auto multiply = [&](const uint32_t (&f)[16]) {
        uint2 xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = p6_lds64(xl + k * 128u + 32u * j);
        p6_mma(c, f[0], f[1], f[2], f[3], xv[0].x, xv[0].y);
        p6_mma(c1, f[4], f[5], f[6], f[7], xv[1].x, xv[1].y);
        p6_mma(c, f[8], f[9], f[10], f[11], xv[2].x, xv[2].y);
        p6_mma(c1, f[12], f[13], f[14], f[15], xv[3].x, xv[3].y);
        if (++k < nk) return;
        // the warp's part of the tile is complete
        float *dst = parts + (tile * kPsWarps + wid) * ps_part(MULTI);
        if (MULTI) {
            ((float4 *)dst)[lane] = make_float4(c[0] + c1[0], c[1] + c1[1], c[2] + c1[2], c[3] + c1[3]);
        } else if (t == 0) {
            dst[g] = c[0] + c1[0];
            dst[g + 8] = c[2] + c1[2];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = c1[j] = 0.f;
        k = 0;
        ++tile;
        s_cur = s_next;
        s_next = p6_scale2(p.scale[min(t0 + tile + 1u, p.rt - 1u) * p.scale_stride]);
    };
#pragma unroll
    for (int i = 0; i < kPsReady; ++i)
        if ((uint32_t)i < n) multiply(fr[i]);
#pragma unroll
    for (int q = 0; q < kPsAhead; ++q) {
        if ((uint32_t)(kPsReady + q) >= n) break;
        if (q + 2 < kPsAhead) fetch_entry(ahead[q + 2]);  // of the block after the next
        uint32_t f[16];
        convert(ahead[q], s_cur, f);
        multiply(f);
    }
    if (!nk) {                                           // fewer column blocks than warps: zeros
        for (uint32_t i = 0; i < tiles * ps_part(MULTI); i += 32u)
            if (i + lane < tiles * ps_part(MULTI)) parts[((i + lane) / ps_part(MULTI) * kPsWarps + wid) * ps_part(MULTI) + (i + lane) % ps_part(MULTI)] = 0.f;
    }
    __syncthreads();
    // ---- sums of the 16 parts: four lanes take four parts each in order, then two shuffles, the same for every m_rows.  MULTI: a
    // lane's float4 of the C fragment, a tile is four warps' work; else a row, two warps'.
    const uint32_t quad = (uint32_t)lane >> 3, kTasks = MULTI ? 4u : 2u;
    for (uint32_t task = wid; task < tiles * kTasks; task += kPsWarps) {
        const uint32_t ti = task / kTasks, l = (task % kTasks) * 8u + ((uint32_t)lane & 7u);       // fragment lane or row
        const float *src = parts + (ti * kPsWarps + quad * 4u) * ps_part(MULTI);
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (MULTI) {
            const float4 *q = (const float4 *)src + l;
            const float4 a0 = q[0], a1 = q[32], a2 = q[64], a3 = q[96];
            v[0] = ((a0.x + a1.x) + a2.x) + a3.x;
            v[1] = ((a0.y + a1.y) + a2.y) + a3.y;
            v[2] = ((a0.z + a1.z) + a2.z) + a3.z;
            v[3] = ((a0.w + a1.w) + a2.w) + a3.w;
        } else {
            v[0] = ((src[l] + src[16 + l]) + src[32 + l]) + src[48 + l];
        }
#pragma unroll
        for (int d = 8; d <= 16; d <<= 1)
#pragma unroll
            for (int j = 0; j < (MULTI ? 4 : 1); ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], d);
        // lane quad j of a fragment lane writes its element j: row l / 4 + 8 (j / 2), activation row 2 (l & 3) + (j & 1)
        const uint32_t m = MULTI ? 2u * (l & 3u) + (quad & 1u) : 0u, r = MULTI ? (l >> 2) + 8u * (quad >> 1) : l;
        const uint32_t row = (t0 + ti) * kTileRows + r;
        if ((!MULTI && quad) || m >= m_rows || row >= p.out_f) continue;
        const float o = !MULTI ? v[0] : quad == 0u ? v[0] : quad == 1u ? v[1] : quad == 2u ? v[2] : v[3];
        p6_put_out(push, push_e, p.out_f, m, row, o, bias, y, y_f32);
    }
    if (push.fin) p6_finish_exchange<kPsThreads>(push, push_e, p.out_f, m_rows, bias, y, y_f32);
}

}  // namespace ixb
