// Causal attention of a prompt's rows over the static KV cache (the many-row counterpart of k_attn_decode): row r of T
// new rows sits at position pos0 + r, its key and value are in the cache already, and it attends to positions
// 0 .. pos0 + r.  The eager path runs this as fp32 matmuls around a masked softmax over the whole static cache.
//
// Bound: the tensor core (8 MMA steps of 16 x 8 x 16 per 16 x 16 scores and head dimension 16: two for Q K^T, six for
// P V): a 1000-row prompt's 16 x 136 pairs of 64-row and 64-key tiles of 16 heads are 17 us at mma.sync's rate.  What it
// has to fight is the chain of key tiles of the last rows and the uneven lengths: CTA = 64 rows of one query head, two
// groups of four warps (16 rows a warp) take the even and the odd key tiles, each through its own two cp.async stages, and
// join at the end; the row tiles with the longest contexts of all heads start first.  Q K^T: bf16 operands, fp32 sums.  The
// probabilities are held in fp32, and so are they multiplied: p = three bf16 numbers of 8 significant bits each, three MMAs.
// The tensor core cuts the low bits of what it adds to a large sum, so a key tile's P V starts from zero and joins the
// running sums by fp32 fused multiply-adds; the denominator is summed from the fp32 values.
// (An infinite value in the cache gives NaN: the parts of a probability may be zero or negative.)
// Against 64 bits (16 / 8 heads of 128, 4 / 4 and 8 / 1 of 64; 65 to 1000 rows, and 200 behind 1500; scores and values of
// three sizes): the share of outputs that are not the correctly rounded bf16 number is 0.5 to 50 in 100,000, that of fp32
// matmuls around a softmax 1 to 130; 5 to 260 with two bf16 numbers and running sums in the tensor core.
// Measured (16 query / 8 KV heads of 128, graph): 65 / 300 / 1000 / 2048 rows 6.9 / 13.5 / 37 / 128 us, with two bf16
// numbers 6.4 / 12.5 / 34 / 115; with one group per CTA and the heads one after the other 50 for 1000 rows.
#pragma once
#include "ixb_p6.cuh"

namespace ixb {

constexpr int kApRows = 64, kApKeys = 64, kApGroup = 128, kApThreads = 2 * kApGroup;

template <int D>
constexpr uint32_t ap_smem_bytes() { return (uint32_t)(kApRows + 8 * kApKeys) * (D + 8) * 2u; }   // Q, two groups' two stages of K and V

__device__ __forceinline__ void ap_ldmatrix_t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t ap_pack(float lo, float hi)
{
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16;
}

// grid (query heads, row tiles)
template <int D>
__global__ void __launch_bounds__(kApThreads)
k_attn_prefill(const __nv_bfloat16 *__restrict__ q, const __nv_bfloat16 *__restrict__ k_cache,
               const __nv_bfloat16 *__restrict__ v_cache, __nv_bfloat16 *__restrict__ out, uint32_t T, uint32_t pos0,
               uint32_t hq, uint32_t hkv, float scale, uint32_t q_stride)
{
    constexpr int PITCH = D + 8;                       // elements; rows 16 bytes apart modulo 128: ldmatrix without conflicts
    constexpr int CH = D / 8;                          // 16-byte chunks per row
    extern __shared__ __align__(128) unsigned char ap_smem[];
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(ap_smem);
    const uint32_t stage_bytes = 2u * kApKeys * PITCH * 2u;
    const int tid = threadIdx.x & (kApGroup - 1), lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t kg = threadIdx.x / kApGroup;        // the group: key tiles kg, kg + 2, ...
    const uint32_t sq = s0, sk = s0 + kApRows * PITCH * 2u + kg * 2u * stage_bytes, sv = sk + kApKeys * PITCH * 2u;
    const uint32_t head = blockIdx.x, kvh = head / (hq / hkv);
    const uint32_t r0 = (gridDim.y - 1u - blockIdx.y) * kApRows;       // longest contexts first
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t n_keys = pos0 + min(r0 + (uint32_t)kApRows, T);     // keys that any row of the tile sees
    const uint32_t n_tiles = (n_keys + kApKeys - 1) / kApKeys;
    const size_t row_stride = (size_t)hkv * D;
    for (int c = threadIdx.x; c < kApRows * CH; c += kApThreads) {
        const uint32_t r = c / CH, ch = c % CH;
        p6_cp16(sq + (r * PITCH + ch * 8u) * 2u, q + (size_t)min(r0 + r, T - 1u) * q_stride + (size_t)head * D + ch * 8u);
    }
    auto fetch = [&](uint32_t kt) {                                     // rows beyond the last key repeat it (masked below)
        const uint32_t st = (kt >> 1 & 1u) * stage_bytes;
        for (int c = tid; c < kApKeys * CH; c += kApGroup) {
            const uint32_t r = c / CH, ch = c % CH;
            const size_t at = (size_t)min(kt * kApKeys + r, n_keys - 1u) * row_stride + (size_t)kvh * D + ch * 8u;
            p6_cp16(sk + st + (r * PITCH + ch * 8u) * 2u, k_cache + at);
            p6_cp16(sv + st + (r * PITCH + ch * 8u) * 2u, v_cache + at);
        }
    };
    if (kg < n_tiles) fetch(kg);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    uint32_t qf[D / 16][4];                            // the warp's 16 rows as A operands
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
        p6_ldmatrix(qf[kk], sq + ((wid * 16 + (lane & 15)) * PITCH + kk * 16 + (lane >> 4) * 8) * 2u);
    float o[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    const float sl2 = scale * 1.4426950408889634f;     // scores in units of log2: probabilities are powers of two
    const uint32_t p_lo = pos0 + r0 + wid * 16 + g;    // position of the lane's first row (the second is 8 further)
    for (uint32_t kt = kg; kt < n_tiles; kt += 2) {
        if (kt + 2 < n_tiles) fetch(kt + 2);           // the other stage: its readers passed the barrier below
        cp_async_commit();
        const uint32_t st = (kt >> 1 & 1u) * stage_bytes;
        float s[kApKeys / 8][4];
#pragma unroll
        for (int n = 0; n < kApKeys / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int n2 = 0; n2 < kApKeys / 16; ++n2) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                uint32_t b[4];                          // keys 16 n2 .. + 15, dimensions 16 kk .. + 15
                p6_ldmatrix(b, sk + st + ((n2 * 16 + (lane & 7) + (lane >> 4) * 8) * PITCH + kk * 16 + ((lane >> 3) & 1) * 8) * 2u);
                p6_mma(s[2 * n2], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], b[0], b[1]);
                p6_mma(s[2 * n2 + 1], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], b[2], b[3]);
            }
        }
        const bool edge = (kt + 1) * kApKeys > pos0 + r0 + wid * 16 + 1u;      // (warp uniform) some score may be masked
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < kApKeys / 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v = s[n][i] * sl2;
                if (edge && kt * kApKeys + n * 8 + 2 * t + (i & 1) > p_lo + 8 * (i >> 1)) v = -INFINITY;
                s[n][i] = v;
                mx[i >> 1] = fmaxf(mx[i >> 1], v);
            }
        float corr[2], base[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            const float mn = fmaxf(m[h], mx[h]);
            base[h] = mn == -INFINITY ? 0.f : mn;       // a row of nothing but -inf so far keeps sum 0
            corr[h] = exp2f(m[h] - base[h]);
            m[h] = mn;
            l[h] *= corr[h];
        }
#pragma unroll
        for (int n = 0; n < kApKeys / 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[n][i] = exp2f(s[n][i] - base[i >> 1]);
                l[i >> 1] += s[n][i];
            }
        // probabilities as three bf16 numbers whose sum they are (8 significant bits each; the differences are exact):
        // [part][keys 16 kk][a0: row g, keys 2 t; a1: row g + 8; a2, a3: keys 8 further]
        uint32_t pa[3][kApKeys / 16][4];
#pragma unroll
        for (int kk = 0; kk < kApKeys / 16; ++kk)
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                float x0 = s[2 * kk + (a >> 1)][2 * (a & 1)], x1 = s[2 * kk + (a >> 1)][2 * (a & 1) + 1];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    pa[c][kk][a] = ap_pack(x0, x1);
                    x0 -= __uint_as_float(pa[c][kk][a] << 16);
                    x1 -= __uint_as_float(pa[c][kk][a] & 0xFFFF0000u);
                }
            }
#pragma unroll
        for (int d2 = 0; d2 < D / 16; ++d2) {
            float w[2][4];                              // the tile's own sums: the tensor core cuts what it adds to a large one
#pragma unroll
            for (int i = 0; i < 4; ++i) w[0][i] = w[1][i] = 0.f;
#pragma unroll
            for (int kk = 0; kk < kApKeys / 16; ++kk) {
                uint32_t b[4];                          // keys 16 kk .. + 15, dimensions 16 d2 .. + 15
                ap_ldmatrix_t(b, sv + st + ((kk * 16 + (lane & 15)) * PITCH + d2 * 16 + (lane >> 4) * 8) * 2u);
#pragma unroll
                for (int c = 2; c >= 0; --c) {
                    p6_mma(w[0], pa[c][kk][0], pa[c][kk][1], pa[c][kk][2], pa[c][kk][3], b[0], b[1]);
                    p6_mma(w[1], pa[c][kk][0], pa[c][kk][1], pa[c][kk][2], pa[c][kk][3], b[2], b[3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[2 * d2][i] = fmaf(o[2 * d2][i], corr[i >> 1], w[0][i]);
                o[2 * d2 + 1][i] = fmaf(o[2 * d2 + 1][i], corr[i >> 1], w[1][i]);
            }
        }
        cp_async_wait<0>();
        asm volatile("bar.sync %0, %1;" ::"r"(kg + 1u), "n"(kApGroup) : "memory");    // the group's next stage has landed, this one is free
    }
    // the odd tiles' group hands its sums over through its own stages
    constexpr int OP = D + 4;                          // floats per row
    float *xo = (float *)(ap_smem + kApRows * PITCH * 2 + 2 * stage_bytes), *xm = xo + kApRows * OP, *xl = xm + kApRows;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
        if (kg == 1) {
            const uint32_t r = wid * 16 + g + 8 * h;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) *(float2 *)(xo + r * OP + n * 8 + 2 * t) = make_float2(o[n][2 * h], o[n][2 * h + 1]);
            if (t == 0) {
                xm[r] = m[h];
                xl[r] = l[h];
            }
        }
    }
    __syncthreads();
    if (kg == 1) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t r = wid * 16 + g + 8 * h, row = r0 + r;
        if (row >= T) continue;
        const float m1 = xm[r], mn = fmaxf(m[h], m1), mb = mn == -INFINITY ? 0.f : mn;
        const float f0 = exp2f(m[h] - mb), f1 = exp2f(m1 - mb), inv = 1.f / (l[h] * f0 + xl[r] * f1);
        __nv_bfloat16 *dst = out + ((size_t)row * hq + head) * D + 2 * t;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
            const float2 v = *(const float2 *)(xo + r * OP + n * 8 + 2 * t);
            *(uint32_t *)(dst + n * 8) = ap_pack((o[n][2 * h] * f0 + v.x * f1) * inv, (o[n][2 * h + 1] * f0 + v.y * f1) * inv);
        }
    }
}

}  // namespace ixb
