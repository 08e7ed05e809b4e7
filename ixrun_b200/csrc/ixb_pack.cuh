// Device-side quantiser and packer (deploy time): bf16 weight -> int8 codes ->
// the five (3,5,8) streams, bit for bit what the reference's CPU quantiser
// writes (ixrun/quantize.py:41-122, ixrun/bitpack.py:13-61).
#pragma once
#include "ixb_common.cuh"

namespace ixb {

// max |w| over the tensor as bf16 bits (non-negative floats order like their bit patterns); NaN payloads are ignored.
// Bound by memory: eight numbers per load, all of a thread's loads independent (5120 x 5120: 15 us, 50 with one number per
// load).
__global__ void __launch_bounds__(256) k_absmax(const uint16_t *__restrict__ w, uint32_t n, uint32_t *out_bits)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const uint32_t n8 = ((uintptr_t)w & 15u) ? 0u : n / 8u;             // whole 16-byte pieces
    uint32_t m2 = 0;
#pragma unroll 4
    for (uint32_t i = t; i < n8; i += nt) {
        const uint4 v = __ldg((const uint4 *)w + i);
        const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t b = r[k] & 0x7fff7fffu;
            m2 = __vmaxu2(m2, b & ~__vcmpgtu2(b, 0x7f807f80u));
        }
    }
    uint32_t m = max(m2 & 0xffffu, m2 >> 16);
    for (uint32_t i = n8 * 8u + t; i < n; i += nt) {
        const uint32_t b = w[i] & 0x7fffu;
        if (b <= 0x7f80u) m = max(m, b);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(out_bits, m);
}

// scale = bf16(bf16(max(absmax, 1e-8)) / 127), each step rounded like the reference does in bf16
__device__ __forceinline__ __nv_bfloat16 scale_from_absmax(uint32_t absmax_bits)
{
    float mx = __uint_as_float(absmax_bits << 16);
    float cl = mx < 1e-8f ? 1e-8f : mx;
    __nv_bfloat16 cl_b = __float2bfloat16_rn(cl);
    return __float2bfloat16_rn(__fdiv_rn(__bfloat162float(cl_b), 127.0f));
}

__device__ __forceinline__ int code_level(int c)
{
    int a = c < 0 ? -c : c;
    return a <= 3 ? 0 : (a <= 15 ? 1 : 2);
}

// ---- four codes at a time, as the bytes of a word (two's complement)
// 0xff where a byte's top bit is set, 0 elsewhere
__device__ __forceinline__ uint32_t byte_signs(uint32_t w)
{
    uint32_t v;
    asm("prmt.b32 %0, %1, %1, 0xBA98;" : "=r"(v) : "r"(w));
    return v;
}
// the top bits of the bytes: |code| > 3, |code| > 15
__device__ __forceinline__ void code_levels4(uint32_t w, uint32_t &over3, uint32_t &over15)
{
    const uint32_t neg = byte_signs(w), a = (w ^ neg) + (neg & 0x01010101u);       // |code|, at most 128: no byte carries
    over3 = (a + 0x7C7C7C7Cu) & 0x80808080u;
    over15 = (a + 0x70707070u) & 0x80808080u;
}
// the top bits of the four bytes as a number (bits 7, 15, 23, 31 meet at 28 .. 31, the other products below without a carry)
__device__ __forceinline__ uint32_t top_bits(uint32_t y) { return (y * 0x00204081u) >> 28; }

// code = clamp(rint(w / sc)), the division rounded to fp32 as the reference does.  w * (1 / sc) is within 2^-22 of the
// quotient, which for |code| < 128 is 3e-5: away from the halves between two codes both round to the same code, and only
// near them (or beyond 128, infinite, NaN, a scale without a reciprocal) the division itself is taken.
__device__ __forceinline__ int quantise_code(uint32_t bf16_bits, float sc, float inv)
{
    const float w = __uint_as_float(bf16_bits << 16);
    float q = w * inv, n = rintf(q);
    if (!(fabsf(q - n) < 0.499f && fabsf(q) < 128.f)) n = rintf(__fdiv_rn(w, sc));
    return (int)fminf(fmaxf(n, -127.f), 127.f);
}

// One warp per 1024-element block.  MODE 0: quantise from bf16 weights and write codes; MODE 1: read existing codes.
// Both write the B1 words and the block's level-1 / level-2 counts.  Whole blocks of aligned tensors: a lane takes
// eight consecutive elements four times, so that loads (16 / 8 bytes), codes and B1 bytes are contiguous across the warp.  The
// fast path rounds by an addition of 1.5 * 2^23, whose low byte is the code, and finds the levels of four codes at a time
// (5120 x 5120 in mode 0: 18.6 us, 27 with a rounding instruction and a comparison per element, 154 when a lane walked its 32
// elements one by one and divided each).
template <int MODE>
__global__ void __launch_bounds__(256)
k_codes_and_counts(const uint16_t *__restrict__ w, const uint32_t *absmax_bits, int8_t *codes, uint32_t n,
                   uint32_t *b1, int32_t *cnt1, int32_t *cnt2, __nv_bfloat16 *scale_out)
{
    uint32_t nb = (n + kBlk - 1) / kBlk;
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= nb) return;
    float sc = 1.f, inv = 1.f;
    if (MODE == 0) {
        __nv_bfloat16 s = scale_from_absmax(*absmax_bits);
        sc = __bfloat162float(s);
        inv = __frcp_rn(sc);
        if (b == 0 && lane == 0) *scale_out = s;
    }
    uint32_t n1 = 0, n2 = 0;
    const bool aligned = ((MODE == 0 ? (uintptr_t)w & 15u : 0u) | ((uintptr_t)codes & 7u)) == 0;
    if (aligned && (b + 1u) * kBlk <= n) {
        uint4 wv[4];
        uint2 cv[4];
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const uint32_t e = b * kBlk + it * 256u + lane * 8u;
            if (MODE == 0) wv[it] = __ldg((const uint4 *)(w + e));
            else cv[it] = *(const uint2 *)(codes + e);
        }
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const uint32_t e = b * kBlk + it * 256u + lane * 8u;
            const uint32_t wr[4] = {wv[it].x, wv[it].y, wv[it].z, wv[it].w}, cr[2] = {cv[it].x, cv[it].y};
            uint32_t co[2] = {cr[0], cr[1]};
            if (MODE == 0) {
                uint32_t r[8];
                bool plain = true;                       // no quotient near a half, none beyond the range
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float v = __uint_as_float(i & 1 ? wr[i >> 1] & 0xffff0000u : wr[i >> 1] << 16), q = v * inv, t = q + 12582912.f;
                    plain = plain && fabsf(q - (t - 12582912.f)) < 0.499f && fabsf(q) < 127.4f;
                    r[i] = __float_as_uint(t);
                }
                if (!plain) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) r[i] = (uint32_t)quantise_code((wr[i >> 1] >> (16 * (i & 1))) & 0xffffu, sc, inv);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    co[k] = __byte_perm(__byte_perm(r[4 * k], r[4 * k + 1], 0x0040), __byte_perm(r[4 * k + 2], r[4 * k + 3], 0x0040), 0x5410);
            }
            uint32_t m1 = 0, e2 = 0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t over3, over15;
                code_levels4(co[k], over3, over15);
                m1 |= (top_bits(over3) ^ 15u) << (4 * k);
                e2 |= top_bits(over3 & ~over15) << (4 * k);
            }
            if (MODE == 0) *(uint2 *)(codes + e) = make_uint2(co[0], co[1]);
            ((uint8_t *)b1)[e >> 3] = (uint8_t)m1;
            n1 += __popc(m1);
            n2 += __popc(e2);
        }
    } else {
        const uint32_t e0 = (b * 32u + lane) * 32u;
        uint32_t m1 = 0, e2 = 0;
        for (uint32_t i = 0; i < 32u && e0 + i < n; ++i) {
            int c;
            if (MODE == 0) {
                c = quantise_code(w[e0 + i], sc, inv);
                codes[e0 + i] = (int8_t)c;
            } else {
                c = codes[e0 + i];
            }
            const int lv = code_level(c);
            m1 |= (uint32_t)(lv == 0) << i;
            e2 |= (uint32_t)(lv == 1) << i;
        }
        if (e0 < n) b1[b * 32u + lane] = m1;
        n1 = __popc(m1);
        n2 = __popc(e2);
    }
    n1 = __reduce_add_sync(0xffffffffu, n1);
    n2 = __reduce_add_sync(0xffffffffu, n2);
    if (lane == 0) { cnt1[b] = (int32_t)n1; cnt2[b] = (int32_t)n2; }
}

// a lane's bits of one stream (NW words, the first bit lowest, zero beyond its end) into the warp's image at bit `bit`
template <int NW>
__device__ __forceinline__ void or_bits(uint32_t *image, uint32_t bit, const uint32_t (&v)[NW])
{
    uint32_t *at = image + (bit >> 5);
    uint32_t carry = 0;
#pragma unroll
    for (int k = 0; k <= NW; ++k) {
        const uint32_t cur = k < NW ? v[k] : 0u, word = __funnelshift_l(carry, cur, bit & 31u);
        if (word) atomicOr(at + k, word);
        carry = cur;
    }
}

// The block's words of one stream (bits [bit0, bit1) of it, image word 0 = stream word bit0 / 32) to memory: the first and
// the last may be shared with the neighbouring blocks.
__device__ __forceinline__ void write_image(uint32_t *stream, const uint32_t *img, uint32_t bit0, uint32_t bit1, int lane)
{
    if (bit0 == bit1) return;
    const uint32_t w0 = bit0 >> 5, nw = ((bit1 - 1u) >> 5) - w0 + 1u;
    for (uint32_t k = lane; k < nw; k += 32) {
        if (k == 0 || k == nw - 1u) atomicOr(stream + w0 + k, img[k]);
        else stream[w0 + k] = img[k];
    }
}

// Streams must be zero on entry.  One warp per block, lane = word of 32 elements.  Bound by instructions: levels and fields
// are made four at a time; a lane runs its elements backwards, eight at a time, and brings every field in at the low end of a
// group's bits (a multiplication and an addition: logic and shifts have half their rate), with predicates and no branches but
// for the rare level 3; a group then goes in at the low end of the lane's bits (3 words of level 1, 5 of level 2, one of the
// second bitmap).  The lanes' bits meet in an image of the block's words in shared memory, which is written in whole words.
// 5120 x 5120: 35 us; 58 with every field shifted into the lane's bits by itself, 91 with a branch per element, 104 with one
// global atomic per field.
constexpr int kPackB2 = 0, kPackL1 = 36, kPackL2 = 140, kPackWords = 308;    // 33, 97 and 161 words at most
__global__ void __launch_bounds__(256)
k_pack(const int8_t *__restrict__ codes, uint32_t n, const int32_t *__restrict__ a_blk, const int32_t *__restrict__ c_blk,
       uint32_t *b2, uint32_t *l1, uint32_t *l2, uint8_t *l3)
{
    __shared__ uint32_t images[8][kPackWords];
    uint32_t nb = (n + kBlk - 1) / kBlk;
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= nb) return;                                 // whole warps leave together
    uint32_t *img = images[threadIdx.x >> 5];
    for (int k = lane; k < kPackWords; k += 32) img[k] = 0;
    uint32_t e0 = (b * 32u + lane) * 32u;
    uint32_t valid = e0 >= n ? 0u : min(32u, n - e0);
    uint32_t cw[8];
    if (valid == 32u && ((uintptr_t)codes & 15u) == 0) {
        const uint4 v0 = __ldg((const uint4 *)(codes + e0)), v1 = __ldg((const uint4 *)(codes + e0) + 1);
        cw[0] = v0.x; cw[1] = v0.y; cw[2] = v0.z; cw[3] = v0.w;
        cw[4] = v1.x; cw[5] = v1.y; cw[6] = v1.z; cw[7] = v1.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) cw[k] = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if ((uint32_t)i < valid) cw[i >> 2] |= (uint32_t)(uint8_t)codes[e0 + i] << (8 * (i & 3));
    }
    uint32_t m1 = 0, e2 = 0, fld[8];                     // levels 1 and 2; the fields of either, four per word
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        uint32_t over3, over15;
        code_levels4(cw[k], over3, over15);
        m1 |= (top_bits(over3) ^ 15u) << (4 * k);
        e2 |= top_bits(over3 & ~over15) << (4 * k);
        const uint32_t f1 = ((cw[k] & 0x07070707u) + 0x03030303u) & 0x07070707u;       // code + 3
        const uint32_t f2 = ((cw[k] & 0x1F1F1F1Fu) + 0x0F0F0F0Fu) & 0x1F1F1F1Fu;       // code + 15
        const uint32_t big = byte_signs(over3);
        fld[k] = (f1 & ~big) | (f2 & big);
    }
    m1 &= lowmask(valid);                                // (elements beyond the tensor are no level 1; codes of 0 are no level 2)
    const uint32_t nl = ~m1 & (valid == 32u ? 0xffffffffu : (1u << valid) - 1u);     // not level 1
    const uint32_t a0 = (uint32_t)a_blk[b], c0 = (uint32_t)c_blk[b], r0 = b * kBlk - a0;    // the block's first ranks
    const uint32_t i1 = warp_incl_scan(__popc(m1), lane), i2 = warp_incl_scan(__popc(e2), lane);
    const uint32_t a1 = a0 + __shfl_sync(0xffffffffu, i1, 31), c1 = c0 + __shfl_sync(0xffffffffu, i2, 31);
    const uint32_t r1 = min((b + 1u) * kBlk, n) - a1;
    uint32_t a = a0 + i1 - __popc(m1), cc = c0 + i2 - __popc(e2);
    uint32_t r = min(e0, n) - a;  // rank among non-L1 elements
    uint32_t t = r - cc;
    // levels 1 and 2 and the second bitmap, from the last element to the first
    uint32_t v1[3] = {0, 0, 0}, v2[5] = {0, 0, 0, 0, 0}, vb[1] = {0};
#pragma unroll
    for (int q = 3; q >= 0; --q) {
        uint32_t g1 = 0, gb = 0;
#pragma unroll
        for (int h = 1; h >= 0; --h) {
            uint32_t g2 = 0;
#pragma unroll
            for (int i = 3; i >= 0; --i) {
                const int at = 8 * q + 4 * h + i;
                const uint32_t f = __byte_perm(fld[2 * q + h], 0, 0x4440 + i);
                const bool is1 = m1 & (1u << at), is2 = e2 & (1u << at), isn = nl & (1u << at);
                if (is1) g1 = g1 * 8u + f;
                if (is2) g2 = g2 * 32u + f;
                if (isn) gb = gb * 2u + (is2 ? 1u : 0u);
            }
            const uint32_t sh = 5u * __popc(e2 & (15u << (8 * q + 4 * h)));
#pragma unroll
            for (int k = 4; k > 0; --k) v2[k] = __funnelshift_l(v2[k - 1], v2[k], sh);
            v2[0] = v2[0] << sh | g2;
        }
        const uint32_t c1q = __popc(m1 & (255u << (8 * q))), cnq = __popc(nl & (255u << (8 * q))), sh = 3u * c1q;
        v1[2] = __funnelshift_l(v1[1], v1[2], sh);
        v1[1] = __funnelshift_l(v1[0], v1[1], sh);
        v1[0] = v1[0] << sh | g1;
        vb[0] = vb[0] << cnq | gb;
    }
    __syncwarp();                                        // the image is zero
    or_bits(img + kPackL1, 3u * a - (3u * a0 & ~31u), v1);
    or_bits(img + kPackL2, 5u * cc - (5u * c0 & ~31u), v2);
    or_bits(img + kPackB2, r - (r0 & ~31u), vb);
    for (uint32_t left = nl & ~e2; left; left &= left - 1u) l3[t++] = (uint8_t)(codes[e0 + __ffs((int)left) - 1] + 127);
    __syncwarp();
    write_image(l1, img + kPackL1, 3u * a0, 3u * a1, lane);
    write_image(l2, img + kPackL2, 5u * c0, 5u * c1, lane);
    write_image(b2, img + kPackB2, r0, r1, lane);
}

// ---------------------------------------------------------------- sibling format: per-group scales
// The group-scale variant of the format (ixgs/quantize.py:35-112, decode ixgs/kernels.py:31-102 and
// ixgs/quantize.py:116-151) stores the same five (3,5,8) streams (fields offset by -3 / -15 / -127, so the stream
// decoder above serves it unchanged) and one fp16 scale per `group` consecutive elements of the flat tensor instead of
// one per tensor: w[e] = bf16(f32(code[e]) * f32(scale[e / group])).  Eight weights per thread where the shape allows.
__global__ void __launch_bounds__(256)
k_group_scale(const int8_t *__restrict__ codes, const __half *__restrict__ gscale, uint32_t n, uint32_t group,
              __nv_bfloat16 *__restrict__ out)
{
    const uint32_t e0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8u;
    if (e0 >= n) return;
    if (e0 + 8u <= n && (group & 7u) == 0 && (((uintptr_t)codes | (uintptr_t)out) & 15u) == 0) {
        const float sc = __half2float(gscale[e0 / group]);             // eight consecutive elements share a group
        const uint2 c = *(const uint2 *)(codes + e0);
        const uint32_t cw[2] = {c.x, c.y};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int a = (int)(int8_t)((cw[k >> 1] >> (16 * (k & 1))) & 0xff);
            const int b = (int)(int8_t)((cw[k >> 1] >> (16 * (k & 1) + 8)) & 0xff);
            o[k] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn((float)a * sc)) |
                   ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn((float)b * sc)) << 16);
        }
        *(uint4 *)(out + e0) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
        for (uint32_t e = e0; e < min(e0 + 8u, n); ++e)
            out[e] = __float2bfloat16_rn((float)codes[e] * __half2float(gscale[e / group]));
    }
}

}  // namespace ixb
