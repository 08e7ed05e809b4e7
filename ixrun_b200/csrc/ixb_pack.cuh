// Device-side quantiser and packer (deploy time): bf16 weight -> int8 codes ->
// the five (3,5,8) streams, bit for bit what the reference's CPU quantiser
// writes (ixrun/quantize.py:41-122, ixrun/bitpack.py:13-61).
#pragma once
#include "ixb_common.cuh"

namespace ixb {

// max |w| over the tensor as bf16 bits (non-negative floats order like their bit patterns); NaN payloads are ignored.
// Bound by memory: eight numbers per load, all of a thread's loads independent (5120 x 5120: 50 us with one number per
// load, before).
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

__device__ __forceinline__ int quantise_code(uint32_t bf16_bits, float sc)
{
    float q = rintf(__fdiv_rn(__uint_as_float(bf16_bits << 16), sc));
    q = fminf(fmaxf(q, -127.f), 127.f);
    return (int)q;
}

// One warp per 1024-element block.  MODE 0: quantise from bf16 weights and write codes; MODE 1: read existing codes.
// Both write the B1 words and the block's level-1 / level-2 counts.  Whole blocks of aligned tensors: a lane takes
// eight consecutive elements four times, so that loads (16 / 8 bytes), codes and B1 bytes are contiguous across the warp
// (5120 x 5120 in mode 0: 154 us when a lane walked its 32 elements one by one, before).
template <int MODE>
__global__ void __launch_bounds__(256)
k_codes_and_counts(const uint16_t *__restrict__ w, const uint32_t *absmax_bits, int8_t *codes, uint32_t n,
                   uint32_t *b1, int32_t *cnt1, int32_t *cnt2, __nv_bfloat16 *scale_out)
{
    uint32_t nb = (n + kBlk - 1) / kBlk;
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= nb) return;
    float sc = 1.f;
    if (MODE == 0) {
        __nv_bfloat16 s = scale_from_absmax(*absmax_bits);
        sc = __bfloat162float(s);
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
            uint32_t co[2] = {0, 0}, m1 = 0, e2 = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                int c;
                if (MODE == 0) {
                    c = quantise_code((wr[i >> 1] >> (16 * (i & 1))) & 0xffffu, sc);
                    co[i >> 2] |= (uint32_t)(c & 0xff) << (8 * (i & 3));
                } else {
                    c = (int)(int8_t)(cr[i >> 2] >> (8 * (i & 3)));
                }
                const int lv = code_level(c);
                m1 |= (uint32_t)(lv == 0) << i;
                e2 |= (uint32_t)(lv == 1) << i;
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
                c = quantise_code(w[e0 + i], sc);
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

// fields of one stream, put down one after the other into a warp's image of the stream's words: whole words and the two
// ends that neighbouring lanes share go in with a shared-memory OR
struct FieldWriter {
    uint32_t *img;                // word of the next bit
    uint64_t buf;
    uint32_t fill;
    __device__ __forceinline__ FieldWriter(uint32_t *image, uint32_t bit) : img(image + (bit >> 5)), buf(0), fill(bit & 31u) {}
    __device__ __forceinline__ void put(uint32_t v, uint32_t width)
    {
        buf |= (uint64_t)v << fill;
        fill += width;
        if (fill >= 32u) {
            atomicOr(img++, (uint32_t)buf);
            buf >>= 32;
            fill -= 32u;
        }
    }
    __device__ __forceinline__ void flush() { if (fill) atomicOr(img, (uint32_t)buf); }
};

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

// Streams must be zero on entry.  One warp per block, lane = word of 32 elements; the block's part of every stream is put
// together in shared memory and written in whole words (one global atomic per field, before: 104 us for 5120 x 5120).
constexpr int kPackB2 = 0, kPackL1 = 34, kPackL2 = 132, kPackWords = 296;    // 33, 97 and 162 words at most
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
    uint32_t m1 = 0, e2 = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int lv = (uint32_t)i < valid ? code_level((int)(int8_t)(cw[i >> 2] >> (8 * (i & 3)))) : 3;
        m1 |= (uint32_t)(lv == 0) << i;
        e2 |= (uint32_t)(lv == 1) << i;
    }
    const uint32_t a0 = (uint32_t)a_blk[b], c0 = (uint32_t)c_blk[b], r0 = b * kBlk - a0;    // the block's first ranks
    const uint32_t i1 = warp_incl_scan(__popc(m1), lane), i2 = warp_incl_scan(__popc(e2), lane);
    const uint32_t a1 = a0 + __shfl_sync(0xffffffffu, i1, 31), c1 = c0 + __shfl_sync(0xffffffffu, i2, 31);
    const uint32_t r1 = min((b + 1u) * kBlk, n) - a1;
    uint32_t a = a0 + i1 - __popc(m1), cc = c0 + i2 - __popc(e2);
    uint32_t r = min(e0, n) - a;  // rank among non-L1 elements
    uint32_t t = r - cc;
    FieldWriter w1(img + kPackL1, 3u * a - (3u * a0 & ~31u)), w2(img + kPackL2, 5u * cc - (5u * c0 & ~31u)),
        wb(img + kPackB2, r - (r0 & ~31u));
    __syncwarp();                                        // the image is zero
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        if ((uint32_t)i >= valid) break;
        const int c = (int)(int8_t)(cw[i >> 2] >> (8 * (i & 3)));
        if ((m1 >> i) & 1u) {
            w1.put((uint32_t)(c + 3), 3u);
        } else {
            const uint32_t two = (e2 >> i) & 1u;
            wb.put(two, 1u);
            if (two) w2.put((uint32_t)(c + 15), 5u);
            else l3[t++] = (uint8_t)(c + 127);
        }
    }
    w1.flush();
    w2.flush();
    wb.flush();
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
