// Resident re-layout "P6" of an INT8-X tensor and the kernels that run on it.
//
// It is built at deploy time, on the GPU, from the int8 codes that the
// reference's (3,5,8) streams decode to (ixrun/quantize.py:80-96), and keeps
// those codes exactly.  Nothing in it is addressed by rank: every 1024-weight
// block (16 rows x 64 columns, one warp) sits at a fixed address, and turning it
// into tensor-core operands costs four instructions per PAIR of weights:
//
//   plane   every element of code -32 .. 31 owns a 6-bit field F = 32 + code; put at the low end of the mantissa it makes
//           a bf16 number of the binade [128, 256):
//             F | 0x4300 = 128 + F = 160 + code
//           so a packed subtraction of 160 gives the code exactly, and the packed multiplication by the scale (plus 0, so
//           that code 0 gives +0.0 whatever the scale's sign) rounds the exact product once: the reference's dequantised
//           weight bf16(f32(code) * f32(scale)) (ixrun/quantize.py:182, ixrun/fused.py:169-170), bit for bit, for any
//           scale (but for the sign of that zero).
//           Other codes ("outliers") leave the placeholder F = 32 (weight 0).  (F used to be bits 6..1 of a number of
//           [64, 128): a shift more for every second pair.  Before that it was part of 1 + code / 32 over
//           two binades, one fused multiply-add per pair instead of two operations, but it held -16 .. 31 only: 1.2 % of
//           the benchmark distribution were outliers, 4 bytes and an extra step each, against 0.07 % now.)
//           Blocks of 16 rows x 64 columns, ragged edges padded with
//           placeholders (p6_elem gives the element of lane / pair / half); a
//           lane owns 32 fields in six 32-bit words,
//           a block is 768 contiguous bytes: 32 x uint4 (words 0..3), then
//           32 x uint2 (words 4, 5).  Word k holds pair 2k at bits 0 / 16 and
//           pair 2k+1 at bits 6 / 22 (low / high element); the 4 + 4 spare
//           bits of words 0..3 hold the low four bits of pairs 12..15, those of
//           words 4, 5 their upper two bits (p6_pair_words).
//   esc     the outliers of every block as 32-bit entries
//             bf16(code * s) << 16 | row_in_tile << 12 | (block & 63) << 6 | column_in_block
//           sorted by block; blk_off[nb + 1] gives the first entry of every block.
//           The low 12 bits are a column offset modulo 4096, so a run of up to
//           64 consecutive blocks of one row tile resolves its columns without
//           knowing which block an entry came from.
//
// Size: 6 + 32 * P(outlier) bits per weight + 4 bytes per block (6.05 bpw for
// the benchmark distribution).
//
// y = W x is one kernel (k_p6_mma): per warp a ring of cp.async-staged blocks,
// four instructions per pair of weights give the A fragments of four mma.sync.m16n8k16 (bf16) with the activations as B;
// the outliers of a warp's run of blocks are staged once in shared memory and added per row-tile segment of the run as
// the k index of further mmas, while the ring keeps fetching.  Products are exact, accumulation is fp32, and no
// floating-point atomics are used: results are reproducible.
#pragma once
#include "ixb_common.cuh"

namespace ixb {

constexpr int kTileRows = 16;      // a block: 16 rows x 64 columns = 1024 weights, one warp
constexpr int kTileCols = 64;

// Lane l of a block: g = l >> 2, t = l & 3.  Its 16 pairs p = 4 j + q (j = 0..3 the mma, q = 0..3 the A register):
//   row    = 16 R + g + 8 (q & 1)
//   column = 64 kb + 16 j + 4 t + 2 (q >> 1) + h          (h = 0 low half, 1 high half of the register)
// i.e. the k index of mma j is permuted inside its 16 columns so that a lane needs four consecutive activations, and a block's
// registers are the words 8 j + 2 t + (q >> 1) of its rows in column order: what tcgen05.st.16x256b makes of them in tensor
// memory, so that k_p6_umma can take the activations as they lie in memory.  (The GEMV alone would rather have 16 consecutive
// activations per lane, 16 t + 4 j: two 16-byte reads per block instead of four 8-byte ones.)
__device__ __forceinline__ void p6_elem(int lane, int p, int h, uint32_t &row_in_tile, uint32_t &col_in_tile)
{
    int g = lane >> 2, t = lane & 3, j = p >> 2, q = p & 3;
    row_in_tile = (uint32_t)(g + 8 * (q & 1));
    col_in_tile = (uint32_t)(16 * j + 4 * t + 2 * (q >> 1) + h);
}
// (SRC & MASK) | ACC
__device__ __forceinline__ uint32_t p6_and_or(uint32_t src, uint32_t mask, uint32_t acc)
{
    uint32_t v;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(src), "r"(mask), "r"(acc));
    return v;
}
__device__ __forceinline__ void p6_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int kP6BlockBytes = 768;
constexpr int kP6Slots = 4;                       // ring slots per warp; blocks are fetched three ahead
constexpr int kP6SlackBlocks = 5;                 // readable blocks behind the plane (the ring fetches past a run end)
constexpr int kP6SlackEntries = 64;               // readable entries behind the outlier list
constexpr int kP6CodeMin = -32, kP6CodeMax = 31;  // codes that the plane holds

struct P6 {
    const unsigned char *plane;  // [(nb + slack) * 768]
    const int32_t *blk_off;      // [nb + 1] first outlier entry of every block
    const uint32_t *esc;         // [n_esc + slack] outlier entries
    const __nv_bfloat16 *scale;  // scale_stride 0: one scale; 1: one per row tile (a tensor fused from several)
    uint32_t out_f, in_f;
    uint32_t rt, kb;             // row tiles, column blocks per row tile; nb = rt * kb
    uint32_t scale_stride;
};

// ------------------------------------------------------------------ build ---
// word j of lane t of a quad <-> word t of lane j
__device__ __forceinline__ void p6_quad_transpose(uint32_t (&a)[4], int lane)
{
#pragma unroll
    for (int d = 1; d <= 2; d <<= 1) {
        const bool up = lane & d;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int lo = d == 1 ? 2 * k : k, hi = lo + d;
            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? a[lo] : a[hi], d);
            if (up) a[lo] = got;
            else a[hi] = got;
        }
    }
}
// the lane's 32 codes of block (R, kbi): out[0..3] row g, out[4..7] row g + 8, the four columns 16 j + 4 t .. + 3 as the bytes
// of word j; elements beyond the tensor are 0.  Two 16-byte loads, dealt out over the quad, where rows and tensor allow.
__device__ __forceinline__ void p6_load_codes(const int8_t *__restrict__ codes, uint32_t out_f, uint32_t in_f, uint32_t R,
                                              uint32_t kbi, int lane, uint32_t (&out)[8])
{
    const bool vec = ((in_f & 15u) | ((uintptr_t)codes & 15u)) == 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const uint32_t row = R * kTileRows + (lane >> 2) + 8 * s;
        const int8_t *src = codes + (size_t)row * in_f + kbi * kTileCols;
        uint32_t w[4] = {0, 0, 0, 0};
        if (vec) {
            const uint32_t c0 = 16 * (lane & 3);
            if (row < out_f && kbi * kTileCols + c0 < in_f) {                   // in_f % 16 == 0: all 16 columns or none
                const uint4 v = __ldg((const uint4 *)(src + c0));
                w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
            }
            p6_quad_transpose(w, lane);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t at = 16 * j + 4 * (lane & 3) + c;
                    if (row < out_f && kbi * kTileCols + at < in_f) w[j] |= (uint32_t)(uint8_t)src[at] << (8 * c);
                }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) out[4 * s + j] = w[j];
    }
}
// element h of pair p out of them (byte 2 ((p & 3) >> 1) + h of word p >> 2 of row g + 8 (p & 1), see p6_elem)
__device__ __forceinline__ int p6_code_of(const uint32_t (&cw)[8], int p, int h)
{
    return (int)(int8_t)(cw[4 * (p & 1) + (p >> 2)] >> (8 * (2 * ((p & 3) >> 1) + h)));
}

// the top bits of the bytes that hold outliers: a code of -32 .. 31 has bits 7, 6 and 5 alike
__device__ __forceinline__ uint32_t p6_outliers4(uint32_t w)
{
    const uint32_t t = w ^ (w << 1);
    return (t | t << 1) & 0x80808080u;
}
// codes [out_f, in_f] -> plane blocks and the number of outliers of every block (one warp per block), four codes at a time:
// F = (code & 63) ^ 32, the bytes of a word are two pairs.  5120 x 5120: 12 us; 17 with a comparison and a shift per code,
// 33 with one byte per load.
__global__ void __launch_bounds__(256)
k_p6_plane(const int8_t *__restrict__ codes, uint32_t out_f, uint32_t in_f, uint32_t rt, uint32_t kb,
           unsigned char *plane, int32_t *blk_cnt)
{
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= rt * kb) return;
    uint32_t R = b / kb, kbi = b - R * kb;
    uint32_t cw[8], w[6] = {0, 0, 0, 0, 0, 0};
    uint32_t n_out = 0;
    p6_load_codes(codes, out_f, in_f, R, kbi, lane, cw);
#pragma unroll
    for (int k = 0; k < 8; ++k) {                    // word j = k & 3 of row half s = k >> 2: pairs 4 j + s and 4 j + 2 + s
        const uint32_t o = p6_outliers4(cw[k]);
        uint32_t out;                                // 0xff where there is an outlier
        asm("prmt.b32 %0, %1, %1, 0xBA98;" : "=r"(out) : "r"(o));
        n_out += __popc(o);
        const uint32_t f = (cw[k] & ~out & 0x3F3F3F3Fu) ^ 0x20202020u;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const uint32_t pair = __byte_perm(f, 0, v ? 0x4342 : 0x4140);          // fields at bits 0 and 16
            const int p = 4 * (k & 3) + 2 * v + (k >> 2);
            if (p < 12) {                            // (see p6_pair_words)
                w[p >> 1] |= pair << (6 * (p & 1));
            } else {
                const int i = p - 12;
                w[i] |= (pair & 0x000F000Fu) << 12;
                w[4 + (i >> 1)] |= (pair & 0x00300030u) << (8 + 2 * (i & 1));
            }
        }
    }
    unsigned char *blk = plane + (size_t)b * kP6BlockBytes;
    ((uint4 *)blk)[lane] = make_uint4(w[0], w[1], w[2], w[3]);
    ((uint2 *)(blk + 512))[lane] = make_uint2(w[4], w[5]);
    n_out = __reduce_add_sync(0xffffffffu, n_out);
    if (lane == 0) blk_cnt[b] = (int32_t)n_out;
}

// outlier entries of every block, in (lane, pair, half) order (one warp per block).  5120 x 5120: 15 us, 25 when every block's
// codes were read and compared one by one.
__global__ void __launch_bounds__(256)
k_p6_esc(const int8_t *__restrict__ codes, uint32_t out_f, uint32_t in_f, uint32_t rt, uint32_t kb,
         const int32_t *__restrict__ blk_off, const __nv_bfloat16 *__restrict__ scale, uint32_t scale_stride, uint32_t *esc,
         uint32_t n_esc)
{
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= rt * kb) return;
    uint32_t R = b / kb, kbi = b - R * kb;
    const int32_t lo = __ldg(blk_off + b);
    if (lo == __ldg(blk_off + b + 1)) return;        // (warp uniform) none, as in most blocks: the codes are not read
    float sc = __bfloat162float(scale[R * scale_stride]);
    uint32_t cw[8];
    p6_load_codes(codes, out_f, in_f, R, kbi, lane, cw);
    uint32_t n_out = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) n_out += __popc(p6_outliers4(cw[k]));
    uint32_t at = (uint32_t)lo + warp_incl_scan(n_out, lane) - n_out;
    if (n_out == 0) return;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int code = p6_code_of(cw, i >> 1, i & 1);
        if (code > kP6CodeMax || code < kP6CodeMin) {
            uint32_t r, c;
            p6_elem(lane, i >> 1, i & 1, r, c);
            uint32_t wbits = __bfloat16_as_ushort(__float2bfloat16_rn((float)code * sc));
            if (at < n_esc) esc[at] = (wbits << 16) | (r << 12) | ((b & 63u) << 6) | c;   // never beyond the caller's buffer
            ++at;
        }
    }
}

// ---------------------------------------------------------------- decode ----
// A lane's plane words with the last four pairs put together: word j of u holds pair 4 j at bits 0 / 16 and 4 j + 1 at 6 / 22, of v
// 4 j + 2 and 4 j + 3 (the other bits are anything).
__device__ __forceinline__ void p6_pair_words(const uint4 &a, const uint2 &b, uint32_t (&u)[4], uint32_t (&v)[4])
{
    u[0] = a.x; u[1] = a.z; u[2] = b.x;
    v[0] = a.y; v[1] = a.w; v[2] = b.y;
    u[3] = p6_and_or(b.x >> 8, 0x00300030u, (a.x >> 12) & 0x000F000Fu) | p6_and_or(b.x >> 4, 0x0C000C00u, (a.y >> 6) & 0x03C003C0u);
    v[3] = p6_and_or(b.y >> 8, 0x00300030u, (a.z >> 12) & 0x000F000Fu) | p6_and_or(b.y >> 4, 0x0C000C00u, (a.w >> 6) & 0x03C003C0u);
}
// the fields at bits 0 / 16 of u and v as four codes, the bytes of a word
__device__ __forceinline__ uint32_t p6_codes4(uint32_t u, uint32_t v)
{
    const uint32_t t = __byte_perm(u & 0x003F003Fu, v & 0x003F003Fu, 0x6420) ^ 0x20202020u, sign = t & 0x20202020u;
    return t | sign << 1 | sign << 2;
}

// plane -> int8 codes (OUT 0) or bf16 weights (OUT 1), row major [out_f, in_f]; outliers come out as 0 here.
// A lane holds four times four consecutive columns of two rows: 4 or 8 bytes per store; codes in aligned rows are dealt out over
// the quad while packed, 16 bytes per store.
// Codes, with the outliers' pass, in a graph: 17408 x 5120 40.5 us, 12288 x 2048 14.8, 8192 x 8200 39.8; 50.1, 16.9 and 40.5 with
// four bytes per store and a code at a time; 39.3, 14.4 and 277 on the layout whose lanes held 16 columns.
template <int OUT>
__global__ void __launch_bounds__(256) k_p6_decode_plane(P6 p, void *out)
{
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= p.rt * p.kb) return;
    uint32_t R = b / p.kb, kbi = b - R * p.kb;
    float sc = __bfloat162float(p.scale[R * p.scale_stride]);
    const unsigned char *blk = p.plane + (size_t)b * kP6BlockBytes;
    uint32_t u[4], v[4];
    p6_pair_words(((const uint4 *)blk)[lane], ((const uint2 *)(blk + 512))[lane], u, v);
    const bool vec = (p.in_f & 3u) == 0 && ((uintptr_t)out & (OUT == 0 ? 3u : 7u)) == 0;
    const bool wide = OUT == 0 && ((p.in_f | (uint32_t)(uintptr_t)out) & 15u) == 0;
    if (wide) {
        p6_quad_transpose(u, lane);
        p6_quad_transpose(v, lane);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {                    // row g, row g + 8
        const uint32_t row = R * kTileRows + (lane >> 2) + 8 * s;
        if (row >= p.out_f) continue;
        uint32_t r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = p6_codes4(u[j] >> 6 * s, v[j] >> 6 * s);
        if (wide) {                                  // columns 16 (lane & 3) .. + 15
            const uint32_t col0 = kbi * kTileCols + 16 * (lane & 3);
            if (col0 < p.in_f) *(uint4 *)((int8_t *)out + (size_t)row * p.in_f + col0) = make_uint4(r[0], r[1], r[2], r[3]);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {                // columns col0 .. col0 + 3
            const uint32_t col0 = kbi * kTileCols + 16 * j + 4 * (lane & 3);
            const size_t o = (size_t)row * p.in_f + col0;
            uint32_t w[2];
            if (OUT == 1) {
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    w[k] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn((float)(int8_t)(r[j] >> 16 * k) * sc)) |
                           (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn((float)(int8_t)(r[j] >> (16 * k + 8)) * sc)) << 16;
            }
            if (vec && col0 < p.in_f) {
                if (OUT == 0) *(uint32_t *)((char *)out + o) = r[j];
                else *(uint2 *)((char *)out + 2 * o) = make_uint2(w[0], w[1]);
            } else {
                for (uint32_t c = 0; c < 4u && col0 + c < p.in_f; ++c) {
                    if (OUT == 0) ((int8_t *)out)[o + c] = (int8_t)((r[j] >> (8 * c)) & 0xff);
                    else ((uint16_t *)out)[o + c] = (uint16_t)((w[c >> 1] >> (16 * (c & 1))) & 0xffff);
                }
            }
        }
    }
}

// The outliers overwrite their placeholders (launched after k_p6_decode_plane on the same stream; one warp per
// block).  An entry carries the bf16 weight w = bf16(code * scale); the code is recovered from it exactly:
// neighbouring codes differ by scale >= |code * scale| / 127, more than one bf16 ulp (2^-7 relative), so no two
// codes share a weight and w / scale is within 0.25 of the code.
template <int OUT>
__global__ void __launch_bounds__(256) k_p6_decode_esc(P6 p, void *out)
{
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (b >= p.rt * p.kb) return;
    uint32_t R = b / p.kb, kbi = b - R * p.kb;
    float sc = __bfloat162float(p.scale[R * p.scale_stride]);
    for (int32_t j = p.blk_off[b] + lane; j < p.blk_off[b + 1]; j += 32) {
        uint32_t ent = p.esc[j];
        uint32_t row = R * kTileRows + ((ent >> 12) & 15u), col = kbi * kTileCols + (ent & 63u);
        if (row >= p.out_f || col >= p.in_f) continue;
        size_t o = (size_t)row * p.in_f + col;
        __nv_bfloat16 wv = __ushort_as_bfloat16((unsigned short)(ent >> 16));
        if (OUT == 1) ((__nv_bfloat16 *)out)[o] = wv;
        else ((int8_t *)out)[o] = (int8_t)__float2int_rn(__bfloat162float(wv) / sc);
    }
}

// ------------------------------------------------------------------ GEMV ----
constexpr int kP6Threads = 768;
constexpr int kP6Warps = kP6Threads / 32;
constexpr int kP6RingBytes = kP6Slots * kP6BlockBytes;                // 3072
constexpr int kP6TailTiles = 32;                                      // row tiles per CTA that the barrier-free tail tracks
constexpr int kP6TailBytes = kP6TailTiles * 12;                       // per tile: arrival counter + two words of plan
// Shared memory of one warp: ring, an outlier step's operand tiles (A: 2 x 16 x 16 bf16, zero between steps; B: 2 x 8 x
// 16), staged entries, two partial row tiles (16 sums at one activation row, else [32] float4).  A CTA: kP6Warps of
// these, the tail's plan, the activations.
template <bool MULTI>
struct P6Smem {
    static constexpr int kEntries = 128;                              // outlier entries a warp stages: five per block of a 24-block run
    static constexpr int kTiles = kP6RingBytes, kStage = kTiles + 1024 + 512;
    static constexpr int kParts = kStage + kEntries * 4, kPart = MULTI ? 32 * 16 : 16 * 4;
    static constexpr int kWarp = kParts + 2 * kPart;
    static constexpr int kFixed = kP6Warps * kWarp + kP6TailBytes;
    static_assert(kWarp % 128 == 0 && kStage % 16 == 0, "per-warp shared memory keeps its alignment");
};

__device__ __forceinline__ void p6_cp16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// the same copy for the lanes with `on` set (a predicate, not a branch: the warp stays converged)
__device__ __forceinline__ void p6_cp16_if(uint32_t dst, const void *src, bool on)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}"
                 ::"r"(dst), "l"(src), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ uint4 p6_lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint2 p6_lds64(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t p6_lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void p6_ldmatrix(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// two bf16 numbers 160 + code -> the two weights; s2: the scale in both halves.  The product is a fused multiply-add of +0:
// the same value, rounded once, but +0.0 for code 0 and a scale of either sign, so that a placeholder is all zero bits.
__device__ __forceinline__ uint32_t p6_weights(uint32_t v, uint32_t s2)
{
    uint32_t w;
    asm("{\n\t.reg .b32 c;\n\tadd.rn.bf16x2 c, %1, %2;\n\tfma.rn.bf16x2 %0, c, %3, %4;\n\t}"
        : "=r"(w) : "r"(v), "r"(0xC320C320u), "r"(s2), "r"(0u));
    return w;
}
// a lane's six plane words -> its 16 pairs of weights; e2 = 0x43004300 (kept in a register by the caller)
__device__ __forceinline__ void p6_unpack(const uint32_t (&w)[6], uint32_t e2, uint32_t s2, uint32_t (&f)[16])
{
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        f[2 * k] = p6_weights(p6_and_or(w[k], 0x003F003Fu, e2), s2);
        f[2 * k + 1] = p6_weights(p6_and_or(w[k] >> 6, 0x003F003Fu, e2), s2);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t v = p6_and_or(w[i] >> 12, 0x000F000Fu, e2);
        v = p6_and_or(w[4 + (i >> 1)] >> (8 + 2 * (i & 1)), 0x00300030u, v);
        f[12 + i] = p6_weights(v, s2);
    }
}
__device__ __forceinline__ uint32_t p6_scale2(const __nv_bfloat16 &s)
{
    const uint32_t b = (uint32_t)__bfloat16_as_ushort(s);
    return b | b << 16;
}

// Where the outputs of a row-parallel shard go instead of y: into this rank's slot of EVERY rank's all-reduce buffer
// (see ixb_allreduce.cuh: slots [2 parities][world][n_max] of {fp32 value, call number} words), as plain peer stores
// straight from the GEMV's epilogue.  world == 0: no push, the outputs are written to y.
struct P6Push {
    uint2 *slots[8];              // every rank's slots, as seen from this rank
    const uint2 *mine;            // this rank's own slots (slots[rank])
    uint32_t *epoch;              // this rank's call counters (whoever finishes the exchange advances them)
    uint32_t world, rank, n_max;
    // fin != 0: the GEMV also finishes the exchange itself.  When a warp is done with its blocks it takes its share
    // of the outputs, waits (bounded) for every rank's words of this call in this rank's own buffer, adds them in
    // rank order (+ bias) and writes y; the last warp of the grid to get there advances the call counters.
    uint32_t fin, counters, spin_limit;
    uint32_t *err;                // the buffer's error word
    uint32_t *done;               // scratch word counting finished warps, zero between launches
};

template <bool V>
struct P6Flag { static constexpr bool value = V; };

// one output (activation row m, weight row `row`): to y (+ bias), or as a marked word to every rank
__device__ __forceinline__ void p6_put_out(const P6Push &push, uint32_t e, uint32_t out_f, uint32_t m, uint32_t row, float v,
                                           const __nv_bfloat16 *__restrict__ bias, void *y, int y_f32)
{
    const size_t o = (size_t)m * out_f + row;
    if (push.world) {
        const size_t at = ((size_t)((e & 1u) * push.world + push.rank)) * push.n_max + o;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if ((uint32_t)r >= push.world) break;
            asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(push.slots[r] + at), "r"(__float_as_uint(v)), "r"(e) : "memory");
        }
    } else if (y_f32) {
        ((float *)y)[o] = bias ? v + __bfloat162float(bias[row]) : v;
    } else {
        __nv_bfloat16 hv = __float2bfloat16_rn(v);
        if (bias) hv = __hadd(hv, bias[row]);
        ((__nv_bfloat16 *)y)[o] = hv;
    }
}

__device__ __forceinline__ void p6_store_tile(const P6Push &push, uint32_t e, uint32_t out_f, uint32_t R, int lane,
                                              const float (&c)[4], uint32_t m_rows, const __nv_bfloat16 *__restrict__ bias,
                                              void *y, int y_f32)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t m = 2u * t + (i & 1), row = R * kTileRows + g + 8 * (i >> 1);
        if (m >= m_rows || row >= out_f) continue;
        p6_put_out(push, e, out_f, m, row, c[i], bias, y, y_f32);
    }
}

// one half of a lane's C fragment: row g + 8 h of the tile, activation rows 2 t and 2 t + 1
__device__ __forceinline__ void p6_store_pair(const P6Push &push, uint32_t e, uint32_t out_f, uint32_t R, int lane, int h,
                                              const float (&v)[2], uint32_t m_rows, const __nv_bfloat16 *__restrict__ bias,
                                              void *y, int y_f32)
{
    const int g = lane >> 2, t = lane & 3;
    const uint32_t row = R * kTileRows + g + 8 * h;
    if (row >= out_f) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t m = 2u * t + i;
        if (m >= m_rows) continue;
        p6_put_out(push, e, out_f, m, row, v[i], bias, y, y_f32);
    }
}

// The exchange's second half, by the same kernel: every thread of the grid looks after one pair of outputs (the first n / 2
// threads have one).  The words of this rank come from this very launch -- from CTAs that are all resident, one per SM -- and the
// other ranks' from their launches of the same call.
template <int THREADS>
__device__ __forceinline__ void p6_finish_exchange(const P6Push &push, uint32_t push_e, uint32_t out_f, uint32_t m_rows,
                                                   const __nv_bfloat16 *__restrict__ bias, void *y, int y_f32)
{
    const uint32_t n = m_rows * out_f, i = (blockIdx.x * THREADS + threadIdx.x) * 2u, W = push.world;
    if (i < n) {
        const uint32_t limit = *(volatile uint32_t *)push.err ? 64u : push.spin_limit;
        const uint2 *mine = push.mine;
        float o0 = 0.f, o1 = 0.f;
        for (uint32_t s = 0; s < W; ++s) {
            const uint2 *src = mine + ((size_t)((push_e & 1u) * W + s)) * push.n_max + i;
            uint32_t v0, m0, v1, m1, polls = 0;
            for (;;) {
                asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v0), "=r"(m0), "=r"(v1), "=r"(m1) : "l"(src) : "memory");
                if (m0 == push_e && m1 == push_e) break;
                __nanosleep(20);
                if (++polls > limit) {
                    *push.err = 1u + s;                // sender s never arrived: the result is wrong, not a hang
                    break;
                }
            }
            o0 += __uint_as_float(v0);
            o1 += __uint_as_float(v1);
        }
        const uint32_t r0 = i % out_f;               // n is even and so is out_f: both values belong to one activation row
        if (y_f32) {
            float2 r;
            r.x = bias ? o0 + __bfloat162float(bias[r0]) : o0;
            r.y = bias ? o1 + __bfloat162float(bias[r0 + 1]) : o1;
            *(float2 *)((float *)y + i) = r;
        } else {
            __nv_bfloat16 h0 = __float2bfloat16_rn(o0), h1 = __float2bfloat16_rn(o1);
            if (bias) {
                h0 = __hadd(h0, bias[r0]);
                h1 = __hadd(h1, bias[r0 + 1]);
            }
            *(__nv_bfloat162 *)((__nv_bfloat16 *)y + i) = __halves2bfloat162(h0, h1);
        }
    }
    // the last warp of the grid to get here advances the call counters: by now every CTA has read them
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) {
        __threadfence();
        if (atomicAdd(push.done, 1u) == gridDim.x * (THREADS / 32u) - 1u) {
            for (uint32_t k = 0; k < push.counters; ++k) push.epoch[k] = push_e;
            *push.done = 0;
        }
    }
}

// n elements cut into `parts` contiguous parts, the first r = n % parts of them one longer than q = n / parts:
// first element of part i, and the part that holds element pos (no 64-bit arithmetic, no division on the way in)
__device__ __forceinline__ uint32_t p6_begin(uint32_t i, uint32_t q, uint32_t r) { return i * q + min(i, r); }
__device__ __forceinline__ uint32_t p6_part_of(uint32_t pos, uint32_t q, uint32_t r)
{
    const uint32_t big = r * (q + 1u);
    return pos < big ? pos / (q + 1u) : r + (pos - big) / q;      // q > 0 whenever pos >= big
}

// An outlier's place in an image [4 mma][32 lanes][4 registers] of a block's registers (the inverse of p6_elem): row r, column c of
// the block sit in lane 4 (r & 7) + ((c >> 2) & 3), pair 4 (c >> 4) + 2 ((c >> 1) & 1) + (r >> 3), half c & 1.
__device__ __forceinline__ uint32_t p6_image_at(uint32_t e)
{
    const uint32_t r = (e >> 12) & 15u, c = e & 63u;
    return (((c >> 4) * 32u + 4u * (r & 7u) + ((c >> 2) & 3u)) * 4u + 2u * ((c >> 1) & 1u) + (r >> 3)) * 4u + 2u * (c & 1u);
}

// An outlier's register in k_p6_decode_bf16: row r, column c of the block sit in lane 4 (r & 7) + (c >> 4), register
// 8 (r >> 3) + ((c & 15) >> 1), half c & 1.
__device__ __forceinline__ uint32_t p6_row_lane(uint32_t e) { return 4u * ((e >> 12) & 7u) + ((e >> 4) & 3u); }
__device__ __forceinline__ uint32_t p6_row_reg(uint32_t e) { return 8u * ((e >> 15) & 1u) + ((e >> 1) & 7u); }

// layout -> bf16 weights in one pass, with the GEMV's own conversion.  Bound by memory (2.76 bytes per weight, the stores to an
// output that stays in L2 faster than that).  The plane is requested before the offsets; the words of a quad's lanes are dealt out
// while they are packed (8 shuffles; as weights it takes 16), so that a lane has 16 consecutive columns of two rows and every weight
// is stored once, a 32-byte sector per lane and row where the alignment allows.  One or two outliers go straight into their
// lane's register, more through an image of the lanes' registers in shared memory; eight CTAs per SM are in flight (six: 17408 x 5120
// 40.7 us, 12288 x 2048 10.9).  In a graph, every launch to its own output / all to one that stays in L2, as a prompt's do: 17408 x
// 5120 40.1 / 40.0 us, 12288 x 2048 13.5 / 10.3, 2048 x 6144 8.0 / 6.5, 4096 x 2048 5.9 / 4.7; with the weights turned round in a
// tile of shared memory 39.8 / 39.8, 13.5 / 11.1, 8.0 / 6.8, 5.8 / 4.8; on the layout whose lanes held 16 columns as it was 39.8 /
// 39.8, 13.2 / 10.3, 7.8 / 6.6, 6.0 / 4.5.
// Needs in_f % 8 == 0 and a 16-byte aligned output.  One warp per block.
__global__ void __launch_bounds__(256, 8) k_p6_decode_bf16(P6 p, __nv_bfloat16 *out)
{
    __shared__ uint4 images[8 * 128];
    const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (b >= p.rt * p.kb) return;                    // whole warps leave together
    const unsigned char *blk = p.plane + (size_t)b * kP6BlockBytes;
    const uint4 a = __ldg((const uint4 *)blk + lane);
    const uint2 a2 = __ldg((const uint2 *)(blk + 512) + lane);
    const int32_t lo = __ldg(p.blk_off + b), hi = __ldg(p.blk_off + b + 1);
    const uint32_t R = b / p.kb, kbi = b - R * p.kb;
    const uint32_t s2 = p6_scale2(p.scale[R * p.scale_stride]);
    uint32_t u[4], v[4];
    p6_pair_words(a, a2, u, v);
    p6_quad_transpose(u, lane);
    p6_quad_transpose(v, lane);
    uint32_t f[16];                                  // row g and row g + 8, columns 16 (lane & 3) .. + 15
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        f[2 * t] = p6_weights(p6_and_or(u[t], 0x003F003Fu, 0x43004300u), s2);
        f[2 * t + 1] = p6_weights(p6_and_or(v[t], 0x003F003Fu, 0x43004300u), s2);
        f[8 + 2 * t] = p6_weights(p6_and_or(u[t] >> 6, 0x003F003Fu, 0x43004300u), s2);
        f[8 + 2 * t + 1] = p6_weights(p6_and_or(v[t] >> 6, 0x003F003Fu, 0x43004300u), s2);
    }
    // placeholders are +0.0, so OR-ing the outlier weights in is exact
    if (hi - lo <= 2) {
        for (int32_t j = lo; j < hi; ++j) {
            const uint32_t e = __ldg(p.esc + j), at = p6_row_reg(e);
            const uint32_t w = (uint32_t)lane == p6_row_lane(e) ? ((e & 1u) ? e & 0xFFFF0000u : e >> 16) : 0u;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (at == (uint32_t)q) f[q] |= w;
        }
    } else {
        uint4 *img = images + (threadIdx.x >> 5) * 128;                 // [4 quads of registers][32 lanes]
#pragma unroll
        for (int q = 0; q < 4; ++q) img[q * 32 + lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        const uint32_t img_s = (uint32_t)__cvta_generic_to_shared(img);
        for (int32_t j = lo + lane; j < hi; j += 32) {
            const uint32_t e = __ldg(p.esc + j), at = p6_row_reg(e);
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(img_s + ((at >> 2) * 32u + p6_row_lane(e)) * 16u + (at & 3u) * 4u + (e & 1u) * 2u), "h"((unsigned short)(e >> 16)) : "memory");
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 w = img[q * 32 + lane];
            f[4 * q] |= w.x;
            f[4 * q + 1] |= w.y;
            f[4 * q + 2] |= w.z;
            f[4 * q + 3] |= w.w;
        }
    }
    const bool wide = (p.in_f & 15u) == 0 && ((uintptr_t)out & 31u) == 0;       // a lane's 32 bytes of a row are one sector
    const uint32_t col0 = kbi * kTileCols + 16u * (lane & 3);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const uint32_t row = R * kTileRows + (lane >> 2) + 8u * s;
        if (row >= p.out_f || col0 >= p.in_f) continue;
        __nv_bfloat16 *dst = out + (size_t)row * p.in_f + col0;
        if (wide) {
            const uint32_t r[8] = {f[8 * s], f[8 * s + 1], f[8 * s + 2], f[8 * s + 3], f[8 * s + 4], f[8 * s + 5], f[8 * s + 6], f[8 * s + 7]};
            st_sector(dst, r);
        } else {                                     // in_f % 8 == 0: eight columns or none
            ((uint4 *)dst)[0] = make_uint4(f[8 * s], f[8 * s + 1], f[8 * s + 2], f[8 * s + 3]);
            if (col0 + 16u <= p.in_f) ((uint4 *)dst)[1] = make_uint4(f[8 * s + 4], f[8 * s + 5], f[8 * s + 6], f[8 * s + 7]);
        }
    }
}

// The nb blocks, in (row tile, column block) order, are cut into gridDim.x contiguous CTA ranges and every CTA range
// into kP6Warps runs.  The CTA ranges are counted in units of `unit` blocks (cq, cr = units / and % gridDim.x):
// unit = 1 balances the CTAs to one block, and row tiles at range boundaries are finished across CTAs; unit = blocks
// per row tile gives every CTA whole row tiles, so nothing crosses CTAs (the host picks the cheaper of the two).  A run is walked segment by segment (its part of one row
// tile): the segment's outliers are added first, from the entries staged in shared memory, then its blocks stream
// through the warp's cp.async ring.  Row tiles that a run covers completely are written straight to y; partial
// tiles are summed per CTA in warp order; a tile shared between CTAs goes through cta_slots and a ticket, the
// last arriver sums the slots in CTA order and clears them.  tickets[] (gridDim.x + 1 words) and cta_slots must be
// zero before the first launch and are left zero, so one scratch buffer serves launches of any shape in turn.  XS = 1: activations staged in shared memory (bf16, padded rows); XS = 0: read from
// global memory.
template <int XS, int MR>
__global__ void __launch_bounds__(kP6Threads, 1)
k_p6_mma(P6 p, const __nv_bfloat16 *__restrict__ x, uint32_t m_rows, const __nv_bfloat16 *__restrict__ bias, void *y,
         int y_f32, float4 *cta_slots, uint32_t *tickets, uint32_t nb, uint32_t xstride, uint32_t cq, uint32_t cr, uint32_t unit,
         P6Push push)
{
    extern __shared__ __align__(128) unsigned char p6_smem[];
    constexpr bool MULTI = MR > 1;
    using SM = P6Smem<MULTI>;
    __nv_bfloat16 *xs = (__nv_bfloat16 *)(p6_smem + SM::kFixed);                         // [m_rows][xstride]

    const int lane = threadIdx.x & 31;
    const int wid = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);   // the same in every lane, and known to be
    const int g = lane >> 2, t = lane & 3;
    const uint32_t KB = p.kb;
    unsigned char *wsm = p6_smem + wid * SM::kWarp;
    uint32_t *estage = (uint32_t *)(wsm + SM::kStage);                 // the run's first SM::kEntries outlier entries

    const uint32_t cb0 = p6_begin(blockIdx.x, cq, cr) * unit, cb1 = p6_begin(blockIdx.x + 1, cq, cr) * unit;
    const uint32_t L = cb1 - cb0, wq = L / kP6Warps, wr = L - wq * kP6Warps;
    const uint32_t b_begin = cb0 + p6_begin(wid, wq, wr), b_end = cb0 + p6_begin(wid + 1, wq, wr);
    const bool active = b_begin < b_end;
    // ---- plan of the tail, made while nothing else can run yet.  For every row tile R0 + i that this CTA touches
    // (fast path: at most kP6TailTiles): which warps' runs meet it, whether it lies inside the CTA's range, how many
    // partial sums will arrive (0: one run covers it and writes y itself), and the CTAs that share it.
    uint32_t *tcnt = (uint32_t *)(p6_smem + kP6Warps * SM::kWarp);   // [kP6TailTiles] arrivals
    uint32_t *tplan = tcnt + kP6TailTiles;                             // [kP6TailTiles][2]
    const uint32_t Rc0 = cb0 / KB, Rc1 = L ? (cb1 - 1u) / KB : Rc0;
    const bool fast_tail = L != 0 && Rc1 - Rc0 < (uint32_t)kP6TailTiles;
    if (fast_tail && lane == 0) {
        for (uint32_t i = wid; i <= Rc1 - Rc0; i += kP6Warps) {
            const uint32_t t0 = (Rc0 + i) * KB, t1 = t0 + KB;
            const uint32_t inside = t0 >= cb0 && t1 <= cb1;
            const uint32_t wlo = p6_part_of(max(t0, cb0) - cb0, wq, wr), whi = p6_part_of(min(t1, cb1) - 1 - cb0, wq, wr);
            const uint32_t need = inside && wlo == whi ? 0u : whi - wlo + 1u;
            uint32_t clo = 0, span = 0;
            if (!inside) {
                clo = p6_part_of(t0, cq, cr);
                span = p6_part_of(t1 - 1u, cq, cr) - clo;
            }
            tcnt[i] = 0;
            tplan[2 * i] = wlo | whi << 8 | need << 16 | inside << 24;
            tplan[2 * i + 1] = clo | span << 16;
        }
    }
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(wsm);
    const uint32_t d16 = ring_s + lane * 16;
    const unsigned char *n16 = p.plane + (size_t)b_begin * kP6BlockBytes + lane * 16;    // this lane's next chunk to fetch
    uint32_t pf_left = b_end - b_begin;                                                  // blocks of the run not yet requested

    // Everything up to griddepcontrol.wait reads only the layer's own (constant) buffers.  When the launch carries
    // the programmatic-stream-serialization attribute this part overlaps the tail of the kernel before it in the
    // stream; without the attribute the two griddepcontrol instructions do nothing.
    asm volatile("griddepcontrol.launch_dependents;");
    // ---- copy group A: the run's first three blocks and the activations
    int32_t j_begin = 0, j_end = 0;
    if (active) {
        j_begin = __ldg(p.blk_off + b_begin);
        j_end = __ldg(p.blk_off + b_end);
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const bool more = pf_left != 0;               // nothing is fetched past the end of the run
            p6_cp16_if(d16 + s * kP6BlockBytes, n16, more);
            p6_cp16_if(d16 + s * kP6BlockBytes + 512, n16 + 512, more && lane < 16);
            n16 += kP6BlockBytes;
            pf_left -= more ? 1u : 0u;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) ((uint4 *)(wsm + SM::kTiles))[k * 32 + lane] = make_uint4(0, 0, 0, 0);
    }
    // the scale of the run's first row tile and of the one after it (a fused tensor has one per row tile); the
    // walk below always holds the next tile's scale one segment ahead, so the load is never waited for
    uint32_t e2, s2 = 0;
    uint32_t sc_cur = 0, sc_next = 0;
    {
        if (p.scale_stride) {                                          // (uniform) a fused tensor: one scale per row tile
            const uint32_t R0 = min(b_begin / KB, p.rt - 1u);
            sc_cur = (uint32_t)__bfloat16_as_ushort(p.scale[R0]);
            sc_next = (uint32_t)__bfloat16_as_ushort(p.scale[min(R0 + 1u, p.rt - 1u)]);
        } else {
            sc_cur = (uint32_t)__bfloat16_as_ushort(p.scale[0]);
        }
        asm volatile("mov.b32 %0, 0x43004300;" : "=r"(e2));            // opaque, so that it stays a register operand
    }
    auto set_scale = [&](uint32_t bits) { s2 = bits | bits << 16; };
    set_scale(sc_cur);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // a pushing launch marks its words with the number of this all-reduce call: one more than the counter that the
    // finishing kernel of the call before left (that kernel is complete: it is ahead of this one in the stream)
    const uint32_t push_e = push.world ? __ldcg(push.epoch) + 1u : 0u;
    if (XS) {
        // whole 16-byte chunks by cp.async; ragged ends are written with plain stores
        const uint32_t chunks = KB * (kTileCols / 8);
        const uint32_t xs_s = (uint32_t)__cvta_generic_to_shared(xs);
        const bool vec = (p.in_f & 7u) == 0;
        for (uint32_t m = 0; m < m_rows; ++m) {
            for (uint32_t k8 = threadIdx.x * 8u; k8 < chunks * 8u; k8 += kP6Threads * 8u) {
                if (vec && k8 + 8u <= p.in_f) {
                    p6_cp16(xs_s + (m * xstride + k8) * 2u, x + (size_t)m * p.in_f + k8);
                } else {
                    unsigned short e[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        e[j] = k8 + j < p.in_f ? __bfloat16_as_ushort(x[(size_t)m * p.in_f + k8 + j]) : (unsigned short)0;
                    *(uint4 *)(xs + (size_t)m * xstride + k8) =
                        make_uint4(e[0] | ((uint32_t)e[1] << 16), e[2] | ((uint32_t)e[3] << 16), e[4] | ((uint32_t)e[5] << 16),
                                   e[6] | ((uint32_t)e[7] << 16));
                }
            }
        }
    }
    cp_async_commit();
    // ---- copy group E: the run's outlier entries, from the 16-byte boundary at or below the first one (their
    // offsets were requested at the top).  From here on every block iteration adds exactly one group, so the
    // entries are complete once three block iterations have waited.
    const int32_t j_base = j_begin & ~3;
    if (active) {
        const uint32_t es = (uint32_t)__cvta_generic_to_shared(estage);
#pragma unroll
        for (int q = 0; q < (SM::kEntries + 127) / 128; ++q) {
            const int32_t ch = j_base + (q * 32 + lane) * 4;
            if (ch < j_end && (q * 32 + lane) * 4 < SM::kEntries) p6_cp16(es + (q * 32 + lane) * 16, p.esc + ch);
        }
    }
    cp_async_commit();
    cp_async_wait<1>();                              // group A has landed for this thread
    __syncthreads();                                 // ... and for the CTA

    // Row tile R is complete in this CTA: sum the partial tiles of warps wlo .. whi in warp order; a tile inside the
    // CTA's range is written to y, a tile shared with other CTAs (clo .. clo + span) is finished across them.
    auto finish_tile = [&](uint32_t R, uint32_t wlo, uint32_t whi, bool inside, uint32_t clo, uint32_t span) {
        const uint32_t t0 = R * KB;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        // (eight warps' parts requested together: one after the other, 24 of them were 0.5 us of a small layer's 5.4)
        for (uint32_t w0 = wlo; w0 <= whi; w0 += 8u) {
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t w = w0 + k, wb = p6_begin(w, wq, wr);
                v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (w > whi || wb == p6_begin(w + 1, wq, wr)) continue;  // not of this tile; a warp without blocks
                // the run of warp w meets tile R: R is its first tile unless the run began in the tile before
                const unsigned char *part = p6_smem + w * SM::kWarp + SM::kParts + (cb0 + wb >= t0 ? 0 : SM::kPart);
                if (MULTI) {
                    v[k] = ((const float4 *)part)[lane];
                } else {                                                // only activation row 0 counts: lanes t == 0, c[0] and c[2]
                    v[k].x = ((const float *)part)[g];
                    v[k].z = ((const float *)part)[g + 8];
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                s.x += v[k].x; s.y += v[k].y; s.z += v[k].z; s.w += v[k].w;
            }
        }
        if (inside) {
            const float cc[4] = {s.x, s.y, s.z, s.w};
            p6_store_tile(push, push_e, p.out_f, R, lane, cc, m_rows, bias, y, y_f32);
            return;
        }
        const uint32_t chi = clo + span;
        if (span == 1u) {
            // Shared by exactly two CTAs (the usual case): one atomic exchange per 64-bit word carries the
            // partial sums themselves -- no slot store, fence, ticket and slot load, a single round trip to L2.
            // A lane swaps its two words (row g: c[0], c[1]; row g + 8: c[2], c[3]), XOR-ed with a constant so
            // that a deposit is never the all-zero "empty" word, into the tile's area.  Whoever finds the
            // other CTA's deposit adds it to its own values (a + b = b + a bit for bit, so it does not matter
            // which of the two that is, word by word), stores the outputs and empties the word again.
            unsigned long long *w2 = (unsigned long long *)(cta_slots + ((size_t)chi * 2) * 32 + lane);
            const unsigned long long K = 0x7FC0DEAD7FC0DEADull;
            const float mine[4] = {s.x, s.y, s.z, s.w};
            unsigned long long got[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned long long dep =
                    ((unsigned long long)__float_as_uint(mine[2 * h + 1]) << 32 | __float_as_uint(mine[2 * h])) ^ K;
                got[h] = atomicExch(w2 + h, dep);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (got[h] == 0ull) continue;                            // first to arrive for this word
                const unsigned long long o = got[h] ^ K;
                const float v[2] = {mine[2 * h] + __uint_as_float((uint32_t)o),
                                    mine[2 * h + 1] + __uint_as_float((uint32_t)(o >> 32))};
                p6_store_pair(push, push_e, p.out_f, R, lane, h, v, m_rows, bias, y, y_f32);
                w2[h] = 0ull;
            }
            return;
        }
        // shared by three or more CTAs: publish this CTA's sum, take a ticket; the last one finishes the tile
        cta_slots[((size_t)blockIdx.x * 2 + (R == Rc0 ? 0 : 1)) * 32 + lane] = s;
        __threadfence();
        __syncwarp();
        uint32_t prev = 0;
        if (lane == 0) prev = atomicAdd(tickets + clo + 1, 1u);
        prev = __shfl_sync(0xffffffffu, prev, 0);
        if (prev != span) return;
        // the other CTAs' slots were fenced before their tickets; they are read from L2 (ld.global.cg), which
        // every SM shares, so nothing cached on this SM can be stale
        float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t cc = clo; cc <= chi; ++cc) {
            float4 *sl = cta_slots + ((size_t)cc * 2 + (p6_begin(cc, cq, cr) >= t0 ? 0 : 1)) * 32 + lane;
            z.x += __ldcg(&sl->x); z.y += __ldcg(&sl->y); z.z += __ldcg(&sl->z); z.w += __ldcg(&sl->w);
            // the slot goes back to zero: a later launch of another shape uses the same words for its two-CTA
            // hand-over, where any non-zero word counts as a deposit
            __stcg(sl, make_float4(0.f, 0.f, 0.f, 0.f));
        }
        const float cc4[4] = {z.x, z.y, z.z, z.w};
        p6_store_tile(push, push_e, p.out_f, R, lane, cc4, m_rows, bias, y, y_f32);
        if (lane == 0) tickets[clo + 1] = 0;
    };
    // Fast tail: a warp that leaves a partial row tile behind counts itself in; the warp that completes the count
    // finishes the tile at once -- no CTA-wide barrier, nobody waits for an unrelated slow warp.
    auto tile_arrive = [&](uint32_t R) {
        const uint32_t i = R - Rc0;
        __syncwarp();                                                    // all lanes' parts are written
        uint32_t prev = 0;
        if (lane == 0) {
            __threadfence_block();
            prev = atomicAdd(tcnt + i, 1u);
        }
        prev = __shfl_sync(0xffffffffu, prev, 0);
        const uint32_t w0 = tplan[2 * i], w1 = tplan[2 * i + 1];
        if (prev + 1u != ((w0 >> 16) & 0xffu)) return;
        __threadfence_block();
        finish_tile(R, w0 & 0xffu, (w0 >> 8) & 0xffu, (w0 >> 24) & 1u, w1 & 0xffffu, w1 >> 16);
    };

    if (active) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t R = b_begin / KB;
        const uint32_t R_first = R;
        // this lane's activations: row min(g, m_rows - 1) (rows beyond m_rows only feed unused C columns)
        const uint32_t xrow = min((uint32_t)g, m_rows - 1u);
        const __nv_bfloat16 *xg = x + (size_t)xrow * p.in_f + 4 * t;                                   // XS = 0
        const uint32_t xs_l = (uint32_t)__cvta_generic_to_shared(xs) + (xrow * xstride + 4 * t) * 2u;    // XS = 1
        uint32_t cs = 0, is = 3 * kP6BlockBytes;     // byte offsets of the ring slot to consume next / to refill next
        const uint32_t d8 = ring_s + 512 + lane * 8;
        const bool lo16 = lane < 16;
        float c1[4] = {0.f, 0.f, 0.f, 0.f};          // second accumulator set: two independent mma chains per block

        // blocks [b0, b1) of row tile R: fetch block b + 3 into the slot consumed last, take block b from its slot
        auto run = [&](uint32_t b0, uint32_t b1) {
            uint32_t xo = (b0 - R * KB) * (kTileCols * 2u);     // byte offset into the activation row
            for (uint32_t n = b1 - b0; n != 0; --n) {
                const bool more = pf_left != 0;                   // the last three iterations of a run fetch nothing
                p6_cp16_if(d16 + is, n16, more);
                p6_cp16_if(d16 + is + 512, n16 + 512, more && lo16);
                cp_async_commit();
                n16 += kP6BlockBytes;
                pf_left -= more ? 1u : 0u;
                uint2 xv[4];
                if (!XS) {                                        // requested ahead of the wait for the block
#pragma unroll
                    for (int j = 0; j < 4; ++j) xv[j] = *(const uint2 *)((const char *)xg + xo + 32 * j);
                }
                cp_async_wait<3>();                               // this lane's chunks of the block have landed ...
                __syncwarp();                                     // ... and so have the other lanes'
                const uint4 a = p6_lds128(d16 + cs);
                const uint2 a2 = p6_lds64(d8 + cs);
                if (XS) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) xv[j] = p6_lds64(xs_l + xo + 32u * j);
                }
                const uint32_t w[6] = {a.x, a.y, a.z, a.w, a2.x, a2.y};
                uint32_t f[16];
                p6_unpack(w, e2, s2, f);
                p6_mma(c, f[0], f[1], f[2], f[3], xv[0].x, xv[0].y);
                p6_mma(c1, f[4], f[5], f[6], f[7], xv[1].x, xv[1].y);
                p6_mma(c, f[8], f[9], f[10], f[11], xv[2].x, xv[2].y);
                p6_mma(c1, f[12], f[13], f[14], f[15], xv[3].x, xv[3].y);
                is = cs;
                cs = cs == (uint32_t)(3 * kP6BlockBytes) ? 0u : cs + (uint32_t)kP6BlockBytes;
                xo += kTileCols * 2u;
            }
        };

        // Outliers of blocks [sb, sb + 64) at most, all in row tile R: entries [jlo, jhi), 32 per step, one per lane, as
        // the k index of two more mmas.  A lane writes its weight into its column of A (at the entry's row) and the
        // activations it meets into its column of B (one per activation row); ldmatrix turns the tiles into operands.
        // So an entry is looked at once for all activation rows, every row of activations gets the same bits alone or
        // beside others, and no sums over lanes are left.  (Products on the CUDA cores and sums over the lanes, row by
        // row of activations: 17408 x 5120 19 us at two rows and 37 us at eight, against 17.4 and 18.4 us now; at one row,
        // with as many outliers, the two forms differ by less than 10 %.)
        // The zeros of A turn infinite and NaN activations into NaN in rows that they do not reach: if a sum is not finite
        // afterwards, the steps are taken again with those activations as 0 in B and their products added one by one.
        const uint32_t tiles = (uint32_t)__cvta_generic_to_shared(wsm + SM::kTiles);
        const uint32_t my_a = tiles + (lane >> 4) * 512u + ((lane >> 3) & 1) * 256u + (lane & 7) * 2u;              // + row * 16
        const uint32_t my_b = tiles + 1024u + (lane >> 4) * 256u + ((lane >> 3) & 1) * 128u + (lane & 7) * 2u;      // + m * 16
        const uint32_t es = (uint32_t)__cvta_generic_to_shared(estage), pitch = XS ? xstride : p.in_f;
        uint32_t at = my_a;                                               // where this lane's weight lies
        auto outlier_steps = [&](uint32_t s64, const __nv_bfloat16 *xm, int32_t jlo, int32_t jhi, auto check) {
            constexpr bool kCheck = decltype(check)::value;
            unsigned short xv[MR];
            auto fetch = [&](int32_t j) -> uint32_t {                     // a lane beyond the end: weight 0, row 0, column 0
                uint32_t e = s64;
                if (j < jhi) {
                    const uint32_t rel = (uint32_t)(j - j_base);
                    e = rel < (uint32_t)SM::kEntries ? p6_lds32(es + rel * 4u) : __ldg(p.esc + j);
                }
                const __nv_bfloat16 *xe = xm + (((e & 0xFFFu) - s64) & 0xFFFu);
#pragma unroll
                for (int m = 0; m < MR; ++m) xv[m] = __bfloat16_as_ushort(xe[min((uint32_t)m, m_rows - 1u) * pitch]);
                return e;
            };
            uint32_t e = fetch(jlo + lane);
            for (int32_t j = jlo; j < jhi; j += 32) {
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"((unsigned short)0) : "memory");
                at = my_a + ((e >> 8) & 0xF0u);
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"((unsigned short)(e >> 16)) : "memory");
                bool bad = false;
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    if (kCheck && (xv[m] & 0x7F80u) == 0x7F80u) {
                        bad = true;
                        xv[m] = 0;
                    }
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(my_b + m * 16u), "h"(xv[m]) : "memory");
                }
                if (kCheck) {
                    for (uint32_t left = __ballot_sync(0xffffffffu, bad && j + lane < jhi); left; left &= left - 1u) {
                        const uint32_t ek = __shfl_sync(0xffffffffu, e, __ffs((int)left) - 1), row = (ek >> 12) & 15u;
                        const __nv_bfloat16 *xk = xm + (((ek & 0xFFFu) - s64) & 0xFFFu);
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t m = 2u * t + i;
                            if (m >= m_rows || (row & 7u) != (uint32_t)g) continue;
                            const float xf = __bfloat162float(xk[(size_t)m * pitch]);
                            if ((__float_as_uint(xf) & 0x7F800000u) != 0x7F800000u) continue;
                            const float v = __uint_as_float(ek & 0xFFFF0000u) * xf;
                            if (row < 8u) c[i] += v;
                            else c[2 + i] += v;
                        }
                        __syncwarp();
                    }
                }
                __syncwarp();                                             // the step's tiles are written
                e = fetch(j + 32 + lane);                                 // (the next step's loads are on their way)
                uint32_t a0[4], a1[4], bf[4];
                p6_ldmatrix(a0, tiles + lane * 16u);
                p6_ldmatrix(a1, tiles + 512u + lane * 16u);
                p6_ldmatrix(bf, tiles + 1024u + lane * 16u);
                p6_mma(c, a0[0], a0[1], a0[2], a0[3], bf[0], bf[1]);
                p6_mma(c1, a1[0], a1[1], a1[2], a1[3], bf[2], bf[3]);
                __syncwarp();                                             // every lane has read them
            }
        };
        auto outlier_pass = [&](uint32_t sb, int32_t jlo, int32_t jhi) {
            if (jlo >= jhi) return;                                       // warp uniform
            const uint32_t s64 = (sb & 63u) << 6;
            const __nv_bfloat16 *xm = (XS ? xs : x) + (sb - R * KB) * kTileCols;
            float before[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                before[i] = c[i];
                before[4 + i] = c1[i];
            }
            outlier_steps(s64, xm, jlo, jhi, P6Flag<false>());
            // the sum of the absolute values is NaN or infinite if one of the eight is
            const float all = fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) + fabsf(c[3]) + fabsf(c1[0]) + fabsf(c1[1]) + fabsf(c1[2]) + fabsf(c1[3]);
            if (__any_sync(0xffffffffu, !(all < INFINITY))) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    c[i] = before[i];
                    c1[i] = before[4 + i];
                }
                outlier_steps(s64, xm, jlo, jhi, P6Flag<true>());
            }
        };

        uint32_t b = b_begin;
        int32_t seg_j = j_begin;
        bool first = true;
        while (b < b_end) {
            const uint32_t seg_e = min((R + 1u) * KB, b_end);
            const bool whole = b == R * KB && seg_e == (R + 1u) * KB;
            const int32_t seg_je = seg_e == b_end ? j_end : __ldg(p.blk_off + seg_e);
            uint32_t mid = b;
            if (first) {
                // three block iterations complete the copy group of the entries for this lane, the warp barrier
                // for all lanes
                mid = min(b + 3u + 2u * ((uint32_t)wid & 7u), seg_e);      // (the warps' outlier passes do not all fall on the same moment)
                run(b, mid);
                if (mid - b < 3u) cp_async_wait<0>();
                __syncwarp();
                first = false;
            }
            for (uint32_t sb = b; sb < seg_e; sb += 64u) {
                const uint32_t se = min(sb + 64u, seg_e);
                const int32_t jlo = sb == b ? seg_j : __ldg(p.blk_off + sb);
                const int32_t jhi = se == seg_e ? seg_je : __ldg(p.blk_off + se);
                outlier_pass(sb, jlo, jhi);
            }
            run(mid, seg_e);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                c[i] += c1[i];
                c1[i] = 0.f;
            }
            if (whole) p6_store_tile(push, push_e, p.out_f, R, lane, c, m_rows, bias, y, y_f32);
            else {
                unsigned char *part = wsm + SM::kParts + (R == R_first ? 0 : SM::kPart);
                if (MULTI) {
                    ((float4 *)part)[lane] = make_float4(c[0], c[1], c[2], c[3]);
                } else if (t == 0) {
                    ((float *)part)[g] = c[0];
                    ((float *)part)[g + 8] = c[2];
                }
                if (fast_tail) tile_arrive(R);
            }
            c[0] = c[1] = c[2] = c[3] = 0.f;
            b = seg_e;
            seg_j = seg_je;
            ++R;
#ifndef IXB_P6_UNIFORM_SCALE
            if (p.scale_stride) {                                         // warp uniform
                set_scale(sc_next);
                sc_next = (uint32_t)__bfloat16_as_ushort(p.scale[min(R + 1u, p.rt - 1u) * p.scale_stride]);
            }
#endif
        }
    }
    cp_async_wait<0>();
    if (!fast_tail) __syncthreads();

    // ---- more row tiles per CTA than the fast tail tracks: after a CTA-wide barrier, sum the parts of every tile
    // that more than one run of this CTA (or another CTA) touched
    if (!fast_tail && L) {
        for (uint32_t R = Rc0 + wid; R <= Rc1; R += kP6Warps) {
            const uint32_t t0 = R * KB, t1 = t0 + KB;                   // the tile's blocks
            const bool inside = t0 >= cb0 && t1 <= cb1;
            const uint32_t wlo = p6_part_of(max(t0, cb0) - cb0, wq, wr), whi = p6_part_of(min(t1, cb1) - 1 - cb0, wq, wr);
            if (inside && wlo == whi) continue;                          // one run had all of it and wrote y itself
            uint32_t clo = 0, span = 0;
            if (!inside) {
                clo = p6_part_of(t0, cq, cr);
                span = p6_part_of(t1 - 1u, cq, cr) - clo;
            }
            finish_tile(R, wlo, whi, inside, clo, span);
        }
    }
    if (push.fin) p6_finish_exchange<kP6Threads>(push, push_e, p.out_f, m_rows, bias, y, y_f32);
}

}  // namespace ixb
