// Per-token glue of a decode step around the packed linears: the work between two GEMVs that the reference leaves
// to HuggingFace eager code and to fla's Triton kernels (ixrun/fla_patch.py:23-72; 63 of 138 ms per token in its own
// breakdown).  Batch-1 (up to 8 rows) kernels, one launch each, all of them usable inside a captured CUDA graph:
// positions and context lengths are read from device memory.
//
//   k_add_rmsnorm   h += delta (bf16), xn = rmsnorm(h) * w          residual add + the norm in front of the next GEMVs
//   k_swiglu        y = silu(g) * u                                 (the GEMV can also do this in its epilogue)
//   k_rope_kv       per-head q/k norm (optional), rotary embedding, K and V written into the static cache
//   k_attn_decode   one query per head over the static KV cache (grouped-query), split over the context; the last CTA
//                   joins the parts (k_attn_combine: in a launch of its own); optional sigmoid output gate
//   k_conv_update   causal depth-wise conv1d over the last K inputs of every channel + SiLU, state shifted
//   k_gdn_step      gated delta rule, one recurrent step per value head: state decay, delta update, read-out,
//                   gated RMSNorm of the head's output
//
// Arithmetic follows the eager reference path: inputs bf16, sums and transcendental functions in fp32, every value
// that the eager code would hold in a bf16 tensor is rounded to bf16 at the same place.
#pragma once
#include "ixb_common.cuh"

namespace ixb {

__device__ __forceinline__ float bf2f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float bfround(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float silu_f(float v) { return v / (1.f + __expf(-v)); }
__device__ __forceinline__ float sigmoid_f(float v) { return 1.f / (1.f + __expf(-v)); }

// sum over the CTA (blockDim.x a multiple of 32, at most 1024); every thread gets the result
__device__ __forceinline__ float cta_sum(float v, float *red)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    __syncthreads();                                   // red may still be read from an earlier call
    if (lane == 0) red[wid] = v;
    __syncthreads();
    float t = lane < nw ? red[lane] : 0.f;
    return warp_sum(t);
}

// ---------------------------------------------------------------- residual add + RMSNorm
// One CTA per row.  h (bf16, in/out) += delta (bf16, may be null); xn = bf16(h * rsqrt(mean(h^2) + eps)) * w.
// Generic form (any hidden size): two passes of scalar accesses.
__global__ void __launch_bounds__(1024)
k_add_rmsnorm_any(__nv_bfloat16 *h, const __nv_bfloat16 *__restrict__ delta, const __nv_bfloat16 *__restrict__ w, float eps,
                  __nv_bfloat16 *xn, uint32_t hidden)
{
    __shared__ float red[32];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const size_t base = (size_t)blockIdx.x * hidden;
    float ss = 0.f;
    for (uint32_t i = threadIdx.x; i < hidden; i += blockDim.x) {
        float v = bf2f(h[base + i]);
        if (delta) {
            v = bfround(v + bf2f(delta[base + i]));
            h[base + i] = __float2bfloat16_rn(v);
        }
        ss += v * v;
    }
    ss = cta_sum(ss, red);
    const float r = rsqrtf(ss / (float)hidden + eps);
    for (uint32_t i = threadIdx.x; i < hidden; i += blockDim.x) {
        const float v = bf2f(h[base + i]);             // this thread wrote it: visible to itself
        xn[base + i] = __hmul(__float2bfloat16_rn(v * r), w[i]);
    }
}

__device__ __forceinline__ void unpack8(const uint4 &r, float (&f)[8])
{
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        f[2 * j] = __uint_as_float(w[j] << 16);
        f[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        w[j] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f[2 * j])) |
               ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f[2 * j + 1])) << 16);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Where the residual's increment comes from when the row-parallel linear before this norm was sharded: the ranks'
// fp32 partial sums lie as marked words in this rank's exchange buffer (see ixb_allreduce.cuh; stored there by the
// epilogue of every rank's GEMV).  world == 0: the increment is the bf16 vector `delta` (or nothing).
struct NormExchange {
    const uint2 *mine;            // this rank's slots [2 parities][world][n_max]
    uint32_t *epoch;              // this rank's call counters
    uint32_t *err;
    uint32_t world, n_max, counters, spin_limit;
};

// Vector form: hidden a multiple of 8 and at most 8192 (5120 with an exchange); thread t keeps elements 8 t .. 8 t + 7 in registers, so the
// row is read once, with all loads in flight together; the norm weights are requested before the dependency wait.
// With an exchange (W > 0) the kernel is also the second half of the all-reduce: it waits (bounded) for every
// rank's words of this call, adds them in rank order and rounds the sum to bf16 (the value a separate finishing
// kernel would have written), then goes on as above; the last step advances the call counters.
constexpr int kNormExchangeThreads = 640;           // the exchange variant holds more registers: hidden <= 5120
template <int W>
__global__ void __launch_bounds__(W > 0 ? kNormExchangeThreads : 1024)
k_add_rmsnorm(__nv_bfloat16 *h, const __nv_bfloat16 *__restrict__ delta, NormExchange ex, const __nv_bfloat16 *__restrict__ w,
              float eps, __nv_bfloat16 *xn, uint32_t hidden)
{
    __shared__ float red[32];
    __shared__ uint32_t e_s;
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t t = threadIdx.x, i = 8u * t;
    const bool on = i < hidden;
    const size_t base = (size_t)blockIdx.x * hidden;
    uint4 wr = make_uint4(0, 0, 0, 0);
    if (on) wr = *(const uint4 *)(w + i);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
    uint32_t e = 0;
    if (W > 0) {
        if (t == 0) e_s = ex.epoch[blockIdx.x] + 1u;
        __syncthreads();
        e = e_s;
    }
    if (on) {
        const uint4 hr = *(const uint4 *)(h + base + i);
        unpack8(hr, v);
        if (W > 0) {
            const uint32_t limit = *(volatile uint32_t *)ex.err ? 64u : ex.spin_limit;
            const uint2 *src0 = ex.mine + (size_t)((e & 1u) * W) * ex.n_max + base + i;
            constexpr int GRP = W < 4 ? (W > 0 ? W : 1) : 4;       // senders polled together (their loads are in flight at once)
            float o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = 0.f;
#pragma unroll
            for (int s0 = 0; s0 < W; s0 += GRP) {
                uint32_t val[GRP][8], mark[GRP][8];
                for (uint32_t polls = 0;; ++polls) {
                    bool all = true;
#pragma unroll
                    for (int s = 0; s < GRP; ++s) {
                        const uint2 *src = src0 + (size_t)(s0 + s) * ex.n_max;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(val[s][2 * q]), "=r"(mark[s][2 * q]), "=r"(val[s][2 * q + 1]), "=r"(mark[s][2 * q + 1])
                                         : "l"(src + 2 * q) : "memory");
                    }
#pragma unroll
                    for (int s = 0; s < GRP; ++s)
#pragma unroll
                        for (int k = 0; k < 8; ++k) all = all && mark[s][k] == e;
                    if (all) break;
                    if (polls > limit) {
#pragma unroll
                        for (int s = 0; s < GRP; ++s)
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (mark[s][k] != e) *ex.err = 1u + (uint32_t)(s0 + s);   // that sender never arrived: wrong result, no hang
                        break;
                    }
                    __nanosleep(20);
                }
#pragma unroll
                for (int s = 0; s < GRP; ++s)                      // in rank order: the same bits on every rank
#pragma unroll
                    for (int k = 0; k < 8; ++k) o[k] += __uint_as_float(val[s][k]);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = bfround(v[k] + bfround(o[k]));
            *(uint4 *)(h + base + i) = pack8(v);
        } else if (delta) {
            float d[8];
            unpack8(*(const uint4 *)(delta + base + i), d);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = bfround(v[k] + d[k]);
            *(uint4 *)(h + base + i) = pack8(v);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
    ss = cta_sum(ss, red);
    const float r = rsqrtf(ss / (float)hidden + eps);
    if (on) {
        float wf[8], o[8];
        unpack8(wr, wf);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = bfround(v[k] * r) * wf[k];
        *(uint4 *)(xn + base + i) = pack8(o);
    }
    if (W > 0 && t == 0)
        for (uint32_t k = blockIdx.x; k < ex.counters; k += gridDim.x) ex.epoch[k] = e;   // all counters advance together
}

// ---------------------------------------------------------------- SwiGLU
// y [rows][cols] = silu(g) * u; g and u may be column slices of a wider matrix (row pitch in_stride elements, e.g. the
// two halves of a fused gate|up output).  vec: cols and in_stride multiples of 8 and 16-byte aligned pointers: eight
// values per thread; otherwise one value per thread.
__global__ void __launch_bounds__(128)
k_swiglu(const __nv_bfloat16 *__restrict__ g, const __nv_bfloat16 *__restrict__ u, __nv_bfloat16 *y, uint32_t rows,
         uint32_t cols, uint32_t in_stride, int vec)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (vec) {
        const uint32_t per_row = cols / 8u, r = t / per_row, c = (t - r * per_row) * 8u;
        if (r >= rows) return;
        float a[8], b[8], o[8];
        unpack8(*(const uint4 *)(g + (size_t)r * in_stride + c), a);
        unpack8(*(const uint4 *)(u + (size_t)r * in_stride + c), b);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = bfround(silu_f(a[k])) * b[k];
        *(uint4 *)(y + (size_t)r * cols + c) = pack8(o);
    } else {
        const uint32_t r = t / cols, c = t - r * cols;
        if (r >= rows) return;
        y[(size_t)r * cols + c] = __hmul(__float2bfloat16_rn(silu_f(bf2f(g[(size_t)r * in_stride + c]))), u[(size_t)r * in_stride + c]);
    }
}

// ---------------------------------------------------------------- q/k norm + RoPE + cache write
// grid (rows, q heads + kv heads), D / 2 threads.  Thread i of a head looks after the pair (i, i + D / 2) of the
// rotate-half convention; the first rot_dim elements are rotated with the caller's tables cos / sin [max_seq][rot_dim / 2]
// (the same fp32 tables as the eager path, so the results agree bit for bit), the rest pass through.
// q_norm / k_norm (per-head RMSNorm weights [D], may be null) are applied first.  q is rotated in place; k and v go
// into the caches [max_seq][kv heads][D].  batch_stride == 0: the rows are consecutive positions pos[0] + row of one
// sequence; batch_stride > 0: row r is the newest token of sequence r, at position pos[r] of the cache that starts
// batch_stride elements after the one before it.  Row pitches of q, k / v: q_stride, kv_stride elements.
__global__ void __launch_bounds__(128)
k_rope_kv(__nv_bfloat16 *q, const __nv_bfloat16 *__restrict__ k, const __nv_bfloat16 *__restrict__ v, const int32_t *pos,
          __nv_bfloat16 *k_cache, __nv_bfloat16 *v_cache, const __nv_bfloat16 *__restrict__ q_norm,
          const __nv_bfloat16 *__restrict__ k_norm, const float *__restrict__ cos_tab, const float *__restrict__ sin_tab,
          uint32_t hq, uint32_t hkv, uint32_t D, uint32_t rot_dim, float eps, uint32_t q_stride, uint32_t max_seq,
          uint32_t kv_stride, size_t batch_stride)
{
    __shared__ float red[32];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t row = blockIdx.x, head = blockIdx.y, i = threadIdx.x, half = D / 2;
    const uint32_t p = batch_stride ? (uint32_t)pos[row] : (uint32_t)pos[0] + row;
    const bool is_q = head < hq;
    __nv_bfloat16 *src = is_q ? q + (size_t)row * q_stride + (size_t)head * D
                              : const_cast<__nv_bfloat16 *>(k) + (size_t)row * kv_stride + (size_t)(head - hq) * D;
    float a = bf2f(src[i]), b = bf2f(src[i + half]);
    const __nv_bfloat16 *nw = is_q ? q_norm : k_norm;
    if (nw) {
        const float ss = cta_sum(a * a + b * b, red);
        const float r = rsqrtf(ss / (float)D + eps);
        a = bf2f(__hmul(__float2bfloat16_rn(a * r), nw[i]));
        b = bf2f(__hmul(__float2bfloat16_rn(b * r), nw[i + half]));
    }
    __nv_bfloat16 *dst_a, *dst_b;
    if (is_q) {
        dst_a = src + i;
        dst_b = src + i + half;
    } else {
        const size_t at = (size_t)row * batch_stride + ((size_t)min(p, max_seq - 1u) * hkv + (head - hq)) * D;
        dst_a = k_cache + at + i;
        dst_b = k_cache + at + i + half;
        const __nv_bfloat16 *vs = v + (size_t)row * kv_stride + (size_t)(head - hq) * D;
        v_cache[at + i] = vs[i];
        v_cache[at + i + half] = vs[i + half];
    }
    // rotate-half over the first rot_dim dimensions: element j < rot_dim / 2 pairs with j + rot_dim / 2 (with
    // rot_dim == D that is this thread's own pair); the head's elements meet in shared memory
    __shared__ float buf[256];
    __syncthreads();
    buf[i] = a;
    buf[i + half] = b;
    __syncthreads();
    const uint32_t rh = rot_dim / 2;
    auto rot = [&](uint32_t e) -> float {              // rotated value of element e
        if (e >= rot_dim) return buf[e];
        const uint32_t j = e < rh ? e : e - rh;
        const size_t ti = (size_t)min(p, max_seq - 1u) * rh + j;
        const float c = cos_tab[ti], s = sin_tab[ti];
        return e < rh ? buf[e] * c - buf[e + rh] * s : buf[e] * c + buf[e - rh] * s;
    };
    const float oa = rot(i), ob = rot(i + half);
    *dst_a = __float2bfloat16_rn(oa);
    *dst_b = __float2bfloat16_rn(ob);
}

// The same without norms and with the whole head rotated, 16-byte aligned rows: a thread takes eight pairs (elements 8 part
// .. + 7 and those D / 2 further), so a head is D / 16 threads and many rows fill their CTAs (1000 rows of 24 heads of 128:
// 5.7 us, against 26 with a CTA of 64 threads per row and head, under the profiler).
__global__ void __launch_bounds__(128)
k_rope_kv8(__nv_bfloat16 *q, const __nv_bfloat16 *__restrict__ k, const __nv_bfloat16 *__restrict__ v, const int32_t *pos,
           __nv_bfloat16 *k_cache, __nv_bfloat16 *v_cache, const float *__restrict__ cos_tab, const float *__restrict__ sin_tab,
           uint32_t rows, uint32_t hq, uint32_t hkv, uint32_t D, uint32_t q_stride, uint32_t max_seq, uint32_t kv_stride,
           size_t batch_stride)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t half = D / 2, parts = D / 16, idx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t part = idx % parts, hr = idx / parts, head = hr % (hq + hkv), row = hr / (hq + hkv);
    if (row >= rows) return;
    const uint32_t p = min(batch_stride ? (uint32_t)pos[row] : (uint32_t)pos[0] + row, max_seq - 1u), i = part * 8u;
    const bool is_q = head < hq;
    const __nv_bfloat16 *src = is_q ? q + (size_t)row * q_stride + (size_t)head * D : k + (size_t)row * kv_stride + (size_t)(head - hq) * D;
    const uint4 ar = *(const uint4 *)(src + i), br = *(const uint4 *)(src + i + half);
    const float4 *ct = (const float4 *)(cos_tab + (size_t)p * half + i), *st = (const float4 *)(sin_tab + (size_t)p * half + i);
    const float4 c0 = ct[0], c1 = ct[1], s0 = st[0], s1 = st[1];
    __nv_bfloat16 *dst = const_cast<__nv_bfloat16 *>(src);
    if (!is_q) {
        const size_t at = (size_t)row * batch_stride + ((size_t)p * hkv + (head - hq)) * D;
        const __nv_bfloat16 *vs = v + (size_t)row * kv_stride + (size_t)(head - hq) * D;
        dst = k_cache + at;
        *(uint4 *)(v_cache + at + i) = *(const uint4 *)(vs + i);
        *(uint4 *)(v_cache + at + i + half) = *(const uint4 *)(vs + i + half);
    }
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    float a[8], b[8], oa[8], ob[8];
    unpack8(ar, a);
    unpack8(br, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        oa[j] = a[j] * c[j] - b[j] * s[j];
        ob[j] = b[j] * c[j] + a[j] * s[j];
    }
    *(uint4 *)(dst + i) = pack8(oa);
    *(uint4 *)(dst + i + half) = pack8(ob);
}

// ---------------------------------------------------------------- single-query attention over the static cache
// grid (groups, CTAs per group, sequences), 256 threads.  A group is G consecutive query heads that share one KV head (G =
// query heads per KV head, or 1): the K and V rows of a position are loaded once and used for all G heads.
// The context [0, n_ctx) (n_ctx = pos[0] + 1) is dealt out in chunks of kAttnChunk positions: part s of at most `splits`
// takes the chunks s, s + splits, ...  A part of a few positions is all fixed cost, so forty sequences of 150 to 300
// positions cut 18 ways took 84 us a layer; which chunks make a part depends on the sequence alone, so it gets the same
// bits alone or in a batch, and a CTA walks as many parts as the grid leaves it.
// Bound by latency at batch 1 (4 MB of cache are 0.7 us of HBM), so a chunk is one short chain: all its K and V rows are
// requested at once (a position's K row by four threads, its V row by D / 8), the scores of all heads take two shuffles,
// a warp per head turns them into weights, every thread sums its positions' V, and the threads' sums are joined once per
// part.  With a running softmax per lane group and joins of eight such states per head instead, a CTA took 10700 cycles
// for 64 positions (12.5 us a launch for 1025 positions of 16 / 8 heads of 128 under the profiler; 29 us for 4097 of
// 6 / 2 heads of 256; 34 us for forty sequences of 225); now 8.2, 16 and 23 us.
// With max_seq (rows of the cache) the first loads do not wait for the position: they read whatever rows the part would
// take at full length, and what lies beyond the position is dropped.  With tickets (one word per sequence and group, zero
// between launches) the last CTA of a group joins the parts itself; otherwise k_attn_combine does.
constexpr uint32_t kAttnChunk = 64;                    // positions: what the 8 warps of a CTA have in flight for D = 128
constexpr int kAttnMaxSplits = 256;
__device__ __forceinline__ uint32_t attn_parts(uint32_t n_ctx, uint32_t splits)
{
    return min(splits, (n_ctx + kAttnChunk - 1u) / kAttnChunk);
}
// Three forms with the same sums in the same order, so the same bits (launch_attn has the rule and what it was measured on):
// kAttnWide  the grid has at most a CTA for every SM, which may have all registers: everything a chunk needs is in flight at once.
//            16 / 8 heads of 128, one sequence of 1100 positions: 5.5 us a launch, 6.2 with two CTAs' registers.
// kAttnMany  more CTAs than SMs: registers as they fall (two CTAs an SM for most sizes).  Five rows of 705 positions verified 9.7
//            us, 11.6 with one CTA's registers; eight sequences of 500 to 1000 positions 15 and 18.5.
// kAttnOne   (heads of 64 and 128) one CTA per group and sequence takes all of its parts.  Their sums stay in shared memory (as many as six kilobytes
// hold; the rest go through the scratch) and nothing is published: the same sums in the same order as by many CTAs, so the same
// bits.  Bound by the chain of a chunk, not by its bytes (a fifth to a half of the copy rate), so three CTAs of an SM run it
// side by side.  Two chunks are in flight through shared memory, a thread's own pieces (nobody else reads
// them, so no barrier waits for them); the warps' sums take the place of the chunk that was taken last, without which only two
// CTAs fit.  Forty sequences of 150 to 300 positions, 16 / 8 heads of 128: 20.9 us by many CTAs, 17.7 so; of 500 to 1000 positions
// 49 and 48.  (One running softmax over all chunks instead of parts: 14.7 and 38, but other bits than the sequence's own.)
enum AttnForm { kAttnWide, kAttnMany, kAttnOne };
__host__ __device__ constexpr int attn_keep(int d, int g) { return 1536 / (g * d) > 0 ? 1536 / (g * d) : 1; }
__host__ __device__ constexpr int attn_one_ctas(int d, int g) { return g * d <= 256 ? 3 : g * d <= 512 ? 2 : 1; }       // per SM: registers
struct AttnJoin {
    uint32_t *tickets;
    __nv_bfloat16 *out;
    const __nv_bfloat16 *gate;
    uint32_t gate_stride, gate_row_stride;
};

template <int D, int G, AttnForm FORM>
__global__ void __launch_bounds__(256, FORM == kAttnOne ? attn_one_ctas(D, G) : FORM == kAttnWide ? 1 : 0)     // 0: no minimum
k_attn_decode(const __nv_bfloat16 *__restrict__ q, const __nv_bfloat16 *__restrict__ k_cache,
              const __nv_bfloat16 *__restrict__ v_cache, const int32_t *pos, float *part, uint32_t hq, uint32_t hkv,
              float scale, uint32_t q_stride, size_t batch_stride, uint32_t splits, uint32_t max_seq, AttnJoin join)
{
    // blockIdx.z: the sequence (its query row, its caches batch_stride elements after the previous one's, its position)
    q += (size_t)blockIdx.z * q_stride;
    k_cache += (size_t)blockIdx.z * batch_stride;
    v_cache += (size_t)blockIdx.z * batch_stride;
    pos += blockIdx.z;
    // scratch: sums [sequences][hq][splits][D], then (maximum, denominator) [sequences][hq][splits]
    float2 *part_ml = (float2 *)(part + (size_t)gridDim.z * hq * splits * D) + (size_t)blockIdx.z * hq * splits;
    part += (size_t)blockIdx.z * hq * splits * D;
    constexpr int NW = 8;                              // warps
    constexpr int C = (int)kAttnChunk;
    constexpr int KC = D / 32;                         // 16-byte pieces of a K row per thread (four threads per position)
    constexpr int VT = D / 8;                          // threads per V row
    constexpr int VG = 256 / VT, VP = C / VG;          // groups of threads, positions of a chunk per group
    constexpr int HG = G * D * NW * 4 <= 16384 ? G : 16384 / (D * NW * 4);        // heads joined at a time
    // the last CTA's join: quads of dimensions, and the groups of threads that share out the parts; their sums take the place
    // of the warps' ([PG][G * D] floats: more than [NW][HG][D] for one head of 64)
    constexpr int QD = G * D / 4, PG = QD >= 256 ? 1 : 256 / QD;
    constexpr int NR = PG * G > NW * HG ? (PG * G + HG - 1) / HG : NW;
    static_assert(PG * G * D <= NR * HG * D && NW <= NR, "sums of the join fit");
    __shared__ __align__(16) float sm_q[G][D];         // scaled queries
    __shared__ float sm_s[G][C], sm_c[G];              // a chunk's scores, then weights; the sums' rescaling
    constexpr bool ONE = FORM == kAttnOne;
    static_assert(!ONE || D <= 128, "two chunks of 256 dimensions do not fit beside one another");
    __shared__ __align__(16) float sm_acc_own[ONE ? 1 : NR * HG * D];
    __shared__ float sm_w[G][kAttnMaxSplits], sm_sum[G];
    __shared__ uint32_t sm_last;
    constexpr int KEEP = ONE ? attn_keep(D, G) : 1;
    __shared__ __align__(16) float sm_part[ONE ? KEEP : 1][ONE ? G * D : 4];
    __shared__ float2 sm_ml[ONE ? G : 1][KEEP];
    extern __shared__ __align__(16) uint4 sm_ring[];   // [2][KC + VP][256 threads]
    // the warps' sums: [NR][HG][D], with a ring in the half of the chunk that was taken last
    static_assert(!ONE || NR * HG * D * 4 <= (KC + VP) * 4096, "fits");
    float *sm_acc = sm_acc_own;
    auto acc_at = [&](int w, int h, int d) -> float & { return sm_acc[(w * HG + h) * D + d]; };
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t head0 = blockIdx.x * G;
    const uint32_t kvh = head0 / (hq / hkv);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int kp = tid >> 2, kt = tid & 3;             // K: position of the chunk, which pieces (kt, kt + 4, ...)
    const int vg = tid / VT, vd = (tid % VT) * 8;      // V: positions vg, vg + VG, ..., eight dimensions
    const size_t row_stride = (size_t)hkv * D;
    const __nv_bfloat16 *kb = k_cache + (size_t)kvh * D + kt * 8, *vb = v_cache + (size_t)kvh * D + vd;
    const uint32_t last = (uint32_t)pos[0];
    uint4 kr[KC], vr[VP];
    const uint32_t ring = ONE ? (uint32_t)__cvta_generic_to_shared(sm_ring) + tid * 16u : 0u;
    uint32_t visit = 0;                                // chunks taken so far; even ones lie in the first half of the ring
    auto piece = [&](uint32_t i, int j) { return ring + ((i & 1u) * (KC + VP) + j) * 4096u; };
    auto request = [&](uint32_t c, uint32_t i, uint32_t limit) {       // chunk c as the i-th to be taken
        const __nv_bfloat16 *src = kb + min(c * kAttnChunk + kp, limit) * row_stride;
#pragma unroll
        for (int j = 0; j < KC; ++j)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(piece(i, j)), "l"(src + j * 32) : "memory");
#pragma unroll
        for (int j = 0; j < VP; ++j)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(piece(i, KC + j)), "l"(vb + min(c * kAttnChunk + vg + j * VG, limit) * row_stride) : "memory");
        cp_async_commit();
    };
    auto taken = [&](uint32_t addr) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
        return v;
    };
    auto fetch_k = [&](uint32_t c, uint32_t limit) {
        const __nv_bfloat16 *src = kb + min(c * kAttnChunk + kp, limit) * row_stride;
#pragma unroll
        for (int j = 0; j < KC; ++j) kr[j] = *(const uint4 *)(src + j * 32);
    };
    auto fetch_v = [&](uint32_t c, uint32_t limit) {
#pragma unroll
        for (int j = 0; j < VP; ++j) vr[j] = *(const uint4 *)(vb + min(c * kAttnChunk + vg + j * VG, limit) * row_stride);
    };
    auto write_out = [&](int h, int d, float v) {      // head h of the group, dimension d
        float o = bfround(v);
        if (join.gate) {
            const float gv = bf2f(join.gate[(size_t)blockIdx.z * join.gate_row_stride + (size_t)(head0 + h) * join.gate_stride + d]);
            o = o * bfround(sigmoid_f(gv));
        }
        join.out[((size_t)blockIdx.z * hq + head0 + h) * D + d] = __float2bfloat16_rn(o);
    };
    if (ONE) {
        request(0u, 0u, max_seq - 1u);                 // (ONE has max_seq)
    } else if (max_seq) {
        fetch_k(blockIdx.y, max_seq - 1u);
        fetch_v(blockIdx.y, max_seq - 1u);
    }
    for (int i = tid; i < G * D; i += 256) sm_q[i / D][i % D] = bf2f(q[(size_t)head0 * D + i]) * scale;
    const uint32_t n_ctx = max_seq ? min(last + 1u, max_seq) : last + 1u, used = attn_parts(n_ctx, splits);
    if (used == 0u && join.tickets && blockIdx.y == 0) {               // position -1: the mean over nothing
        for (int i = tid; i < G * D; i += 256)
            join.out[((size_t)blockIdx.z * hq + head0 + i / D) * D + i % D] = __float2bfloat16_rn(__int_as_float(0x7FFFFFFF));
    }
    if (blockIdx.y >= used) {
        if (ONE) cp_async_wait<0>();
        return;
    }
    uint32_t ps = 0, pc = 0;                           // part and chunk requested last
    auto request_next = [&](uint32_t i) {
        pc = (pc + splits) * kAttnChunk < n_ctx ? pc + splits : ++ps;
        if (ps < used) request(pc, i, n_ctx - 1u);
        else cp_async_commit();
    };
    if (ONE) request_next(1u);
    __syncthreads();
    if (!max_seq) {
        fetch_k(blockIdx.y, n_ctx - 1u);
        fetch_v(blockIdx.y, n_ctx - 1u);
    }
    for (uint32_t s = blockIdx.y; s < used; s += gridDim.y) {
        float acc[G][8];
#pragma unroll
        for (int h = 0; h < G; ++h)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[h][j] = 0.f;
        float M = -INFINITY, L = 0.f;                  // of head wid, in warp wid
        for (uint32_t c = s; c * kAttnChunk < n_ctx; c += splits) {
            const bool more = (c + splits) * kAttnChunk < n_ctx;
            const uint32_t nxt = more ? c + splits : s + gridDim.y;       // the part's next chunk, or the next part's first
            const bool ahead = more || nxt < used;
            float sc[G];
#pragma unroll
            for (int h = 0; h < G; ++h) sc[h] = 0.f;
            if (ONE) {
                cp_async_wait<1>();                    // the chunk is there, the next one may be on its way
#pragma unroll
                for (int j = 0; j < KC; ++j) kr[j] = taken(piece(visit, j));
            }
#pragma unroll
            for (int j = 0; j < KC; ++j) {
                float kf[8];
                unpack8(kr[j], kf);
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float4 q0 = *(const float4 *)&sm_q[h][kt * 8 + j * 32], q1 = *(const float4 *)&sm_q[h][kt * 8 + j * 32 + 4];
                    sc[h] = fmaf(kf[3], q0.w, fmaf(kf[2], q0.z, fmaf(kf[1], q0.y, fmaf(kf[0], q0.x, sc[h]))));
                    sc[h] = fmaf(kf[7], q1.w, fmaf(kf[6], q1.z, fmaf(kf[5], q1.y, fmaf(kf[4], q1.x, sc[h]))));
                }
            }
            if (!ONE && ahead) fetch_k(nxt, n_ctx - 1u);
            const bool live = c * kAttnChunk + kp < n_ctx;
#pragma unroll
            for (int h = 0; h < G; ++h) {
                sc[h] += __shfl_xor_sync(0xffffffffu, sc[h], 1);
                sc[h] += __shfl_xor_sync(0xffffffffu, sc[h], 2);
                if (kt == (h & 3)) sm_s[h][kp] = live ? sc[h] : -INFINITY;
            }
            __syncthreads();
            if (wid < G) {                             // a warp per head (a chunk has at least one live position)
                const float s0 = sm_s[wid][lane], s1 = sm_s[wid][lane + 32];
                float mx = fmaxf(s0, s1);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
                mx = fmaxf(mx, M);
                const float base = mx == -INFINITY ? 0.f : mx;     // nothing but -inf so far: weights 0
                const float p0 = __expf(s0 - base), p1 = __expf(s1 - base), cr = __expf(M - base);
                sm_s[wid][lane] = p0;
                sm_s[wid][lane + 32] = p1;
                if (lane == 0) sm_c[wid] = cr;
                L = L * cr + warp_sum(p0 + p1);
                M = mx;
            }
            __syncthreads();
            if (c != s) {
#pragma unroll
                for (int h = 0; h < G; ++h)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[h][j] *= sm_c[h];
            }
#pragma unroll
            for (int j = 0; j < VP; ++j) {
                float vf[8];
                if (ONE) vr[j] = taken(piece(visit, KC + j));
                unpack8(vr[j], vf);
                if (c * kAttnChunk + vg + j * VG >= n_ctx) continue;       // (not read, or rows beyond the position)
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float p = sm_s[h][vg + j * VG];
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[h][k] = fmaf(p, vf[k], acc[h][k]);
                }
            }
            if (!ONE && ahead) fetch_v(nxt, n_ctx - 1u);
            if (ONE && more) {
                request_next(visit + 2u);              // into the pieces that this thread has just taken
                ++visit;
            }
            if (more) __syncthreads();                 // the weights are read: the next chunk's scores may follow
        }
        // join: the warp's groups of threads by shuffles, the warps in shared memory, HG heads at a time
        if (ONE) {
            sm_acc = (float *)(sm_ring + (visit & 1u) * (KC + VP) * 256u);
            __syncthreads();                           // nobody takes pieces of it any more
        }
        float *dst = part + ((size_t)head0 * splits + s) * D;
#pragma unroll
        for (int h0 = 0; h0 < G; h0 += HG) {
            if (h0 || (!ONE && s != blockIdx.y)) __syncthreads();  // sm_acc is free
#pragma unroll
            for (int hh = 0; hh < HG; ++hh) {
                if (h0 + hh >= G) break;
                float (&v)[8] = acc[h0 + hh < G ? h0 + hh : 0];
#pragma unroll
                for (int d = VT; d < 32; d <<= 1)
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], d);
                if (lane < VT) {
                    *(float4 *)&acc_at(wid, hh, vd) = make_float4(v[0], v[1], v[2], v[3]);
                    *(float4 *)&acc_at(wid, hh, vd + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
            }
            __syncthreads();
            for (int i = tid; i < HG * D && h0 + i / D < G; i += 256) {
                float a = 0.f;
#pragma unroll
                for (int w = 0; w < NW; ++w) a += acc_at(w, i / D, i % D);
                if (ONE && s < (uint32_t)KEEP) sm_part[s][h0 * D + i] = a;
                else dst[(size_t)(h0 + i / D) * splits * D + i % D] = a;
            }
        }
        if (ONE && s + 1u < used) {
            __syncthreads();                           // the sums are read
            request_next(visit + 2u);
            ++visit;
        }
        if (wid < G && lane == 0) {
            if (ONE && s < (uint32_t)KEEP) sm_ml[wid][s] = make_float2(M, L);
            else part_ml[(size_t)(head0 + wid) * splits + s] = make_float2(M, L);
        }
    }
    if (!ONE && !join.tickets) return;
    // ---- the last CTA of the group joins the parts.  The CTAs with work add numbers whose sum is zero to the ticket, the first
    // one 1 - ctas and the others 1: it is zero again exactly when all of them have come.  So nobody resets it, and it is zero
    // after launches that overlapped too (whose own results are lost).
    const uint32_t ctas = min(gridDim.y, used);
    uint32_t *ticket = join.tickets + (size_t)blockIdx.z * gridDim.x + blockIdx.x;
    if (!ONE) __threadfence();                       // this thread's share of the parts, before the ticket
    __syncthreads();
    if (!ONE && ctas > 1u) {
        const uint32_t mine = blockIdx.y ? 1u : 1u - ctas;
        if (threadIdx.x == 0) sm_last = atomicAdd(ticket, mine) + mine == 0u;
        __syncthreads();
        if (!sm_last) return;
        __threadfence();
    }
    // all of the group's sums are requested at once, as far as registers go: a thread takes four dimensions of a head and
    // every PG-th part (rounds of eight dependent loads of one value: 29 us a launch at a 4097-token context, not 16.5)
    constexpr int MAXQ = (QD + 255) / 256;             // quads per thread
    constexpr int UN = ONE ? 1 : 16;
    const int pg = QD >= 256 ? 0 : tid / QD, q0 = QD >= 256 ? tid : tid % QD;
    float4 first[UN];
    auto sums = [&](int qd, uint32_t s) -> float4 {
        if (ONE && s < (uint32_t)KEEP) return *(const float4 *)&sm_part[s][qd * 4];
        return __ldcg((const float4 *)(part + ((size_t)(head0 + qd * 4 / D) * splits + s) * D + qd * 4 % D));
    };
#pragma unroll
    for (int k = 0; k < UN; ++k) {
        const uint32_t s = pg + k * PG;
        first[k] = q0 < QD && pg < PG && s < used ? sums(q0, s) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (wid < G) {                                     // a warp per head: the parts' weights and their sum
        const float2 *p = part_ml + (size_t)(head0 + wid) * splits;
        auto max_sum = [&](uint32_t s) { return ONE && s < (uint32_t)KEEP ? sm_ml[wid][s] : __ldcg(p + s); };
        float mx = -INFINITY, sum = 0.f;
        for (uint32_t s = lane; s < used; s += 32) mx = fmaxf(mx, max_sum(s).x);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
        for (uint32_t s = lane; s < used; s += 32) {
            const float2 ml = max_sum(s);
            const float c = ml.x == -INFINITY ? 0.f : __expf(ml.x - mx);
            sm_w[wid][s] = c;
            sum += ml.y * c;
        }
        sum = warp_sum(sum);
        if (lane == 0) sm_sum[wid] = sum;
    }
    __syncthreads();
    float *sm_p = sm_acc;                              // [PG][G * D]
#pragma unroll
    for (int i = 0; i < MAXQ; ++i) {
        const int qd = q0 + i * 256;
        if (qd >= QD || pg >= PG) continue;
        const int h = qd * 4 / D;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](const float4 &v, float w) {
            a.x = fmaf(v.x, w, a.x); a.y = fmaf(v.y, w, a.y); a.z = fmaf(v.z, w, a.z); a.w = fmaf(v.w, w, a.w);
        };
#pragma unroll
        for (int k = 0; k < UN; ++k) {
            const uint32_t s = pg + k * PG;
            if (s < used) add(i ? sums(qd, s) : first[k], sm_w[h][s]);
        }
        for (uint32_t s0 = pg + UN * PG; s0 < used; s0 += UN * PG) {
            float4 v[UN];
#pragma unroll
            for (int k = 0; k < UN; ++k) {
                const uint32_t s = s0 + k * PG;
                v[k] = s < used ? sums(qd, s) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < UN; ++k)
                if (s0 + k * PG < used) add(v[k], sm_w[h][s0 + k * PG]);
        }
        *(float4 *)(sm_p + (size_t)pg * G * D + qd * 4) = a;
    }
    __syncthreads();
    for (int i = tid; i < G * D; i += 256) {
        const int h = i / D, d = i % D;
        float a = sm_p[i];
#pragma unroll
        for (int g = 1; g < PG; ++g) a += sm_p[g * G * D + i];
        write_out(h, d, a / sm_sum[h]);
    }
}

// grid q heads, D threads: out[head][d] = sum over the splits, optional sigmoid gate (gate[head][d], bf16).
// The splits' maxima and denominators are fetched by one thread each, the weighted sums with independent loads.
__global__ void __launch_bounds__(256)
k_attn_combine(const float *__restrict__ part, __nv_bfloat16 *out, const __nv_bfloat16 *__restrict__ gate, const int32_t *pos,
               uint32_t max_splits, uint32_t D, uint32_t gate_stride, uint32_t gate_row_stride)
{
    __shared__ float wgt[kAttnMaxSplits], red[32];
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t head = blockIdx.x, t = threadIdx.x;
    // blockIdx.y: the sequence
    const float2 *part_ml = (const float2 *)(part + (size_t)gridDim.y * gridDim.x * max_splits * D) +
                            ((size_t)blockIdx.y * gridDim.x + head) * max_splits;
    part += (size_t)blockIdx.y * gridDim.x * max_splits * D;
    out += (size_t)blockIdx.y * gridDim.x * D;
    if (gate) gate += (size_t)blockIdx.y * gate_row_stride;
    float gv = 0.f;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (gate && t < D) gv = bf2f(gate[(size_t)head * gate_stride + t]);
    const uint32_t splits = attn_parts((uint32_t)pos[blockIdx.y] + 1u, max_splits);
    const float *p = part + (size_t)head * max_splits * D;
    float ms = -INFINITY, ls = 0.f;
    if (t < splits) {
        const float2 ml = part_ml[t];
        ms = ml.x;
        ls = ml.y;
    }
    // CTA-wide maximum
    float M = ms;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
    if ((t & 31u) == 0) red[t >> 5] = M;
    __syncthreads();
    M = red[0];
    for (uint32_t i = 1; i < (blockDim.x >> 5); ++i) M = fmaxf(M, red[i]);
    const float c = ms == -INFINITY ? 0.f : __expf(ms - M);
    if (t < splits) wgt[t] = c;
    const float L = cta_sum(ls * c, red);              // (its barriers also publish wgt)
    if (t >= D) return;
    float a0 = 0.f, a1 = 0.f;
    const float *pt = p + t;
    uint32_t s2 = 0;
    for (; s2 + 16 <= splits; s2 += 16) {              // sixteen independent loads in flight
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = pt[(size_t)(s2 + k) * D];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
            a0 = fmaf(v[k], wgt[s2 + k], a0);
            a1 = fmaf(v[k + 1], wgt[s2 + k + 1], a1);
        }
    }
    {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = s2 + k < splits ? pt[(size_t)(s2 + k) * D] : 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) a0 = fmaf(v[k], s2 + k < splits ? wgt[s2 + k] : 0.f, a0);
    }
    const float a = a0 + a1;
    float o = bfround(a / L);
    if (gate) o = bfround(o) * bfround(sigmoid_f(gv));
    out[(size_t)head * D + t] = __float2bfloat16_rn(o);
}

// ---------------------------------------------------------------- causal conv1d update (depth-wise)
// state [C][K - 1] (bf16, oldest first) holds the last K - 1 inputs of every channel;
// y_c = silu(sum_j w[c][j] * input_{t - K + 1 + j} + bias_c), then the state takes x in.
// K == 4 and C a multiple of 4: a thread looks after four channels with 8- and 16-byte accesses, everything
// requested at once (the weights before the dependency wait); other shapes take the scalar kernel.
__global__ void __launch_bounds__(64)
k_conv_update4(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *state, const __nv_bfloat16 *__restrict__ w,
               const __nv_bfloat16 *__restrict__ bias, __nv_bfloat16 *y, uint32_t C)
{
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t c = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    const bool on = c < C;
    uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
    uint2 bb = make_uint2(0, 0);
    if (on) {
        w0 = *(const uint4 *)(w + (size_t)c * 4);
        w1 = *(const uint4 *)(w + (size_t)c * 4 + 8);
        if (bias) bb = *(const uint2 *)(bias + c);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!on) return;
    uint2 *sp = (uint2 *)(state + (size_t)c * 3);      // 12 state values of the four channels: 24 bytes
    const uint2 s0 = sp[0], s1 = sp[1], s2 = sp[2];
    const uint2 xr = *(const uint2 *)(x + c);
    const uint32_t sw[6] = {s0.x, s0.y, s1.x, s1.y, s2.x, s2.y}, ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    const uint32_t xw[2] = {xr.x, xr.y}, bw[2] = {bb.x, bb.y};
    auto half = [](const uint32_t *a, int i) { return __uint_as_float((i & 1) ? (a[i >> 1] & 0xffff0000u) : (a[i >> 1] << 16)); };
    auto bits = [](const uint32_t *a, int i) { return (i & 1) ? (a[i >> 1] >> 16) : (a[i >> 1] & 0xffffu); };
    uint32_t ns[12], yo[4];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        float acc = half(bw, ch);
#pragma unroll
        for (int j = 0; j < 3; ++j) acc = fmaf(half(ww, 4 * ch + j), half(sw, 3 * ch + j), acc);
        acc = fmaf(half(ww, 4 * ch + 3), half(xw, ch), acc);
        yo[ch] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(silu_f(acc)));
        ns[3 * ch] = bits(sw, 3 * ch + 1);
        ns[3 * ch + 1] = bits(sw, 3 * ch + 2);
        ns[3 * ch + 2] = bits(xw, ch);
    }
    sp[0] = make_uint2(ns[0] | ns[1] << 16, ns[2] | ns[3] << 16);
    sp[1] = make_uint2(ns[4] | ns[5] << 16, ns[6] | ns[7] << 16);
    sp[2] = make_uint2(ns[8] | ns[9] << 16, ns[10] | ns[11] << 16);
    *(uint2 *)(y + c) = make_uint2(yo[0] | yo[1] << 16, yo[2] | yo[3] << 16);
}

__global__ void __launch_bounds__(256)
k_conv_update(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *state, const __nv_bfloat16 *__restrict__ w,
              const __nv_bfloat16 *__restrict__ bias, __nv_bfloat16 *y, uint32_t C, uint32_t K)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    __nv_bfloat16 *st = state + (size_t)c * (K - 1);
    const __nv_bfloat16 *wc = w + (size_t)c * K;
    const float xv = bf2f(x[c]);
    float acc = bias ? bf2f(bias[c]) : 0.f;
    for (uint32_t j = 0; j + 1 < K; ++j) {
        const float s = bf2f(st[j]);
        acc = fmaf(bf2f(wc[j]), s, acc);
        if (j + 2 < K) st[j] = st[j + 1];
    }
    acc = fmaf(bf2f(wc[K - 1]), xv, acc);
    st[K - 2] = x[c];
    y[c] = __float2bfloat16_rn(silu_f(acc));
}

// ---------------------------------------------------------------- gated delta rule, one step
// One CTA per value head, 256 threads: thread (j = tid & 127, ih = tid >> 7) owns column j of the head's state
// S [DK = 128][DV = 128] (fp32, row i = key dimension) for rows [64 ih, 64 ih + 64), in registers.
//   q, k: the key head's vectors (value head / (hv / hk)), L2-normalised here; q scaled by DK^-0.5
//   g = exp(-exp(A_log) * softplus(a + dt_bias)),  beta = sigmoid(b)
//   S <- g S;  delta = (v - S^T k) beta;  S <- S + k delta^T;  o = S^T q
//   o <- rmsnorm(o) * norm_w * silu(z)                                  (the head's gated output norm)
// The state is read once and written once.
// CONV: the causal depth-wise conv (K = 4) + SiLU of the layer runs in the same kernel on the channels this head needs
// (its key head's q and k, its own v): qkv is then the raw projection, conv_state [2][C][3] holds the last three inputs
// of every channel twice -- the step at position p reads copy p & 1 and writes copy (p + 1) & 1, because the value heads
// that share a key head all read its q / k channels while one of them (the first) writes them.
template <bool CONV>
__global__ void __launch_bounds__(256)
k_gdn_step(const __nv_bfloat16 *__restrict__ qkv, const __nv_bfloat16 *__restrict__ z, const __nv_bfloat16 *__restrict__ a_in,
           const __nv_bfloat16 *__restrict__ b_in, const float *__restrict__ A_log, const float *__restrict__ dt_bias,
           const __nv_bfloat16 *__restrict__ norm_w, float *state, __nv_bfloat16 *out, uint32_t hk, uint32_t hv, float eps,
           __nv_bfloat16 *conv_state, const __nv_bfloat16 *__restrict__ conv_w, const int32_t *pos, uint32_t C)
{
    constexpr int DK = 128, DV = 128;
    __shared__ float red[32], qs[DK], ks[DK], vs[DV], part_k[2][DV], part_q[2][DV];
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t vh = blockIdx.x, rep = hv / hk, kh = vh / rep;
    const uint32_t tid = threadIdx.x, j = tid & 127u, ih = tid >> 7;
    // the head's state was last written by this kernel one token ago and its parameters are constants: both are
    // requested before the dependency wait, so the longest loads overlap the tail of the kernel ahead
    float *S = state + (size_t)vh * DK * DV;
    float s[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) s[i] = S[(size_t)(64 * ih + i) * DV + j];
    const float a_log = A_log[vh], dtb = dt_bias[vh], nw = bf2f(norm_w[j]);
    // qkv = [q (hk * DK) | k (hk * DK) | v (hv * DV)]; channels of this head
    const uint32_t cq = kh * DK + j, ck = (hk + kh) * DK + j, cv = 2u * hk * DK + vh * DV + j;
    // conv: thread j < 128 looks after q channel j and v channel j, thread 128 + j after k channel j
    const uint32_t c0 = ih == 0 ? cq : ck, c1 = cv;
    float cw0[4] = {0.f, 0.f, 0.f, 0.f}, cw1[4] = {0.f, 0.f, 0.f, 0.f}, st0[3] = {0.f, 0.f, 0.f}, st1[3] = {0.f, 0.f, 0.f};
    uint32_t par = 0;
    if (CONV) {
        par = (uint32_t)pos[0] & 1u;                     // (written at the end of the token step before this one)
        const __nv_bfloat16 *rd = conv_state + (size_t)par * C * 3;
#pragma unroll
        for (int k = 0; k < 4; ++k) cw0[k] = bf2f(conv_w[(size_t)c0 * 4 + k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) st0[k] = bf2f(rd[(size_t)c0 * 3 + k]);
        if (ih == 0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cw1[k] = bf2f(conv_w[(size_t)c1 * 4 + k]);
#pragma unroll
            for (int k = 0; k < 3; ++k) st1[k] = bf2f(rd[(size_t)c1 * 3 + k]);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float qe = 0.f, ke = 0.f;
    if (CONV) {
        auto conv = [&](uint32_t c, const float (&w)[4], const float (&st)[3], bool write) -> float {
            const __nv_bfloat16 xin = qkv[c];
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) acc = fmaf(w[k], st[k], acc);
            acc = fmaf(w[3], bf2f(xin), acc);
            if (write) {
                __nv_bfloat16 *wr = conv_state + ((size_t)(par ^ 1u) * C + c) * 3;
                wr[0] = __float2bfloat16_rn(st[1]);
                wr[1] = __float2bfloat16_rn(st[2]);
                wr[2] = xin;
            }
            return bfround(silu_f(acc));                 // the conv's output is a bf16 tensor in the eager path
        };
        const float y0 = conv(c0, cw0, st0, vh % rep == 0);      // q or k: written by the key head's first value head
        if (ih == 0) {
            qe = y0;
            vs[j] = conv(c1, cw1, st1, true);
        } else {
            ke = y0;
        }
    } else {
        if (ih == 0) {
            qe = bf2f(qkv[cq]);
            vs[j] = bf2f(qkv[cv]);
        } else {
            ke = bf2f(qkv[ck]);
        }
    }
    const float qn = cta_sum(qe * qe, red), kn = cta_sum(ke * ke, red);     // (q lives in threads 0..127, k in 128..255)
    if (ih == 0) qs[j] = qe * rsqrtf(qn + 1e-6f) * rsqrtf((float)DK);
    else ks[j] = ke * rsqrtf(kn + 1e-6f);
    __syncthreads();
    const float av = bf2f(a_in[vh]) + dtb;
    const float sp = av > 20.f ? av : log1pf(__expf(av));
    const float g = __expf(-__expf(a_log) * sp), beta = sigmoid_f(bf2f(b_in[vh]));
    float sk = 0.f, sq = 0.f;
#pragma unroll
    for (int i = 0; i < 64; ++i) {
        s[i] *= g;
        sk = fmaf(s[i], ks[64 * ih + i], sk);
        sq = fmaf(s[i], qs[64 * ih + i], sq);
    }
    part_k[ih][j] = sk;
    part_q[ih][j] = sq;
    float kq = 0.f;
    if (tid < DK) kq = ks[tid] * qs[tid];
    kq = cta_sum(kq, red);                             // k . q (also the barrier for part_k / part_q)
    const float kv_mem = part_k[0][j] + part_k[1][j];
    const float delta = (vs[j] - kv_mem) * beta;
#pragma unroll
    for (int i = 0; i < 64; ++i) S[(size_t)(64 * ih + i) * DV + j] = fmaf(ks[64 * ih + i], delta, s[i]);
    // o_j = sum_i (S_ij + k_i delta_j) q_i = (S^T q)_j + delta_j (k . q)
    const float o = part_q[0][j] + part_q[1][j] + delta * kq;
    const float ob = bfround(o);                       // the recurrence's output is a bf16 tensor in the eager path
    const float ss = cta_sum(ih == 0 ? ob * ob : 0.f, red);
    if (ih == 0) {
        const float r = rsqrtf(ss / (float)DV + eps);
        const __nv_bfloat16 nv = __float2bfloat16_rn(bfround(ob * r) * nw);
        const float zg = silu_f(bf2f(z[(size_t)vh * DV + j]));
        out[(size_t)vh * DV + j] = __hmul(nv, __float2bfloat16_rn(zg));
    }
}

}  // namespace ixb
