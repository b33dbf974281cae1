// The weight-only NVFP4 lane: y[t][r] = dot_nvfp4_a16_q8_f32(W_r, x_t), taken when a weight carries no
// input_scale_inv (crates/muser-engine/src/weights.rs:117-121).
//
// Reproduces quant::quantize_nvfp4_q8_block and dot_nvfp4_a16_q8_f32 bit for bit (src/quant/nvfp4.rs:62-99,348-379;
// the GB10 twin is scripts/gx10/vllm/muser_vllm/exact_fp4_a16_mm.py): every 256 activations are rounded to f16 and
// quantized to int8 against the FIRST element of largest magnitude (inverse scale -127 / that element, nearest
// through the 12582912 magic-number FMA, capped at 127); a block's contraction is an exact integer: E2M1 codes in
// halves times int8, the sum of a 16-group times its E4M3 scale in units of 2^-9, sixteen groups added in 64 bits;
// then four FMAs in a fixed order turn it into f32, the blocks are added front to back, and the result is rounded
// to f16.  Nothing here is approximate, so outputs are compared for equal bits.
//
// This is the lane for checkpoints without activation scales, not the prefill hot path.  The activations of a call are
// quantized once into the context workspace by a kernel of their own; the contraction runs on the int8 tensor pipe.
#include <cuda_fp8.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "nvfp4_a16_exchange.h"

namespace muser {

// int8 codes [tokens][n_in] followed by one f32 d per (token, 256-block)
__global__ void __launch_bounds__(256) nvfp4_q8_quantize_kernel(const void *x, uint32_t x_f32, uint32_t n_in,
                                                                int8_t *qs, float *ds) {
    __shared__ float s_mag[8];
    __shared__ uint32_t s_idx[8];
    __shared__ float s_val[8];
    pdl_wait();
    pdl_release(); // the contraction may start fetching its weights
    const uint32_t block = blockIdx.x, tok = blockIdx.y, i = threadIdx.x, blocks = n_in / 256;
    const size_t at = (size_t)tok * n_in + (size_t)block * 256 + i;
    const float raw = x_f32 ? reinterpret_cast<const float *>(x)[at] : __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(x)[at]);
    const float v = __half2float(__float2half_rn(raw));
    // first element of largest magnitude: larger magnitude wins, the lower index wins a tie
    float mag = v == v ? fabsf(v) : -1.0f, val = v; // a NaN never wins the reference's `>` scan
    uint32_t idx = i;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, mag, o), v2 = __shfl_xor_sync(0xffffffffu, val, o);
        const uint32_t i2 = __shfl_xor_sync(0xffffffffu, idx, o);
        if (m2 > mag || (m2 == mag && i2 < idx)) mag = m2, val = v2, idx = i2;
    }
    if ((i & 31) == 0) s_mag[i >> 5] = mag, s_idx[i >> 5] = idx, s_val[i >> 5] = val;
    __syncthreads();
    mag = s_mag[0], val = s_val[0], idx = s_idx[0];
#pragma unroll
    for (int w = 1; w < 8; ++w)
        if (s_mag[w] > mag || (s_mag[w] == mag && s_idx[w] < idx)) mag = s_mag[w], val = s_val[w], idx = s_idx[w];
    int q = 0;
    float d = 0.0f;
    if (mag > 0.0f) {
        const float inverse_scale = __fdiv_rn(-127.0f, val);
        const float rounded = __fmaf_rn(inverse_scale, v, 12582912.0f);
        q = (int)(__float_as_uint(rounded) & 0x007fffffu) - 0x00400000;
        q = q < 127 ? q : 127;
        d = __fdiv_rn(1.0f, inverse_scale);
    }
    qs[at] = (int8_t)q;
    if (i == 0) ds[(size_t)tok * blocks + block] = d;
}

struct A16Args {
    const uint8_t *packed, *scales; // the repacked image: codes [n_out_pad][n_in/2], swizzled unsigned scales
    const int8_t *qs;
    const float *ds;
    void *y;
    float scale2;
    uint32_t n_out, n_in, kt, tokens, y_dtype, ksplit, row_tiles;
};

// Four E2M1 codes (the low 16 bits of w, one per nibble) -> the positive ones' values in halves as four bytes
// (quant/nvfp4.rs:16-30).  A byte permute looks the magnitude up by the nibble's low three bits; with the nibble's sign bit
// set it replicates the looked-up byte's top bit instead, i.e. gives 0.
__device__ __forceinline__ uint32_t e2m1_positive(uint32_t w) {
    uint32_t v; // (the __byte_perm intrinsic uses three bits of a selector)
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(0x03020100u), "r"(0x0C080604u), "r"(w));
    return v;
}
// Four int8 of the codes' values: on the codes with their sign bits flipped the permute yields the negative ones' magnitudes;
// the bias keeps the borrows of the 32-bit difference inside their bytes.
__device__ __forceinline__ uint32_t e2m1_halves(uint32_t w, uint32_t w_flipped) {
    return (e2m1_positive(w) + 0x80808080u - e2m1_positive(w_flipped)) ^ 0x80808080u;
}
__device__ __forceinline__ void imma_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Four unsigned, finite E4M3 scale codes in units of 2^-9 (nvfp4.rs:33-51), at most 229376: through f16, exact.
__device__ __forceinline__ void e4m3_q9(uint32_t codes, int (&q9)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float2 f = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(codes >> (16 * i)), __NV_E4M3)));
        q9[2 * i] = __float_as_int(__fmaf_rn(f.x, 512.0f, 12582912.0f)) - 0x4B400000;
        q9[2 * i + 1] = __float_as_int(__fmaf_rn(f.y, 512.0f, 12582912.0f)) - 0x4B400000;
    }
}
__device__ __forceinline__ uint32_t word(const uint4 &v, int i) { return (&v.x)[i]; } // compile-time i only

constexpr int kA16Warps = 8;
constexpr int a16_ctas_per_sm(int pairs) { return pairs == 1 ? 3 : 2; } // what the registers allow

// A warp contracts one 256-value block of 16 weight rows with 2 * PAIRS tokens at a time.  The codes come as they lie in
// memory: lane (g, t) loads 16 bytes of row g (and of row g + 8) of each 128-value chunk, which are the two 16-groups
// 2t and 2t + 1.  Word i of the four lanes of a row feeds one m16n8k32 product, so its 32 inputs belong to FOUR groups;
// they are told apart by the columns: column (token, q) carries the token's int8 inputs in lane q of the four and zeros
// in the others.  Three quarters of such a product are zeros, but the tensor pipe has the time (8 cycles a product and
// 4 products for 2 tokens beside ~145 other instructions), nothing is regrouped, and weights go from memory to
// registers.  Two products accumulate a group; its exact sum then meets the group's scale in a 64-bit multiply-add.
//
// CTA: 8 / ksplit row tiles; the ksplit warps of a tile take neighbouring blocks, leave their f32 contributions in
// shared memory, meet at a named barrier, and every (row, token) sum is continued front to back by one thread, so the
// order of the additions is the reference's whatever ksplit is.
//
// Two tokens: 27648 x 5120 151 -> 30 us, 5120 x 27648 222 -> 40, 1024 x 5120 23 -> 6, a layer's seven calls 699 -> 137
// (bound by instruction issue; the weights' bytes take 12 us each for the large ones).  The earlier form, one warp per
// row with eight scalar multiply-adds per lane and a 64-bit shuffle tree per token and block, had about five times the
// instructions per weight.
template <int PAIRS, int CTAS>
__global__ void __launch_bounds__(kA16Warps * 32, CTAS) nvfp4_a16_kernel(const __grid_constant__ A16Args a) {
    // With three CTAs an SM the byte-and-logic pipe bounds the kernel, and positive and negative values in products of their
    // own, which meet in the sums, cost it four instructions less per eight codes (us at two tokens: 27648 x 5120 30.9 -> 28.3,
    // 5120 x 27648 40.5 -> 36.6); with fewer warps or more tokens the products do (1024 x 5120 5.9 -> 6.4, 27648 x 5120 at 8
    // tokens 62 -> 73).
    constexpr bool kApart = CTAS == 3;
    __shared__ float contrib[2][kA16Warps][2 * PAIRS * 16];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t slot = warp / a.ksplit, part = warp % a.ksplit, slots = kA16Warps / a.ksplit;
    const uint32_t rt = blockIdx.x * slots + slot;
    // Tile u of a 128-row group holds rows 32 (m & 3) + 4 u + (m >> 2), m = 0..15: four rows that share 16 bytes of the
    // swizzled scale plane sit side by side.
    const uint32_t tile_row = (rt / 8) * 128 + 4 * (rt % 8);
    auto row_of = [&](uint32_t m) { return tile_row + 32 * (m & 3) + (m >> 2); };
    if (rt >= a.row_tiles || tile_row >= a.n_out) return; // whole slots leave; barriers are per slot
    const uint32_t blocks = a.n_in / 256, steps = (blocks + a.ksplit - 1) / a.ksplit;
    const uint8_t *code0 = a.packed + (size_t)row_of(g) * (a.n_in / 2) + 16 * t, *code1 = a.packed + (size_t)row_of(g + 8) * (a.n_in / 2) + 16 * t;
    auto scale_ptr = [&](uint32_t row) {
        return a.scales + (size_t)(row / 128) * ((size_t)a.kt * 512) + (row % 32) * 16 + ((row % 128) / 32) * 4 + (t & 1) * 512;
    };
    const uint8_t *sc0 = scale_ptr(row_of(g)), *sc1 = scale_ptr(row_of(g + 8));
    struct Block {
        uint4 c[2][2];    // [chunk][row g, row g + 8]
        uint32_t s[2][2];
    };
    auto fetch = [&](uint32_t b, Block &k) {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            k.c[ch][0] = __ldg(reinterpret_cast<const uint4 *>(code0 + (size_t)b * 128 + ch * 64));
            k.c[ch][1] = __ldg(reinterpret_cast<const uint4 *>(code1 + (size_t)b * 128 + ch * 64));
            k.s[ch][0] = __ldg(reinterpret_cast<const uint32_t *>(sc0 + (size_t)(4 * b + 2 * ch) * 512));
            k.s[ch][1] = __ldg(reinterpret_cast<const uint32_t *>(sc1 + (size_t)(4 * b + 2 * ch) * 512));
        }
    };
    Block cur, nxt;
    if (part < blocks) fetch(part, nxt);
    pdl_wait(); // the int8 activations come from the kernel before this one; weights are constants
    // (released behind the wait: what starts early finds the kernel before THIS one complete and takes no room from it)
    pdl_release();
    for (uint32_t t0 = 0; t0 < a.tokens; t0 += 2 * PAIRS) {
        if (t0 > 0 && part < blocks) fetch(part, nxt);
        const uint32_t live = min(a.tokens - t0, 2u * PAIRS);
        float total[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) total[i] = 0.0f;
        uint32_t step = 0;
        for (uint32_t b0 = 0; b0 < blocks; b0 += a.ksplit, ++step) {
            const uint32_t b = b0 + part, buffer = a16_buffer(t0 / (2 * PAIRS), steps, step);
            float *mine = contrib[buffer][warp];
            if (b < blocks) {
                cur = nxt;
                if (b + a.ksplit < blocks) fetch(b + a.ksplit, nxt);
                long long sum[PAIRS][2];
#pragma unroll
                for (int p = 0; p < PAIRS; ++p) sum[p][0] = sum[p][1] = 0;
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t av[4][4], neg[4][4]; // kApart: the positive values, and the negative ones' magnitudes
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const uint32_t w = word(cur.c[ch][r], i), f = w ^ 0x88888888u;
                            if constexpr (kApart) {
                                av[i][r] = e2m1_positive(w), neg[i][r] = e2m1_positive(f);
                                av[i][2 + r] = e2m1_positive(w >> 16), neg[i][2 + r] = e2m1_positive(f >> 16);
                            } else {
                                av[i][r] = e2m1_halves(w, f);
                                av[i][2 + r] = e2m1_halves(w >> 16, f >> 16);
                            }
                        }
                    int q0[4], q1[4]; // groups 4 (t & 1) .. + 3 of the chunk, rows g and g + 8
                    e4m3_q9(cur.s[ch][0], q0);
                    e4m3_q9(cur.s[ch][1], q1);
#pragma unroll
                    for (int p = 0; p < PAIRS; ++p) {
                        uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
                        const uint32_t tok = 2 * p + (g >> 2);
                        if ((g & 3) == t && tok < live) {
                            const uint4 *src = reinterpret_cast<const uint4 *>(a.qs + (size_t)(t0 + tok) * a.n_in + (size_t)b * 256 + ch * 128 + 32 * t);
                            x0 = ld_after_wait(src), x1 = ld_after_wait(src + 1);
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) { // groups 2q + h of the four lanes q
                            int d[4] = {0, 0, 0, 0};
                            const uint4 &x = h ? x1 : x0;
                            imma_k32(d, av[2 * h][0], av[2 * h][1], av[2 * h][2], av[2 * h][3], x.x, x.y);
                            imma_k32(d, av[2 * h + 1][0], av[2 * h + 1][1], av[2 * h + 1][2], av[2 * h + 1][3], x.z, x.w);
                            if constexpr (kApart) {
                                int n[4] = {0, 0, 0, 0};
                                imma_k32(n, neg[2 * h][0], neg[2 * h][1], neg[2 * h][2], neg[2 * h][3], x.x, x.y);
                                imma_k32(n, neg[2 * h + 1][0], neg[2 * h + 1][1], neg[2 * h + 1][2], neg[2 * h + 1][3], x.z, x.w);
#pragma unroll
                                for (int i = 0; i < 4; ++i) d[i] -= n[i];
                            }
                            sum[p][0] += (long long)d[0] * q0[h] + (long long)d[1] * q0[2 + h];
                            sum[p][1] += (long long)d[2] * q1[h] + (long long)d[3] * q1[2 + h];
                        }
                    }
                }
                // lanes t and t ^ 1 hold the two halves of the block for token 2 p + (t >> 1): the even one ends up with
                // row g, the odd one with row g + 8
                const uint32_t odd = t & 1, m = g + 8 * odd;
#pragma unroll
                for (int p = 0; p < PAIRS; ++p) {
                    const long long other = __shfl_xor_sync(0xffffffffu, odd ? sum[p][0] : sum[p][1], 1);
                    const long long whole = (odd ? sum[p][1] : sum[p][0]) + other;
                    const uint32_t tok = 2 * p + (t >> 1);
                    float c = -0.0f; // a block of zeros is skipped (nvfp4.rs:356-358): adding -0 changes nothing
                    const float d = tok < live ? ld_after_wait(a.ds + (size_t)(t0 + tok) * blocks + b) : 0.0f;
                    if (d != 0.0f) {
                        c = __fmaf_rn(__ll2float_rn(whole), 1.0f / 1024.0f, 0.0f);
                        c = __fmaf_rn(c, d, 0.0f);
                        c = __fmaf_rn(c, a.scale2, 0.0f);
                    }
                    mine[tok * 16 + m] = c;
                }
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(a.ksplit * 32) : "memory");
            const uint32_t n_here = min(a.ksplit, blocks - b0);
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const uint32_t e = part * 32 + lane + (uint32_t)i * a.ksplit * 32;
                if (e < 32u * PAIRS)
                    for (uint32_t s = 0; s < n_here; ++s) total[i] = __fmaf_rn(1.0f, contrib[buffer][slot * a.ksplit + s][e], total[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const uint32_t e = part * 32 + lane + (uint32_t)i * a.ksplit * 32, tok = e / 16, row = row_of(e % 16);
            if (e >= 32u * PAIRS || tok >= live || row >= a.n_out) continue;
            const __half h = __float2half_rn(total[i]); // the lane's output boundary (nvfp4.rs:378)
            const size_t o = (size_t)(t0 + tok) * a.n_out + row;
            if (a.y_dtype == MUSER_DTYPE_F16) reinterpret_cast<__half *>(a.y)[o] = h;
            else if (a.y_dtype == MUSER_DTYPE_BF16) reinterpret_cast<__nv_bfloat16 *>(a.y)[o] = __float2bfloat16_rn(__half2float(h));
            else reinterpret_cast<float *>(a.y)[o] = __half2float(h);
        }
    }
}

// Warps per row tile.  A block costs a warp about 500 cycles of its scheduler (mostly the byte-and-logic pipe, which takes
// an instruction every two cycles) and no less than 2500 from end to end, so a split is worth the rounds of CTAs over the
// GPU times the blocks in turn times the longer of the two.  Few rows (attn_k: 64 tiles) want all eight warps on a tile;
// so do 5120 x 27648 (320 CTAs at once against 160, one to an SM).
static uint32_t a16_ksplit(uint32_t row_tiles, uint32_t blocks, uint32_t tokens, int sm_count) {
    const int per_sm = a16_ctas_per_sm(tokens <= 2 ? 1 : 2);
    const double issue = 500.0 + 70.0 * std::min(tokens, 16u);
    uint32_t best = 1;
    double best_cost = 1e300;
    for (uint32_t ks = 1; ks <= kA16Warps; ks *= 2) {
        const uint32_t ctas = (row_tiles + kA16Warps / ks - 1) / (kA16Warps / ks);
        const double rounds = std::ceil((double)ctas / (per_sm * sm_count)), busy = std::min<double>(per_sm, std::ceil((double)ctas / sm_count));
        const double cost = rounds * std::ceil((double)blocks / ks) * std::max(busy * kA16Warps / 4 * issue, 2000.0 + issue);
        if (cost < best_cost * 0.999) best = ks, best_cost = cost;
    }
    return best;
}

// x: [tokens][n_in] f32 or bf16; the int8 codes and block scales pass through `workspace`.
muser_cuda_status launch_nvfp4_a16(Ctx *ctx, const Weight *w, const void *x, uint32_t x_dtype, void *y, uint32_t y_dtype,
                                   uint32_t tokens, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    if (w->n_in % 256) return fail(ctx, MUSER_CUDA_BAD_SHAPE, "the weight-only NVFP4 lane quantizes activations per 256: n_in % 256 != 0");
    if (w->shard.axis == MUSER_SHARD_K && w->shard.world > 1)
        return fail(ctx, MUSER_CUDA_BAD_SHAPE, "the weight-only NVFP4 lane rounds its result to f16: it cannot produce a K shard's partial sums");
    const size_t q_bytes = ((size_t)tokens * w->n_in + 15) / 16 * 16, d_bytes = (size_t)tokens * (w->n_in / 256) * sizeof(float);
    if (q_bytes + d_bytes > workspace_bytes)
        return fail(ctx, MUSER_CUDA_WORKSPACE_TOO_SMALL, "context workspace holds " + std::to_string(workspace_bytes) + " bytes, this call needs " + std::to_string(q_bytes + d_bytes));
    int8_t *qs = reinterpret_cast<int8_t *>(workspace);
    float *ds = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(workspace) + q_bytes);
    MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_q8_quantize_kernel, dim3((unsigned)(w->n_in / 256), tokens), dim3(256), 0, stream, x,
                                   (uint32_t)(x_dtype == MUSER_DTYPE_F32), (uint32_t)w->n_in, qs, ds));
    A16Args a;
    a.packed = w->packed, a.scales = w->scales, a.qs = qs, a.ds = ds, a.y = y;
    a.scale2 = w->scale2;
    a.n_out = (uint32_t)w->n_out, a.n_in = (uint32_t)w->n_in, a.kt = (uint32_t)((w->n_in + 63) / 64), a.tokens = tokens, a.y_dtype = y_dtype;
    a.row_tiles = (a.n_out + 127) / 128 * 8;
    a.ksplit = a16_ksplit(a.row_tiles, a.n_in / 256, tokens, ctx->sm_count);
    const dim3 grid((a.row_tiles * a.ksplit + kA16Warps - 1) / kA16Warps), threads(kA16Warps * 32);
    // three CTAs an SM cost the kernel for two tokens a third of its registers: only where there are as many
    // (1024 x 5120: 5.8 us with 2 an SM, 7.3 with 3; 5120 x 27648: 56 and 40)
    if (tokens <= 2 && grid.x > 2 * (unsigned)ctx->sm_count) MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_a16_kernel<1, 3>, grid, threads, 0, stream, a));
    else if (tokens <= 2) MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_a16_kernel<1, 2>, grid, threads, 0, stream, a));
    else if (tokens <= 4) MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_a16_kernel<2, 2>, grid, threads, 0, stream, a));
    else if (tokens <= 8) MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_a16_kernel<4, 2>, grid, threads, 0, stream, a));
    else MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_a16_kernel<8, 2>, grid, threads, 0, stream, a));
    return MUSER_CUDA_OK;
}

} // namespace muser
