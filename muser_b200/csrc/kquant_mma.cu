// Batched projection for Q4_K, Q5_K and Q6_K weights on the warp-level tensor instructions: y[t][r] = dot(W_r, x_t) for
// 13 to 64 tokens, up to four projections of the same input (or a fused gate/up pair) in one launch.
//
// Stands in for the batched routes of MetalKernels::encode_quantized_matmul and the speculative-verify batches of
// encode_quantized_decode_group (crates/muser-engine/src/metal/encode/qkv.rs:234-281,414-449); on the CPU lane,
// weights::matmul with quant::dot_q4_k_f32 / dot_q6_k_f32 (src/weights.rs:398-421) in the deferred-scale order of
// quant/k_block.rs:178-240 and quant/k_block/q6.rs:90-141.
//
// A kernel of its own first turns the activations into f16 fragments: every (token, 256 inputs) is scaled by a power of
// two that puts its largest magnitude between 2^9 and 2^10 (no range limit; bf16 inputs are exact down to 2^-24 of that
// maximum), f32 inputs become a head and a remainder (22 bits).  The contraction kernel's operands are then exact:
//   Q4_K, Q5_K  the integer sc * q (6-bit scale x 4- or 5-bit quant, at most 1953) times 2^-24 as f16.  Sixteen m16n8k16 products
//               accumulate a super-block of 256 inputs in f32 registers, one more product multiplies the 6-bit mins
//               with the sub-block sums (f16 head + remainder), and acc += s * (d * sum - dmin * mins) once per 256.
//   Q6_K        up to 16 tokens q - 32 as f16; one product is one 16-input sub-block, whose int8 scale is applied to the
//               f32 result (sc * (q - 32) needs 12 bits and a sign, f16 has 11); beyond 16 tokens sc * (q - 32) itself,
//               exact to 2048 and rounded to even above, as the tcgen05 kernel (kquant_tc.cu) takes it; d once per 256.
// A remainder plane accumulates into the same registers.
//
// Layout: warp = one 16-row tile of the image (kquant_layout.cuh: a lane already owns its fragment's bytes), all token
// columns in its registers; the warps of a CTA walk the same K range, so the activation fragments of a super-block are
// fetched once per CTA: one producer warp brings them and the warps' weight tiles with bulk copies into a ring of stages
// (a full and an empty barrier each).  K is cut between the CTAs of a cluster; the slices meet through distributed shared
// memory and are added in slice order, every CTA finishing its share of the outputs.
//
// What bounds it: no one unit.  Three or four warps a scheduler run chains of unpack, product and scale whose latencies are only
// partly covered.  m16n8k16 takes the tensor pipe 8.3 cycles: from 48 tokens the products are the largest part.  Figures beside takes_mma() in kquant_decode.cu.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kquant_layout.cuh"
#include "rmsnorm.cuh"
#include "tcgen05.cuh"

namespace muser {

constexpr int kMmaMaxJobs = 4, kMmaMaxSplit = 8;
// Warps on an SM, one of every CTA's being its producer, at 128 registers a thread.  (24 warps of 80 registers were no
// faster: 27648 x 5120 at 16 tokens 41.7 us against 40.2 under the same plan.)
constexpr int kMmaWarps = 16;

struct MmaJob {
    const uint8_t *image, *image_up; // image_up: second weight of the fused gate/up call, else null
    void *y;
    const float *row_scale;
    const void *residual;
    float out_scale, softcap; // LM-head tail
    uint32_t dtype, n_out, row_tiles, y_bf16, group0; // group0: first row group of this job
};
struct MmaArgs {
    MmaJob job[kMmaMaxJobs];
    const uint8_t *blob; // per super-block: fragments, min operand, scales (MmaBlob)
    int *status;
    uint32_t n_jobs, nsb, tokens, ksplit, warps, stages, stage_bytes, tile_slot;
};

// One super-block of prepared activations: [plane][32-input block j][token group][8 tokens][64 bytes], then per token
// group 256 bytes of sub-block sums (lane (g, t): heads of sums 2t, 2t + 1, remainders of the same), then one f32 scale
// per token.  The 16-byte chunk of lane t lies at chunk t ^ (g & 2), which keeps the Q6_K kernel's 8-byte reads free of
// bank conflicts.
template <int NG, int PLANES> struct MmaBlob {
    static constexpr uint32_t kPlane = 8 * NG * 512, kSums = PLANES * kPlane, kScales = kSums + NG * 256, kBytes = kScales + NG * 32;
};

__device__ __forceinline__ void hmma16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
namespace mm {
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }
__device__ __forceinline__ uint32_t gw(const uint4 &v, int i) { return (&v.x)[i]; } // compile-time i only
// bytes 2 i, 2 i + 1 of w as an f16 pair: 0x6400 | v is 1024 + v
__device__ __forceinline__ __half2 byte_pair(uint32_t w, uint32_t i, float bias = 1024.0f) {
    return __hsub2(u2h(__byte_perm(w, 0x64646464u, i ? 0x4342u : 0x4140u)), __float2half2_rn(bias));
}
// one of a pair's halves on both sides (an operand's half selection, not an instruction)
__device__ __forceinline__ __half2 both(__half2 v, int half) { return half ? __high2half2(v) : __low2half2(v); }
// byte i of w on both sides
__device__ __forceinline__ __half2 byte_twice(uint32_t w, uint32_t i) {
    return __hsub2(u2h(__byte_perm(w, 0x64646464u, 0x4040u | i | (i << 8))), __float2half2_rn(1024.0f));
}
// int8 byte i of w (biased by 128: b ^ 0x80) as f32
__device__ __forceinline__ float biased_byte(uint32_t w, uint32_t i) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | i)) - 8388736.0f; // bytes i, 0, 0, 0x4B: 2^23 + b
}

struct HdrQ45 {
    float d, dmin;
    uint32_t sc[2], mn[2]; // 6-bit values as bytes: sub-blocks 0-3, 4-7 (quant/k_block.rs:22-31)
};
__device__ __forceinline__ HdrQ45 hdr_q45(uint4 h) {
    HdrQ45 s;
    const __half2 dd = *reinterpret_cast<const __half2 *>(&h.x);
    s.d = __low2float(dd), s.dmin = __high2float(dd);
    s.sc[0] = h.y & 0x3F3F3F3Fu, s.mn[0] = h.z & 0x3F3F3F3Fu;
    s.sc[1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    s.mn[1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    return s;
}

// One tile (16 rows x 256 inputs) times all token columns, added to out[gp][i]: i = 0, 1 row g, tokens 8 gp + 2t, + 1;
// i = 2, 3 row g + 8.
template <int NG, int PLANES, bool Q5>
__device__ __forceinline__ void tile_q45(const uint8_t *tile, const uint8_t *blob, uint32_t lane, float (&out)[NG][4]) {
    using B = MmaBlob<NG, PLANES>;
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint4 *qp = reinterpret_cast<const uint4 *>(tile);
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = qp[32 * i + lane];
    uint4 hbits = make_uint4(0, 0, 0, 0);
    if constexpr (Q5) hbits = reinterpret_cast<const uint4 *>(tile + kQ5OffHi)[lane];
    const uint4 *hp = reinterpret_cast<const uint4 *>(tile + (Q5 ? kQ5OffHdr : 2048));
    const HdrQ45 ha = hdr_q45(hp[g]), hb = hdr_q45(hp[g + 8]);
    const uint8_t *frag = blob + g * 64 + ((t ^ (g & 2)) * 16);
    // A product's sum is cut off, not rounded, at its accumulator's last place: twice the products into one accumulator
    // are twice the error (1.1e-6 of the result's norm with head and remainder in one at 27 tokens, 4e-7 apart).
    constexpr bool kApart = PLANES == 2 && NG <= 4;
    float acc[NG][4], rem[kApart ? NG : 1][4];
#pragma unroll
    for (int gp = 0; gp < NG; ++gp) acc[gp][0] = acc[gp][1] = acc[gp][2] = acc[gp][3] = 0.0f;
#pragma unroll
    for (int gp = 0; gp < (kApart ? NG : 1); ++gp) rem[gp][0] = rem[gp][1] = rem[gp][2] = rem[gp][3] = 0.0f;
    // Scales two sub-blocks at a time from 17 tokens on (27648 x 5120 at 48 tokens 49.7 -> 48.6 us, 5120 x 27648 Q6_K at 32
    // 49.8 -> 48.3); below, where the kernel's Q6_K form keeps its scales in f32, that form lost its registers to it (5120 x
    // 27648 at 16 tokens 41.6 -> 44.2).
    constexpr bool kPairs = NG > 2;
    __half2 scales[2], scales16[2]; // kPairs: of sub-blocks j and j + 1, rows g and g + 8
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (kPairs && j % 2 == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                scales[r] = byte_pair(r ? hb.sc[j >> 2] : ha.sc[j >> 2], (j >> 1) & 1);
                scales16[r] = __hmul2(scales[r], __float2half2_rn(0.0625f));
            }
        }
        uint32_t av[2][4]; // [product][a0..a3]
#pragma unroll
        for (int r = 0; r < 2; ++r) { // row g, row g + 8
            const uint32_t w = gw(q[2 * r + (j >> 2)], j & 3);
            // A quant in the low bits of an f16 is that many of its smallest subnormals, 2^-24: the operand is sc * q * 2^-24,
            // exact, one mask and one product a pair.  (From 1024 + q by a fused multiply-add with -1024 sc, 27648 x 5120 at 16
            // tokens took 32.5 us instead of 28.3, 5120 x 5120 12.3 instead of 11.1.)
            const __half2 sc = kPairs ? both(scales[r], j & 1) : byte_twice(r ? hb.sc[j >> 2] : ha.sc[j >> 2], j & 3);
            auto pair = [&](uint32_t bits) { return h2u(__hmul2(u2h(bits), sc)); };
            if constexpr (Q5) {
                const uint32_t fifth = gw(hbits, 2 * r + (j >> 2));
                const uint32_t wl = (w & 0x0F0F0F0Fu) | q5_fifth(fifth, 2 * (j & 3)), wh = ((w >> 4) & 0x0F0F0F0Fu) | q5_fifth(fifth, 2 * (j & 3) + 1);
                av[0][r] = pair(wl & 0x00FF00FFu), av[0][2 + r] = pair(wh & 0x00FF00FFu);
                av[1][r] = pair((wl >> 8) & 0x00FF00FFu), av[1][2 + r] = pair((wh >> 8) & 0x00FF00FFu);
            } else {
                // the nibbles at bits 4-7 and 20-23 stay where they are, sixteen times as large
                const __half2 sc16 = kPairs ? both(scales16[r], j & 1) : __hmul2(sc, __float2half2_rn(0.0625f));
                auto pair16 = [&](uint32_t bits) { return h2u(__hmul2(u2h(bits), sc16)); };
                const uint32_t w8 = w >> 8;
                av[0][r] = pair(w & 0x000F000Fu), av[0][2 + r] = pair16(w & 0x00F000F0u);
                av[1][r] = pair(w8 & 0x000F000Fu), av[1][2 + r] = pair16(w8 & 0x00F000F0u);
            }
        }
#pragma unroll
        for (int pl = 0; pl < PLANES; ++pl)
#pragma unroll
            for (int gp = 0; gp < NG; ++gp) {
                const uint4 b = *reinterpret_cast<const uint4 *>(frag + pl * B::kPlane + (j * NG + gp) * 512);
                float(&sum)[4] = kApart && pl == 1 ? rem[kApart ? gp : 0] : acc[gp];
                hmma16(sum, av[0][0], av[0][1], av[0][2], av[0][3], b.x, b.y);
                hmma16(sum, av[1][0], av[1][1], av[1][2], av[1][3], b.z, b.w);
            }
    }
    if constexpr (kApart) {
#pragma unroll
        for (int gp = 0; gp < NG; ++gp)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[gp][i] += rem[gp][i];
    }
    const float da = ha.d * 16777216.0f, db = hb.d * 16777216.0f;
    const uint32_t sel = 0x4140u + (t & 1) * 0x0202u; // bytes 2t, 2t + 1 of the eight mins
    const uint32_t ma = h2u(__hsub2(u2h(__byte_perm(t & 2 ? ha.mn[1] : ha.mn[0], 0x64646464u, sel)), __float2half2_rn(1024.0f)));
    const uint32_t mb = h2u(__hsub2(u2h(__byte_perm(t & 2 ? hb.mn[1] : hb.mn[0], 0x64646464u, sel)), __float2half2_rn(1024.0f)));
#pragma unroll
    for (int gp = 0; gp < NG; ++gp) {
        const uint2 b = *reinterpret_cast<const uint2 *>(blob + B::kSums + gp * 256 + lane * 8);
        float m[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        hmma16(m, ma, mb, ma, mb, b.x, b.y);
        const float2 s = *reinterpret_cast<const float2 *>(blob + B::kScales + (gp * 8 + 2 * t) * 4);
        out[gp][0] = fmaf(s.x, fmaf(-ha.dmin, m[0], da * acc[gp][0]), out[gp][0]);
        out[gp][1] = fmaf(s.y, fmaf(-ha.dmin, m[1], da * acc[gp][1]), out[gp][1]);
        out[gp][2] = fmaf(s.x, fmaf(-hb.dmin, m[2], db * acc[gp][2]), out[gp][2]);
        out[gp][3] = fmaf(s.y, fmaf(-hb.dmin, m[3], db * acc[gp][3]), out[gp][3]);
    }
}

template <int NG, int PLANES>
__device__ __forceinline__ void tile_q6(const uint8_t *tile, const uint8_t *blob, uint32_t lane, float (&out)[NG][4]) {
    using B = MmaBlob<NG, PLANES>;
    constexpr bool kScaled = NG > 2; // the operand carries the sub-block's scale
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint4 *qp = reinterpret_cast<const uint4 *>(tile), *lp = reinterpret_cast<const uint4 *>(tile + kQ6OffHi);
    const uint4 *sp = reinterpret_cast<const uint4 *>(tile + kQ6OffSc);
    uint4 top[4], low[2], sc[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) top[i] = qp[32 * i + lane];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        low[i] = lp[32 * i + lane];
        sc[i] = sp[g + 8 * i];
#pragma unroll
        for (int v = 0; v < 4; ++v) (&sc[i].x)[v] ^= 0x80808080u;
    }
    const __half *dp = reinterpret_cast<const __half *>(tile + kQ6OffD);
    const float da = __half2float(dp[g]), db = __half2float(dp[g + 8]);
    // sub-block 2j + par: 8 bytes t & 1 of chunk (2 par + t / 2), see MmaBlob
    const uint8_t *frag0 = blob + g * 64 + (((t >> 1) ^ (g & 2)) * 16) + (t & 1) * 8;
    const uint8_t *frag1 = blob + g * 64 + (((2 + (t >> 1)) ^ (g & 2)) * 16) + (t & 1) * 8;
    float acc[NG][4];
#pragma unroll
    for (int gp = 0; gp < NG; ++gp) acc[gp][0] = acc[gp][1] = acc[gp][2] = acc[gp][3] = 0.0f;
    __half2 scales4[2], offsets[2]; // kScaled: sc / 4 and -288 sc of sub-blocks s and s + 1, rows g and g + 8
#pragma unroll
    for (int s = 0; s < 16; ++s) {
        if (kScaled && s % 2 == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const __half2 k = byte_pair(gw(sc[r], s >> 2), (s >> 1) & 1, 1152.0f);
                scales4[r] = __hmul2(k, __float2half2_rn(0.25f)), offsets[r] = __hmul2(k, __float2half2_rn(-288.0f));
            }
        }
        uint32_t a[4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t tw = gw(top[2 * r + (s >> 3)], (s & 7) >> 1), lw = gw(low[r], s >> 2);
            const uint32_t tp = (s & 1) ? tw : tw << 4;
            const uint32_t lo = (s & 3) == 0 ? lw << 2 : (s & 3) == 1 ? lw : (s & 3) == 2 ? lw >> 2 : lw >> 4;
            const uint32_t b = ((tp & 0xF0F0F0F0u) | (lo & 0x0C0C0C0Cu)) ^ 0x80808080u; // 4 (q - 32) + 128 per byte
            const __half2 b01 = u2h(__byte_perm(b, 0x64646464u, 0x4140u)), b23 = u2h(__byte_perm(b, 0x64646464u, 0x4342u)); // 1024 + b
            if constexpr (kScaled) { // (1024 + b) * (sc / 4) - 288 sc = sc (q - 32), rounded once
                const __half2 k4 = both(scales4[r], s & 1), off = both(offsets[r], s & 1);
                a[r] = h2u(__hfma2(b01, k4, off)), a[2 + r] = h2u(__hfma2(b23, k4, off));
            } else {
                a[r] = h2u(__hsub2(b01, __float2half2_rn(1152.0f))), a[2 + r] = h2u(__hsub2(b23, __float2half2_rn(1152.0f)));
            }
        }
        const float sa = biased_byte(gw(sc[0], s >> 2), s & 3), sb = biased_byte(gw(sc[1], s >> 2), s & 3);
#pragma unroll
        for (int gp = 0; gp < NG; ++gp) {
            float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int pl = 0; pl < PLANES; ++pl) {
                const uint2 b = *reinterpret_cast<const uint2 *>(((s & 1) ? frag1 : frag0) + pl * B::kPlane + ((s >> 1) * NG + gp) * 512);
                hmma16(kScaled ? acc[gp] : d, a[0], a[1], a[2], a[3], b.x, b.y);
            }
            if constexpr (!kScaled) {
                acc[gp][0] = fmaf(sa, d[0], acc[gp][0]);
                acc[gp][1] = fmaf(sa, d[1], acc[gp][1]);
                acc[gp][2] = fmaf(sb, d[2], acc[gp][2]);
                acc[gp][3] = fmaf(sb, d[3], acc[gp][3]);
            }
        }
    }
#pragma unroll
    for (int gp = 0; gp < NG; ++gp) {
        float2 s = *reinterpret_cast<const float2 *>(blob + B::kScales + (gp * 8 + 2 * t) * 4);
        if constexpr (!kScaled) s.x *= 0.25f, s.y *= 0.25f; // the operand was 4 (q - 32)
        out[gp][0] = fmaf(s.x * da, acc[gp][0], out[gp][0]);
        out[gp][1] = fmaf(s.y * da, acc[gp][1], out[gp][1]);
        out[gp][2] = fmaf(s.x * db, acc[gp][2], out[gp][2]);
        out[gp][3] = fmaf(s.y * db, acc[gp][3], out[gp][3]);
    }
}

__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer(uint32_t addr, uint32_t rank) { // 16 bytes of another CTA's shared memory
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
} // namespace mm

// FAM 0: Q4_K and Q6_K jobs in any mix; FAM 1: Q5_K jobs.
template <int NG, int PLANES, int FAM>
__global__ void __launch_bounds__(kMmaWarps * 32, 1) kquant_mma_kernel(const __grid_constant__ MmaArgs a) {
    using B = MmaBlob<NG, PLANES>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
    uint8_t *smem = smem_raw + (base - smem_u32(smem_raw));
    __shared__ uint64_t bars[16]; // full[8], empty[8]
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const uint32_t full = smem_u32(bars), empty = full + 64;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, W = a.warps;
    const uint32_t rank = blockIdx.x % a.ksplit, group = blockIdx.x / a.ksplit;
    uint32_t ji = 0;
#pragma unroll
    for (uint32_t i = 1; i < kMmaMaxJobs; ++i)
        if (i < a.n_jobs && group >= a.job[i].group0) ji = i;
    const MmaJob &jb = a.job[ji];
    const uint32_t lgroup = group - jb.group0, dual = jb.image_up ? 1u : 0u;
    const uint32_t tiles_cta = W >> dual, tile0 = lgroup * tiles_cta; // row tiles of this CTA (gate and up share one)
    const uint32_t k0 = a.nsb * rank / a.ksplit, n_k = a.nsb * (rank + 1) / a.ksplit - k0;
    const uint32_t tile_bytes = FAM == 1 ? kQ5TileBytes : jb.dtype == MUSER_DTYPE_Q4_K ? kQ4TileBytes : kQ6TileBytes;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, W);
        }
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    float out[NG][4];
#pragma unroll
    for (int gp = 0; gp < NG; ++gp) out[gp][0] = out[gp][1] = out[gp][2] = out[gp][3] = 0.0f;

    if (warp == W) {
        // ---------------------------------------------------------------- producer (whole warp, one elected lane issues)
        const uint32_t n_tiles = min(jb.row_tiles - tile0, tiles_cta), n_copies = n_tiles << dual;
        auto weights = [&](uint32_t i, uint32_t s) {
            const uint32_t dst = base + s * a.stage_bytes + B::kBytes;
            mbar_expect_tx_elect(full + 8 * s, B::kBytes + n_copies * tile_bytes);
            for (uint32_t c = 0; c < n_copies; ++c) {
                const uint8_t *image = dual && (c & 1) ? jb.image_up : jb.image;
                bulk_load_elect(dst + c * a.tile_slot, image + ((uint64_t)(tile0 + (c >> dual)) * a.nsb + k0 + i) * tile_bytes, tile_bytes, full + 8 * s);
            }
        };
        auto activations = [&](uint32_t i, uint32_t s) {
            bulk_load_elect(base + s * a.stage_bytes, a.blob + (size_t)(k0 + i) * B::kBytes, B::kBytes, full + 8 * s);
        };
        const uint32_t ahead = min(a.stages, n_k);
        for (uint32_t i = 0; i < ahead; ++i) weights(i, i); // constants: under the tail of the kernel that prepares the activations
        pdl_wait();
        pdl_release(); // (behind the wait: see nvfp4_a16.cu)
        for (uint32_t i = 0; i < ahead; ++i) activations(i, i);
        bool ok = true;
        uint32_t issued = ahead, s = 0, phase = 0;
        for (uint32_t i = ahead; i < n_k && ok; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait_relaxed(empty + 8 * s, phase, abort_flag, 20));
            if (!ok) break;
            weights(i, s);
            activations(i, s);
            issued = i + 1;
            if (++s == a.stages) s = 0, phase ^= 1;
        }
        if (!ok && lane == 0) {
            *abort_flag = 1;
            atomicExch(a.status + 1, 311);
        }
        // The copies in flight land before the shared memory is used for anything else, also when a consumer gave up
        // after the last copy was issued (otherwise the consumers have waited for them anyway).
        for (uint32_t i = issued > a.stages ? issued - a.stages : 0; i < issued; ++i) mbar_wait_alone(full + 8 * (i % a.stages), (i / a.stages) & 1);
    } else {
        // ---------------------------------------------------------------- one row tile per warp
        pdl_wait(); // the epilogue reads and writes what earlier kernels may still use
        const bool mine = (warp >> dual) < tiles_cta && tile0 + (warp >> dual) < jb.row_tiles; // (an odd warp has no pair)
        uint32_t s = 0, phase = 0;
        for (uint32_t i = 0; i < n_k; ++i) {
            if (!mbar_wait_warp(full + 8 * s, phase, abort_flag)) {
                if (lane == 0) {
                    *abort_flag = 1;
                    atomicExch(a.status + 1, 312);
                }
                break;
            }
            const uint8_t *blob = smem + s * a.stage_bytes, *tile = blob + B::kBytes + warp * a.tile_slot;
            if (mine) {
                if constexpr (FAM == 1) mm::tile_q45<NG, PLANES, true>(tile, blob, lane, out);
                else if (jb.dtype == MUSER_DTYPE_Q4_K) mm::tile_q45<NG, PLANES, false>(tile, blob, lane, out);
                else mm::tile_q6<NG, PLANES>(tile, blob, lane, out);
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * s) : "memory");
            if (++s == a.stages) s = 0, phase ^= 1;
        }
    }
    // ---------------------------------------------------------------- the K slices meet, and out
    __syncthreads(); // every stage has been read, or given up, and every copy has landed: the ring becomes scratch
    const uint32_t rows_cta = W * 16, row_pitch = rows_cta + 4; // (pitch: conflict-free stores)
    float *red = reinterpret_cast<float *>(smem);               // [token][row of the CTA]
    if (warp < W) {
        const uint32_t g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int gp = 0; gp < NG; ++gp)
#pragma unroll
            for (int i = 0; i < 4; ++i) red[(8 * gp + 2 * t + (i & 1)) * row_pitch + warp * 16 + g + (i >> 1) * 8] = out[gp][i];
    }
    if (a.ksplit > 1) mm::cluster_meet();
    else __syncthreads();
    const uint32_t rows_out = tiles_cta * 16, quads = a.tokens * (rows_out / 4); // four neighbouring rows of a token per step
    for (uint32_t e = rank * blockDim.x + threadIdx.x; e < quads; e += a.ksplit * blockDim.x) {
        const uint32_t tok = e / (rows_out / 4), r = (e % (rows_out / 4)) * 4, row = tile0 * 16 + r;
        if (row >= jb.n_out) continue;
        auto gather = [&](uint32_t at) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (uint32_t sl = 0; sl < a.ksplit; ++sl) {
                const float4 p = a.ksplit > 1 ? mm::ld_peer(base + (tok * row_pitch + at) * 4, sl) : *reinterpret_cast<const float4 *>(red + tok * row_pitch + at);
                v.x += p.x, v.y += p.y, v.z += p.z, v.w += p.w;
            }
            return v;
        };
        float4 v4 = gather(dual ? (r / 16) * 32 + r % 16 : r);
        float v[4] = {v4.x, v4.y, v4.z, v4.w};
        if (dual) { // silu_fast(gate) * up, quant/helpers.rs:72
            const float4 u4 = gather((r / 16) * 32 + 16 + r % 16);
            const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = __fdiv_rn(v[i], 1.0f + expf(-v[i])) * u[i];
        }
        const size_t o = (size_t)tok * jb.n_out + row;
        const uint32_t valid = min(4u, jb.n_out - row);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (jb.row_scale) v[i] *= jb.row_scale[tok];
            v[i] = logit_tail(v[i], jb.out_scale, jb.softcap);
            if (jb.residual && i < (int)valid)
                v[i] += jb.y_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(jb.residual)[o + i]) : reinterpret_cast<const float *>(jb.residual)[o + i];
        }
        if (jb.y_bf16) {
            __nv_bfloat16 *y = reinterpret_cast<__nv_bfloat16 *>(jb.y) + o;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < (int)valid) y[i] = __float2bfloat16_rn(v[i]);
        } else {
            float *y = reinterpret_cast<float *>(jb.y) + o;
            if (valid == 4 && (jb.n_out & 3) == 0) {
                *reinterpret_cast<float4 *>(y) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < (int)valid) y[i] = v[i];
            }
        }
    }
    if (a.ksplit > 1) mm::cluster_meet(); // no CTA leaves while another may read its sums
}

// Activations -> MmaBlob.  One warp per (token, super-block): lane l holds inputs 8 l .. 8 l + 7, which are chunk l % 4 of
// 32-input block l / 4.  Token columns past `tokens` are zeros.  `clamp`: magnitudes beyond f16's largest number are
// taken as that number.  With norm_weight the row is first normalized (reference.rs:73-80); every block recomputes the
// row's mean square, which costs less than a pass of its own.
template <int NG, int PLANES, bool XF32>
__global__ void __launch_bounds__(256) kquant_mma_prepare_kernel(const void *x, uint32_t tokens, uint32_t n_in, uint32_t k_off, uint32_t nsb,
                                                                 uint32_t clamp, const float *norm_weight, float norm_eps,
                                                                 uint8_t *blobs) {
    using B = MmaBlob<NG, PLANES>;
    __shared__ float red[33];
    pdl_wait();
    pdl_release(); // the contraction may fetch its first weight tiles
    const uint32_t tok = blockIdx.y, sb = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const void *row = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)tok * n_in)
                           : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)tok * n_in);
    float inv_rms = 1.0f;
    if (norm_weight && tok < tokens) inv_rms = block_inv_rms<XF32>(row, n_in, norm_eps, red); // (uniform over the block)
    if (sb >= nsb) return;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    const int64_t k = (int64_t)sb * 256 + 8 * lane - (int64_t)k_off; // a multiple of 8, like n_in: eight in or eight out
    if (tok < tokens && k >= 0 && k < (int64_t)n_in) {
        load8<XF32>(row, (uint32_t)(k / 8), v);
        if (norm_weight) {
            const float4 w0 = ld_after_wait(reinterpret_cast<const float4 *>(norm_weight + k)), w1 = ld_after_wait(reinterpret_cast<const float4 *>(norm_weight + k) + 1);
            const float nw[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], inv_rms), nw[i]);
        }
        if (clamp) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = v[i] == v[i] ? fminf(fmaxf(v[i], -65504.0f), 65504.0f) : v[i];
        }
    }
    float amax = 0.0f;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i])), nan = nan || v[i] != v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    // a NaN or an infinity makes every output of its token NaN (its operands are zero and its scale is NaN), as such
    // inputs do on the CPU lane
    const bool poisoned = __any_sync(0xffffffffu, nan) || !(amax < 3.0e38f);
    int ex = amax > 0.0f && !poisoned ? 9 - ilogbf(amax) : 0; // 2^ex brings amax to 2^9 .. 2^10
    ex = ex > 120 ? 120 : ex; // (amax below 2^-111: the operands stay smaller, nothing is lost that f32 outputs could show)
    const float up = __int_as_float((127 + ex) << 23), down = poisoned ? __int_as_float(0x7FC00000) : __int_as_float((127 - ex) << 23);
    __half2 head[4], rest[4];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float f0 = poisoned ? 0.0f : v[2 * i] * up, f1 = poisoned ? 0.0f : v[2 * i + 1] * up;
        head[i] = __floats2half2_rn(f0, f1);
        const float2 h = __half22float2(head[i]);
        rest[i] = __floats2half2_rn(f0 - h.x, f1 - h.y);
        const float2 r = __half22float2(rest[i]);
        sum += PLANES == 2 ? (h.x + r.x) + (h.y + r.y) : h.x + h.y; // of what the products see
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    uint8_t *blob = blobs + (size_t)sb * B::kBytes;
    const uint32_t gp = tok >> 3, g = tok & 7, j = lane >> 2, t = lane & 3;
    uint8_t *dst = blob + (j * NG + gp) * 512 + g * 64 + ((t ^ (g & 2)) * 16);
    *reinterpret_cast<uint4 *>(dst) = make_uint4(mm::h2u(head[0]), mm::h2u(head[1]), mm::h2u(head[2]), mm::h2u(head[3]));
    if constexpr (PLANES == 2)
        *reinterpret_cast<uint4 *>(dst + B::kPlane) = make_uint4(mm::h2u(rest[0]), mm::h2u(rest[1]), mm::h2u(rest[2]), mm::h2u(rest[3]));
    if (t == 0) { // sum j: column lane (g, j / 2), half j % 2 of its head pair and of its remainder pair
        const __half sh = __float2half_rn(sum), sr = __float2half_rn(sum - __half2float(sh));
        __half *s = reinterpret_cast<__half *>(blob + B::kSums + gp * 256 + (g * 4 + (j >> 1)) * 8);
        s[j & 1] = sh, s[2 + (j & 1)] = sr;
    }
    if (lane == 0) *reinterpret_cast<float *>(blob + B::kScales + tok * 4) = down;
}

// ------------------------------------------------------------------------------------------ host side
namespace {

struct MmaPlan {
    uint32_t warps, ksplit, stages;
};

// How many clusters of n CTAs (one CTA an SM) the device holds at once: a cluster stays inside one GPC, so sizes that do
// not divide a GPC's SMs leave some idle (a B200: 74, 45, 33, 26, 22, 15, 15 for two to eight).  Asked once per device
// and kept whatever the answer, so that the process's calls agree: a device that cannot say holds no clusters (its error is
// taken off: a launch without clusters reports errors of its own).
struct ClusterRoom {
    int n[kMmaMaxSplit + 1] = {};
};
cudaError_t cluster_room(int device, int sm_count, ClusterRoom *out) {
    static PerDevice<ClusterRoom> rooms;
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(rooms.mu);
    ClusterRoom &r = rooms.slot[device];
    if (!r.n[1]) {
        constexpr size_t kSmem = 200 * 1024;
        const void *fn = reinterpret_cast<const void *>(kquant_mma_kernel<1, 1, 0>);
        cudaError_t e = ensure_dynamic_smem(fn, device, kSmem);
        ClusterRoom found;
        for (int n = 2; n <= kMmaMaxSplit && e == cudaSuccess; ++n) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(n * 64), cfg.blockDim = dim3(kMmaWarps * 32), cfg.dynamicSmemBytes = kSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = n, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr, cfg.numAttrs = 1;
            e = cudaOccupancyMaxActiveClusters(&found.n[n], fn, &cfg);
        }
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            found = ClusterRoom{};
        }
        found.n[1] = sm_count;
        r = found;
    }
    *out = r;
    return cudaSuccess;
}

// Warps per CTA (= row tiles), K slices per cluster and ring depth.  A warp's tile costs about `tile` cycles of its
// scheduler and takes at least 1500 + 1.1 tile from end to end; the plan with the
// fewest (rounds over the GPU) x (tiles that share a scheduler) x (columns in turn) wins, the meeting of the slices
// counted as 2500 cycles.
MmaPlan mma_plan(const uint32_t *tiles, uint32_t n_jobs, bool dual, uint32_t nsb, uint32_t blob_bytes, uint32_t tile_slot, uint32_t red_tokens,
                 const ClusterRoom &room, double tile) {
    MmaPlan best{0, 0, 0};
    double best_cost = 1e300;
    // (every warp count: 1728 row tiles want twelve, 144 CTAs, where fifteen would leave a fifth of the SMs idle)
    for (uint32_t w = kMmaWarps - 1; w >= 3; --w) {
        const uint32_t stage = blob_bytes + w * tile_slot;
        for (uint32_t per_sm = 1; per_sm <= std::max(1u, kMmaWarps / ((w + 4) / 4 * 4)); ++per_sm) {
            const uint32_t bytes = (227u * 1024) / per_sm - 1024 - 512, stages = std::min(8u, bytes / stage);
            if (stages < 2 || red_tokens * (w * 16 + 4) * 4 > stages * stage) continue;
            const uint32_t per_cta = dual ? w / 2 : w;
            uint32_t groups = 0;
            for (uint32_t i = 0; i < n_jobs; ++i) groups += (tiles[i] + per_cta - 1) / per_cta;
            for (uint32_t ks = 1; ks <= (uint32_t)kMmaMaxSplit && ks <= nsb; ++ks) {
                const double slots = (double)room.n[ks] * per_sm;
                if (slots < 1.0) continue;
                const double rounds = std::ceil(groups / slots);
                const double ctas = std::min<double>(per_sm, std::ceil((double)groups / room.n[ks]));
                const double column = std::max(ctas * w / 4.0 * tile, 1500.0 + 1.1 * tile);
                const double cost = rounds * (std::ceil((double)nsb / ks) * column + (ks > 1 ? 2500.0 : 800.0));
                if (cost < best_cost * 0.999) best_cost = cost, best = {w, ks, stages};
            }
        }
    }
    return best;
}

template <int NG, int PLANES, int FAM> cudaError_t mma_launch(Ctx *ctx, const MmaArgs &a, uint32_t grid, size_t smem, cudaStream_t stream) {
    const void *fn = reinterpret_cast<const void *>(kquant_mma_kernel<NG, PLANES, FAM>);
    const cudaError_t e = ensure_dynamic_smem(fn, ctx->device, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid), cfg.blockDim = dim3((a.warps + 1) * 32), cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = a.ksplit, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = a.ksplit > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kquant_mma_kernel<NG, PLANES, FAM>, a);
}

template <int NG, int PLANES>
cudaError_t mma_run(Ctx *ctx, MmaArgs &a, const uint32_t *tiles, bool dual, bool q5, bool q6, const void *x, bool x_f32, uint32_t n_in, uint32_t k_off,
                    bool clamp, const float *norm_weight, float norm_eps, cudaStream_t stream) {
    using B = MmaBlob<NG, PLANES>;
    if ((size_t)a.nsb * B::kBytes > ctx->tc_scratch_bytes) return cudaErrorNotSupported;
    a.tile_slot = q5 ? kQ5TileBytes : q6 ? kQ6TileBytes : kQ4TileBytes;
    // the plans of the geometries this instantiation was launched with lately: working one out takes microseconds
    struct Cached {
        uint32_t nsb = 0, n_jobs = 0, tiles[kMmaMaxJobs] = {}, slot = 0;
        bool dual = false;
        MmaPlan plan{0, 0, 0};
    };
    struct CacheSet {
        Cached entry[16];
        uint32_t next = 0;
    };
    static PerDevice<CacheSet> cached;
    ClusterRoom room;
    cudaError_t e = cluster_room(ctx->device, ctx->sm_count, &room);
    if (e != cudaSuccess) return e;
    MmaPlan p;
    {
        std::lock_guard<std::mutex> lock(cached.mu);
        CacheSet &set = cached.slot[ctx->device];
        const Cached *hit = nullptr;
        for (const Cached &c : set.entry) {
            bool same = c.nsb == a.nsb && c.n_jobs == a.n_jobs && c.slot == a.tile_slot && c.dual == dual;
            for (uint32_t i = 0; same && i < a.n_jobs; ++i) same = c.tiles[i] == tiles[i];
            if (same) {
                hit = &c;
                break;
            }
        }
        if (!hit) {
            Cached &c = set.entry[set.next];
            set.next = (set.next + 1) % 16;
            c.nsb = a.nsb, c.n_jobs = a.n_jobs, c.slot = a.tile_slot, c.dual = dual;
            for (uint32_t i = 0; i < a.n_jobs; ++i) c.tiles[i] = tiles[i];
            // cycles of a scheduler per tile, fitted to 27648 x 5120 (Q4_K) and 5120 x 27648 (Q6_K) at 8 to 64 tokens
            const double tile = (q6 ? 1050.0 : 950.0) + (q6 && NG <= 2 ? 190.0 : 30.0) * NG + 130.0 * NG * PLANES;
            c.plan = mma_plan(tiles, a.n_jobs, dual, a.nsb, B::kBytes, a.tile_slot, NG * 8, room, tile);
            hit = &c;
        }
        p = hit->plan;
    }
    if (!p.warps) return cudaErrorNotSupported;
    a.warps = p.warps, a.ksplit = p.ksplit, a.stages = p.stages;
    a.stage_bytes = (B::kBytes + p.warps * a.tile_slot + 15) / 16 * 16;
    uint32_t group = 0;
    for (uint32_t i = 0; i < a.n_jobs; ++i) {
        a.job[i].group0 = group;
        const uint32_t per_cta = dual ? p.warps / 2 : p.warps;
        group += (tiles[i] + per_cta - 1) / per_cta;
    }
    uint8_t *blobs = reinterpret_cast<uint8_t *>(ctx->tc_scratch);
    a.blob = blobs;
    const dim3 pgrid((a.nsb + 7) / 8, NG * 8);
    auto prepare = [&](auto kernel) {
        return launch_pdl(kernel, pgrid, dim3(256), 0, stream, x, a.tokens, n_in, k_off, a.nsb, (uint32_t)clamp, norm_weight, norm_eps, blobs);
    };
    if constexpr (PLANES == 2) e = x_f32 ? prepare(kquant_mma_prepare_kernel<NG, 2, true>) : prepare(kquant_mma_prepare_kernel<NG, 2, false>);
    else e = prepare(kquant_mma_prepare_kernel<NG, 1, false>);
    if (e != cudaSuccess) return e;
    const size_t smem = (size_t)a.stages * a.stage_bytes + 128;
    if (q5) return mma_launch<NG, PLANES, 1>(ctx, a, group * p.ksplit, smem, stream);
    return mma_launch<NG, PLANES, 0>(ctx, a, group * p.ksplit, smem, stream);
}

} // namespace

// Up to four K-quant weights of one n_in (and one K shard geometry) applied to the same tokens; w_up: the fused gate/up
// form (one job).  cudaErrorNotSupported when the shape does not fit this kernel.  bf16 inputs behind a fused norm
// travel as f32 (two planes), like f32 inputs.
cudaError_t launch_kquant_mma(Ctx *ctx, const Weight *const *w, const Weight *w_up, uint32_t n_jobs, const void *x, uint32_t x_dtype, void *const *y,
                              const uint32_t *y_dtype, uint32_t tokens, const Epilogue *ep, bool clamp, cudaStream_t stream) {
    if (n_jobs == 0 || n_jobs > (uint32_t)kMmaMaxJobs || tokens == 0 || tokens > 64 || !ctx->tc_scratch) return cudaErrorNotSupported;
    MmaArgs a;
    uint32_t tiles[kMmaMaxJobs], n_q5 = 0, n_q6 = 0;
    for (uint32_t i = 0; i < n_jobs; ++i) {
        if (w[i]->nsb != w[0]->nsb || w[i]->k_off != w[0]->k_off || w[i]->n_in != w[0]->n_in) return cudaErrorNotSupported;
        n_q5 += w[i]->dtype == MUSER_DTYPE_Q5_K, n_q6 += w[i]->dtype == MUSER_DTYPE_Q6_K;
        MmaJob &j = a.job[i];
        j.image = w[i]->image, j.image_up = w_up ? w_up->image : nullptr;
        j.y = y[i], j.row_scale = ep[i].row_scale, j.residual = ep[i].residual;
        j.out_scale = ep[i].out_scale, j.softcap = ep[i].softcap;
        j.dtype = w[i]->dtype, j.n_out = (uint32_t)w[i]->n_out, j.row_tiles = w[i]->row_tiles;
        j.y_bf16 = y_dtype[i] == MUSER_DTYPE_BF16;
        tiles[i] = w[i]->row_tiles;
    }
    if (n_q5 != 0 && (n_q5 != n_jobs || w_up)) return cudaErrorNotSupported;
    for (uint32_t i = n_jobs; i < (uint32_t)kMmaMaxJobs; ++i) a.job[i] = a.job[0];
    a.status = ctx->dev_status;
    a.n_jobs = n_jobs, a.nsb = w[0]->nsb, a.tokens = tokens;
    const uint32_t n_in = (uint32_t)w[0]->n_in, k_off = w[0]->k_off;
    const bool xf32 = x_dtype == MUSER_DTYPE_F32;
    auto run = [&](auto ng, auto planes) {
        return mma_run<decltype(ng)::value, decltype(planes)::value>(ctx, a, tiles, w_up != nullptr, n_q5 != 0, n_q6 != 0, x, xf32, n_in, k_off, clamp,
                                                                     ep[0].norm_weight, ep[0].norm_eps, stream);
    };
    auto pick = [&](auto planes) {
        const uint32_t ng = (tokens + 7) / 8;
        if (ng <= 1) return run(std::integral_constant<int, 1>{}, planes);
        if (ng <= 2) return run(std::integral_constant<int, 2>{}, planes);
        if (ng <= 3) return run(std::integral_constant<int, 3>{}, planes);
        if (ng <= 4) return run(std::integral_constant<int, 4>{}, planes);
        if (ng <= 6) return run(std::integral_constant<int, 6>{}, planes);
        return run(std::integral_constant<int, 8>{}, planes);
    };
    return xf32 || ep[0].norm_weight ? pick(std::integral_constant<int, 2>{}) : pick(std::integral_constant<int, 1>{});
}

} // namespace muser
