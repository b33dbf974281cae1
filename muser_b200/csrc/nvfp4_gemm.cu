// NVFP4 x NVFP4 block-scaled GEMM on the 5th-generation tensor cores: y[t][n] = sum_k x[t][k] * w[n][k].
//
// Stands in for MetalKernels::encode_nvfp4_matmul / encode_nvfp4_w4a4_prequant_m16
// (crates/muser-engine/src/metal/encode/qkv.rs:13-65,128-227) and the W4A4 lane of weights::matmul
// (src/weights.rs:111-121, quant/nvfp4.rs:304-338): E2M1 codes of activations and weights, one E4M3 scale per
// 16 values on each side, then (acc * weight_scale2) * (1 / input_scale_inv) in that order.
//
// Shape of the kernel: persistent CTAs, one per SM, each walking 128-token x 256-row output tiles, or pairs of CTAs on
// 256 tokens x 256 rows where that is faster (pairs_pay; the PAIR form below).  Warp 0 streams 128-byte-swizzled
// K slabs (256 values) of both operands with TMA plus their scale factors with bulk copies through a
// 4-stage shared-memory ring; warp 1 copies each K = 64 block's scale factors into tensor memory (tcgen05.cp) and
// issues its tcgen05.mma kind::mxf4nvf4 right behind them (for pairs: a slab's copies, then its products) into a 128 x 256 f32 accumulator in tensor memory (both
// warps run their loops converged and issue through an elected lane: tcgen05.cuh);
// warps 2-17 read the accumulator back (tcgen05.ld), apply the two tensor scales and the fused epilogue, and
// store.  Every mbarrier wait is bounded: on expiry the CTA records a code in the context's status word,
// stops issuing work, waits (bounded) for its own copies in flight, frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "nvfp4_codec.cuh"
#include "nvfp4_pairs_rule.h"
#include "tcgen05.cuh"

namespace muser {

// Development aid, compiled in only with -DMUSER_GEMM_WAIT_PROFILE: the single-thread roles of the first CTAs add
// up the SM cycles they spend in each kind of wait, and a debug entry point copies the sums out.
#ifdef MUSER_GEMM_WAIT_PROFILE
__device__ unsigned long long g_wait_prof[4 * 8 * 4]; // [cta < 4][role < 8][slot < 4]
#define PROF_DECL long long prof_t0 = 0, prof_start = clock64(); unsigned long long prof_acc[3] = {0, 0, 0};
#define PROF_BEGIN prof_t0 = clock64();
#define PROF_END(i) prof_acc[i] += (unsigned long long)(clock64() - prof_t0);
#define PROF_FLUSH(role)                                                                              \
    if (blockIdx.x < 4) {                                                                             \
        for (int i_ = 0; i_ < 3; ++i_) g_wait_prof[(blockIdx.x * 8 + (role)) * 4 + i_] = prof_acc[i_]; \
        g_wait_prof[(blockIdx.x * 8 + (role)) * 4 + 3] = (unsigned long long)(clock64() - prof_start); \
    }
#else
#define PROF_DECL
#define PROF_BEGIN
#define PROF_END(i)
#define PROF_FLUSH(role)
#endif

constexpr int BM = 128, BN = 256, BK = 256;      // tile: tokens x weight rows x values
constexpr int kStages = 4;
constexpr int kABytes = BM * BK / 2;             // 16 KiB
constexpr int kBBytes = BN * BK / 2;             // 32 KiB
constexpr int kSfaBytes = 4 * 512;               // 128 rows x 16 scales
constexpr int kSfbBytes = 2 * 4 * 512;           // 256 rows x 16 scales
constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
static_assert(kSmemBytes <= 227 * 1024, "stage ring exceeds the shared memory of one CTA");
constexpr int kEpiWarps = 16, kGemmThreads = 32 * (2 + kEpiWarps);
constexpr uint32_t kTmemCols = 512;              // 256 accumulator + 16 SFA + 32 SFB, rounded to a power of two
constexpr uint32_t kSfCol = 256, kSfBufCols = 48, kSfBufs = 4; // scale buffers of 16 (SFA) + 32 (SFB) columns behind the accumulator

struct GemmArgs {
    const uint8_t *a_scales; // activations, swizzled
    const uint8_t *b_scales; // weights, swizzled
    const uint8_t *b2_scales; // second weight (up projection) of the fused gate/up form, else null
    void *y;
    const float *row_scale;
    float out_scale, softcap; // LM-head tail
    const void *residual;
    int *status;
    uint32_t tokens, n_out, k_tiles, kt64; // kt64: 64-value blocks per row (one MMA and one scale chunk each)
    uint32_t n_tiles;                      // 256-row tiles of the weight
    uint32_t y_dtype;
    float scale2, scale2_up, inv_input_scale;
    // QOUT form: the output leaves as NVFP4 activations for the next projection instead of as numbers
    uint8_t *q_packed;  // [tokens][n_out / 2]
    uint8_t *q_scales;  // swizzled, ceil(tokens / 128) x (n_out / 64) chunks
    float q_isi;        // the next projection's input_scale_inv
    uint32_t q_kt;      // n_out / 64
    uint32_t group_m;   // token tiles per raster group (tile_coords)
    uint32_t a_bytes;   // of a stage's activation box: 128 bytes per token row
    uint32_t ksplit;    // SPLIT form: CTAs of a cluster that share one tile's K
    // GROUP form: up to four projections of the same activations in one launch; weight-row tiles are numbered through
    // all of them (projection p owns tiles grp_tile0[p] .. grp_tile0[p + 1] - 1)
    uint32_t grp_tile0[5];
    const uint8_t *grp_b_scales[4];
    void *grp_y[4];
    uint32_t grp_n_out[4];
    float grp_scale2[4];
    uint32_t grp_slices[4]; // SLICED form: slices that a projection's K is summed in
};

// Output tile number -> (token tile, weight-row tile).  Tiles are numbered group by group: a group is `group_m` token
// tiles; inside it the token tile runs fastest, then the weight-row tile.  The CTAs that run side by side thus share
// a few weight tiles (read from HBM once per group, from L2 by the others) and together touch only the group's
// activations, which stay in L2 while the group sweeps all weight rows.  With every token tile in one group
// (group_m >= m_tiles, the case up to a few thousand tokens) this is "token tile fastest"; at 32768 tokens the
// activations of ffn_down alone are 453 MB, and without groups each of its 20 weight-row tiles re-read them from HBM.
__device__ __forceinline__ void tile_coords(uint32_t tile, uint32_t m_tiles, uint32_t n_tiles, uint32_t group_m, uint32_t &tile_m, uint32_t &tile_n) {
    const uint32_t per_group = group_m * n_tiles, group = tile / per_group, r = tile - group * per_group;
    const uint32_t gm = min(group_m, m_tiles - group * group_m); // the last group may be short
    tile_n = r / gm;
    tile_m = group * group_m + (r - tile_n * gm);
}

// Scale-factor chunk: 32 rows x 16 bytes, unswizzled, 8-row groups 128 bytes apart.
__device__ __forceinline__ uint64_t scale_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)(128 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// A scale copy and a product, issued by the elected lane of a warp that runs its role converged (tcgen05.cuh).
__device__ __forceinline__ void tmem_cp_scales_elect(uint32_t tmem_addr, uint64_t desc) {
    asm volatile("{\n\t" MUSER_ELECT_PRED "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n\t}" ::"r"(tmem_addr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mma_nvf4_elect(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t" MUSER_ELECT_PRED
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
        : "memory");
}
__device__ __forceinline__ void ld_32b(const void *p, uint32_t (&r)[8]) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_32b(void *p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// 64 neighbouring bytes of outputs, 16 f32 or 32 16-bit ones, in 32-byte stores where the row's pieces are whole sectors
// (`wide`; a lane's row is its own: narrower stores write half sectors) and in 16-byte stores otherwise, with the residual,
// fetched the same way (ld_64), added in f32.
__device__ __forceinline__ void ld_64(const void *p, bool wide, uint32_t (&r)[2][8]) {
    const uint8_t *at = reinterpret_cast<const uint8_t *>(p);
    if (wide) {
        ld_32b(at, r[0]), ld_32b(at + 32, r[1]);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 v = ld_after_wait(reinterpret_cast<const uint4 *>(at) + i);
        uint32_t *o = &r[i >> 1][4 * (i & 1)];
        o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
    }
}
template <typename T>
__device__ __forceinline__ void st_64(const float *v, T *y, bool has_res, const uint32_t (&res)[2][8], bool wide) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t w = res[h][i];
            if constexpr (sizeof(T) == 4) {
                o[i] = __float_as_uint(has_res ? v[8 * h + i] + __uint_as_float(w) : v[8 * h + i]);
            } else {
                float a = v[16 * h + 2 * i], b = v[16 * h + 2 * i + 1];
                if constexpr (std::is_same<T, __half>::value) {
                    const float2 r = __half22float2(*reinterpret_cast<const __half2 *>(&w));
                    if (has_res) a += r.x, b += r.y;
                    const __half2 packed = __floats2half2_rn(a, b);
                    o[i] = *reinterpret_cast<const uint32_t *>(&packed);
                } else {
                    if (has_res) a += __uint_as_float(w << 16), b += __uint_as_float(w & 0xFFFF0000u);
                    const __nv_bfloat162 packed = __floats2bfloat162_rn(a, b);
                    o[i] = *reinterpret_cast<const uint32_t *>(&packed);
                }
            }
        }
        uint8_t *at = reinterpret_cast<uint8_t *>(y) + 32 * h;
        if (wide) {
            st_32b(at, o);
        } else {
            reinterpret_cast<uint4 *>(at)[0] = make_uint4(o[0], o[1], o[2], o[3]);
            reinterpret_cast<uint4 *>(at)[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
    }
}
// One strip of 32 (or 8) columns of one accumulator row: scale, fuse, convert, store (16-byte stores when the row allows).
template <typename T, int N = 32>
__device__ __forceinline__ void store_strip(const float (&v)[N], T *y, const T *res, uint32_t valid, bool vec_ok) {
    if constexpr (sizeof(T) == 4) {
        if (vec_ok && valid == N) {
#pragma unroll
            for (int i = 0; i < N; i += 4) {
                float4 q = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                if (res) {
                    const float4 r = *reinterpret_cast<const float4 *>(res + i);
                    q.x += r.x, q.y += r.y, q.z += r.z, q.w += r.w;
                }
                *reinterpret_cast<float4 *>(y + i) = q;
            }
            return;
        }
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) // (unrolled with a predicate: a run-time index would push v[] out of registers)
            if (i < valid) y[i] = v[i] + (res ? res[i] : 0.0f);
    } else {
        auto to_f = [](T h) { if constexpr (std::is_same<T, __half>::value) return __half2float(h); else return __bfloat162float(h); };
        auto pack = [](float a, float b) -> uint32_t {
            if constexpr (std::is_same<T, __half>::value) {
                const __half2 h = __floats2half2_rn(a, b);
                return *reinterpret_cast<const uint32_t *>(&h);
            } else {
                const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
                return *reinterpret_cast<const uint32_t *>(&h);
            }
        };
        if (vec_ok && valid == N) {
#pragma unroll
            for (int i = 0; i < N; i += 8) {
                float f[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] = v[i + k];
                if (res) {
                    const uint4 r = *reinterpret_cast<const uint4 *>(res + i);
                    const T *rt = reinterpret_cast<const T *>(&r);
#pragma unroll
                    for (int k = 0; k < 8; ++k) f[k] += to_f(rt[k]);
                }
                *reinterpret_cast<uint4 *>(y + i) = make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7]));
            }
            return;
        }
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            if (i >= valid) continue;
            const float f = v[i] + (res ? to_f(res[i]) : 0.0f);
            if constexpr (std::is_same<T, __half>::value) y[i] = __float2half_rn(f); else y[i] = __float2bfloat16_rn(f);
        }
    }
}

// Clusters (SPLIT and PAIR): an address in another CTA's shared memory, and all threads of all CTAs meeting.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t cta_addr, uint32_t rank) { // shared::cta address -> that CTA's window
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(cta_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// SPLIT form: f32 sums of a tile as [row][256 columns + padding] in shared memory.
constexpr uint32_t kRedPitch = BN + 4;
static_assert((uint32_t)BM * kRedPitch * 4 <= (uint32_t)(kStages * kStageBytes), "the slices' sums exceed the stage ring");
__device__ __forceinline__ float4 split_load(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// PAIR form: a cluster of two CTAs owns a 256-token x 256-row tile (tcgen05 cta_group::2).  Each CTA holds 128 of the tokens
// (their activations, their accumulator) and HALF of the weight rows of every slab; the pair's tensor cores read both halves.
constexpr int kPStages = 5;
constexpr int kPBBytes = (BN / 2) * BK / 2; // 16 KiB: this CTA's half of the pair's 256 weight rows
constexpr int kPStageBytes = kABytes + kPBBytes + kSfaBytes + kSfbBytes;
constexpr int kOutPiece = 32 * 64;           // an epilogue warp's staging buffer: 32 rows of 64 bytes
constexpr int kPSmemBytes = kPStages * kPStageBytes + kEpiWarps * kOutPiece + 1024 + 256;
static_assert(kPSmemBytes <= 227 * 1024, "stage ring exceeds the shared memory of one CTA");

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// "Accumulator read", the one arrival of a thread on the other CTA's barrier: relaxed, because all that it orders is tensor-memory
// reads, which tcgen05.wait::ld has completed and the tcgen05 fences in front of it and behind the wait order.
__device__ __forceinline__ void mbar_arrive_accumulator_read(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Staging buffer (64-byte rows, 64-byte swizzle) -> a box of the output; columns and rows past its end are not written.
__device__ __forceinline__ void tma_store_2d_elect(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("{\n\t" MUSER_ELECT_PRED
                 "@e cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n\t@e cp.async.bulk.commit_group;\n\t}"
                 ::"l"(map), "r"(x), "r"(y), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void store_buffer_free() { // the warp's last store has read its buffer
    asm volatile("{\n\t" MUSER_ELECT_PRED "@e cp.async.bulk.wait_group.read 0;\n\t}" ::: "memory");
    __syncwarp();
}
__device__ __forceinline__ uint4 lds_16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void sts_16(uint32_t at, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// mbar_wait_relaxed and mbar_wait_warp for barriers that the other CTA of the pair arrives on (by its loads, its products' commits or its warps).
__device__ __forceinline__ bool mbar_try_pair(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done;
}
__device__ __forceinline__ bool mbar_wait_pair_relaxed(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t ns) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_pair(bar, parity)) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
        __nanosleep(ns);
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait_pair_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    bool ok = false;
    for (uint32_t i = 0; i < kSpinLimit && !ok; ++i) {
        ok = mbar_try_pair(bar, parity);
        if ((i & 1023u) == 1023u && *abort_flag) break;
    }
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void tma_load_2d_pair_elect(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("{\n\t" MUSER_ELECT_PRED
                 "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void pair_commit_elect(uint32_t cluster_addr) {
    asm volatile("{\n\t" MUSER_ELECT_PRED "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void pair_cp_scales_elect(uint32_t tmem_addr, uint64_t desc) {
    asm volatile("{\n\t" MUSER_ELECT_PRED "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n\t}" ::"r"(tmem_addr), "l"(desc) : "memory");
}
__device__ __forceinline__ void pair_mma_nvf4_elect(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                    uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t" MUSER_ELECT_PRED
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
        : "memory");
}

// A whole slab's twelve scale copies, four products and two commits ("stage consumed", to both CTAs) behind ONE election.  With
// one commit an elect.sync each and a loop around them took the issuing warp 1080 cycles a slab, unrolled 740, one election
// about 400, and the products take 512.  Chunks of 512 bytes follow one another in shared memory: four of the activations, then
// four of either half of the weight rows.  The role is entered by a branch that does not tell the compiler that its warp runs
// converged: told so, as the other roles are (they issue their loads in 128 cycles instead of 304, and the single CTAs' slabs
// are 10 % shorter), it takes 923 cycles to issue them.
#define PAIR_CP(COL, CHUNK)                                                                                                  \
    "add.u32 t, %4, " #COL ";\n\tadd.u32 v, %5, " #CHUNK " * 32;\n\tmov.b64 d, {v, %7};\n\t"                                     \
    "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [t], d;\n\t"
#define PAIR_MMA(KB, SFA, SFB, P)                                                                                            \
    "add.u32 v, %1, 2 * " #KB ";\n\tmov.b64 a, {v, %8};\n\tadd.u32 v, %2, 2 * " #KB ";\n\tmov.b64 b, {v, %8};\n\t"              \
    "add.u32 t, %4, " #SFA ";\n\tadd.u32 u, %4, " #SFB ";\n\t"                                                                 \
    "@e tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], a, b, %3, [t], [u], " P ";\n\t"
#define PAIR_HEAD "{\n\t.reg .pred q;\n\t.reg .b32 t, u, v;\n\t.reg .b64 a, b, d;\n\t" MUSER_ELECT_PRED "setp.eq.b32 q, 0, 0;\n\t"
#define PAIR_CPS                                                                                     \
    PAIR_CP(0, 0) PAIR_CP(16, 4) PAIR_CP(20, 8) PAIR_CP(4, 1) PAIR_CP(24, 5) PAIR_CP(28, 9)          \
    PAIR_CP(8, 2) PAIR_CP(32, 6) PAIR_CP(36, 10) PAIR_CP(12, 3) PAIR_CP(40, 7) PAIR_CP(44, 11)
#define PAIR_MMAS(FIRST)                                                                             \
    PAIR_MMA(0, 0, 16, FIRST) PAIR_MMA(1, 4, 24, "q") PAIR_MMA(2, 8, 32, "q") PAIR_MMA(3, 12, 40, "q") \
    "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"                                      \
    "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%9];\n\t}"
// (shared-memory addresses lie below 256 KB: the low words of operand_desc() and scale_desc() are address / 16 and constants)
#define PAIR_ARGS                                                                                                          \
    ::"r"(tmem_d), "r"((a >> 4) | (1u << 16)), "r"((b >> 4) | (1u << 16)), "r"(idesc), "r"(sf), "r"(scales >> 4),         \
        "r"(empty), "n"((128 >> 4) | (1 << 14)), "n"((1024 >> 4) | (1 << 14) | (2 << 29)), "r"(peer_empty)        \
        : "memory"
__device__ __forceinline__ void pair_slab_elect(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t sf, uint32_t scales, uint32_t empty, uint32_t peer_empty) {
    asm volatile(PAIR_HEAD PAIR_CPS PAIR_MMAS("q") PAIR_ARGS);
}
// A tile's first slab in two parts: its copies, and the products that start the accumulator anew.
__device__ __forceinline__ void pair_first_copies_elect(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t sf, uint32_t scales, uint32_t empty, uint32_t peer_empty) {
    asm volatile(PAIR_HEAD PAIR_CPS "}" PAIR_ARGS);
}
__device__ __forceinline__ void pair_first_products_elect(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t sf, uint32_t scales, uint32_t empty, uint32_t peer_empty) {
    asm volatile(PAIR_HEAD PAIR_MMAS("!q") PAIR_ARGS);
}
#undef PAIR_CP
#undef PAIR_MMA
#undef PAIR_HEAD
#undef PAIR_CPS
#undef PAIR_MMAS
#undef PAIR_ARGS

enum : int { kWhole = 0, kCluster = 1, kSliced = 2 }; // how a tile's K is cut (SPLIT)

// Tensor maps of a launch beside the activations': the weights (one, gate and up, or a group's), and for PAIR the outputs, the
// residual and all scales
// (tiled loads with the pair's qualifier run a little faster than untiled bulk copies: 560 against 594 cycles per 32 KB).
struct GemmMaps {
    CUtensorMap b[4], a_scales, b_scales[4], y[4], residual;
};

// Persistent: CTA b takes output tiles b, b + gridDim.x, ...; tile index -> (n tile, m tile) with m fastest, so the
// CTAs that run side by side share one weight tile (read from HBM once, from L2 afterwards).
//
// DUAL is the fused FFN front half (reference: encode_ffn_q4k_gate_up_silu_4r2s, src/metal/encode/ffn.rs:10-36, and
// reference.rs:511-513 on the CPU lane): the 256 accumulator columns of a tile are 128 rows of the gate weight next to
// the same 128 rows of the up weight (map_b, map_b2: 128-row boxes), and the epilogue writes silu_fast(gate) * up,
// each factor first rounded to f16 as the unfused W4A4 lane returns it (quant/nvfp4.rs:337).
// TAIL compiles the LM-head tail (logit scale, tanh soft cap) into the epilogue; the common instantiation has none of it.
// QOUT (with DUAL): silu(gate) * up is not stored but quantized on the spot for the down projection, exactly as
// quant::quantize_nvfp4_activation would quantize the f32 product (quant/nvfp4.rs:173-238): a thread holds 32
// consecutive outputs of its token, i.e. two 16-value groups = half a chunk of the swizzled scale plane, and writes
// 16 bytes of codes and two of scales.  The 27648-wide intermediate is never written or read as numbers.
// GROUP: several projections that read the same quantized activations (q | k | v) share one launch: their weight-row
// tiles form one tile space, so the small ones fill the SMs that a launch of their own would leave idle.  Plain
// outputs only (no fused tail, row scale or residual).
// SPLIT = kCluster: the slabs of one output tile are cut between the CTAs of a cluster (gemm_ksplit()): each leaves its f32 sums in
// its shared memory, and all of them add the slices up in slice order, every CTA finishing a share of the tile's outputs.
// SPLIT = kSliced (with GROUP): a group that holds weights which SPLIT cuts when they are called alone.  Tiles are whole, but
// the accumulator starts anew with every slice of such a weight and the epilogue adds the slices up as kCluster does: the bits
// of the single call in the group's one launch (where that is the faster way: group_cost).
// PAIR: pairs of SMs on 256-token tiles (above).  Both CTAs' loads report to the leader's (rank 0's) barrier of their stage, which
// expects the bytes of both; the leader issues the scale copies and the products for both and commits "stage consumed" and
// "accumulator complete" to both CTAs' barriers.  So what either CTA acts on comes from the loads and products themselves.  (A
// thread that passed its own CTA's observation on would have to release it at cluster scope: 1.7 times the time of the whole
// GEMM for "landed", 1.9 times for "consumed", at 2048 tokens.)
template <bool DUAL, bool TAIL, bool QOUT = false, bool GROUP = false, int SPLIT = kWhole, bool PAIR = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
nvfp4_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ GemmMaps maps, const GemmArgs g) {
    constexpr uint32_t kTileRows = DUAL ? BN / 2 : BN; // output columns (weight rows) per tile
    constexpr bool CLUSTER = SPLIT == kCluster, SLICED = SPLIT == kSliced;
    constexpr uint32_t kStages = PAIR ? kPStages : muser::kStages, kStageBytes = PAIR ? kPStageBytes : muser::kStageBytes;
    constexpr uint32_t kBBytes = PAIR ? kPBBytes : muser::kBBytes;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // swizzled tiles need 1024-byte alignment
    uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t out_base = base + kStages * kStageBytes; // PAIR: the epilogue warps' staging buffers
    uint64_t *bars = reinterpret_cast<uint64_t *>(aligned + kStages * kStageBytes + (PAIR ? kEpiWarps * kOutPiece : 0));
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kStages);
    const uint32_t bar_acc_full = smem_u32(bars + 2 * kStages), bar_acc_empty = smem_u32(bars + 2 * kStages + 1);
    const uint32_t bar_res = smem_u32(bars + 2 * kStages + 2); // PAIR: one per epilogue warp, "the residual has landed"
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kStages + 2 + (PAIR ? kEpiWarps : 0));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31; // (told to be the same in the whole warp)
    const uint32_t m_tiles = (g.tokens + (PAIR ? 2 : 1) * BM - 1) / ((PAIR ? 2 : 1) * BM), n_tiles_total = g.n_tiles * m_tiles;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    // This CTA's tiles and, of each, its slabs.  (Macros, so that the other forms compile as if CLUSTER did not exist: with
    // variables in their place the roles' lambdas kept them in registers and every form's slab took 10 % longer.)
#define GEMM_SLICE (CLUSTER ? blockIdx.x % g.ksplit : 0u)
#define GEMM_TILE_FIRST (CLUSTER ? blockIdx.x / g.ksplit : PAIR ? blockIdx.x >> 1 : blockIdx.x)
#define GEMM_TILE_STEP (CLUSTER ? n_tiles_total : PAIR ? gridDim.x >> 1 : gridDim.x)
#define GEMM_KT_FIRST (CLUSTER ? g.k_tiles * GEMM_SLICE / g.ksplit : 0u)
#define GEMM_KT_END (CLUSTER ? g.k_tiles * (GEMM_SLICE + 1) / g.ksplit : g.k_tiles)

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc_full, 1);
        mbar_init(bar_acc_empty, (PAIR ? 2 : 1) * kEpiWarps); // one arrival per epilogue warp (of the pair, in the leader)
        if constexpr (PAIR)
            for (int e = 0; e < kEpiWarps; ++e) mbar_init(bar_res + 8 * e, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if constexpr (PAIR) { // one warp of each CTA takes part in the paired allocation, and both CTAs' barriers exist before anything reports to them
        __syncthreads();
        cluster_barrier();
        if (warp == 1) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 0) {
        // ---------------------------------------------------------------- producer (whole warp; one elected lane issues)
        {
            uint32_t it = 0, issued = 0; // k slabs issued so far, over all tiles
            uint32_t stage = 0, phase = 1; // PAIR: of slab `it`
            bool ok = true; PROF_DECL
            const uint32_t landed = PAIR ? map_to_rank(bar_full, 0) : bar_full; // where this CTA's loads report
            const CUtensorMap *ms = nullptr; // PAIR: the scales of `mb`
            uint32_t tile_m, tile_n;
            const uint8_t *sfa, *sfb0, *sfb1;
            const CUtensorMap *mb;
            auto locate = [&](uint32_t tile) {
                tile_coords(tile, m_tiles, g.n_tiles, g.group_m, tile_m, tile_n);
                const uint8_t *b_scales = g.b_scales;
                mb = &maps.b[0];
                if constexpr (PAIR) ms = &maps.b_scales[0];
                if constexpr (GROUP) {
                    const uint32_t p = (tile_n >= g.grp_tile0[1]) + (tile_n >= g.grp_tile0[2]) + (tile_n >= g.grp_tile0[3]);
                    tile_n -= g.grp_tile0[p];
                    b_scales = g.grp_b_scales[p];
                    mb = &maps.b[p];
                    if constexpr (PAIR) ms = &maps.b_scales[p];
                }
                sfa = g.a_scales + (size_t)tile_m * g.kt64 * 512;
                sfb0 = b_scales + (size_t)(DUAL ? tile_n : 2 * tile_n) * g.kt64 * 512;
                sfb1 = DUAL ? g.b2_scales + (size_t)tile_n * g.kt64 * 512 : sfb0 + (size_t)g.kt64 * 512;
            };
            // the last slab may hold fewer than four 64-value blocks: the operand boxes are zero-filled past the row
            // end, and only the scale chunks that exist are fetched
            auto sf_bytes = [&](uint32_t kt) { return min(4u, g.kt64 - 4 * kt) * 512; };
            auto load_weights = [&](uint32_t kt, uint32_t s) {
                const uint32_t st = base + s * kStageBytes, full = landed + 8 * s;
                if constexpr (PAIR) { // (scale rows of 8-byte elements; what lies past a row's or the tensor's end arrives as zeros)
                    if (rank == 0) mbar_expect_tx_elect(bar_full + 8 * s, 2 * (g.a_bytes + kBBytes + kSfaBytes + kSfbBytes));
                    // the leader holds the tile's first 128 weight rows (the gate rows of the fused form), the other CTA the rest (up)
                    const CUtensorMap *half = DUAL ? &maps.b[rank] : mb;
                    tma_load_2d_pair_elect(st + kABytes, half, (int)(kt * (BK / 2)), (int)(DUAL ? tile_n * kTileRows : tile_n * BN + rank * (BN / 2)), full);
                    const uint32_t sfb = st + kABytes + kBBytes + kSfaBytes, x = kt * (4 * 512 / 8);
                    tma_load_2d_pair_elect(sfb, ms, (int)x, (int)(DUAL ? tile_n : 2 * tile_n), full);
                    tma_load_2d_pair_elect(sfb + 2048, DUAL ? &maps.b_scales[1] : ms, (int)x, (int)(DUAL ? tile_n : 2 * tile_n + 1), full);
                    return;
                }
                mbar_expect_tx_elect(full, g.a_bytes + kBBytes + 3 * sf_bytes(kt));
                if constexpr (DUAL) {
                    tma_load_2d_elect(st + kABytes, &maps.b[0], (int)(kt * (BK / 2)), (int)(tile_n * kTileRows), full);
                    tma_load_2d_elect(st + kABytes + kBBytes / 2, &maps.b[1], (int)(kt * (BK / 2)), (int)(tile_n * kTileRows), full);
                } else {
                    tma_load_2d_elect(st + kABytes, mb, (int)(kt * (BK / 2)), (int)(tile_n * BN), full);
                }
                bulk_load_elect(st + kABytes + kBBytes + kSfaBytes, sfb0 + (size_t)kt * 2048, sf_bytes(kt), full);
                bulk_load_elect(st + kABytes + kBBytes + kSfaBytes + 2048, sfb1 + (size_t)kt * 2048, sf_bytes(kt), full);
            };
            auto load_activations = [&](uint32_t kt, uint32_t s) {
                const uint32_t st = base + s * kStageBytes, full = landed + 8 * s;
                if constexpr (PAIR) {
                    tma_load_2d_pair_elect(st, &map_a, (int)(kt * (BK / 2)), (int)((2 * tile_m + rank) * BM), full);
                    tma_load_2d_pair_elect(st + kABytes + kBBytes, &maps.a_scales, (int)(kt * (4 * 512 / 8)), (int)(2 * tile_m + rank), full);
                    return;
                }
                tma_load_2d_elect(st, &map_a, (int)(kt * (BK / 2)), (int)(tile_m * BM), full);
                bulk_load_elect(st + kABytes + kBBytes, sfa + (size_t)kt * kSfaBytes, sf_bytes(kt), full);
            };
            // weights are constants: the first stages' are on their way before the kernel that makes the activations is done
            locate(GEMM_TILE_FIRST);
            const uint32_t ahead = min(kStages, GEMM_KT_END - GEMM_KT_FIRST);
            for (uint32_t i = 0; i < ahead; ++i) load_weights(GEMM_KT_FIRST + i, i);
            pdl_wait();
            pdl_release(); // (behind the wait: what starts early starts when the kernel before this one is complete)
            for (uint32_t tile = GEMM_TILE_FIRST; tile < n_tiles_total && ok; tile += GEMM_TILE_STEP) {
                locate(tile);
                for (uint32_t kt = GEMM_KT_FIRST; kt < GEMM_KT_END; ++kt, ++it) {
                    const uint32_t s = PAIR ? stage : it % kStages, round = it / kStages;
                    PROF_BEGIN if (PAIR) { if (it >= kStages) ok = mbar_wait_pair_warp(bar_empty + 8 * s, phase, abort_flag); } else if (round > 0) ok = mbar_wait_warp(bar_empty + 8 * s, (round - 1) & 1, abort_flag); PROF_END(0)
                    if (!ok) break;
                    if (it >= ahead) load_weights(kt, s);
                    load_activations(kt, s);
                    issued = it + 1;
                    if (PAIR && ++stage == kStages) stage = 0, phase ^= 1;
                }
            }
            if (lane == 0) { PROF_FLUSH(0) }
            if constexpr (PAIR) { // the last commits have reached this CTA's barriers before it may leave
                for (uint32_t k = issued > kStages ? issued - kStages : 0; k < issued && ok; ++k)
                    ok = mbar_wait_pair_warp(bar_empty + 8 * (k % kStages), (k / kStages) & 1, abort_flag);
            }
            if (!ok) {
                if (lane == 0) {
                    *abort_flag = 1;
                    atomicExch(g.status + 1, 101);
                }
                // let the copies already in flight land before the CTA's shared memory goes away
                // (the second CTA's report to the leader's barriers, which it cannot ask: it stays for one wait that runs out)
                if (PAIR && rank) mbar_wait_alone(bar_full, 0);
                const uint32_t first = issued > kStages ? issued - kStages : 0;
                for (uint32_t k = first; k < issued && !(PAIR && rank); ++k) {
                    uint32_t done = 0;
                    for (uint32_t i = 0; i < kSpinLimit && !done; ++i)
                        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                                     : "=r"(done) : "r"(bar_full + 8 * (k % kStages)), "r"((k / kStages) & 1) : "memory");
                }
            }
        }
    } else if (PAIR && warp == 1 && rank) { // (the leader issues for both)
    } else if (PAIR && (threadIdx.x >> 5) == 1) { // (see pair_slab_elect)
        // ---------------------------------------------------------------- MMA issuer of a pair (whole warp; one elected lane issues)
        // A pair's copies run beside the products only when the slab's are issued together in front of them (512 cycles per
        // slab in isolation, the four products' own time; three in front of each product 642).  The loop over a tile's slabs
        // holds nothing that it could do without: with the first slab's and the last one's cases inside it a slab took 545
        // cycles, and 30 more with one more flag to look at; now the products' 512 (gate/up at 2048 tokens 234 -> 220 us).
        // What is left is the change of tiles, about 1800 cycles from the last slab's issue to the next tile's first.
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
        const uint32_t peer_empty = map_to_rank(bar_empty, 1), peer_acc_full = map_to_rank(bar_acc_full, 1), whole_slabs = g.kt64 / 4;
        uint32_t local = 0, stage = 0, phase = 0;
        bool ok = true;
        auto landed = [&] {
            ok = mbar_wait_pair_warp(bar_full + 8 * stage, phase, abort_flag);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return ok;
        };
        auto drained = [&] { // the epilogue warps of both CTAs have read the previous tile
            if (local == 0) return true;
            ok = mbar_wait_pair_warp(bar_acc_empty, (local - 1) & 1, abort_flag);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return ok;
        };
        auto next_stage = [&] {
            if (++stage == kStages) stage = 0, phase ^= 1;
        };
#define PAIR_STAGE base + stage * kStageBytes, base + stage * kStageBytes + kABytes
#define PAIR_SCALES tmem + kSfCol + stage * kSfBufCols, base + stage * kStageBytes + kABytes + kBBytes
        auto ragged = [&](bool fresh) { // the end of a row
            const uint32_t st = base + stage * kStageBytes, sf = tmem + kSfCol + stage * kSfBufCols, sfa = st + kABytes + kBBytes, sfb = sfa + kSfaBytes;
            const uint64_t da = operand_desc(st), db = operand_desc(st + kABytes);
            for (uint32_t kb = 0; kb < g.kt64 % 4; ++kb) {
                pair_cp_scales_elect(sf + 4 * kb, scale_desc(sfa + 512 * kb));
                pair_cp_scales_elect(sf + 16 + 8 * kb, scale_desc(sfb + 512 * kb));
                pair_cp_scales_elect(sf + 16 + 8 * kb + 4, scale_desc(sfb + 2048 + 512 * kb));
            }
            for (uint32_t kb = 0; kb < g.kt64 % 4; ++kb)
                pair_mma_nvf4_elect(tmem, da + 2 * kb, db + 2 * kb, idesc, sf + 4 * kb, sf + 16 + 8 * kb, !fresh || kb != 0);
            pair_commit_elect(bar_empty + 8 * stage);
            pair_commit_elect(peer_empty + 8 * stage);
            next_stage();
        };
        for (uint32_t tile = GEMM_TILE_FIRST; tile < n_tiles_total; tile += GEMM_TILE_STEP, ++local) {
            if (!landed()) break;
            if (whole_slabs) {
                // the first copies go into the tensor pipe's queue behind the last tile's products, before the accumulator is free
                pair_first_copies_elect(tmem, PAIR_STAGE, idesc, PAIR_SCALES, 0, 0);
                if (!drained()) break;
                pair_first_products_elect(tmem, PAIR_STAGE, idesc, PAIR_SCALES, bar_empty + 8 * stage, peer_empty + 8 * stage);
                next_stage();
            } else {
                if (!drained()) break;
                ragged(true);
            }
            for (uint32_t i = 1; i < whole_slabs; ++i) {
                if (!landed()) break;
                pair_slab_elect(tmem, PAIR_STAGE, idesc, PAIR_SCALES, bar_empty + 8 * stage, peer_empty + 8 * stage);
                next_stage();
            }
            if (!ok) break;
            if (whole_slabs && g.kt64 % 4) {
                if (!landed()) break;
                ragged(false);
            }
            pair_commit_elect(bar_acc_full);
            pair_commit_elect(peer_acc_full);
        }
#undef PAIR_STAGE
#undef PAIR_SCALES
        if (!ok && lane == 0) {
            *abort_flag = 1;
            atomicExch(g.status + 1, 102);
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (whole warp; one elected lane issues)
        {
            // kind::mxf4nvf4: A and B E2M1 (format 1), K-major, UE4M3 scales, N >> 3 at bit 17, M >> 4 at bit 24
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            uint32_t it = 0, local = 0;
            bool ok = true; PROF_DECL
            for (uint32_t tile = GEMM_TILE_FIRST; tile < n_tiles_total && ok; tile += GEMM_TILE_STEP, ++local) {
                // the accumulator is free again once the epilogue warps have read the previous tile out of it
                if (local > 0) {
                    PROF_BEGIN ok = mbar_wait_warp(bar_acc_empty, (local - 1) & 1, abort_flag); PROF_END(0)
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                uint32_t slices = 1, slice = 0, slice_first = 0, slice_end = 0; // SLICED only
                if constexpr (SLICED) {
                    uint32_t tile_m, tile_n;
                    tile_coords(tile, m_tiles, g.n_tiles, g.group_m, tile_m, tile_n);
                    slices = g.grp_slices[(tile_n >= g.grp_tile0[1]) + (tile_n >= g.grp_tile0[2]) + (tile_n >= g.grp_tile0[3])];
                    slice_end = g.k_tiles / slices; // (kept: a division a slab took the issuing warp longer than the slab's products)
                }
                for (uint32_t kt = GEMM_KT_FIRST; kt < GEMM_KT_END; ++kt, ++it) {
                    if constexpr (SLICED) {
                        if (kt == slice_end) { // (never true at the last slice's end, where the loop ends)
                            mma_commit_elect(bar_acc_full);
                            PROF_BEGIN ok = mbar_wait_warp(bar_acc_empty, local & 1, abort_flag); PROF_END(0)
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            ++local, ++slice, slice_first = kt, slice_end = g.k_tiles * (slice + 1) / slices;
                        }
                    }
                    const uint32_t s = it % kStages, round = it / kStages;
                    PROF_BEGIN ok = mbar_wait_warp(bar_full + 8 * s, round & 1, abort_flag); PROF_END(1)
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = base + s * kStageBytes;
                    const uint64_t da = operand_desc(st), db = operand_desc(st + kABytes);
                    const uint32_t nkb = min(4u, g.kt64 - 4 * kt);
                    const uint32_t buf = it % kSfBufs, sf = tmem + kSfCol + buf * kSfBufCols;
                    // Each MMA's scale factors go to tensor memory right in front of it, from the same lane: the tensor
                    // pipe takes both in issue order, so no barrier stands between a copy and the MMA that reads it, and
                    // the copies run under the MMAs before them (691 cycles per slab in isolation against 548 for the
                    // MMAs alone).  The buffers alternate so that a copy never lands in what an earlier MMA still reads.
                    const uint32_t sfa = st + kABytes + kBBytes, sfb = sfa + kSfaBytes;
                    for (uint32_t kb = 0; kb < nkb; ++kb) { // 64 values = 32 bytes further along the swizzled 128-byte rows: +2 in 16-byte units
                        tmem_cp_scales_elect(sf + 4 * kb, scale_desc(sfa + 512 * kb));
                        tmem_cp_scales_elect(sf + 16 + 8 * kb, scale_desc(sfb + 512 * kb));
                        tmem_cp_scales_elect(sf + 16 + 8 * kb + 4, scale_desc(sfb + 2048 + 512 * kb));
                        mma_nvf4_elect(tmem, da + 2 * kb, db + 2 * kb, idesc, sf + 4 * kb, sf + 16 + 8 * kb, ((kt - (SLICED ? slice_first : GEMM_KT_FIRST)) | kb) != 0);
                    }
                    mma_commit_elect(bar_empty + 8 * s); // the stage may be overwritten once these MMAs have read it
                }
                if (ok) mma_commit_elect(bar_acc_full);
            }
            if (lane == 0) { PROF_FLUSH(1) }
            if (!ok && lane == 0) {
                *abort_flag = 1;
                atomicExch(g.status + 1, 102);
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..17)
        // Sixteen warps: four per 32-lane quarter of the accumulator, one for each quarter of the tile's output columns
        // (64, or 32 gate + 32 up).  There is room for one accumulator only, so the MMA warp cannot start the next tile
        // before the last tcgen05.ld of this one, and the rest of the epilogue runs under the next tile's products: it
        // must not take longer than those do.  With eight warps it did wherever it does more than store: gate/up +
        // quantize at 32768 tokens had two warps a scheduler waiting on each other's chains of conversions, and o_proj
        // waited for its residual behind the accumulator.
        const uint32_t quad = warp & 3;                 // the 32 accumulator lanes this warp may read
        const uint32_t part = (uint32_t)(warp - 2) >> 2; // which quarter of the output columns
        constexpr uint32_t kOutCols = DUAL ? BN / 2 : BN, kPartCols = kOutCols / 4, kStrips = kPartCols / 32;
        const uint32_t leader_acc_empty = PAIR ? map_to_rank(bar_acc_empty, 0) : 0u;
        uint32_t local = 0, res_phase = 0;
        pdl_wait(); // the residual and row scales come from, and the outputs may still be read by, earlier kernels
        for (uint32_t tile = GEMM_TILE_FIRST; tile < n_tiles_total; tile += GEMM_TILE_STEP, ++local) {
            uint32_t tile_m, tile_n;
            tile_coords(tile, m_tiles, g.n_tiles, g.group_m, tile_m, tile_n);
            uint32_t n_out = g.n_out; // (of this tile's projection)
            void *y_out = g.y;
            float scale2 = g.scale2;
            uint32_t slices = 1, grp = 0; // SLICED, GROUP only
            if constexpr (GROUP) {
                const uint32_t p = grp = (tile_n >= g.grp_tile0[1]) + (tile_n >= g.grp_tile0[2]) + (tile_n >= g.grp_tile0[3]);
                tile_n -= g.grp_tile0[p];
                n_out = g.grp_n_out[p], y_out = g.grp_y[p], scale2 = g.grp_scale2[p];
                if constexpr (SLICED) slices = g.grp_slices[p];
            }
            const uint32_t tok = (PAIR ? 2 * tile_m + rank : tile_m) * BM + quad * 32 + lane, col0 = part * kPartCols, out0 = tile_n * kOutCols + col0;
            const bool live = tok < g.tokens && out0 < n_out;
            // rows whose pieces lie on 16 bytes, and on whole 32-byte sectors
            const bool is_f32 = g.y_dtype == MUSER_DTYPE_F32;
            const uint32_t align = (uint32_t)(reinterpret_cast<uintptr_t>(y_out) | reinterpret_cast<uintptr_t>(g.residual));
            const bool vec_ok = (n_out & 7) == 0 && (align & 15) == 0, vec = vec_ok && live && out0 + kPartCols <= n_out;
            const bool wide = (align & 31) == 0 && (is_f32 || (n_out & 15) == 0);
            // the residual is fetched while the products still run: its first 64 bytes to registers, the others to L2
            uint32_t res[2][8];
            const bool vec_res = !PAIR && !DUAL && !GROUP && vec && g.residual;
            const uint8_t *res_at = reinterpret_cast<const uint8_t *>(g.residual) + ((size_t)tok * n_out + out0) * (is_f32 ? 4 : 2);
            auto load_res = [&](uint32_t piece) {
                if (vec_res) ld_64(res_at + 64 * piece, wide, res);
            };
            // PAIR: outputs leave (and the residual comes) through the warp's staging buffer, 64 bytes of 32 rows at a time.  Stored
            // straight from the registers, a row per lane, a tile's outputs kept the load/store pipe for 4000 cycles, behind
            // which the copies and products of the next tile could not be issued.
            const uint32_t buf = out_base + (uint32_t)(warp - 2) * kOutPiece, row0 = tok - lane;
            const CUtensorMap *map_y = &maps.y[0];
            if constexpr (PAIR && GROUP) map_y = &maps.y[grp];
            const bool staged_res = PAIR && !DUAL && !GROUP && g.residual;
            auto fetch_piece = [&](uint32_t n0) { // (warp-uniform)
                mbar_expect_tx_elect(bar_res + 8 * (warp - 2), kOutPiece);
                tma_load_2d_elect(buf, &maps.residual, (int)n0, (int)row0, bar_res + 8 * (warp - 2));
            };
            if constexpr (PAIR && !QOUT) {
                store_buffer_free();
                if (staged_res && row0 < g.tokens && out0 < n_out) fetch_piece(out0);
            }
            if constexpr (!PAIR && !DUAL && !GROUP) {
                load_res(0);
                if (vec_res)
                    for (uint32_t at = 64; at < kPartCols * (is_f32 ? 4 : 2); at += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(res_at + at));
            }
            // (with a sleep between the polls: sixteen polling warps cost the SM power that the products could use)
            bool ok = __all_sync(0xffffffffu, (PAIR ? mbar_wait_pair_relaxed(bar_acc_full, local & 1, abort_flag, 20) : mbar_wait_relaxed(bar_acc_full, local & 1, abort_flag, 64)));
            if (!ok) {
                if (lane == 0) {
                    *abort_flag = 1;
                    atomicCAS(g.status + 1, 0, 103);
                }
                if (staged_res && row0 < g.tokens && out0 < n_out) mbar_wait_alone(bar_res + 8 * (warp - 2), res_phase); // (it is in flight)
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float rs = (g.row_scale && tok < g.tokens) ? g.row_scale[tok] : 1.0f;
            const uint32_t lane_base = tmem + ((quad * 32) << 16);
            // All of this warp's part of the accumulator goes to registers first (64 values a thread) and the
            // accumulator is handed back at once: the MMA warp cannot start the next tile before that, so nothing
            // that touches global memory may sit in between.
            uint32_t r[2][32];
#pragma unroll
            for (uint32_t s = 0; s < 2; ++s) // fused form: strip 0 is gate columns, strip 1 the same columns of up
                tmem_ld32(lane_base + col0 + s * (DUAL ? kOutCols : 32), r[s]);
            tmem_ld_wait();
            if constexpr (SLICED) {
                if (slices > 1) { // (as SPLIT adds: from zero, in slice order)
#pragma unroll
                    for (int i = 0; i < 64; ++i) r[i >> 5][i & 31] = __float_as_uint(0.0f + __uint_as_float(r[i >> 5][i & 31]));
                }
                for (uint32_t slice = 1; slice < slices; ++slice) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty) : "memory");
                    ++local;
                    ok = mbar_wait_warp(bar_acc_full, local & 1, abort_flag); // (no sleep: the tensor pipe stands still from here on)
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 64; c += 16) { // (sixteen columns at a time: the sums so far fill the registers)
                        uint32_t v[16];
                        tmem_ld16(lane_base + col0 + c, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            uint32_t &sum = r[(c + i) >> 5][(c + i) & 31];
                            sum = __float_as_uint(__uint_as_float(sum) + __uint_as_float(v[i]));
                        }
                    }
                }
                if (!ok) {
                    if (lane == 0) {
                        *abort_flag = 1;
                        atomicCAS(g.status + 1, 0, 103);
                    }
                    break;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) mbar_arrive_accumulator_read(leader_acc_empty);
                else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty) : "memory");
            }
            if constexpr (CLUSTER) {
                // (every stage has been consumed: the ring is scratch now)
                if (tok < g.tokens) {
                    float4 *row = reinterpret_cast<float4 *>(aligned + ((quad * 32 + lane) * kRedPitch + col0) * 4);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint32_t *v = &r[i >> 3][4 * (i & 7)];
                        row[i] = make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3]));
                    }
                }
                continue;
            }
            if constexpr (QOUT) {
                // rows of the last 128-token block that hold no token get zero scale bytes: the next GEMM reads the
                // block's whole scale chunk (their codes come from TMA's zero fill)
                if (out0 < n_out && (!PAIR || (2 * tile_m + rank) * BM < g.tokens)) { // (the plane ends with the last block that holds a token)
                    uint32_t q_scales = 0; // the two scale bytes of this thread's 32 outputs
                    if (tok < g.tokens) {
                        float v[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float gate = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(__uint_as_float(r[0][i]), scale2), g.inv_input_scale)));
                            const float up = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(__uint_as_float(r[1][i]), g.scale2_up), g.inv_input_scale)));
                            v[i] = __fdiv_rn(gate, 1.0f + expf(-gate)) * up;
                        }
                        uint8_t *codes = g.q_packed + (size_t)tok * (n_out / 2) + out0 / 2;
                        const bool vec_codes = (reinterpret_cast<uintptr_t>(g.q_packed) & 15) == 0; // (rows are whole 32 bytes)
                        float(&lo)[16] = *reinterpret_cast<float(*)[16]>(&v[0]);
                        float(&hi)[16] = *reinterpret_cast<float(*)[16]>(&v[16]);
                        uint4 packed;
                        q_scales = quantize_group(lo, g.q_isi, packed.x, packed.y);
                        q_scales |= quantize_group(hi, g.q_isi, packed.z, packed.w) << 8;
                        if (vec_codes) {
                            *reinterpret_cast<uint4 *>(codes) = packed;
                        } else {
                            *reinterpret_cast<uint2 *>(codes) = make_uint2(packed.x, packed.y);
                            *reinterpret_cast<uint2 *>(codes + 8) = make_uint2(packed.z, packed.w);
                        }
                    }
                    *reinterpret_cast<uint16_t *>(g.q_scales + swizzled_scale_offset(tok, out0 / 16, g.q_kt)) = (uint16_t)q_scales;
                }
                continue;
            }
            if constexpr (PAIR) {
                auto leave = [&](auto type) {
                    using T = decltype(type);
                    constexpr int kCols = 64 / sizeof(T), kChunk = 16 / sizeof(T), kPieces = kPartCols / kCols;
#pragma unroll
                    for (int piece = 0; piece < kPieces; ++piece) {
                        const uint32_t n0 = out0 + piece * kCols;
                        if (row0 >= g.tokens || n0 >= n_out) break; // (the whole warp's)
                        if (piece > 0) {
                            store_buffer_free();
                            if (staged_res) fetch_piece(n0);
                        }
                        if (staged_res) {
                            if (!mbar_wait_warp(bar_res + 8 * (warp - 2), res_phase, abort_flag)) {
                                if (lane == 0) {
                                    *abort_flag = 1;
                                    atomicCAS(g.status + 1, 0, 105);
                                }
                                ok = false;
                                break;
                            }
                            res_phase ^= 1;
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            float v[kChunk];
#pragma unroll
                            for (int i = 0; i < kChunk; ++i) {
                                const int at = piece * kCols + c * kChunk + i;
                                v[i] = __fmul_rn(__fmul_rn(__uint_as_float(r[at >> 5][at & 31]), scale2), g.inv_input_scale);
                                if constexpr (DUAL) {
                                    const float gate = __half2float(__float2half_rn(v[i]));
                                    const float up = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(__uint_as_float(r[1][at & 31]), g.scale2_up), g.inv_input_scale)));
                                    v[i] = __fdiv_rn(gate, 1.0f + expf(-gate)) * up; // silu_fast, quant/helpers.rs:72
                                }
                                v[i] *= rs;
                                if constexpr (TAIL) v[i] = logit_tail(v[i], g.out_scale, g.softcap);
                            }
                            const uint32_t at = buf + lane * 64 + ((c ^ ((lane >> 1) & 3)) * 16);
                            uint32_t o[4], w[4] = {0, 0, 0, 0};
                            if (staged_res) {
                                const uint4 q = lds_16(at);
                                w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
                            }
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if constexpr (sizeof(T) == 4) {
                                    o[i] = __float_as_uint(staged_res ? v[i] + __uint_as_float(w[i]) : v[i]);
                                } else {
                                    float a = v[2 * i], b = v[2 * i + 1];
                                    if constexpr (std::is_same<T, __half>::value) {
                                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
                                        if (staged_res) a += f.x, b += f.y;
                                        const __half2 packed = __floats2half2_rn(a, b);
                                        o[i] = *reinterpret_cast<const uint32_t *>(&packed);
                                    } else {
                                        if (staged_res) a += __uint_as_float(w[i] << 16), b += __uint_as_float(w[i] & 0xFFFF0000u);
                                        const __nv_bfloat162 packed = __floats2bfloat162_rn(a, b);
                                        o[i] = *reinterpret_cast<const uint32_t *>(&packed);
                                    }
                                }
                            }
                            sts_16(at, o);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        tma_store_2d_elect(map_y, buf, (int)n0, (int)row0);
                    }
                };
                if (is_f32) leave(float{});
                else if (g.y_dtype == MUSER_DTYPE_BF16) leave(__nv_bfloat16{});
                else leave(__half{});
                if (!ok) break;
                continue;
            }
#pragma unroll
            for (uint32_t s = 0; s < kStrips; ++s) {
                const uint32_t n0 = out0 + 32 * s;
                if (tok >= g.tokens || n0 >= n_out) continue;
                if constexpr (!DUAL && !GROUP) {
                    if (s > 0) load_res(is_f32 ? 2 * s : s);
                }
                const size_t o = (size_t)tok * n_out + n0;
                const uint32_t valid = min(32u, n_out - n0);
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) { // quant/nvfp4.rs:334-336: tensor scales applied one after the other
                    v[i] = __fmul_rn(__fmul_rn(__uint_as_float(r[s][i]), scale2), g.inv_input_scale);
                    if constexpr (DUAL) {
                        const float gate = __half2float(__float2half_rn(v[i]));
                        const float up = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(__uint_as_float(r[1][i]), g.scale2_up), g.inv_input_scale)));
                        v[i] = __fdiv_rn(gate, 1.0f + expf(-gate)) * up; // silu_fast, quant/helpers.rs:72
                    }
                    v[i] *= rs;
                    if constexpr (TAIL) v[i] = logit_tail(v[i], g.out_scale, g.softcap);
                }
                auto store = [&](auto *y) {
                    using T = std::remove_pointer_t<decltype(y)>;
                    if (!vec) {
                        store_strip<T>(v, y + o, g.residual ? reinterpret_cast<const T *>(g.residual) + o : nullptr, valid, vec_ok);
                    } else if constexpr (sizeof(T) == 4) {
                        st_64(v, y + o, vec_res, res, wide);
                        if constexpr (!DUAL && !GROUP) load_res(2 * s + 1);
                        st_64(v + 16, y + o + 16, vec_res, res, wide);
                    } else {
                        st_64(v, y + o, vec_res, res, wide);
                    }
                };
                if (is_f32) store(reinterpret_cast<float *>(y_out));
                else if (g.y_dtype == MUSER_DTYPE_BF16) store(reinterpret_cast<__nv_bfloat16 *>(y_out));
                else store(reinterpret_cast<__half *>(y_out));
            }
        }
    }
    if constexpr (PAIR && !QOUT) // the stores are done with the staging buffers
        if (warp >= 2) asm volatile("{\n\t" MUSER_ELECT_PRED "@e cp.async.bulk.wait_group 0;\n\t}" ::: "memory");
    if constexpr (CLUSTER) {
        cluster_barrier();
        pdl_wait(); // (every warp stores here)
        uint32_t tile_m, tile_n;
        tile_coords(GEMM_TILE_FIRST, m_tiles, g.n_tiles, g.group_m, tile_m, tile_n);
        const uint32_t rows = min((uint32_t)BM, g.tokens - tile_m * BM);
        uint32_t n_out = g.n_out; // (of this tile's projection)
        void *y = g.y;
        float scale2 = g.scale2;
        if constexpr (GROUP) {
            const uint32_t p = (tile_n >= g.grp_tile0[1]) + (tile_n >= g.grp_tile0[2]) + (tile_n >= g.grp_tile0[3]);
            tile_n -= g.grp_tile0[p];
            n_out = g.grp_n_out[p], y = g.grp_y[p], scale2 = g.grp_scale2[p];
        }
        // eight columns of one row at a time: neighbouring lanes read and store neighbouring pieces
        for (uint32_t e = GEMM_SLICE * blockDim.x + threadIdx.x; e < rows * (BN / 8); e += g.ksplit * blockDim.x) {
            const uint32_t row = e / (BN / 8), c0 = (e % (BN / 8)) * 8, tok = tile_m * BM + row, n0 = tile_n * BN + c0;
            if (n0 >= n_out) continue;
            float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
            for (uint32_t p = 0; p < g.ksplit; ++p) {
                const uint32_t at = map_to_rank(base + (row * kRedPitch + c0) * 4, p);
                const float4 q0 = split_load(at), q1 = split_load(at + 16);
                v[0] += q0.x, v[1] += q0.y, v[2] += q0.z, v[3] += q0.w, v[4] += q1.x, v[5] += q1.y, v[6] += q1.z, v[7] += q1.w;
            }
            const float rs = g.row_scale ? g.row_scale[tok] : 1.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], scale2), g.inv_input_scale) * rs;
            const size_t o = (size_t)tok * n_out + n0;
            const uint32_t valid = min(8u, n_out - n0);
            const bool vec_ok = (n_out & 7) == 0 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(g.residual)) & 15) == 0;
            if (g.y_dtype == MUSER_DTYPE_F32)
                store_strip<float, 8>(v, reinterpret_cast<float *>(y) + o, g.residual ? reinterpret_cast<const float *>(g.residual) + o : nullptr, valid, vec_ok);
            else if (g.y_dtype == MUSER_DTYPE_BF16)
                store_strip<__nv_bfloat16, 8>(v, reinterpret_cast<__nv_bfloat16 *>(y) + o,
                                              g.residual ? reinterpret_cast<const __nv_bfloat16 *>(g.residual) + o : nullptr, valid, vec_ok);
            else
                store_strip<__half, 8>(v, reinterpret_cast<__half *>(y) + o, g.residual ? reinterpret_cast<const __half *>(g.residual) + o : nullptr, valid, vec_ok);
        }
        cluster_barrier(); // no CTA leaves while another may read its sums
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) {
        cluster_barrier(); // nothing of the pair is in flight towards this CTA any more
        if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    } else if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

#undef GEMM_SLICE
#undef GEMM_TILE_FIRST
#undef GEMM_TILE_STEP
#undef GEMM_KT_FIRST
#undef GEMM_KT_END

// Tensor-pipe ceiling for this instruction: every SM issues `iters` x 4 block-scaled FP4 MMAs (128 x 256 x 64 each)
// on whatever its shared and tensor memory hold, with no loads, no scale copies and no epilogue.  The time of this
// kernel is the denominator for the GEMM's roofline fraction.
__global__ void __launch_bounds__(192, 1) nvfp4_peak_kernel(uint32_t iters, int *status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
    uint64_t *bars = reinterpret_cast<uint64_t *>(aligned + kStageBytes);
    const uint32_t bar_done = smem_u32(bars);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < kStageBytes / 16; i += blockDim.x) reinterpret_cast<uint4 *>(aligned)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        mbar_init(bar_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    if (warp == 1) { // whole warp, one elected lane issues
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        const uint64_t da = operand_desc(base), db = operand_desc(base + kABytes);
        // scale factors: one copy of zeroed chunks so that the accumulator stays finite
        for (uint32_t kb = 0; kb < 4; ++kb) {
            tmem_cp_scales_elect(tmem + kSfCol + 4 * kb, scale_desc(base + kABytes + kBBytes));
            tmem_cp_scales_elect(tmem + kSfCol + 16 + 8 * kb, scale_desc(base + kABytes + kBBytes));
            tmem_cp_scales_elect(tmem + kSfCol + 16 + 8 * kb + 4, scale_desc(base + kABytes + kBBytes));
        }
        for (uint32_t i = 0; i < iters; ++i)
#pragma unroll
            for (uint32_t kb = 0; kb < 4; ++kb)
                mma_nvf4_elect(tmem, da + 2 * kb, db + 2 * kb, idesc, tmem + kSfCol + 4 * kb, tmem + kSfCol + 16 + 8 * kb, (i | kb) != 0);
        mma_commit_elect(bar_done);
        if (!mbar_wait_warp(bar_done, 0, abort_flag) && lane == 0) atomicExch(status + 1, 104);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// What the tensor pipe and the shared-memory ports do with the GEMM's instruction mix, measured in isolation: one
// thread per SM issues, per iteration (= one 256-value slab of a 128 x 256 tile), the slab's four MMAs and / or its
// scale-factor copies in a chosen order, on resident operands; another thread may stream bulk copies from an
// L2-resident buffer into shared memory beside it, as the GEMM's producer does.
//   mode 0: 4 MMAs                       mode 1: 12 copies (32x128b.warpx4), then 4 MMAs
//   mode 2: (3 copies, 1 MMA) x 4         mode 3: 12 copies only
//   mode 4: 6 copies of 128x256b only     mode 5: 6 copies of 128x256b, then 4 MMAs        mode 6: nothing (loads only)
constexpr int kProbeLoadRing = 6, kProbeLoadChunk = 18 * 1024;
constexpr int kProbeSmemBytes = kStageBytes + 16384 + kProbeLoadRing * kProbeLoadChunk + 2048;
__global__ void __launch_bounds__(192, 1) nvfp4_pipe_probe_kernel(uint32_t mode, uint32_t iters, uint32_t load_chunks, uint32_t random,
                                                                  const uint8_t *src, uint32_t src_chunks, int *status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t scales = base + kABytes + kBBytes, load_base = base + kStageBytes + 16384;
    uint64_t *bars = reinterpret_cast<uint64_t *>(aligned + kStageBytes + 16384 + kProbeLoadRing * kProbeLoadChunk);
    const uint32_t bar_done = smem_u32(bars), bar_load = smem_u32(bars + 1);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 1 + kProbeLoadRing);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < (kStageBytes + 16384) / 16; i += blockDim.x) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (random) { // non-zero E2M1 codes; scale bytes 0x30..0x3f (E4M3 0.5 .. 1.9) so that the sums stay finite
            uint32_t h = (i + 1u) * 2654435761u + blockIdx.x * 40503u;
            auto next = [&]() { h ^= h << 13; h ^= h >> 17; h ^= h << 5; return h; };
            v = make_uint4(next(), next(), next(), next());
            if (16 * i >= (uint32_t)(kABytes + kBBytes)) v.x = (v.x & 0x0f0f0f0fu) | 0x30303030u, v.y = (v.y & 0x0f0f0f0fu) | 0x30303030u, v.z = (v.z & 0x0f0f0f0fu) | 0x30303030u, v.w = (v.w & 0x0f0f0f0fu) | 0x30303030u;
        }
        reinterpret_cast<uint4 *>(aligned)[i] = v;
    }
    if (threadIdx.x == 0) {
        mbar_init(bar_done, 1);
        for (int i = 0; i < kProbeLoadRing; ++i) mbar_init(bar_load + 8 * i, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, sf = tmem + kSfCol, sf2 = sf + kSfBufCols;
    if (warp == 1 && mode != 6) { // whole warp, one elected lane issues: as the GEMM's roles do
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        const uint64_t da = operand_desc(base), db = operand_desc(base + kABytes);
        auto wide_desc = [&](uint32_t a) { // 128 rows x 32 bytes, the two halves of a row 8 KiB apart
            return (uint64_t)((a >> 4) & 0x3FFF) | (uint64_t)(8192 >> 4) << 16 | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
        };
        for (uint32_t c = 0; c < 12; ++c) tmem_cp_scales_elect(sf + 4 * c, scale_desc(scales + 512 * c)); // what the MMAs read
        for (uint32_t i = 0; i < iters; ++i) {
            if (mode == 1 || mode == 3)
                for (uint32_t c = 0; c < 12; ++c) tmem_cp_scales_elect(sf2 + 4 * c, scale_desc(scales + 512 * c));
            if (mode == 4 || mode == 5)
                for (uint32_t c = 0; c < 6; ++c) asm volatile("{\n\t" MUSER_ELECT_PRED "@e tcgen05.cp.cta_group::1.128x256b [%0], %1;\n\t}" ::"r"(sf2 + 8 * c), "l"(wide_desc(scales + 2048 * (c % 3))) : "memory");
            if (mode == 2) {
#pragma unroll
                for (uint32_t kb = 0; kb < 4; ++kb) {
                    for (uint32_t c = 0; c < 3; ++c) tmem_cp_scales_elect(sf2 + 4 * (3 * kb + c), scale_desc(scales + 512 * (3 * kb + c)));
                    mma_nvf4_elect(tmem, da + 2 * kb, db + 2 * kb, idesc, sf + 4 * kb, sf + 16 + 8 * kb, (i | kb) != 0);
                }
            } else if (mode == 0 || mode == 1 || mode == 5) {
#pragma unroll
                for (uint32_t kb = 0; kb < 4; ++kb) mma_nvf4_elect(tmem, da + 2 * kb, db + 2 * kb, idesc, sf + 4 * kb, sf + 16 + 8 * kb, (i | kb) != 0);
            }
        }
        mma_commit_elect(bar_done);
        if (!mbar_wait_warp(bar_done, 0, abort_flag) && lane == 0) atomicExch(status + 1, 107);
    }
    if (warp == 0 && load_chunks) {
        uint32_t at = (blockIdx.x * 977u) % src_chunks;
        for (uint32_t it = 0; it < load_chunks + kProbeLoadRing; ++it) {
            const uint32_t slot = it % kProbeLoadRing, bar = bar_load + 8 * slot;
            if (it >= (uint32_t)kProbeLoadRing && !mbar_wait_warp(bar, ((it / kProbeLoadRing) - 1) & 1, abort_flag)) {
                if (lane == 0) atomicExch(status + 1, 108);
                break;
            }
            if (it < load_chunks) {
                mbar_expect_tx_elect(bar, kProbeLoadChunk);
                bulk_load_elect(load_base + slot * kProbeLoadChunk, src + (size_t)at * kProbeLoadChunk, kProbeLoadChunk, bar);
                at = (at + 149u) % src_chunks;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

muser_cuda_status launch_nvfp4_pipe_probe(Ctx *ctx, uint32_t mode, uint32_t iters, uint32_t load_kib, uint32_t random, cudaStream_t stream) {
    const uint32_t chunks_per_iter = load_kib / 18, src_chunks = (uint32_t)std::min<size_t>(1024, ctx->workspace_bytes / kProbeLoadChunk);
    if (mode > 6 || load_kib % 18 || (chunks_per_iter && src_chunks < 2))
        return fail(ctx, MUSER_CUDA_BAD_ARG, "pipe probe: mode 0..6, loads in multiples of 18 KiB, and a context workspace of at least 36 KiB to read them from");
    MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(reinterpret_cast<const void *>(nvfp4_pipe_probe_kernel), ctx->device, kProbeSmemBytes));
    nvfp4_pipe_probe_kernel<<<ctx->sm_count, 192, kProbeSmemBytes, stream>>>(mode, iters, chunks_per_iter * iters, random,
                                                                            reinterpret_cast<const uint8_t *>(ctx->workspace), src_chunks, ctx->dev_status);
    MUSER_CUDA_TRY(ctx, cudaGetLastError());
    return MUSER_CUDA_OK;
}

muser_cuda_status launch_nvfp4_peak(Ctx *ctx, uint32_t iters, double *flops, cudaStream_t stream) {
    MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(reinterpret_cast<const void *>(nvfp4_peak_kernel), ctx->device, kStageBytes + 2048));
    nvfp4_peak_kernel<<<ctx->sm_count, 192, kStageBytes + 2048, stream>>>(iters, ctx->dev_status);
    MUSER_CUDA_TRY(ctx, cudaGetLastError());
    *flops = 2.0 * BM * BN * 64 * 4.0 * iters * ctx->sm_count;
    return MUSER_CUDA_OK;
}

// ------------------------------------------------------------------------------------------ host side
#ifdef MUSER_GEMM_WAIT_PROFILE
extern "C" __attribute__((visibility("default"))) int muser_cuda_debug_wait_profile(unsigned long long *out) {
    return (int)cudaMemcpyFromSymbol(out, g_wait_prof, sizeof(g_wait_prof));
}
#endif
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// rows x row_bytes, K contiguous; box = box_rows x box_bytes with the swizzle of the same width, zero fill outside.
bool tma_make_map(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t box_bytes) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {row_bytes, rows};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {box_bytes, box_rows};
    cuuint32_t elem[2] = {1, 1};
    const CUtensorMapSwizzle sw = box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                  : box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                  : box_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static bool make_map(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
    return tma_make_map(map, ptr, rows, row_bytes, box_rows, 128);
}
// A swizzled scale plane as one row of 8-byte elements per 128 operand rows; box = one slab's chunks (2048 bytes, zero fill).
static bool make_scale_map(CUtensorMap *map, const void *ptr, uint64_t blocks, uint64_t kt64) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {kt64 * 64, blocks}, strides[1] = {kt64 * 512};
    cuuint32_t box[2] = {256, 1}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void *>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// [tokens][n_out] outputs or residuals in boxes of 32 rows x 64 bytes, and whether they can be reached so.
static bool pair_rows_fit(const void *y, const void *residual, uint64_t n_out, uint32_t y_dtype) {
    return aligned16(y) && aligned16(residual) && n_out * (y_dtype == MUSER_DTYPE_F32 ? 4 : 2) % 16 == 0;
}
static bool make_out_map(CUtensorMap *map, const void *ptr, uint64_t tokens, uint64_t n_out, uint32_t y_dtype) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const uint32_t size = y_dtype == MUSER_DTYPE_F32 ? 4 : 2;
    cuuint64_t dims[2] = {n_out, tokens}, strides[1] = {n_out * size};
    cuuint32_t box[2] = {64 / size, 32}, elem[2] = {1, 1};
    return fn(map, size == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(ptr), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

muser_cuda_status nvfp4_build_tensor_map(Ctx *ctx, Weight *w) {
    struct Form {
        void **slot;
        bool scales;
        uint32_t box_rows;
    };
    const Form forms[3] = {{&w->tmap_cache, false, BN}, {&w->tmap_half, false, BN / 2}, {&w->tmap_scales, true, 1}};
    for (const Form &f : forms) {
        CUtensorMap *m = new CUtensorMap;
        *f.slot = m; // (freed with the weight)
        if (!(f.scales ? make_scale_map(m, w->scales, w->n_out_pad / 128, w->n_in / 64) : make_map(m, w->packed, w->n_out_pad, w->n_in / 2, f.box_rows)))
            return fail(ctx, MUSER_CUDA_ERROR, "cuTensorMapEncodeTiled failed for the weight image");
    }
    return MUSER_CUDA_OK;
}

void nvfp4_free_tensor_map(Weight *w) {
    delete reinterpret_cast<CUtensorMap *>(w->tmap_cache);
    delete reinterpret_cast<CUtensorMap *>(w->tmap_half);
    delete reinterpret_cast<CUtensorMap *>(w->tmap_scales);
    w->tmap_cache = w->tmap_half = w->tmap_scales = nullptr;
}

// Token rows of an activation box.  A single token tile that is not full fetches whole 8-row swizzle atoms of its tokens
// only; the stage's other rows hold whatever was there (any byte is a pair of finite E2M1 codes) and belong to outputs
// that nobody stores (gate/up + quantize at 16 tokens: 36 -> 32 us).
static uint32_t box_tokens(uint32_t tokens) { return std::min<uint32_t>(BM, (tokens + 7) / 8 * 8); }

// CTAs that share the K of one output tile.  A slab takes a CTA 0.45 us, so a long K over few tiles leaves most SMs idle:
// 5120 x 27648 has 20 tiles of 108 slabs per 128 tokens.  Split where all tiles with all their slices are on the GPU at once
// (clusters stay inside a GPC).  From 48 slabs on as often as a slice keeps eight slabs: measured are 108 slabs
// (us, whole -> split: 48 -> 20 at 16 tokens, 52 -> 29 at 128, 52 -> 34 at 384; 509 tokens are 80 tiles, whole) and rows of
// 48 (1024 x 12288 24 -> 10 at 16 tokens, 28 -> 17 at 128).  Rows of kSplitMin to 47 slabs in four or two where there are so
// few tokens that the meeting costs clearly less than the slabs: 20 slabs up to 43 tokens (5120 + 1024 + 1024 rows of 5120
// inputs 9.9 -> 6.8 us at one token, 8.7 at 16, 9.0 at 32, 9.9 at 48; 5120 x 5120 with residual 10.3 -> 8.5 at 16), 12 slabs up
// to 22 (3072 x 3072 7.4 -> 5.2 at one, 6.8 at 16).
// What the bits of a result depend on: the number of slices, i.e. the weight's rows and row length, the token count and the
// device (its SMs, and how many clusters of a size it holds).  Calls with a logit scale or soft cap, the fused gate/up form
// and contexts told to use pairs never split; a group gives the bits of the single calls.
constexpr uint32_t kSplitMin = 12;
struct SplitRoom {
    bool asked = false;
    int n[9] = {}; // clusters of n CTAs the device holds at once
};
static SplitRoom split_room(Ctx *ctx) {
    if (ctx->device < 0 || ctx->device >= kMaxDevices) return SplitRoom{};
    static PerDevice<SplitRoom> rooms;
    std::lock_guard<std::mutex> lock(rooms.mu);
    SplitRoom &room = rooms.slot[ctx->device];
    if (!room.asked) {
        // Asked once and kept whatever the answer, so that the process's calls agree: a device that cannot say holds no
        // clusters.  (Its error is taken off: whole tiles need no clusters, and the launch reports errors of its own.)
        room.asked = true;
        const auto kernel = nvfp4_gemm_kernel<false, false, false, false, kCluster>;
        cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kSmemBytes);
        for (int n = 2; n <= 8 && e == cudaSuccess; ++n) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = n, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(n * 64), cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = kSmemBytes, cfg.attrs = attr, cfg.numAttrs = 1;
            e = cudaOccupancyMaxActiveClusters(&room.n[n], kernel, &cfg);
        }
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            for (int &n : room.n) n = 0;
        }
    }
    return room;
}
// us of a tile in `ks` slices beside its launch: a slab 0.43, the meeting of the slices 0.6 and 0.075 per token row
static double split_us(uint32_t k_tiles, uint32_t ks, uint32_t tokens) {
    return std::ceil((double)k_tiles / ks) * 0.43 + (ks > 1 ? 0.6 + 0.075 * std::min<uint32_t>(tokens, BM) : 0.0);
}
static uint32_t gemm_ksplit(Ctx *ctx, const Weight *w, uint32_t tokens) {
    const uint32_t k_tiles = (uint32_t)((w->n_in + BK - 1) / BK), tiles = (uint32_t)(w->n_out_pad / BN) * ((tokens + BM - 1) / BM);
    if (k_tiles < kSplitMin || tiles * 2 > (uint32_t)ctx->sm_count) return 1;
    const SplitRoom room = split_room(ctx);
    if (k_tiles < 48) {
        for (uint32_t ks = 4; ks >= 2; ks -= 2)
            if (tokens <= (uint32_t)BM && tiles <= (uint32_t)room.n[ks] && split_us(k_tiles, ks, tokens) <= 0.7 * split_us(k_tiles, 1, tokens)) return ks;
        return 1;
    }
    for (uint32_t ks = 8; ks >= 2; --ks)
        if (tiles <= (uint32_t)room.n[ks] && k_tiles / ks >= 8) return ks;
    return 1;
}
static void cluster_launch(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&attr)[2], uint32_t ctas, uint32_t size, size_t smem, cudaStream_t stream) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = size, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas), cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cfg.attrs = attr, cfg.numAttrs = 2;
}

// ------------------------------------------------------------------------------------------ paired CTAs
// Clusters of two that the device holds at once, asked once and kept (a device that cannot say holds none).
static uint32_t pair_room(Ctx *ctx) {
    struct Room { int n = -1; };
    static PerDevice<Room> rooms;
    if (ctx->device < 0 || ctx->device >= kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(rooms.mu);
    Room &room = rooms.slot[ctx->device];
    if (room.n < 0) {
        const auto kernel = nvfp4_gemm_kernel<false, false, false, false, kWhole, true>;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(2 * 64), cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = kPSmemBytes, cfg.attrs = attr, cfg.numAttrs = 1;
        cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kPSmemBytes);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&room.n, kernel, &cfg);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            room.n = 0;
        }
    }
    return (uint32_t)std::max(0, std::min(room.n, ctx->sm_count / 2));
}
static bool takes_pairs(Ctx *ctx, uint32_t n_tiles, uint32_t tokens, uint64_t n_in, PairForm form) {
    if (ctx->nvfp4_pair != 2) return ctx->nvfp4_pair == 1;
    return pairs_pay((uint32_t)ctx->sm_count, pair_room(ctx), n_tiles, tokens, (uint32_t)((n_in + BK - 1) / BK), form);
}
template <bool DUAL, bool TAIL, bool QOUT, bool GROUP>
static cudaError_t launch_pairs(Ctx *ctx, const CUtensorMap &map_a, const GemmMaps &maps, const GemmArgs &g, cudaStream_t stream) {
    const auto kernel = nvfp4_gemm_kernel<DUAL, TAIL, QOUT, GROUP, kWhole, true>;
    const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kPSmemBytes);
    if (e != cudaSuccess) return e;
    const uint32_t room = pair_room(ctx);
    if (!room) return cudaErrorNotSupported;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cluster_launch(cfg, attr, 2 * std::min(room, g.n_tiles * ((g.tokens + 2 * BM - 1) / (2 * BM))), 2, kPSmemBytes, stream);
    return cudaLaunchKernelEx(&cfg, kernel, map_a, maps, g);
}

// Token tiles (of 128, or of 256 where pairs take them) per raster group: about 32 MB of activations, at least 8 x 128 tokens.
static uint32_t raster_group(Ctx *ctx, const Weight *w, uint32_t m_blocks, bool pair) {
    const uint64_t tile_bytes = (uint64_t)BM * (w->n_in / 2 + w->n_in / 16);
    uint32_t gm = (uint32_t)std::max<uint64_t>(8, (32ull << 20) / std::max<uint64_t>(1, tile_bytes));
    if (ctx->nvfp4_group_m) gm = ctx->nvfp4_group_m;
    gm = std::max<uint32_t>(1, std::min<uint32_t>(gm, m_blocks));
    return pair ? (gm + 1) / 2 : gm;
}

muser_cuda_status launch_nvfp4_gemm(Ctx *ctx, const Weight *w, const uint8_t *x_packed, const uint8_t *x_scales, void *y,
                                    uint32_t y_dtype, uint32_t tokens, const Epilogue &ep, cudaStream_t stream,
                                    const Weight *w_up, const NvFp4Out *qout) {
    const uint32_t m_blocks = (tokens + BM - 1) / BM, n_tiles = w_up ? (uint32_t)((w->n_out + BN / 2 - 1) / (BN / 2)) : (uint32_t)(w->n_out_pad / BN);
    const bool tail = ep.out_scale != 1.0f || ep.softcap > 0.0f;
    const uint32_t ks = w_up || tail || ctx->nvfp4_pair == 1 ? 1 : gemm_ksplit(ctx, w, tokens);
    const bool pair = ks == 1 && takes_pairs(ctx, n_tiles, tokens, w->n_in, w_up ? PairForm::fused : PairForm::plain) && (qout || pair_rows_fit(y, ep.residual, w->n_out, y_dtype));
    const uint32_t a_rows = pair ? BM : box_tokens(tokens);
    CUtensorMap map_a;
    GemmMaps maps;
    if (!make_map(&map_a, x_packed, tokens, w->n_in / 2, a_rows) || (pair && !make_scale_map(&maps.a_scales, x_scales, m_blocks, w->n_in / 64)))
        return fail(ctx, MUSER_CUDA_ERROR, "cuTensorMapEncodeTiled failed for the activations");
    GemmArgs g;
    g.a_scales = x_scales;
    g.b_scales = w->scales;
    g.b2_scales = w_up ? w_up->scales : nullptr;
    g.y = y;
    g.row_scale = ep.row_scale;
    g.out_scale = ep.out_scale;
    g.softcap = ep.softcap;
    g.residual = ep.residual;
    g.status = ctx->dev_status;
    g.tokens = tokens;
    g.a_bytes = a_rows * (BK / 2);
    g.ksplit = 1;
    g.n_out = (uint32_t)w->n_out;
    g.k_tiles = (uint32_t)((w->n_in + BK - 1) / BK);
    g.kt64 = (uint32_t)(w->n_in / 64);
    g.y_dtype = y_dtype;
    g.scale2 = w->scale2;
    g.scale2_up = w_up ? w_up->scale2 : 0.0f;
    g.inv_input_scale = 1.0f / w->input_scale_inv;
    g.n_tiles = n_tiles;
    g.q_packed = qout ? qout->packed : nullptr;
    g.q_scales = qout ? qout->scales : nullptr;
    g.q_isi = qout ? qout->input_scale_inv : 0.0f;
    g.q_kt = (uint32_t)(w->n_out / 64);
    g.group_m = raster_group(ctx, w, m_blocks, pair);
    if (qout && (!w_up || w->n_out % 64)) return fail(ctx, MUSER_CUDA_BAD_SHAPE, "quantized outputs come from the fused gate/up form, with n_out % 64 == 0");
    // (the fused form's boxes hold 128 rows of either weight, a pair's the 128 rows of one CTA)
    maps.b[0] = *reinterpret_cast<const CUtensorMap *>(w_up || pair ? w->tmap_half : w->tmap_cache);
    if (w_up) maps.b[1] = *reinterpret_cast<const CUtensorMap *>(w_up->tmap_half);
    if (pair) {
        maps.b_scales[0] = *reinterpret_cast<const CUtensorMap *>(w->tmap_scales);
        if (w_up) maps.b_scales[1] = *reinterpret_cast<const CUtensorMap *>(w_up->tmap_scales);
        if (!qout && (!make_out_map(&maps.y[0], y, tokens, w->n_out, y_dtype) || (ep.residual && !make_out_map(&maps.residual, ep.residual, tokens, w->n_out, y_dtype))))
            return fail(ctx, MUSER_CUDA_ERROR, "cuTensorMapEncodeTiled failed for the outputs");
        MUSER_CUDA_TRY(ctx, qout   ? (launch_pairs<true, false, true, false>(ctx, map_a, maps, g, stream))
                            : w_up ? (launch_pairs<true, false, false, false>(ctx, map_a, maps, g, stream)) // (the fused FFN form has no tail)
                            : tail ? (launch_pairs<false, true, false, false>(ctx, map_a, maps, g, stream))
                                   : (launch_pairs<false, false, false, false>(ctx, map_a, maps, g, stream)));
        return MUSER_CUDA_OK;
    }
    const uint32_t tiles = g.n_tiles * m_blocks;
    if (ks > 1) {
        g.ksplit = ks;
        const auto kernel = nvfp4_gemm_kernel<false, false, false, false, kCluster>;
        MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kSmemBytes));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        cluster_launch(cfg, attr, tiles * ks, ks, kSmemBytes, stream);
        MUSER_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, map_a, maps, g));
        return MUSER_CUDA_OK;
    }
    const uint32_t grid = tiles < (uint32_t)ctx->sm_count ? tiles : (uint32_t)ctx->sm_count;
    // (the attribute is per device: set where the launch happens, with the launching context's device current)
    const void *kfn = w_up ? reinterpret_cast<const void *>(nvfp4_gemm_kernel<true, false>)
                      : tail ? reinterpret_cast<const void *>(nvfp4_gemm_kernel<false, true>)
                             : reinterpret_cast<const void *>(nvfp4_gemm_kernel<false, false>);
    MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(kfn, ctx->device, kSmemBytes));
    if (qout) {
        const void *qfn = reinterpret_cast<const void *>(nvfp4_gemm_kernel<true, false, true>);
        MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(qfn, ctx->device, kSmemBytes));
        MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_gemm_kernel<true, false, true>, dim3(grid), dim3(kGemmThreads), kSmemBytes, stream, map_a, maps, g));
    } else if (w_up)
        MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_gemm_kernel<true, false>, dim3(grid), dim3(kGemmThreads), kSmemBytes, stream, map_a, maps, g)); // (the fused FFN form has no tail)
    else if (tail)
        MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_gemm_kernel<false, true>, dim3(grid), dim3(kGemmThreads), kSmemBytes, stream, map_a, maps, g));
    else
        MUSER_CUDA_TRY(ctx, launch_pdl(nvfp4_gemm_kernel<false, false>, dim3(grid), dim3(kGemmThreads), kSmemBytes, stream, map_a, maps, g));
    MUSER_CUDA_TRY(ctx, cudaGetLastError());
    return MUSER_CUDA_OK;
}

// A group that holds weights which are split when they are called alone: one launch of whole tiles (SLICED), or each of
// those weights in a launch of its own and the rest in one?  In us: a slab of a tile 0.43 or the weights' bytes at 6.5 TB/s,
// a launch about 4, a change of slices 0.5, the meeting of the slices 0.6 and 0.075 per token row of a tile.  Measured, one
// launch / apart: 3 x 1024 rows of 27648 inputs 53 / 40 at 16 tokens, 54 / 54 at 100, 55 / 64 at 200; 2048 + 512 + 512 of
// 12288 27 / 25 at 8, 26 / 29 at 16, 28 / 51 at 128; 12288 + 1024 + 1024 of 12288 28 / 36 at 8, 31 / 63 at 256.  (Not split
// at all, with other bits than the single calls': 50, 51, 52; 25, 25, 27; 28, 32.)
struct GroupCost {
    double one_launch, apart;
};
static GroupCost group_cost(const uint32_t *slices, const Weight *const *ws, uint32_t n, uint32_t tokens, int sm_count) {
    const uint32_t m_tiles = (tokens + BM - 1) / BM, k_tiles = (uint32_t)((ws[0]->n_in + BK - 1) / BK);
    const auto bytes_us = [&](uint32_t tiles) { return (double)tiles / m_tiles * BN * ws[0]->n_in * 0.5625 / 6.5e6; };
    const auto whole_us = [&](uint32_t tiles) { return tiles ? std::max(std::ceil((double)tiles / sm_count) * k_tiles * 0.43, bytes_us(tiles)) + 4.0 : 0.0; };
    uint32_t all = 0, unsplit = 0, most = 1;
    double apart = 0.0;
    for (uint32_t p = 0; p < n; ++p) {
        const uint32_t tiles = (uint32_t)(ws[p]->n_out_pad / BN) * m_tiles;
        all += tiles, most = std::max(most, slices[p]);
        if (slices[p] > 1) apart += std::max(std::ceil((double)k_tiles / slices[p]) * 0.43, bytes_us(tiles)) + 4.6 + 0.075 * std::min<uint32_t>(tokens, BM);
        else unsplit += tiles;
    }
    return GroupCost{whole_us(all) + (most - 1) * 0.5, apart + whole_us(unsplit)};
}

// Up to four projections of the same quantized activations in one launch (GROUP form of the kernel).
muser_cuda_status launch_nvfp4_gemm_group(Ctx *ctx, const Weight *const *ws, uint32_t n, const uint8_t *x_packed, const uint8_t *x_scales,
                                          void *const *ys, uint32_t y_dtype, uint32_t tokens, cudaStream_t stream) {
    const Weight *w0 = ws[0];
    uint32_t slices[4] = {1, 1, 1, 1}; // (the paired kernel, which serves single calls where it is on, never splits)
    bool sliced = false;
    for (uint32_t p = 0; p < n && ctx->nvfp4_pair != 1; ++p) slices[p] = gemm_ksplit(ctx, ws[p], tokens), sliced = sliced || slices[p] > 1;
    // All of them in the same number of slices and all clusters on the GPU at once: clusters.  (In two rounds 5120 + 2560 + 2560
    // rows of 5120 inputs took 15.4 us at 16 tokens, whole tiles with sliced sums 12.)
    const uint32_t m_blocks = (tokens + BM - 1) / BM;
    uint32_t tiles_n = 0;
    for (uint32_t p = 0; p < n; ++p) tiles_n += (uint32_t)(ws[p]->n_out_pad / BN);
    bool clusters = sliced;
    for (uint32_t p = 1; p < n; ++p) clusters = clusters && slices[p] == slices[0];
    const GroupCost cost = group_cost(slices, ws, n, tokens, ctx->sm_count);
    if (clusters) {
        const uint32_t k_tiles = (uint32_t)((w0->n_in + BK - 1) / BK);
        clusters = tiles_n * m_blocks <= (uint32_t)split_room(ctx).n[slices[0]] && split_us(k_tiles, slices[0], tokens) + 4.0 <= std::min(cost.one_launch, cost.apart);
    }
    if (sliced && !clusters && cost.one_launch > cost.apart) {
        const Weight *rest[4];
        void *rest_y[4];
        uint32_t n_rest = 0;
        for (uint32_t p = 0; p < n; ++p) {
            if (slices[p] == 1) {
                rest[n_rest] = ws[p], rest_y[n_rest++] = ys[p];
                continue;
            }
            const muser_cuda_status st = launch_nvfp4_gemm(ctx, ws[p], x_packed, x_scales, ys[p], y_dtype, tokens, Epilogue{}, stream);
            if (st != MUSER_CUDA_OK) return st;
        }
        return n_rest ? launch_nvfp4_gemm_group(ctx, rest, n_rest, x_packed, x_scales, rest_y, y_dtype, tokens, stream) : MUSER_CUDA_OK;
    }
    bool pair = !sliced && takes_pairs(ctx, tiles_n, tokens, w0->n_in, PairForm::group);
    for (uint32_t p = 0; p < n; ++p) pair = pair && pair_rows_fit(ys[p], nullptr, ws[p]->n_out, y_dtype);
    const uint32_t a_rows = pair ? BM : box_tokens(tokens);
    CUtensorMap map_a;
    GemmMaps maps;
    if (!make_map(&map_a, x_packed, tokens, w0->n_in / 2, a_rows) || (pair && !make_scale_map(&maps.a_scales, x_scales, m_blocks, w0->n_in / 64)))
        return fail(ctx, MUSER_CUDA_ERROR, "cuTensorMapEncodeTiled failed for the activations");
    GemmArgs g = {};
    g.a_scales = x_scales;
    g.status = ctx->dev_status;
    g.tokens = tokens;
    g.a_bytes = a_rows * (BK / 2);
    g.ksplit = 1;
    g.k_tiles = (uint32_t)((w0->n_in + BK - 1) / BK);
    g.kt64 = (uint32_t)(w0->n_in / 64);
    g.y_dtype = y_dtype;
    g.out_scale = 1.0f;
    g.inv_input_scale = 1.0f / w0->input_scale_inv;
    tiles_n = 0;
    for (uint32_t p = 0; p < 4; ++p) {
        maps.b[p] = *reinterpret_cast<const CUtensorMap *>(pair ? ws[p < n ? p : 0]->tmap_half : ws[p < n ? p : 0]->tmap_cache);
        if (pair) maps.b_scales[p] = *reinterpret_cast<const CUtensorMap *>(ws[p < n ? p : 0]->tmap_scales);
        if (pair && p < n && !make_out_map(&maps.y[p], ys[p], tokens, ws[p]->n_out, y_dtype))
            return fail(ctx, MUSER_CUDA_ERROR, "cuTensorMapEncodeTiled failed for the outputs");
        g.grp_tile0[p] = tiles_n;
        if (p >= n) continue;
        g.grp_b_scales[p] = ws[p]->scales;
        g.grp_y[p] = ys[p];
        g.grp_n_out[p] = (uint32_t)ws[p]->n_out;
        g.grp_scale2[p] = ws[p]->scale2;
        g.grp_slices[p] = slices[p];
        tiles_n += (uint32_t)(ws[p]->n_out_pad / BN);
    }
    g.grp_tile0[4] = tiles_n;
    for (uint32_t p = n; p < 4; ++p) g.grp_tile0[p] = tiles_n; // no tile falls into a projection that is not there
    g.n_tiles = tiles_n;
    g.n_out = g.grp_n_out[0], g.y = g.grp_y[0], g.scale2 = g.grp_scale2[0], g.b_scales = g.grp_b_scales[0];
    g.group_m = raster_group(ctx, w0, m_blocks, pair);
    if (pair) {
        MUSER_CUDA_TRY(ctx, (launch_pairs<false, false, false, true>(ctx, map_a, maps, g, stream)));
        return MUSER_CUDA_OK;
    }
    const uint32_t tiles = tiles_n * m_blocks;
    const uint32_t grid = tiles < (uint32_t)ctx->sm_count ? tiles : (uint32_t)ctx->sm_count;
    if (clusters) {
        const auto kernel = nvfp4_gemm_kernel<false, false, false, true, kCluster>;
        MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kSmemBytes));
        g.ksplit = slices[0];
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        cluster_launch(cfg, attr, tiles * slices[0], slices[0], kSmemBytes, stream);
        MUSER_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, map_a, maps, g));
        return MUSER_CUDA_OK;
    }
    const auto kernel = sliced ? nvfp4_gemm_kernel<false, false, false, true, kSliced> : nvfp4_gemm_kernel<false, false, false, true>;
    MUSER_CUDA_TRY(ctx, ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kSmemBytes));
    MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(grid), dim3(kGemmThreads), kSmemBytes, stream, map_a, maps, g));
    MUSER_CUDA_TRY(ctx, cudaGetLastError());
    return MUSER_CUDA_OK;
}

} // namespace muser
