// NVFP4 activation quantizer: f32/bf16 rows -> packed E2M1 codes + one E4M3FN scale per 16 values.
//
// Reproduces quant::activation_group_codes / quantize_nvfp4_activation bit for bit
// (crates/muser-engine/src/quant/nvfp4.rs:173-238): round to f16, amax/6 * input_scale_inv saturated at 448
// and rounded to E4M3 (nearest, ties to even), then threshold compares of |x| * input_scale_inv against
// scale * {0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5} with the reference's <= / < pattern.  Scales are written in
// the 128-row x 4-group swizzle of scripts/gx10/vllm/muser_vllm/exact_fp4_quant.py:149-162, which is also
// the order the block-scaled MMA wants them in tensor memory.
#include "common.cuh"
#include "nvfp4_codec.cuh"
#include "rmsnorm.cuh"

namespace muser {

// Grids of up to two blocks an SM release their successor in front of their own wait (pdl_turn): norm, q | k | v, quantizer and o of
// a 5120-wide layer 29.5 -> 26.8 us at 16 tokens, 34.1 -> 33.3 at 200; larger ones gain nothing (509 tokens 40.0 / 39.9) or, with
// the whole layer, lose (168.5 -> 173).
static bool few_blocks(const Ctx *ctx, uint32_t blocks) { return blocks <= 2 * (uint32_t)ctx->sm_count; }
// Four neighbouring threads (groups 4q .. 4q+3 of one row) merge their scale bytes into one aligned 32-bit store.
// Every lane of the warp calls this; lanes past the row's last group slot pass live = false.
__device__ __forceinline__ void store_scale_quad(uint32_t scale_code, uint32_t row, uint32_t grp, uint32_t kt, uint8_t *scales,
                                                 bool live = true) {
    uint32_t word = scale_code;
    word |= __shfl_down_sync(0xffffffffu, scale_code, 1) << 8;
    word |= __shfl_down_sync(0xffffffffu, scale_code, 2) << 16;
    word |= __shfl_down_sync(0xffffffffu, scale_code, 3) << 24;
    if (live && (grp & 3) == 0) {
        const size_t off = (size_t)(row / 128) * ((size_t)kt * 512) + (size_t)(grp / 4) * 512 + (row % 32) * 16 + ((row % 128) / 32) * 4;
        *reinterpret_cast<uint32_t *>(scales + off) = word;
    }
}

// One thread per 16-value group; the four threads of a 64-value span merge their scale bytes into one
// aligned 32-bit store.  Rows tokens..tokens_pad-1 only clear their scale slots.
template <bool XF32>
__global__ void nvfp4_quantize_kernel(const void *x, uint32_t tokens, uint32_t tokens_pad, uint32_t n_in, uint32_t kt, float isi, uint8_t *packed,
                                      uint8_t *scales, bool early) {
    pdl_turn(early);
    const uint32_t groups_pad = kt * 4; // group slots per row in the swizzled plane
    const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (idx >= (uint64_t)tokens_pad * groups_pad) return; // groups_pad % 4 == 0: quads never straddle the edge
    const uint32_t row = (uint32_t)(idx / groups_pad), grp = (uint32_t)(idx % groups_pad);
    uint32_t scale_code = 0;
    if (row < tokens && grp * 16 < n_in) {
        const void *xr = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)row * n_in)
                              : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)row * n_in);
        float r[16];
        float(&lo)[8] = *reinterpret_cast<float(*)[8]>(&r[0]);
        float(&hi)[8] = *reinterpret_cast<float(*)[8]>(&r[8]);
        load8<XF32>(xr, 2 * grp, lo);
        load8<XF32>(xr, 2 * grp + 1, hi);
        scale_code = quantize_group(r, isi, packed + (size_t)row * (n_in / 2) + grp * 8);
    }
    store_scale_quad(scale_code, row, grp, kt, scales);
}

// 1 / sqrt(mean(x^2) + eps) per row with the squares added FRONT TO BACK in f32, one rounding per step, exactly as
// rms_norm does on the CPU lane (crates/muser-engine/src/reference.rs:59-72).  The order matters here more than
// anywhere else on the path: the NVFP4 quantizer that consumes the normalized row is a chain of threshold compares,
// so a factor that differs in its last bits flips a 4-bit code now and then, and one flipped code moves that
// token's outputs by a few 1e-3 of their norm.  One thread owns one row's chain; its warp stages 256 inputs of its 32
// rows at a time through shared memory (asynchronous copies, two buffers), so that global loads stay coalesced
// (consecutive threads read consecutive 16 bytes of one row) while the sums stay sequential.
template <bool XF32>
__global__ void __launch_bounds__(32) rms_rows_sequential_kernel(const void *x, uint32_t tokens, uint32_t n_in, float eps, float *inv_rms, bool early) {
    pdl_turn(early);
    constexpr int kRows = 32, kChunk = 256;                       // rows per block (one warp), inputs per row and step
    constexpr int kParts = kChunk * (XF32 ? 4 : 2) / 16;          // 16-byte pieces per row and step
    constexpr int kStride = kParts + 1;                           // row stride in pieces: conflict-free 16-byte reads down a column
    extern __shared__ uint4 rms_tile[];                           // two buffers of kRows x kStride pieces
    const uint32_t row0 = blockIdx.x * kRows, lane = threadIdx.x, my_row = row0 + lane;
    const size_t row_bytes = (size_t)n_in * (XF32 ? 4 : 2);
    const uint8_t *base = reinterpret_cast<const uint8_t *>(x);
    const uint32_t steps = (n_in + kChunk - 1) / kChunk;
    // the next step's pieces travel global -> shared asynchronously while this step's chain runs
    auto stage = [&](uint32_t step, uint4 *buf) {
        const uint32_t k0 = step * kChunk;
        const uint32_t parts_here = min((uint32_t)kParts, (n_in - k0) * (XF32 ? 4u : 2u) / 16u);
        for (uint32_t i = lane; i < kRows * kParts; i += 32) {
            const uint32_t r = i / kParts, part = i % kParts;
            uint4 *dst = buf + r * kStride + part;
            if (row0 + r < tokens && part < parts_here) {
                const void *src = base + (size_t)(row0 + r) * row_bytes + (size_t)k0 * (XF32 ? 4 : 2) + (size_t)part * 16;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
            } else {
                *dst = make_uint4(0, 0, 0, 0); // zeros add nothing to the chain
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float ss = 0.0f;
    stage(0, rms_tile);
    for (uint32_t step = 0; step < steps; ++step) {
        uint4 *cur = rms_tile + (step & 1) * (kRows * kStride);
        if (step + 1 < steps) {
            stage(step + 1, rms_tile + ((step + 1) & 1) * (kRows * kStride));
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
#pragma unroll 4
        for (int part = 0; part < kParts; ++part) {
            const uint4 v = cur[lane * kStride + part];
            if constexpr (XF32) {
                const float f[4] = {__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)};
#pragma unroll
                for (int i = 0; i < 4; ++i) ss = __fadd_rn(ss, __fmul_rn(f[i], f[i]));
            } else {
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xFFFF0000u);
                    ss = __fadd_rn(ss, __fmul_rn(lo, lo));
                    ss = __fadd_rn(ss, __fmul_rn(hi, hi));
                }
            }
        }
        __syncwarp(); // this buffer is refilled by the step after next
    }
    if (my_row < tokens) inv_rms[my_row] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)n_in), eps)));
}

// The same chains for few rows, where one warp that fetches, unpacks, squares and adds takes 11 cycles an input: here the
// first warp's lanes only read squares and add (four cycles an addition is the floor, 11 us for 5120 values), and the
// block's other seven warps fetch, square and lay the squares out for it, 256 inputs of 16 rows ahead (of 32 rows the
// seven could not keep up: 2048 rows 41 us, 37 with 16).  From some thousands of rows the shared-memory traffic costs more
// than the latency saved (us with the quantizer behind it, 5120 values: 2048 rows 51 -> 37, 4096 rows 46 against about 50).
constexpr int kRmsThreads = 256, kRmsRows = 16, kRmsChunk = 256;
constexpr int kRmsPitch = kRmsRows + 1;                                     // float4 per four inputs: rows side by side, padded
constexpr int kRmsBuffer = kRmsChunk / 4 * kRmsPitch;                       // float4 of one buffer
constexpr size_t kRmsSmem = 2 * kRmsBuffer * sizeof(float4);
template <bool XF32>
__global__ void __launch_bounds__(kRmsThreads) rms_rows_staged_kernel(const void *x, uint32_t tokens, uint32_t n_in, float eps, float *inv_rms, bool early) {
    extern __shared__ float4 rms_squares[]; // two buffers
    pdl_turn(early);
    const uint32_t row0 = blockIdx.x * kRmsRows, steps = (n_in + kRmsChunk - 1) / kRmsChunk;
    // warps 1 .. 7: pieces of eight inputs, neighbouring lanes along a row; all of a thread's loads before the first is used
    constexpr uint32_t kPieces = kRmsRows * (kRmsChunk / 8), kLoaders = kRmsThreads - 32, kPer = (kPieces + kLoaders - 1) / kLoaders;
    auto stage = [&](uint32_t step, float4 *buf) {
        float v[kPer][8];
#pragma unroll
        for (uint32_t n = 0; n < kPer; ++n) {
            const uint32_t p = threadIdx.x - 32 + n * kLoaders, r = p / (kRmsChunk / 8), i8 = step * (kRmsChunk / 8) + p % (kRmsChunk / 8);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[n][k] = 0.0f; // zeros add nothing to the chain
            if (p < kPieces && row0 + r < tokens && i8 < n_in / 8)
                load8<XF32>(XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)(row0 + r) * n_in)
                                 : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)(row0 + r) * n_in), i8, v[n]);
        }
#pragma unroll
        for (uint32_t n = 0; n < kPer; ++n) {
            const uint32_t p = threadIdx.x - 32 + n * kLoaders, r = p / (kRmsChunk / 8), j = p % (kRmsChunk / 8);
            if (p >= kPieces) break;
#pragma unroll
            for (int k = 0; k < 8; ++k) v[n][k] = __fmul_rn(v[n][k], v[n][k]);
            buf[(2 * j) * kRmsPitch + r] = make_float4(v[n][0], v[n][1], v[n][2], v[n][3]);
            buf[(2 * j + 1) * kRmsPitch + r] = make_float4(v[n][4], v[n][5], v[n][6], v[n][7]);
        }
    };
    float ss = 0.0f;
    if (threadIdx.x >= 32) stage(0, rms_squares);
    for (uint32_t step = 0; step < steps; ++step) {
        __syncthreads(); // this step's squares are there, and the other buffer has been read
        if (threadIdx.x >= 32) {
            if (step + 1 < steps) stage(step + 1, rms_squares + ((step + 1) & 1) * kRmsBuffer);
        } else {
            const float4 *cur = rms_squares + (step & 1) * kRmsBuffer + min(threadIdx.x, kRmsRows - 1u); // (lanes without a row repeat the last)
#pragma unroll 32
            for (int q = 0; q < kRmsChunk / 4; ++q) {
                const float4 v = cur[q * kRmsPitch];
                ss = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(ss, v.x), v.y), v.z), v.w);
            }
        }
    }
    if (threadIdx.x < kRmsRows && row0 + threadIdx.x < tokens)
        inv_rms[row0 + threadIdx.x] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)n_in), eps)));
}

constexpr uint32_t kRmsStagedRows = 4096; // beyond: the warp per 32 chains above

// ---- the chain without its latency ----------------------------------------------------------------------------------
// A chain of n dependent additions takes 4 cycles each at best.  A block cuts the row into one segment per thread.  While
// the running sum S stays inside one binade, adding a square moves S's bit pattern by a whole number of units that
// depends on the square and, for a tie, on whether the pattern is even; so a whole segment acts on the pattern as
// "add `even` if it is even, `odd` if it is odd", and two chains of the segment's own squares, from the bottom of the binade
// and from one unit above it, give the two numbers.  The binade is guessed from a parallel prefix sum.  Segments of one
// binade that follow one another in a warp are composed by a scan; one warp then walks the warps' runs, checks for each
// that S was in the guessed binade before and is after (S never falls, so it was in between), takes the segments of a run
// that fails one at a time, and adds the squares of a segment that fails one by one: one or two per power of two that the sum
// passes.  (A run that fails at its first segment, where the guess and the sum part, happens to one row in some hundred; added
// value by value to its end it took the kernel from 7 to 18 us at rows of 4096, segment by segment 10.7.)  The sum that results
// is the chain's.
constexpr int kChainThreads = 1024; // most threads of a block, one segment each
struct ChainThread {
    uint2 add, own;  // units of its run up to and with its segment, and of the segment alone, from an even and an odd pattern
    uint32_t binade; // exponent field that the segment's additions hold for, kNoBinade: one by one
    uint32_t unused;
};
struct ChainBlock {
    uint32_t starts[32]; // per warp: the lanes that begin a run
    float warp_sum[32];
    float inv_rms;
};
constexpr int kChainResident = 1152; // threads an SM holds (56 registers each)
// At least 12 KB: beside a block with less, a CTA of the GEMM behind finds room on the same SM and is set up there while the
// row's chain runs (an NVFP4 layer of 16 tokens 88.2 us instead of 87.1).
constexpr size_t chain_smem(uint32_t threads) { return threads < 512 ? 512 * sizeof(ChainThread) : threads * sizeof(ChainThread); }
static_assert(kChainResident / 96 * (chain_smem(96) + sizeof(ChainBlock) + 1024) < 227 * 1024, "shared memory holds fewer blocks than registers");
constexpr uint32_t kNoBinade = 256;
static uint32_t chain_threads(uint32_t n_in, uint32_t eights) { return ((n_in / 8 + eights - 1) / eights + 31) / 32 * 32; }
__device__ __forceinline__ uint2 chain_compose(uint2 first, uint2 then) {
    return make_uint2(first.x + ((first.x & 1) ? then.y : then.x), first.y + ((first.y & 1) ? then.x : then.y)); // (odd + odd: even)
}
// What a segment of `n` squares adds to an even and to an odd pattern, if the sum is about `before` in front of it and `after`
// behind it and stays in the binade that is returned with it.
__device__ __forceinline__ uint2 chain_segment(float before, float after, const float *v, int n, uint32_t &binade) {
    binade = __float_as_uint(before) >> 23; // (sums of squares: no sign; infinities and NaN are 255)
    if (binade != __float_as_uint(after) >> 23 || binade == 255) binade = kNoBinade;
    const uint32_t bottom = binade << 23; // (no binade: sums that nobody looks at)
    float even = __uint_as_float(bottom), odd = __uint_as_float(bottom + 1);
#pragma unroll
    for (int i = 0; i < n; ++i) even = __fadd_rn(even, v[i]), odd = __fadd_rn(odd, v[i]);
    return make_uint2(__float_as_uint(even) - bottom, __float_as_uint(odd) - (bottom + 1));
}
// The lanes that begin a run of segments of one binade; `add` becomes the run's up to and with the lane's segment.
__device__ __forceinline__ uint32_t chain_runs(uint32_t binade, uint2 &add) {
    const uint32_t lane = threadIdx.x & 31, left = __shfl_up_sync(0xffffffffu, binade, 1);
    const uint32_t starts = __ballot_sync(0xffffffffu, lane == 0 || binade != left || binade == kNoBinade);
    const uint32_t start = 31 - __clz(starts & (0xffffffffu >> (31 - lane))); // of this lane's run
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint2 l = make_uint2(__shfl_up_sync(0xffffffffu, add.x, o), __shfl_up_sync(0xffffffffu, add.y, o));
        if (lane >= start + o) add = chain_compose(l, add);
    }
    return starts;
}
// 1 / sqrt(mean(x^2) + eps) of one row of n_in <= 8 K blockDim values, for every thread of the block.
template <bool XF32, int K>
__device__ __forceinline__ float chain_inv_rms(const void *xr, uint32_t n_in, float eps, ChainThread *th, ChainBlock &sh) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5, n8 = n_in / 8;
    float v[K][8];
#pragma unroll
    for (int i = 0; i < K; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[i][k] = 0.0f; // (zeros leave any sum as it is)
        if (tid * K + i < n8) load8<XF32>(xr, tid * K + i, v[i]);
    }
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) v[i][k] = __fmul_rn(v[i][k], v[i][k]), sum += v[i][k];
    float after = sum; // of the segments up to and including this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, after, o);
        if (lane >= (uint32_t)o) after += up;
    }
    float before = __shfl_up_sync(0xffffffffu, after, 1);
    if (lane == 0) before = 0.0f;
    if (lane == 31) sh.warp_sum[warp] = after;
    __syncthreads();
    float carry = 0.0f;
    for (uint32_t w = 0; w < warp; ++w) carry += sh.warp_sum[w];
    before += carry, after += carry;
    uint32_t binade;
    uint2 add = chain_segment(before, after, &v[0][0], 8 * K, binade);
    th[tid].own = add;
    const uint32_t starts = chain_runs(binade, add);
    th[tid].add = add, th[tid].binade = binade;
    if (lane == 0) sh.starts[warp] = starts;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = 0; // the running sum's bit pattern, the same in every lane
        const auto step = [&](uint32_t e, uint32_t even, uint32_t odd) {
            const uint32_t next = s + ((s & 1) ? odd : even);
            const bool holds = (s >> 23) == e && (next >> 23) == e;
            if (holds) s = next;
            return holds;
        };
        // what there is to know of a warp that is one run, a warp per lane
        const uint32_t w_starts = lane < warps ? sh.starts[lane] : 0u, w_last = min(lane, warps - 1) * 32 + 31;
        const uint32_t w_binade = th[w_last].binade;
        const uint2 w_add = th[w_last].add;
        for (uint32_t w = 0; w < warps; ++w) {
            uint32_t runs = __shfl_sync(0xffffffffu, w_starts, w);
            const uint32_t e = __shfl_sync(0xffffffffu, w_binade, w), x = __shfl_sync(0xffffffffu, w_add.x, w), y = __shfl_sync(0xffffffffu, w_add.y, w);
            if (runs == 1 && step(e, x, y)) continue;
            const uint2 my_add = th[w * 32 + lane].add, my_own = th[w * 32 + lane].own;
            const uint32_t my_binade = th[w * 32 + lane].binade;
            for (uint32_t pos = 0; pos < 32;) {
                const uint32_t rest = runs & ~(0xffffffffu >> (31 - pos)); // starts behind `pos`
                const uint32_t end = rest ? __ffs(rest) - 1 : 32;
                const bool start = (runs >> pos) & 1; // (else inside a run whose first segment failed)
                const uint32_t last = start ? end - 1 : pos, units_x = start ? my_add.x : my_own.x, units_y = start ? my_add.y : my_own.y;
                if (step(__shfl_sync(0xffffffffu, my_binade, last), __shfl_sync(0xffffffffu, units_x, last), __shfl_sync(0xffffffffu, units_y, last))) {
                    pos = last + 1;
                    continue;
                }
                float t = __uint_as_float(s);
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    const uint32_t i8 = (w * 32 + pos) * K + i;
                    float q[8];
                    if (i8 >= n8) break;
                    load8<XF32>(xr, i8, q);
#pragma unroll
                    for (int k = 0; k < 8; ++k) t = __fadd_rn(t, __fmul_rn(q[k], q[k]));
                }
                s = __float_as_uint(t);
                ++pos;
            }
        }
        if (lane == 0) sh.inv_rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(__uint_as_float(s), (float)n_in), eps)));
    }
    __syncthreads();
    return sh.inv_rms;
}

// The same factors for many rows: a warp takes a row, 1024 values at a time (a segment of 32 per lane), and knows the running
// sum at the start of each step, so nothing waits for another warp.  Each square is added twice and the 31 lanes' prefixes
// are scanned twice per step: more work than a chain of plain additions, but 32 lanes share it and no value passes through
// shared memory.  Segments of 8 or 16 values cost more scans for the same row (2048 rows of 2048 values, norm and quantizer:
// 15.5 and 12.2 us against 11.5) and gain nothing on short rows (512 values: 7.8, 7.2, 7.4).
constexpr int kChainRowWarps = 4;
template <bool XF32>
__global__ void __launch_bounds__(32 * kChainRowWarps) rms_rows_chain_kernel(const void *x, uint32_t tokens, uint32_t n_in, float eps, float *inv_rms, bool early) {
    constexpr int K = 4; // eights per lane and step
    pdl_turn(early);
    const uint32_t lane = threadIdx.x & 31, row = blockIdx.x * kChainRowWarps + (threadIdx.x >> 5), n8 = n_in / 8;
    if (row >= tokens) return; // (whole warps)
    const void *xr = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)row * n_in)
                          : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)row * n_in);
    constexpr int kWords = XF32 ? 2 : 1; // 16-byte pieces of eight values
    uint4 next[K][kWords];
    auto fetch = [&](uint32_t first8) {
#pragma unroll
        for (int i = 0; i < K; ++i) {
            const uint32_t at = first8 + lane * K + i;
#pragma unroll
            for (int k = 0; k < kWords; ++k)
                next[i][k] = at < n8 ? ld_after_wait(reinterpret_cast<const uint4 *>(xr) + (size_t)at * kWords + k) : make_uint4(0, 0, 0, 0);
        }
    };
    uint32_t s = 0; // the running sum's bit pattern, the same in every lane
    fetch(0);
    for (uint32_t first8 = 0; first8 < n8; first8 += 32 * K) {
        float v[K][8], sum = 0.0f;
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t w = XF32 ? (&next[i][(k / 4) % kWords].x)[k % 4] : (&next[i][0].x)[k / 2];
                const float f = __uint_as_float(XF32 ? w : (k & 1) ? w & 0xFFFF0000u : w << 16);
                v[i][k] = __fmul_rn(f, f), sum += v[i][k];
            }
        if (first8 + 32 * K < n8) fetch(first8 + 32 * K);
        float after = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, after, o);
            if (lane >= (uint32_t)o) after += up;
        }
        float before = __shfl_up_sync(0xffffffffu, after, 1);
        before = __uint_as_float(s) + (lane ? before : 0.0f), after += __uint_as_float(s);
        uint32_t binade;
        uint2 add = chain_segment(before, after, &v[0][0], 8 * K, binade);
        const uint32_t starts = chain_runs(binade, add);
        for (uint32_t pos = 0; pos < 32;) {
            const uint32_t rest = starts & ~(0xffffffffu >> (31 - pos)), end = rest ? __ffs(rest) - 1 : 32;
            const uint32_t e = __shfl_sync(0xffffffffu, binade, end - 1);
            const uint32_t even = __shfl_sync(0xffffffffu, add.x, end - 1), odd = __shfl_sync(0xffffffffu, add.y, end - 1);
            const uint32_t sum_bits = s + ((s & 1) ? odd : even);
            if (((starts >> pos) & 1) && (s >> 23) == e && (sum_bits >> 23) == e) {
                s = sum_bits, pos = end;
                continue;
            }
            float t = __uint_as_float(s); // (every lane adds its own squares, the segment's lane is heard)
#pragma unroll
            for (int i = 0; i < K; ++i)
#pragma unroll
                for (int k = 0; k < 8; ++k) t = __fadd_rn(t, v[i][k]);
            s = __shfl_sync(0xffffffffu, __float_as_uint(t), pos);
            ++pos;
        }
    }
    if (lane == 0) inv_rms[row] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(__uint_as_float(s), (float)n_in), eps)));
}

// Which of the three leaves the factors.  The plain chains (few values per row, or enough rows that a lane each fills the chip)
// do half the additions.  us with the quantizer of a row a block, plain / warp per row, bf16: 512 values 4.5 / 4.8 at 148 rows, 6.4 / 7.4 at
// 2048; 1024 values 6.6 / 5.4 at 449, 9.0 / 8.7 at 2048, 11.8 / 12.5 at 4096; 2048 values 14.3 / 11.5 at 2048, 18.3 / 16.9 at
// 4096, 28.4 / 29 at 8192; 3136 values 27.5 / 23.6 at 4096, 42.6 / 40.2 at 8192, 139 / 153 at 32768; 4608
// values 59 / 58 at 10000, 82 / 89 at 16384, 168 / 169 at 32768 (f32, where the line could lie lower: 90 / 90, 161 / 141, 279 / 269); 5120 values 45 / 32 at
// 4096, 66 / 57 at 8192, 224 / 212 at 32768; 12288 values 77 / 46 at 2048.  f32: 5120 values 72 / 52 at 4096, 352 / 353 at
// 32768; 12288 values 136 / 72 at 2048; 27648 values 304 / 160 at 2048.
static cudaError_t launch_rms_rows(Ctx *ctx, const void *x, uint32_t x_dtype, uint32_t tokens, uint32_t n_in, float eps, float *inv_rms,
                                   cudaStream_t stream) {
    const bool f32 = x_dtype == MUSER_DTYPE_F32;
    if (n_in >= 5120 || (n_in >= 1024 && tokens <= 2 * n_in))
        return launch_pdl(f32 ? rms_rows_chain_kernel<true> : rms_rows_chain_kernel<false>, dim3((tokens + kChainRowWarps - 1) / kChainRowWarps),
                          dim3(32 * kChainRowWarps), 0, stream, x, tokens, n_in, eps, inv_rms,
                          few_blocks(ctx, (tokens + kChainRowWarps - 1) / kChainRowWarps));
    if (tokens <= kRmsStagedRows) {
        const auto kernel = f32 ? rms_rows_staged_kernel<true> : rms_rows_staged_kernel<false>;
        const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), ctx->device, kRmsSmem);
        if (e != cudaSuccess) return e;
        return launch_pdl(kernel, dim3((tokens + kRmsRows - 1) / kRmsRows), dim3(kRmsThreads), kRmsSmem, stream, x, tokens, n_in, eps, inv_rms,
                          few_blocks(ctx, (tokens + kRmsRows - 1) / kRmsRows));
    }
    const unsigned blocks = (tokens + 31) / 32;
    const size_t smem = (size_t)2 * 32 * ((f32 ? 64 : 32) + 1) * sizeof(uint4);
    const void *fn = f32 ? reinterpret_cast<const void *>(rms_rows_sequential_kernel<true>) : reinterpret_cast<const void *>(rms_rows_sequential_kernel<false>);
    const cudaError_t e = ensure_dynamic_smem(fn, ctx->device, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(f32 ? rms_rows_sequential_kernel<true> : rms_rows_sequential_kernel<false>, dim3(blocks), dim3(32), smem, stream, x, tokens, n_in, eps, inv_rms,
                      few_blocks(ctx, blocks));
}

// (x * inv_rms) * w of one row, quantized group by group by the whole block; rows past `tokens` only clear their scales.
template <bool XF32>
__device__ __forceinline__ void norm_quantize_row(const void *xr, uint32_t row, uint32_t tokens, uint32_t n_in, uint32_t kt, float isi,
                                                  const float *norm_w, float inv, uint8_t *packed, uint8_t *scales) {
    const uint32_t groups_pad = kt * 4;
    for (uint32_t g0 = 0; g0 < groups_pad; g0 += blockDim.x) { // blockDim % 4 == 0: quads stay together
        const uint32_t grp = g0 + threadIdx.x;
        uint32_t scale_code = 0;
        if (row < tokens && grp * 16 < n_in) {
            float r[16], a[8], b[8];
            load8<XF32>(xr, 2 * grp, a);
            load8<XF32>(xr, 2 * grp + 1, b);
            const float4 *wp = reinterpret_cast<const float4 *>(norm_w + grp * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 w = ld_after_wait(wp + i);
                const float *src = i < 2 ? a + 4 * i : b + 4 * (i - 2);
                r[4 * i] = __fmul_rn(__fmul_rn(src[0], inv), w.x);
                r[4 * i + 1] = __fmul_rn(__fmul_rn(src[1], inv), w.y);
                r[4 * i + 2] = __fmul_rn(__fmul_rn(src[2], inv), w.z);
                r[4 * i + 3] = __fmul_rn(__fmul_rn(src[3], inv), w.w);
            }
            scale_code = quantize_group(r, isi, packed + (size_t)row * (n_in / 2) + grp * 8);
        }
        store_scale_quad(scale_code, row, grp, kt, scales, grp < groups_pad);
    }
}

// The same quantizer behind a fused input RMSNorm (reference.rs:59-80): one block per token row takes the row's factor
// (chain_inv_rms) and quantizes (x * inv_rms) * w group by group.
template <bool XF32, int K>
__global__ void __maxnreg__(56) nvfp4_norm_quantize_kernel(const void *x, uint32_t tokens, uint32_t n_in, uint32_t kt, float isi,
                                                                            const float *norm_w, float eps, uint8_t *packed, uint8_t *scales, bool early) {
    extern __shared__ ChainThread chain_threads_shared[]; // (by the block's size: 1024 of them left room for ten blocks of 96 where twelve are counted on)
    __shared__ ChainBlock sh;
    const uint32_t row = blockIdx.x;
    // the norm weights are read last, from L2 if they are asked for now (between two layers' weights they go to memory)
    if (row < min(tokens, 16u))
        for (uint32_t i = 32 * threadIdx.x; i < n_in; i += 32 * blockDim.x) asm volatile("prefetch.global.L2 [%0];" ::"l"(norm_w + i));
    pdl_turn(early);
    const void *xr = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)row * n_in)
                          : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)row * n_in);
    const float inv = row < tokens ? chain_inv_rms<XF32, K>(xr, n_in, eps, chain_threads_shared, sh) : 0.0f; // (uniform over the block)
    norm_quantize_row<XF32>(xr, row, tokens, n_in, kt, isi, norm_w, inv, packed, scales);
}

// The quantizer behind a kernel that leaves the rows' factors in memory (chain_eights).  Blocks of a row's own size (64 threads
// for 1024 values) were slower from 700 rows on: 9.9 against 8.7 us at 2048 rows.
template <bool XF32>
__global__ void __launch_bounds__(256) nvfp4_scaled_quantize_kernel(const void *x, uint32_t tokens, uint32_t n_in, uint32_t kt, float isi,
                                                                    const float *norm_w, const float *inv_rms, uint8_t *packed,
                                                                    uint8_t *scales, bool early) {
    const uint32_t row = blockIdx.x;
    pdl_turn(early);
    const void *xr = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)row * n_in)
                          : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)row * n_in);
    norm_quantize_row<XF32>(xr, row, tokens, n_in, kt, isi, norm_w, row < tokens ? ld_after_wait(inv_rms + row) : 0.0f, packed, scales);
}

// Both quantizers for many rows: a thread takes one group of the four rows whose scales are neighbours in the swizzled plane
// (r, r + 32, r + 64, r + 96 of a 128-row block), all of them on their way before the first is used, and four lanes' scale bytes
// leave as 16 bytes instead of four times 4 (a sector each); the norm's weights are read once for four rows.  32768 rows of
// 5120 values: 117 -> 79 us from bf16 (5.5 TB/s), 135 -> 109 from f32 (7 TB/s); behind the norm 212 -> 180 and 353 -> 297 with
// the norm's own kernel.  (Blocks of 256 threads 85 and 127; two of the four rows ahead 87 and 120.)
template <bool XF32, bool NORM>
__global__ void __launch_bounds__(128) nvfp4_quantize_quads_kernel(const void *x, uint32_t tokens, uint32_t n_in, uint32_t kt, float isi,
                                                                   const float *norm_w, const float *inv_rms, uint8_t *packed, uint8_t *scales) {
    pdl_turn(false); // (thousands of blocks)
    const uint32_t groups_pad = kt * 4;
    const uint64_t idx = blockIdx.x * (uint64_t)128 + threadIdx.x; // (128 x kt of them per 128 rows: whole blocks)
    const uint32_t quad = (uint32_t)(idx / groups_pad), grp = (uint32_t)(idx % groups_pad);
    const uint32_t row0 = quad / 32 * 128 + quad % 32;
    constexpr int kWords = XF32 ? 4 : 2; // 16-byte pieces of a group
    const bool live = grp * 16 < n_in;
    uint4 raw[4][kWords];
    float inv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t row = row0 + 32 * i;
        const bool there = live && row < tokens;
        const uint4 *p = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(x) + ((size_t)row * n_in + grp * 16) * (XF32 ? 4 : 2));
#pragma unroll
        for (int k = 0; k < kWords; ++k) raw[i][k] = there ? ld_after_wait(p + k) : make_uint4(0, 0, 0, 0);
        if (NORM) inv[i] = there ? ld_after_wait(inv_rms + row) : 0.0f;
    }
    float4 w[4];
    if (NORM && live) {
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = ld_after_wait(reinterpret_cast<const float4 *>(norm_w + grp * 16) + k);
    }
    uint32_t word[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t row = row0 + 32 * i;
        word[i] = 0;
        if (live && row < tokens) {
            float r[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const uint32_t bits = XF32 ? (&raw[i][(k / 4) % kWords].x)[k % 4] : (&raw[i][(k / 8) % kWords].x)[(k % 8) / 2];
                const float f = __uint_as_float(XF32 ? bits : (k & 1) ? bits & 0xFFFF0000u : bits << 16);
                r[k] = NORM ? __fmul_rn(__fmul_rn(f, inv[i]), (&w[k / 4].x)[k % 4]) : f;
            }
            word[i] = quantize_group(r, isi, packed + (size_t)row * (n_in / 2) + grp * 8);
        }
        word[i] |= __shfl_down_sync(0xffffffffu, word[i], 1) << 8;
        word[i] |= __shfl_down_sync(0xffffffffu, word[i], 2) << 16;
    }
    if ((grp & 3) == 0) // (the four rows' words are neighbours)
        *reinterpret_cast<uint4 *>(scales + (size_t)(row0 / 128) * ((size_t)kt * 512) + (size_t)(grp / 4) * 512 + (row0 % 32) * 16) =
            make_uint4(word[0], word[1], word[2], word[3]);
}
// Where a quarter of the threads still fills the chip: us, a row / four rows a thread, bf16 rows of 2048 values 3.9 / 3.9 at 2048
// rows, 6.4 / 5.4 at 4096; 5120 values 4.5 / 5.2 at 1024, 7.7 / 6.6 at 2048; f32 rows, whose loads are twice as many, 2048 values
// 7.0 / 7.3 at 4096, 12.6 / 11.8 at 8192; 5120 values 8.3 / 8.6 at 2048, 17.0 / 15.0 at 4096.  Behind a norm, which leaves the
// SMs unevenly free for a grid of one round: bf16 2048 values 11.6 / 13.6 at 2048 rows, 17.1 / 15.7 at 4096; f32 1024 values
// 14.1 / 16.9 at 4096, 23.0 / 20.1 at 8192; 5120 values 30.6 / 22.4 at 1500.
static bool takes_quads(uint32_t tokens_pad, uint32_t kt, bool f32, bool norm) {
    return (uint64_t)tokens_pad * kt >= (f32 && !norm ? 16u << 14 : 8u << 14); // (in 64 values)
}

// Eights a thread holds in the kernel above, 0: a kernel of its own leaves the rows' factors and the quantizer reads the rows
// again.  One block per row pays where one round of blocks takes all rows: a second round waits for the first one's chains.
// us, factors on their own / two eights / four, bf16 rows of 5120 values: 7.8 / 7.4 / 9.3 at 1 row, 9.4 / 8.2 / 10 at 148,
// 17.5 / 18 / 13.7 at 1024, 18.3 / - / 21.1 at 1500 (a second round); 12288 values: 15.7 / 9.7 / - at 148, 17.5 / 26 / - at
// 300 (two eights: the second round of three); 27648 values: 23.8 / - / 13.4 at 1 row, 28.1 / - / 13.3 at 148, 31.8 / - / 38
// at 300.  Shorter rows are the warp's: 2048 values 4.7 / 6.0 / - at 1 row, 6.4 / 6.6 / - at 148.
static uint32_t chain_eights(const Ctx *ctx, uint32_t tokens, uint32_t n_in) {
    if (n_in < 2560) return 0;
    for (uint32_t eights = 2; eights <= 4; eights *= 2) {
        const uint32_t threads = chain_threads(n_in, eights);
        if (threads <= kChainThreads && tokens <= (uint32_t)ctx->sm_count * (kChainResident / threads)) return eights;
    }
    return 0;
}

// Plain rows: out[t][k] = (x[t][k] * inv_rms_t) * w[k] in f32, for the kernels that read their activations as they go.
template <bool XF32>
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const void *__restrict__ x, uint32_t n_in, const float *__restrict__ norm_w,
                                                           const float *__restrict__ inv_rms, float *__restrict__ out) {
    const uint32_t row = blockIdx.x;
    const void *xr = XF32 ? (const void *)(reinterpret_cast<const float *>(x) + (size_t)row * n_in)
                          : (const void *)(reinterpret_cast<const __nv_bfloat16 *>(x) + (size_t)row * n_in);
    const float inv = inv_rms[row];
    for (uint32_t i = threadIdx.x; i < n_in / 8; i += blockDim.x) {
        float v[8];
        load8<XF32>(xr, i, v);
        const float4 w0 = __ldg(reinterpret_cast<const float4 *>(norm_w) + 2 * i), w1 = __ldg(reinterpret_cast<const float4 *>(norm_w) + 2 * i + 1);
        float4 *o = reinterpret_cast<float4 *>(out + (size_t)row * n_in) + 2 * i;
        o[0] = make_float4(__fmul_rn(__fmul_rn(v[0], inv), w0.x), __fmul_rn(__fmul_rn(v[1], inv), w0.y),
                           __fmul_rn(__fmul_rn(v[2], inv), w0.z), __fmul_rn(__fmul_rn(v[3], inv), w0.w));
        o[1] = make_float4(__fmul_rn(__fmul_rn(v[4], inv), w1.x), __fmul_rn(__fmul_rn(v[5], inv), w1.y),
                           __fmul_rn(__fmul_rn(v[6], inv), w1.z), __fmul_rn(__fmul_rn(v[7], inv), w1.w));
    }
}

muser_cuda_status launch_rmsnorm_rows(Ctx *ctx, const void *x, uint32_t x_dtype, uint32_t tokens, uint64_t n_in,
                                      const float *norm_weight, float norm_eps, float *out, cudaStream_t stream) {
    // the factors sit behind the rows in the same scratch (the caller sized it for tokens x n_in floats and more)
    float *inv = ctx->inv_rms;
    if (tokens > ctx->inv_rms_rows) return fail(ctx, MUSER_CUDA_WORKSPACE_TOO_SMALL, "fused input norm: more rows than the context's per-row scratch holds");
    MUSER_CUDA_TRY(ctx, launch_rms_rows(ctx, x, x_dtype, tokens, (uint32_t)n_in, norm_eps, inv, stream));
    if (x_dtype == MUSER_DTYPE_F32)
        rmsnorm_rows_kernel<true><<<tokens, 256, 0, stream>>>(x, (uint32_t)n_in, norm_weight, inv, out);
    else
        rmsnorm_rows_kernel<false><<<tokens, 256, 0, stream>>>(x, (uint32_t)n_in, norm_weight, inv, out);
    MUSER_CUDA_TRY(ctx, cudaGetLastError());
    return MUSER_CUDA_OK;
}

muser_cuda_status launch_nvfp4_quantize(Ctx *ctx, const void *x, uint32_t x_dtype, uint32_t tokens, uint64_t n_in,
                                        float isi, uint8_t *packed, uint8_t *scales, cudaStream_t stream,
                                        const float *norm_weight, float norm_eps) {
    const uint32_t kt = (uint32_t)((n_in + 63) / 64);
    const uint32_t tokens_pad = (tokens + 127) / 128 * 128;
    if (norm_weight) {
        float *inv = ctx->inv_rms;
        if (!inv || tokens > ctx->inv_rms_rows) return fail(ctx, MUSER_CUDA_WORKSPACE_TOO_SMALL, "fused input norm: more rows than the context's per-row scratch holds");
        const uint32_t eights = chain_eights(ctx, tokens, (uint32_t)n_in);
        const bool f32 = x_dtype == MUSER_DTYPE_F32;
        if (!eights) {
            MUSER_CUDA_TRY(ctx, launch_rms_rows(ctx, x, x_dtype, tokens, (uint32_t)n_in, norm_eps, inv, stream));
            if (takes_quads(tokens_pad, kt, f32, true)) {
                const auto kernel = f32 ? nvfp4_quantize_quads_kernel<true, true> : nvfp4_quantize_quads_kernel<false, true>;
                MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(tokens_pad / 128 * kt), dim3(128), 0, stream, x, tokens, (uint32_t)n_in, kt, isi,
                                               norm_weight, (const float *)inv, packed, scales));
                return MUSER_CUDA_OK;
            }
            const auto kernel = f32 ? nvfp4_scaled_quantize_kernel<true> : nvfp4_scaled_quantize_kernel<false>;
            MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(tokens_pad), dim3(256), 0, stream, x, tokens, (uint32_t)n_in, kt, isi, norm_weight, (const float *)inv,
                                           packed, scales, few_blocks(ctx, tokens_pad)));
            return MUSER_CUDA_OK;
        }
        const auto kernel = eights == 2 ? (f32 ? nvfp4_norm_quantize_kernel<true, 2> : nvfp4_norm_quantize_kernel<false, 2>)
                                        : (f32 ? nvfp4_norm_quantize_kernel<true, 4> : nvfp4_norm_quantize_kernel<false, 4>);
        const uint32_t threads = chain_threads((uint32_t)n_in, eights);
        MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(tokens_pad), dim3(threads), chain_smem(threads), stream, x, tokens, (uint32_t)n_in, kt, isi, norm_weight, norm_eps, packed,
                                       scales, few_blocks(ctx, tokens_pad)));
        return MUSER_CUDA_OK;
    }
    if (takes_quads(tokens_pad, kt, x_dtype == MUSER_DTYPE_F32, false)) {
        const auto kernel = x_dtype == MUSER_DTYPE_F32 ? nvfp4_quantize_quads_kernel<true, false> : nvfp4_quantize_quads_kernel<false, false>;
        MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(tokens_pad / 128 * kt), dim3(128), 0, stream, x, tokens, (uint32_t)n_in, kt, isi,
                                       (const float *)nullptr, (const float *)nullptr, packed, scales));
        return MUSER_CUDA_OK;
    }
    const uint64_t total = (uint64_t)tokens_pad * kt * 4;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    const auto kernel = x_dtype == MUSER_DTYPE_F32 ? nvfp4_quantize_kernel<true> : nvfp4_quantize_kernel<false>;
    MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(blocks), dim3(256), 0, stream, x, tokens, tokens_pad, (uint32_t)n_in, kt, isi, packed, scales,
                                   few_blocks(ctx, blocks)));
    return MUSER_CUDA_OK;
}

} // namespace muser
