// The step either side of the projections, so that a layer's non-attention work can stay on the device between two
// projection calls: the sandwich-norm tail, the attention output gate, and the per-head QK norm.
//
// Reference semantics (CPU lane, f32): crates/muser-engine/src/reference.rs:59-80 (rms_norm, rms_norm_mul),
// :384-393 (per-head norm of q and k), :447-455 (sigmoid gate in front of o_proj), :466-480 and :530-542 (post-norm
// with its own epsilon, then the residual), :484-490 (the next pre-norm).  On the reference's GPU path the tail is one
// kernel, muser_fused_norm_residual_rms_norm_32sg (src/shaders/ferrite/rmsnorm_batch_tail.metal:147-200):
//     hidden += rms_norm(src, eps1) * weight1;  output = rms_norm(hidden, eps2) * weight2
// Sums of squares are block-wide trees here (the CPU lane adds front to back, the shader in simdgroups): results
// agree to rounding, not bit for bit, and are compared by relative error.
#include "common.cuh"

namespace muser {

// These kernels are a few microseconds of latency between two projections.  Up to one block an SM (decode: a row per token)
// each lets its successor launch in front of its own wait (`early`): the launches of a chain of them, and the set-up and first
// weight copies of the projection that follows, lie under the projection before (a layer at one token 88.1 -> 87.1 us, at eight
// 126.2 -> 124.6, against a release behind the wait).  Larger grids do not: the successor's blocks only took the slots of
// their own later ones (head norm, gate and tail of 512 rows of 2048, us: 12.6 with the release, 10.6 without; of 16 rows of
// 5120: 6.0 and 6.9).  They work in place, and a caller may make the norm weights on the stream: both are read behind the wait
// (ld_after_wait).

// Sum over the block of one value per thread; `red` holds 33 floats; every thread gets the total.
__device__ __forceinline__ float block_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (blockDim.x + 31) >> 5;
    __syncthreads(); // `red` may still be read from an earlier call
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < warps ? red[lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

// One block per token row.  n % 4 == 0; rows 16-byte aligned.
// HELD: the row's first kHeld pieces per thread (8192 values a block of 512) stay in registers from one fetch: reading them
// again for each of the three passes is two more trips to L2 in a kernel that, with one block an SM, is nothing but such
// trips (16 rows of 5120 values: 2.8 us against 3.8).  The registers leave an SM room for one block, so more rows read again
// and have their trips covered by other blocks (512 rows of 2048: 7.2 us held, 5.7 read again).
template <bool HELD>
__global__ void __launch_bounds__(512) norm_residual_norm_kernel(float *hidden, const float *src, float *output,
                                                                 const float *w1, const float *w2, uint32_t n, float eps1,
                                                                 float eps2) {
    __shared__ float red[33];
    if constexpr (HELD) pdl_release();
    pdl_wait();
    const uint32_t n4 = n / 4;
    float4 *h4 = reinterpret_cast<float4 *>(hidden + (size_t)blockIdx.x * n);
    const float4 *s4 = reinterpret_cast<const float4 *>(src + (size_t)blockIdx.x * n);
    const float4 *w14 = reinterpret_cast<const float4 *>(w1), *w24 = reinterpret_cast<const float4 *>(w2);
    constexpr uint32_t kHeld = HELD ? 4 : 0;
    float4 s[kHeld + 1], h[kHeld + 1], u1[kHeld + 1], u2[kHeld + 1]; // (the weights' pieces with them)
    float ss = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kHeld; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        s[k] = h[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n4) s[k] = ld_after_wait(s4 + i), h[k] = ld_after_wait(h4 + i);
    }
#pragma unroll
    for (uint32_t k = 0; k < kHeld; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        if (i < n4) u1[k] = ld_after_wait(w14 + i);
        if (i < n4 && output) u2[k] = ld_after_wait(w24 + i);
    }
#pragma unroll
    for (uint32_t k = 0; k < kHeld; ++k) ss += s[k].x * s[k].x + s[k].y * s[k].y + s[k].z * s[k].z + s[k].w * s[k].w;
    for (uint32_t i = threadIdx.x + kHeld * blockDim.x; i < n4; i += blockDim.x) {
        const float4 v = ld_after_wait(s4 + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    const float inv_src = __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(block_sum(ss, red), (float)n) + eps1));
    float sh = 0.0f;
    auto tail = [&](uint32_t i, const float4 &sv, float4 &hv, const float4 &w) {
        hv.x += sv.x * inv_src * w.x, hv.y += sv.y * inv_src * w.y, hv.z += sv.z * inv_src * w.z, hv.w += sv.w * inv_src * w.w;
        h4[i] = hv;
        sh += hv.x * hv.x + hv.y * hv.y + hv.z * hv.z + hv.w * hv.w;
    };
#pragma unroll
    for (uint32_t k = 0; k < kHeld; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        if (i < n4) tail(i, s[k], h[k], u1[k]);
    }
    for (uint32_t i = threadIdx.x + kHeld * blockDim.x; i < n4; i += blockDim.x) {
        float4 hv = ld_after_wait(h4 + i);
        tail(i, ld_after_wait(s4 + i), hv, ld_after_wait(w14 + i));
    }
    if (!output) return;
    const float inv_h = __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(block_sum(sh, red), (float)n) + eps2));
    float4 *o4 = reinterpret_cast<float4 *>(output + (size_t)blockIdx.x * n);
    auto out = [&](uint32_t i, const float4 &hv, const float4 &w) {
        o4[i] = make_float4(hv.x * inv_h * w.x, hv.y * inv_h * w.y, hv.z * inv_h * w.z, hv.w * inv_h * w.w);
    };
#pragma unroll
    for (uint32_t k = 0; k < kHeld; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        if (i < n4) out(i, h[k], u2[k]);
    }
    for (uint32_t i = threadIdx.x + kHeld * blockDim.x; i < n4; i += blockDim.x) out(i, ld_after_wait(h4 + i), ld_after_wait(w24 + i)); // (this thread's own)
}

// x[i] *= 1 / (1 + exp(-gate[i])), four at a time.
__global__ void __launch_bounds__(256) sigmoid_gate_kernel(float *x, const float *gate, size_t n4, bool early) {
    if (early) pdl_release();
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (size_t)gridDim.x * 256) {
        float4 v = ld_after_wait(reinterpret_cast<const float4 *>(x) + i);
        const float4 g = ld_after_wait(reinterpret_cast<const float4 *>(gate) + i);
        v.x *= __fdiv_rn(1.0f, 1.0f + expf(-g.x)), v.y *= __fdiv_rn(1.0f, 1.0f + expf(-g.y));
        v.z *= __fdiv_rn(1.0f, 1.0f + expf(-g.z)), v.w *= __fdiv_rn(1.0f, 1.0f + expf(-g.w));
        reinterpret_cast<float4 *>(x)[i] = v;
    }
}

// One warp per (token, head): x <- x * 1/sqrt(mean(x^2) + eps) * w, head_dim % 4 == 0, head_dim <= 1024.
__global__ void __launch_bounds__(256) head_rms_norm_kernel(float *x, const float *w, float eps, uint32_t heads_total,
                                                            uint32_t head_dim, bool early) {
    if (early) pdl_release();
    pdl_wait();
    const uint32_t head = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (head >= heads_total) return;
    float4 *row = reinterpret_cast<float4 *>(x + (size_t)head * head_dim);
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    const uint32_t n4 = head_dim / 4;
    // A lane's first piece of the row and of the weights, all of them up to heads of 128, are fetched together and held.  (us, weights
    // fetched ahead and the row read twice / held: 40 heads 1.63 / 1.45 at one token, 5.46 / 3.97 at 512, 16.9 / 12.1 at 2048.)
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v0 = lane < n4 ? ld_after_wait(row + lane) : zero, w0 = lane < n4 ? ld_after_wait(w4 + lane) : zero;
    float ss = v0.x * v0.x + v0.y * v0.y + v0.z * v0.z + v0.w * v0.w;
    for (uint32_t i = lane + 32; i < n4; i += 32) {
        const float4 v = ld_after_wait(row + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(ss, (float)head_dim) + eps));
    auto scaled = [&](const float4 &v, const float4 &ww) { return make_float4(v.x * inv * ww.x, v.y * inv * ww.y, v.z * inv * ww.z, v.w * inv * ww.w); };
    if (lane < n4) row[lane] = scaled(v0, w0);
    for (uint32_t i = lane + 32; i < n4; i += 32) row[i] = scaled(ld_after_wait(row + i), ld_after_wait(w4 + i));
}

muser_cuda_status launch_norm_residual_norm(Ctx *ctx, float *hidden, const float *src, float *output, const float *w1, const float *w2,
                                            uint32_t tokens, uint32_t n, float eps1, float eps2, cudaStream_t stream) {
    const unsigned threads = n / 4 >= 512 ? 512 : n / 4 >= 256 ? 256 : 128;
    const auto kernel = tokens <= (uint32_t)ctx->sm_count ? norm_residual_norm_kernel<true> : norm_residual_norm_kernel<false>;
    MUSER_CUDA_TRY(ctx, launch_pdl(kernel, dim3(tokens), dim3(threads), 0, stream, hidden, src, output, w1, w2, n, eps1, eps2));
    return MUSER_CUDA_OK;
}

muser_cuda_status launch_sigmoid_gate(Ctx *ctx, float *x, const float *gate, size_t count, cudaStream_t stream) {
    const size_t n4 = count / 4;
    const unsigned blocks = (unsigned)std::min<size_t>((n4 + 255) / 256, (size_t)ctx->sm_count * 8);
    MUSER_CUDA_TRY(ctx, launch_pdl(sigmoid_gate_kernel, dim3(blocks), dim3(256), 0, stream, x, gate, n4, blocks <= (unsigned)ctx->sm_count));
    return MUSER_CUDA_OK;
}

muser_cuda_status launch_head_rms_norm(Ctx *ctx, float *x, const float *w, float eps, uint32_t tokens, uint32_t heads, uint32_t head_dim,
                                       cudaStream_t stream) {
    const uint32_t total = tokens * heads;
    const uint32_t blocks = (total + 7) / 8;
    MUSER_CUDA_TRY(ctx, launch_pdl(head_rms_norm_kernel, dim3(blocks), dim3(256), 0, stream, x, w, eps, total, head_dim, blocks <= (uint32_t)ctx->sm_count));
    return MUSER_CUDA_OK;
}

} // namespace muser
