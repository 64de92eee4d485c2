// Device pieces shared by the input quantisers (quantize_input_q8_0, rmsnorm_quantize_q8_0; flare-core/src/model.rs:
// 5507-5527, 5610-5641): used by the standalone kernels and by the matrix-vector kernel's prologue.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

__device__ __forceinline__ int8_t flare_to_i8_saturating(float r) {       // Rust `as i8`
    return (int8_t)((r != r) ? 0 : (r >= 127.0f ? 127 : (r <= -128.0f ? -128 : (int)r)));
}

// One warp, one block of 32 values (lane = element): amax, scale = amax / 127, code = round(n * (127 / amax)) as i8.
// Returns this lane's code; every lane gets the scale.
__device__ __forceinline__ int flare_q8_code(float n, float& scale) {
    float amax = fabsf(n);
#pragma unroll
    for (int off = 16; off; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    scale = __fdiv_rn(amax, 127.0f);
    const float inv_scale = scale != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    return flare_to_i8_saturating(roundf(__fmul_rn(n, inv_scale)));
}
__device__ __forceinline__ void flare_quantize_block_of_32(float n, int lane, int8_t* q_out, float* s_out) {
    float scale;
    q_out[lane] = (int8_t)flare_q8_code(n, scale);
    if (lane == 0) *s_out = scale;
}

// Four values per lane, eight lanes per block (all of a block's lanes take part): this lane's four codes, and the block's
// scale on every lane.
__device__ __forceinline__ uint32_t flare_q8_quad(const float (&n)[4], float& scale) {
    float amax = fmaxf(fmaxf(fabsf(n[0]), fabsf(n[1])), fmaxf(fabsf(n[2]), fabsf(n[3])));
#pragma unroll
    for (int off = 4; off; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    scale = __fdiv_rn(amax, 127.0f);
    const float inv_scale = scale != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) c |= (uint32_t)(uint8_t)flare_to_i8_saturating(roundf(__fmul_rn(n[i], inv_scale))) << (8 * i);
    return c;
}

// The sum of squares of a vector that one warp of eight contributes (warp w: blocks w, w + 8, .., lane = element) and
// the norm's factor from all eight: one order of additions for every kernel that normalises.
__device__ __forceinline__ float flare_sum_sq_of_warp(const float* __restrict__ x, int dim, int warp, int lane) {
    float s = 0.0f;
#pragma unroll 8
    for (int i = warp * 32 + lane; i < dim; i += 256) s = fmaf(x[i], x[i], s);
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}
__device__ __forceinline__ float flare_inv_rms(const float* s_sq, int dim, float eps) {
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++) sum += s_sq[w];
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)dim), eps)));
}
// The two norms of the CPU multiply in different order: rmsnorm_quantize_q8_0 (x * weight) * inv_rms, rmsnorm_into
// (x * inv_rms) * weight.
__device__ __forceinline__ void flare_norm_quad(float (&n)[4], const float* __restrict__ weight, float inv_rms, bool weight_first) {
    const float4 w4 = __ldg(reinterpret_cast<const float4*>(weight));
    const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
        n[i] = weight_first ? __fmul_rn(__fmul_rn(n[i], w[i]), inv_rms) : __fmul_rn(__fmul_rn(n[i], inv_rms), w[i]);
}
