// What the prompt attention kernels (flash_tc.cu, flash_prompt_kernel in layer_ops.cu) share on the device.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace amv {

constexpr float kLog2e = 1.44269504088896340736f;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One row by a whole warp, masked keys left out instead of multiplied by zero: a lane's D / 32 columns (from column lane * D / 32)
// of sum p V over the keys of the split, p = exp(score - ref). For rows whose accumulator is not finite: the products above
// multiply every key of a step with every row, so a NaN or an infinity in V would reach rows that do not see its key, and an
// infinity would meet the remainder of its probability, which may be zero or negative. Rare, so simple: a lane per key for the
// scores, all lanes on a key's columns for the sum.
template <int D>
__device__ __noinline__ float4 seen_keys_row(const float* qrow, const __half* k, const __half* v, const __half* mrow, uint32_t k_s1,
                                             uint32_t v_s1, uint32_t key_begin, uint32_t key_end, float scale, float softcap, float ref) {
    constexpr int C = D / 32;
    const uint32_t lane = threadIdx.x & 31u;
    const float ninf = __uint_as_float(0xFF800000u);
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t key0 = key_begin; key0 < key_end; key0 += 32u) {
        const uint32_t key = key0 + lane;
        const float mv = key >= key_end ? ninf : mrow ? __half2float(mrow[key]) : 0.0f;
        float p = 0.0f;
        if (mv != ninf) {
            const uint4* row = reinterpret_cast<const uint4*>(k + (uint64_t)key * k_s1);
            float s = 0.0f;
            for (uint32_t c = 0; c < (uint32_t)D / 8u; ++c) {
                const uint4 x = row[c];
                const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 kf = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                    s = fmaf(h2f(f2h(qrow[8u * c + 2u * j])), kf.x, s);
                    s = fmaf(h2f(f2h(qrow[8u * c + 2u * j + 1u])), kf.y, s);
                }
            }
            s *= scale;
            if (softcap != 0.0f) s = softcap * tanhf(s / softcap);
            p = ex2((s + mv - ref) * kLog2e);
        }
        for (uint32_t seen = __ballot_sync(0xffffffffu, mv != ninf); seen; seen &= seen - 1u) {
            const int b = __ffs(seen) - 1;
            const float pb = __shfl_sync(0xffffffffu, p, b);
            const __half* row = v + (uint64_t)(key0 + b) * v_s1 + C * lane;
#pragma unroll
            for (int c = 0; c < C; ++c) acc[c] = fmaf(pb, __half2float(row[c]), acc[c]);
        }
    }
    return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

}  // namespace amv
