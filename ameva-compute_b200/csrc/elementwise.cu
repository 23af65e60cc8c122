// The f32 row operations that sit between the quantized mul_mats of a decoder layer: residual ADD, MUL, the split
// SWIGLU gate and RMS normalisation (alone or with the weight multiply that follows it). They keep a llama.cpp graph on
// the device between two MUL_MATs; the first three are also what the decode GEMV's fused epilogue computes when the
// consumer directly follows a one-row product.
//
// Reference: the corresponding ops of the reference's graph engine (adapters/llama/ggml-ameva/ggml-ameva.cpp:5249-5285;
// fusion pairs RMS_NORM + MUL and MUL_MAT + ADD / GLU, :4345-4378). Arithmetic as ggml's CPU backend states it:
// silu(x) = x / (1 + exp(-x)); rms_norm: y = x * (1 / sqrt(mean(x^2) + eps)), the mean accumulated here in fp32 by a
// tree (ggml accumulates in double: results agree to fp32 rounding of the scale).
#include <cstring>

#include "common.cuh"

namespace amv {

// Elements per thread of the vector forms: two 16-byte pieces half a CTA's span apart, so that a thread has two (binary,
// SWIGLU: four) independent 16-byte loads in flight. Bound by HBM / L2. One 4-byte element per thread (the scalar forms
// below) measured 34 us for the SWIGLU of 512 x 14336 and 11 us for the residual ADD of 512 x 4096.
constexpr uint32_t kVecThreads = 256, kVecPieces = 2;

template <int OP>
__device__ __forceinline__ float binary_op(float x, float y) { return OP == 0 ? x + y : x * y; }

// dst[i] = a[i] (+ | *) b[i], 16 bytes at a time; the last total % 4 elements by the first threads of the last CTA
template <int OP>
__global__ void __launch_bounds__(kVecThreads) binary_f32_vec_kernel(const float* a, const float* b, float* dst,
                                                                     uint64_t total) {
    pdl_trigger();
    pdl_wait();
    const uint64_t n4 = total >> 2, i0 = (uint64_t)blockIdx.x * (kVecThreads * kVecPieces) + threadIdx.x;
    float4 x[kVecPieces], y[kVecPieces];
#pragma unroll
    for (uint32_t k = 0; k < kVecPieces; ++k) {
        const uint64_t i = i0 + k * kVecThreads;
        if (i < n4) {
            x[k] = reinterpret_cast<const float4*>(a)[i];
            y[k] = reinterpret_cast<const float4*>(b)[i];
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kVecPieces; ++k) {
        const uint64_t i = i0 + k * kVecThreads;
        if (i < n4)
            reinterpret_cast<float4*>(dst)[i] = make_float4(binary_op<OP>(x[k].x, y[k].x), binary_op<OP>(x[k].y, y[k].y),
                                                            binary_op<OP>(x[k].z, y[k].z), binary_op<OP>(x[k].w, y[k].w));
    }
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x < (total & 3u)) {
        const uint64_t i = 4u * n4 + threadIdx.x;
        dst[i] = binary_op<OP>(a[i], b[i]);
    }
}

// dst[r][c] = a[r][c] (+ | *) b[r % b_rows][c]; rows are `cols` floats apart in all three
template <int OP>
__global__ void __launch_bounds__(256) binary_f32_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                         float* __restrict__ dst, uint64_t total, uint32_t cols,
                                                         uint32_t b_rows) {
    pdl_trigger();
    pdl_wait();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const uint64_t r = i / cols;
    const uint32_t c = (uint32_t)(i - r * cols);
    dst[i] = binary_op<OP>(a[i], b[(r % b_rows) * cols + c]);
}

// dst = silu(gate) * up
__global__ void __launch_bounds__(kVecThreads) swiglu_f32_vec_kernel(const float* gate, const float* up, float* dst,
                                                                     uint64_t total) {
    pdl_trigger();
    pdl_wait();
    const uint64_t n4 = total >> 2, i0 = (uint64_t)blockIdx.x * (kVecThreads * kVecPieces) + threadIdx.x;
    float4 g[kVecPieces], u[kVecPieces];
#pragma unroll
    for (uint32_t k = 0; k < kVecPieces; ++k) {
        const uint64_t i = i0 + k * kVecThreads;
        if (i < n4) {
            g[k] = reinterpret_cast<const float4*>(gate)[i];
            u[k] = reinterpret_cast<const float4*>(up)[i];
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kVecPieces; ++k) {
        const uint64_t i = i0 + k * kVecThreads;
        if (i < n4)
            reinterpret_cast<float4*>(dst)[i] =
                make_float4(swiglu_f32(g[k].x, u[k].x), swiglu_f32(g[k].y, u[k].y), swiglu_f32(g[k].z, u[k].z), swiglu_f32(g[k].w, u[k].w));
    }
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x < (total & 3u)) {
        const uint64_t i = 4u * n4 + threadIdx.x;
        dst[i] = swiglu_f32(gate[i], up[i]);
    }
}
__global__ void __launch_bounds__(256) swiglu_f32_kernel(const float* __restrict__ gate, const float* __restrict__ up,
                                                         float* __restrict__ dst, uint64_t total) {
    pdl_trigger();
    pdl_wait();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < total) dst[i] = swiglu_f32(gate[i], up[i]);
}

// one CTA per row: y = x * rsqrt(mean(x^2) + eps) [* w]
__global__ void __launch_bounds__(256) rms_norm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                           float* __restrict__ dst, uint32_t cols, float eps,
                                                           uint32_t has_weight) {
    pdl_trigger();
    pdl_wait();
    __shared__ float red[8];
    const float* row = x + (size_t)blockIdx.x * cols;
    float* out = dst + (size_t)blockIdx.x * cols;
    float ss = 0.0f;
    for (uint32_t c = threadIdx.x; c < cols; c += 256u) ss = fmaf(row[c], row[c], ss);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += red[i];
    const float scale = __fdiv_rn(1.0f, sqrtf(__fdiv_rn(tot, (float)cols) + eps));
    for (uint32_t c = threadIdx.x; c < cols; c += 256u) {
        const float v = __fmul_rn(row[c], scale);
        out[c] = has_weight ? __fmul_rn(v, w[c]) : v;
    }
}

// The same for rows of whole 16-byte pieces that fit the registers (J per thread): the row and the weight row
// are each read once, all loads of a thread in flight together, instead of twice with a 4-byte load per step.
template <int J>
__global__ void __launch_bounds__(256) rms_norm_f32_vec_kernel(const float* x, const float* w, float* dst, uint32_t cols,
                                                               float eps, uint32_t has_weight) {
    __shared__ float red[8];
    const uint32_t P = cols >> 2;
    const float4* row = reinterpret_cast<const float4*>(x + (size_t)blockIdx.x * cols);
    float4* out = reinterpret_cast<float4*>(dst + (size_t)blockIdx.x * cols);
    pdl_trigger();
    pdl_wait();
    float4 v[J], g[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t i = threadIdx.x + 256u * j;
        v[j] = i < P ? row[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (has_weight && i < P) g[j] = reinterpret_cast<const float4*>(w)[i];
    }
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < J; ++j) ss = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, ss))));
    ss = warp_sum(ss);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += red[i];
    const float scale = __fdiv_rn(1.0f, sqrtf(__fdiv_rn(tot, (float)cols) + eps));
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t i = threadIdx.x + 256u * j;
        if (i >= P) continue;
        float4 y = make_float4(__fmul_rn(v[j].x, scale), __fmul_rn(v[j].y, scale), __fmul_rn(v[j].z, scale), __fmul_rn(v[j].w, scale));
        if (has_weight)
            y = make_float4(__fmul_rn(y.x, g[j].x), __fmul_rn(y.y, g[j].y), __fmul_rn(y.z, g[j].z), __fmul_rn(y.w, g[j].w));
        out[i] = y;
    }
}

// From here on the vector forms: below it (rows of token generation) one element per thread spreads the few thousand elements
// over more SMs (a decoder layer at one row, 4096 wide: 93.0 against 93.9 us).
constexpr uint64_t kVecMin = 1u << 16;
// SWIGLU: eight exponentials and divisions in a row per thread take longer than the loads they save until the chip is full
// (us, vector form / scalar: 65536 elements 2.8 / 1.8, 524288 3.6 / 3.3, 2097152 6.2 / 9.5)
constexpr uint64_t kVecMinGate = 1u << 20;

// ameva_add_f32 / ameva_mul_f32: bindings 0 a f32 [rows][cols], 1 b f32 [b_rows][cols], 2 dst f32 [rows][cols];
//   push {rows, cols, b_rows (rows % b_rows == 0; 1 = one row broadcast over all)}
template <int OP>
static AcResult launch_binary(const LaunchArgs& a) {
    const uint32_t rows = a.push[0], cols = a.push[1], b_rows = a.push[2];
    if (rows == 0 || cols == 0 || b_rows == 0 || rows % b_rows) return AC_ERR_KERNEL_ARG_INVALID;
    const uint64_t total = (uint64_t)rows * cols;
    if (a.range[0] < total * 4u || a.range[1] < (uint64_t)b_rows * cols * 4u || a.range[2] < total * 4u)
        return AC_ERR_INVALID_BUFFER_SIZE;
    const uint64_t blocks = (total + 255u) / 256u;
    if (blocks > 0x7FFFFFFFull) return AC_ERR_INVALID_WORK_ITEM_DIMS;
    // same-shape operands are one linear walk of 16-byte pieces (bindings start on 64 bytes; a broadcast b stays on the scalar
    // form: its index needs the column)
    if (b_rows == rows && total >= kVecMin) {
        const uint64_t span = 4u * kVecThreads * kVecPieces;
        launch_pdl(binary_f32_vec_kernel<OP>, dim3((unsigned)((total + span - 1u) / span)), dim3(kVecThreads), 0, a.stream,
                   (const float*)a.ptr[0], (const float*)a.ptr[1], (float*)a.ptr[2], total);
        return check_launch();
    }
    launch_pdl(binary_f32_kernel<OP>, dim3((unsigned)blocks), dim3(256), 0, a.stream, (const float*)a.ptr[0],
               (const float*)a.ptr[1], (float*)a.ptr[2], total, cols, b_rows);
    return check_launch();
}
AcResult launch_add_f32(const LaunchArgs& a) { return launch_binary<0>(a); }
AcResult launch_mul_f32(const LaunchArgs& a) { return launch_binary<1>(a); }

// ameva_swiglu_f32: bindings 0 gate f32 [n], 1 up f32 [n], 2 dst f32 [n]; push {n}
AcResult launch_swiglu_f32(const LaunchArgs& a) {
    const uint64_t n = a.push[0];
    if (n == 0) return AC_ERR_KERNEL_ARG_INVALID;
    if (a.range[0] < n * 4u || a.range[1] < n * 4u || a.range[2] < n * 4u) return AC_ERR_INVALID_BUFFER_SIZE;
    if (n >= kVecMinGate) {
        const uint64_t span = 4u * kVecThreads * kVecPieces;
        launch_pdl(swiglu_f32_vec_kernel, dim3((unsigned)((n + span - 1u) / span)), dim3(kVecThreads), 0, a.stream,
                   (const float*)a.ptr[0], (const float*)a.ptr[1], (float*)a.ptr[2], n);
        return check_launch();
    }
    launch_pdl(swiglu_f32_kernel, dim3((unsigned)((n + 255u) / 256u)), dim3(256), 0, a.stream, (const float*)a.ptr[0],
               (const float*)a.ptr[1], (float*)a.ptr[2], n);
    return check_launch();
}

// ameva_rms_norm_f32: bindings 0 x f32 [rows][cols], 1 w f32 [cols] (any buffer when has_weight = 0), 2 dst f32;
//   push {rows, cols, eps (float bits), has_weight}
AcResult launch_rms_norm_f32(const LaunchArgs& a) {
    const uint32_t rows = a.push[0], cols = a.push[1], has_weight = a.push[3];
    if (rows == 0 || cols == 0 || has_weight > 1u) return AC_ERR_KERNEL_ARG_INVALID;
    const uint64_t total = (uint64_t)rows * cols;
    if (a.range[0] < total * 4u || (has_weight && a.range[1] < (uint64_t)cols * 4u) || a.range[2] < total * 4u)
        return AC_ERR_INVALID_BUFFER_SIZE;
    float eps;
    memcpy(&eps, &a.push[2], 4);
    if (!(eps >= 0.0f)) return AC_ERR_KERNEL_ARG_INVALID;
    // rows of whole 16-byte pieces, at most eight of them per thread (64 registers): the form that reads a row once
    if ((cols & 3u) == 0u && cols <= 8192u) {
        const uint32_t J = ((cols >> 2) + 255u) / 256u;
        auto go = [&](void (*kernel)(const float*, const float*, float*, uint32_t, float, uint32_t)) {
            launch_pdl(kernel, dim3(rows), dim3(256), 0, a.stream, (const float*)a.ptr[0], (const float*)a.ptr[1],
                       (float*)a.ptr[2], cols, eps, has_weight);
        };
        if (J <= 1) go(rms_norm_f32_vec_kernel<1>);
        else if (J <= 2) go(rms_norm_f32_vec_kernel<2>);
        else if (J <= 4) go(rms_norm_f32_vec_kernel<4>);
        else go(rms_norm_f32_vec_kernel<8>);
        return check_launch();
    }
    launch_pdl(rms_norm_f32_kernel, dim3(rows), dim3(256), 0, a.stream, (const float*)a.ptr[0], (const float*)a.ptr[1],
               (float*)a.ptr[2], cols, eps, has_weight);
    return check_launch();
}

}  // namespace amv
