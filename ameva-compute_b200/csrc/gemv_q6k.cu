// Q6_K x Q8_K (and, below, Q5_K x Q8_K) mul_mat for up to 8 activation rows (token generation; more rows run in chunks
// of 8).
//
// A Q6_K weight is d * scale[e / 16] * (q6 - 32) with 6-bit q6 split over ql / qh (ggml-common.h block_q6_K: ql[128],
// qh[64], scales[16] int8, d fp16: 210 bytes per 256 weights). The upload decodes q6 - 32 to int8 in element order and
// keeps the scale bytes (registry.cu decode_q6_K; 274 bytes per block on the device), so the kernel reads a 16-weight
// group with one 16-byte load and multiplies it with the int8 activations by four dp4a:
//   y[m][n] = sum_blocks (d_w * d_a) * sum_{g < 16} scale[g] * sum_{i < 16} (q6 - 32)[16 g + i] * q8[16 g + i]
// which is ggml_vec_dot_q6_K_q8_K's arithmetic (generic branch: aux32 += scale * (q8 * (q6 - 32)), sumf += d * aux32)
// with the integers exact and the fp32 products summed per lane and then over the warp (ggml sums per block in lane
// order 0..7; the results agree to fp32 rounding). The reference serves Q6_K through its f32 GEMV with the weights
// decoded in the shader (adapters/llama/ggml-ameva/shaders/ameva_qdecode.glsl, decode of type 14;
// ggml-ameva-repack.cpp:21-28 lists q6_K in the repacked family).
//
// All seven byte-decoded types run in one kernel body (byte_gemv_kernel) with a policy for the scale records: one warp per
// weight row, eight rows per CTA; a lane walks the row's 16-weight groups with stride 32, so a warp's loads are 512
// contiguous bytes; weights bypass L1, which keeps the activation rows. Bound by HBM (Q6_K: 274 bytes per 256 weights) and, at
// token-generation sizes, by the latency of a launch's dependent loads: the scale records and the first two steps of weights
// (eight 16-byte loads per lane) are requested before the wait for the preceding kernel, and the step after next is in
// flight during the arithmetic. 4096 x 11008 in a decoder layer: 16.6 us as one launch of its own before, the layer 85.0 -> 81.1 us.
#include "common.cuh"

namespace amv {

constexpr int kQ6Warps = 8;
constexpr uint32_t kQ6ScaleBytes = 18;   // 16 int8 sub-block scales + fp16 d, as in the ggml block

// one 16-weight group of a row against the M activation rows
template <int M>
__device__ __forceinline__ void group_dot(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ,
                                          const uint8_t* __restrict__ AB, uint32_t K, uint32_t B, float (&acc)[M]) {
    const uint32_t blk = gi >> 4, g = gi & 15u;
    const uint8_t* rec = s + blk * kQ6ScaleBytes;
    const int sc = (int)(int8_t)rec[g];
    const float dw = h2f((uint16_t)(rec[16] | ((uint32_t)rec[17] << 8)));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint4 a = *reinterpret_cast<const uint4*>(AQ + (size_t)m * K + 16u * gi);
        int t = dp4a_ss(w.x, a.x, 0);
        t = dp4a_ss(w.y, a.y, t);
        t = dp4a_ss(w.z, a.z, t);
        t = dp4a_ss(w.w, a.w, t);
        const float da = *reinterpret_cast<const float*>(AB + ((size_t)m * B + blk) * kABBytes + 32);
        acc[m] = fmaf(dw * da, (float)(sc * t), acc[m]);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Q5_K x Q8_K, the same way: a Q5_K weight is d * sc[j] * q5 - dmin * m[j] for sub-block j = e / 32 (ggml-common.h
// block_q5_K: d, dmin, scales[12] with packed 6-bit sc / m, qh[32], qs[128]: 176 bytes per 256 weights). The upload
// decodes q5 (0..31) to bytes in element order and keeps the first 16 bytes of the block as the scale record (the
// record of Q4_K), 272 bytes per block on the device.
//   y[m][n] = sum_blocks d_a * ( d * sum_j sc[j] * sum_i q5 * q8  -  dmin * sum_j m[j] * bsum(j) )
// as ggml_vec_dot_q5_K_q8_K (generic branch) forms it; a lane takes 16 weights (half a sub-block) with the Q8_K half-sum
// of the same 16 activations for the min term.
// ---------------------------------------------------------------------------------------------------------------------
template <int M>
__device__ __forceinline__ void group_dot_q5(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ,
                                             const uint8_t* __restrict__ AB, uint32_t K, uint32_t B, float (&acc)[M]) {
    const uint32_t blk = gi >> 4, g = gi & 15u, j = g >> 1;
    const uint8_t* rec = s + blk * 16u;
    const uint32_t hd = *reinterpret_cast<const uint32_t*>(rec);
    const uint8_t* sm = rec + 4;
    int sc, mn;   // get_scale_min_k4
    if (j < 4u) {
        sc = sm[j] & 63;
        mn = sm[j + 4u] & 63;
    } else {
        sc = (sm[j + 4u] & 0x0F) | ((sm[j - 4u] >> 6) << 4);
        mn = (sm[j + 4u] >> 4) | ((sm[j] >> 6) << 4);
    }
    const float dw = h2f((uint16_t)(hd & 0xFFFFu)), dmin = h2f((uint16_t)(hd >> 16));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint4 a = *reinterpret_cast<const uint4*>(AQ + (size_t)m * K + 16u * gi);
        int t = dp4a_ss(w.x, a.x, 0);
        t = dp4a_ss(w.y, a.y, t);
        t = dp4a_ss(w.z, a.z, t);
        t = dp4a_ss(w.w, a.w, t);
        const uint8_t* ab = AB + ((size_t)m * B + blk) * kABBytes;
        const float da = *reinterpret_cast<const float*>(ab + 32);
        const int bs = (int)reinterpret_cast<const int16_t*>(ab)[g];
        acc[m] += (dw * da) * (float)(sc * t) - (dmin * da) * (float)(mn * bs);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// IQ4_XS x Q8_K: a weight is d * (ls[e / 32] - 32) * kvalues_iq4nl[q4] (ggml-common.h block_iq4_xs: d, scales_h,
// scales_l[4], qs[128]: 136 bytes per 256 weights; ls is 6 bits: four from scales_l, two from scales_h). The upload
// decodes kvalues[q4] to int8 in element order and keeps the first 8 bytes of the block as the scale record (264 bytes
// per block on the device). y = sum_blocks (d * d_a) * sum_ib (ls[ib] - 32) * sum_i kv * q8, as
// ggml_vec_dot_iq4_xs_q8_K forms it.
// ---------------------------------------------------------------------------------------------------------------------
template <int M>
__device__ __forceinline__ void group_dot_iq4xs(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ,
                                                const uint8_t* __restrict__ AB, uint32_t K, uint32_t B, float (&acc)[M]) {
    const uint32_t blk = gi >> 4, ib = (gi & 15u) >> 1;
    const uint2 rec = *reinterpret_cast<const uint2*>(s + blk * 8u);   // d | scales_h << 16, scales_l[0..3]
    const uint32_t lo = (rec.y >> (4u * ib)) & 0x0Fu, hi = ((rec.x >> 16) >> (2u * ib)) & 3u;
    const int ls = (int)(lo | (hi << 4)) - 32;
    const float dw = h2f((uint16_t)(rec.x & 0xFFFFu));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint4 a = *reinterpret_cast<const uint4*>(AQ + (size_t)m * K + 16u * gi);
        int t = dp4a_ss(w.x, a.x, 0);
        t = dp4a_ss(w.y, a.y, t);
        t = dp4a_ss(w.z, a.z, t);
        t = dp4a_ss(w.w, a.w, t);
        const float da = *reinterpret_cast<const float*>(AB + ((size_t)m * B + blk) * kABBytes + 32);
        acc[m] = fmaf(dw * da, (float)(ls * t), acc[m]);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Q4_1 / Q5_1 x Q8_0-with-sums (ggml's Q8_1): a weight is d * q + m per 32 (q = 0..15 / 0..31), so
//   y = sum_blocks (d_w * d_a) * sum_i q * q8 + m_w * (d_a * sum_i q8)
// as ggml_vec_dot_q4_1_q8_1 / _q5_1_q8_1 form it (there d_a * sum q8 is the fp16 field s of the Q8_1 block; here it is
// the product of the activation record's fp16 d and int16 sum in fp32). The upload decodes q to bytes (32 per block) and
// keeps (d, m) as a 4-byte record; one kernel serves both types.
// ---------------------------------------------------------------------------------------------------------------------
template <int M>
__device__ __forceinline__ void group_dot_q41(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ,
                                              const uint8_t* __restrict__ ADb, uint32_t K, uint32_t U, float (&acc)[M]) {
    const uint32_t* AD = reinterpret_cast<const uint32_t*>(ADb);
    const uint32_t u = gi >> 1, rec = reinterpret_cast<const uint32_t*>(s)[u];
    const float dw = h2f((uint16_t)(rec & 0xFFFFu)), mw = (gi & 1u) ? 0.0f : h2f((uint16_t)(rec >> 16));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint4 a = *reinterpret_cast<const uint4*>(AQ + (size_t)m * K + 16u * gi);
        int t = dp4a_ss(w.x, a.x, 0);
        t = dp4a_ss(w.y, a.y, t);
        t = dp4a_ss(w.z, a.z, t);
        t = dp4a_ss(w.w, a.w, t);
        const uint32_t adw = AD[(size_t)m * U + u];
        const float da = h2f((uint16_t)(adw & 0xFFFFu));
        acc[m] += (dw * da) * (float)t + mw * (da * (float)(int)(int16_t)(adw >> 16));
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Q3_K and Q2_K x Q8_K. Q3_K: a weight is d * (scale[e / 16] - 32) * q3, q3 = -4..3 from two bits of qs and one of hmask,
// scale six bits packed in scales[12] (ggml-common.h block_q3_K: hmask[32], qs[64], scales[12], d: 110 bytes per 256
// weights); the upload decodes q3 to int8 and keeps scales[12] + d as a 14-byte record. Q2_K: d * (sc[e / 16] & 15) * q2
// - dmin * (sc[e / 16] >> 4), q2 = 0..3 (block_q2_K: scales[16], qs[64], d, dmin: 84 bytes); the upload decodes q2 to
// bytes and keeps scales[16], d, dmin as a 20-byte record. Sums as ggml_vec_dot_q3_K_q8_K / _q2_K_q8_K (generic branch)
// form them; Q2_K's min term uses the Q8_K sum of the same 16 activations. KIND 3 / 2 selects the type.
// ---------------------------------------------------------------------------------------------------------------------
template <int M, int KIND>
__device__ __forceinline__ void group_dot_q23(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ,
                                              const uint8_t* __restrict__ AB, uint32_t K, uint32_t B, float (&acc)[M]) {
    constexpr uint32_t kRec = KIND == 3 ? 14u : 20u;
    const uint32_t blk = gi >> 4, g = gi & 15u;
    const uint8_t* rec = s + blk * kRec;
    int sc, mn = 0;
    float dw, dmin = 0.0f;
    if (KIND == 3) {
        const uint32_t lo = g < 8u ? (rec[g] & 0x0Fu) : (rec[g - 8u] >> 4);
        const uint32_t hi = (rec[8u + (g & 3u)] >> (2u * (g >> 2))) & 3u;
        sc = (int)(lo | (hi << 4)) - 32;
        dw = h2f((uint16_t)(rec[12] | ((uint32_t)rec[13] << 8)));
    } else {
        sc = rec[g] & 0x0F;
        mn = rec[g] >> 4;
        dw = h2f((uint16_t)(rec[16] | ((uint32_t)rec[17] << 8)));
        dmin = h2f((uint16_t)(rec[18] | ((uint32_t)rec[19] << 8)));
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint4 a = *reinterpret_cast<const uint4*>(AQ + (size_t)m * K + 16u * gi);
        int t = dp4a_ss(w.x, a.x, 0);
        t = dp4a_ss(w.y, a.y, t);
        t = dp4a_ss(w.z, a.z, t);
        t = dp4a_ss(w.w, a.w, t);
        const uint8_t* ab = AB + ((size_t)m * B + blk) * kABBytes;
        const float da = *reinterpret_cast<const float*>(ab + 32);
        if (KIND == 3) {
            acc[m] = fmaf(dw * da, (float)(sc * t), acc[m]);
        } else {
            const int bs = (int)reinterpret_cast<const int16_t*>(ab)[g];
            acc[m] += (dw * da) * (float)(sc * t) - (dmin * da) * (float)(mn * bs);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// The kernel. A policy names the weights per scale record (1 << kUnit), the bytes of a record and the dot product of one
// 16-weight group. add: the ADD behind the product, when the launch carries it (M rows of N floats without gaps).
// ---------------------------------------------------------------------------------------------------------------------
#define AMV_BYTE_POLICY(NAME, UNIT, REC, AHEAD, DOT)                                                                       \
    struct NAME {                                                                                                          \
        static constexpr uint32_t kUnit = UNIT, kRec = REC;                                                                \
        static constexpr bool kAhead = AHEAD;                                                                              \
        template <int M>                                                                                                   \
        static __device__ __forceinline__ void dot(const uint4 w, uint32_t gi, const uint8_t* s, const int8_t* __restrict__ AQ, \
                                                   const uint8_t* __restrict__ AD, uint32_t K, uint32_t units, float (&acc)[M]) { \
            DOT(w, gi, s, AQ, AD, K, units, acc);                                                                          \
        }                                                                                                                  \
    };
AMV_BYTE_POLICY(ByteQ6K, 8, kQ6ScaleBytes, true, group_dot<M>)
AMV_BYTE_POLICY(ByteQ5K, 8, 16, false, group_dot_q5<M>)
AMV_BYTE_POLICY(ByteIq4Xs, 8, 8, true, group_dot_iq4xs<M>)
AMV_BYTE_POLICY(ByteQ41, 5, 4, true, group_dot_q41<M>)
AMV_BYTE_POLICY(ByteQ3K, 8, 14, true, (group_dot_q23<M, 3>))
AMV_BYTE_POLICY(ByteQ2K, 8, 20, true, (group_dot_q23<M, 2>))
#undef AMV_BYTE_POLICY

struct ByteAdd {
    const float* e;
    float* out;
};

// AHEAD (see the launcher): the first two steps of weights are requested before the wait, and a step is always in flight during
// the arithmetic. Otherwise a step is requested when it is needed. 64 registers for both, four CTAs per SM: left to itself the
// compiler takes 32-60 without AHEAD and keeps fewer loads in flight (Q5_K x 8 rows, 4096 x 14336: 60.8 us, with the bound 42.4;
// the kernels of the single types took 45.1).
template <class T, int M, bool AHEAD>
__global__ void __launch_bounds__(kQ6Warps * 32, 4)
byte_gemv_kernel(const uint8_t* __restrict__ Q, const uint8_t* __restrict__ S, const int8_t* __restrict__ AQ,
                 const uint8_t* __restrict__ AD, float* __restrict__ dst, uint32_t N, uint32_t K, uint32_t dst_stride,
                 const ByteAdd add) {
    constexpr uint32_t UN = 4, STEP = 32u * UN;   // groups per step of a warp
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t row = blockIdx.x * kQ6Warps + warp;
    if (row >= N) return;
    const uint32_t units = K >> T::kUnit, groups = K >> 4;
    const uint4* q = reinterpret_cast<const uint4*>(Q + (size_t)row * K);
    extern __shared__ __align__(16) uint8_t byte_smem[];
    const uint32_t rec_bytes = units * T::kRec;
    uint8_t* s = byte_smem + (size_t)warp * ((rec_bytes + 15u) & ~15u);
    // neither the weights nor their scale records depend on the kernel before this one
    uint4 ahead[AHEAD ? 2u * UN : 1u];
    if constexpr (AHEAD) {
#pragma unroll
        for (uint32_t u = 0; u < 2u * UN; ++u)
            if (32u * u + lane < groups) ahead[u] = ld_stream_u4(q + 32u * u + lane);
    }
    const uint8_t* src = S + (size_t)row * rec_bytes;
    if (((uintptr_t)src & 3u) == 0u && (rec_bytes & 3u) == 0u) {
        for (uint32_t i = lane; i < rec_bytes / 4u; i += 32u) reinterpret_cast<uint32_t*>(s)[i] = __ldg(reinterpret_cast<const uint32_t*>(src) + i);
    } else {   // (records of 18 or 14 bytes)
        for (uint32_t i = lane; i < rec_bytes / 2u; i += 32u) reinterpret_cast<uint16_t*>(s)[i] = __ldg(reinterpret_cast<const uint16_t*>(src) + i);
    }
    pdl_trigger();   // the kernel behind this one may be scheduled (it waits for this grid before touching what it wrote)
    pdl_wait();      // the activations come from the preceding kernel
    __syncwarp();
    float acc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[m] = 0.0f;
    if constexpr (AHEAD) {
        for (uint32_t base = 0; base < groups; base += STEP) {
#pragma unroll
            for (uint32_t u = 0; u < UN; ++u) {
                const uint32_t gi = base + 32u * u + lane;
                if (gi < groups) T::template dot<M>(ahead[u], gi, s, AQ, AD, K, units, acc);
            }
#pragma unroll
            for (uint32_t u = 0; u < UN; ++u) {
                ahead[u] = ahead[UN + u];
                const uint32_t gi = base + 2u * STEP + 32u * u + lane;
                if (gi < groups) ahead[UN + u] = ld_stream_u4(q + gi);
            }
        }
    } else {
        uint32_t gi = lane;
        for (; gi + 32u * (UN - 1u) < groups; gi += STEP) {
            uint4 w[UN];
#pragma unroll
            for (uint32_t u = 0; u < UN; ++u) w[u] = ld_stream_u4(q + gi + 32u * u);
#pragma unroll
            for (uint32_t u = 0; u < UN; ++u) T::template dot<M>(w[u], gi + 32u * u, s, AQ, AD, K, units, acc);
        }
        for (; gi < groups; gi += 32u) T::template dot<M>(ld_stream_u4(q + gi), gi, s, AQ, AD, K, units, acc);
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const float v = warp_sum(acc[m]);
        if (lane == 0) {
            dst[(size_t)m * dst_stride + row] = v;
            if (add.out) add.out[(size_t)m * N + row] = v + add.e[(size_t)m * N + row];
        }
    }
}

// Bindings 0 Q (one byte per weight, decoded at upload, [N][K]), 1 S (the type's scale records), 2 AQ int8 [M][K], 3 AB
// (48-byte Q8_K records [M][K/256]) or AD (per-32 scale words), 4 dst f32 [M][dst_stride]; push {M (1..8), N, K, dst_stride}
template <class T>
static AcResult launch_byte_gemv(const LaunchArgs& a, uint32_t max_k, uintptr_t s_align) {
    const uint32_t M = a.push[0], N = a.push[1], K = a.push[2], dst_stride = a.push[3];
    if (M == 0 || M > 8) return AC_ERR_INVALID_SHAPE;
    if (N == 0 || K == 0 || (K & ((1u << T::kUnit) - 1u)) || K > max_k || dst_stride < N) return AC_ERR_KERNEL_ARG_INVALID;
    const uint64_t units = K >> T::kUnit;
    if (a.range[0] < (uint64_t)N * K || a.range[1] < (uint64_t)N * units * T::kRec || a.range[2] < (uint64_t)M * K ||
        a.range[3] < (uint64_t)M * units * (T::kUnit == 8u ? kABBytes : 4u) ||
        a.range[4] < ((uint64_t)(M - 1) * dst_stride + N) * 4u)
        return AC_ERR_INVALID_BUFFER_SIZE;
    if ((((uintptr_t)a.ptr[0] | (uintptr_t)a.ptr[2]) & 15u) || ((uintptr_t)a.ptr[1] & (s_align - 1u)) ||
        (T::kUnit == 5u && ((uintptr_t)a.ptr[3] & 3u)))
        return AC_ERR_BUFFER_ALIGNMENT_INVALID;
    const size_t smem = (size_t)kQ6Warps * ((units * T::kRec + 15u) & ~15ull);   // (at most 41 KB)
    const ByteAdd add = {a.add_e, a.add_out};
    auto go = [&](auto kernel) {
        launch_pdl(kernel, dim3((N + kQ6Warps - 1) / kQ6Warps), dim3(kQ6Warps * 32), smem, a.stream, (const uint8_t*)a.ptr[0],
                   (const uint8_t*)a.ptr[1], (const int8_t*)a.ptr[2], (const uint8_t*)a.ptr[3], (float*)a.ptr[4], N, K, dst_stride, add);
    };
    // AHEAD where its four CTAs per SM are a wave of their own or one of many (us, AHEAD / not, Q6_K x 1 row: 4096 x 14336 10.0 /
    // 14.6, 4096 x 4096 3.4 / 4.6, 28672 x 4096 20.0 / 20.9; 5203 x 4096 5.5 / 4.9, 1024 x 4096 2.8 / 2.6); never for Q5_K, whose
    // dot product does not fit 64 registers with it (5203 x 4096 10.2 / 5.6)
    const uint64_t ctas = (N + kQ6Warps - 1) / kQ6Warps, sms = a.sm_count > 0 ? (uint64_t)a.sm_count : 148u;
    const bool ahead = (ctas > sms && ctas <= 4u * sms) || ctas >= 16u * sms;
    switch (M) {
        case 1:
            if constexpr (T::kAhead) {
                if (ahead) {
                    go(byte_gemv_kernel<T, 1, true>);
                    break;
                }
            }
            go(byte_gemv_kernel<T, 1, false>);
            break;
        case 2: go(byte_gemv_kernel<T, 2, false>); break;
        case 3: go(byte_gemv_kernel<T, 3, false>); break;
        case 4: go(byte_gemv_kernel<T, 4, false>); break;
        case 5: go(byte_gemv_kernel<T, 5, false>); break;
        case 6: go(byte_gemv_kernel<T, 6, false>); break;
        case 7: go(byte_gemv_kernel<T, 7, false>); break;
        default: go(byte_gemv_kernel<T, 8, false>); break;
    }
    return check_launch();
}
// S records: Q6_K 18 bytes (scales[16], d), Q5_K 16 (d, dmin, packed scales), IQ4_XS 8 (d, scales_h, scales_l), Q4_1 / Q5_1 4
// per 32 weights (fp16 d | fp16 m << 16; activations per 32), Q3_K 14 (scales[12], d), Q2_K 20 (scales[16], d, dmin)
AcResult launch_mmvqb_q6_K(const LaunchArgs& a) { return launch_byte_gemv<ByteQ6K>(a, 65536u, 1u); }
AcResult launch_mmvqb_q5_K(const LaunchArgs& a) { return launch_byte_gemv<ByteQ5K>(a, 65536u, 16u); }
AcResult launch_mmvqb_iq4_xs(const LaunchArgs& a) { return launch_byte_gemv<ByteIq4Xs>(a, 65536u, 8u); }
AcResult launch_mmvq_q4_1(const LaunchArgs& a) { return launch_byte_gemv<ByteQ41>(a, 32768u, 4u); }
AcResult launch_mmvqb_q3_K(const LaunchArgs& a) { return launch_byte_gemv<ByteQ3K>(a, 65536u, 2u); }
AcResult launch_mmvqb_q2_K(const LaunchArgs& a) { return launch_byte_gemv<ByteQ2K>(a, 65536u, 2u); }

// ---------------------------------------------------------------------------------------------------------------------
// Scale table of the tensor-core GEMM for the types above (ameva_mmtc_b8): per 16 weights an fp16 pair (s, o) with
// w = s * q + o for the stored byte q, decoded from the type's scale records: Q6_K s = d * scale[g]; Q5_K s = d * sc[g / 2],
// o = -dmin * m[g / 2]; IQ4_XS s = d * (ls[g / 2] - 32); Q3_K s = d * (scale6[g] - 32); Q2_K s = d * (scales[g] & 15),
// o = -dmin * (scales[g] >> 4); Q4_1 / Q5_1 s = d, o = m of the 32-weight block g / 2. The products are exact in fp32
// (an fp16 times at most 6 bits) and rounded once to fp16. One thread per 256 weights; it runs once per weight (the
// host keeps the table) or once per prompt, and moves 64 bytes per 256 weights.
// ---------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) mmtc_scales_kernel(const uint8_t* __restrict__ S, uint32_t* __restrict__ H, uint32_t type,
                                                          uint64_t blocks) {
    pdl_wait();
    pdl_trigger();
    const uint64_t b = (uint64_t)blockIdx.x * 256u + threadIdx.x;
    if (b >= blocks) return;
    const uint32_t rec_bytes = type == 14u ? 18u : type == 13u ? 16u : type == 23u ? 8u : type == 11u ? 14u : type == 10u ? 20u : 32u;
    const uint8_t* rec = S + b * rec_bytes;
    auto half_at = [&](uint32_t off) { return h2f((uint16_t)(rec[off] | ((uint32_t)rec[off + 1u] << 8))); };
    uint32_t out[16];
#pragma unroll
    for (uint32_t g = 0; g < 16u; ++g) {
        float sv = 0.0f, ov = 0.0f;
        if (type == 14u) {
            sv = half_at(16) * (float)(int8_t)rec[g];
        } else if (type == 13u) {
            const uint32_t j = g >> 1;
            const uint8_t* sm = rec + 4;
            int sc, mn;
            if (j < 4u) {
                sc = sm[j] & 63;
                mn = sm[j + 4u] & 63;
            } else {
                sc = (sm[j + 4u] & 0x0F) | ((sm[j - 4u] >> 6) << 4);
                mn = (sm[j + 4u] >> 4) | ((sm[j] >> 6) << 4);
            }
            sv = half_at(0) * (float)sc;
            ov = -(half_at(2) * (float)mn);
        } else if (type == 23u) {
            const uint32_t ib = g >> 1, sh = rec[2] | ((uint32_t)rec[3] << 8);
            const uint32_t lo = (rec[4u + (ib >> 1)] >> (4u * (ib & 1u))) & 0x0Fu, hi = (sh >> (2u * ib)) & 3u;
            sv = half_at(0) * (float)((int)(lo | (hi << 4)) - 32);
        } else if (type == 11u) {
            const uint32_t lo = g < 8u ? (rec[g] & 0x0Fu) : (rec[g - 8u] >> 4);
            const uint32_t hi = (rec[8u + (g & 3u)] >> (2u * (g >> 2))) & 3u;
            sv = half_at(12) * (float)((int)(lo | (hi << 4)) - 32);
        } else if (type == 10u) {
            sv = half_at(16) * (float)(rec[g] & 0x0F);
            ov = -(half_at(18) * (float)(rec[g] >> 4));
        } else {   // Q4_1 / Q5_1: eight (d, m) records per 256 weights
            sv = half_at(4u * (g >> 1));
            ov = half_at(4u * (g >> 1) + 2u);
        }
        const __half2 pr = __floats2half2_rn(sv, ov);
        out[g] = *reinterpret_cast<const uint32_t*>(&pr);
    }
    uint4* dst = reinterpret_cast<uint4*>(H + b * 16u);
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) dst[i] = make_uint4(out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3]);
}

// ameva_mmtc_scales: bindings 0 S (the weight's scale records), 1 H (fp16 pairs, 64 bytes per 256 weights);
// push {device type (14, 13, 23, 11, 10, 3, 7), N, K (% 256)}
AcResult launch_mmtc_scales(const LaunchArgs& a) {
    const uint32_t type = a.push[0], N = a.push[1], K = a.push[2];
    uint32_t rec;
    switch (type) {
        case 14: rec = 18; break;
        case 13: rec = 16; break;
        case 23: rec = 8; break;
        case 11: rec = 14; break;
        case 10: rec = 20; break;
        case 3: case 7: rec = 32; break;
        default: return AC_ERR_FEATURE_NOT_SUPPORTED;
    }
    if (N == 0 || K == 0 || (K & 255u)) return AC_ERR_KERNEL_ARG_INVALID;
    const uint64_t blocks = (uint64_t)N * (K >> 8);
    if (a.range[0] < blocks * rec || a.range[1] < blocks * 64u) return AC_ERR_INVALID_BUFFER_SIZE;
    if ((uintptr_t)a.ptr[1] & 15u) return AC_ERR_BUFFER_ALIGNMENT_INVALID;
    const uint64_t grid = (blocks + 255u) / 256u;
    if (grid > 0x7fffffffull) return AC_ERR_INVALID_WORK_ITEM_DIMS;
    launch_pdl(mmtc_scales_kernel, dim3((unsigned)grid), dim3(256), 0, a.stream, (const uint8_t*)a.ptr[0], (uint32_t*)a.ptr[1],
               type, blocks);
    return check_launch();
}

}  // namespace amv
