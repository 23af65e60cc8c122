// FLASH_ATTN_EXT for prompts (ameva_flash_attn with more than sixteen rows of query positions x grouped heads, D 64 or
// 128) on the 5th-generation tensor cores. The launcher of ameva_flash_attn (layer_ops.cu) validates the arguments,
// chooses the key splits and calls launch_flash_tc.
//
// A CTA owns 128 rows = 128 / G query positions x the G heads of a KV head (row r: position q0 + r / G, head h0 + r % G)
// and walks the keys of its split in tiles of 64:
//   warp 5      streams K and V tiles with TMA (128-byte swizzle) through two stages each;
//   warp 4      issues the MMAs: S = Q K^T (both in shared memory) into one of two TMEM buffers, then O += P V with P read
//               from tensor memory and V as an MN-major shared-memory operand; S of tile j + 1 is issued before P V of tile
//               j, so the softmax of the next tile starts while the tensor core multiplies this one;
//   warps 0-3   one row per thread: read the 64 scores, online softmax in fp32, write P over the scores as two fp16 halves
//               (rounded value and remainder: the 64 columns of the scores hold both). The accumulator is rescaled only
//               when a row's maximum has grown by more than kGrowth since its last rescale (probabilities then stay below
//               e^kGrowth, well inside fp16, and the sum carries the same factor).
// Before the tiles of a window are processed the mask is scanned once: tiles that are masked for all 128 rows are left out
// of the list every role walks, tiles whose mask is all zero skip the mask arithmetic (a causal prompt has one or two mixed
// tiles per CTA), and of a mixed tile only the k-steps of 16 keys that some row sees are multiplied with V: what lies in the
// cache behind the last visible key (never written, perhaps NaN) takes no part. Up to two CTAs per SM.
// Bound by latency: 512 positions x 2048 keys of 32 heads on 8 of 128 are 128 CTAs, one per SM with one softmax warp per
// scheduler, tensor pipe 15 % active, DRAM idle (64 exponentials per thread and tile, S and P V in turn). 64 us at 2748 keys,
// 327 TFLOP/s of unmasked products; the mma.sync form (64 rows per CTA) takes 242 us. For prompts of little work that form is the
// faster one (flash_small in layer_ops.cu).
// Rounding: Q to fp16 once as in the other attention kernels, scores, sums and accumulation in fp32. P with its remainder:
// with the lazy reference the largest probability of a row is no longer exactly 1, and P rounded once left an error 1-5 %
// above the mma.sync form's (2.9e-4 against 2.8e-4 of the result); with the remainder it is 2.1e-4. Rescaling at every
// new maximum instead cost the same time and left 2.8e-4.
// Every wait on a barrier is bounded (sync_ptx.cuh); a CTA that gives up drains its copies and MMAs, frees its TMEM and
// returns. The allocation of TMEM has no bound of its own: it waits for CTAs that are resident already, and those end.
#include <cuda.h>
#include <cuda_fp16.h>

#include <cstring>

#include "common.cuh"
#include "flash_args.h"
#include "flash_row.cuh"
#include "sync_ptx.cuh"
#include "tcgen05_ptx.cuh"
#include "tensor_map.h"

namespace amv {
namespace ftc {

using namespace ptx;
using namespace tc;

constexpr uint32_t kRows = 128, kKeys = 64, kStages = 2;
constexpr uint32_t kSoftmaxWarps = 4, kWarpMma = 4, kWarpLoad = 5, kThreads = 192;
constexpr uint32_t kWindow = 512;      // key tiles scanned and listed at a time
// An entry of the list: tile of the window, a bit per 16 keys that some row sees, mixed.
constexpr uint32_t kTileMask = kWindow - 1u, kStepShift = 9, kAllSteps = 15u << kStepShift, kMixed = 0x8000u, kNoTile = 0x7FFFu;
constexpr uint32_t kTmemCols = 256;    // two S buffers of 64 columns, then D columns of O
constexpr float kGrowth = 5.0f;        // e^5 = 148

template <int D>
struct Smem {
    static constexpr uint32_t kAtoms = D / 64;                  // 64-column (128-byte) groups of a row
    static constexpr uint32_t kQ = kAtoms * kRows * 128u, kTile = kAtoms * kKeys * 128u;
    static constexpr uint32_t kBytes = 1024u + kQ + 2u * kStages * kTile + 256u + 2u * kWindow;
};

__device__ __forceinline__ uint32_t pack_halves(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Descriptor of a V tile as the B operand with its columns (N) contiguous: 64-column groups of the 128-byte swizzle
// kKeys * 128 bytes apart (leading offset), groups of eight keys 1024 bytes apart (stride offset).
__device__ __forceinline__ uint64_t make_v_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(kKeys * 128u >> 4) << 16) | (64ull << 32) | (1ull << 46) |
           (2ull << 61);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2)
flash_tc_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, const float* __restrict__ q,
                const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ mask, float* __restrict__ o, float* __restrict__ part, const FlashArgs pc,
                uint32_t n_splits, uint32_t vec, uint32_t* status) {
    using L = Smem<D>;
    constexpr uint32_t A = L::kAtoms;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sQ = base, *sK = sQ + L::kQ, *sV = sK + kStages * L::kTile;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kStages * L::kTile);
    Ctl* ctl = reinterpret_cast<Ctl*>(bars + 24);
    uint32_t* s_count = reinterpret_cast<uint32_t*>(ctl + 1);
    uint16_t* s_list = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(bars) + 256);   // see kTileMask
    const uint32_t k_full = smem_u32(bars), k_empty = k_full + 8u * kStages, v_full = k_empty + 8u * kStages,
                   v_empty = v_full + 8u * kStages, s_full = v_empty + 8u * kStages, p_full = s_full + 16u, pv_done = p_full + 16u,
                   drain = pv_done + 16u;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(k_full + 8u * s, 1u);
            mbar_init(k_empty + 8u * s, 1u);
            mbar_init(v_full + 8u * s, 1u);
            mbar_init(v_empty + 8u * s, 1u);
        }
        for (uint32_t s = 0; s < 2u; ++s) {
            mbar_init(s_full + 8u * s, 1u);
            mbar_init(p_full + 8u * s, kSoftmaxWarps);
            mbar_init(pv_done + 8u * s, 1u);   // two of them: S of tile j says that P V of tile j - 2 is complete, so a wait
        }                                      // for tile j - 1's own barrier meets it at most one phase behind
        mbar_init(drain, 1u);
        ctl->abort = 0u;
        fence_barrier_init();
    }
    if (warp == kWarpMma) tmem_alloc<false>(smem_u32(&ctl->tmem_base), kTmemCols);
    pdl_wait();
    const uint32_t z = blockIdx.x, hkv = blockIdx.y;
    const uint32_t G = pc.n_head / pc.n_head_kv, h0 = hkv * G, QT = kRows / G;
    // the last positions first: under a causal mask they have the most unmasked keys, and the grid is dealt in order
    const uint32_t q0 = (gridDim.z - 1u - blockIdx.z) * QT;
    const uint32_t key_begin = z * pc.split_keys, key_end = min(pc.n_kv, key_begin + pc.split_keys);
    const uint32_t n_tiles = key_end > key_begin ? (key_end - key_begin + kKeys - 1u) / kKeys : 0u;
    const float ninf = __uint_as_float(0xFF800000u);
    const float scale = __uint_as_float(pc.scale), softcap = __uint_as_float(pc.softcap);
    const bool q_vec = (vec & 1u) != 0u, m_vec = (vec & 2u) != 0u, o_vec = (vec & 4u) != 0u;

    // Q rows to fp16 in the K-major 128-byte swizzle; idle rows are zero. Eight rows of a warp in flight at once: this and the
    // scan below are chains of global loads in front of the first tile otherwise (23 of 82 us at 512 x 2048 positions).
    constexpr uint32_t kBatch = 8, kWarps = kThreads / 32u;
#pragma unroll 1
    for (uint32_t r0 = warp; r0 < kRows; r0 += kBatch * kWarps) {
        const uint32_t c = 4u * lane;   // (D = 64: the upper half of the warp idles)
        float4 x[kBatch];
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
            const uint32_t r = r0 + u * kWarps, iq = q0 + r / G;
            x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < (uint32_t)D && r < QT * G && iq < pc.n_q) {
                const float* row = q + pc.q_off + (uint64_t)iq * pc.q_s1 + (uint64_t)(h0 + r % G) * pc.q_s2;
                if (q_vec) x[u] = *reinterpret_cast<const float4*>(row + c);
                else x[u] = make_float4(row[c], row[c + 1u], row[c + 2u], row[c + 3u]);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
            const uint32_t r = r0 + u * kWarps, piece = (c & 63u) >> 3;
            if (c < (uint32_t)D && r < kRows)
                *reinterpret_cast<uint2*>(sQ + (c >> 6) * (kRows * 128u) + r * 128u + ((piece ^ (r & 7u)) << 4) + ((c & 4u) << 1)) =
                    make_uint2(pack_halves(x[u].x, x[u].y), pack_halves(x[u].z, x[u].w));
        }
    }
    fence_async_smem();   // the MMAs read Q through the async proxy
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Not earlier than the barrier that publishes the allocation: a CTA of the kernel behind this one could otherwise take the
    // tensor memory this CTA is still waiting for, and hold it while it waits for this grid.
    pdl_trigger();
    const uint32_t tmem = ctl->tmem_base, tmem_o = tmem + 2u * kKeys;

    // softmax state of this thread's row (warps 0-3)
    const uint32_t my_row = threadIdx.x;
    const uint32_t my_iq = q0 + my_row / G, my_head = h0 + my_row % G;
    const bool my_valid = my_row < QT * G && my_iq < pc.n_q;
    const __half* my_mask = mask;
    if (my_valid && pc.has_mask) my_mask += pc.m_off + (uint64_t)my_iq * pc.m_s1 + (uint64_t)(my_head % pc.m_ne2) * pc.m_s2;
    float m_run = ninf, l_run = 0.0f;
    // positions in the rings, kept across windows
    Ring kl(kStages), vl(kStages);       // loads
    Ring km(kStages), vm(kStages);       // MMAs
    uint32_t done = 0;                   // tiles processed by this role in earlier windows
    uint32_t k_issued = 0, v_issued = 0;
    bool ok = true;

    for (uint32_t w0 = 0; w0 < n_tiles; w0 += kWindow) {
        const uint32_t nw = min(kWindow, n_tiles - w0);
        // ---- scan: class of every tile of the window, kept in s_list as a dense array first, then compacted ----
        if (pc.has_mask) {
            // distinct mask rows of the CTA: one per position, or one per row when the heads have masks of their own
            const uint32_t positions = min(QT, pc.n_q - q0), n_rows = pc.m_ne2 == 1u ? positions : positions * G;
            for (uint32_t t = warp; t < nw; t += kThreads / 32u) {
                const uint32_t key0 = key_begin + (w0 + t) * kKeys;
                const bool whole = key0 + kKeys <= key_end;
                bool open = false, nonzero = !whole;
                const uint32_t sub = lane >> 3, piece = lane & 7u;   // four rows at a time, eight keys per lane
                auto mask_at = [&](uint32_t i) {   // this lane's eight keys of distinct row i
                    const uint32_t pos = pc.m_ne2 == 1u ? i : i / G, hd = pc.m_ne2 == 1u ? 0u : (h0 + i % G) % pc.m_ne2;
                    return mask + pc.m_off + (uint64_t)(q0 + pos) * pc.m_s1 + (uint64_t)hd * pc.m_s2 + key0 + 8u * piece;
                };
                if (m_vec && whole) {
#pragma unroll 1
                    for (uint32_t i0 = sub; i0 < n_rows; i0 += 4u * kBatch) {
                        uint4 v[kBatch];
#pragma unroll
                        for (uint32_t u = 0; u < kBatch; ++u) {   // (rows past the last repeat it)
                            const uint32_t i = i0 + 4u * u;
                            v[u] = *reinterpret_cast<const uint4*>(mask_at(i < n_rows ? i : i0));
                        }
#pragma unroll
                        for (uint32_t u = 0; u < kBatch; ++u) {
                            const uint32_t x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                open = open || x[k] != 0xFC00FC00u;
                                nonzero = nonzero || x[k] != 0u;
                            }
                        }
                    }
                } else {
                    for (uint32_t i = sub; i < n_rows; i += 4u) {
                        const __half* row = mask_at(i);
                        for (uint32_t k = 0; k < 8u; ++k) {
                            if (key0 + 8u * piece + k >= key_end) break;
                            const uint16_t x = *reinterpret_cast<const uint16_t*>(row + k);
                            open = open || x != 0xFC00u;
                            nonzero = nonzero || x != 0u;
                        }
                    }
                }
                const uint32_t seen = __ballot_sync(0xffffffffu, open);   // lanes 8 r + p: keys 8 p .. 8 p + 7
                nonzero = __any_sync(0xffffffffu, nonzero);
                uint32_t steps = 0;
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k) steps |= (seen & (0x03030303u << (2u * k))) ? 1u << k : 0u;
                if (lane == 0) s_list[t] = (uint16_t)(seen ? (t | steps << kStepShift | (nonzero ? kMixed : 0u)) : kNoTile);
            }
        } else {
            for (uint32_t t = threadIdx.x; t < nw; t += kThreads)
                s_list[t] = (uint16_t)(t | kAllSteps | (key_begin + (w0 + t + 1u) * kKeys <= key_end ? 0u : kMixed));
        }
        __syncthreads();
        if (warp == 0) {   // compaction in place: entries move to lower positions, 32 at a time
            uint32_t n = 0;
            for (uint32_t t = 0; t < nw; t += 32u) {
                const uint16_t e = t + lane < nw ? s_list[t + lane] : (uint16_t)kNoTile;
                const uint32_t keep = __ballot_sync(0xffffffffu, e != kNoTile);
                __syncwarp();
                if (e != kNoTile) s_list[n + __popc(keep & ((1u << lane) - 1u))] = e;
                __syncwarp();
                n += __popc(keep);
            }
            if (lane == 0) *s_count = n;
        }
        __syncthreads();
        const uint32_t n = *s_count;

        if (warp == kWarpLoad) {
            if (lane == 0) {
                for (uint32_t i = 0; i < n && ok; ++i) {
                    const int key0 = (int)(key_begin + (w0 + (s_list[i] & kTileMask)) * kKeys);
                    ok = mbar_wait(k_empty + 8u * kl.idx, kl.phase ^ 1u, ctl, status, 0xB00u);
                    if (!ok) break;
                    mbar_arrive_expect_tx(k_full + 8u * kl.idx, L::kTile);
                    for (uint32_t a = 0; a < A; ++a)
                        tma_load_3d(smem_u32(sK + kl.idx * L::kTile + a * (kKeys * 128u)), &k_map, k_full + 8u * kl.idx, (int)(64u * a),
                                    key0, (int)hkv);
                    ++k_issued;
                    kl.advance();
                    ok = mbar_wait(v_empty + 8u * vl.idx, vl.phase ^ 1u, ctl, status, 0xB10u);
                    if (!ok) break;
                    mbar_arrive_expect_tx(v_full + 8u * vl.idx, L::kTile);
                    for (uint32_t a = 0; a < A; ++a)
                        tma_load_3d(smem_u32(sV + vl.idx * L::kTile + a * (kKeys * 128u)), &v_map, v_full + 8u * vl.idx, (int)(64u * a),
                                    key0, (int)hkv);
                    ++v_issued;
                    vl.advance();
                }
            }
        } else if (warp == kWarpMma) {
            if (lane == 0) {
                const uint32_t idesc_s = make_idesc(1u, 0u, kKeys, kRows);
                const uint32_t idesc_o = make_idesc(1u, 0u, (uint32_t)D, kRows) | (1u << 16);   // B is MN-major
                auto issue_s = [&](uint32_t j) {   // S of tile number j (over all windows)
                    ok = mbar_wait<false>(k_full + 8u * km.idx, km.phase, ctl, status, 0xB20u);
                    if (!ok) return;
                    tc_fence_after();
#pragma unroll
                    for (uint32_t a = 0; a < A; ++a) {
                        const uint64_t da = make_smem_desc(smem_u32(sQ + a * (kRows * 128u)));
                        const uint64_t db = make_smem_desc(smem_u32(sK + km.idx * L::kTile + a * (kKeys * 128u)));
#pragma unroll
                        for (uint32_t k = 0; k < 4u; ++k)
                            umma_ss_f16(tmem + (j & 1u) * kKeys, da + 2u * k, db + 2u * k, idesc_s, (uint32_t)((a | k) != 0u));
                    }
                    umma_commit<false>(k_empty + 8u * km.idx);
                    umma_commit<false>(s_full + 8u * (j & 1u));
                    km.advance();
                };
                if (n && ok) issue_s(done);
                for (uint32_t i = 0; i < n && ok; ++i) {
                    const uint32_t j = done + i;
                    if (i + 1u < n) issue_s(j + 1u);
                    ok = ok && mbar_wait<false>(v_full + 8u * vm.idx, vm.phase, ctl, status, 0xB30u);
                    ok = ok && mbar_wait<false>(p_full + 8u * (j & 1u), (j >> 1) & 1u, ctl, status, 0xB40u);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t dv = make_v_desc(smem_u32(sV + vm.idx * L::kTile));
                    const uint32_t steps = (uint32_t)s_list[i] >> kStepShift;   // (at least one of a listed tile)
                    uint32_t acc = j != 0u;
#pragma unroll
                    for (uint32_t k = 0; k < kKeys / 16u; ++k) {   // 16 keys: 8 columns of P (high, then low), two groups of eight V rows
                        if (!(steps >> k & 1u)) continue;
                        const uint32_t ta = tmem + (j & 1u) * kKeys + 8u * k;
                        umma_ts<false, false>(tmem_o, ta, dv + 128u * k, idesc_o, acc);
                        umma_ts<false, false>(tmem_o, ta + 32u, dv + 128u * k, idesc_o, 1u);
                        acc = 1u;
                    }
                    umma_commit<false>(v_empty + 8u * vm.idx);
                    umma_commit<false>(pv_done + 8u * (j & 1u));
                    vm.advance();
                }
            }
        } else {
            const uint32_t lanes = (warp * 32u) << 16;
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t j = done + i, b = j & 1u, e = s_list[i];
                const uint32_t key0 = key_begin + (w0 + (e & kTileMask)) * kKeys;
                const bool mixed = (e & kMixed) != 0u;
                ok = ok && mbar_wait(s_full + 8u * b, (j >> 1) & 1u, ctl, status, 0xB50u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                float x[kKeys];
                tmem_ld32_async(tmem + lanes + b * kKeys, reinterpret_cast<uint32_t*>(x));
                tmem_ld32_async(tmem + lanes + b * kKeys + 32u, reinterpret_cast<uint32_t*>(x) + 32);
                tmem_wait_ld();
                const bool plain = !mixed && softcap == 0.0f && scale > 0.0f;   // the same for every thread of the CTA
                float mx = ninf;
                if (plain) {
#pragma unroll
                    for (uint32_t k = 0; k < kKeys; ++k) mx = fmaxf(mx, x[k]);
                    mx *= scale;
                } else {
                    const bool whole = key0 + kKeys <= key_end;
#pragma unroll
                    for (uint32_t p8 = 0; p8 < kKeys / 8u; ++p8) {
                        uint32_t mk[4] = {0u, 0u, 0u, 0u};   // eight mask values; -inf past the last key
                        if (m_vec && whole && pc.has_mask) {
                            if (my_valid) {
                                const uint4 v = *reinterpret_cast<const uint4*>(my_mask + key0 + 8u * p8);
                                mk[0] = v.x; mk[1] = v.y; mk[2] = v.z; mk[3] = v.w;
                            }
                        } else {
#pragma unroll
                            for (uint32_t k = 0; k < 8u; ++k) {
                                const uint32_t key = key0 + 8u * p8 + k;
                                uint32_t h = 0xFC00u;
                                if (key < key_end) h = (pc.has_mask && my_valid) ? *reinterpret_cast<const uint16_t*>(my_mask + key) : 0u;
                                mk[k >> 1] |= h << (16u * (k & 1u));
                            }
                        }
#pragma unroll
                        for (uint32_t k = 0; k < 8u; ++k) {
                            const float mv = h2f((uint16_t)(mk[k >> 1] >> (16u * (k & 1u))));
                            float xv = x[8u * p8 + k] * scale;
                            if (softcap != 0.0f) xv = softcap * tanhf(xv / softcap);
                            xv = mv == ninf ? ninf : xv + mv;
                            x[8u * p8 + k] = xv;
                            mx = fmaxf(mx, xv);
                        }
                    }
                }
                // a row whose maximum grew: its sum and accumulator move to the new reference
                const bool grow = mx > m_run + kGrowth || (m_run == ninf && mx != ninf);
                if (__any_sync(0xffffffffu, grow)) {
                    const float f = !grow ? 1.0f : m_run == ninf ? 0.0f : ex2((m_run - mx) * kLog2e);
                    if (grow) m_run = mx;
                    l_run *= f;
                    if (j != 0u) {
                        ok = mbar_wait(pv_done + 8u * ((j - 1u) & 1u), ((j - 1u) >> 1) & 1u, ctl, status, 0xB60u);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll 1
                        for (uint32_t c = 0; c < (uint32_t)D; c += 32u) {
                            uint32_t v[32];
                            tmem_ld32_async(tmem_o + lanes + c, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * f);
                            tmem_st32(tmem_o + lanes + c, v);
                        }
                    }
                }
                const float ref = (m_run == ninf ? 0.0f : m_run) * kLog2e, mul = plain ? scale * kLog2e : kLog2e;
                const float m_nat = m_run == ninf ? 0.0f : m_run;
                uint32_t ph[kKeys / 2u], pl[kKeys / 2u];   // P as fp16 and what that rounding left, again as fp16
                auto split = [&](uint32_t k, float p0, float p1) {
                    const __half2 h = __floats2half2_rn(p0, p1);
                    const float2 f = __half22float2(h);
                    ph[k] = *reinterpret_cast<const uint32_t*>(&h);
                    pl[k] = pack_halves(p0 - f.x, p1 - f.y);
                };
                float s0 = 0.0f, s1 = 0.0f;
                if (plain) {
#pragma unroll
                    for (uint32_t k = 0; k < kKeys / 2u; ++k) {
                        const float p0 = ex2(fmaf(x[2u * k], mul, -ref)), p1 = ex2(fmaf(x[2u * k + 1u], mul, -ref));
                        s0 += p0;
                        s1 += p1;
                        split(k, p0, p1);
                    }
                } else {   // the difference first: scores next to a large mask value keep their spacing
#pragma unroll
                    for (uint32_t k = 0; k < kKeys / 2u; ++k) {
                        const float p0 = ex2((x[2u * k] - m_nat) * kLog2e), p1 = ex2((x[2u * k + 1u] - m_nat) * kLog2e);
                        s0 += p0;
                        s1 += p1;
                        split(k, p0, p1);
                    }
                }
                l_run += s0 + s1;
                tmem_st32(tmem + lanes + b * kKeys, ph);   // over this tile's scores (waits for the stores)
                tmem_st32(tmem + lanes + b * kKeys + 32u, pl);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + 8u * b);
            }
        }
        done += n;
        __syncthreads();   // every role is done with the list (the loads and MMAs of its last tiles may still run)
    }

    // ---- results ----
    if (warp < kSoftmaxWarps) {
        if (done) ok = ok && mbar_wait(pv_done + 8u * ((done - 1u) & 1u), ((done - 1u) >> 1) & 1u, ctl, status, 0xB70u) && !ctl->abort;
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after();
            // through shared memory (Q's and K's, which no MMA reads any more), so that a row leaves as whole lines
            constexpr uint32_t kChunks = D / 4;
            float* stage = reinterpret_cast<float*>(base) + warp * 32u * D;
            const float inv = n_splits == 1u ? 1.0f / l_run : 1.0f;
            const uint32_t lanes = (warp * 32u) << 16;
            float check = 0.0f;   // NaN once a column is not finite
#pragma unroll 1
            for (uint32_t c = 0; c < (uint32_t)D; c += 32u) {
                uint32_t x[32];
                if (done) {
                    tmem_ld32_async(tmem_o + lanes + c, x);
                    tmem_wait_ld();
                } else {   // every key was masked: nothing was accumulated
#pragma unroll
                    for (int j = 0; j < 32; ++j) x[j] = 0u;
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) check = fmaf(__uint_as_float(x[j]), 0.0f, check);
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j)
                    reinterpret_cast<float4*>(stage)[lane * kChunks + (((c >> 2) + j) ^ (lane & 7u))] =
                        make_float4(__uint_as_float(x[4u * j]) * inv, __uint_as_float(x[4u * j + 1u]) * inv,
                                    __uint_as_float(x[4u * j + 2u]) * inv, __uint_as_float(x[4u * j + 3u]) * inv);
            }
            __syncwarp();
            // (a sum of probabilities that is not finite says that the scores are not: the row is NaN either way)
            for (uint32_t bad = __ballot_sync(0xffffffffu, my_valid && check != 0.0f && l_run - l_run == 0.0f); bad; bad &= bad - 1u) {
                const int i = __ffs(bad) - 1;
                const uint32_t r = warp * 32u + i, iq = q0 + r / G, head = h0 + r % G;
                const float m = __shfl_sync(0xffffffffu, m_run, i), f = __shfl_sync(0xffffffffu, inv, i);
                const __half* mrow = pc.has_mask ? mask + pc.m_off + (uint64_t)iq * pc.m_s1 + (uint64_t)(head % pc.m_ne2) * pc.m_s2 : nullptr;
                const float4 x = seen_keys_row<D>(q + pc.q_off + (uint64_t)iq * pc.q_s1 + (uint64_t)head * pc.q_s2,
                                                  k + pc.k_off + (uint64_t)hkv * pc.k_s2, v + pc.v_off + (uint64_t)hkv * pc.v_s2, mrow, pc.k_s1,
                                                  pc.v_s1, key_begin, key_end, scale, softcap, m == ninf ? 0.0f : m);
                const float y[4] = {x.x * f, x.y * f, x.z * f, x.w * f};
#pragma unroll
                for (uint32_t c = 0; c < D / 32u; ++c) {
                    const uint32_t e = lane * (D / 32u) + c;
                    stage[4u * (i * kChunks + ((e >> 2) ^ (i & 7u))) + (e & 3u)] = y[c];
                }
            }
            __syncwarp();
            for (uint32_t i = 0; i < 32u; ++i) {
                const uint32_t r = warp * 32u + i, iq = q0 + r / G;
                if (r >= QT * G || iq >= pc.n_q) break;   // (rows are ordered by position)
                const uint64_t orow = (uint64_t)iq * pc.n_head + h0 + r % G;
                float* dst = n_splits == 1u ? o + pc.o_off + orow * D
                                            : part + pc.part_off + ((uint64_t)z * pc.n_q * pc.n_head + orow) * (D + 4) + 4;
                if (o_vec || n_splits != 1u) {
                    if (lane < kChunks)
                        reinterpret_cast<float4*>(dst)[lane] = reinterpret_cast<const float4*>(stage)[i * kChunks + (lane ^ (i & 7u))];
                } else {
                    for (uint32_t e = lane; e < (uint32_t)D; e += 32u)
                        dst[e] = stage[4u * (i * kChunks + ((e >> 2) ^ (i & 7u))) + (e & 3u)];
                }
            }
            if (n_splits != 1u && my_valid) {
                float* pr = part + pc.part_off + ((uint64_t)z * pc.n_q * pc.n_head + (uint64_t)my_iq * pc.n_head + my_head) * (D + 4);
                pr[0] = m_run;
                pr[1] = l_run;
            }
        }
    } else if (lane == 0 && ctl->abort) {   // copies and MMAs already requested finish before the CTA leaves
        if (warp == kWarpLoad) {
            for (uint32_t i = k_issued > kStages ? k_issued - kStages : 0u; i < k_issued; ++i)
                mbar_wait(k_full + 8u * (i % kStages), (i / kStages) & 1u, ctl, status, 0xB80u);
            for (uint32_t i = v_issued > kStages ? v_issued - kStages : 0u; i < v_issued; ++i)
                mbar_wait(v_full + 8u * (i % kStages), (i / kStages) & 1u, ctl, status, 0xB90u);
        } else if (warp == kWarpMma) {
            umma_commit<false>(drain);
            for (uint32_t spins = 0; spins < 4096u && !mbar_try_wait(drain, 0u); ++spins) __nanosleep(64);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kWarpMma) tmem_dealloc<false>(tmem, kTmemCols);
}

// [heads][keys][D] fp16 with the caller's strides (elements, multiples of 8), boxes of 64 keys x 64 columns
static bool encode_kv(EncodeTiledFn enc, CUtensorMap* map, const void* ptr, uint32_t off, uint32_t D, uint32_t n_kv,
                      uint32_t n_head_kv, uint32_t s1, uint32_t s2) {
    const cuuint64_t dims[3] = {D, n_kv, n_head_kv};
    // (the stride of a dimension of one element is never used, but has to be a valid one)
    const cuuint64_t strides[2] = {n_kv > 1u ? 2ull * s1 : 2ull * D, n_head_kv > 1u ? 2ull * s2 : 2ull * D};
    const cuuint32_t box[3] = {64, kKeys, 1}, estr[3] = {1, 1, 1};
    if (!strides[0] || !strides[1]) return false;
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<char*>((const char*)ptr + 2ull * off), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D>
static bool launch_d(const LaunchArgs& a, const CUtensorMap& km, const CUtensorMap& vm, const FlashArgs& pc, uint32_t n_splits,
                     uint32_t q_tiles, uint32_t vec) {
    if (!ensure_dynamic_smem<flash_tc_kernel<D>>((int)Smem<D>::kBytes)) return false;
    launch_pdl(flash_tc_kernel<D>, dim3(n_splits, pc.n_head_kv, q_tiles), dim3(kThreads), Smem<D>::kBytes, a.stream, km, vm,
               (const float*)a.ptr[0], (const __half*)a.ptr[1], (const __half*)a.ptr[2], (const __half*)a.ptr[3], (float*)a.ptr[4],
               (float*)a.ptr[5], pc, n_splits, vec, a.status);
    return true;
}

}  // namespace ftc

bool flash_tc_maps(const LaunchArgs& a, const FlashArgs& pc, FlashMaps* maps) {
    tc::EncodeTiledFn enc = tc::encode_fn();
    return enc && ftc::encode_kv(enc, &maps->k, a.ptr[1], pc.k_off, pc.D, pc.n_kv, pc.n_head_kv, pc.k_s1, pc.k_s2) &&
           ftc::encode_kv(enc, &maps->v, a.ptr[2], pc.v_off, pc.D, pc.n_kv, pc.n_head_kv, pc.v_s1, pc.v_s2);
}

bool launch_flash_tc(const LaunchArgs& a, const FlashMaps& maps, const FlashArgs& pc, uint32_t n_splits, uint32_t q_tiles) {
    const uint32_t q_vec = !((pc.q_off | pc.q_s1 | pc.q_s2) & 3u) && !((uintptr_t)a.ptr[0] & 15u);
    const uint32_t m_vec = pc.has_mask && !((pc.m_off | pc.m_s1 | pc.m_s2) & 7u) && !((uintptr_t)a.ptr[3] & 15u);
    const uint32_t o_vec = !(pc.o_off & 3u) && !((uintptr_t)a.ptr[4] & 15u);
    const uint32_t vec = q_vec | m_vec << 1 | o_vec << 2;
    return pc.D == 64u ? ftc::launch_d<64>(a, maps.k, maps.v, pc, n_splits, q_tiles, vec)
                       : ftc::launch_d<128>(a, maps.k, maps.v, pc, n_splits, q_tiles, vec);
}

}  // namespace amv
